// Compile-time-sized line FFTs (the fast path of the solver's FFT engine).
//
// For a transform length N known at compile time, the radix plan, the
// per-stage butterfly counts, the thread -> butterfly mapping and every
// index division fold to constants.  T threads cooperate on one line; in pass
// s each runs ceil((N / R_s) / T) radix-R_s butterflies held in registers.
// Passes (called stages below) run in place: all butterfly inputs of a thread
// are loaded to registers, the block synchronises, and the outputs are
// written back to the same buffer, so a transform needs a single shared-
// memory tile (one buffer per field instead of a ping-pong pair).
#pragma once
#include "fft_engine.cuh"

namespace kwb {

// ---------------------------------------------------------------------------
// Radix plans.  The arithmetic of a transform is fixed by its length: the
// radices of the runtime-plan engine's first order (make_fft_plan: 16, then 8 /
// 4 / 2, then 7, 5, 3), each with its twiddles from the FP64-built table, so
// every plan of a length gives the same bits as that engine and a result does
// not depend on the plan, its variant or the tile.  What a plan chooses is how
// the radices are grouped into passes.  A pass costs each thread a read and a
// write of shared memory per point and two block barriers, so neighbouring
// radices are run on one set of registers (180 = 4 x 5 x 3 x 3 as (4 x 5)
// (3 x 3): two passes instead of four), and a radix of 16 or 8 may be split
// between two passes where that balances them: its first part is a smaller
// codelet on every (16 / part)-th input, the rest the radix-2 layers that the
// codelet would end with.
// The grouping of a length is found by exhaustive search with the cost model
// below.  Variant 1 is for grids too small to fill the device, where a step is
// a chain of latencies: the model then counts one thread's own work, so more
// threads share a line (128 = 16 x 8 as 4, 4, 8 on 32 threads instead of 8).
// ---------------------------------------------------------------------------
constexpr int kCtMaxSteps = 16;
struct CtStep {
  int r;       // this step's radix
  int radix;   // the radix it is a part of (r itself unless split)
  int done;    // product of the parts before it: 1 at the first, which has the twiddles
  bool open;   // first step of a pass
};
struct CtPlan {
  int nst;                // steps
  CtStep st[kCtMaxSteps];
  int s;                  // passes
  int t;                  // threads per line
};

__host__ __device__ constexpr int ct_codelet_cost(int r) {  // packed arithmetic instructions, roughly
  switch (r) {
    case 2: return 2;
    case 3: return 8;
    case 4: return 8;
    case 5: return 20;
    case 7: return 48;
    case 8: return 26;
    default: return 90;
  }
}

constexpr int kCtMaxHeld = 20;  // elements a thread holds at most (two registers each)

// Passes of a plan: radix and instructions of one butterfly each (loads,
// stores and addresses, distinct twiddle loads, twiddle products, codelets).
struct CtCost {
  int np;
  int radix[kCtMaxSteps];
  int work[kCtMaxSteps];
};
__host__ __device__ constexpr CtCost ct_passes(const CtPlan& p) {
  CtCost c{};
  for (int i = 0; i < p.nst; ++i) {
    if (p.st[i].open) {
      c.radix[c.np] = 1;
      c.work[c.np] = 12;
      ++c.np;
    }
    c.radix[c.np - 1] *= p.st[i].r;
  }
  int at = -1, in = 1;
  for (int i = 0; i < p.nst; ++i) {
    if (p.st[i].open) {
      ++at;
      in = 1;
      c.work[at] += 4 * c.radix[at];
    }
    const int r = p.st[i].r, nb = c.radix[at] / r;
    if (p.st[i].done == 1)
      c.work[at] += nb * ct_codelet_cost(r) + (i ? 2 * (r - 1) * in + 4 * (r - 1) * nb : 0);
    else
      c.work[at] += nb * (p.st[i].done == 2 ? 4 : 10);
    in *= r;
  }
  return c;
}

// Cost of a plan on t threads per line, -1 where a thread would hold too many
// elements.  Instructions of one thread, per line element it owns (variant 0:
// block throughput; 10 % more in a pass whose butterflies do not fill the
// threads evenly, 12 % where a thread holds over 16 elements, which costs
// occupancy) or in all (variant 1: latency, with 150 for a pass' barriers and
// shared-memory round trip and 60 per element for the work around the
// transform; up to 80 % more where threads have no butterfly in a pass), times
// 1000.  Runs of whole cases with the overhead of a pass, the held elements'
// share and the threads varied moved them by up to 20 %: 180 x 150 x 125 Stokes,
// 100 steps, 31.2 to 37.5 ms (125 as 5 x 5 x 5 on 25 or 9 threads), 432 x 360 x
// 288, 24 steps, 104.7 to 113.8 ms (432 on 48 or 27 threads).  Variant 1, us per
// 2D lossless step with a thread per butterfly of the widest pass or of any:
// 42 x 256 51 / 37, 1000 x 500 58 / 56, but 256 x 256 27 / 35, 64^3 69 / 82,
// where most threads then idle.
__host__ __device__ constexpr long long ct_plan_cost(int n, const CtCost& c, int t, int variant) {
  long long sum = 0;
  int held = 0, busy = 0;  // busy: thousandths of the threads, summed over the passes
  for (int i = 0; i < c.np; ++i) {
    const int nr = n / c.radix[i], nb = (nr + t - 1) / t;
    busy += 1000 * nr / (nb * t);
    held = nb * c.radix[i] > held ? nb * c.radix[i] : held;
    sum += variant ? nb * c.work[i] + 150 : nb * c.work[i] * (nr % t ? 11 : 10) + 150;
  }
  if (held > kCtMaxHeld) return -1;
  if (variant) return (sum + 60 * n / t) * (1800 - 800 * busy / (1000 * c.np));
  return sum * t * (held > 16 ? 112 : 100) / n;
}

__host__ __device__ constexpr void ct_rate(int n, CtPlan& p, CtPlan& best, long long& cost, int variant) {
  const CtCost c = ct_passes(p);
  if (c.np < 2) return;
  // threads per line: one butterfly each of any pass (variant 1), or 1 to 4
  const int most = variant ? 1 : 4;
  for (int i = 0; i < most * c.np; ++i) {
    const int nr = n / c.radix[i / most], nb = i % most + 1;
    const int t = (nr + nb - 1) / nb;
    if (t > 256) continue;
    const long long v = ct_plan_cost(n, c, t, variant);
    if (v >= 0 && (best.nst == 0 || v < cost)) {
      best = p;
      best.s = c.np;
      best.t = t;
      cost = v;
    }
  }
}

// Radices from `rest` on, of the current one `done` parts are in the plan;
// `width`: the radix of the pass under way, 0 where a new one must start.
__host__ __device__ constexpr void ct_search(int n, int rest, int radix, int done, int width, CtPlan& p, CtPlan& best,
                                             long long& cost, int variant) {
  if (p.nst == kCtMaxSteps) return;
  if (done == 1) {  // a new radix
    if (rest == 1) return ct_rate(n, p, best, cost, variant);
    constexpr int radices[7] = {16, 8, 4, 2, 7, 5, 3};
    for (int i = 0; i < 7; ++i)
      if (rest % radices[i] == 0) {
        radix = radices[i];
        break;
      }
    const int least = radix == 16 ? (variant ? 4 : 8) : (radix == 8 ? 4 : radix);
    for (int m = radix; m >= least; m /= 2)
      for (int open = 0; open < 2; ++open) {
        if (!open && (width == 0 || width * m > kCtMaxHeld)) continue;
        p.st[p.nst++] = CtStep{m, radix, 1, open == 1};
        if (m == radix)
          ct_search(n, rest / radix, 0, 1, open ? m : width * m, p, best, cost, variant);
        else  // the rest of the radix in the passes that follow
          ct_search(n, rest, radix, m, 0, p, best, cost, variant);
        --p.nst;
      }
    return;
  }
  int added = 0;
  for (int q = done; q < radix; q *= 2) {  // radix-2 layers
    p.st[p.nst++] = CtStep{2, radix, q, added++ == 0};
    if (2 * q == radix)
      ct_search(n, rest / radix, 0, 1, radix / done, p, best, cost, variant);
    else
      ct_search(n, rest, radix, 2 * q, 0, p, best, cost, variant);
  }
  p.nst -= added;
}

__host__ __device__ constexpr CtPlan ct_plan(int n, int variant) {
  CtPlan cur{}, best{};
  long long cost = 0;
  if (n > 1) ct_search(n, n, 0, 1, 0, cur, best, cost, variant);
  return best;
}

// Ct<N, V>: the plan of length N.
template <int N, int V = 0>
struct Ct {
  static constexpr CtPlan P = ct_plan(N, V);
  static constexpr int S = P.s;
  static constexpr int T = P.t;  // threads per line
  static_assert(S > 1, "transform length must factor into 2, 3, 5 and 7");
  static constexpr int first(int pass) {  // first step of a pass (pass S: the end)
    int at = -1;
    for (int i = 0; i < P.nst; ++i) {
      at += P.st[i].open;
      if (at == pass) return i;
    }
    return P.nst;
  }
  static constexpr int radix(int pass) {
    int r = 1;
    for (int i = first(pass); i < first(pass + 1); ++i) r *= P.st[i].r;
    return r;
  }
  static constexpr int ns(int pass) {  // product of the radices before `pass`
    int r = 1;
    for (int i = 0; i < first(pass); ++i) r *= P.st[i].r;
    return r;
  }
  static constexpr int held() {  // most elements a thread holds in a pass
    int h = 0;
    for (int i = 0; i < S; ++i) {
      const int v = (N / radix(i) + T - 1) / T * radix(i);
      h = v > h ? v : h;
    }
    return h;
  }
  static constexpr bool has7() {  // a radix-7 codelet (the heaviest)
    for (int i = 0; i < P.nst; ++i)
      if (P.st[i].r == 7) return true;
    return false;
  }
};

template <int V>
struct Ct<0, V> {
  static constexpr int S = 0, T = 1;
  static constexpr int radix(int) { return 1; }
  static constexpr int held() { return 16; }
};

// ---------------------------------------------------------------------------
// Tile shapes
// ---------------------------------------------------------------------------
// Columns per column tile: rows of 32 to 256 bytes in global memory (a
// multiple of 4 bins, so a tile's rows are whole 32-byte sectors), 128 to 400
// threads, and a tile of at most 36 KB.
__host__ __device__ constexpr int ct_col_lines(int n, int t) {
  int l = t <= 8 ? 32 : (t <= 20 ? 16 : (t <= 40 ? 8 : 4));
  while (l > 4 && l * n > 4608) l /= 2;
  return l;
}

// Row pairs per row tile: about 128 threads (variant 1: 64) in as few partly
// idle warps as possible; an even count where the threads per line are odd
// (the tile's element count is then even: 16-byte aligned bulk copies).
__host__ __device__ constexpr int ct_row_lines(int t, int variant) {
  const int lo = variant ? 32 : 80, hi = variant ? 96 : 160, mid = variant ? 64 : 128;
  int best = 1, best_score = -1000000;
  for (int l = 1; l * t <= hi || l == 1; ++l) {
    if (l * t < lo && (l + 1) * t <= hi) continue;
    if (l > 1 && (l & 1) && (t & 1)) continue;
    const int th = l * t, full = (th + 31) / 32 * 32;
    const int off = th > mid ? th - mid : mid - th;
    const int score = 1000 * th / full - off;
    if (score > best_score) {
      best_score = score;
      best = l;
    }
  }
  return best;
}

// Row tile layout: element (l, n) at l * LS + n + n / PAD.  One element of
// padding per 16 where the first pass' outputs, a multiple of 8 or 4 apart,
// would fall in a few banks; per 32 where they are 12 or 20 apart; none for
// lengths that are not multiples of 4, whose radices are odd or twice an odd
// number.  LS = T mod 16, so the lines that share a warp continue the bank
// sequence of a line's butterflies.  Counted over all passes' accesses:
// 1.0 to 1.7 shared-memory wavefronts per ideal one (up to 2.5 with padding
// per 16 at every length).
//
// at(base, l, n0, c, block): the index of element n0 + c given base = (l, n0),
// c and block compile-time constants once the stage loops are unrolled: base
// plus a constant where the padding allows it.  block > 0: n0 + c lies in the
// aligned block of that many elements that n0 lies in.
template <int N, int V = 0>
struct CtRow {
  static constexpr int shift() {
    if (N == 0) return 5;
    if (N % 4) return 10;  // none: lengths are at most 1024
    return Ct<N, V>::radix(0) % 8 == 0 || Ct<N, V>::radix(0) == 4 ? 4 : 5;
  }
  static constexpr int SH = shift();
  static constexpr int PAD = 1 << SH;
  static constexpr int stride() {
    int ls = N + ((N - 1) >> SH);
    if (N % 4 == 0 && ls < N + 4) ls = N + 4;  // two raw half-spectrum rows fit one line (RowBulk)
    // one line of an odd number of threads: an even stride, for the bulk copies' 16 bytes
    const int t = Ct<N, V>::T, even = N % 4 == 0 && t % 2 == 1 && ct_row_lines(t, V) == 1;
    while (ls % 16 != (t + even) % 16) ++ls;
    return ls;
  }
  static constexpr int LS = stride();
  __device__ __forceinline__ int operator()(int l, int n) const { return l * LS + n + (n >> SH); }
  __device__ __forceinline__ int at(int base, int l, int n0, int c, int block) const {
    if (PAD >= N || (block > 0 && PAD % block == 0)) return base + c;
    if (c % PAD == 0) return base + c + c / PAD;
    return (*this)(l, n0 + c);
  }
};

// Column tile layout: element (l, n) at n * TL + l.
template <int TL>
struct CtCol {
  __device__ __forceinline__ int operator()(int l, int n) const { return n * TL + l; }
  __device__ __forceinline__ int at(int base, int, int, int c, int) const { return base + c * TL; }
};

// ---------------------------------------------------------------------------
// Stages
// ---------------------------------------------------------------------------
// threadIdx.x made opaque to the optimiser: the word it is summed with is 0
// (tw[0] = exp(0) = 1), but only a shared-memory read at run time tells.  The
// transforms take the thread's butterfly index from it: without it ptxas
// hoists every stage's addresses out of a loop over a tile's fields and spills
// them (by ptxas' report when it came: k_x_eos at 540 points 132 against 72
// registers, k_x_rho at 144 points up to 0.9 KB of spills a thread).  Powers of two keep the plain index: their
// addresses are base + constant, and recomputing them cost k_x_u and k_x_rho
// 5 % at 256 points.
template <int N>
__device__ __forceinline__ int ct_tid(const float2* tw) {
  if constexpr ((N & (N - 1)) == 0)
    return (int)threadIdx.x;
  else
    return (int)threadIdx.x + (*reinterpret_cast<const volatile int*>(tw) - 0x3f800000);
}

// A pass of the plan: N / R butterflies of R points, NB per thread.
template <int N, int V, int PASS>
struct CtStage {
  static constexpr int LEN = N;
  using Plan = Ct<N, V>;
  static constexpr int FIRST = Plan::first(PASS), LAST = Plan::first(PASS + 1);  // its steps
  static constexpr int R = Plan::radix(PASS);
  static constexpr int NS = Plan::ns(PASS);
  static constexpr int NR = N / R;
  static constexpr int T = Plan::T;
  static constexpr int NB = (NR + T - 1) / T;
  static __device__ __forceinline__ bool has(int j) { return NR % T == 0 || j < NR; }
};

// One radix-2 layer of a split radix, between the `done` x 2 points of an even
// and an odd half: w = o exp(-+ pi i q / done), in the very operations of
// dft4, dft8 and dft16.
template <int N, int DONE, bool INV>
__device__ __forceinline__ float2 ct_layer_twiddle(float2 o, int q, const float2* __restrict__ tw) {
  if constexpr (DONE == 2) {
    const float2 t = c_rot<INV>(o);
    return q ? t : o;
  } else if constexpr (DONE == 4) {
    const float r = 0.707106781186547524400844362104849039f;
    const float s = r * (o.x + o.y), d = INV ? r * (o.x - o.y) : r * (o.y - o.x);
    const float2 odd = (q == 1) ? (INV ? make_float2(d, s) : make_float2(s, d))
                                : (INV ? make_float2(-s, d) : make_float2(d, -s));
    const float2 t = c_rot<INV>(o);
    return (q & 1) ? odd : (q ? t : o);
  } else {
    const float2 w = tw[q * (N / 16)];  // exp(-2 pi i q / 16)
    const float2 t = c_rot<INV>(o), m = w16_mul<INV>(o, make_float2(w.x, -w.y), q);
    return q == 4 ? t : m;
  }
}

// Steps STEP .. LAST - 1 of butterfly j, whose steps before (product IN) are
// done: element b * IN + q of v is output q of the sub-transform that holds
// inputs b, b + R / IN, ...  jk = j mod NS.  OTHER: the twiddles of the last
// radix take the other form of their product (c_twiddle).
template <class G, int STEP, int IN, bool INV, bool OTHER>
__device__ __forceinline__ void ct_steps(float2 (&v)[G::R], const float2* __restrict__ tw, int j, int jk) {
  if constexpr (STEP < G::LAST) {
    constexpr CtStep st = G::Plan::P.st[STEP];
    constexpr int r = st.r, left = G::R / IN, per = left / r;
    float2 w[G::R];
#pragma unroll
    for (int b = 0; b < per; ++b) {
#pragma unroll
      for (int q = 0; q < IN; ++q) {
        float2 x[r];
#pragma unroll
        for (int i = 0; i < r; ++i) x[i] = v[(b + i * per) * IN + q];
        if constexpr (st.done == 1) {
          constexpr int ns = G::NS * IN, sub = st.radix / r;  // sub: inputs of the radix between two of this part
          if constexpr (ns > 1) {
            constexpr int step = G::LEN / (ns * st.radix);
            const int base = (jk + q * G::NS) * step;
            // which of the `sub` interleaved parts: all of them lie in this
            // pass, or (a split radix ends its pass) one per thread
            const int h = sub == 1 ? 0 : j / (G::LEN / (st.radix * IN));
            static_assert(sub == 1 || per == 1, "a split radix ends its pass");
            if (G::NS > 1 || q > 0) {
#pragma unroll
              for (int i = 0; i < r; ++i) {
                if (sub == 1 && i == 0) continue;
                x[i] = c_twiddle<INV, OTHER && ns * st.radix == G::LEN>(x[i], tw[base * (i * sub + h)]);
              }
            }
          }
          dft<r, INV>(x);
        } else {
          // NS = (product before this radix) * (its parts before this pass)
          constexpr int before = st.done / IN, unit = G::NS / before;
          const float2 t = ct_layer_twiddle<G::LEN, st.done, INV>(x[1], jk / unit + q * before, tw);
          x[1] = c_sub(x[0], t);
          x[0] = c_add(x[0], t);
        }
#pragma unroll
        for (int i = 0; i < r; ++i) w[b * (IN * r) + q + IN * i] = x[i];
      }
    }
#pragma unroll
    for (int i = 0; i < G::R; ++i) v[i] = w[i];
    ct_steps<G, STEP + 1, IN * r, INV, OTHER>(v, tw, j, jk);
  }
}

// Butterfly j of a pass, twiddles included.
template <class G, bool INV, bool OTHER = false>
__device__ __forceinline__ void ct_butterfly(float2 (&v)[G::R], const float2* __restrict__ tw, int j) {
  ct_steps<G, G::FIRST, 1, INV, OTHER>(v, tw, j, G::NR <= G::NS ? j : j % G::NS);
}

// Inputs of a thread's butterflies from `buf`.
template <class G, class L>
__device__ __forceinline__ void ct_load(float2 (&v)[G::R], const float2* buf, int l, int j, L lay) {
  const int base = lay(l, j);
#pragma unroll
  for (int r = 0; r < G::R; ++r) v[r] = buf[lay.at(base, l, j, r * G::NR, 0)];
}

// Outputs of butterfly j to `buf`.
template <class G, class L>
__device__ __forceinline__ void ct_store(const float2 (&v)[G::R], float2* buf, int l, int j, L lay) {
  const int idx = (j / G::NS) * (G::NS * G::R) + j % G::NS;
  const int base = lay(l, idx);
#pragma unroll
  for (int r = 0; r < G::R; ++r) buf[lay.at(base, l, idx, r * G::NS, G::NS * G::R)] = v[r];
}

// One in-place stage: inputs to registers, barrier, outputs, barrier.
template <int N, int V, int STAGE, bool INV, bool OTHER = false, class L>
__device__ __forceinline__ void ct_stage(float2* buf, const float2* __restrict__ tw, int l, int tid, L lay) {
  using G = CtStage<N, V, STAGE>;
  float2 v[G::NB][G::R];
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    const int j = tid + i * G::T;
    if (G::has(j)) {
      ct_load<G>(v[i], buf, l, j, lay);
      ct_butterfly<G, INV, OTHER>(v[i], tw, j);
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    const int j = tid + i * G::T;
    if (G::has(j)) ct_store<G>(v[i], buf, l, j, lay);
  }
  __syncthreads();
}

// Stages FIRST .. LAST - 1.
template <int N, int V, int FIRST, int LAST, bool INV, bool OTHER = false, class L>
__device__ __forceinline__ void ct_stages(float2* buf, const float2* __restrict__ tw, int l, int tid, L lay) {
  if constexpr (FIRST < LAST) {
    ct_stage<N, V, FIRST, INV, OTHER>(buf, tw, l, tid, lay);
    ct_stages<N, V, FIRST + 1, LAST, INV, OTHER>(buf, tw, l, tid, lay);
  }
}

// The last stage with a caller-supplied output: st(pos, v) receives element
// pos of this thread's line.  No barriers.
template <int N, int V, bool INV, class L, class ST>
__device__ __forceinline__ void ct_last_st(const float2* buf, const float2* __restrict__ tw, int l, int tid, L lay,
                                           ST st) {
  using G = CtStage<N, V, Ct<N, V>::S - 1>;
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    const int j = tid + i * G::T;
    if (G::has(j)) {
      float2 v[G::R];
      ct_load<G>(v, buf, l, j, lay);
      ct_butterfly<G, INV>(v, tw, j);
#pragma unroll
      for (int r = 0; r < G::R; ++r) st(j + r * G::NS, v[r]);  // j < NS in the last stage
    }
  }
}

// The first stage with a caller-supplied loader: ld(l, j, c, span) returns
// input element j + c of line l, 0 <= j < span, c and span compile-time
// constants once unrolled, from wherever the caller keeps it (the row kernels
// build each packed line from two raw half-spectrum rows on the fly).  In
// place like ct_stage: every input is loaded before the block barrier and
// every output stored after it, so the inputs may alias the output buffer.
template <int N, int V, bool INV, class L, class LD>
__device__ __forceinline__ void ct_stage0_ld(float2* buf, const float2* __restrict__ tw, int l, int tid, L lay, LD ld) {
  using G = CtStage<N, V, 0>;
  float2 v[G::NB][G::R];
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    const int j = tid + i * G::T;
    if (G::has(j)) {
#pragma unroll
      for (int r = 0; r < G::R; ++r) v[i][r] = ld(l, j, r * G::NR, G::NR);
      ct_butterfly<G, INV>(v[i], tw, j);
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    const int j = tid + i * G::T;
    if (G::has(j)) ct_store<G>(v[i], buf, l, j, lay);
  }
  __syncthreads();
}

// From a forward transform through a spectral operator to an inverse one of
// the same line.  The operator is applied to the inputs of the inverse
// transform's first pass as a thread loads them: element i R + r of u is input
// r of its butterfly i, position pos(tid, m).  Where the forward transform's
// last pass leaves a thread the very positions its first inverse pass takes
// (DIRECT: both passes' butterflies fill the threads evenly, as for 64 = 16 x 4,
// 128 = 16 x 8 and 256 = 16 x 16) they stay in registers; otherwise they go
// through shared memory once.
template <int N, int V>
struct CtHandoff {
  using G = CtStage<N, V, Ct<N, V>::S - 1>;  // forward, last pass
  using H = CtStage<N, V, 0>;                // inverse, first pass
  static constexpr int M = H::NB * H::R;     // elements of u
  static constexpr bool DIRECT = G::NR % G::T == 0 && H::NR % H::T == 0;
  static __device__ __forceinline__ int pos(int tid, int m) {
    return tid + (m / H::R) * H::T + (m % H::R) * H::NR;
  }
  static __device__ __forceinline__ bool has(int tid, int m) { return H::has(tid + (m / H::R) * H::T); }
};

// Forward last pass of line `l` read from `src` into u (DIRECT).
template <int N, int V, bool OTHER, class L>
__device__ __forceinline__ void ct_fwd_last_to_regs(const float2* __restrict__ src, const float2* __restrict__ tw,
                                                    int l, int tid, L lay, float2 (&u)[CtHandoff<N, V>::M]) {
  using G = typename CtHandoff<N, V>::G;
  using H = typename CtHandoff<N, V>::H;
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    float2 v[G::R];
    ct_load<G>(v, src, l, tid + i * G::T, lay);
    ct_butterfly<G, false, OTHER>(v, tw, tid + i * G::T);
#pragma unroll
    for (int r = 0; r < G::R; ++r) {
      const int m = i + r * G::NB;  // position tid + m T
      u[(m % H::NB) * H::R + m / H::NB] = v[r];
    }
  }
}

// Inverse first pass from u; stores its outputs to `dst` for the next pass.
template <int N, int V, class L>
__device__ __forceinline__ void ct_inv_first_from_regs(float2 (&u)[CtHandoff<N, V>::M], const float2* __restrict__ tw,
                                                       float2* __restrict__ dst, int l, int tid, L lay) {
  using H = typename CtHandoff<N, V>::H;
#pragma unroll
  for (int i = 0; i < H::NB; ++i) {
    const int j = tid + i * H::T;
    if (H::has(j)) {
      float2 v[H::R];
#pragma unroll
      for (int r = 0; r < H::R; ++r) v[r] = u[i * H::R + r];
      ct_butterfly<H, true>(v, tw, j);
      ct_store<H>(v, dst, l, j, lay);
    }
  }
}

// In-place transform of LINES lines by T * LINES threads.  LINE_FAST maps
// consecutive threads to consecutive lines (column tiles, whose lines are
// adjacent in shared memory); otherwise to consecutive butterflies of one
// line (row tiles).  Must be called by every thread of the block (it
// synchronises); the caller synchronises before the call.
template <int N, int V, bool INV, bool LINE_FAST, int LINES, class L>
__device__ __forceinline__ void ct_fft(float2* buf, const float2* __restrict__ tw, L lay) {
  constexpr int T = Ct<N, V>::T;
  const int id = ct_tid<N>(tw);
  const int l = LINE_FAST ? id % LINES : id / T;
  const int tid = LINE_FAST ? id / LINES : id - l * T;
  ct_stages<N, V, 0, Ct<N, V>::S, INV>(buf, tw, l, tid, lay);
}

// Row tiles (consecutive threads on consecutive butterflies of a line): the
// first stage reads its inputs through `ld`, the others run in place.
template <int N, int V, bool INV, class L, class LD>
__device__ __forceinline__ void ct_fft_rows_ld(float2* buf, const float2* __restrict__ tw, L lay, LD ld) {
  constexpr int T = Ct<N, V>::T;
  const int id = ct_tid<N>(tw);
  const int l = id / T, tid = id - l * T;
  ct_stage0_ld<N, V, INV>(buf, tw, l, tid, lay, ld);
  ct_stages<N, V, 1, Ct<N, V>::S, INV>(buf, tw, l, tid, lay);
}

}  // namespace kwb
