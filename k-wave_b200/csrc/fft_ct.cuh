// Compile-time-sized line FFTs (the fast path of the solver's FFT engine).
//
// For a transform length N known at compile time, the radix plan, the
// per-stage butterfly counts, the thread -> butterfly mapping and every
// index division fold to constants.  T = N / RMAX threads cooperate on one
// line; in stage s each thread runs ceil((N / R_s) / T) radix-R_s butterflies
// held in registers.  Stages run in place: all butterfly inputs of a thread
// are loaded to registers, the block synchronises, and the outputs are
// written back to the same buffer, so a transform needs a single shared-
// memory tile (one buffer per field instead of a ping-pong pair).
#pragma once
#include "fft_engine.cuh"

namespace kwb {

// ---------------------------------------------------------------------------
// Radix plans.  A stage costs each thread a read and a write of shared memory
// per point, two block barriers, the twiddles and the butterflies, so few
// stages of large, nearly equal radices win (180 = 15 x 12 instead of
// 4 x 5 x 3 x 3: half the stages, and every thread busy in each).  The plan
// of a length is found by exhaustive search over its factorisations into the
// radices there are codelets for, largest first, with the cost model below.
// Variant 1 is for grids too small to fill the device, where a step is a
// chain of latencies: the model then counts one thread's own work, so more
// threads share a line (128 = 8 x 4 x 4 on 16 threads instead of 16 x 8 on 8).
// ---------------------------------------------------------------------------
constexpr int kCtMaxStages = 10;
struct CtPlan {
  int s;
  int r[kCtMaxStages];
};

__host__ __device__ constexpr int ct_codelet_cost(int r) {  // packed arithmetic instructions, roughly
  switch (r) {
    case 2: return 2;
    case 3: return 8;
    case 4: return 8;
    case 5: return 20;
    case 6: return 22;
    case 7: return 48;
    case 8: return 26;
    case 9: return 62;
    case 10: return 50;
    case 12: return 56;
    case 14: return 110;
    case 15: return 100;
    default: return 86;
  }
}

// Instructions of one thread per line element it owns (variant 0: block
// throughput) or in all (variant 1: latency, with 150 for a stage's barriers
// and shared-memory round trip and 60 per element for the work around the
// transform), times 1000.  (250 and 40, fewer stages on fewer threads, was
// slower: 128 x 128 lossless 32 against 25 us per step, 64 x 72 x 80
// absorbing 124 against 96.)
__host__ __device__ constexpr long long ct_plan_cost(int n, const CtPlan& p, int variant) {
  int rmax = 1;
  for (int i = 0; i < p.s; ++i) rmax = p.r[i] > rmax ? p.r[i] : rmax;
  const int t = n / rmax;
  long long c = 0;
  for (int i = 0; i < p.s; ++i) {
    const int r = p.r[i], nb = (n / r + t - 1) / t;
    c += nb * (4 * r + (i ? 6 * (r - 1) : 0) + ct_codelet_cost(r) + 12) + (variant ? 150 : 40);
  }
  return variant ? 1000 * (c + 60 * rmax) : 1000 * c / rmax;
}

__host__ __device__ constexpr void ct_search(int n, int rest, int first, CtPlan& cur, CtPlan& best, long long& cost,
                                             int variant) {
  constexpr int radices[13] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  if (rest == 1) {
    const long long c = ct_plan_cost(n, cur, variant);
    if (best.s == 0 || c < cost) {
      best = cur;
      cost = c;
    }
    return;
  }
  if (cur.s == kCtMaxStages) return;
  for (int i = first; i < 13; ++i) {
    if (rest % radices[i]) continue;
    cur.r[cur.s++] = radices[i];
    ct_search(n, rest / radices[i], i, cur, best, cost, variant);
    --cur.s;
  }
}

__host__ __device__ constexpr CtPlan ct_plan(int n, int variant) {
  CtPlan cur{}, best{};
  long long cost = 0;
  if (n > 1) ct_search(n, n, 0, cur, best, cost, variant);
  return best;
}

// Ct<N, V>: the plan of length N.  REV (below) runs its stages in the opposite
// radix order, so that an inverse transform can start from the registers a
// forward one ends in (CtHandoff).
template <int N, int V = 0>
struct Ct {
  static constexpr CtPlan P = ct_plan(N, V);
  static constexpr int S = P.s;
  static_assert(S > 0, "transform length must factor into 2, 3, 5 and 7");
  static constexpr int rmax() {
    int r = 1;
    for (int i = 0; i < P.s; ++i) r = P.r[i] > r ? P.r[i] : r;
    return r;
  }
  static constexpr int RMAX = rmax();
  static constexpr int T = N / RMAX;  // threads per line
  static constexpr int held() {       // most elements a thread holds in a stage
    int h = 0;
    for (int i = 0; i < P.s; ++i) {
      const int v = (N / P.r[i] + T - 1) / T * P.r[i];
      h = v > h ? v : h;
    }
    return h;
  }
  static constexpr bool has7() {  // a radix-7 or radix-14 stage (the heaviest codelets)
    for (int i = 0; i < P.s; ++i)
      if (P.r[i] % 7 == 0) return true;
    return false;
  }
  static constexpr int radix(int stage, bool rev) { return rev ? P.r[S - 1 - stage] : P.r[stage]; }
  static constexpr int ns(int stage, bool rev) {  // product of the radices before `stage`
    int p = 1;
    for (int i = 0; i < stage; ++i) p *= radix(i, rev);
    return p;
  }
};

template <int V>
struct Ct<0, V> {
  static constexpr int S = 0, RMAX = 1, T = 1;
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
// padding per 16 where the first radix is 16 (its outputs, 16 apart, would all
// fall in one bank), per 32 otherwise; and LS = T mod 16, so the lines that
// share a warp continue the bank sequence of a line's butterflies.  Over the
// lengths this gives 1.0-1.6 shared-memory wavefronts per ideal one (the same
// layout with LS = n + n / 16 + 1: 2 to 6).
//
// at(base, l, n0, c, block): the index of element n0 + c given base = (l, n0),
// c and block compile-time constants once the stage loops are unrolled: base
// plus a constant where the padding allows it.  block > 0: n0 + c lies in the
// aligned block of that many elements that n0 lies in.
template <int N, int V = 0>
struct CtRow {
  static constexpr int SH = (N > 0 && Ct<N, V>::RMAX == 16) ? 4 : 5;
  static constexpr int PAD = 1 << SH;
  static constexpr int stride() {
    int ls = N + ((N - 1) >> SH);
    if (N % 4 == 0 && ls < N + 4) ls = N + 4;  // two raw half-spectrum rows fit one line (RowBulk)
    while (ls % 16 != Ct<N, V>::T % 16) ++ls;
    return ls;
  }
  static constexpr int LS = stride();
  __device__ __forceinline__ int operator()(int l, int n) const { return l * LS + n + (n >> SH); }
  __device__ __forceinline__ int at(int base, int l, int n0, int c, int block) const {
    if (block > 0 && PAD % block == 0) return base + c;
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
// them (k_x_eos at 540 points 132 against 72 registers, k_x_rho at 144 points
// up to 0.9 KB of spills a thread).  Powers of two keep the plain index: their
// addresses are base + constant, and recomputing them cost k_x_u and k_x_rho
// 5 % at 256 points.
template <int N>
__device__ __forceinline__ int ct_tid(const float2* tw) {
  if constexpr ((N & (N - 1)) == 0)
    return (int)threadIdx.x;
  else
    return (int)threadIdx.x + (*reinterpret_cast<const volatile int*>(tw) - 0x3f800000);
}

// Butterflies per thread in a stage.
template <int N, int V, int STAGE, bool REV>
struct CtStage {
  static constexpr int R = Ct<N, V>::radix(STAGE, REV);
  static constexpr int NS = Ct<N, V>::ns(STAGE, REV);
  static constexpr int NR = N / R;
  static constexpr int T = Ct<N, V>::T;
  static constexpr int NB = (NR + T - 1) / T;
  static constexpr int TWS = N / (NS * R);
  static __device__ __forceinline__ bool has(int j) { return NR % T == 0 || j < NR; }
};

// Twiddles and butterfly j of a stage.
template <class G, bool INV>
__device__ __forceinline__ void ct_butterfly(float2 (&v)[G::R], const float2* __restrict__ tw, int j) {
  if constexpr (G::NS > 1) {
    const int step = (j % G::NS) * G::TWS;
#pragma unroll
    for (int r = 1; r < G::R; ++r) {
      float2 w = tw[step * r];
      if (INV) w.y = -w.y;
      v[r] = c_mul(v[r], w);
    }
  }
  dft<G::R, INV>(v);
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
template <int N, int V, int STAGE, bool INV, bool REV, class L>
__device__ __forceinline__ void ct_stage(float2* buf, const float2* __restrict__ tw, int l, int tid, L lay) {
  using G = CtStage<N, V, STAGE, REV>;
  float2 v[G::NB][G::R];
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    const int j = tid + i * G::T;
    if (G::has(j)) {
      ct_load<G>(v[i], buf, l, j, lay);
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

// Stages FIRST .. LAST - 1.
template <int N, int V, int FIRST, int LAST, bool INV, bool REV, class L>
__device__ __forceinline__ void ct_stages(float2* buf, const float2* __restrict__ tw, int l, int tid, L lay) {
  if constexpr (FIRST < LAST) {
    ct_stage<N, V, FIRST, INV, REV>(buf, tw, l, tid, lay);
    ct_stages<N, V, FIRST + 1, LAST, INV, REV>(buf, tw, l, tid, lay);
  }
}

// The last stage with a caller-supplied output: st(pos, v) receives element
// pos of this thread's line.  No barriers.
template <int N, int V, bool INV, bool REV, class L, class ST>
__device__ __forceinline__ void ct_last_st(const float2* buf, const float2* __restrict__ tw, int l, int tid, L lay,
                                           ST st) {
  using G = CtStage<N, V, Ct<N, V>::S - 1, REV>;
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
__device__ __forceinline__ void ct_stage0_ld(float2* buf, int l, int tid, L lay, LD ld) {
  using G = CtStage<N, V, 0, false>;
  float2 v[G::NB][G::R];
#pragma unroll
  for (int i = 0; i < G::NB; ++i) {
    const int j = tid + i * G::T;
    if (G::has(j)) {
#pragma unroll
      for (int r = 0; r < G::R; ++r) v[i][r] = ld(l, j, r * G::NR, G::NR);
      ct_butterfly<G, INV>(v[i], nullptr, j);  // first stage: no twiddles
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

// Register hand-off between a forward transform and an inverse one of the
// same line.  The forward transform runs its stages in the opposite radix
// order (REV), so its last stage has the largest radix, one butterfly per
// thread, and leaves butterfly tid's outputs at positions tid + T m, m <
// RMAX; the inverse transform's first stage has the same radix and its
// butterfly tid reads exactly those positions.  So the thread that ends the
// one starts the other, and a spectral operator is applied in between in
// registers with no shared-memory pass, for every length.
template <int N, int V>
struct CtHandoff {
  using G = CtStage<N, V, Ct<N, V>::S - 1, true>;  // forward, last stage
  using H = CtStage<N, V, 0, false>;               // inverse, first stage
  static constexpr int M = Ct<N, V>::RMAX;         // positions per thread
  static_assert(Ct<N, V>::S >= 2 && G::NB == 1 && H::NB == 1 && G::R == M && H::R == M && G::NS == Ct<N, V>::T &&
                    H::NR == Ct<N, V>::T,
                "the last and first stages face each other");
};

// Forward last stage of line `l` read from `src`; u[m] receives position tid + T m.
template <int N, int V, class L>
__device__ __forceinline__ void ct_fwd_last_to_regs(const float2* __restrict__ src, const float2* __restrict__ tw,
                                                    int l, int tid, L lay, float2 (&u)[CtHandoff<N, V>::M]) {
  using G = typename CtHandoff<N, V>::G;
  ct_load<G>(u, src, l, tid, lay);
  ct_butterfly<G, false>(u, tw, tid);
}

// Inverse first stage from u; stores its outputs to `dst` for the next stage.
template <int N, int V, class L>
__device__ __forceinline__ void ct_inv_first_from_regs(float2 (&u)[CtHandoff<N, V>::M], float2* __restrict__ dst,
                                                       int l, int tid, L lay) {
  using H = typename CtHandoff<N, V>::H;
  ct_butterfly<H, true>(u, nullptr, tid);
  ct_store<H>(u, dst, l, tid, lay);
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
  ct_stages<N, V, 0, Ct<N, V>::S, INV, false>(buf, tw, l, tid, lay);
}

// Row tiles (consecutive threads on consecutive butterflies of a line): the
// first stage reads its inputs through `ld`, the others run in place.
template <int N, int V, bool INV, class L, class LD>
__device__ __forceinline__ void ct_fft_rows_ld(float2* buf, const float2* __restrict__ tw, L lay, LD ld) {
  constexpr int T = Ct<N, V>::T;
  const int id = ct_tid<N>(tw);
  const int l = id / T, tid = id - l * T;
  ct_stage0_ld<N, V, INV>(buf, l, tid, lay, ld);
  ct_stages<N, V, 1, Ct<N, V>::S, INV, false>(buf, tw, l, tid, lay);
}

}  // namespace kwb
