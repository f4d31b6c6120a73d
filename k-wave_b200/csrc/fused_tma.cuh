// The TMA-fed fused last-axis operator (forward transform, k-space operator
// multiply, inverse transform) and the launchers of one length.
#pragma once
#include "col_tma.cuh"
#include "spec_ops.cuh"

namespace kwb {

// Operator classes of the fused kernel: one instantiation per class keeps
// only that operator's arithmetic in the kernel body.
enum FusedClass { FC_GRAD = 0, FC_NABLA = 1, FC_SRCK = 2 };

// The operations an operator is evaluated in, and so its rounding: from |k|^2
// (no square root) for the 2^a 3^b 5^c lengths from 64 to 256, whose results
// have always been rounded so; from |k|, the very operations of eval_op, for
// the others, so that they get the same bits here and in k_fused_last.
template <int N>
constexpr bool kOpFromK = N < 64 || N > 256 || N % 7 == 0;

// Blocks per SM the register budget is sized for: about 768 threads for the
// single-output pass, 512 otherwise and where a stage holds more than 16
// elements a thread or a radix is 7, which spill at 768.
template <int NC, int V, int MODE>
struct FusedBounds {
  static constexpr int TH = TTile<NC, V>::THREADS;
  static constexpr int WANT = MODE && Ct<NC, V>::held() <= 16 && !Ct<NC, V>::has7() ? 768 : 512;
  static constexpr int MIN_BLOCKS = WANT / TH > 0 ? WANT / TH : 1;
};

// MODE 1: every input has a single output (in place in the input stage: two
// tile buffers, three blocks per SM).
// MODE 0: the forward transform is kept and each output multiplied from it
// into a third buffer (two blocks per SM).
// The operator is applied in registers between the forward transform's last
// stage and the inverse's first (CtHandoff), and the inverse's last stage
// writes the output.  (The gradient's pair of outputs, kappa and kappa times
// the transform axis' derivative, also fits the in-place form with both taken
// from the hand-off registers, but at three blocks per SM that spills and
// measured slower at 256 points: 1.338 against 1.330 ms per 256^3 step.)
template <int NC, int V, int CLS, int MODE>
__global__ void __launch_bounds__(TTile<NC, V>::THREADS, FusedBounds<NC, V, MODE>::MIN_BLOCKS) k_fused_tma(const __grid_constant__ FusedTmaArgs a,
                                                                     const float2* __restrict__ tw_g,
                                                                     const __grid_constant__ SpecTables T) {
  constexpr int TL = TTile<NC, V>::LINES;
  constexpr int E = TTile<NC, V>::STRIDE;  // stage stride (the tile, padded to 128 bytes)
  constexpr int TH = TTile<NC, V>::THREADS;
  constexpr int S = Ct<NC, V>::S;
  extern __shared__ __align__(128) unsigned char smraw[];
  float2* inb = reinterpret_cast<float2*>(smraw);  // 2 input stages
  float2* W = MODE ? nullptr : inb + 2 * E;        // product / inverse-transform buffer (MODE 0)
  float2* tw = inb + (MODE ? 2 : 3) * E;
  uint64_t* bar = reinterpret_cast<uint64_t*>(tw + NC);
  // per-line tables of the transform axis: shifted derivatives (+, -) and k^2
  float2* dpos = reinterpret_cast<float2*>(bar + 2);
  float2* dneg = dpos + NC;
  float2* dsh = dneg + NC;
  float* kl2 = reinterpret_cast<float*>(dsh + NC);
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  const int lax = (a.dim == 3) ? 2 : 1;
  for (int i = threadIdx.x; i < NC; i += blockDim.x) {
    tw[i] = tw_g[i];
    kl2[i] = T.k2[lax][i];
    if constexpr (CLS == FC_GRAD) {
      dpos[i] = T.ddk_pos[lax][i];
      dneg[i] = T.ddk_neg[lax][i];
      dsh[i] = T.shift_neg[lax] ? T.shift_neg[lax][i] : make_float2(1.f, 0.f);
    }
  }
  __syncthreads();
  const int main_in = a.ncx * a.nouter;  // column tiles of one input
  const int per_in = main_in + a.nrem;
  const int ntiles = a.nin * per_in;
  // tile t -> input g and, for a column tile, its first column cx and outer
  // index o; a remainder tile has cx = -1 and its first outer index in o
  auto decode = [&](int t, int& g, int& cx, int& o) {
    g = t / per_in;
    const int r = t - g * per_in;
    if (r < main_in) {
      o = r / a.ncx;
      cx = r - o * a.ncx;
    } else {
      cx = -1;
      o = (r - main_in) * a.rem_y;
    }
  };
  __shared__ unsigned inflight, parity_bits;  // thread 0: as in k_col_tma
  if (threadIdx.x == 0) inflight = parity_bits = 0;
  auto issue = [&](int t, int j) {  // tile t, consumed at loop iteration j
    const int s = j & 1;
    int g, cx, o;
    decode(t, g, cx, o);
    mbar_expect_tx(&bar[s], TTile<NC, V>::BYTES);  // a remainder box holds as many bytes
    if (t == a.wait.skip_tile) return;  // test hook: announced, never issued
    if (cx >= 0) {
      tma_load_4d(inb + s * E, &a.in[g], cx * TL, 0, 0, o, &bar[s]);
    } else {
      tma_load_4d(inb + s * E, &a.in_rem[g], a.ncols - 1, o, 0, 0, &bar[s]);
    }
    inflight |= 1u << s;
    parity_bits = (parity_bits & ~(1u << s)) | ((unsigned)((j >> 1) & 1) << s);
  };
  pdl_wait();  // the inputs are the predecessors' outputs
  pdl_trigger();
  if (threadIdx.x == 0) {
    // the step's first kernel advances the clock: the previous step's kernels,
    // its last readers, have completed, and this step's wait for this one
    if (blockIdx.x == 0 && a.clock) *a.clock += 1;
    if (blockIdx.x < ntiles) issue(blockIdx.x, 0);
    if (blockIdx.x + gridDim.x < ntiles) issue(blockIdx.x + gridDim.x, 1);
  }
  const CtCol<TL> lay{};
  const float cdt2sq = T.cdt2 * T.cdt2;
  constexpr int TPL = TH / TL;  // threads per line
  using HO = CtHandoff<NC, V>;
  constexpr int M = HO::M;
  static_assert(TPL == Ct<NC, V>::T, "one line per group of T threads");
  bool aborted = false;
  int it = 0;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
    const int s = it & 1;
    float2* F = inb + s * E;
    const int id = ct_tid<NC>(tw), l = id % TL, tid = id / TL;
    int g, cx, o;
    decode(t, g, cx, o);
    // this thread's line: its column ix and outer index ol, where its
    // output goes (loff) and whether it is a real column (valid)
    int ix, ol;
    long long loff;
    bool valid;
    if (cx >= 0) {
      const int x0 = cx * TL;
      ix = min(x0 + l, a.ncols - 1);
      ol = o;
      loff = (long long)o * a.ostride + x0 + l;
      valid = (x0 + l) < a.ncols;
    } else {  // lines alternate the last column and the padding bin
      ix = a.ncols - 1;
      ol = o + (l >> 1);
      loff = (long long)ol * a.ostride + ix;
      valid = (l & 1) == 0;
    }
    const float kxy2 = __ldg(T.k2[0] + ix) + ((a.dim == 3) ? __ldg(T.k2[1] + ol) : 0.f);
    // the operator of output q: a real factor m(|k|^2), times a complex
    // factor that is constant along the line or read from a line table
    struct OpEval {
      float2 dconst;
      const float2* dline;
      float e;
      bool kappa;
    };
    auto setup = [&](int q) {
      const SpecOp op = a.op[g * a.fanout + q];
      OpEval ev{make_float2(1.f, 0.f), nullptr, 0.f, true};
      if constexpr (CLS == FC_GRAD) {
        if (op.kind != OP_KAPPA) {
          ev.kappa = op.kind != OP_SHIFT_NEG;  // the shift operator carries no kappa
          if (op.axis == lax) {
            ev.dline = (op.kind == OP_GRAD_POS) ? dpos : (op.kind == OP_GRAD_NEG ? dneg : dsh);
          } else {
            const float2* tab = (op.kind == OP_GRAD_POS)   ? T.ddk_pos[op.axis]
                                : (op.kind == OP_GRAD_NEG) ? T.ddk_neg[op.axis]
                                                           : T.shift_neg[op.axis];  // shift, kappa * shift
            ev.dconst = __ldg(tab + (op.axis == 0 ? ix : ol));
          }
        }
      } else if constexpr (CLS == FC_NABLA) {
        ev.e = (op.kind == OP_NABLA1) ? T.ym2 : T.ym1;
      }
      return ev;
    };
    // the operator of element p of the line on u; prescaled: u already holds
    // kappa * scale times the transform (GRAD)
    auto apply1 = [&](const OpEval& ev, float2 u, int p, bool prescaled) -> float2 {
      const float k2 = kxy2 + kl2[p];
      if constexpr (CLS == FC_GRAD) {
        const float2 d = ev.dline ? ev.dline[p] : ev.dconst;
        if constexpr (kOpFromK<NC>) {
          const float f = ev.kappa ? sinc_series(T.cdt2 * sqrtf(k2)) * T.scale : T.scale;
          return c_op_mul(u, make_float2(d.x * f, d.y * f));
        }
        if (prescaled) return c_op_mul(u, d);
        const float f = ev.kappa ? sinc_sq(cdt2sq * k2) * T.scale : T.scale;
        return c_op_mul(c_scale(u, f), d);
      } else {
        float f;
        if constexpr (CLS == FC_NABLA) {  // |k|^y = (|k|^2)^(y/2)
          const float k = kOpFromK<NC> ? sqrtf(k2) : k2, e = kOpFromK<NC> ? ev.e : 0.5f * ev.e;
          f = (k == 0.f) ? (e == 0.f ? T.scale : 0.f) : exp2f(e * log2f(k)) * T.scale;
        } else {
          f = (kOpFromK<NC> ? cos_series(T.cdt2 * sqrtf(k2)) : cos_sq(cdt2sq * k2)) * T.scale;
        }
        return c_scale(u, f);
      }
    };
    auto apply = [&](const OpEval& ev, float2 (&u)[M], bool prescaled = false) {
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (HO::has(tid, m)) u[m] = apply1(ev, u[m], HO::pos(tid, m), prescaled);
    };
    // inverse last stage, straight from W to the output (and the optional
    // second output scaled by a factor constant along the line)
    auto finish = [&](int q, const float2* src) {
      float2* dst = a.outp[g * a.fanout + q] + loff;
      float2* dst2 = a.dual_outp[g * a.fanout + q];
      float2 dsc = make_float2(0.f, 0.f);
      if (dst2) {
        dst2 += loff;
        dsc = __ldg(a.dual_tab[g * a.fanout + q] + ol);
      }
      auto st_g = [&](int pos, float2 v) {  // (the line is this thread's, folded into loff)
        if (valid) {
          dst[pos * a.lstride] = v;
          if (dst2) dst2[pos * a.lstride] = c_mul(v, dsc);
        }
      };
      ct_last_st<NC, V, true>(src, tw, l, tid, lay, st_g);
      fence_async_smem();  // the reads of src come before a TMA refill of it
      __syncthreads();     // src is reused by the next inverse
    };
    auto refill = [&]() {  // F is consumed: refill this input stage with the tile two ahead
      if (threadIdx.x == 0) {
        const int t2 = t + 2 * gridDim.x;
        if (t2 < ntiles) issue(t2, it + 2);
      }
    };
    const bool ok = mbar_wait(&bar[s], (it >> 1) & 1, a.err, a.wait.limit_ns);
    if (__syncthreads_or(!ok)) {  // every thread leaves together; nothing more is issued
      aborted = true;
      break;
    }
    if (threadIdx.x == 0) inflight &= ~(1u << s);
    float2 u[M];
    auto load_u = [&]() {  // the inverse transform's first inputs
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (HO::has(tid, m)) u[m] = F[lay(l, HO::pos(tid, m))];
    };
    if constexpr (MODE == 1) {
      // operator and inverse first stage in registers, the latter's outputs
      // back into F once every thread has read its inputs; inverse last
      // stage to the output; then F takes the tile two ahead
      constexpr bool OTHER = NC == 64 || NC == 128 || NC == 256;  // as their results have always been rounded
      if constexpr (HO::DIRECT) {
        ct_stages<NC, V, 0, S - 1, false, OTHER>(F, tw, l, tid, lay);
        ct_fwd_last_to_regs<NC, V, OTHER>(F, tw, l, tid, lay, u);
      } else {
        ct_stages<NC, V, 0, S, false, OTHER>(F, tw, l, tid, lay);
        load_u();
      }
      apply(setup(0), u);
      __syncthreads();
      ct_inv_first_from_regs<NC, V>(u, tw, F, l, tid, lay);
      __syncthreads();
      ct_stages<NC, V, 1, S - 1, true>(F, tw, l, tid, lay);
      finish(0, F);
      refill();
    } else {
      // several outputs of one input: the forward transform is kept in F; each
      // output's first inverse inputs are read from it, multiplied in
      // registers and given the inverse first stage on the way to W
      ct_stages<NC, V, 0, S, false>(F, tw, l, tid, lay);
      // a first output of kappa alone (the gradient pass: kappa P, then kappa
      // P times the axis derivative) leaves kappa * scale * F in F, so the
      // later outputs carrying kappa skip its evaluation (c_mul by 1 + 0i is
      // exact, so each output's value is unchanged)
      bool kf = false;
#pragma unroll 1
      for (int q = 0; q < a.fanout; ++q) {
        load_u();
        const OpEval ev = setup(q);
        apply(ev, u, kf && ev.kappa);
        if constexpr (CLS == FC_GRAD && !kOpFromK<NC>) {
          if (q == 0 && a.fanout > 1 && a.op[g * a.fanout].kind == OP_KAPPA) {
#pragma unroll
            for (int m = 0; m < M; ++m)
              if (HO::has(tid, m)) F[lay(l, HO::pos(tid, m))] = u[m];  // no other thread reads them
            kf = true;
          }
        }
        ct_inv_first_from_regs<NC, V>(u, tw, W, l, tid, lay);
        if (q + 1 == a.fanout) fence_async_smem();
        __syncthreads();
        if (q + 1 == a.fanout) refill();
        ct_stages<NC, V, 1, S - 1, true>(W, tw, l, tid, lay);
        finish(q, W);
      }
    }
  }
  if (threadIdx.x == 0 && aborted)  // the loads still in flight land before shared memory is released
    for (int s = 0; s < 2; ++s)
      if (inflight & (1u << s)) mbar_wait(&bar[s], (parity_bits >> s) & 1, nullptr, a.wait.limit_ns);
}

template <int NC, int V, int CLS, int MODE>
cudaError_t fused_tma_t(const FusedTmaArgs& a, const float2* tw, const SpecTables& T, cudaStream_t st) {
  const size_t sm = (MODE ? 2 : 3) * TTile<NC, V>::STRIDE * sizeof(float2) + NC * sizeof(float2) + 2 * sizeof(uint64_t) +
                    3 * NC * sizeof(float2) + NC * sizeof(float);
  auto k = k_fused_tma<NC, V, CLS, MODE>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, TTile<NC, V>::THREADS, sm);
  const int ntiles = a.nin * (a.ncx * a.nouter + a.nrem);
  const int grid = std::min(ntiles, std::max(1, per_sm) * tma_num_sms());
  const cudaError_t e = launch_pdl(k, dim3(grid), dim3(TTile<NC, V>::THREADS), sm, st, a, tw, T);
  return e != cudaSuccess ? e : cudaGetLastError();
}

// The fused last-axis pass of one length, dispatched on the plan variant and
// the operator class (MODE 0, several outputs per input, only for the
// gradient class).
template <int NC, int V>
cudaError_t fused_tma_v(const FusedTmaArgs& a, const float2* tw, const SpecTables& T, cudaStream_t st) {
  const int kind = a.op[0].kind;
  const bool one = a.fanout == 1;
  if (kind == OP_GRAD_POS || kind == OP_GRAD_NEG || kind == OP_KAPPA || kind == OP_SHIFT_NEG ||
      kind == OP_KAPPA_SHIFT_NEG) {
    return one ? fused_tma_t<NC, V, FC_GRAD, 1>(a, tw, T, st) : fused_tma_t<NC, V, FC_GRAD, 0>(a, tw, T, st);
  }
  if (!one) return cudaErrorInvalidValue;
  if (kind == OP_NABLA1 || kind == OP_NABLA2) return fused_tma_t<NC, V, FC_NABLA, 1>(a, tw, T, st);
  return fused_tma_t<NC, V, FC_SRCK, 1>(a, tw, T, st);
}

// The launchers of one length, on the plan variant the arguments name.
// Member functions are defined out of class (so not inline): each length is
// instantiated in its own translation unit (generated by build.py from
// tma_sizes.h and tma_more_sizes.h).
template <int NC>
struct TmaKernels {
  static int lines(int v);  // columns per tile
  static cudaError_t col(bool inv, const ColTmaArgs& a, const float2* tw, cudaStream_t st);
  static cudaError_t fused(const FusedTmaArgs& a, const float2* tw, const SpecTables& T, cudaStream_t st);
};
template <int NC>
int TmaKernels<NC>::lines(int v) {
  return v ? TTile<NC, 1>::LINES : TTile<NC, 0>::LINES;
}
template <int NC>
cudaError_t TmaKernels<NC>::col(bool inv, const ColTmaArgs& a, const float2* tw, cudaStream_t st) {
  if (a.v) return inv ? col_tma_t<NC, 1, true>(a, tw, st) : col_tma_t<NC, 1, false>(a, tw, st);
  return inv ? col_tma_t<NC, 0, true>(a, tw, st) : col_tma_t<NC, 0, false>(a, tw, st);
}
template <int NC>
cudaError_t TmaKernels<NC>::fused(const FusedTmaArgs& a, const float2* tw, const SpecTables& T, cudaStream_t st) {
  return a.v ? fused_tma_v<NC, 1>(a, tw, T, st) : fused_tma_v<NC, 0>(a, tw, T, st);
}

}  // namespace kwb
