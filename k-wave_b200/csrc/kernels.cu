// Solver kernels: size dispatch, the compile-time-length instantiations'
// lookup table, the runtime-plan instantiation (NC = 0) and the small
// elementwise kernels.  The FFT-carrying kernel templates are in
// kernels_impl.cuh; each compile-time length is instantiated in its own
// translation unit, generated by build.py from ct_sizes.h and ct_more_sizes.h.
#include <algorithm>
#include <cstdlib>

#include "ct_more_sizes.h"
#include "ct_sizes.h"
#include "kernels_impl.cuh"

namespace kwb {

#define KWB_EXTERN(N) extern template struct CtKernels<N>;
KWB_CT_SIZES(KWB_EXTERN)
KWB_CT_MORE_SIZES(KWB_EXTERN)
#undef KWB_EXTERN

// ---------------------------------------------------------------------------
// small elementwise kernels
// ---------------------------------------------------------------------------
// scatter one time sample of a source into a zeroed field
__global__ void k_scatter(float* f, const int* __restrict__ idx, const int* __restrict__ slot, int n,
                          const float* __restrict__ sig, int nrows_sig, int t, const float* __restrict__ weight) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int row = (nrows_sig == 1) ? 0 : slot[j];
  const float v = sig[(long long)(t - 1) * nrows_sig + row];
  f[idx[j]] = weight ? weight[j] * v : v;
}

// out[x, y] = in[x, y] * r[y] on a 2D grid (the axisymmetric u_r / r)
__global__ void k_scale_rows(float* __restrict__ out, const float* __restrict__ in, const float* __restrict__ r,
                             int nx, int ny, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = in[i] * r[(i / nx) % ny];
}

// Cartesian sensor points by linear interpolation: each point's value is
// the weighted sum of its simplex vertices' values recorded this step
// (kspaceFirstOrder_extractSensorData.m:296-420, sum(p(tri) .* bc, 2)),
// then the point's series / max / min / rms as for a grid sensor.
__global__ void k_interp_sensor(Sensor s, const float* __restrict__ vals, const int* __restrict__ vslot,
                                const float* __restrict__ w, int K, Clock clk) {
  const int fi = record_index(clk);
  if (fi <= 0) return;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < s.ns; j += gridDim.x * blockDim.x) {
    float v = 0.f;
    for (int k = 0; k < K; ++k) v += __ldg(w + (long long)j * K + k) * __ldg(vals + __ldg(vslot + (long long)j * K + k));
    sensor_put(s, fi, j, v);
  }
}

// rho_i = p0 / (dim c0^2) (kspaceFirstOrder3D.m:1027-1030, 2D.m:915-916);
// points whose density is stored merged (RhoBox) hold the sum dim * rho_i
// in r0 alone.
__global__ void k_rho_init(float* r0, float* r1, float* r2, const float* __restrict__ p0, Map c0sq, int dim,
                           RhoBox box, int nx, int ny, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = p0[i] / ((float)dim * c0sq.at(i));
    const long long row = i / nx;
    if (box.at((int)(i - row * nx), (int)(row % ny), (int)(row / ny), dim)) {
      r0[i] = (float)dim * v;
      continue;
    }
    r0[i] = v;
    r1[i] = v;
    if (dim == 3) r2[i] = v;
  }
}

// sensors from a materialised real field (initial-pressure step)
__global__ void k_record_field(const float* __restrict__ f, Sensor s, Clock clk, long long n) {
  const int fi = record_index(clk);
  if (fi <= 0) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = f[i];
    if (s.mode == 1) sensor_put(s, fi, i, v);
    sensor_all(s, fi, i, v);
  }
  if (s.mode == 2) {
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < s.ns;
         j += (long long)gridDim.x * blockDim.x)
      sensor_put(s, fi, s.slot[j], f[s.idx[j]]);
  }
}

__global__ void k_advance(int* t) {
  pdl_wait();  // the previous step's kernels have read the clock
  *t += 1;
}

// rms = sqrt(sum / n): the completed blocks' Kahan sum plus the partial sum
// of a block still in progress (partial != 0), kRmsBlock.
__global__ void k_rms_final(const float2* __restrict__ acc, const float* __restrict__ blk, int partial, float* out,
                            long long n, float inv_n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = sqrtf((acc[i].x + (partial ? blk[i] : 0.f)) * inv_n);
}

// Last axis without TMA: forward transform, multiply by `fanout` operators,
// inverse transform each product (runtime-plan engine, any length).
__global__ void __launch_bounds__(kThreads) k_fused_last(const __grid_constant__ FusedArgs a,
                                                         const __grid_constant__ FFTPlan plan,
                                                         const float2* __restrict__ tw_g,
                                                         const __grid_constant__ SpecTables T, int dim) {
  extern __shared__ __align__(16) float2 sm[];
  const int n = plan.n, tl = a.tl;
  float2* tw = sm;
  float2* A = sm + n;
  float2* B = A + tl * n;
  float2* C = B + tl * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) tw[i] = tw_g[i];
  const int g = blockIdx.z;
  const int outer = blockIdx.y;
  if (a.clock && threadIdx.x == 0 && blockIdx.x + outer + g == 0) *a.clock += 1;
  const long long off = (long long)outer * a.ostride;
  const float2* src = a.in[g] + off;
  const int c0 = blockIdx.x * tl;
  const int total = tl * n;
#pragma unroll 4
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int l = i % tl, p = i / tl, c = c0 + l;
    A[i] = (c < a.ncols) ? src[p * a.lstride + c] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const ColLayout lay{tl};
  float2* F = fft_lines<false, true>(A, B, tw, plan, tl, lay);
  float2* W1 = (F == A) ? B : A;
  for (int o = 0; o < a.fanout; ++o) {
    const SpecOp op = a.op[g * a.fanout + o];
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
      const int l = i % tl, p = i / tl;
      int c = c0 + l;
      if (c >= a.ncols) c = 0;
      const int iy = (dim == 3) ? outer : p;
      const int iz = (dim == 3) ? p : 0;
      W1[i] = c_op_mul(F[i], eval_op(op, T, dim, c, iy, iz));
    }
    __syncthreads();
    float2* R = fft_lines<true, true>(W1, C, tw, plan, tl, lay);
    float2* dst = a.out[g * a.fanout + o] + off;
    float2* dst2 = a.dual_out[g * a.fanout + o];
    const float2 dsc = dst2 ? __ldg(a.dual_tab[g * a.fanout + o] + outer) : make_float2(0.f, 0.f);
    if (dst2) dst2 += off;
#pragma unroll 4
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
      const int l = i % tl, p = i / tl, c = c0 + l;
      if (c < a.ncols) {
        dst[p * a.lstride + c] = R[i];
        if (dst2) dst2[p * a.lstride + c] = c_mul(R[i], dsc);
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// host-side launch helpers, dispatching on the transform length
// ---------------------------------------------------------------------------
namespace {

struct CtEntry {
  int n;
  decltype(&CtKernels<0>::col_fft) col_fft;
  decltype(&CtKernels<0>::x_u) x_u;
  decltype(&CtKernels<0>::x_rho) x_rho;
  decltype(&CtKernels<0>::x_eos) x_eos;
  decltype(&CtKernels<0>::x_r2c) x_r2c;
  decltype(&CtKernels<0>::x_c2r) x_c2r;
  decltype(&CtKernels<0>::threads_per_line) threads_per_line;
};

#define KWB_ENTRY(N)                                                                                  \
  {N, &CtKernels<N>::col_fft, &CtKernels<N>::x_u, &CtKernels<N>::x_rho,          \
   &CtKernels<N>::x_eos, &CtKernels<N>::x_r2c, &CtKernels<N>::x_c2r, &CtKernels<N>::threads_per_line},
const CtEntry kCtTable[] = {KWB_CT_SIZES(KWB_ENTRY) KWB_CT_MORE_SIZES(KWB_ENTRY)};
#undef KWB_ENTRY

const CtEntry kRuntime = {0,
                          &CtKernels<0>::col_fft,
                          &CtKernels<0>::x_u,
                          &CtKernels<0>::x_rho,
                          &CtKernels<0>::x_eos,
                          &CtKernels<0>::x_r2c,
                          &CtKernels<0>::x_c2r,
                          &CtKernels<0>::threads_per_line};

// the kernels of transform length n: compile-time if listed, else runtime
// (plan variant v < 0: runtime)
const CtEntry& kernels_for(int n, int v = 0) {
  if (v >= 0)
    for (const CtEntry& e : kCtTable)
      if (e.n == n) return e;
  return kRuntime;
}

}  // namespace

bool ct_supported(int n) { return kernels_for(n).n == n && n > 0; }

// The radix-plan variant (fft_ct.cuh) of `lines` transforms of length n per
// pass: 1 where variant 0 would leave most of the device idle (fewer than 240
// threads per SM, 35 520 in all).  us per step, variants 1 / 0 of every axis, at
// the threads a row pass of variant 0 has: 2D lossless 256^2 (2 k) 27 / 50, 768^2
// (18 k) 58 / 74, 1024 x 768 (25 k) 72 / 81, 900^2 (27 k) 89 / 96, 960^2 (31 k)
// 97 / 99, 800^2 (32 k) 72 / 72, 980^2 (34 k) 87 / 105, 1008^2 (36 k) 109 / 90; 3D
// lossless 64^3 (8 k) 48 / 76, 84^3 (21 k) 89 / 141, 100^3 (25 k) 127 / 129, 98^3
// (34 k) 138 / 159, 96^3 (37 k) 111 / 105, 90^3 (40 k) 138 / 115, 128^3 (66 k)
// 190 / 154.
constexpr long long kNarrowThreads = 148 * 240;
int plan_variant(int n, long long lines) {
  if (!ct_supported(n)) return 0;
  return lines * kernels_for(n).threads_per_line() < kNarrowThreads ? 1 : 0;
}

cudaError_t launch_col_fft(bool inv, const ColArgs& a, int nfields, long long nouter, const FFTPlan& plan,
                           const float2* tw, cudaStream_t st) {
  kernels_for(plan.n, a.v).col_fft(inv, a, nfields, nouter, plan, tw, st);
  return cudaGetLastError();
}

cudaError_t launch_fused_last(const FusedArgs& a, int ninputs, long long nouter, const FFTPlan& plan,
                              const float2* tw, const SpecTables& T, int dim, cudaStream_t st) {
  const dim3 grid((a.ncols + a.tl - 1) / a.tl, (unsigned)nouter, ninputs);
  const size_t sm = smem_col(plan.n, a.tl, 3);
  set_smem(k_fused_last, sm);
  k_fused_last<<<grid, kThreads, sm, st>>>(a, plan, tw, T, dim);
  return cudaGetLastError();
}

cudaError_t launch_x_u(const UArgs& a, const Dims& d, const FFTPlan& plan, const float2* tw, int L,
                       cudaStream_t st) {
  kernels_for(d.nx, d.v).x_u(a, d, plan, tw, L, st);
  return cudaGetLastError();
}

cudaError_t launch_x_rho(const RhoArgs& a, const Dims& d, const FFTPlan& plan, const float2* tw, int L,
                         cudaStream_t st) {
  kernels_for(d.nx, d.v).x_rho(a, d, plan, tw, L, st);
  return cudaGetLastError();
}

cudaError_t launch_x_eos(const EosArgs& a, const Dims& d, const FFTPlan& plan, const float2* tw, int L,
                         cudaStream_t st) {
  kernels_for(d.nx, d.v).x_eos(a, d, plan, tw, L, st);
  return cudaGetLastError();
}

cudaError_t launch_x_r2c(const float* f, float2* S, const Dims& d, const FFTPlan& plan, const float2* tw, int L,
                         cudaStream_t st) {
  kernels_for(d.nx, d.v).x_r2c(f, S, d, plan, tw, L, st);
  return cudaGetLastError();
}

cudaError_t launch_x_c2r(const float2* S, float* out, int accumulate, const Dims& d, const FFTPlan& plan,
                         const float2* tw, int L, cudaStream_t st) {
  kernels_for(d.nx, d.v).x_c2r(S, out, accumulate, d, plan, tw, L, st);
  return cudaGetLastError();
}

static inline unsigned ew_blocks(long long n) {
  long long b = (n + kThreads - 1) / kThreads;
  if (b > 148LL * 16) b = 148LL * 16;
  if (b < 1) b = 1;
  return (unsigned)b;
}

cudaError_t launch_scatter(float* f, const int* idx, const int* slot, int n, const float* sig, int nrows_sig,
                           int t, const float* weight, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_scatter<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(f, idx, slot, n, sig, nrows_sig, t, weight);
  return cudaGetLastError();
}

cudaError_t launch_interp_sensor(const Sensor& s, const float* vals, const int* vslot, const float* w, int K,
                                 const Clock& clk, cudaStream_t st) {
  if (s.mode == 0 || s.ns <= 0) return cudaSuccess;
  const int blocks = std::min((s.ns + kThreads - 1) / kThreads, 4096);
  k_interp_sensor<<<blocks, kThreads, 0, st>>>(s, vals, vslot, w, K, clk);
  return cudaGetLastError();
}

cudaError_t launch_scale_rows(float* out, const float* in, const float* r, int nx, int ny, long long n,
                              cudaStream_t st) {
  k_scale_rows<<<ew_blocks(n), kThreads, 0, st>>>(out, in, r, nx, ny, n);
  return cudaGetLastError();
}

cudaError_t launch_rho_init(float* r0, float* r1, float* r2, const float* p0, Map c0sq, int dim, const RhoBox& box,
                            int nx, int ny, long long n, cudaStream_t st) {
  k_rho_init<<<ew_blocks(n), kThreads, 0, st>>>(r0, r1, r2, p0, c0sq, dim, box, nx, ny, n);
  return cudaGetLastError();
}

cudaError_t launch_record_field(const float* f, const Sensor& s, const Clock& clk, long long n, cudaStream_t st) {
  k_record_field<<<ew_blocks(n), kThreads, 0, st>>>(f, s, clk, n);
  return cudaGetLastError();
}

cudaError_t launch_advance(int* t, cudaStream_t st) {
  const cudaError_t e = launch_pdl(k_advance, dim3(1), dim3(1), 0, st, t);
  return e != cudaSuccess ? e : cudaGetLastError();
}

bool pdl_enabled() {
  static const bool on = [] {
    const char* v = std::getenv("KWAVE_B200_NO_PDL");
    return !(v && v[0] == '1');
  }();
  return on;
}

// Medium maps from the uploaded sound speed (in place: c0 -> c0^2) and, for
// absorption, c0^2 tau and c0^2 eta in FP64 (kspaceFirstOrder_createAbsorptionVariables.m:27-99):
// tau = -2 a c0^(y-1), eta = 2 a c0^y tan(pi y / 2), a = alpha_coeff in Np
// (db2neper is linear in the coefficient: `np_per_db`).  eos 2 (Stokes): tau
// = -2 a c0 itself, with a for y = 2.
__global__ void k_medium_maps(float* c0_to_c0sq, float c0_scalar, float* ctau, float* ceta,
                              const float* __restrict__ alpha, float alpha_scalar, double np_per_db, double y,
                              double tan_py, int eos, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float cf = c0_to_c0sq ? c0_to_c0sq[i] : c0_scalar;
    const double c = (double)cf;
    if (ctau) {
      const double a = (double)(alpha ? alpha[i] : alpha_scalar) * np_per_db;
      if (eos == 1) {
        const double csq = (double)(cf * cf);
        const double cy1 = pow(c, y - 1.0);
        ctau[i] = (float)(csq * (double)(float)(-2.0 * a * cy1));
        ceta[i] = (float)(csq * (double)(float)(2.0 * a * cy1 * c * tan_py));
      } else {
        ctau[i] = (float)(-2.0 * a * c);
      }
    }
    if (c0_to_c0sq) c0_to_c0sq[i] = cf * cf;
  }
}

__global__ void k_reciprocal(float* v, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    v[i] = 1.0f / v[i];
}

cudaError_t launch_medium_maps(float* c0_to_c0sq, float c0_scalar, float* ctau, float* ceta, const float* alpha,
                               float alpha_scalar, double np_per_db, double y, double tan_py, int eos, long long n,
                               cudaStream_t st) {
  k_medium_maps<<<ew_blocks(n), kThreads, 0, st>>>(c0_to_c0sq, c0_scalar, ctau, ceta, alpha, alpha_scalar, np_per_db,
                                                   y, tan_py, eos, n);
  return cudaGetLastError();
}

cudaError_t launch_reciprocal(float* v, long long n, cudaStream_t st) {
  k_reciprocal<<<ew_blocks(n), kThreads, 0, st>>>(v, n);
  return cudaGetLastError();
}

cudaError_t launch_rms_final(const float2* acc, const float* blk, int partial, float* out, long long n, float inv_n,
                             cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_rms_final<<<ew_blocks(n), kThreads, 0, st>>>(acc, blk, partial, out, n, inv_n);
  return cudaGetLastError();
}

}  // namespace kwb
