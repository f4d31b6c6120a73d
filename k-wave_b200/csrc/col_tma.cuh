// The TMA-fed y pass: a persistent, pipelined column transform, and the tile
// geometry it shares with the fused last-axis operator.
//
// Each thread block loops over column tiles (TL adjacent kx columns x the
// whole line).  Tiles arrive by cp.async.bulk.tensor into a ring of shared
// memory stages while the previous tile is being transformed, and leave by
// bulk tensor stores, so the memory system streams continuously instead of
// stalling on each block's load phase.  The shared-memory tile layout
// [position][column] is exactly the TMA box layout and the column layout
// the in-place FFT engine uses.
#pragma once
#include <algorithm>

#include "fft_ct.cuh"
#include "kernels.cuh"
#include "kernels_tma.cuh"
#include "tma.cuh"

namespace kwb {

int tma_num_sms();  // multiprocessors of the current device

// Lines per TMA tile: the column tile's, a multiple of 4, so every tile starts
// at a bin index x = cx * LINES whose byte offset (8-byte bins) is a multiple
// of 32 (tensor copies require 16).
template <int NC, int V>
struct TTile {
  static constexpr int LINES = ct_col_lines(NC, Ct<NC, V>::T);
  static constexpr int THREADS = Ct<NC, V>::T * LINES;
  static constexpr int ELEMS = LINES * NC;
  static constexpr unsigned BYTES = ELEMS * sizeof(float2);
  // Stage stride in elements: tensor copies read and write shared memory at
  // 128-byte aligned addresses, so each stage is padded to a multiple of 128
  // bytes.
  static constexpr int STRIDE = (int)((BYTES + 127u) / 128u * 128u / sizeof(float2));
};

// Shared-memory stages of the y pass: tiles t + grid and t + 2 grid load
// while tile t is transformed and stored (two blocks per SM at 256 points).
// Two stages, three blocks per SM, measured slower at 256^3 (1.348 against
// 1.336 ms per step).
constexpr int kColStages = 3;

// Blocks per SM the register budget is sized for: as many as three stages of
// shared memory allow, at most about 640 threads (512 where a stage holds more
// than 16 elements a thread); without a bound ptxas takes up to 190 registers,
// which leaves one block per SM.
template <int NC, int V>
struct ColBounds {
  static constexpr int TH = TTile<NC, V>::THREADS;
  static constexpr int BY_REGS = (Ct<NC, V>::held() <= 16 ? 640 : 512) / TH;
  static constexpr int BY_SMEM = (int)(220 * 1024 / (kColStages * TTile<NC, V>::STRIDE * sizeof(float2) + 9 * NC));
  static constexpr int MIN_BLOCKS = BY_REGS < 1 || BY_SMEM < 1 ? 1 : (BY_REGS < BY_SMEM ? BY_REGS : BY_SMEM);
};

template <int NC, int V, bool INV>
__global__ void __launch_bounds__(TTile<NC, V>::THREADS, ColBounds<NC, V>::MIN_BLOCKS) k_col_tma(const __grid_constant__ ColTmaArgs a,
                                                                const float2* __restrict__ tw_g) {
  constexpr int TL = TTile<NC, V>::LINES;
  constexpr int E = TTile<NC, V>::STRIDE;  // stage stride (the tile, padded to 128 bytes)
  constexpr int ST = kColStages;
  extern __shared__ __align__(128) unsigned char smraw[];
  float2* bufs = reinterpret_cast<float2*>(smraw);
  float2* tw = bufs + ST * E;
  uint64_t* bar = reinterpret_cast<uint64_t*>(tw + NC);
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) mbar_init(&bar[s], 1);
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i < NC; i += blockDim.x) tw[i] = tw_g[i];
  __syncthreads();
  const int per_field = a.ncx * a.nouter;
  const int ntiles = a.nfields * per_field;
  // Tiles are numbered f * per_field + r (field f, position r).  Without a
  // derived field, block b takes tiles b, b + grid, ...  With one, block b
  // takes positions b, b + grid, ... and at each position every field,
  // the derived field first: its load from the source field and the source
  // field's own load both come before the source tile is stored back in
  // place, in one block's program order, and the second load hits L2.
  const bool grouped = a.dual_field >= 0;
  auto tile_at = [&](int k) -> int {  // this block's k-th tile, -1 past the end
    if (!grouped) {
      const int t = blockIdx.x + k * gridDim.x;
      return t < ntiles ? t : -1;
    }
    const int q = k / a.nfields, j = k - q * a.nfields;
    const int r = blockIdx.x + q * gridDim.x;
    if (r >= per_field) return -1;
    const int f = (j == 0) ? a.dual_field : (j - 1 < a.dual_field ? j - 1 : j);
    return f * per_field + r;
  };
  auto coords = [&](int t, int& f, int& x, int& o) {  // field, first column, outer index
    f = t / per_field;
    const int r = t - f * per_field;
    const int q = r / a.ncx;
    x = (r - q * a.ncx) * TL;
    o = a.outer0 + q;
  };
  // thread 0's record of the stages with a load in flight (bit s) and the
  // parity of each one's pending phase, for the drain after a failed wait
  // (in shared memory: it costs no registers in the transform loop)
  __shared__ unsigned inflight, parity_bits;
  if (threadIdx.x == 0) inflight = parity_bits = 0;
  auto issue = [&](int t, int j) {  // tile t, consumed at loop iteration j
    const int s = j % ST;
    int f, x, o;
    coords(t, f, x, o);
    mbar_expect_tx(&bar[s], TTile<NC, V>::BYTES);
    if (t == a.wait.skip_tile) return;  // test hook: announced, never issued
    tma_load_4d(bufs + s * E, &a.map[f == a.dual_field ? a.dual_src : f], x, 0, 0, o, &bar[s]);
    inflight |= 1u << s;
    parity_bits = (parity_bits & ~(1u << s)) | ((unsigned)((j / ST) & 1) << s);
  };
  if (threadIdx.x == 0)
    for (int f = 0; f < a.nfields; ++f) prefetch_tmap(&a.map[f]);
  pdl_wait();  // the fields are the predecessors' outputs
  pdl_trigger();
  if (threadIdx.x == 0) {
    const int t0 = tile_at(0), t1 = tile_at(1);
    if (t0 >= 0) issue(t0, 0);
    if (t1 >= 0) issue(t1, 1);
  }
  const CtCol<TL> lay{};
  bool aborted = false;
  for (int it = 0;; ++it) {
    const int t = tile_at(it);
    if (t < 0) break;
    const int s = it % ST;
    float2* b = bufs + s * E;
    const bool ok = mbar_wait(&bar[s], (it / ST) & 1, a.err, a.wait.limit_ns);
    if (__syncthreads_or(!ok)) {  // every thread leaves together; nothing more is issued
      aborted = true;
      break;
    }
    if (threadIdx.x == 0) inflight &= ~(1u << s);
    int f, x, o;
    coords(t, f, x, o);
    if (f == a.dual_field) {  // the derived field: the first stage reads its input times the axis factor
      const int id = ct_tid<NC>(tw), l = id % TL, tid = id / TL;
      const float2* tab = a.dual_tab;
      ct_stage0_ld<NC, V, INV>(b, tw, l, tid, lay, [&](int ll, int j, int c, int) { return c_mul(b[lay(ll, j + c)], __ldg(tab + j + c)); });
      ct_stages<NC, V, 1, Ct<NC, V>::S, INV>(b, tw, l, tid, lay);
    } else {
      ct_fft<NC, V, INV, true, TL>(b, tw, lay);
    }
    fence_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      tma_store_4d(&a.map[f], x, 0, 0, o, b);
      bulk_commit();
      const int t2 = tile_at(it + 2);
      if (t2 >= 0) {
        bulk_wait_read<ST - 2>();  // the store out of the stage being refilled has read it
        issue(t2, it + 2);
      }
    }
  }
  if (threadIdx.x == 0) {
    bulk_wait<0>();
    if (aborted)  // the loads still in flight land before the block's shared memory is released
      for (int s = 0; s < ST; ++s)
        if (inflight & (1u << s)) mbar_wait(&bar[s], (parity_bits >> s) & 1, nullptr, a.wait.limit_ns);
  }
}

template <int NC, int V, bool INV>
cudaError_t col_tma_t(const ColTmaArgs& a, const float2* tw, cudaStream_t st) {
  const size_t sm = kColStages * TTile<NC, V>::STRIDE * sizeof(float2) + NC * sizeof(float2) + kColStages * sizeof(uint64_t);
  auto k = k_col_tma<NC, V, INV>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, TTile<NC, V>::THREADS, sm);
  const int ntiles = a.nfields * a.ncx * a.nouter;
  const int grid = std::min(ntiles, std::max(1, per_sm) * tma_num_sms());
  const cudaError_t e = launch_pdl(k, dim3(grid), dim3(TTile<NC, V>::THREADS), sm, st, a, tw);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace kwb
