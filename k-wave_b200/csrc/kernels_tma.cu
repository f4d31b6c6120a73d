// Host side of the TMA-fed column passes: the y pass (col_tma.cuh) and the
// fused last-axis operator (fused_tma.cuh), instantiated per length in
// generated translation units; tensor maps and the per-length dispatch.
#include <cudaTypedefs.h>

#include <algorithm>

#include "fused_tma.cuh"
#include "tma_more_sizes.h"
#include "tma_sizes.h"

namespace kwb {

#define KWB_EXTERN(N) extern template struct TmaKernels<N>;
KWB_TMA_COL_SIZES(KWB_EXTERN)
KWB_TMA_MORE_SIZES(KWB_EXTERN)
#undef KWB_EXTERN

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {

struct TmaEntry {
  int n;
  decltype(&TmaKernels<64>::lines) lines;
  decltype(&TmaKernels<64>::col) col;
  decltype(&TmaKernels<64>::fused) fused;
};
#define KWB_ENTRY(N) {N, &TmaKernels<N>::lines, &TmaKernels<N>::col, &TmaKernels<N>::fused},
const TmaEntry kTmaTable[] = {KWB_TMA_COL_SIZES(KWB_ENTRY) KWB_TMA_MORE_SIZES(KWB_ENTRY)};
#undef KWB_ENTRY

const TmaEntry* tma_entry(int n) {
  for (const TmaEntry& e : kTmaTable)
    if (e.n == n) return &e;
  return nullptr;
}

}  // namespace

int tma_lines(int n, int v) {
  const TmaEntry* e = tma_entry(n);
  return e ? e->lines(v) : 0;
}

static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

static bool get_encoder() {
  if (g_encode) return true;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
    return false;
  g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  return true;
}

bool tma_supported(int n) { return tma_entry(n) != nullptr; }

// A tensor copy's box holds at most 256 elements along a dimension, so a line
// of n points is addressed as nseg segments of equal length, two dimensions of
// one box, which land one after the other in shared memory: the fewest
// segments of at most 256 points that divide n.
static int line_segments(int n) {
  int s = (n + 255) / 256;
  while (n % s) ++s;
  return s;
}

static bool encode(CUtensorMap* m, void* base, const cuuint64_t (&dims)[4], const cuuint64_t (&strides)[3],
                   const cuuint32_t (&box)[4]) {
  const cuuint32_t es[4] = {1, 1, 1, 1};
  return g_encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map over a half-spectrum buffer [nz][ny][nxp] (8-byte elements) for
// transforms along y (yaxis 1) or z (2): dimensions {kx, position in segment,
// segment, outer index}, box {columns per tile, n / segments, segments, 1}.
// The x extent is the nxh bins in use, not the pitch: the last column tile
// of a row is loaded with zeros past bin nxh - 1 and stored clipped there,
// so padding costs no memory traffic.  Tiles start at x = cx * lines, a
// multiple of 32 bytes.
bool make_spec_map(CUtensorMap* m, void* base, const Dims& d, int yaxis, int n, int v) {
  if (!get_encoder()) return false;
  const int lines = tma_lines(n, v), nseg = line_segments(n), seg = n / nseg;
  if (d.nxp % 2 != 0 || lines < 2 || lines % 2 != 0 || lines > 256 || nseg > 256) return false;
  const cuuint64_t row = (cuuint64_t)d.nxp * 8, plane = row * d.ny;
  const cuuint64_t ls = yaxis == 1 ? row : plane, os = yaxis == 1 ? plane : row;
  return encode(m, base,
                {(cuuint64_t)d.nxh, (cuuint64_t)seg, (cuuint64_t)nseg, (cuuint64_t)(yaxis == 1 ? d.nz : d.ny)},
                {ls, ls * seg, os}, {(cuuint32_t)lines, (cuuint32_t)seg, (cuuint32_t)nseg, 1u});
}

// Tensor map of the remainder tiles of the last-axis pass (3D): box {2,
// rows, n / segments, segments} at x = nxh - 1, the lone last column and the
// bin past it (zero-filled on load; its lines are not stored).
bool make_spec_map_rem(CUtensorMap* m, void* base, const Dims& d, int n, int rows) {
  if (!get_encoder()) return false;
  const int nseg = line_segments(n), seg = n / nseg;
  if (d.nxp % 2 != 0 || (d.nxh - 1) % 2 != 0 || rows < 1 || rows > 256 || nseg > 256) return false;
  const cuuint64_t row = (cuuint64_t)d.nxp * 8, plane = row * d.ny;
  return encode(m, base, {(cuuint64_t)d.nxh, (cuuint64_t)d.ny, (cuuint64_t)seg, (cuuint64_t)nseg},
                {row, plane, plane * seg}, {2u, (cuuint32_t)rows, (cuuint32_t)seg, (cuuint32_t)nseg});
}

static int g_num_sms = 0;
int tma_num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return g_num_sms;
}

cudaError_t launch_col_tma(bool inv, int n, const ColTmaArgs& a, const float2* tw, cudaStream_t st) {
  const TmaEntry* e = tma_entry(n);
  return e ? e->col(inv, a, tw, st) : cudaErrorInvalidValue;
}

cudaError_t launch_fused_tma(int n, const FusedTmaArgs& a, const float2* tw, const SpecTables& T, cudaStream_t st) {
  const TmaEntry* e = tma_entry(n);
  return e ? e->fused(a, tw, T, st) : cudaErrorInvalidValue;
}

}  // namespace kwb
