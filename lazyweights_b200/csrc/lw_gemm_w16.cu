// Launcher of the tcgen05 GEMM over decoded fp16 weights; see lw_gemm_w16.cuh.
#include <cuda.h>

#include <algorithm>

#include "lw_gemv1.h"

#include "lw_gemm_w16.cuh"

namespace lw {

constexpr size_t kSmemLimit = 227 * 1024;

int launch_gemm_w16(const __half* X, const __half* W, float* Y, int m, int rows, int K, int ldy, float* partials,
                    size_t partial_capacity, const float* unscale, cudaStream_t st) {
  if (m < 1 || rows % 64 || K % kW16SlabK) {
    set_kernel_error_text("gemm (fp16 weights)", "shape must be a multiple of 64 rows x 64 columns");
    return kErrArg;
  }
  GemmW16Args a = {};
  a.tok_tiles = (m + kW16MaxTokens - 1) / kW16MaxTokens;
  a.ntok = ((m + a.tok_tiles - 1) / a.tok_tiles + 15) / 16 * 16;
  a.tok_tiles = (m + a.ntok - 1) / a.ntok;
  a.row_tiles = (rows + kW16Rows - 1) / kW16Rows;
  const int slabs = K / kW16SlabK, sms = sm_count(), tiles = a.row_tiles * a.tok_tiles;
  // Split K where the tiles alone leave blocks idle: the time of a launch is its rounds of work items times an item's
  // slabs (plus about four slabs' worth of filling and draining), and the planes cost their own traffic: about as long
  // as 16 slabs for the extra kernel and one per 2 MB written and read again.
  a.splits = 1;
  double best = 0;
  for (int z = 1; z <= 8; z *= 2) {
    const size_t plane = static_cast<size_t>(z) * m * rows;
    if (slabs % z || (z > 1 && (!partials || plane > partial_capacity))) continue;
    const int rounds = (tiles * z + sms - 1) / sms;
    const double cost = rounds * (slabs / z + 4.0) + (z > 1 ? 16.0 + plane * 4.0 / (2 << 20) : 0.0);
    if (z == 1 || cost < best) {
      best = cost;
      a.splits = z;
    }
  }
  a.slabs = slabs / a.splits;
  const size_t stage = kW16ABytes + static_cast<size_t>(a.ntok) * kW16SlabK * 2;
  a.stages = static_cast<int>(std::min<size_t>(kW16MaxStages, (kSmemLimit - 2048) / stage));   // 1 KB: the stages' alignment, 1 KB: barriers
  alignas(64) CUtensorMap wm, xm;
  if (!make_half_slab_map(&wm, W, K, rows, kW16Rows) || !make_half_slab_map(&xm, X, K, m, a.ntok)) {
    set_kernel_error_text("gemm (fp16 weights)", "no tensor map: the activations must be 16-byte aligned");
    return kErrArg;
  }
  a.y = a.splits > 1 ? partials : Y;
  a.ldy = a.splits > 1 ? rows : ldy;
  a.unscale = a.splits > 1 ? nullptr : unscale;
  a.err = error_word();
  a.wait_limit = debug_knobs().wait_limit;
  a.m = m;
  a.rows = rows;
  a.K = K;
  if (!a.err) return kErrCuda;
  static bool configured_per_device[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  bool& configured = configured_per_device[dev & 63];
  if (!configured) {
    if (cudaFuncSetAttribute(k_gemm_w16, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit - 1024)) != cudaSuccess)
      return note_launch("cudaFuncSetAttribute(k_gemm_w16)");
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min(sms, tiles * a.splits));
  cfg.blockDim = dim3(kW16Threads);
  cfg.dynamicSmemBytes = a.stages * stage + 1024;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_gemm_w16, wm, xm, a);
  const int rc = note_launch("k_gemm_w16");
  if (rc || a.splits == 1) return rc;
  return launch_sum_partials(partials, Y, m, rows, ldy, a.splits, unscale, st);
}

}  // namespace lw
