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
  const int slabs = K / kW16SlabK, sms = sm_count();
  // The tile's rows and the K split, by the time of a launch in ns: rounds of work items times an item's slabs.  A slab takes
  // what its bytes take at 95 GB/s per SM or its multiply-adds at 1.1 ns per token and 128 rows, whichever is more; filling and
  // draining about 2 us per launch, and per round where the accumulator is not double-buffered (the tile's results leave
  // meanwhile: 12 ns per token and 128 rows).  Planes of a split cost the extra kernel, about 4 us, and their own traffic:
  // 0.35 us per MB.  Fitted on Q4_K 14336 x 4096, where 256 rows win from 257 tokens on (300: 77 against 87 us)
  // and 128 rows up to 256 (128: 61 against 66).  It errs by 3 to 7 per cent on 4096 x 14336 at 128 and 200 tokens, where it takes
  // 256 rows (63.0 and 72.4 us; 128 rows 61.4 and 67.4).
  a.splits = a.blocks_m = 1;
  double best = 0;
  for (int b = 1; b <= 2; ++b)
    for (int z = 1; z <= 8; z *= 2) {
      const size_t plane = static_cast<size_t>(z) * m * rows;
      if (slabs % z || (z > 1 && (!partials || plane > partial_capacity))) continue;
      const int tiles = (rows + b * kW16Rows - 1) / (b * kW16Rows) * a.tok_tiles, rounds = (tiles * z + sms - 1) / sms;
      const double slab = std::max((b * kW16Rows + a.ntok) * 128.0 / 95.0, b * a.ntok * 1.1), out = 2000.0 + b * a.ntok * 12.0;
      const double cost = rounds * (slabs / z) * slab + (b == 1 ? 1 : rounds) * out + (z > 1 ? 4000.0 + plane * 4.0 / (1 << 20) * 350.0 : 0.0);
      if (best == 0 || cost < best) {
        best = cost;
        a.splits = z;
        a.blocks_m = b;
      }
    }
  a.row_tiles = (rows + a.blocks_m * kW16Rows - 1) / (a.blocks_m * kW16Rows);
  const int tiles = a.row_tiles * a.tok_tiles;
  a.slabs = slabs / a.splits;
  const size_t stage = a.blocks_m * kW16ABytes + static_cast<size_t>(a.ntok) * kW16SlabK * 2;
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
  a.drop_slab = debug_knobs().drop_unit;
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
