// Tensor-core GEMM over decoded fp16 weights, for products of more rows than the fused kernels take (and path 2 of
// rt_test_matmul): Y[token, row] = sum_k X[token, k] W[row, k], fp16 operands, fp32 accumulation.  The role of the
// reference's k_gemm_raw8 / k_gemm2_raw8 (kernels/llmrt.cu:211-343), which run SIMT float FMAs on decoded codes.
//
//   D[weight row, token] = sum_k W[weight row, k] X[token, k]     tcgen05.mma, kind::f16, M = 128, N = tokens, K = 16
//
// Bound: the L2-to-SM traffic of the operand tiles, about 95 GB/s per SM (32 KB in 0.34 us, 48 KB in 0.50 us): a tile of
// R rows x N tokens reads (R + N) x 128 bytes per 64 columns for R x N x 64 multiply-adds.  So N is as large as the tokens
// allow, up to the 256 of one instruction, and R is 256 (two instructions per step, `blocks_m`) where that brings the launch
// down: 512 tokens x 14336 x 4096 take 1 round of 64 KB steps instead of 2 rounds of 48 KB steps.
//  * One persistent block per SM: warp 0 starts the TMA loads (128-byte swizzled 64-column slabs of both operands, a
//    ring of stages), warp 1 issues the MMAs (one lane each), warps 2..5 read finished tiles from tensor memory.
//  * The accumulator of a 128-row tile is double-buffered in tensor memory, so the tile before is written while the next one
//    runs; a 256-row tile of 256 tokens fills the tensor memory once.
//  * A lane of the epilogue holds a weight row, i.e. one output column: a warp's store of one token is 128 bytes.
//  * Few tiles: K is split (a work item is tile x K range) and each range writes a plane of partial sums,
//    added in order by k_sum_partials.
//  * Every wait is bounded; a warp that gives up sets the error word and a block-wide flag that ends every loop.  Whoever
//    gave up, the block ends only after the copies it started have landed and the multiplications it issued are done (waits
//    with a limit of their own; after a pass that ran through they return at once).
#pragma once
#include "lw_tcgen05.cuh"

namespace lw {

constexpr int kW16Rows = 128;                  // M: weight rows of an instruction; a tile has one or two such blocks
constexpr int kW16MaxTokens = 256;             // N: tokens of a tile, a multiple of 16
constexpr int kW16SlabK = 64;                  // columns of a stage: one 128-byte swizzle row
constexpr int kW16MaxStages = 8;
constexpr int kW16Threads = 6 * 32;
constexpr uint32_t kW16ABytes = kW16Rows * kW16SlabK * 2;

struct GemmW16Args {
  float* y;              // [m][ldy] (splits == 1) or planes [splits][m][rows]
  const float* unscale;  // factor per token of the finished sum (splits == 1 only; may be null)
  unsigned int* err;
  uint32_t wait_limit;
  int m, rows, K, ldy;
  int ntok;              // N of a tile
  int tok_tiles, row_tiles, splits;
  int slabs;             // 64-column slabs per split (K / 64 / splits)
  int stages;
  int blocks_m;          // 128-row blocks of a tile: 1 or 2
  int drop_slab;         // a test's lost copy: block 0 never loads this slab of its first item (-1: none)
};

__global__ void __launch_bounds__(kW16Threads, 1)
    k_gemm_w16(const __grid_constant__ CUtensorMap WM, const __grid_constant__ CUtensorMap XM, const __grid_constant__ GemmW16Args A) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[kW16MaxStages], empty[kW16MaxStages], d_full[2], d_empty[2], mma_done;
  __shared__ uint32_t tmem_slot[1];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
  const uint32_t a_bytes = A.blocks_m * kW16ABytes, stage_bytes = a_bytes + A.ntok * (kW16SlabK * 2);   // a multiple of 1024: ntok is one of 16s, 8 rows = 1 KB
  if (threadIdx.x == 0) {
    for (int i = 0; i < A.stages; ++i) {
      mbar_init(smem_addr(full + i), 1);
      mbar_init(smem_addr(empty + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_addr(d_full + i), 1);
      mbar_init(smem_addr(d_empty + i), 4);
    }
    mbar_init(smem_addr(&mma_done), 1);
    abort_word = 0;
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot[0];
  // items: splits x row tiles x token tiles, token tiles fastest: the blocks that read the same rows of W run at one time
  const int items = A.row_tiles * A.tok_tiles * A.splits;
  const int log_buffers = A.blocks_m == 1 ? 1 : 0;   // accumulators of a tile in tensor memory: item n of the block uses n % buffers
  pdl_trigger();
  if (warp == 0) {
    if (lane == 0) {   // ---- TMA loads
      pdl_wait();      // the decoded weights and the converted activations come from the kernels before
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
        const int tt = it % A.tok_tiles, q = it / A.tok_tiles, rt = q % A.row_tiles, z = q / A.row_tiles;
        for (int k = 0; k < A.slabs; ++k) {
          if (!(ok = t5_wait(empty + s, ph ^ 1u, A.wait_limit, A.err, abort_flag))) break;
          const uint32_t dst = base + s * stage_bytes;
          if (k != A.drop_slab || it != 0) {
            mbar_expect(full + s, stage_bytes);
            for (int i = 0; i < A.blocks_m; ++i)   // rows past the end arrive as zeros
              tma_load_2d(dst + i * kW16ABytes, &WM, (z * A.slabs + k) * kW16SlabK, (rt * A.blocks_m + i) * kW16Rows, full + s);
            tma_load_2d(dst + a_bytes, &XM, (z * A.slabs + k) * kW16SlabK, tt * A.ntok, full + s);
          }
          if (++s == A.stages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      // the copies still in flight land before the block gives its shared memory back (stages below s were last filled in
      // round ph, the others in the round before)
      for (int i = 0; i < A.stages; ++i) mbar_wait(smem_addr(full + i), i < s ? ph : ph ^ 1u, A.err, 1u << 16);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {   // ---- MMAs
      const uint32_t idesc = idesc_f16_m128(A.ntok);
      int s = 0, n = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++n) {
        const int db = n & log_buffers;
        if (!(ok = t5_wait(d_empty + db, ((n >> log_buffers) & 1) ^ 1u, A.wait_limit, A.err, abort_flag))) break;
        tc_fence_after();
        for (int k = 0; k < A.slabs; ++k) {
          if (!(ok = t5_wait(full + s, ph, A.wait_limit, A.err, abort_flag))) break;
          tc_fence_after();
          const uint64_t dbd = smem_desc_sw128(base + s * stage_bytes + a_bytes);
          for (int i = 0; i < A.blocks_m; ++i) {
            const uint64_t da = smem_desc_sw128(base + s * stage_bytes + i * kW16ABytes);
#pragma unroll
            for (int j = 0; j < kW16SlabK / 16; ++j)   // 32 bytes further inside the swizzle row
              mma_ss_f16(tmem + (db + i) * kW16MaxTokens, da + 2 * j, dbd + 2 * j, idesc, k > 0 || j > 0);
          }
          mma_commit(empty + s);
          if (++s == A.stages) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (ok) mma_commit(d_full + db);
      }
      mma_commit(&mma_done);   // they read shared memory and write tensor memory, which the block is about to give back
      mbar_wait(smem_addr(&mma_done), 0, A.err, 1u << 16);
    }
    __syncwarp();
  } else {   // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4) ..
    const int quad = warp & 3;
    pdl_wait();   // the factors come from a kernel before, and what it reads may be this kernel's result
    int n = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x, ++n) {
      const int tt = it % A.tok_tiles, q = it / A.tok_tiles, rt = q % A.row_tiles, z = q / A.row_tiles;
      const int db = n & log_buffers, t0 = tt * A.ntok;
      if (!__all_sync(0xffffffffu, t5_wait(d_full + db, (n >> log_buffers) & 1, A.wait_limit, A.err, abort_flag))) break;
      tc_fence_after();
      const int nt = min(A.ntok, A.m - t0);
      for (int i = 0; i < A.blocks_m; ++i) {
        const int row = (rt * A.blocks_m + i) * kW16Rows + quad * 32 + lane;
        float* y = A.y + static_cast<size_t>(z) * A.m * A.rows + static_cast<size_t>(t0) * A.ldy + row;
        const uint32_t src = tmem + (static_cast<uint32_t>(32 * quad) << 16) + (db + i) * kW16MaxTokens;
        for (int c0 = 0; c0 < nt; c0 += 16) {
          uint32_t v[16];
          tmem_load16(src + c0, v);
          tmem_wait_load();
          if (row < A.rows) {
#pragma unroll
            for (int c = 0; c < 16; ++c)
              if (c0 + c < nt) {
                const float f = __uint_as_float(v[c]);
                y[static_cast<size_t>(c0 + c) * A.ldy] = A.unscale ? f * A.unscale[t0 + c0 + c] : f;
              }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(d_empty + db);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace lw
