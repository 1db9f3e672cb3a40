// Pieces shared by the tensor-core grouped GEMM kernels: the tile walk over
// ragged expert segments, output conversion, and host-side tensor-map encoding.
#pragma once

#include <atomic>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace b200moe {
namespace {

constexpr int kFeat = 128;          // features per tile (UMMA M)
constexpr int kMaxExperts = 1024;
constexpr size_t kMaxSmem = 227 * 1024;   // dynamic shared memory of a CTA

// Depth of a ring whose blocks `sets` converter sets take in turn, each putting what it makes of a block
// into one of `operands` stages that one issuer's MMAs free in order.  A set waits for the n-th fill of a stage by
// parity, which also looks complete while fill n - 1 is still on its way: that fill, block i - stages, has
// landed for sure only if the MMA was done with it when the set stored its last block, i - sets, i.e. if it
// is no later than block i - sets - operands.  (Two issuers free operands out of order: gemm_tc_i4.cu therefore also
// keeps its depth a multiple of the sets, so that a stage's fills are all seen by the same set.)
constexpr int converter_ring_depth(int sets, int operands) { return sets + operands; }

struct TileInfo {
  int e, n_tile, m_tile, row0, valid;   // e: index of the weights the tile multiplies with
};

// The tile walk of a CTA, in shared memory: row and tile prefix sums over the experts that have
// rows (decode batches leave most experts of a layer empty; walking over those, an element at a
// time in every role, cost more than a tile's multiplications), and those experts' ids.
struct TileWalk {
  const int* tile_start;     // [n + 1] first tile of an expert, then the number of tiles
  const int* row_start;      // [n + 1]
  const uint16_t* expert;    // [n]
  int n;                     // experts with rows
  int total;                 // tiles
};
__host__ __device__ constexpr int tile_walk_bytes(int num_experts) {
  return ((2 * (num_experts + 1) + 1) * 4 + 2 * num_experts + 15) & ~15;
}
__device__ __forceinline__ TileWalk tile_walk_at(const void* mem, int num_experts) {
  TileWalk w;
  const int* p = reinterpret_cast<const int*>(mem);
  w.n = p[0];
  w.tile_start = p + 1;
  w.row_start = w.tile_start + num_experts + 1;
  w.expert = reinterpret_cast<const uint16_t*>(w.row_start + num_experts + 1);
  w.total = w.tile_start[w.n];
  return w;
}

// Tiles of one expert are numbered feature-tile-major with the token tiles
// adjacent, so CTAs that run at the same time share a weight tile in L2.
// With w_experts > 0 the row segments outnumber the weight sets: segment s multiplies with
// weights s % w_experts (the segments are the (source rank, local expert) pairs of an
// expert-parallel exchange, source-major).
// `cursor` is the position in the walk of the caller's previous tile; t does not decrease.
template <int BT>
__device__ __forceinline__ void locate_tile(const TileWalk& w, int t, int& cursor, TileInfo& ti, int w_experts = 0) {
  if (t >= w.tile_start[cursor + 1]) {
    ++cursor;
    if (t >= w.tile_start[cursor + 1]) {   // further than the next one: bisect
      int lo = cursor + 1, hi = w.n - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (w.tile_start[mid] <= t) lo = mid;
        else hi = mid - 1;
      }
      cursor = lo;
    }
  }
  const int local = t - w.tile_start[cursor];
  const int rows = w.row_start[cursor + 1] - w.row_start[cursor];
  const int m_tiles = (rows + BT - 1) / BT;
  const int e = w.expert[cursor];
  ti.e = w_experts > 0 ? e % w_experts : e;
  ti.n_tile = m_tiles == 1 ? local : local / m_tiles;
  ti.m_tile = local - ti.n_tile * m_tiles;
  ti.row0 = w.row_start[cursor] + ti.m_tile * BT;
  const int left = rows - ti.m_tile * BT;
  ti.valid = left < BT ? left : BT;
}

// A bounded wait gave up: tell the caller through its status word.  A plain store, so the
// word may live in device memory or in mapped host memory that the host polls without a
// synchronisation.
__device__ __forceinline__ void report_timeout(int32_t* status) {
  if (status != nullptr) {
    *reinterpret_cast<volatile int32_t*>(status) = 1;
    __threadfence_system();
  }
}
__device__ __forceinline__ float load_bias(const void* b, int out_f16, int64_t idx) {
  if (out_f16) return __half2float(reinterpret_cast<const __half*>(b)[idx]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(b)[idx]);
}


// Output path of the epilogue warps.  A warp holds a block of the result as
// vals[i] = D(token i, feature lane) (one TMEM lane per thread), but D is
// row-major over features, so a direct store would write 2 bytes per lane into
// 32 different 64-byte pieces.  The block is transposed through a per-warp
// shared-memory tile ([token][feature], 16-bit) and written as 16-byte vectors:
// kFeat/8 lanes cover one token row, 256/kFeat rows per store instruction.
// kFeat = 32 (one value per lane) or 16 (values on the even lanes only).
template <int kTok, int kFeatW>
__device__ __forceinline__ void store_tile_rows(uint32_t xp_s, void* d, int64_t row0, int tok_valid, int64_t m_limit, int n_out,
                                                int feat0, int lane) {
  __syncwarp();
  constexpr int kLanesPerRow = kFeatW / 8;          // 16-byte pieces per token row
  constexpr int kRowsPerIter = 32 / kLanesPerRow;
  const int piece = lane % kLanesPerRow;
  const int f = feat0 + piece * 8;
#pragma unroll
  for (int it = 0; it < kTok / kRowsPerIter; ++it) {
    const int tok = lane / kLanesPerRow + it * kRowsPerIter;
    if (tok < tok_valid && row0 + tok < m_limit && f < n_out) {
      const uint4 q = ptx::lds128(xp_s + (tok * kFeatW + piece * 8) * 2);
      *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(d) + (row0 + tok) * (int64_t)n_out + f) = q;
    }
  }
  __syncwarp();
}
__device__ __forceinline__ uint16_t bits16(float x, int out_f16) {
  if (out_f16) { const __half h = __float2half_rn(x); return *reinterpret_cast<const uint16_t*>(&h); }
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  return *reinterpret_cast<const uint16_t*>(&h);
}
// The same for gated outputs shared out over lane pairs: vals[j] = D(token 2 j + (lane & 1), feature lane / 2).
template <int kHalfTok>
__device__ __forceinline__ void store_pairs_transposed(uint16_t* xp, const float (&vals)[kHalfTok], void* d, int out_f16,
                                                       int64_t row0, int tok_valid, int64_t m_limit, int n_out, int feat0,
                                                       int lane) {
  const uint32_t xp_s = ptx::smem_u32(xp);
  const uint32_t at = xp_s + ((lane & 1) * 16 + (lane >> 1)) * 2;
#pragma unroll
  for (int j = 0; j < kHalfTok; ++j) ptx::sts16(at + j * 64, bits16(vals[j], out_f16));
  store_tile_rows<2 * kHalfTok, 16>(xp_s, d, row0, tok_valid, m_limit, n_out, feat0, lane);
}
template <int kTok, int kFeatW>
__device__ __forceinline__ void store_block_transposed(uint16_t* xp, const float (&vals)[kTok],
                                                       void* d, int out_f16, int64_t row0,
                                                       int tok_valid, int64_t m_limit, int n_out,
                                                       int feat0, int lane) {
  const int col = (kFeatW == 32) ? lane : (lane >> 1);
  const bool writer = (kFeatW == 32) || !(lane & 1);
  const uint32_t xp_s = ptx::smem_u32(xp);
#pragma unroll
  for (int i = 0; i < kTok; ++i) {
    const uint16_t bits = bits16(vals[i], out_f16);
    if (writer) ptx::sts16(xp_s + (i * kFeatW + col) * 2, bits);
  }
  store_tile_rows<kTok, kFeatW>(xp_s, d, row0, tok_valid, m_limit, n_out, feat0, lane);
}

// Fills the tile walk at `mem` (tiles of expert e = ceil(rows_e / BT) * n_tiles).  Called by one
// full warp; a lane takes eight consecutive experts of every 256, so that their loads are in
// flight together and one scan serves them all.
template <int BT>
__device__ __forceinline__ void build_tile_walk(const int32_t* rows_per_expert, int num_experts, int n_tiles, void* mem) {
  const int lane = threadIdx.x & 31;
  int* head = reinterpret_cast<int*>(mem);
  int* tile_start = head + 1;
  int* row_start = tile_start + num_experts + 1;
  uint16_t* expert = reinterpret_cast<uint16_t*>(row_start + num_experts + 1);
  int carry_r = 0, carry_t = 0, carry_n = 0;
  for (int base = 0; base < num_experts; base += 256) {
    int r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = base + lane * 8 + i;
      r[i] = e < num_experts ? __ldcg(rows_per_expert + e) : 0;   // (read twice, see prefetch_first_tiles: not through L1)
    }
    int sum_r = 0, sum_t = 0, sum_n = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (r[i] < 0) r[i] = 0;
      sum_r += r[i];
      sum_t += ((r[i] + BT - 1) / BT) * n_tiles;
      sum_n += r[i] > 0 ? 1 : 0;
    }
    int ir = sum_r, it = sum_t, in = sum_n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o_r = __shfl_up_sync(0xffffffffu, ir, d);
      const int o_t = __shfl_up_sync(0xffffffffu, it, d);
      const int o_n = __shfl_up_sync(0xffffffffu, in, d);
      if (lane >= d) { ir += o_r; it += o_t; in += o_n; }
    }
    int row = carry_r + ir - sum_r, tile = carry_t + it - sum_t, pos = carry_n + in - sum_n;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (r[i] > 0) {
        row_start[pos] = row;
        tile_start[pos] = tile;
        expert[pos] = (uint16_t)(base + lane * 8 + i);
        ++pos;
        row += r[i];
        tile += ((r[i] + BT - 1) / BT) * n_tiles;
      }
    }
    carry_r += __shfl_sync(0xffffffffu, ir, 31);
    carry_t += __shfl_sync(0xffffffffu, it, 31);
    carry_n += __shfl_sync(0xffffffffu, in, 31);
  }
  if (lane == 0) {
    head[0] = carry_n;
    row_start[carry_n] = carry_r;
    tile_start[carry_n] = carry_t;
  }
}

// Weights of the CTA's first tiles to L2, in the time in which an early launched kernel only waits for the one
// before it (6 to 10 us for the second GEMM of a decode layer: the end of the first GEMM and the activation).
// One full warp, before pdl_wait(): `rows_per_expert` must be complete already (gemm_args.rows_ready), but
// nothing depends on it: from any counts the walk ends and asks for blocks of the weights only, and it is built
// again after the wait.  `load(tile, kb)` asks for a K block.
// Second GEMM of qwen3 fp8 at 16 tokens 33.6 -> 31.2 us, of the small 16-bit layer at 64 tokens 11.1 -> 10.4; the
// layer calls with 128 / 256 / 512 KB a CTA: 96.9 / 96.2 / 97.1 (98.2 without) and 39.1 / 39.6 / 39.9 (39.9); one
// Mixtral token 118.9 / 119.3 / 120.3 (119.3).
constexpr int kPreBytes = 131072;
template <int BT, typename Load>
__device__ __forceinline__ void prefetch_first_tiles(const int32_t* rows_per_expert, int num_experts, int w_experts,
                                                     int n_tiles, int num_kb, int blocks, void* mem, Load&& load) {
  build_tile_walk<BT>(rows_per_expert, num_experts, n_tiles, mem);
  __syncwarp();
  if (ptx::elect_one()) {
    const TileWalk walk = tile_walk_at(mem, num_experts);
    int cursor = 0;
    for (int t = blockIdx.x; t < walk.total && blocks > 0; t += gridDim.x) {
      TileInfo ti;
      locate_tile<BT>(walk, t, cursor, ti, w_experts);
      if ((uint32_t)ti.n_tile >= (uint32_t)n_tiles) break;   // the counts were not complete: no such tile, so no more
      for (int kb = 0; kb < num_kb && blocks > 0; ++kb, --blocks) load(ti, kb);
    }
  }
  __syncwarp();
}

// ------------------------------ host side ------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static const EncodeTiledFn fn = [] {   // (threads that come first together wait for one look-up)
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
                       qres == cudaDriverEntryPointSuccess;
    return found ? reinterpret_cast<EncodeTiledFn>(ptr) : nullptr;
  }();
  return fn;
}

int encode_map(CUtensorMap* map, CUtensorMapDataType dt, int rank, const void* base,
               const cuuint64_t* dims, const cuuint64_t* strides_bytes, const cuuint32_t* box,
               CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return fail(B200MOE_E_CUDA, "cuTensorMapEncodeTiled is not available");
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, dt, (cuuint32_t)rank, const_cast<void*>(base), dims, strides_bytes, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(B200MOE_E_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return B200MOE_OK;
}

// cudaFuncAttributeMaxDynamicSharedMemorySize belongs to a (kernel, device) pair, so a process that
// drives several GPUs sets it on each of them.  It is always set to the most a CTA may have, not to what
// the call needs: threads that come first together with different needs set the same.  One static
// instance per kernel instantiation.
struct SmemConfig {
  std::atomic<bool> done[kMaxDevices];
  template <typename Kern>
  int ensure(Kern kern) {
    const int dev = current_device();
    if (!done[dev].load(std::memory_order_acquire)) {
      B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
      done[dev].store(true, std::memory_order_release);
    }
    return B200MOE_OK;
  }
};

}  // namespace
}  // namespace b200moe
