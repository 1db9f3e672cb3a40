// Block-scaled tensor-core grouped GEMM: MXFP4 weights (two e2m1 codes per byte,
// [E,N,K/2], one e8m0 scale per 32 elements, [E,N,K/32]) times MXFP8 activations
// (e4m3 codes [terms][M,K], one e8m0 scale per 32 elements as 32-bit words
// [terms][K/128][M]).  With terms == 2 the second plane is the residual of the
// first (activation = plane0 + plane1): each weight tile is multiplied with
// both planes, which gives 16-bit-like activation accuracy at fp8 MMA speed.
//
// tcgen05.mma kind::mxf8f6f4.block_scale multiplies both operands by their
// power-of-two scales inside the tensor core, so nothing is dequantised by CUDA
// cores: HBM and shared memory see 4-bit weights and 8-bit activations only.
//
// Same orientation, tile walk and epilogue as the other tensor-core kernels
// (weights' output features on the 128-row M side, tokens on the N side).  Roles:
//   warp 0    : weight producer.  Weight tile of 128 rows x 128 codes, fetched by TMA with
//               the 16U4_ALIGN16B tensor-map type, which spreads every 8 packed
//               bytes into a 16-byte slot (the operand format the MMA reads),
//               128-byte swizzle; asks for blocks further on to be brought into L2.
//   warp 1    : MMA issuer, owns tensor memory; also copies the scale factors of each
//               K block from shared to tensor memory (tcgen05.cp, which replicates them
//               over the four lane quarters as the MMA wants them)
//   warps 2-5 : scale preparers: bring the e8m0 bytes of the tile's 128 weight rows
//               (one contiguous piece of the scale tensor) into shared memory
//               with cp.async one tile ahead, read the tokens' scale words (one
//               coalesced 32-bit word per token and K block) a group of K blocks
//               ahead, and write both to a ring of groups in the layout tcgen05.cp
//               reads
//   warp 10   : token producer: the tile's rows (rounded up to 16) x 128 bytes of every plane
//   warps 6-9 : epilogue.  When K is not a multiple of 128 (the weights' tensor-map type
//               needs it) they also bring and spread the last, partial block of a tile.
//
// The same kernel (kW8) multiplies per-tensor-scaled fp8 weights ([E,K,N], e4m3 or
// e5m2, one fp32 scale per expert: the reference's w8a16 recipe,
// csrc/xpu/grouped_gemm/xe_2/grouped_gemm_xe2_interface.hpp:322-360) with the same
// two-plane activations: the weight tile then is a plain byte tile read as an
// MN-major operand, its scale factors are 2^0, and the expert's scale
// multiplies the accumulator in the epilogue.  MXFP8 weights ([E,K,N] e4m3 with one
// e8m0 scale per 32 K rows, [E,K/32,N]: the reference's "mxfp8" recipe,
// vllm_xpu_kernels/moe_utils.py:76-78, 236-403) take the same path with their real
// scale factors, staged from the transposed scale tensor.
//
// What bounds it (128 experts, two planes): shared memory.  A K block writes 16 KB of spread weights and 256
// bytes a token row, and its MMAs read the same again: 64 KB or 512 cycles at 128 bytes a cycle with 64 rows,
// where the MMAs themselves take 320; with loads left out a K block takes 360 to 410 cycles, with them about
// 660.  With few rows it is 320 cycles and DRAM (about 370 at the copy rate); measured about 400.  So a tile brings
// and multiplies only the rows it has, and the second plane follows directly (both planes in boxes of 96 rows and
// N = 96 + rows before: 430 -> 396 us at 64 rows per expert, N 5760, K 2880).
//
// Numerics: products of e2m1 and e4m3 codes are exact, scaling by powers of two is
// exact, accumulation is fp32; the difference from the reference's w4a16 path
// (csrc/xpu/grouped_gemm/xe_2/gemm_xe2.hpp:411-471 of vllm-xpu-kernels) is the
// rounding of the activations to MXFP8 only.
#include "common.cuh"
#include "gemm_tc_common.cuh"
#include "mx_quant.cuh"
#include "sm100_ptx.cuh"


namespace b200moe {
namespace {

constexpr int kMxWBytes = 16384;    // 128 rows x 128 codes in 16-byte slots of 16
constexpr int kMxWTx = 8192;        // the spreading load reports the packed bytes it read to its barrier
constexpr int kMxThreads = 352;
constexpr int kMxMaxStages = 8;
// K blocks the weights are asked for into L2 ahead of their load.  A row's piece of a K block is 64 bytes and L2
// fetches 256, so every fourth block comes from DRAM, and the ring is too short for that latency (stamps: 1500 to
// 1900 cycles for that block, 750 for the others).  128 experts, N 5760, K 2880, gated, with / without: 4 rows per
// expert 204 / 217 us, 16 rows 262 / 283, 64 rows 385 / 393; 4, 8 and 10 blocks ahead, or on into the next tile, are
// slower.  Not for token tiles of 16: their calls run into the power cap when they follow one another, and the
// asking costs energy: layer calls of 128 tokens, in short runs 342 / 349 us, in a loop of seconds 391 / 384.
constexpr int kMxAhead = 6;
// Routed rows up to which this kernel launches early (launch_pdl); the layer's other kernels gain by it further on
// (kEarlyLaunchRows), this one does not.  gpt-oss layer calls, single bursts, this kernel plain / early, us: 1 token 42.2 /
// 39.7, 128 tokens 348 / 344, 400 tokens (1600 rows) 416.2 / 416.1, 512 tokens 428.5 / 429.1, 1024 tokens 499.5 / 505.1, 1500
// tokens 558 / 571, 2048 tokens (8192 rows) 665 / 697.
constexpr int64_t kMxEarlyLaunchRows = 2048;
constexpr int kMxGroup = 4;         // K blocks per scale group (one hand-over from the scale preparers)
constexpr int kMxSlots = 4;         // scale groups in the ring, at most
constexpr int kMxSfwCap = 24576 + 32;    // largest weight-scale piece (128 rows x K/32 bytes) staged in shared memory

struct MxParams {
  const uint8_t* w;         // [E, N, K/2]: the partial K block's source
  const uint8_t* w_scale;   // [E, N, K/32] e8m0; kW8 with w8_block: [E, K/32, N]; else unused
  const float* w_tensor_scale;  // kW8 without w8_block: [E] fp32, multiplies the result
  int w8_block;             // kW8: 1 = MXFP8 weights (scales per 32 K rows), 0 = one scale per expert
  const uint32_t* a_scale;  // [terms][num_kb][M] words of four e8m0 bytes
  const void* bias;
  void* d;
  const int32_t* rows_per_expert;
  int32_t* status;
  int64_t m;
  int n, k, num_experts;
  int n_tiles, num_kb;
  int terms;       // activation planes (1 or 2)
  int tail;        // 1: the last K block is partial, its weights are brought by the epilogue warps
  int stages;
  int sfw_bytes;   // bytes of one staged weight-scale buffer
  uint32_t tmem_cols;
  uint32_t idesc;
  int out_f16;
  int swiglu;      // 1: D[m, f/2] = swigluoai(acc[m,f], acc[m,f+1]) for even f
  float alpha, limit, clamp_limit;
  uint32_t* d_scale;   // swiglu: not null, D leaves as e4m3 planes [terms][M, n/2] with their scale words [terms][n/2 / 128][M]
};

struct MxCtrl {
  uint64_t full[kMxMaxStages];
  uint64_t empty[kMxMaxStages];
  uint64_t sf_full[kMxSlots];
  uint64_t sf_empty[kMxSlots];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t sfw_full[2];
  uint64_t sfw_empty[2];
  uint64_t tail_full;    // the tile's partial block has been spread
  uint64_t pair_full[2]; // quantised output: both halves of a 32-wide group are in shared memory
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) uint16_t xpose[4][32 * 32];   // a warp's transpose tile; quantised output: two buffers per pair of warps
};

// Quantised output of a gated tile: lane pair lane / 2 takes one token's group of 32 outputs, 16 values each (16-bit, as
// they would have been stored), through the planes of quant_mxfp8_kernel, value for value.
template <int kTerms>
__device__ __forceinline__ void store_quantised(uint32_t src, const MxParams& p, int64_t row, bool live, int group, int lane) {
  const int n_out = p.n >> 1, words = (n_out + 127) / 128;
  uint32_t x[8];
  *reinterpret_cast<uint4*>(x) = ptx::lds128(src);
  *reinterpret_cast<uint4*>(x + 4) = ptx::lds128(src + 16);
  float v[16], amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (p.out_f16) {
      const float2 h = __half22float2(*reinterpret_cast<const __half2*>(x + i));
      v[2 * i] = h.x; v[2 * i + 1] = h.y;
    } else {
      v[2 * i] = __uint_as_float(x[i] << 16); v[2 * i + 1] = __uint_as_float(x[i] & 0xffff0000u);
    }
  }
#pragma unroll
  for (int term = 0; term < kTerms; ++term) {
    amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    float sc, inv;
    const int e = mx_scale(amax, kMxLeast, sc, inv);
    uint32_t c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = mx_codes4(v + 4 * i, sc, inv, term + 1 < kTerms);
    if (live) {
      uint8_t* to = reinterpret_cast<uint8_t*>(p.d) + (term * p.m + row) * n_out + group * 32 + (lane & 1) * 16;
      *reinterpret_cast<uint4*>(to) = make_uint4(c[0], c[1], c[2], c[3]);
      if ((lane & 1) == 0) {
        uint8_t* s = reinterpret_cast<uint8_t*>(p.d_scale + ((int64_t)term * words + (group >> 2)) * p.m + row) + (group & 3);
        *s = (uint8_t)e;
        if ((group + 1) * 32 == n_out)    // the groups that fill the row's last word: 2^0
          for (int g = 1; (group & 3) + g < 4; ++g) s[g] = 0x7f;
      }
    }
  }
}
// Shared memory after the pipeline stages: one buffer for the partial K block, the ring
// of scale groups, MxCtrl, the tile walk and two weight-scale staging buffers.
// One group of the scale ring: per K block 512 bytes for the weight rows and 512 per 128 token rows.
template <int kNT>
__host__ __device__ constexpr int mx_slot_bytes() { return kMxGroup * 512 * (kNT > 128 ? 3 : 2); }
// Wide token tiles give the room of two groups to another pipeline stage.
template <int kNT>
__host__ __device__ constexpr int mx_slots() { return kNT > 128 ? 2 : kMxSlots; }

// Weight scales of a tile's rows: one contiguous piece of the scale tensor,
// copied to staging buffer (seq & 1) asynchronously by the 128 feeder threads
// (`ft` = index among them); every thread arrives on sfw_full when its part has
// landed.  Returns false when the wait for the buffer gave up.
__device__ __forceinline__ bool stage_w_scales(const MxParams& p, MxCtrl* ctrl, uint8_t* sfw,
                                               const TileInfo& ti, uint32_t seq, int ft, int kgroups,
                                               volatile int* abort_flag) {
  const uint32_t b = seq & 1;
  if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctrl->sfw_empty[b], ((seq >> 1) & 1) ^ 1, abort_flag)))
    return false;
  const int n0 = ti.n_tile * kFeat;
  const int rows_here = (p.n - n0) < kFeat ? (p.n - n0) : kFeat;
  const int len = rows_here * kgroups;
  const uint8_t* src = p.w_scale + ((int64_t)ti.e * p.n + n0) * kgroups;
  const uint32_t dst = ptx::smem_u32(sfw + b * p.sfw_bytes);
  for (int off = ft * 16; off < len; off += 128 * 16)
    ptx::cp_async_16(dst + off, src + off, (len - off) < 16 ? (len - off) : 16);
  ptx::cp_async_mbar_arrive(&ctrl->sfw_full[b]);
  return true;
}

// The same for MXFP8 weights, whose scales are [E, K/32, N]: for every K group the
// 128 bytes of the tile's features, stored as [group][128] in the staging buffer.
// N is a multiple of 16, so a tile's valid bytes per group are whole 16-byte chunks;
// chunks past N are zero-filled (their rows get 2^0 when the scales are packed).
__device__ __forceinline__ bool stage_w_scales_kn(const MxParams& p, MxCtrl* ctrl, uint8_t* sfw,
                                                  const TileInfo& ti, uint32_t seq, int ft, int kgroups,
                                                  volatile int* abort_flag) {
  const uint32_t b = seq & 1;
  if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctrl->sfw_empty[b], ((seq >> 1) & 1) ^ 1, abort_flag)))
    return false;
  const int n0 = ti.n_tile * kFeat;
  const int valid = (p.n - n0) < kFeat ? (p.n - n0) : kFeat;
  const uint8_t* src = p.w_scale + (int64_t)ti.e * kgroups * p.n + n0;
  const uint32_t dst = ptx::smem_u32(sfw + b * p.sfw_bytes);
  for (int c = ft; c < kgroups * 8; c += 128) {
    const int g = c >> 3, part = c & 7;
    const int bytes = valid - part * 16 >= 16 ? 16 : 0;
    ptx::cp_async_16(dst + c * 16, src + (int64_t)g * p.n + (bytes ? part * 16 : 0), bytes);
  }
  ptx::cp_async_mbar_arrive(&ctrl->sfw_full[b]);
  return true;
}

// Maps of the activation planes with boxes of 16, 32, ... BT rows: a tile brings and multiplies its rows
// rounded up to 16, the second plane's directly behind the first one's.
template <int BT>
struct MxTokenMaps {
  CUtensorMap rows[BT / 16];
};

// BT tokens per tile, kTerms activation planes, kSub 128-wide K blocks per
// pipeline stage (one barrier hand-over per stage: with small token tiles the
// roles' fixed cost per hand-over, not the data, bounds the rate).
template <int BT, int kTerms, int kSub, bool kW8>
__global__ void __launch_bounds__(kMxThreads, 1)
grouped_gemm_mx_kernel(const __grid_constant__ MxTokenMaps<BT> tmap_a,
                       const __grid_constant__ CUtensorMap tmap_w, const MxParams p) {
  static_assert(kMxGroup % kSub == 0, "a scale group is a whole number of stages");
  constexpr int kChunk = BT >= 32 ? 32 : 16;
  constexpr int kNT = kTerms * BT;                  // UMMA N: the planes side by side
  constexpr int kTokChunks = kNT > 128 ? 2 : 1;      // 512-byte scale chunks of the tokens per K block
  constexpr uint32_t kSfBase = 2 * kNT;
  constexpr int kSfPer = kTokChunks == 1 ? 8 : 16;   // scale columns of a K block: the weight rows' four, then the tokens'
  constexpr int kSlotBytes = mx_slot_bytes<kNT>(), kSlots = mx_slots<kNT>();
  constexpr int kABytes = kNT * 128;                // activation bytes of one K block (all planes)
  constexpr int kAOff = kSub * kMxWBytes;           // stage: [W blocks][A blocks]
  constexpr int kStageBytes = kSub * (kMxWBytes + kABytes);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int stages = p.stages;
  uint8_t* tail_w = smem + stages * kStageBytes;   // the weights of the partial K block, if there is one
  uint8_t* sf_ring = tail_w + (p.tail ? kMxWBytes : 0);
  uint8_t* ctrl_at = sf_ring + kSlots * kSlotBytes;
  MxCtrl* ctrl = reinterpret_cast<MxCtrl*>(ctrl_at);
  uint8_t* after = ctrl_at + ((sizeof(MxCtrl) + 15) & ~(size_t)15);
  uint8_t* sfw = after + tile_walk_bytes(p.num_experts);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    pdl_wait();
    build_tile_walk<BT>(p.rows_per_expert, p.num_experts, p.n_tiles, after);
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a.rows[BT / 16 - 1]);
      ptx::prefetch_tensormap(&tmap_w);
    }
  } else if (warp == 1) {
    ptx::tmem_alloc(&ctrl->tmem_base, p.tmem_cols);
    ptx::tmem_relinquish();
  } else if (warp == 2 && lane == 0) {
    for (int s = 0; s < kMxMaxStages; ++s) {
      ptx::mbar_init(&ctrl->full[s], 2);
      ptx::mbar_init(&ctrl->empty[s], 1);
    }
    for (int g = 0; g < kMxSlots; ++g) {
      ptx::mbar_init(&ctrl->sf_full[g], 4);
      ptx::mbar_init(&ctrl->sf_empty[g], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&ctrl->acc_full[a], 1);
      ptx::mbar_init(&ctrl->acc_empty[a], 4);
      ptx::mbar_init(&ctrl->sfw_full[a], 128);
      ptx::mbar_init(&ctrl->sfw_empty[a], 4);
    }
    ptx::mbar_init(&ctrl->tail_full, 4);
    for (int x = 0; x < 2; ++x) ptx::mbar_init(&ctrl->pair_full[x], 2);
    ctrl->abort_flag = 0;
    ptx::fence_barrier_init();
  }
  pdl_wait();
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();

  const uint32_t tmem_base = ctrl->tmem_base;
  const TileWalk walk = tile_walk_at(after, p.num_experts);
  const int total_tiles = walk.total;
  const int tail_kb = (!kW8 && p.tail) ? p.num_kb - 1 : -1;
  constexpr int kWTx = kW8 ? kMxWBytes : kMxWTx;   // bytes a weight-tile load reports
  const int n_groups = (p.num_kb + kMxGroup - 1) / kMxGroup;

  if (warp == 0) {
    // ------------------------------ weight producer ---------------------------
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 1;
      int cursor = 0;
      bool ok = true;
      const uint32_t full0 = ptx::smem_u32(&ctrl->full[0]), empty0 = ptx::smem_u32(&ctrl->empty[0]);
      const uint32_t st0 = ptx::smem_u32(smem);
      uint32_t st = st0;
      const int whole_kb = tail_kb >= 0 ? tail_kb : p.num_kb;   // the partial block does not come this way
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<BT>(walk, t, cursor, ti);
        const int n0 = ti.n_tile * kFeat;
        for (int kb0 = 0; kb0 < p.num_kb; kb0 += kSub) {
          if (!ptx::paced::mbar_wait_s(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          const uint32_t full = full0 + 8 * s;
          ptx::mbar_expect_tx_s(full, max(0, min(kSub, whole_kb - kb0)) * kWTx);
#pragma unroll
          for (int sub = 0; sub < kSub; ++sub) {
            if (kb0 + sub < whole_kb) {
              // kW8: 128 K rows x 128 features, one byte each; rows past K are zero-filled
              if (kW8) ptx::tma_load_3d_s(st + sub * kMxWBytes, &tmap_w, full, n0, (kb0 + sub) * 128, ti.e);
              else ptx::tma_load_3d_s(st + sub * kMxWBytes, &tmap_w, full, (kb0 + sub) * 128, n0, ti.e);
            }
          }
          if (!kW8 && BT > 16 && kb0 + kMxAhead < whole_kb) ptx::tma_prefetch_3d(&tmap_w, (kb0 + kMxAhead) * 128, n0, ti.e);
          st += kStageBytes;
          if (++s == (uint32_t)stages) { s = 0; ph ^= 1; st = st0; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 10) {
    // ------------------------------ token producer ----------------------------
    // (a thread of its own: a TMA instruction occupies the thread that issues it for about 130 cycles)
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 1;
      int cursor = 0;
      bool ok = true;
      const uint32_t full0 = ptx::smem_u32(&ctrl->full[0]), empty0 = ptx::smem_u32(&ctrl->empty[0]);
      const uint32_t st0 = ptx::smem_u32(smem) + kAOff;
      uint32_t st = st0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<BT>(walk, t, cursor, ti);
        const CUtensorMap* tok_map = &tmap_a.rows[BT == 16 ? 0 : (ti.valid - 1) >> 4];
        const int tok_bytes = BT == 16 ? kABytes : ((ti.valid + 15) & ~15) * (kTerms * 128);
        for (int kb0 = 0; kb0 < p.num_kb; kb0 += kSub) {
          if (!ptx::paced::mbar_wait_s(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          const uint32_t full = full0 + 8 * s;
          ptx::mbar_expect_tx_s(full, min(kSub, p.num_kb - kb0) * tok_bytes);
#pragma unroll
          for (int sub = 0; sub < kSub; ++sub)
            if (kb0 + sub < p.num_kb)
              ptx::tma_load_3d_s(st + sub * kABytes, tok_map, full, (kb0 + sub) * 128, ti.row0, 0);   // all planes
          st += kStageBytes;
          if (++s == (uint32_t)stages) { s = 0; ph ^= 1; st = st0; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    // One thread.  A K block is one asm statement on descriptors that differ by an addition from
    // the ring's first: the issuer is a serial chain, and with token tiles of 16 and 64 the chain,
    // not the tensor pipe (38 to 64 cycles per instruction), sets the rate.
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 0, acc_it = 0, slot = 0, slot_ph = 0;
      int cursor = 0;
      bool ok = true;
      const uint32_t full0 = ptx::smem_u32(&ctrl->full[0]), empty0 = ptx::smem_u32(&ctrl->empty[0]);
      const uint32_t sf_full0 = ptx::smem_u32(&ctrl->sf_full[0]), sf_empty0 = ptx::smem_u32(&ctrl->sf_empty[0]);
      const uint32_t tail_full = ptx::smem_u32(&ctrl->tail_full);
      const uint32_t acc_full0 = ptx::smem_u32(&ctrl->acc_full[0]), acc_empty0 = ptx::smem_u32(&ctrl->acc_empty[0]);
      // descriptors: the upper halves do not change, the lower ones hold the address
      const uint64_t adesc_at0 = ptx::make_smem_desc(ptx::smem_u32(smem) + kAOff, 16, 1024);
      const uint64_t wdesc_at0 = ptx::make_smem_desc(ptx::smem_u32(smem), kW8 ? 16384 : 16, 1024);
      const uint64_t sfdesc_at0 = ptx::make_smem_desc_plain(ptx::smem_u32(sf_ring), 128);
      const uint32_t a_hi = (uint32_t)(adesc_at0 >> 32), w_hi = (uint32_t)(wdesc_at0 >> 32), sf_hi = (uint32_t)(sfdesc_at0 >> 32);
      const uint32_t adesc0 = (uint32_t)adesc_at0, wdesc0 = (uint32_t)wdesc_at0, sfdesc0 = (uint32_t)sfdesc_at0;
      const uint32_t tdesc = (uint32_t)ptx::make_smem_desc(ptx::smem_u32(tail_w), 16, 1024);
      uint32_t wdesc = wdesc0, adesc = adesc0, sfdesc = sfdesc0;
      const int whole_kb = tail_kb >= 0 ? tail_kb : p.num_kb;   // K blocks before the partial one
      // A partly filled token tile multiplies only up to its last valid row (UMMA N in steps of 16).
      auto instruction = [&](int t) {
        TileInfo ti;
        locate_tile<BT>(walk, t, cursor, ti);
        return (p.idesc & ~(0x3fu << 17)) | ((uint32_t)(kTerms * ((ti.valid + 15) & ~15)) >> 3 << 17);
      };
      uint32_t idesc_next = (int)blockIdx.x < total_tiles ? instruction(blockIdx.x) : 0u;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const uint32_t a = acc_it & 1;
        const uint32_t idesc = idesc_next;
        const uint32_t d_tmem = tmem_base + a * kNT;
        if (!ptx::mbar_wait_s(acc_empty0 + 8 * a, ((acc_it >> 1) & 1) ^ 1, abort_flag)) break;
        ptx::tc_fence_after();
        auto wait_stage = [&]() {
          const bool go = ptx::mbar_wait_s(full0 + 8 * s, ph, abort_flag);
          ptx::tc_fence_after();
          return go;
        };
        // scales first: tcgen05.cp and tcgen05.mma of one thread execute in issue order
        auto issue = [&](int u, uint32_t w, uint32_t accumulate) {
          ptx::umma_mx_block<kTokChunks, kW8 ? 4096 / 16 : 32 / 16>(
              d_tmem, w, w_hi, adesc + (u % kSub) * (kABytes >> 4), a_hi, idesc, accumulate, tmem_base + kSfBase + u * kSfPer,
              sfdesc + u * 32, sfdesc + kMxGroup * 32 + u * (kTokChunks * 32), sf_hi);
        };
        auto release_stage = [&]() {
          ptx::umma_commit(empty0 + 8 * s);
          wdesc += kStageBytes >> 4;
          adesc += kStageBytes >> 4;
          if (++s == (uint32_t)stages) { s = 0; ph ^= 1; wdesc = wdesc0; adesc = adesc0; }
        };
        for (int kb0 = 0; kb0 < p.num_kb && ok; kb0 += kMxGroup) {
          // the next tile's, while the pipe has work (not between two tiles)
          if (kb0 + kMxGroup >= p.num_kb && t + (int)gridDim.x < total_tiles) idesc_next = instruction(t + gridDim.x);
          if (!ptx::mbar_wait_s(sf_full0 + 8 * slot, slot_ph, abort_flag)) { ok = false; break; }
          ptx::fence_proxy_async();
          if (kb0 + kMxGroup <= whole_kb) {
#pragma unroll
            for (int u = 0; u < kMxGroup; ++u) {
              if (u % kSub == 0 && !wait_stage()) { ok = false; break; }
              issue(u, wdesc + (u % kSub) * (kMxWBytes >> 4), (kb0 > 0 || u > 0) ? 1u : 0u);
              if (u % kSub == kSub - 1) release_stage();
            }
          } else {   // the tile's last, partial group (and the partial K block)
#pragma unroll
            for (int u = 0; u < kMxGroup; ++u) {
              const int kb = kb0 + u;
              if (kb < p.num_kb) {
                if (u % kSub == 0 && !wait_stage()) { ok = false; break; }
                if (kb == tail_kb) {
                  if (!ptx::mbar_wait_s(tail_full, acc_it & 1, abort_flag)) { ok = false; break; }
                  ptx::tc_fence_after();
                }
                issue(u, kb == tail_kb ? tdesc : wdesc + (u % kSub) * (kMxWBytes >> 4), kb > 0 ? 1u : 0u);
                if (u % kSub == kSub - 1 || kb == p.num_kb - 1) release_stage();
              }
            }
          }
          if (!ok) break;
          ptx::umma_commit(sf_empty0 + 8 * slot);
          sfdesc += kSlotBytes >> 4;
          if (++slot == kSlots) { slot = 0; slot_ph ^= 1; sfdesc = sfdesc0; }
        }
        if (ok) { ptx::umma_commit(acc_full0 + 8 * a); ++acc_it; }
      }
    }
    __syncwarp();
  } else if (warp < 6) {
    // ------------------------------ scale preparers ------------------------------
    const int ft = (warp - 2) * 32 + lane;         // 0..127: index in the cooperative copies
    // The weight row whose scales this thread lays out: the word of row r goes to byte
    // (r % 32) * 16 + (r / 32) * 4 of a K block's chunk, so these rows make a warp's stores contiguous.
    const int wrow = (warp - 2) * 8 + (lane >> 2) + 32 * (lane & 3);
    const int kgroups = p.k / 32;
    const int64_t plane_words = (int64_t)p.num_kb * p.m;
    constexpr int kPer = (kMxGroup * kNT + 127) / 128;   // token words per thread and group
    uint32_t slot = 0, slot_ph = 0;
    int cursor = 0, cursor_next = 0, cursor_la = 0;
    bool ok = true;

    // Token scales of one group: thread ft takes words ft + 128 i of [K block][plane][token], coalesced over
    // the lanes, read one group ahead of their use by a look-ahead position (la_*) that runs over the same
    // sequence.  (Two register sets that change roles: a move from one to the other would wait for the loads.)
    auto word_u = [&](int i) { return (ft + 128 * i) / kNT; };
    auto word_tok = [&](int i) { return (ft + 128 * i) % BT; };
    auto word_term = [&](int i) { return (ft + 128 * i) % kNT / BT; };
    uint32_t tok_a[kPer], tok_b[kPer];
    int64_t src[kPer];                                   // word of K block u, row 0
#pragma unroll
    for (int i = 0; i < kPer; ++i) src[i] = word_term(i) * plane_words + (int64_t)word_u(i) * p.m + word_tok(i);
    bool odd = false;
    auto fetch_b = [&](const TileInfo& ti, int g, uint32_t (&db)[kPer]) {
      const uint32_t* base = p.a_scale + (int64_t)(g * kMxGroup) * p.m + ti.row0;
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        db[i] = (ft + 128 * i < kMxGroup * kNT && word_u(i) < p.num_kb - g * kMxGroup && word_tok(i) < ti.valid)
                    ? base[src[i]] : 0x7f7f7f7fu;
    };
    int la_t = blockIdx.x, la_g = 0;
    TileInfo la_ti;
    bool la_valid = la_t < total_tiles;
    if (la_valid) {
      locate_tile<BT>(walk, la_t, cursor_la, la_ti);
      fetch_b(la_ti, 0, tok_a);
    }

    uint32_t tile_seq = 0;
    TileInfo ti, ti_next;
    const bool staged = !kW8 || p.w8_block != 0;   // weight scales come through shared memory
    auto stage = [&](const TileInfo& tn, uint32_t seq) {
      return kW8 ? stage_w_scales_kn(p, ctrl, sfw, tn, seq, ft, kgroups, abort_flag)
                 : stage_w_scales(p, ctrl, sfw, tn, seq, ft, kgroups, abort_flag);
    };
    if (staged && (int)blockIdx.x < total_tiles) {
      locate_tile<BT>(walk, blockIdx.x, cursor_next, ti_next);
      if (!stage(ti_next, 0u)) { *abort_flag = 1; ok = false; }
    }
    for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++tile_seq) {
      locate_tile<BT>(walk, t, cursor, ti);
      const int t_next = t + gridDim.x;
      if (staged && t_next < total_tiles) {
        locate_tile<BT>(walk, t_next, cursor_next, ti_next);
        if (!stage(ti_next, tile_seq + 1)) {
          *abort_flag = 1; ok = false; break;
        }
      }
      const uint32_t b = tile_seq & 1;
      if (staged && !__all_sync(0xffffffffu, ptx::mbar_wait(&ctrl->sfw_full[b], (tile_seq >> 1) & 1, abort_flag))) {
        *abort_flag = 1; ok = false; break;
      }
      const uint32_t sfw_s = ptx::smem_u32(sfw + b * p.sfw_bytes);
      const bool row_ok = ti.n_tile * kFeat + wrow < p.n;
      // Where the token words go: row n of the side-by-side token operand (planes of v16 rows) in the layout
      // tcgen05.cp reads.
      const int v16 = (ti.valid + 15) & ~15;
      uint32_t dst[kPer];
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int n = word_term(i) * v16 + word_tok(i);
        dst[i] = kMxGroup * 512 + word_u(i) * (kTokChunks * 512) + (n >> 7) * 512 + (n & 31) * 16 + ((n >> 5) & 3) * 4;
      }
      auto group = [&](int g, const uint32_t (&use)[kPer], uint32_t (&fill)[kPer]) {
        if (++la_g == n_groups) {
          la_g = 0;
          la_t += gridDim.x;
          la_valid = la_t < total_tiles;
          if (la_valid) locate_tile<BT>(walk, la_t, cursor_la, la_ti);
        }
        if (la_valid) fetch_b(la_ti, la_g, fill);
        // this row's scale bytes of the group's four K blocks, one word each; bytes of groups past
        // the row's end become 0x7f
        uint32_t wa[kMxGroup];
        const int left = kgroups - 16 * g;
        if (!kW8) {
          const uint32_t addr = sfw_s + wrow * kgroups + 16 * g;   // any alignment: aligned words and a funnel shift
          uint32_t v[kMxGroup + 1];
#pragma unroll
          for (int u = 0; u <= kMxGroup; ++u) v[u] = ptx::lds32((addr & ~3u) + 4 * u);
#pragma unroll
          for (int u = 0; u < kMxGroup; ++u) wa[u] = __funnelshift_r(v[u], v[u + 1], (addr & 3u) * 8);
        } else if (p.w8_block) {
          // staged as [group][128 features]: one byte per group
#pragma unroll
          for (int u = 0; u < kMxGroup; ++u) {
            wa[u] = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (4 * u + q < left) wa[u] |= ptx::lds8(sfw_s + (16 * g + 4 * u + q) * 128 + wrow) << (8 * q);
          }
        }
        if (!staged || !row_ok) {   // per-tensor scale: applied in the epilogue
#pragma unroll
          for (int u = 0; u < kMxGroup; ++u) wa[u] = 0x7f7f7f7fu;
        } else if (left < 4 * kMxGroup) {
#pragma unroll
          for (int u = 0; u < kMxGroup; ++u) {
            const int lu = left - 4 * u;
            const uint32_t keep = lu >= 4 ? 0xffffffffu : (lu <= 0 ? 0u : ((1u << (8 * lu)) - 1u));
            wa[u] = (wa[u] & keep) | (0x7f7f7f7fu & ~keep);
          }
        }
        // the ring slot's previous group has been copied to tensor memory
        if (!__all_sync(0xffffffffu, ptx::paced::mbar_wait_s(ptx::smem_u32(&ctrl->sf_empty[slot]), slot_ph ^ 1, abort_flag))) {
          *abort_flag = 1;
          return false;
        }
        const uint32_t ring = ptx::smem_u32(sf_ring) + slot * kSlotBytes;
#pragma unroll
        for (int u = 0; u < kMxGroup; ++u) ptx::sts32(ring + u * 512 + (wrow & 31) * 16 + (wrow >> 5) * 4, wa[u]);
#pragma unroll
        for (int i = 0; i < kPer; ++i)
          if (ft + 128 * i < kMxGroup * kNT && word_tok(i) < v16) ptx::sts32(ring + dst[i], use[i]);
        // (the issuer's proxy fence stands between these writes and its tcgen05.cp: one here would wait for the
        // loads of the next group as well)
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&ctrl->sf_full[slot]);
        if (++slot == kSlots) { slot = 0; slot_ph ^= 1; }
        return true;
      };
      for (int g = 0; g < n_groups && ok; ++g, odd = !odd) ok = odd ? group(g, tok_b, tok_a) : group(g, tok_a, tok_b);
      if (!ok) break;
      if (staged) {
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&ctrl->sfw_empty[b]);
      }
    }
    ptx::cp_async_wait_all();   // staged pieces of an aborted walk
  } else {
    // ------------------------------ epilogue ----------------------------------
    const int q = warp & 3;
    const int et = q * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const int n_out = p.swiglu ? p.n / 2 : p.n;
    uint32_t acc_it = 0, xit = 0;
    int cursor = 0, cursor_next = 0;
    bool ok = true;
    // The partial K block (K = 64 past a multiple of 128): row et's 32 packed bytes, fetched a tile
    // ahead; the other half of the block's codes stay zero, like the tokens' there.
    uint4 tail_q[2] = {};
    auto fetch_tail = [&](const TileInfo& tn) {
      const int f = tn.n_tile * kFeat + et;
      const uint4* src = reinterpret_cast<const uint4*>(p.w + ((int64_t)tn.e * p.n + f) * (p.k / 2) + tail_kb * 64);
      tail_q[0] = f < p.n ? __ldg(src) : make_uint4(0, 0, 0, 0);
      tail_q[1] = f < p.n ? __ldg(src + 1) : make_uint4(0, 0, 0, 0);
    };
    if (tail_kb >= 0) {
      const uint32_t dst = ptx::smem_u32(tail_w) + (et >> 3) * 1024 + (et & 7) * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c) ptx::sts128(dst + c * 16, make_uint4(0, 0, 0, 0));
      if ((int)blockIdx.x < total_tiles) {
        TileInfo tn;
        locate_tile<BT>(walk, blockIdx.x, cursor_next, tn);
        fetch_tail(tn);
      }
    }
    for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      TileInfo ti;
      locate_tile<BT>(walk, t, cursor, ti);
      const int feat = ti.n_tile * kFeat + et;
      const bool feat_ok = feat < p.n;
      float bias_v = 0.f;
      if (p.bias != nullptr && feat_ok) bias_v = load_bias(p.bias, p.out_f16, (int64_t)ti.e * p.n + feat);
      const float w_mul = (kW8 && !p.w8_block) ? p.w_tensor_scale[ti.e] : 1.0f;
      const uint32_t a = acc_it & 1;
      if (tail_kb >= 0) {
        // The previous tile's MMAs are complete (its accumulator has been waited for): write this
        // tile's partial block, row et: 32 packed bytes -> four of the row's eight 16-byte slots
        // (8 data bytes each), slot index xor-ed with (et & 7).
        const uint32_t dst = ptx::smem_u32(tail_w) + (et >> 3) * 1024 + (et & 7) * 128;
        ptx::sts64(dst + ((0 ^ (et & 7)) << 4), tail_q[0].x, tail_q[0].y);
        ptx::sts64(dst + ((1 ^ (et & 7)) << 4), tail_q[0].z, tail_q[0].w);
        ptx::sts64(dst + ((2 ^ (et & 7)) << 4), tail_q[1].x, tail_q[1].y);
        ptx::sts64(dst + ((3 ^ (et & 7)) << 4), tail_q[1].z, tail_q[1].w);
        ptx::fence_proxy_async();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&ctrl->tail_full);
        const int t_next = t + gridDim.x;
        if (t_next < total_tiles) {
          TileInfo tn;
          locate_tile<BT>(walk, t_next, cursor_next, tn);
          fetch_tail(tn);
        }
      }
      // a whole tile's MMAs away: poll from one lane, sleeping in between, so that the
      // wait does not take issue slots from the feeder warp on the same scheduler
      if (!ptx::mbar_wait_warp(&ctrl->acc_full[a], (acc_it >> 1) & 1, abort_flag, 128)) { ok = false; break; }
      ptx::tc_fence_after();
      const uint32_t second = (uint32_t)((ti.valid + 15) & ~15);   // the second plane's first column
#pragma unroll
      for (int c0 = 0; c0 < BT; c0 += kChunk) {
        if (c0 < ti.valid) {
          uint32_t v[kTerms][kChunk];
#pragma unroll
          for (int term = 0; term < kTerms; ++term) {
            const uint32_t col = tmem_base + a * kNT + term * second + c0 + lane_sel;
            if (kChunk == 32) ptx::tmem_ld_32x32(col, reinterpret_cast<uint32_t(&)[32]>(v[term]));
            else ptx::tmem_ld_32x16(col, reinterpret_cast<uint32_t(&)[16]>(v[term]));
          }
          ptx::tmem_wait_ld(v[0], v[kTerms - 1]);
          float vals[kChunk];
#pragma unroll
          for (int i = 0; i < kChunk; ++i) {
            float acc = 0.f + __uint_as_float(v[0][i]);
            if (kTerms == 2) acc += __uint_as_float(v[kTerms - 1][i]);   // the planes' partial results add up
            vals[i] = kW8 ? fmaf(acc, w_mul, bias_v) : acc + bias_v;
          }
          if (p.swiglu) {
            // Gate sits on even features, up on the next odd one: neighbours in the warp.  Of two tokens the even
            // lane takes the first and the odd lane the second, so a pair computes each output once.
            // One branch around the whole block: the unrolled body stays straight-line code, so
            // the shuffle / exp / divide chains overlap instead of running one after another.
            const float c_lim = p.clamp_limit > 0.f ? p.clamp_limit : INFINITY;
            const bool odd = lane & 1;
            float out[kChunk / 2];
#pragma unroll
            for (int j = 0; j < kChunk / 2; ++j) {
              const float mine = odd ? vals[2 * j + 1] : vals[2 * j];
              const float other = __shfl_xor_sync(0xffffffffu, odd ? vals[2 * j] : vals[2 * j + 1], 1);
              float gate = odd ? other : mine;
              float up = odd ? mine : other;
              gate = fminf(gate, c_lim);
              up = fminf(fmaxf(up, -c_lim), c_lim);
              gate = fminf(gate, p.limit);
              up = fminf(fmaxf(up, -p.limit), p.limit);
              out[j] = (up + 1.0f) * gate * __fdividef(1.0f, 1.0f + __expf(-gate * p.alpha));
            }
            if (BT == 16 && p.d_scale != nullptr) {
              // A group of 32 outputs is spread over two warps (q and q ^ 1): both put their 16 of every token into one
              // buffer, from where the first takes them.  Two buffers in turn: who writes one again has seen the
              // other warp arrive for the tile in between, after its reads of the tile before.
              const uint32_t pair = q >> 1, side = q & 1;
              const uint32_t buf = ptx::smem_u32(ctrl->xpose[pair * 2 + (xit & 1)]);
              const uint32_t at = buf + ((lane & 1) * 32 + side * 16 + (lane >> 1)) * 2;
#pragma unroll
              for (int j = 0; j < kChunk / 2; ++j) ptx::sts16(at + j * 128, bits16(out[j], p.out_f16));
              __syncwarp();
              if (lane == 0) ptx::mbar_arrive(&ctrl->pair_full[pair]);
              if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctrl->pair_full[pair], xit & 1, abort_flag))) { ok = false; break; }
              ++xit;
              const int tok = lane >> 1, group = ti.n_tile * 2 + pair;
              if (side == 0)
                store_quantised<kTerms>(buf + lane * 32, p, (int64_t)ti.row0 + tok, tok < ti.valid && group * 32 < n_out, group, lane);
              continue;
            }
            store_pairs_transposed(ctrl->xpose[warp - 6], out, p.d, p.out_f16, (int64_t)ti.row0 + c0, ti.valid - c0, p.m,
                                   n_out, (ti.n_tile * kFeat + q * 32) >> 1, lane);
          } else {
            store_block_transposed<kChunk, 32>(ctrl->xpose[warp - 6], vals, p.d, p.out_f16,
                                               (int64_t)ti.row0 + c0, ti.valid - c0, p.m, n_out,
                                               ti.n_tile * kFeat + q * 32, lane);
          }
        }
      }
      if (!ok) break;
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&ctrl->acc_empty[a]);
      ++acc_it;
    }
  }

  pdl_trigger();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if (*abort_flag != 0) __nanosleep(20000);
    ptx::tmem_dealloc(tmem_base, p.tmem_cols);
  }
  if (tid == 0 && *abort_flag != 0) report_timeout(p.status);
}

template <int BT, int kTerms, int kSub, bool kW8>
int launch_mx(const b200moe_gemm_args* a, const CUtensorMap& tw, MxParams& p, int grid, cudaStream_t st) {
  MxTokenMaps<BT> ta;
  for (int i = 0; i < BT / 16; ++i) {
    cuuint64_t dims[3] = {(cuuint64_t)a->k, (cuuint64_t)a->m, (cuuint64_t)kTerms};
    cuuint64_t strides[2] = {(cuuint64_t)a->k, (cuuint64_t)a->k * (cuuint64_t)a->m};
    cuuint32_t box[3] = {128, (cuuint32_t)(16 * (i + 1)), (cuuint32_t)kTerms};
    if (int rc = encode_map(&ta.rows[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a->a, dims, strides, box)) return rc;
  }
  auto kern = grouped_gemm_mx_kernel<BT, kTerms, kSub, kW8>;
  const uint32_t need = 2 * kTerms * BT + kMxGroup * (kTerms * BT > 128 ? 16 : 8);
  p.tmem_cols = need <= 128 ? 128u : (need <= 256 ? 256u : 512u);
  const int body = kSub * (kMxWBytes + kTerms * BT * 128);
  const int fixed = 1024 + (p.tail ? kMxWBytes : 0) + mx_slots<kTerms * BT>() * mx_slot_bytes<kTerms * BT>() +
                    (int)((sizeof(MxCtrl) + 15) & ~(size_t)15) + tile_walk_bytes(p.num_experts) + 2 * p.sfw_bytes;
  p.stages = (227 * 1024 - fixed) / body;
  if (p.stages > kMxMaxStages) p.stages = kMxMaxStages;
  if (p.stages < 2) return fail(B200MOE_E_UNSUPPORTED, "block-scaled GEMM: tile does not fit shared memory");
  const size_t smem = (size_t)fixed + (size_t)p.stages * body;
  static SmemConfig configured;
  if (int rc = configured.ensure(kern)) return rc;
  B200_LAUNCHED("grouped_gemm_mx_kernel", launch_pdl(p.m <= kMxEarlyLaunchRows, kern, dim3(grid), dim3(kMxThreads), smem, st, ta, tw, p));
  return B200MOE_OK;
}

}  // namespace

// MXFP4 weights x MXFP8 activations (one plane, or two with the residual) on the
// block-scaled tensor-core path.  a: codes [terms][M,K]; a_scale: 32-bit words
// [terms][ceil(K/128)][M] of four e8m0 bytes (what b200moe_quant_mxfp8 writes).
// Returns B200MOE_E_UNSUPPORTED (no launch) for anything else.
int grouped_gemm_tc_mx(const b200moe_gemm_args* a, cudaStream_t st) {
  const bool x2 = a->a_dtype == B200MOE_FP8_E4M3_X2;
  const bool w4 = a->w_format == B200MOE_W_MXFP4_NK;
  const bool w8mx = a->w_format == B200MOE_W_MXFP8_KN;
  const bool w8 = a->w_format == B200MOE_W_FP8_TENSOR_KN || a->w_format == B200MOE_W_FP8E5M2_TENSOR_KN || w8mx;
  if (!(w4 || w8) || !(a->a_dtype == B200MOE_FP8_E4M3 || x2) || a->a_scale == nullptr)
    return fail(B200MOE_E_UNSUPPORTED,
                "block-scaled GEMM takes MXFP4, MXFP8 or per-tensor fp8 weights and MXFP8 activations");
  if (a->epilogue == B200MOE_EPI_SILU_MUL)
    return fail(B200MOE_E_UNSUPPORTED, "block-scaled GEMM: SiLU epilogue not available");
  if (a->num_experts > kMaxExperts || a->k % 32 != 0 || a->k < 128 || (w4 && a->k % 64 != 0))
    return fail(B200MOE_E_UNSUPPORTED, "block-scaled GEMM: K must be a multiple of 64 (fp8 weights: 32), at least 128");
  if (w8 && a->n % 16 != 0)
    return fail(B200MOE_E_UNSUPPORTED, "block-scaled GEMM: N must be a multiple of 16 for [E,K,N] fp8 weights");
  if (((uintptr_t)a->a & 15) || ((uintptr_t)a->w & 31) || ((uintptr_t)a->d & 15) || ((uintptr_t)a->a_scale & 3))
    return fail(B200MOE_E_BADARG, "block-scaled GEMM: A and D must be 16-byte, W 32-byte, A scales 4-byte aligned");
  if (a->epilogue == B200MOE_EPI_SWIGLUOAI && (a->n / 2) % 8 != 0)
    return fail(B200MOE_E_UNSUPPORTED, "block-scaled GEMM: gated output width must be a multiple of 8");
  if (x2 && (a->m * (int64_t)a->k) % 16 != 0)
    return fail(B200MOE_E_UNSUPPORTED, "block-scaled GEMM: the second activation plane must be 16-byte aligned");
  if (a->m == 0 || a->n == 0) return B200MOE_OK;

  MxParams p;
  p.w = reinterpret_cast<const uint8_t*>(a->w);
  p.w_scale = reinterpret_cast<const uint8_t*>(a->w_scale);
  p.w_tensor_scale = reinterpret_cast<const float*>(a->w_scale);
  p.a_scale = reinterpret_cast<const uint32_t*>(a->a_scale);
  p.bias = a->bias; p.d = a->d; p.rows_per_expert = a->rows_per_expert; p.status = a->status;
  p.m = a->m; p.n = a->n; p.k = a->k; p.num_experts = a->num_experts;
  p.n_tiles = (a->n + kFeat - 1) / kFeat;
  p.num_kb = (a->k + 127) / 128;
  p.terms = x2 ? 2 : 1;
  p.tail = w4 && (a->k % 128) != 0;
  p.sfw_bytes = 0;
  p.w8_block = w8mx ? 1 : 0;
  if (w8mx) {
    // per K group the tile's 128 scale bytes: whole 16-byte chunks from a 16-byte aligned tensor
    const int piece = 128 * (a->k / 32);
    if (((uintptr_t)a->w_scale & 15) != 0 || piece > kMxSfwCap)
      return fail(B200MOE_E_UNSUPPORTED, "block-scaled GEMM: K at most 6144, scales 16-byte aligned");
    p.sfw_bytes = piece;
  }
  if (w4) {
    // The weight scales of a tile (128 rows x K/32 bytes, contiguous in the scale
    // tensor) are staged in shared memory: every tile's piece must start on a
    // 16-byte boundary and two pieces must fit.
    const int kgroups = a->k / 32;
    const int piece = ((128 * kgroups + 15) & ~15) + 32;   // the last row's words are read past its end
    if (((uintptr_t)a->w_scale & 15) != 0 || ((int64_t)a->n * kgroups) % 16 != 0 || piece > kMxSfwCap)
      return fail(B200MOE_E_UNSUPPORTED,
                  "block-scaled GEMM: N * K / 32 must be a multiple of 16, K at most 6144, scales 16-byte aligned");
    p.sfw_bytes = piece;
  }
  p.out_f16 = a->d_dtype == B200MOE_F16;
  p.swiglu = a->epilogue == B200MOE_EPI_SWIGLUOAI;
  p.alpha = a->act_alpha; p.limit = a->act_limit; p.clamp_limit = a->clamp_limit;
  const bool quantised = a->d_dtype == B200MOE_FP8_E4M3 || a->d_dtype == B200MOE_FP8_E4M3_X2;
  p.d_scale = quantised ? reinterpret_cast<uint32_t*>(a->d_scale) : nullptr;
  if (quantised) p.out_f16 = a->mid_dtype == B200MOE_F16;

  const int64_t rows_in_use = (a->rows_hint > 0 && a->rows_hint < a->m) ? a->rows_hint : a->m;
  const int64_t avg = (rows_in_use + a->num_experts - 1) / a->num_experts;
  int bt = avg <= 8 ? 16 : (avg <= 40 ? 64 : 128);
  // both planes' accumulators share tensor memory: two planes of 96 tokens are one MMA of
  // N = 192 (enough work per instruction to keep the tensor pipe busy), two stages of them
  // and the scale columns fill the 512 columns
  if (x2 && bt > 64) bt = avg > 48 ? 96 : 64;
  if (!x2 && avg > 128) bt = 192;               // one plane: the same N = 192 instruction
  if (quantised) bt = 16;   // (the other tiles have no such epilogue)
  // Measured, 128 experts, N 5760, K 2880.  Two planes at 16 / 64 / 96 tokens: 8 rows per expert 238 / 305
  // / 373 us, 16 rows 305 / 309 / 373, 48 rows 670 / 356 / 426, 64 rows - / 469 / 430; one plane at 16 / 64
  // / 128 / 192: 8 rows 232 / 283 / 301 / 347, 16 rows 313 / 285 / 300 / 350, 40 rows 549 / 318 / 322 / 367,
  // 64 rows - / 416 / 330 / 385, 128 rows - / 635 / 811 / 562.  Segments around a multiple of the tile
  // cost a second tile: at 96 rows two planes take 667 us with 64 tokens and 842 with 96 (K 2880, N 2880:
  // 313 and 293), at 192 rows 1178 and 1381 (534 and 498).
  // weights: e2m1 K-major, or e4m3 / e5m2 MN-major; activations e4m3 K-major
  const uint32_t a_fmt = w4 ? 5u : (a->w_format == B200MOE_W_FP8E5M2_TENSOR_KN ? 1u : 0u);
  p.idesc = ptx::make_idesc_mx(a_fmt, 0u, kFeat, (uint32_t)(bt * p.terms)) | (w8 ? (1u << 15) : 0u);

  CUtensorMap tw;
  if (w8) {
    cuuint64_t dims[3] = {(cuuint64_t)a->n, (cuuint64_t)a->k, (cuuint64_t)a->num_experts};
    cuuint64_t strides[2] = {(cuuint64_t)a->n, (cuuint64_t)a->k * a->n};
    cuuint32_t box[3] = {128, 128, 1};
    int rc = encode_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a->w, dims, strides, box);
    if (rc) return rc;
  } else {
    {
      // Whole 128-code blocks only: this tensor-map type wants the inner extent to be
      // a multiple of 128 codes; the row pitch stays K/2 bytes.
      cuuint64_t dims[3] = {(cuuint64_t)(a->k - a->k % 128), (cuuint64_t)a->n, (cuuint64_t)a->num_experts};
      cuuint64_t strides[2] = {(cuuint64_t)(a->k / 2), (cuuint64_t)(a->k / 2) * a->n};
      cuuint32_t box[3] = {128, (cuuint32_t)kFeat, 1};
      int rc = encode_map(&tw, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 3, a->w, dims, strides, box);
      if (rc) return rc;
    }
  }
  const int64_t tile_bound = ((a->m + bt - 1) / bt + a->num_experts) * (int64_t)p.n_tiles;
  int grid = sm_count();
  if (a->max_ctas > 0 && a->max_ctas < grid) grid = a->max_ctas;
  if (tile_bound < grid) grid = (int)tile_bound;
  if (grid < 1) grid = 1;
  // Small token tiles move two K blocks per pipeline stage.
#define B200_MX_CASES(W8)                                                              \
  if (x2) {                                                                            \
    if (bt == 16) return launch_mx<16, 2, 2, W8>(a, tw, p, grid, st);                 \
    if (bt == 96) return launch_mx<96, 2, 1, W8>(a, tw, p, grid, st);                 \
    return launch_mx<64, 2, 1, W8>(a, tw, p, grid, st);                               \
  }                                                                                    \
  if (bt == 192) return launch_mx<192, 1, 1, W8>(a, tw, p, grid, st);                 \
  if (bt == 16) return launch_mx<16, 1, 2, W8>(a, tw, p, grid, st);                   \
  if (bt == 64) return launch_mx<64, 1, 2, W8>(a, tw, p, grid, st);                   \
  return launch_mx<128, 1, 1, W8>(a, tw, p, grid, st);
  if (w8) { B200_MX_CASES(true) }
  B200_MX_CASES(false)
#undef B200_MX_CASES
}

}  // namespace b200moe
