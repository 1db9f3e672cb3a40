// INT4 x quantised activations on the block-scaled tensor-core instruction.
//
//   D[m, f] = sum_g scale[f, g] * sum_{k in g} (u[f, k] - 8) * a[m, k]  (+ bias),  u = nibble ^ 8
//
// Weights [E,N,K/2] are two's-complement nibbles with one 16-bit scale per row and 128 or 256 K
// elements.  A nibble u in 0..15, put into a byte, IS the e4m3 number u * 2^-9 (the subnormals and
// the first binade of e4m3 are linear), so unpacking is the whole conversion: three instructions per
// eight weights where the tokens' codes come with the even ones first, too (a layer's do), two more to put the
// weights in order where they don't (33 tokens x top-2 of 8 experts of 4096 x 14336, a layer call 223 -> 219 us
// without), against seventeen for the 16-bit expansion of gemm_tc_dq.cu, whose integer pipe is the bound when there
// are few tokens.  The activations are e4m3 planes with one power-of-two
// scale per 32 values (mx_quant.cuh): two planes hold a bfloat16 exactly, three a float16 (values
// 2^-14 of the group's largest and smaller excepted, whose error stays below 2^-21 of it), so
// nothing is lost against 16-bit activations, and the weight is not rounded after its scale is applied.
//
// The zero point and the group scales are applied where a 128-wide K block's sum leaves tensor
// memory: with features on the lanes the scale is one register per thread, and 8 * sum_k a[m, k] (kept
// by the quantiser for every block) comes from shared memory, the same for all lanes.
//
// Roles (768 threads in warpgroups that re-balance registers, one persistent CTA per SM; tiles of
// 128 features x BT tokens):
//   warp 0       : TMA producer: per K block 128 x 64 packed bytes and the planes' BT x 128 bytes
//   warps 1-2    : MMA issuers, a thread each, which take K blocks in turn; they copy the tokens' scale
//                  factors to tensor memory (tcgen05.cp); the planes accumulate in the same columns, so the
//                  promotion reads BT columns only
//   warp 3       : brings the tokens' scale words and sums, four K blocks at a time
//   warps 4-15   : converters, three sets that take K blocks in turn (a set is one long chain of
//                  latencies, 630 cycles per block): a thread unpacks a row's 64 bytes into 32 columns
//                  of tensor memory, from where the MMA reads the weights (nothing goes back through
//                  shared memory)
//   warps 16-23  : promotion and epilogue; warp w owns lane quarter w & 3 and half of the columns
// What bounds it is none of the units but the chain of hand-overs of a K block: a look at an mbarrier that is
// already complete costs its warp about 100 cycles, an arrival as much, and one issuer that waited for the stage,
// the operand, the accumulator and the scales needed 620 cycles a block.  So there are two issuers, and each
// hand-over stands for all that it implies: the converters' arrival for the stage's tokens (they waited for the
// same stage), an accumulator's completion for its operand columns and for the group's scales, and a stage is
// released with the arrival of the block kI4Conv further on, which waited for the MMAs of the one before.
// 33 tokens x top-2 of 8 experts, 28672 x 4096 and 4096 x 14336: 144 -> 135 and 97 -> 94.5 us; the next in the
// row are the promotion warps (540 cycles a block).
// Waits are bounded as in the other kernels (sm100_ptx.cuh).
#include <algorithm>

#include "common.cuh"
#include "gemm_tc_common.cuh"
#include "sm100_ptx.cuh"

namespace b200moe {
namespace {

constexpr int kI4RawBytes = 8192;    // 128 rows x 64 packed bytes
constexpr int kI4Threads = 768;
constexpr int kI4LaunchRegs = 80, kI4FeedRegs = 64, kI4ConvRegs = 56, kI4PromoRegs = 120;   // warpgroups 0, 1-3, 4-5
static_assert(128 * kI4FeedRegs + 384 * kI4ConvRegs + 256 * kI4PromoRegs <= kI4Threads * kI4LaunchRegs, "setmaxnreg budget");
constexpr int kI4MaxStages = 12;
constexpr int kI4Group = 4;          // K blocks per hand-over of token scales
constexpr int kI4Slots = 3;
constexpr int kI4Sets = 3;           // converter sets
constexpr int kI4Issuers = 2;        // threads that issue MMAs
// Blocks in tensor memory: operand (32 columns), token scales and accumulator of block i are slot i % kI4Conv.
constexpr int kI4Conv = 6;
// A slot stays with one issuer, whose instructions execute in order, and with one converter set, which has seen
// the slot's block before the last complete when it waits for the last by parity.
static_assert(kI4Conv % kI4Issuers == 0 && kI4Conv % kI4Sets == 0, "slots");

struct I4Params {
  const uint16_t* w_scale;   // [E, N, groups] in the activation type
  const uint32_t* a_scale;   // [planes][num_kb][M] words of four e8m0 bytes, then float sums [num_kb][M]
  const void* bias;
  void* d;
  const int32_t* rows_per_expert;
  int32_t* status;
  int64_t m;
  int n, k, num_experts;
  int n_tiles, num_kb;
  int groups, kb_shift;      // scales per weight row; scale index = K block >> kb_shift
  int stages, stages_wide;   // of the ring (with the 32-token tile, where the kernel chooses)
  int ctrl_at;
  int rows_ready;            // 1: prefetch_first_tiles
  uint32_t idesc;
  int out_f16;
};

constexpr uint32_t kI4Tmem = 512;    // columns

template <int BT, int kTerms>
struct I4Shape {
  static constexpr int kTokChunks = kTerms > 2 ? 2 : 1;       // scale chunks: two columns per plane
  static constexpr int kABytes = kTerms * BT * 128;
  static constexpr int kStageBytes = kI4RawBytes + kABytes;
  static constexpr int kSfPer = 4 * kTokChunks;               // tokens' scale columns of a K block
  static constexpr uint32_t kConvBase = kI4Conv * BT;
  static constexpr uint32_t kSfBase = kConvBase + kI4Conv * 32;   // weights' scale columns (constant), then the tokens'
  static constexpr uint32_t kCols = kSfBase + 8 + kI4Conv * kSfPer;
  static constexpr int kSlotBytes = kI4Group * (512 * kTokChunks + BT * 4);
  static_assert(BT <= 32 && kCols <= kI4Tmem, "tensor memory");
};

struct I4Ctrl {
  uint64_t full[kI4MaxStages];
  uint64_t empty[kI4MaxStages];      // the converters, which have read the packed weights, and one of them for the MMA
  uint64_t conv_full[kI4Conv];
  uint64_t acc_full[kI4Conv];        // the block's MMAs are complete (its operand columns are free, too)
  uint64_t acc_empty[kI4Conv];
  uint64_t sf_full[kI4Slots];
  uint64_t sf_empty[kI4Slots];       // the promotion warps, which have seen the group's MMAs complete
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) uint16_t xpose[8][16 * 32];   // per promotion warp: output transpose tile
};

// Shared memory: ring and token scales, then from p.ctrl_at on the control block and the tile walk (or two).
constexpr int kI4CtrlBytes = (int)((sizeof(I4Ctrl) + 15) & ~(size_t)15);
__device__ __forceinline__ uint8_t* i4_smem() {
  extern __shared__ uint8_t smem_raw[];
  return reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
}

// Everything that comes before the first tile; with kEither the walk over 32-token tiles, too, behind the other one.
template <int BT, bool kEither>
__device__ __forceinline__ void grouped_gemm_i4_kernel_prologue(const CUtensorMap& tmap_a, const CUtensorMap& tmap_w,
                                                                const I4Params& p, I4Ctrl* ctrl, uint8_t* walk_mem) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    if (p.rows_ready)
      prefetch_first_tiles<BT>(p.rows_per_expert, p.num_experts, 0, p.n_tiles, p.num_kb, kPreBytes / kI4RawBytes, walk_mem,
                               [&](const TileInfo& ti, int kb) { ptx::tma_prefetch_3d(&tmap_w, kb * 64, ti.n_tile * kFeat, ti.e); });
    pdl_wait();
    build_tile_walk<BT>(p.rows_per_expert, p.num_experts, p.n_tiles, walk_mem);
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a);
      ptx::prefetch_tensormap(&tmap_w);
    }
  } else if (warp == 1) {
    ptx::tmem_alloc(&ctrl->tmem_base, kI4Tmem);
    ptx::tmem_relinquish();
  } else if (warp == 2 && lane == 0) {
    for (int s = 0; s < kI4MaxStages; ++s) {
      ptx::mbar_init(&ctrl->full[s], 1);
      ptx::mbar_init(&ctrl->empty[s], 1 + 4);
    }
    for (int c = 0; c < kI4Conv; ++c) {
      ptx::mbar_init(&ctrl->conv_full[c], 4);
    }
    for (int a = 0; a < kI4Conv; ++a) {
      ptx::mbar_init(&ctrl->acc_full[a], 2);   // the MMAs, and the issuer for the sums it has seen
      ptx::mbar_init(&ctrl->acc_empty[a], 8);
    }
    for (int g = 0; g < kI4Slots; ++g) {
      ptx::mbar_init(&ctrl->sf_full[g], 1);
      ptx::mbar_init(&ctrl->sf_empty[g], 8);
    }
    ctrl->abort_flag = 0;
    ptx::fence_barrier_init();
  } else if (kEither && warp == 3) {
    pdl_wait();
    build_tile_walk<32>(p.rows_per_expert, p.num_experts, p.n_tiles, walk_mem + tile_walk_bytes(p.num_experts));
  }
  pdl_wait();
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
}

template <int BT, int kTerms, bool kEvensFirst>
__device__ __forceinline__ void grouped_gemm_i4_kernel_body(const CUtensorMap& tmap_a, const CUtensorMap& tmap_w,
                                                            const I4Params& p, int stages, uint8_t* smem, I4Ctrl* ctrl,
                                                            const uint8_t* walk_mem) {
  using S = I4Shape<BT, kTerms>;
  constexpr int kStageBytes = S::kStageBytes, kSlotBytes = S::kSlotBytes;
  uint8_t* sf_ring = smem + stages * kStageBytes;
  volatile int* abort_flag = &ctrl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t tmem_base = ctrl->tmem_base;
  if (warp >= 4 && warp < 8) {
    // the weights' scale factors: 2^9 everywhere, which makes the codes the integers 0..15
    const uint32_t c9[4] = {0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u};
    ptx::tmem_st_32x4(tmem_base + S::kSfBase + ((uint32_t)((warp & 3) * 32) << 16), c9[0], c9[1], c9[2], c9[3]);
    ptx::tmem_wait_st();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();

  const TileWalk walk = tile_walk_at(walk_mem, p.num_experts);
  const int total_tiles = walk.total;
  const uint32_t full0 = ptx::smem_u32(&ctrl->full[0]), empty0 = ptx::smem_u32(&ctrl->empty[0]);
  const uint32_t conv_full0 = ptx::smem_u32(&ctrl->conv_full[0]);
  const uint32_t acc_full0 = ptx::smem_u32(&ctrl->acc_full[0]), acc_empty0 = ptx::smem_u32(&ctrl->acc_empty[0]);
  const uint32_t sf_full0 = ptx::smem_u32(&ctrl->sf_full[0]), sf_empty0 = ptx::smem_u32(&ctrl->sf_empty[0]);
  int my_tiles = 0;
  for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) ++my_tiles;

  if (warp < 4) {
    ptx::setmaxnreg_dec<kI4FeedRegs>();
    if (warp == 0) {
      // ------------------------------ TMA producer ------------------------------
      if (ptx::elect_one()) {
        uint32_t s = 0, ph = 1;
        int cursor = 0;
        bool ok = true;
        const uint32_t st0 = ptx::smem_u32(smem);
        uint32_t st = st0;
        for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
          TileInfo ti;
          locate_tile<BT>(walk, t, cursor, ti);
          const int n0 = ti.n_tile * kFeat;
          for (int kb = 0; kb < p.num_kb; ++kb) {
            const uint32_t full = full0 + 8 * s;
            if (!ptx::paced::mbar_wait_s(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
            ptx::mbar_expect_tx_s(full, kStageBytes);
            ptx::tma_load_3d_s(st, &tmap_w, full, kb * 64, n0, ti.e);
            ptx::tma_load_3d_s(st + kI4RawBytes, &tmap_a, full, kb * 128, ti.row0, 0);   // all planes
            st += kStageBytes;
            if (++s == (uint32_t)stages) { s = 0; ph ^= 1; st = st0; }
          }
        }
      }
      __syncwarp();
    } else if (warp <= kI4Issuers) {
      // ------------------------------ MMA issuers -------------------------------
      // Every kI4Issuers-th block each: blocks have accumulators of their own, so their order does not matter.
      if (ptx::elect_one()) {
        const uint32_t mine = warp - 1;
        uint32_t turn = 0, c = 0, cph = 0, s = 0;      // whose block, its slot, its ring stage
        uint32_t u = 0, slot = 0, slot_ph = 0;         // its place in the group of scales, the group's
        int cursor = 0;
        bool ok = true;
        const uint64_t adesc_at0 = ptx::make_smem_desc(ptx::smem_u32(smem) + kI4RawBytes, 16, 1024);
        const uint32_t adesc0 = (uint32_t)adesc_at0, a_hi = (uint32_t)(adesc_at0 >> 32);
        const uint64_t sfdesc0 = ptx::make_smem_desc_plain(ptx::smem_u32(sf_ring), 128);
        const uint32_t sf = tmem_base + S::kSfBase;
        for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
          TileInfo ti;
          locate_tile<BT>(walk, t, cursor, ti);
          // a partly filled token tile multiplies only its valid columns (UMMA N in steps of 16)
          const uint32_t n_eff = (uint32_t)((ti.valid + 15) & ~15);
          const uint32_t idesc = (p.idesc & ~(0x3fu << 17)) | ((n_eff >> 3) << 17);
#pragma unroll 1
          for (int kb = 0; kb < p.num_kb; ++kb) {
            if (turn == mine) {
              // (the converters have seen the block's loads land, the tokens' among them)
              if ((u < kI4Issuers && !ptx::mbar_wait_s(sf_full0 + 8 * slot, slot_ph, abort_flag)) ||
                  !ptx::mbar_wait_s(conv_full0 + 8 * c, cph, abort_flag) ||
                  !ptx::mbar_wait_s(acc_empty0 + 8 * c, cph ^ 1, abort_flag)) { ok = false; break; }
              // tcgen05.commit completes the MMAs and orders nothing else: the group's sums, written by warp 3, reach
              // the promotion warps through this arrival (acquired above, released here)
              ptx::mbar_arrive_s(acc_full0 + 8 * c);
              ptx::tc_fence_after();
              const uint32_t sfa = sf + 8 + c * S::kSfPer, adesc = adesc0 + s * (kStageBytes >> 4);
              const uint64_t sfd = sfdesc0 + slot * (kSlotBytes >> 4) + u * (S::kTokChunks * 32);
              ptx::tmem_cp_scales(sfa, sfd);
              if (S::kTokChunks == 2) ptx::tmem_cp_scales(sfa + 4, sfd + 32);
#pragma unroll
              for (int term = 0; term < kTerms; ++term)
                ptx::umma_mx_block_ts(tmem_base + c * BT, tmem_base + S::kConvBase + c * 32, adesc + term * (BT * 128 >> 4), a_hi,
                                      idesc, term > 0 ? 1u : 0u, sf, sfa + 2 * term);
              ptx::umma_commit(acc_full0 + 8 * c);
            }
            if (++turn == kI4Issuers) turn = 0;
            if (++c == kI4Conv) { c = 0; cph ^= 1; }
            if (++s == (uint32_t)stages) s = 0;
            if (++u == kI4Group || kb + 1 == p.num_kb) {
              u = 0;
              if (++slot == kI4Slots) { slot = 0; slot_ph ^= 1; }
            }
          }
        }
      }
      __syncwarp();
    } else {
      // ------------------------ tokens' scales and sums ---------------------------
      const int ft = lane;
      constexpr int kPer = kI4Group * kTerms * BT / 32, kPerSum = kI4Group * BT / 32;
      const int tok = ft % BT;
      const int64_t plane_words = (int64_t)p.num_kb * p.m;
      uint32_t slot = 0, slot_ph = 1;
      int cursor = 0;
      bool ok = true;
      // (the ring is deep enough to hide the loads' latency)
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<BT>(walk, t, cursor, ti);
        for (int kb0 = 0; kb0 < p.num_kb; kb0 += kI4Group) {
          const uint32_t* words = p.a_scale + ((int64_t)kb0 * p.m + ti.row0 + tok);
          uint32_t w[kPer];
          float m[kPerSum];
          // token, plane and K block of a word: lane % BT, then planes, then blocks (with all three from one number, lane +
          // 32 * i, the addresses did not fit the registers: three planes in the choosing kernel 4 to 5 % slower)
  #pragma unroll
          for (int i = 0; i < kPer; ++i) {
            const int j = i * (32 / BT) + ft / BT, u = j / kTerms, kb = kb0 + u;
            w[i] = (kb < p.num_kb && tok < ti.valid) ? words[(j % kTerms) * plane_words + (int64_t)u * p.m] : 0x7f7f7f7fu;
          }
  #pragma unroll
          for (int i = 0; i < kPerSum; ++i) {
            const int u = i * (32 / BT) + ft / BT, kb = kb0 + u;
            m[i] = (kb < p.num_kb && tok < ti.valid) ? -8.0f * __uint_as_float(words[kTerms * plane_words + (int64_t)u * p.m]) : 0.f;
          }
          if (!__all_sync(0xffffffffu, ptx::paced::mbar_wait_s(sf_empty0 + 8 * slot, slot_ph, abort_flag))) { ok = false; break; }
          const uint32_t ring = ptx::smem_u32(sf_ring) + slot * kSlotBytes;
  #pragma unroll
          for (int i = 0; i < kPer; ++i) {
            // plane `term` takes the columns 2 * term and 2 * term + 1 (an MMA's scales start on an even one)
            const int j = i * (32 / BT) + ft / BT, u = j / kTerms, term = j % kTerms;
            ptx::sts32(ring + u * (S::kTokChunks * 512) + (term >> 1) * 512 + (tok & 31) * 16 + ((2 * term + (tok >> 5)) & 3) * 4,
                       w[i]);
          }
  #pragma unroll
          for (int i = 0; i < kPerSum; ++i)
            ptx::sts32f(ring + kI4Group * 512 * S::kTokChunks + (ft + 32 * i) * 4, m[i]);
          ptx::fence_proxy_async();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_s(sf_full0 + 8 * slot);
          if (++slot == kI4Slots) { slot = 0; slot_ph ^= 1; }
        }
      }
    }
  } else if (warp < 16) {
    ptx::setmaxnreg_dec<kI4ConvRegs>();
    // ------------------------------ converters ------------------------------
    const int row = (warp & 3) * 32 + lane, set = (warp - 4) >> 2;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t src0 = ptx::smem_u32(smem) + row * 64;
    const uint32_t swz = (uint32_t)((row >> 1) & 3) << 4;      // 64-byte swizzle: chunk index xor row bits 1..2
    uint32_t s = set, ph = 0, c = set, cph = 0;
    const uint32_t blocks = (uint32_t)my_tiles * p.num_kb;      // every tile: the same K loop
    for (uint32_t i = set; i < blocks; i += kI4Sets) {
      if (!__all_sync(0xffffffffu, ptx::paced::mbar_wait_s(full0 + 8 * s, ph, abort_flag))) break;
      const uint32_t src = src0 + s * kStageBytes;
      uint32_t o[32];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 v = ptx::lds128(src + ((uint32_t)(q * 16) ^ swz));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // nibbles of even and of odd k as bytes (sign bit flipped: 0..15), in the order of the tokens' codes
          const uint32_t e = (w[j] & 0x0f0f0f0fu) ^ 0x08080808u, d = ((w[j] >> 4) & 0x0f0f0f0fu) ^ 0x08080808u;
          o[q * 8 + 2 * j] = kEvensFirst ? e : __byte_perm(e, d, 0x5140);
          o[q * 8 + 2 * j + 1] = kEvensFirst ? d : __byte_perm(e, d, 0x7362);
        }
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_s(empty0 + 8 * s);
      // the operand columns are free when the MMAs of the slot's block before are complete: its accumulator is full
      if (!__all_sync(0xffffffffu, ptx::paced::mbar_wait_s(acc_full0 + 8 * c, cph ^ 1, abort_flag))) break;
      ptx::tc_fence_after();
      ptx::tmem_st_32x32(tmem_base + S::kConvBase + c * 32 + lane_sel, o);
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      // ... and the MMAs of block i - kI4Conv are done with their stage's tokens
      const uint32_t old = s >= kI4Conv ? s - kI4Conv : s + stages - kI4Conv;
      __syncwarp();
      ptx::mbar_arrive_if(conv_full0 + 8 * c, lane == 0, empty0 + 8 * old, (warp & 3) == 0 && i >= kI4Conv);
      c += kI4Sets;
      if (c >= kI4Conv) { c -= kI4Conv; cph ^= 1; }
      s += kI4Sets;
      if (s >= (uint32_t)stages) { s -= stages; ph ^= 1; }
    }
  } else {
    ptx::setmaxnreg_inc<kI4PromoRegs>();
    // ------------------------ promotion and epilogue --------------------------
    constexpr int kHalf = BT / 2;                  // columns of this warp
    const int q = warp & 3, half = (warp - 16) >> 2;
    const int et = q * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const int col0 = half * kHalf;
    uint32_t a = 0, aph = 0, slot = 0;
    int cursor = 0;
    bool ok = true;
    const bool vec4 = p.kb_shift == 0 && p.groups % 4 == 0 && (reinterpret_cast<uintptr_t>(p.w_scale) & 7) == 0;
    for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      TileInfo ti;
      locate_tile<BT>(walk, t, cursor, ti);
      const int feat = ti.n_tile * kFeat + et;
      const bool feat_ok = feat < p.n;
      const float bias_v = (p.bias != nullptr && feat_ok) ? load_bias(p.bias, p.out_f16, (int64_t)ti.e * p.n + feat) : 0.f;
      const uint16_t* srow = p.w_scale + ((int64_t)ti.e * p.n + (feat_ok ? feat : 0)) * p.groups;
      const bool mine = col0 < ti.valid;           // any valid column in this warp's half
      // the four scales of a group of K blocks (packed 16-bit), read one group ahead
      auto scales_of = [&](int kb0) {
        uint2 r = make_uint2(0u, 0u);
        if (vec4) {
          if (kb0 < p.groups) r = __ldg(reinterpret_cast<const uint2*>(srow + kb0));
        } else {
          uint32_t h[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int g = (kb0 + u) >> p.kb_shift;
            h[u] = g < p.groups ? __ldg(srow + g) : 0;
          }
          r = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
        }
        return r;
      };
      float2 acc[kHalf / 2];
#pragma unroll
      for (int i = 0; i < kHalf / 2; ++i) acc[i] = make_float2(0.f, 0.f);
      uint2 nxt = scales_of(0);
      for (int kb0 = 0; kb0 < p.num_kb && ok; kb0 += kI4Group) {
        const uint2 cur = nxt;
        nxt = scales_of(kb0 + kI4Group);
        float sc[kI4Group];
        if (p.out_f16) {
          const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&cur.x));
          const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&cur.y));
          sc[0] = lo.x; sc[1] = lo.y; sc[2] = hi.x; sc[3] = hi.y;
        } else {
          sc[0] = __uint_as_float(cur.x << 16); sc[1] = __uint_as_float(cur.x & 0xffff0000u);
          sc[2] = __uint_as_float(cur.y << 16); sc[3] = __uint_as_float(cur.y & 0xffff0000u);
        }
        // (the group's sums are there when its first accumulator is: the issuer has waited for them)
        const uint32_t sums = ptx::smem_u32(sf_ring) + slot * kSlotBytes + kI4Group * 512 * S::kTokChunks + col0 * 4;
#pragma unroll
        for (int u = 0; u < kI4Group; ++u) {
          if (kb0 + u >= p.num_kb) break;
          if (!__all_sync(0xffffffffu, ptx::mbar_wait_inline_s(acc_full0 + 8 * a, aph, abort_flag))) { ok = false; break; }
          ptx::tc_fence_after();
          uint32_t v[kHalf];
          if (mine) {
            const uint32_t col = tmem_base + a * BT + col0 + lane_sel;
            if (kHalf == 16) ptx::tmem_ld_32x16(col, reinterpret_cast<uint32_t(&)[16]>(v));
            else ptx::tmem_ld_32x8(col, reinterpret_cast<uint32_t(&)[8]>(v));
            ptx::tmem_wait_ld(v);
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_s(acc_empty0 + 8 * a);   // the accumulator is in registers
          if (++a == kI4Conv) { a = 0; aph ^= 1; }
          if (mine) {
#pragma unroll
            for (int i = 0; i < kHalf; i += 4) {
              const float4 m = ptx::lds128f(sums + (u * BT + i) * 4);   // -8 * the block's sum of the token
              ptx::add_fma_f32x2(acc[i / 2], v[i], v[i + 1], m.x, m.y, sc[u]);
              ptx::add_fma_f32x2(acc[i / 2 + 1], v[i + 2], v[i + 3], m.z, m.w, sc[u]);
            }
          }
        }
        if (!ok) break;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_s(sf_empty0 + 8 * slot);
        if (++slot == kI4Slots) slot = 0;
      }
      if (!ok) break;
      if (mine) {
        constexpr int kChunk = kHalf < 16 ? kHalf : 16;
#pragma unroll
        for (int c0 = 0; c0 < kHalf; c0 += kChunk) {
          if (col0 + c0 < ti.valid) {
            float vals[kChunk];
#pragma unroll
            for (int i = 0; i < kChunk; ++i) vals[i] = ((i & 1) ? acc[(c0 + i) / 2].y : acc[(c0 + i) / 2].x) + bias_v;
            store_block_transposed<kChunk, 32>(ctrl->xpose[warp - 16], vals, p.d, p.out_f16, (int64_t)ti.row0 + col0 + c0,
                                               ti.valid - col0 - c0, p.m, p.n, ti.n_tile * kFeat + q * 32, lane);
          }
        }
      }
    }
  }

  pdl_trigger();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if (*abort_flag != 0) __nanosleep(20000);
    ptx::tmem_dealloc(tmem_base, kI4Tmem);
  }
  if (tid == 0 && *abort_flag != 0) report_timeout(p.status);
}

template <int BT, int kTerms, bool kEvensFirst>
__global__ void __launch_bounds__(kI4Threads, 1)
grouped_gemm_i4_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                       const I4Params p) {
  uint8_t *smem = i4_smem(), *walk = smem + p.ctrl_at + kI4CtrlBytes;
  I4Ctrl* ctrl = reinterpret_cast<I4Ctrl*>(smem + p.ctrl_at);
  grouped_gemm_i4_kernel_prologue<BT, false>(tmap_a, tmap_w, p, ctrl, walk);
  grouped_gemm_i4_kernel_body<BT, kTerms, kEvensFirst>(tmap_a, tmap_w, p, p.stages, smem, ctrl, walk);
}

// The tile by the rows that the experts really have, which the host does not know: 32 tokens where the tiles of 16
// would be more by an eighth (two planes) or a third (three); see grouped_gemm_tc_i4.  Both walks are made at once and
// all else ahead of them as in the other kernel.  The choice costs 0 to 1 % (Mixtral, 33 tokens, 16-token tiles alone / so, on
// four inputs: 211.8 / 214.5, 221.0 / 223.5, 222.8 / 224.3, 226.4 / 227.4 us).
template <int kTerms, bool kEvensFirst>
__global__ void __launch_bounds__(kI4Threads, 1)
grouped_gemm_i4_either_kernel(const __grid_constant__ CUtensorMap tmap_a16, const __grid_constant__ CUtensorMap tmap_a32,
                              const __grid_constant__ CUtensorMap tmap_w, const I4Params p) {
  uint8_t *smem = i4_smem(), *walk16 = smem + p.ctrl_at + kI4CtrlBytes, *walk32 = walk16 + tile_walk_bytes(p.num_experts);
  I4Ctrl* ctrl = reinterpret_cast<I4Ctrl*>(smem + p.ctrl_at);
  grouped_gemm_i4_kernel_prologue<16, true>(tmap_a16, tmap_w, p, ctrl, walk16);
  const int64_t tiles16 = tile_walk_at(walk16, p.num_experts).total, tiles32 = tile_walk_at(walk32, p.num_experts).total;
  if (kTerms == 2 ? 8 * tiles16 > 9 * tiles32 : 3 * tiles16 > 4 * tiles32)
    grouped_gemm_i4_kernel_body<32, kTerms, kEvensFirst>(tmap_a32, tmap_w, p, p.stages_wide, smem, ctrl, walk32);
  else
    grouped_gemm_i4_kernel_body<16, kTerms, kEvensFirst>(tmap_a16, tmap_w, p, p.stages, smem, ctrl, walk16);
}

template <int BT, int kTerms>
int i4_token_map(CUtensorMap* map, const b200moe_gemm_args* a) {
  cuuint64_t dims[3] = {(cuuint64_t)a->k, (cuuint64_t)a->m, (cuuint64_t)kTerms};
  cuuint64_t strides[2] = {(cuuint64_t)a->k, (cuuint64_t)a->k * (cuuint64_t)a->m};
  cuuint32_t box[3] = {128, (cuuint32_t)BT, (cuuint32_t)kTerms};
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a->a, dims, strides, box);
}

// Stages of the ring, and in ctrl_at (at least) the end of ring and token scales.
template <int BT, int kTerms>
int i4_ring(int walk_bytes, int& ctrl_at) {
  using S = I4Shape<BT, kTerms>;
  constexpr int kScales = kI4Slots * S::kSlotBytes, kOther = 1024 + kScales + kI4CtrlBytes;
  // A multiple of the converter sets: then a stage is always read by the same set, which has seen the fill before
  // the one that it waits for by parity (the issuers finish blocks out of order).  And deeper than the slots: a
  // stage is released when the block kI4Conv further on is stored.
  constexpr int kLeast = ((int)kMaxSmem - kOther - 2 * tile_walk_bytes(kMaxExperts)) / S::kStageBytes;
  constexpr int kDepth = converter_ring_depth(kI4Sets, kI4Conv);
  static_assert(kLeast / kI4Sets * kI4Sets >= kDepth && kI4MaxStages >= kDepth && kI4MaxStages % kI4Sets == 0,
                "ring depth that the converters' waits need");
  int stages = ((int)kMaxSmem - kOther - walk_bytes) / S::kStageBytes / kI4Sets * kI4Sets;
  if (stages > kI4MaxStages) stages = kI4MaxStages;
  ctrl_at = std::max(ctrl_at, stages * S::kStageBytes + kScales);
  return stages;
}

// kEither: the kernel chooses between BT and 32 tokens.
template <int BT, int kTerms, bool kEvensFirst, bool kEither = false>
int launch_i4(const b200moe_gemm_args* a, I4Params& p, cudaStream_t st) {
  p.idesc = ptx::make_idesc_mx(0u, 0u, kFeat, (uint32_t)BT);   // (a tile puts its number of columns in)
  CUtensorMap ta, ta32, tw;
  if (int rc = i4_token_map<BT, kTerms>(&ta, a)) return rc;
  if (kEither)
    if (int rc = i4_token_map<32, kTerms>(&ta32, a)) return rc;
  {
    cuuint64_t dims[3] = {(cuuint64_t)(a->k / 2), (cuuint64_t)a->n, (cuuint64_t)a->num_experts};
    cuuint64_t strides[2] = {(cuuint64_t)(a->k / 2), (cuuint64_t)(a->k / 2) * a->n};
    cuuint32_t box[3] = {64, (cuuint32_t)kFeat, 1};
    if (int rc = encode_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a->w, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B))
      return rc;
  }
  const int walk_bytes = (kEither ? 2 : 1) * tile_walk_bytes(p.num_experts);
  p.ctrl_at = 0;
  p.stages = i4_ring<BT, kTerms>(walk_bytes, p.ctrl_at);
  p.stages_wide = kEither ? i4_ring<32, kTerms>(walk_bytes, p.ctrl_at) : 0;
  const size_t smem = 1024 + (size_t)p.ctrl_at + kI4CtrlBytes + walk_bytes;
  const int64_t tile_bound = ((a->m + BT - 1) / BT + a->num_experts) * (int64_t)p.n_tiles;
  int grid = sm_count();
  if (a->max_ctas > 0 && a->max_ctas < grid) grid = a->max_ctas;
  if (tile_bound < grid) grid = (int)tile_bound;
  static SmemConfig configured;
  if constexpr (kEither) {
    auto kern = grouped_gemm_i4_either_kernel<kTerms, kEvensFirst>;
    if (int rc = configured.ensure(kern)) return rc;
    B200_LAUNCHED("grouped_gemm_i4_either_kernel",
                  launch_pdl(p.m <= kEarlyLaunchRows, kern, dim3(grid), dim3(kI4Threads), smem, st, ta, ta32, tw, p));
  } else {
    auto kern = grouped_gemm_i4_kernel<BT, kTerms, kEvensFirst>;
    if (int rc = configured.ensure(kern)) return rc;
    B200_LAUNCHED("grouped_gemm_i4_kernel",
                  launch_pdl(p.m <= kEarlyLaunchRows, kern, dim3(grid), dim3(kI4Threads), smem, st, ta, tw, p));
  }
  return B200MOE_OK;
}

}  // namespace

// INT4 weights x two (bfloat16 output) or three (float16 output) e4m3 planes: a codes [planes][M,K],
// a_scale words [planes][K/128][M] and fp32 block sums [K/128][M] behind them (what
// b200moe_quant_mxfp8_ex writes, in either order of the codes).  Returns B200MOE_E_UNSUPPORTED (no launch) for anything else.
int grouped_gemm_tc_i4(const b200moe_gemm_args* a, cudaStream_t st) {
  const bool evens_first = a->a_dtype == B200MOE_FP8_E4M3_X2_EVENS_FIRST || a->a_dtype == B200MOE_FP8_E4M3_X3_EVENS_FIRST;
  const int planes = a->a_dtype == B200MOE_FP8_E4M3_X2 || a->a_dtype == B200MOE_FP8_E4M3_X2_EVENS_FIRST ? 2 :
                     a->a_dtype == B200MOE_FP8_E4M3_X3 || a->a_dtype == B200MOE_FP8_E4M3_X3_EVENS_FIRST ? 3 : 0;
  if (a->w_format != B200MOE_W_INT4_NK || planes == 0 || a->a_scale == nullptr || a->epilogue != B200MOE_EPI_NONE)
    return fail(B200MOE_E_UNSUPPORTED, "int4 GEMM takes int4 weights and two or three e4m3 activation planes");
  if (a->num_experts > kMaxExperts || a->k % 128 != 0 || (a->group_size != 128 && a->group_size != 256) || a->n % 8 != 0)
    return fail(B200MOE_E_UNSUPPORTED, "int4 GEMM: K a multiple of 128, one scale per 128 or 256 of it");
  if (((uintptr_t)a->a & 15) || ((uintptr_t)a->w & 15) || ((uintptr_t)a->d & 15) || ((uintptr_t)a->a_scale & 3))
    return fail(B200MOE_E_BADARG, "int4 GEMM: A, W and D must be 16-byte aligned");
  I4Params p;
  p.w_scale = reinterpret_cast<const uint16_t*>(a->w_scale);
  p.a_scale = reinterpret_cast<const uint32_t*>(a->a_scale);
  p.bias = a->bias; p.d = a->d; p.rows_per_expert = a->rows_per_expert; p.status = a->status;
  p.rows_ready = a->rows_ready == 1 && a->m <= kEarlyLaunchRows;
  p.m = a->m; p.n = a->n; p.k = a->k; p.num_experts = a->num_experts;
  p.n_tiles = (a->n + kFeat - 1) / kFeat;
  p.num_kb = a->k / 128;
  p.groups = a->k / a->group_size;
  p.kb_shift = a->group_size == 256 ? 1 : 0;
  p.out_f16 = a->d_dtype == B200MOE_F16;
  const int64_t in_use = (a->rows_hint > 0 && a->rows_hint < a->m) ? a->rows_hint : a->m;
  const int64_t avg = (in_use + a->num_experts - 1) / a->num_experts;
  // Both the MMA and the promotion cost grow with the tile; experts with more rows than the tile take another, whose
  // weights come from L2.  How many do is not known here, so from 9 to 10 rows per expert (13 for float16, whose three
  // planes make the wide tile dearer) the kernel chooses.  Layer calls, time with 16-token tiles / with the kernel's
  // choice, each against 32-token tiles in the same run (calls that follow one another, outputs the same bit for bit), where
  // the router's logits have an offset per expert of deviation 0, 0.5, 1, 2 and 4:
  //   8 experts of 4096 x 14336, top 2, bfloat16, 9 rows    .94 / .96   .97 / .97    .99 / 1.00  1.02 / 1.00  1.09 / 1.00  (of 171 to 240 us)
  //   64 experts of 2048 x 1408, top 6, bfloat16, 9 rows    .96 / .96   1.01 / 1.01  1.05 / 1.01  1.13 / 1.01  1.17 / 1.01  (of 72 to 114)
  //   the same, float16, 9 rows                             .84 / .85   .90 / .93    .95 / .99   1.03 / .98   1.09 / .96  (of 83 to 138)
  //   the 8 experts, float16, 13 rows                       .88 / .94   1.01 / .99   1.04 / 1.01  1.11 / 1.00  1.04 / .99  (of 251 to 310)
  // By those, 16 tokens win while their tiles are no more than by a tenth to a sixth (two planes) or 0.28 to 0.35 (three) as
  // many again: a wide tile multiplies only columns that have rows.
  auto run = [&](auto order) {
    constexpr bool kEvens = decltype(order)::value;
    if (planes == 2) return avg <= 8 ? launch_i4<16, 2, kEvens>(a, p, st) : avg <= 10 ? launch_i4<16, 2, kEvens, true>(a, p, st) :
                                                                                       launch_i4<32, 2, kEvens>(a, p, st);
    return avg <= 8 ? launch_i4<16, 3, kEvens>(a, p, st) : avg <= 13 ? launch_i4<16, 3, kEvens, true>(a, p, st) :
                                                                      launch_i4<32, 3, kEvens>(a, p, st);
  };
  return evens_first ? run(std::true_type()) : run(std::false_type());
}

}  // namespace b200moe
