// Tensor-core grouped GEMM for weights that are dequantised on the way in:
// MXFP4 (two e2m1 codes per byte, [E,N,K/2], one e8m0 scale per 32 elements,
// [E,N,K/32]) or INT4 (two's-complement nibbles, [E,N,K/2], one 16-bit scale per
// group of 32..256 elements, [E,N,K/group]) times 16-bit activations.
//
// Same orientation, tile walk and epilogue as grouped_gemm_tc_kernel (weights'
// output features on the 128-row M side of tcgen05.mma, tokens on the N side).
// The expanded weights go from the converters' registers into tensor memory,
// from where the MMA takes them: shared memory sees the packed bytes once, and
// one expansion serves up to 256 tokens (two accumulators of 128 columns).
//   warp 0      : TMA: the tokens (BT rows x 128 bytes per 64 K, 128B swizzle)
//   warp 1      : MMA issuer (kind::f16, A from tensor memory), owns tensor memory
//   warp 2      : TMA: the packed weights, 128 rows x 64 bytes per 128 K (64B swizzle)
//   warps 4-    : converters, two or three sets that take the 128-wide K blocks in turn (a
//                 block is one chain of latencies: barrier, shared loads, expansion,
//                 tensor-memory store, about 650 cycles); a thread owns one weight row
//                 and asks for the scales of its next block before it starts on this one
//   last four   : epilogue
// HBM sees only the 4-bit weights (0.53 bytes per element with scales).
// Large tiles are bound by the matrix instructions and the tokens' way from L2 (32 KB per 512 cycles),
// small ones by the integer pipe of the converters (nine of the seventeen instructions per eight
// weights).  Measured, int4 layer of 8 experts 4096 x 14336, 2 a token, against an expansion through
// shared memory with tiles of at most 128 tokens, the two in turn: 128 tokens 349 us (718), 512 tokens
// 606 us (1190), 2048 tokens 1662 us (3403: 0.87 against 0.42 PFLOP/s).
//
// Numerics follow csrc/xpu/grouped_gemm/xe_2/gemm_xe2.hpp:400-419, 455-471 of
// vllm-xpu-kernels: LUT[code] * 2^(byte-127) (INT4: nibble * scale) rounded to
// the activation type before the multiply, fp32 accumulation, bias added in fp32.
#include <cuda_fp4.h>
#include "common.cuh"
#include "gemm_tc_common.cuh"
#include "sm100_ptx.cuh"

namespace b200moe {
namespace {

constexpr int kDqRawBytes = 8192;  // 128 rows x 64 packed bytes
constexpr int kDqMaxRaw = 12, kDqMaxTok = 8, kDqMaxSlots = 6, kDqMaxAcc = 3;

struct DqParams {
  const uint8_t* w_scale;  // MXFP4: [E, N, K/32] e8m0; INT4: [E, N, K/group] 16-bit values
  int group_shift;         // log2 of the K elements per scale
  int scales;              // scales per weight row
  const void* bias;
  void* d;
  const int32_t* rows_per_expert;
  int32_t* status;
  int64_t m;
  int n, k, num_experts;
  int n_tiles, num_kb;     // num_kb: 128-wide K blocks (TMA fills what is past K with zeros)
  int raw_stages, tok_stages;
  uint32_t idesc;
  int out_f16;
  int swiglu;      // 1: D[m, f/2] = swigluoai(acc[m,f], acc[m,f+1]) for even f
  float alpha, limit, clamp_limit;
};

// A token tile of BT rows is computed in units of at most 128 accumulator columns.  Large tiles hand
// tokens and weights over 64 K at a time (a stage of 256 rows is 32 KB), small ones 128 K.
template <int BT>
struct DqShape {
  static constexpr int kUnit = BT < 128 ? BT : 128;
  static constexpr int kHalves = BT > 64 ? 2 : 1;              // hand-overs per 128-wide K block
  static constexpr int kPieces = 2 / kHalves;                  // 64-wide pieces per hand-over
  static constexpr int kTokBytes = kPieces * BT * 128;
  static constexpr int kSlotCols = kPieces * 32;               // weights of a hand-over in tensor memory
  static constexpr int kSlots = BT > 64 ? 4 : 6;
  // Converter sets of four warps.  Not more than a ring of slots holds blocks: a set's wait for its next
  // slot tells one turn of the ring from the next only if its own last block came at most a turn ago.
  static constexpr int kSets = BT > 64 ? 2 : 3;
  static constexpr int kEpiWarp = 4 + 4 * kSets;
  static constexpr int kThreads = 32 * (kEpiWarp + 4);
  // accumulators in turn: with three the first unit of a tile starts while the last one's is read
  static constexpr int kAcc = BT > 128 ? 3 : 2;
  static constexpr uint32_t kSlotBase = kAcc * kUnit;
  static constexpr uint32_t kCols = kSlotBase + kSlots * kSlotCols;
  static constexpr uint32_t kTmem = kCols <= 256 ? 256u : 512u;
  static_assert(kCols <= 512 && kSlots <= kDqMaxSlots && kAcc <= kDqMaxAcc, "tensor memory");
  static_assert(kSets * kHalves <= kSlots, "slots of a converter set");
};

struct DqCtrl {
  uint64_t raw_full[kDqMaxRaw];
  uint64_t raw_empty[kDqMaxRaw];
  uint64_t tok_full[kDqMaxTok];
  uint64_t tok_empty[kDqMaxTok];
  uint64_t slot_full[kDqMaxSlots];
  uint64_t slot_empty[kDqMaxSlots];
  uint64_t acc_full[kDqMaxAcc];
  uint64_t acc_empty[kDqMaxAcc];
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) uint8_t walk[tile_walk_bytes(kMaxExperts)];
  alignas(16) uint16_t xpose[4][32 * 32];  // per epilogue warp: output transpose tile
};

// Two e2m1 codes (low nibble = even k) -> two fp32 values.
__device__ __forceinline__ float2 e2m1x2_to_float2(uint32_t byte) {
  const __half2_raw h = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)byte, __NV_E2M1);
  return __half22float2(*reinterpret_cast<const __half2*>(&h));
}
template <bool kF16>
__device__ __forceinline__ uint32_t mul16(uint32_t a, uint32_t b) {
  if (kF16) {
    const __half2 v = __hmul2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <bool kF16>
__device__ __forceinline__ uint32_t sub16(uint32_t a, uint32_t b) {
  if (kF16) {
    const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}

// What a scale becomes once per 32 values: INT4 the 16-bit scale in both halves; MXFP4 the e8m0 byte
// as a float (fp16) or as two bf16 factors in both halves.
template <bool kInt4, bool kF16>
struct DqScale {
  uint32_t a, b;
  __device__ __forceinline__ explicit DqScale(uint32_t v) {
    if (kInt4) { a = v | (v << 16); b = 0; return; }
    if (kF16) { a = __float_as_uint(e8m0_to_f32(v)); b = 0; return; }
    // 2^(v - 1) would leave the bf16 range above 128: the rest goes into a second factor
    a = ((v < 128u ? v : 128u) + 126u) << 7;
    b = v <= 128u ? 0x3f80u : (v == 255u ? 0x7fc0u : (v - 1u) << 7);
    a |= a << 16;
    b |= b << 16;
  }
};

// Eight packed values (low nibble first) -> four words of two 16-bit values.
template <bool kInt4, bool kF16>
__device__ __forceinline__ void expand8(uint32_t w, const DqScale<kInt4, kF16>& sc, uint32_t* o) {
  const uint32_t h = w >> 4;   // odd k in the low nibbles
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    // byte j of w in the low half, byte j of h in the high half
    const uint32_t q = __byte_perm(w, h, (uint32_t)(j | (j << 4) | ((4 + j) << 8) | ((4 + j) << 12)));
    if (kInt4) {
      // nibble n (two's complement) -> 128 + (n ^ 8) (bf16 0x4300 | .; fp16: 1024 +, 0x6400 | .)
      // exactly, minus 136 (1032) = n as a signed value, times the scale: one rounding, as the
      // reference's product in the activation type.
      constexpr uint32_t magic = kF16 ? 0x64086408u : 0x43084308u;   // 1032.0 / 136.0
      o[j] = mul16<kF16>(sub16<kF16>((q & 0x000f000fu) ^ magic, magic), sc.a);
    } else if (kF16) {
      const float2 f = e2m1x2_to_float2((w >> (8 * j)) & 0xffu);
      const __half2 v = __floats2half2_rn(f.x * __uint_as_float(sc.a), f.y * __uint_as_float(sc.a));
      o[j] = *reinterpret_cast<const uint32_t*>(&v);
    } else {
      // The code's exponent and mantissa bits where bf16 keeps them ((c & 7) << 6, sign to bit 15):
      // read as bf16 that is the code's value times 2^-126, subnormal codes included, so the exact
      // multiply by 2^(scale - 1) yields code * 2^(scale - 127).
      const uint32_t bits = ((q << 6) & 0x01C001C0u) | ((q << 12) & 0x80008000u);
      o[j] = mul16<kF16>(mul16<kF16>(bits, sc.a), sc.b);
    }
  }
}

// BT tokens per tile.
template <int BT, bool kInt4, bool kF16>
__global__ void __launch_bounds__(DqShape<BT>::kThreads, 1)
grouped_gemm_dq_kernel(const __grid_constant__ CUtensorMap tmap_a,
                       const __grid_constant__ CUtensorMap tmap_w, const DqParams p) {
  using S = DqShape<BT>;
  constexpr int kUnit = S::kUnit, kHalves = S::kHalves, kPieces = S::kPieces, kSlots = S::kSlots, kAcc = S::kAcc;
  constexpr int kSets = S::kSets, kEpiWarp = S::kEpiWarp;
  constexpr int kChunk = BT >= 32 ? 32 : 16;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int raw_stages = p.raw_stages, tok_stages = p.tok_stages;
  uint8_t* raw_ring = smem + tok_stages * S::kTokBytes;
  DqCtrl* ctrl = reinterpret_cast<DqCtrl*>(raw_ring + raw_stages * kDqRawBytes);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    pdl_wait();
    build_tile_walk<BT>(p.rows_per_expert, p.num_experts, p.n_tiles, ctrl->walk);
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a);
      ptx::prefetch_tensormap(&tmap_w);
    }
  } else if (warp == 1) {
    ptx::tmem_alloc(&ctrl->tmem_base, S::kTmem);
    ptx::tmem_relinquish();
  } else if (warp == 2 && lane == 0) {
    for (int s = 0; s < kDqMaxRaw; ++s) {
      ptx::mbar_init(&ctrl->raw_full[s], 1);
      ptx::mbar_init(&ctrl->raw_empty[s], 4);
    }
    for (int s = 0; s < kDqMaxTok; ++s) {
      ptx::mbar_init(&ctrl->tok_full[s], 1);
      ptx::mbar_init(&ctrl->tok_empty[s], 1);
    }
    for (int c = 0; c < kDqMaxSlots; ++c) {
      ptx::mbar_init(&ctrl->slot_full[c], 4);
      ptx::mbar_init(&ctrl->slot_empty[c], 1);
    }
    for (int a = 0; a < kDqMaxAcc; ++a) {
      ptx::mbar_init(&ctrl->acc_full[a], 1);
      ptx::mbar_init(&ctrl->acc_empty[a], 4);
    }
    ctrl->abort_flag = 0;
    ptx::fence_barrier_init();
  }
  pdl_wait();
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();

  const uint32_t tmem_base = ctrl->tmem_base;
  const TileWalk walk = tile_walk_at(ctrl->walk, p.num_experts);
  const int total_tiles = walk.total;
  const uint32_t raw_full0 = ptx::smem_u32(&ctrl->raw_full[0]), raw_empty0 = ptx::smem_u32(&ctrl->raw_empty[0]);
  const uint32_t tok_full0 = ptx::smem_u32(&ctrl->tok_full[0]), tok_empty0 = ptx::smem_u32(&ctrl->tok_empty[0]);
  const uint32_t slot_full0 = ptx::smem_u32(&ctrl->slot_full[0]), slot_empty0 = ptx::smem_u32(&ctrl->slot_empty[0]);
  const uint32_t acc_full0 = ptx::smem_u32(&ctrl->acc_full[0]), acc_empty0 = ptx::smem_u32(&ctrl->acc_empty[0]);

  if (warp == 0) {
    // ------------------------------ TMA: tokens --------------------------------
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 1;
      int cursor = 0;
      bool ok = true;
      const uint32_t st0 = ptx::smem_u32(smem);
      uint32_t st = st0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<BT>(walk, t, cursor, ti);
        const bool second = BT > kUnit && ti.valid > kUnit;   // rows past the first unit
        const uint32_t bytes = (BT > kUnit && !second) ? kPieces * kUnit * 128 : S::kTokBytes;
        for (int hb = 0; hb < p.num_kb * kHalves; ++hb) {
          const uint32_t full = tok_full0 + 8 * s;
          if (!ptx::paced::mbar_wait_s(tok_empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          ptx::mbar_expect_tx_s(full, bytes);
#pragma unroll
          for (int j = 0; j < kPieces; ++j)
            ptx::tma_load_2d_s(st + j * BT * 128, &tmap_a, full, (hb * kPieces + j) * 64, ti.row0);
          if (second) ptx::tma_load_2d_s(st + kUnit * 128, &tmap_a, full, hb * 64, ti.row0 + kUnit);
          st += S::kTokBytes;
          if (++s == (uint32_t)tok_stages) { s = 0; ph ^= 1; st = st0; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------ TMA: packed weights ------------------------
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 1;
      int cursor = 0;
      bool ok = true;
      const uint32_t st0 = ptx::smem_u32(raw_ring);
      uint32_t st = st0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<BT>(walk, t, cursor, ti);
        const int n0 = ti.n_tile * kFeat;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          const uint32_t full = raw_full0 + 8 * s;
          if (!ptx::paced::mbar_wait_s(raw_empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          ptx::mbar_expect_tx_s(full, kDqRawBytes);
          ptx::tma_load_3d_s(st, &tmap_w, full, kb * 64, n0, ti.e);
          st += kDqRawBytes;
          if (++s == (uint32_t)raw_stages) { s = 0; ph ^= 1; st = st0; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 0, c = 0, cph = 0, a = 0, aph = 1;
      int cursor = 0;
      bool ok = true;
      const uint64_t desc0 = ptx::make_smem_desc(ptx::smem_u32(smem), 16, 1024);
      uint64_t desc = desc0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<BT>(walk, t, cursor, ti);
        const bool second = BT > kUnit && ti.valid > kUnit;
        // a partly filled unit multiplies only its valid columns (UMMA N in steps of 16)
        auto idesc_of = [&](int valid) { return (p.idesc & ~(0x3fu << 17)) | ((uint32_t)((valid + 15) & ~15) >> 3 << 17); };
        const uint32_t idesc1 = idesc_of(second ? kUnit : ti.valid), idesc2 = idesc_of(ti.valid - kUnit);
        const uint32_t acc1 = tmem_base + a * kUnit, bar1 = 8 * a;
        if (!ptx::mbar_wait_s(acc_empty0 + bar1, aph, abort_flag)) break;
        if (++a == kAcc) { a = 0; aph ^= 1; }
        const uint32_t acc2 = tmem_base + a * kUnit, bar2 = 8 * a;
        ptx::tc_fence_after();
        for (int hb = 0; hb < p.num_kb * kHalves; ++hb) {
          if (!ptx::mbar_wait_s(tok_full0 + 8 * s, ph, abort_flag) ||
              !ptx::mbar_wait_s(slot_full0 + 8 * c, cph, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after();
          const uint32_t w = tmem_base + S::kSlotBase + c * S::kSlotCols;
#pragma unroll
          for (int j = 0; j < kPieces; ++j)
            ptx::umma_f16_block_ts(acc1, w + j * 32, desc + j * (BT * 128 >> 4), idesc1, hb + j > 0 ? 1u : 0u);
          if (second) {
            if (hb == 0) {
              if (!ptx::mbar_wait_s(acc_empty0 + bar2, aph, abort_flag)) { ok = false; break; }
              ptx::tc_fence_after();
            }
            ptx::umma_f16_block_ts(acc2, w, desc + (kUnit * 128 >> 4), idesc2, hb > 0 ? 1u : 0u);
          }
          ptx::umma_commit(slot_empty0 + 8 * c);
          ptx::umma_commit(tok_empty0 + 8 * s);
          desc += S::kTokBytes >> 4;
          if (++s == (uint32_t)tok_stages) { s = 0; ph ^= 1; desc = desc0; }
          if (++c == kSlots) { c = 0; cph ^= 1; }
        }
        if (!ok) break;
        ptx::umma_commit(acc_full0 + bar1);
        if (second) {
          ptx::umma_commit(acc_full0 + bar2);
          if (++a == kAcc) { a = 0; aph ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4 && warp < kEpiWarp) {
    // ------------------------------ converters --------------------------------
    const int row = (warp & 3) * 32 + lane, set = (warp - 4) >> 2;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t src0 = ptx::smem_u32(raw_ring) + row * 64;
    const uint32_t swz = (uint32_t)((row >> 1) & 3) << 4;      // 64-byte swizzle: chunk index xor row bits 1..2
    const uint32_t slot_base = tmem_base + S::kSlotBase + lane_sel;
    // this set's K blocks: kb of tile t, advanced kSets at a time across tiles
    int t = blockIdx.x, kb = set, cursor = 0;
    bool feat_ok = false;
    const uint8_t* srow = p.w_scale;
    auto enter_tile = [&]() {
      TileInfo ti;
      locate_tile<BT>(walk, t, cursor, ti);
      const int feat = ti.n_tile * kFeat + row;
      feat_ok = feat < p.n;
      srow = p.w_scale + ((int64_t)ti.e * p.n + (feat_ok ? feat : 0)) * p.scales * (kInt4 ? 2 : 1);
    };
    auto settle = [&]() {   // kb past the tile: on to the next one (a tile may have fewer blocks than sets)
      bool moved = false;
      while (kb >= p.num_kb && t < total_tiles) { kb -= p.num_kb; t += gridDim.x; moved = true; }
      if (moved && t < total_tiles) enter_tile();
    };
    // the four scales (one per 32 values) of the block, INT4: 16-bit values, MXFP4: bytes
    struct Scales { uint32_t v[4]; };
    auto load_scales = [&]() {
      Scales r;
      if (kInt4) {
        const uint16_t* s16 = reinterpret_cast<const uint16_t*>(srow);
        if (p.group_shift >= 7) {
          const uint32_t v = feat_ok ? (uint32_t)__ldg(s16 + ((kb * 128) >> p.group_shift)) : 0u;
          r.v[0] = r.v[1] = r.v[2] = r.v[3] = v;
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int g = (kb * 128 + 32 * u) >> p.group_shift;
            r.v[u] = (feat_ok && g < p.scales) ? (uint32_t)__ldg(s16 + g) : 0u;
          }
        }
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          r.v[u] = (feat_ok && kb * 4 + u < p.scales) ? (uint32_t)__ldg(srow + kb * 4 + u) : 127u;
      }
      return r;
    };
    if (t < total_tiles) { enter_tile(); settle(); }
    Scales nxt;
    if (t < total_tiles) nxt = load_scales();
    uint32_t s = set, ph = 0;
    uint32_t c = (set * kHalves) % kSlots, cph = 1 ^ (((set * kHalves) / kSlots) & 1);
    while (t < total_tiles) {
      const Scales cur = nxt;
      kb += kSets;
      settle();
      if (t < total_tiles) nxt = load_scales();
      if (!__all_sync(0xffffffffu, ptx::paced::mbar_wait_s(raw_full0 + 8 * s, ph, abort_flag))) break;
      const uint32_t src = src0 + s * kDqRawBytes;
      uint4 raw[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) raw[q] = ptx::lds128(src + ((uint32_t)(q * 16) ^ swz));
      bool ok = true;
#pragma unroll
      for (int h = 0; h < 2; ++h) {                 // 64 values: 32 words of two
        uint32_t o[32];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint4 v = raw[2 * h + q];
          const DqScale<kInt4, kF16> sc(cur.v[2 * h + q]);
          expand8<kInt4, kF16>(v.x, sc, o + q * 16);
          expand8<kInt4, kF16>(v.y, sc, o + q * 16 + 4);
          expand8<kInt4, kF16>(v.z, sc, o + q * 16 + 8);
          expand8<kInt4, kF16>(v.w, sc, o + q * 16 + 12);
        }
        if (h == 0) {
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_s(raw_empty0 + 8 * s);   // the block is in registers
        }
        if (h == 0 || kHalves == 2) {
          if (!__all_sync(0xffffffffu, ptx::paced::mbar_wait_s(slot_empty0 + 8 * c, cph, abort_flag))) { ok = false; break; }
          ptx::tc_fence_after();
        }
        ptx::tmem_st_32x32(slot_base + c * S::kSlotCols + (kHalves == 1 ? h * 32 : 0), o);
        if (h == 1 || kHalves == 2) {
          ptx::tmem_wait_st();
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_s(slot_full0 + 8 * c);
          if (kHalves == 2 && h == 0) c = c + 1 == kSlots ? 0 : c + 1, cph ^= c == 0;
        }
      }
      if (!ok) break;
      s += kSets;
      if (s >= (uint32_t)raw_stages) { s -= raw_stages; ph ^= 1; }
      c += kHalves == 2 ? 2 * kSets - 1 : kSets;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (c >= kSlots) { c -= kSlots; cph ^= 1; }
    }
  } else if (warp >= kEpiWarp) {
    // ------------------------------ epilogue ----------------------------------
    const int q = warp & 3;
    const int et = q * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const int n_out = p.swiglu ? p.n / 2 : p.n;
    uint32_t a = 0, aph = 0;
    int cursor = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      TileInfo ti;
      locate_tile<BT>(walk, t, cursor, ti);
      const int feat = ti.n_tile * kFeat + et;
      const bool feat_ok = feat < p.n;
      float bias_v = 0.f;
      if (p.bias != nullptr && feat_ok) bias_v = load_bias(p.bias, p.out_f16, (int64_t)ti.e * p.n + feat);
      for (int u0 = 0; u0 < ti.valid; u0 += kUnit) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait_inline_s(acc_full0 + 8 * a, aph, abort_flag))) { ok = false; break; }
        ptx::tc_fence_after();
        const int valid = ti.valid - u0;
#pragma unroll 1
        for (int c0 = 0; c0 < kUnit; c0 += kChunk) {
          if (c0 < valid) {
            uint32_t v[kChunk];
            if (kChunk == 32) ptx::tmem_ld_32x32(tmem_base + a * kUnit + c0 + lane_sel, reinterpret_cast<uint32_t(&)[32]>(v));
            else ptx::tmem_ld_32x16(tmem_base + a * kUnit + c0 + lane_sel, reinterpret_cast<uint32_t(&)[16]>(v));
            ptx::tmem_wait_ld(v);
            float vals[kChunk];
#pragma unroll
            for (int i = 0; i < kChunk; ++i) vals[i] = __uint_as_float(v[i]) + bias_v;
            if (p.swiglu) {
              // One branch around the whole block: the unrolled body stays straight-line code, so
              // the shuffle / exp / divide chains of the columns overlap.
              const float c_lim = p.clamp_limit > 0.f ? p.clamp_limit : INFINITY;
#pragma unroll
              for (int i = 0; i < kChunk; ++i) {
                // gate sits on even features, up on the next odd one: neighbours in the warp
                const float x = vals[i];
                const float other = __shfl_xor_sync(0xffffffffu, x, 1);
                float gate = (lane & 1) ? other : x;
                float up = (lane & 1) ? x : other;
                gate = fminf(gate, c_lim);
                up = fminf(fmaxf(up, -c_lim), c_lim);
                gate = fminf(gate, p.limit);
                up = fminf(fmaxf(up, -p.limit), p.limit);
                vals[i] = (up + 1.0f) * gate * __fdividef(1.0f, 1.0f + __expf(-gate * p.alpha));
              }
            }
            if (p.swiglu)
              store_block_transposed<kChunk, 16>(ctrl->xpose[warp - kEpiWarp], vals, p.d, p.out_f16,
                                                 (int64_t)ti.row0 + u0 + c0, valid - c0, p.m, n_out,
                                                 (ti.n_tile * kFeat + q * 32) >> 1, lane);
            else
              store_block_transposed<kChunk, 32>(ctrl->xpose[warp - kEpiWarp], vals, p.d, p.out_f16,
                                                 (int64_t)ti.row0 + u0 + c0, valid - c0, p.m, n_out,
                                                 ti.n_tile * kFeat + q * 32, lane);
          }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_s(acc_empty0 + 8 * a);
        if (++a == kAcc) { a = 0; aph ^= 1; }
      }
    }
  }

  pdl_trigger();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if (*abort_flag != 0) __nanosleep(20000);
    ptx::tmem_dealloc(tmem_base, S::kTmem);
  }
  if (tid == 0 && *abort_flag != 0) report_timeout(p.status);
}

template <int BT, bool kInt4, bool kF16>
int launch_dq(const b200moe_gemm_args* a, DqParams& p, cudaStream_t st) {
  using S = DqShape<BT>;
  auto kern = grouped_gemm_dq_kernel<BT, kInt4, kF16>;
  const uint32_t fmt = kF16 ? 0u : 1u;
  p.idesc = ptx::make_idesc(fmt, fmt, 0u, 0u, kFeat, (uint32_t)S::kUnit);
  CUtensorMap ta, tw;
  {
    cuuint64_t dims[2] = {(cuuint64_t)a->k, (cuuint64_t)a->m};
    cuuint64_t strides[1] = {(cuuint64_t)a->k * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)S::kUnit};
    if (int rc = encode_map(&ta, kF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                            a->a, dims, strides, box)) return rc;
  }
  {
    cuuint64_t dims[3] = {(cuuint64_t)(a->k / 2), (cuuint64_t)a->n, (cuuint64_t)a->num_experts};
    cuuint64_t strides[2] = {(cuuint64_t)(a->k / 2), (cuuint64_t)(a->k / 2) * a->n};
    cuuint32_t box[3] = {64, (cuuint32_t)kFeat, 1};
    if (int rc = encode_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a->w, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B))
      return rc;
  }
  // Shared memory: the weights of small tiles stream at HBM's rate and get most of it, the tokens of
  // large ones (32 KB per 64 K) what four raw stages leave.
  constexpr int kRoom = (int)kMaxSmem - 1024 - (int)((sizeof(DqCtrl) + 15) & ~(size_t)15);
  constexpr int kTokFit = BT > 64 ? (kRoom - 4 * kDqRawBytes) / S::kTokBytes : 6;
  constexpr int kTok = kTokFit < kDqMaxTok ? kTokFit : kDqMaxTok;
  constexpr int kRawFit = (kRoom - kTok * S::kTokBytes) / kDqRawBytes;
  constexpr int kRaw = kRawFit < kDqMaxRaw ? kRawFit : kDqMaxRaw;
  static_assert(kRaw >= converter_ring_depth(S::kSets, S::kSlots / S::kHalves), "ring depth that the converters' waits need");
  p.tok_stages = kTok;
  p.raw_stages = kRaw;
  constexpr size_t smem = kMaxSmem - kRoom + (size_t)kTok * S::kTokBytes + (size_t)kRaw * kDqRawBytes;
  static SmemConfig configured;
  if (int rc = configured.ensure(kern)) return rc;
  const int64_t tile_bound = ((a->m + BT - 1) / BT + a->num_experts) * (int64_t)p.n_tiles;
  int grid = sm_count();
  if (a->max_ctas > 0 && a->max_ctas < grid) grid = a->max_ctas;
  if (tile_bound < grid) grid = (int)tile_bound;
  B200_LAUNCHED("grouped_gemm_dq_kernel",
                launch_pdl(p.m <= kEarlyLaunchRows, kern, dim3(grid), dim3(S::kThreads), smem, st, ta, tw, p));
  return B200MOE_OK;
}

}  // namespace

// MXFP4 or INT4 weights x 16-bit activations on the tensor cores.  Returns
// B200MOE_E_UNSUPPORTED (no launch) for anything else.
int grouped_gemm_tc_dq(const b200moe_gemm_args* a, cudaStream_t st) {
  const bool int4 = a->w_format == B200MOE_W_INT4_NK;
  if (!(a->w_format == B200MOE_W_MXFP4_NK || int4) || a->a_dtype == B200MOE_FP8_E4M3)
    return fail(B200MOE_E_UNSUPPORTED, "dequantising tensor-core GEMM takes MXFP4 or INT4 weights only");
  if (int4 && ((uintptr_t)a->w_scale & 1))
    return fail(B200MOE_E_BADARG, "grouped GEMM: INT4 scales must be 2-byte aligned");
  if (a->epilogue == B200MOE_EPI_SILU_MUL)
    return fail(B200MOE_E_UNSUPPORTED, "dequantising tensor-core GEMM: SiLU epilogue not available");
  if (a->num_experts > kMaxExperts || a->k % 64 != 0 || (a->k / 2) % 16 != 0)
    return fail(B200MOE_E_UNSUPPORTED, "dequantising tensor-core GEMM: K must be a multiple of 64");
  if (((uintptr_t)a->a & 15) || ((uintptr_t)a->w & 15) || ((uintptr_t)a->d & 15))
    return fail(B200MOE_E_BADARG, "grouped GEMM: A, W and D must be 16-byte aligned");
  if (a->epilogue == B200MOE_EPI_SWIGLUOAI && (a->n / 2) % 8 != 0)
    return fail(B200MOE_E_UNSUPPORTED, "dequantising tensor-core GEMM: gated output width must be a multiple of 8");
  if (a->m == 0 || a->n == 0) return B200MOE_OK;

  DqParams p;
  p.w_scale = reinterpret_cast<const uint8_t*>(a->w_scale);
  const int group = int4 ? a->group_size : 32;
  p.group_shift = group == 32 ? 5 : group == 64 ? 6 : group == 128 ? 7 : 8;
  p.scales = a->k / group;
  p.bias = a->bias; p.d = a->d; p.rows_per_expert = a->rows_per_expert; p.status = a->status;
  p.m = a->m; p.n = a->n; p.k = a->k; p.num_experts = a->num_experts;
  p.n_tiles = (a->n + kFeat - 1) / kFeat;
  p.num_kb = (a->k + 127) / 128;
  p.out_f16 = a->d_dtype == B200MOE_F16;
  p.swiglu = a->epilogue == B200MOE_EPI_SWIGLUOAI;
  p.alpha = a->act_alpha; p.limit = a->act_limit; p.clamp_limit = a->clamp_limit;

  const int64_t rows_in_use = (a->rows_hint > 0 && a->rows_hint < a->m) ? a->rows_hint : a->m;
  const int64_t avg = (rows_in_use + a->num_experts - 1) / a->num_experts;
  const bool f16 = a->a_dtype == B200MOE_F16;
  // Tile of tokens: what the average expert fills; the large one computes 128 columns where it holds
  // no more rows, so it serves everything above.  Measured at 16 / 64 / 256 tokens, int4, 8 experts, N
  // 28672, K 4096: 8 rows per expert 182 / 184 / 248 us, 16 rows 242 / 185 / 248, 40 rows 508 / 188 / 254,
  // 48 rows 604 / 191 / 252, 64 rows - / 315 / 254, 256 rows - / 772 / 510.
#define B200_DQ_CASES(I4, F16)                                  \
  if (avg <= 8) return launch_dq<16, I4, F16>(a, p, st);        \
  if (avg <= 40) return launch_dq<64, I4, F16>(a, p, st);       \
  return launch_dq<256, I4, F16>(a, p, st);
  if (int4 && f16) { B200_DQ_CASES(true, true) }
  if (int4) { B200_DQ_CASES(true, false) }
  if (f16) { B200_DQ_CASES(false, true) }
  B200_DQ_CASES(false, false)
#undef B200_DQ_CASES
}

}  // namespace b200moe
