// fp8 x block-scaled fp8 grouped GEMM for prefill-sized expert segments, tokens on the
// 128-row M side of tcgen05.mma and the weight's output features on its N side.
//
//   D[r0:r0+rows_e, :] = sum_kb a_scale[row, kb] * w_scale[e, n/128, kb] * (A_kb * W_e,kb^T)
//
// The block-scaled recipe (csrc/xpu/grouped_gemm/xe_2/grouped_gemm_xe2_interface.hpp:361-383
// of vllm-xpu-kernels: e4m3 activations with one fp32 scale per 1x128 group, e4m3 weights with
// one per 128x128 block) needs every 128-wide K block's partial sum multiplied by its own
// scale before it is added up.  With tokens on the tensor-memory lanes an epilogue thread
// owns one token row, and the 128 features of the tile share one weight block: the scale of
// a K block is a single register per thread.  The promotion then is one fused
// multiply-add per accumulator, and the finished row goes to global memory as
// consecutive 16-byte stores.  (The feature-major kernel of gemm_tc.cu, which serves the
// smaller token tiles, has a different scale in every accumulator column and has to stage
// them through shared memory.)
//
// Two kernels: 128 x 128 tiles (below, used when N is a single 128-feature block) and
// 128 x 256 tiles (further down, the one prefill shapes run).
//
// Roles of the 128 x 128 kernel (320 threads, one persistent CTA per SM):
//   warp 0    : TMA producer, ring of 6 stages of [weights 128x128 B | tokens 128x128 B]
//   warp 1    : MMA issuer (one lane), kind::f8f6f4, one accumulator stage (128 columns of
//               tensor memory, four stages) per K block
//   warps 2-9 : promotion + epilogue; warp w reads lane quarter w & 3, columns
//               64 * ((w - 2) / 4) .. + 63: 64 accumulators per thread
// Every mbarrier wait is bounded; on expiry the CTA raises its abort flag, all roles leave
// their loops, tensor memory is freed and *status is set to 1.
#include "common.cuh"
#include "gemm_tc_common.cuh"
#include "sm100_ptx.cuh"


namespace b200moe {
namespace {

constexpr int kTTok = 128;            // tokens per tile (UMMA M)
constexpr int kTStages = 6;
constexpr int kTStageBytes = 32768;   // weights 16 KB, tokens 16 KB
constexpr int kTAcc = 4;              // accumulator stages
constexpr int kTThreads = 320;
constexpr int kTCols = 64;            // accumulator columns per epilogue thread
constexpr int kTGroup = 4;            // K blocks per scale prefetch group

struct TParams {
  const float* a_scale;   // [M, K/128]
  const float* w_scale;   // [E, N/128, K/128]
  const void* bias;
  void* d;
  const int32_t* rows_per_expert;
  int32_t* status;
  int64_t m;
  int n, k, num_experts;
  int w_experts;          // >0: segment s uses weight set s % w_experts
  int n_tiles, num_kb;
  uint32_t idesc;
  int out_f16;
  // gated epilogue of the 128 x 256 kernel (kGated): D is [M, n/2] e4m3 with one fp32 scale per
  // token and 128 features in d_scale [M, n/256]
  float* d_scale;
  float clamp;            // >0: gate = min(gate, clamp), up = clamp(up, -clamp, clamp)
  int rows_ready;         // 128 x 256 kernel, 1: prefetch_first_tiles
  int stages;             // 128 x 256 kernel: pipeline stages
  int d_aligned32;        // 128 x 256 kernel: rows of D begin on 32-byte boundaries
};

struct TCtrl {
  uint64_t full[kTStages];
  uint64_t empty[kTStages];
  uint64_t acc_full[kTAcc];
  uint64_t acc_empty[kTAcc];
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) uint8_t walk[tile_walk_bytes(kMaxExperts)];
};

constexpr size_t kTSmem = 1024 + (size_t)kTStages * kTStageBytes + sizeof(TCtrl);

template <bool kWKn>
__global__ void __launch_bounds__(kTThreads, 1)
grouped_gemm_fp8t_kernel(const __grid_constant__ CUtensorMap tmap_a,
                         const __grid_constant__ CUtensorMap tmap_w, const TParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  TCtrl* ctrl = reinterpret_cast<TCtrl*>(smem + kTStages * kTStageBytes);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    pdl_wait();
    build_tile_walk<kTTok>(p.rows_per_expert, p.num_experts, p.n_tiles, ctrl->walk);
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a);
      ptx::prefetch_tensormap(&tmap_w);
    }
  } else if (warp == 1) {
    ptx::tmem_alloc(&ctrl->tmem_base, 512);
    ptx::tmem_relinquish();
  } else if (warp == 2 && lane == 0) {
    for (int s = 0; s < kTStages; ++s) {
      ptx::mbar_init(&ctrl->full[s], 1);
      ptx::mbar_init(&ctrl->empty[s], 1);
    }
    for (int a = 0; a < kTAcc; ++a) {
      ptx::mbar_init(&ctrl->acc_full[a], 1);
      ptx::mbar_init(&ctrl->acc_empty[a], 8);
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

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 1;
      int cursor = 0;
      bool ok = true;
      const uint32_t full0 = ptx::smem_u32(&ctrl->full[0]), empty0 = ptx::smem_u32(&ctrl->empty[0]);
      const uint32_t st0 = ptx::smem_u32(smem);
      uint32_t st = st0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<kTTok>(walk, t, cursor, ti, p.w_experts);
        const int n0 = ti.n_tile * kFeat;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          const uint32_t full = full0 + 8 * s;
          if (!ptx::paced::mbar_wait_s(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          ptx::mbar_expect_tx_s(full, kTStageBytes);
          if (!kWKn) ptx::tma_load_3d_s(st, &tmap_w, full, kb * 128, n0, ti.e);
          else ptx::tma_load_3d_s(st, &tmap_w, full, n0, kb * 128, ti.e);
          ptx::tma_load_2d_s(st + 16384, &tmap_a, full, kb * 128, ti.row0);
          st += kTStageBytes;
          if (++s == (uint32_t)kTStages) { s = 0; ph ^= 1; st = st0; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (ptx::elect_one()) {
      uint32_t s = 0, ph = 0, a = 0, aph = 1;
      const uint32_t full0 = ptx::smem_u32(&ctrl->full[0]), empty0 = ptx::smem_u32(&ctrl->empty[0]);
      const uint32_t acc_full0 = ptx::smem_u32(&ctrl->acc_full[0]), acc_empty0 = ptx::smem_u32(&ctrl->acc_empty[0]);
      // weights: K-major rows of 128 bytes, or (kWKn) the [K, N] tile read as an MN-major operand
      const uint64_t wdesc0 = ptx::make_smem_desc(ptx::smem_u32(smem), kWKn ? 16384u : 16u, 1024);
      const uint64_t adesc0 = ptx::make_smem_desc(ptx::smem_u32(smem) + 16384, 16, 1024);
      uint64_t wdesc = wdesc0, adesc = adesc0;
      int my_tiles = 0;
      for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) ++my_tiles;
      const int64_t blocks = (int64_t)my_tiles * p.num_kb;   // every tile: same K loop, no tile state needed
      for (int64_t i = 0; i < blocks; ++i) {
        if (!ptx::mbar_wait_s(full0 + 8 * s, ph, abort_flag)) break;
        if (!ptx::mbar_wait_s(acc_empty0 + 8 * a, aph, abort_flag)) break;
        ptx::tc_fence_after();
        ptx::umma_block<true, 2, kWKn ? 4096 / 16 : 2>(tmem_base + a * 128, adesc, wdesc, p.idesc, 0u);
        ptx::umma_commit(acc_full0 + 8 * a);
        ptx::umma_commit(empty0 + 8 * s);
        wdesc += kTStageBytes >> 4;
        adesc += kTStageBytes >> 4;
        if (++s == (uint32_t)kTStages) { s = 0; ph ^= 1; wdesc = wdesc0; adesc = adesc0; }
        if (++a == (uint32_t)kTAcc) { a = 0; aph ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ------------------------ promotion and epilogue --------------------------
    const int q = warp & 3;
    const int r = q * 32 + lane;                       // token row inside the tile
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const int col0 = ((warp - 2) >> 2) * kTCols;       // first feature column of this warp
    const int kbs = p.num_kb;
    const bool vec4_ok = (kbs % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.a_scale) & 15) == 0);
    struct ScaleRegs { float a[kTGroup]; float w[kTGroup]; };
    ScaleRegs cur, pre;
    bool pre_valid = false;
    auto fetch_group = [&](const TileInfo& tt, int g, ScaleRegs& sr) {
      const int kb0 = g * kTGroup;
      const int64_t wsb = ((int64_t)tt.e * p.n_tiles + tt.n_tile) * kbs + kb0;
#pragma unroll
      for (int jb = 0; jb < kTGroup; ++jb) sr.w[jb] = (kb0 + jb < kbs) ? p.w_scale[wsb + jb] : 0.f;
      const bool live = r < tt.valid;
      const float* src = p.a_scale + (int64_t)(tt.row0 + r) * kbs + kb0;
      if (live && vec4_ok) {
        const float4 q4 = *reinterpret_cast<const float4*>(src);
        sr.a[0] = q4.x; sr.a[1] = q4.y; sr.a[2] = q4.z; sr.a[3] = q4.w;
      } else {
#pragma unroll
        for (int jb = 0; jb < kTGroup; ++jb) sr.a[jb] = (live && kb0 + jb < kbs) ? src[jb] : 0.f;
      }
    };
    uint32_t a = 0, aph = 0;
    const uint32_t acc_empty0 = ptx::smem_u32(&ctrl->acc_empty[0]);
    int cursor = 0;
    bool ok = true;
    const int n_groups = (p.num_kb + kTGroup - 1) / kTGroup;
    for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      TileInfo ti;
      locate_tile<kTTok>(walk, t, cursor, ti, p.w_experts);
      float acc[kTCols];
#pragma unroll
      for (int i = 0; i < kTCols; ++i) acc[i] = 0.f;
      uint32_t va[32], vb[32];
      // scales are read one group of K blocks ahead of their use (the next tile's first group
      // during this tile's last)
      if (!pre_valid) fetch_group(ti, 0, cur);
      else cur = pre;
      pre_valid = false;
      for (int g = 0; g < n_groups && ok; ++g) {
        if (g + 1 < n_groups) {
          fetch_group(ti, g + 1, pre);
        } else if (t + (int)gridDim.x < total_tiles) {
          int cursor2 = cursor;
          TileInfo tn;
          locate_tile<kTTok>(walk, t + gridDim.x, cursor2, tn, p.w_experts);
          fetch_group(tn, 0, pre);
          pre_valid = true;
        }
#pragma unroll
        for (int jb = 0; jb < kTGroup; ++jb) {
          if (g * kTGroup + jb >= p.num_kb) break;
          const float sc = cur.a[jb] * cur.w[jb];
          if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctrl->acc_full[a], aph, abort_flag))) {
            *abort_flag = 1; ok = false; break;
          }
          ptx::tc_fence_after();
          // both halves in flight together, one wait: tcgen05.wait::ld covers every load before it
          ptx::tmem_ld_32x32(tmem_base + a * 128 + col0 + lane_sel, va);
          ptx::tmem_ld_32x32(tmem_base + a * 128 + col0 + 32 + lane_sel, vb);
          ptx::tmem_wait_ld(va, vb);
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_s(acc_empty0 + 8 * a);   // the stage is in registers
          if (++a == (uint32_t)kTAcc) { a = 0; aph ^= 1; }
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            acc[i] = fmaf(__uint_as_float(va[i]), sc, acc[i]);
            acc[32 + i] = fmaf(__uint_as_float(vb[i]), sc, acc[32 + i]);
          }
        }
        if (g + 1 < n_groups) cur = pre;
      }
      if (ok && r < ti.valid) {
        const int f0 = ti.n_tile * kFeat + col0;
        uint16_t* drow = reinterpret_cast<uint16_t*>(p.d) + (int64_t)(ti.row0 + r) * p.n + f0;
#pragma unroll
        for (int c = 0; c < kTCols; c += 8) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            float x0 = acc[c + i], x1 = acc[c + i + 1];
            if (p.bias != nullptr) {
              x0 += load_bias(p.bias, p.out_f16, (int64_t)ti.e * p.n + f0 + c + i);
              x1 += load_bias(p.bias, p.out_f16, (int64_t)ti.e * p.n + f0 + c + i + 1);
            }
            if (p.out_f16) {
              const __half2 h = __floats2half2_rn(x0, x1);
              w[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
            } else {
              const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
              w[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
            }
          }
          *reinterpret_cast<uint4*>(drow + c) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }

  // Teardown: everyone meets here, also after an aborted wait.
  pdl_trigger();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if (*abort_flag != 0) __nanosleep(20000);  // let copies still in flight land
    ptx::tmem_dealloc(tmem_base, 512);
  }
  if (tid == 0 && *abort_flag != 0) report_timeout(p.status);
}

// ---------------------------------------------------------------------------------
// Wide variant: 128 tokens x 256 features per tile, so that every tcgen05.mma carries
// twice the work (the issuing thread, not the tensor pipe, bounds the 128-feature tile).
// A thread then owns 128 accumulators, more than the even register split of 384 threads
// allows: the warps are laid out in warpgroups and re-balance registers with setmaxnreg
//   warps 0-3  : producer (warp 0), MMA issuer (warp 1), scale preparers (warps 2 and 3); 56 registers
//   warps 4-11 : promotion + epilogue, 224 registers; warp w reads lane quarter w & 3 and
//                the 128 columns of feature block (w - 4) / 4, in two passes of 64
// Tensor memory holds two accumulator stages of 256 columns.  A CTA's K blocks are one stream over all its
// tiles: every role counts them, and stages, scale slots and parities follow from the count.
//
// What bounds a K block: its MMAs take 512 cycles; their operands and the loads that bring the next ones
// pass 96 KB through shared memory (768 cycles at 128 bytes a cycle); a promotion warp's own path is about
// 600 cycles (clock64, MMAs and loads left out), of which loads and additions are 380 and the rest is
// hand-overs: a wait for a barrier that is complete already costs a warp 100 cycles or more, and two warps a
// scheduler cannot hide it.  So the warp waits once per K block, for the accumulator alone: the issuer has
// seen the block's scales before it issues, and the accumulator of the next block is looked at before the
// last additions.  (The same warp with waits for scales and stage and its two arrivals apart: 850 cycles.
// Loads that ran ahead of the wait, 64-bit accumulators and scalar additions all cost registers or moves:
// slower.)  Under load about 850 cycles a K block remain, at 1.3 to 1.4 GHz under the power cap where the
// same loop on zeros runs at 1.85.
//
// Finished 16-bit rows leave by TMA: a warp puts its 32 rows x 128 features into shared memory and goes on.
// Storing from the registers (32 bytes of 32 rows an instruction) cost every warp about 3600 cycles per tile
// that nothing overlapped, staging through a smaller tile and storing 64-byte pieces 4000; now about 2500,
// most of it the additional passes through shared memory.  The last, partly filled 32 rows of an expert are
// stored from the registers, because the rows behind them belong to another tile.  The buffer takes the room
// of one ring stage; three stages are as fast as four were.  (The gated form has no such buffer and would have room
// for a fourth, but is slower with it: layer calls 616 -> 622 us with 512 rows for each of 128 experts, 4286 -> 4347 with 256
// for each of 256.)
//
// Before / after, 64 experts x 256 rows, N 4096, K 7168: 570 -> 528 us; N 7168, K 2048: 309 -> 287;
// 128 experts of 188 rows, N 1536, K 2048: 140 -> 126; N 2048, K 768: 94 -> 78; 64 experts x 140 rows,
// N 4096, K 7168: 622 -> 519; 32 experts of 32 rows on average: 175 -> 170.
constexpr int kT2Threads = 384;
// setmaxnreg.inc waits - without any limit - until the CTA's register pool holds what it asks
// for, so the re-balanced total must fit what the CTA got at launch (threads x launch registers)
constexpr int kT2LaunchRegs = 168, kT2LowRegs = 56, kT2HighRegs = 224;
static_assert(128 * kT2LowRegs + 256 * kT2HighRegs <= kT2Threads * kT2LaunchRegs, "setmaxnreg budget");
constexpr int kT2Stages = 3;          // ring: 144 KB in flight per SM (one stage less beside a walk of many hundred experts)
constexpr int kT2Slots = 2;           // scale groups handed over ahead
constexpr int kT2Tiles = 16;          // tile coordinates handed over ahead
constexpr int kT2StageBytes = 49152;   // weights 2 x 16 KB, tokens 16 KB
constexpr int kT2Acc = 2;

// A group of K blocks' scales as the promotion warps read them.
struct alignas(16) T2Slot {
  float s[kTGroup][2][128];  // [K block][feature block of the tile][token row]: a_scale * w_scale
};
struct T2Ctrl {
  uint64_t full[kT2Stages];
  uint64_t empty[kT2Stages];
  uint64_t acc_full[kT2Acc];
  uint64_t acc_empty[kT2Acc];
  uint64_t sf_full[kT2Slots];
  uint64_t sf_empty[kT2Slots];
  uint32_t tmem_base;
  int abort_flag;
  float xchg[2][2][128];   // gated epilogue: group maxima exchanged between the two warps of a token row
  uint64_t xbar[4];        // ... and the barrier of each such pair of warps (one per lane quarter)
  alignas(16) T2Slot slot[kT2Slots];
  // The CTA's tile i (first row, valid rows, feature tile, expert) at i % kT2Tiles, written before the group of
  // scales in which it begins, that is when every warp has read the last block of the third group before
  // that one: the tiles in use span at most 13 blocks, and a block begins at most one tile.
  int4 tile[kT2Tiles];
};
// shared memory: the ring, (not gated) the finished tile, T2Ctrl, the tile walk
constexpr int kT2OutBytes = 8 * 8192;   // 32 rows x 128 features of 16 bits a promotion warp
constexpr size_t kT2Fixed = 1024 + ((sizeof(T2Ctrl) + 15) & ~(size_t)15);
static_assert(kT2Fixed + 2 * (size_t)kT2StageBytes + kT2OutBytes + tile_walk_bytes(kMaxExperts) <= kMaxSmem, "shared memory");

//
// kGated (the first grouped GEMM of a SiLU layer with block-scaled fp8 experts): a tile pairs the
// 128 gate features j0.. with the 128 up features n/2 + j0.. of the same tokens; warp w reads
// lane quarter w & 3 and, of both blocks, the 64 columns of half (w - 4) / 4, so a thread holds
// gate and up of the same 64 features of its token.  The epilogue rounds both to the 16-bit
// type an unfused GEMM would have stored, applies silu(gate) * up, finds the maximum of the
// token's 128-feature group together with the partner warp (shared memory, a named barrier of
// the two warps) and stores e4m3 codes and the group's fp32 scale: the arithmetic of
// silu_and_mul_per_block_quant on the unfused output, value for value, without the [M, n]
// round trip through HBM.
// (D's rows begin on 16-byte boundaries; on 32-byte ones unless the caller's buffer does not)
__device__ __forceinline__ void store32(void* to, const uint32_t (&w)[8], int aligned32) {
  if (aligned32) ptx::stg256(to, w);
  else {
    reinterpret_cast<uint4*>(to)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(to)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// Maps of the tokens with boxes of 32, 64, 96 and 128 rows.  A partly filled tile brings the quarters that have
// rows, and zeros (a box that begins behind the matrix) for the others: they would be multiplied all the same, and
// the next expert's rows there cost L2 traffic and power, which under the power cap is time.  Whole boxes / with
// zeros: 256 experts of 256 rows on average (N 4096, K 7168 and N 7168, K 2048; 2.5 tiles of 128) 5013 -> 4951 us a layer
// call, one of 8 ranks at 1024 tokens 281 -> 276, 128 experts of 188 rows 321 -> 318.
struct T2TokenMaps {
  CUtensorMap rows[4];
};

template <bool kWKn, bool kGated>
__global__ void __launch_bounds__(kT2Threads, 1)
grouped_gemm_fp8t256_kernel(const __grid_constant__ T2TokenMaps tmap_a,
                            const __grid_constant__ CUtensorMap tmap_w,
                            const __grid_constant__ CUtensorMap tmap_d, const TParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int stages = p.stages;
  uint8_t* out_base = smem + stages * kT2StageBytes;
  T2Ctrl* ctrl = reinterpret_cast<T2Ctrl*>(out_base + (kGated ? 0 : kT2OutBytes));
  uint8_t* walk_mem = reinterpret_cast<uint8_t*>(ctrl) + ((sizeof(T2Ctrl) + 15) & ~(size_t)15);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // 256-feature tiles; gated: one tile per 128 gate features (p.n_tiles counts 128-feature blocks of n)
  const int n_tiles2 = kGated ? p.n_tiles / 2 : (p.n_tiles + 1) / 2;
  const int up_block0 = p.n_tiles / 2;        // gated: first 128-feature block of the up half

  if (warp == 0) {
    if (!kGated && p.rows_ready) {
      prefetch_first_tiles<kTTok>(p.rows_per_expert, p.num_experts, p.w_experts, n_tiles2, p.num_kb, kPreBytes / 32768,
                                  walk_mem, [&](const TileInfo& ti, int kb) {
        const int n0 = ti.n_tile * 256;
        if (!kWKn) {
          ptx::tma_prefetch_3d(&tmap_w, kb * 128, n0, ti.e);
          ptx::tma_prefetch_3d(&tmap_w, kb * 128, n0 + 128, ti.e);
        } else {
          ptx::tma_prefetch_3d(&tmap_w, n0, kb * 128, ti.e);
          ptx::tma_prefetch_3d(&tmap_w, n0 + 128, kb * 128, ti.e);
        }
      });
    }
    pdl_wait();
    build_tile_walk<kTTok>(p.rows_per_expert, p.num_experts, n_tiles2, walk_mem);
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a.rows[3]);
      ptx::prefetch_tensormap(&tmap_w);
    }
  } else if (warp == 1) {
    ptx::tmem_alloc(&ctrl->tmem_base, 512);
    ptx::tmem_relinquish();
  } else if (warp == 2 && lane == 0) {
    for (int s = 0; s < kT2Stages; ++s) {
      ptx::mbar_init(&ctrl->full[s], 1);
      ptx::mbar_init(&ctrl->empty[s], 1);
    }
    for (int a = 0; a < kT2Acc; ++a) {
      ptx::mbar_init(&ctrl->acc_full[a], 2);   // the MMAs, and the issuer for the scales it has seen
      ptx::mbar_init(&ctrl->acc_empty[a], 8);
    }
    for (int g = 0; g < kT2Slots; ++g) {
      ptx::mbar_init(&ctrl->sf_full[g], 2);
      ptx::mbar_init(&ctrl->sf_empty[g], 8);
    }
    for (int x = 0; x < 4; ++x) ptx::mbar_init(&ctrl->xbar[x], 2);
    ctrl->abort_flag = 0;
    ptx::fence_barrier_init();
  }
  pdl_wait();
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();

  const uint32_t tmem_base = ctrl->tmem_base;
  const TileWalk walk = tile_walk_at(walk_mem, p.num_experts);
  const int total_tiles = walk.total;
  const int my_tiles = (int)blockIdx.x < total_tiles ? (total_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  // The CTA's K blocks are one stream over all its tiles: every role counts them, stages, slots and
  // parities follow from the count.
  const uint32_t blocks = (uint32_t)my_tiles * (uint32_t)p.num_kb;
  const uint32_t sf_full0 = ptx::smem_u32(&ctrl->sf_full[0]), sf_empty0 = ptx::smem_u32(&ctrl->sf_empty[0]);

  if (warp < 4) {
    ptx::setmaxnreg_dec<kT2LowRegs>();
    const uint32_t full0 = ptx::smem_u32(&ctrl->full[0]), empty0 = ptx::smem_u32(&ctrl->empty[0]);
    if (warp == 0 && ptx::elect_one()) {
      // ------------------------------ TMA producer ------------------------------
      uint32_t s = 0, ph = 1;
      int cursor = 0;
      bool ok = true;
      const uint32_t st0 = ptx::smem_u32(smem);
      uint32_t st = st0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        locate_tile<kTTok>(walk, t, cursor, ti, p.w_experts);
        const int n0 = kGated ? ti.n_tile * 128 : ti.n_tile * 256;
        const int n1 = kGated ? (up_block0 + ti.n_tile) * 128 : n0 + 128;
        const int quarters = (ti.valid + 31) >> 5;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          const uint32_t full = full0 + 8 * s;
          if (!ptx::paced::mbar_wait_s(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          ptx::mbar_expect_tx_s(full, kT2StageBytes);
          // two 128-feature blocks (the second one is zero-filled past N)
          if (!kWKn) {
            ptx::tma_load_3d_s(st, &tmap_w, full, kb * 128, n0, ti.e);
            ptx::tma_load_3d_s(st + 16384, &tmap_w, full, kb * 128, n1, ti.e);
          } else {
            ptx::tma_load_3d_s(st, &tmap_w, full, n0, kb * 128, ti.e);
            ptx::tma_load_3d_s(st + 16384, &tmap_w, full, n1, kb * 128, ti.e);
          }
          ptx::tma_load_2d_s(st + 32768, &tmap_a.rows[quarters - 1], full, kb * 128, ti.row0);
          if (quarters < 4) ptx::tma_load_2d_s(st + 32768 + quarters * 4096, &tmap_a.rows[3 - quarters], full, kb * 128, (int)p.m);
          st += kT2StageBytes;
          if (++s == (uint32_t)stages) { s = 0; ph ^= 1; st = st0; }
        }
      }
    } else if (warp == 1 && ptx::elect_one()) {
      // ------------------------------ MMA issuer --------------------------------
      // One thread; descriptors advance by additions.
      uint32_t s = 0, ph = 0, a = 0, aph = 1;
      const uint32_t acc_full0 = ptx::smem_u32(&ctrl->acc_full[0]), acc_empty0 = ptx::smem_u32(&ctrl->acc_empty[0]);
      const uint64_t wdesc0 = ptx::make_smem_desc(ptx::smem_u32(smem), kWKn ? 16384u : 16u, 1024);
      const uint64_t adesc0 = ptx::make_smem_desc(ptx::smem_u32(smem) + 32768, 16, 1024);
      uint64_t wdesc = wdesc0, adesc = adesc0;
      const uint32_t idesc = (p.idesc & ~(0x3fu << 17)) | ((256u >> 3) << 17);
      for (uint32_t i = 0; i < blocks; ++i) {
        // (the block's scales: acc_full stands for them too)
        if (i % kTGroup == 0 && !ptx::paced::mbar_wait_s(sf_full0 + 8 * ((i >> 2) & 1), (i >> 3) & 1, abort_flag)) break;
        if (!ptx::paced::mbar_wait_s(full0 + 8 * s, ph, abort_flag)) break;
        if (!ptx::paced::mbar_wait_s(acc_empty0 + 8 * a, aph, abort_flag)) break;
        // tcgen05.commit completes the MMAs and orders nothing else: scales and tile, written by the preparers,
        // reach the promotion warps through this arrival (acquired above, released here)
        ptx::mbar_arrive_s(acc_full0 + 8 * a);
        ptx::tc_fence_after();
        ptx::umma_block<true, 2, kWKn ? 4096 / 16 : 2>(tmem_base + a * 256, adesc, wdesc, idesc, 0u);
        ptx::umma_commit(acc_full0 + 8 * a);
        ptx::umma_commit(empty0 + 8 * s);
        wdesc += kT2StageBytes >> 4;
        adesc += kT2StageBytes >> 4;
        if (++s == (uint32_t)stages) { s = 0; ph ^= 1; wdesc = wdesc0; adesc = adesc0; }
        if (++a == (uint32_t)kT2Acc) { a = 0; aph ^= 1; }
      }
    } else if (warp >= 2) {
      // ------------------------------ scale preparers ---------------------------
      const int ft = tid - 64, kbs = p.num_kb;            // 0..63: rows ft and ft + 64
      const bool whole = kbs % kTGroup == 0;              // no group spans two tiles
      const bool vec4 = whole && (reinterpret_cast<uintptr_t>(p.a_scale) & 15) == 0;
      int cursor = 0, kb = kbs, t = (int)blockIdx.x - (int)gridDim.x;
      uint32_t seq = 0;
      const float *a0 = nullptr, *w0 = nullptr;
      int64_t w1 = 0;
      bool live[2] = {false, false};
      for (uint32_t b = 0; b < blocks; b += kTGroup) {
        const uint32_t slot = (b / kTGroup) % kT2Slots;
        float av[2][kTGroup], wv[2][kTGroup];
#pragma unroll
        for (int j = 0; j < kTGroup; ++j) {
          if (kb == kbs && b + j < blocks) {
            TileInfo ti;
            t += gridDim.x;
            locate_tile<kTTok>(walk, t, cursor, ti, p.w_experts);
            const int nb0 = kGated ? ti.n_tile : ti.n_tile * 2, nb1 = kGated ? ti.n_tile + up_block0 : nb0 + 1;
            w0 = p.w_scale + ((int64_t)ti.e * p.n_tiles + nb0) * kbs;
            w1 = nb1 < p.n_tiles ? (int64_t)(nb1 - nb0) * kbs : 0;   // past N: any scale, the block's values are zero
            a0 = p.a_scale + (int64_t)(ti.row0 + ft) * kbs;
            live[0] = ft < ti.valid;
            live[1] = ft + 64 < ti.valid;
            if (ft == 0) ctrl->tile[seq % kT2Tiles] = make_int4(ti.row0, ti.valid, ti.n_tile, ti.e);
            ++seq;
            kb = 0;
          }
          const bool in = b + j < blocks;
          wv[0][j] = in ? __ldg(w0 + kb) : 0.f;
          wv[1][j] = in ? __ldg(w0 + w1 + kb) : 0.f;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float* src = a0 + (int64_t)(64 * i) * kbs + kb;
            if (!vec4) {
              av[i][j] = in && live[i] ? *src : 0.f;
            } else if (j == 0) {
              const float4 v = live[i] ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
              av[i][0] = v.x; av[i][1] = v.y; av[i][2] = v.z; av[i][3] = v.w;
            }
          }
          if (in) ++kb;
        }
        if (!__all_sync(0xffffffffu, ptx::paced::mbar_wait_s(sf_empty0 + 8 * slot, ((b / (kTGroup * kT2Slots)) & 1) ^ 1, abort_flag))) break;
        T2Slot* out = &ctrl->slot[slot];
#pragma unroll
        for (int j = 0; j < kTGroup; ++j) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            out->s[j][0][ft + 64 * i] = av[i][j] * wv[0][j];
            out->s[j][1][ft + 64 * i] = av[i][j] * wv[1][j];
          }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_s(sf_full0 + 8 * slot);
      }
    }
  } else {
    // ------------------------ promotion and epilogue --------------------------
    ptx::setmaxnreg_inc<kT2HighRegs>();
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const int half = (warp - 4) >> 2;                  // which 128-feature block of the tile (gated: which 64 features of both)
    // one shared address, the rest are constants from there (registers are full)
    const uint32_t cs = ptx::smem_u32(ctrl);
    constexpr uint32_t kAccFull = offsetof(T2Ctrl, acc_full), kAccEmpty = offsetof(T2Ctrl, acc_empty), kAbort = offsetof(T2Ctrl, abort_flag);
    constexpr uint32_t kSfFull = offsetof(T2Ctrl, sf_full), kSfEmpty = offsetof(T2Ctrl, sf_empty), kSlot = offsetof(T2Ctrl, slot);
    static_assert(kT2Slots * kTGroup == 8 && kT2Acc == 2 && sizeof(T2Slot) == kTGroup * 1024, "parities of the block count");
    const uint32_t my_scales = cs + kSlot + (kGated ? 0 : half * 512) + r * 4;
    // Chunks of 32 columns (chunk c of a stage -> acc[16 c ..]).  plain: the 128 columns of this warp's
    // block; gated: 64 gate columns, then the 64 up columns of the same features.
    const uint32_t col_base = tmem_base + (kGated ? half * 64 : half * 128) + lane_sel;
    constexpr uint32_t kSecond = kGated ? 128 : 64;
    uint32_t b = 0, xpar = 0;
    bool ok = true, seen = false;   // seen: the next block's accumulator was there when last looked at
    for (int tile = 0; tile < my_tiles; ++tile) {
      float2 acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int left = p.num_kb; left > 0; --left, ++b) {
        if (!__all_sync(0xffffffffu, seen)) {
          ok = __all_sync(0xffffffffu, ptx::mbar_wait_lean(cs + kAccFull + 8 * (b & 1), (b >> 1) & 1, cs + kAbort));
          if (!ok) break;
        }
        ptx::tc_fence_after();
        const uint32_t col = col_base + (b & 1) * 256;
        uint32_t va[32], vb[32];
        ptx::tmem_ld_32x32(col, va);
        ptx::tmem_ld_32x32(col + 32, vb);
        const float c0 = ptx::lds32f(my_scales + (b & 7) * 1024);
        const float c1 = kGated ? ptx::lds32f(my_scales + (b & 7) * 1024 + 512) : c0;
        ptx::tmem_wait_ld(va, vb);
        ptx::fma_f32x2(acc, va, c0);
        ptx::fma_f32x2(acc + 16, vb, c0);
        ptx::tmem_ld_32x32(col + kSecond, va);
        ptx::tmem_ld_32x32(col + kSecond + 32, vb);
        ptx::tmem_wait_ld(va, vb);
        ptx::tc_fence_before();   // the whole stage is in registers
        __syncwarp();             // ... of all lanes, which have also read the block's scales
        ptx::mbar_arrive_if(cs + kAccEmpty + 8 * (b & 1), lane == 0, cs + kSfEmpty + 8 * ((b >> 2) & 1), (b & 3) == 3);
        seen = ptx::mbar_test_wait_s(cs + kAccFull + 8 * ((b + 1) & 1), ((b + 1) >> 1) & 1);
        ptx::fma_f32x2(acc + 32, va, c1);
        ptx::fma_f32x2(acc + 48, vb, c1);
      }
      if (!ok) break;
      const int4 here = ctrl->tile[tile % kT2Tiles];
      TileInfo ti;
      ti.row0 = here.x; ti.valid = here.y; ti.n_tile = here.z; ti.e = here.w;
      if (kGated) {
        // values 0..63 = gate, 64..127 = up of features j0 + half * 64 ..
        const int half_n = p.n >> 1;
        const int j0 = ti.n_tile * 128 + half * 64;
        float amax = 0.f;
        // the first half of acc becomes the activated values of features j0 ..
        auto activate = [&](auto round16) {
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            float g = (i & 1) ? acc[i >> 1].y : acc[i >> 1].x, u = (i & 1) ? acc[32 + (i >> 1)].y : acc[32 + (i >> 1)].x;
            if (p.bias != nullptr) {
              g += load_bias(p.bias, p.out_f16, (int64_t)ti.e * p.n + j0 + i);
              u += load_bias(p.bias, p.out_f16, (int64_t)ti.e * p.n + half_n + j0 + i);
            }
            // what the unfused GEMM would have stored, then (optionally) the clamp on those values
            g = round16(g);
            u = round16(u);
            if (p.clamp > 0.f) {
              g = round16(fminf(g, p.clamp));
              u = round16(fminf(fmaxf(u, -p.clamp), p.clamp));
            }
            const float v = __fmul_rn(__fdividef(g, 1.0f + __expf(-g)), u);
            amax = fmaxf(amax, fabsf(v));
            if (i & 1) acc[i >> 1].y = v;
            else acc[i >> 1].x = v;
          }
        };
        if (p.out_f16) activate([](float x) { return __half2float(__float2half_rn(x)); });
        else activate([](float x) { return __bfloat162float(__float2bfloat16_rn(x)); });
        // the other 64 features of the token's 128-feature group are with the partner warp
        // (two buffers by tile parity: the partner has read the previous value of a buffer before
        // it arrived at the barrier of the tile in between)
        ctrl->xchg[xpar][half][r] = amax;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&ctrl->xbar[q]);
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctrl->xbar[q], xpar, abort_flag))) { *abort_flag = 1; ok = false; }
        amax = fmaxf(amax, ctrl->xchg[xpar][half ^ 1][r]);
        xpar ^= 1u;
        if (ok && r < ti.valid) {
          const float scale = fmaxf(__fdiv_rn(amax, 448.0f), 1.0f / (448.0f * 512.0f));
          uint8_t* drow = reinterpret_cast<uint8_t*>(p.d) + (int64_t)(ti.row0 + r) * half_n + j0;
#pragma unroll
          for (int c = 0; c < 64; c += 32) {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              uint32_t x = 0;
#pragma unroll
              for (int b4 = 0; b4 < 4; ++b4)
              {
                const float2 v2 = acc[(c + i + b4) >> 1];
                x |= (uint32_t)f32_to_e4m3(fmaxf(-448.0f, fminf(__fdividef((b4 & 1) ? v2.y : v2.x, scale), 448.0f))) << (8 * b4);
              }
              w[i >> 2] = x;
            }
            store32(drow + c, w, p.d_aligned32);
          }
          if (half == 0) p.d_scale[(int64_t)(ti.row0 + r) * (half_n >> 7) + ti.n_tile] = scale;
        }
        __syncwarp();
      } else {
        const int f0 = ti.n_tile * 256 + half * 128;
        if (p.bias != nullptr && f0 < p.n) {
          const int64_t at = (int64_t)ti.e * p.n + f0;
#pragma unroll
          for (int c = 0; c < 64; c += 8) {
#pragma unroll
            for (int i = c; i < c + 8; ++i) {
              acc[i].x += load_bias(p.bias, p.out_f16, at + 2 * i);
              acc[i].y += load_bias(p.bias, p.out_f16, at + 2 * i + 1);
            }
            asm volatile("" ::: "memory");   // a few loads at a time: registers are full
          }
        }
        uint32_t w[64];
        if (p.out_f16) {
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            const __half2 h = __floats2half2_rn(acc[i].x, acc[i].y);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(acc[i].x, acc[i].y);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
          }
        }
        const bool whole = f0 < p.n && q * 32 + 32 <= ti.valid;   // the warp's 32 rows: by TMA
        const uint32_t out = ptx::smem_u32(out_base) + (warp - 4) * 8192;
        if (whole) {
          if (lane == 0) ptx::bulk_wait_read();   // the tile before has left the buffer
          __syncwarp();
          // two boxes of 32 rows x 64 features, 128-byte swizzle
#pragma unroll
          for (int j = 0; j < 16; ++j)
            ptx::sts128(out + (j >> 3) * 4096 + lane * 128 + (((j & 7) ^ (lane & 7)) << 4),
                        make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]));
        } else if (f0 < p.n && r < ti.valid) {
          uint16_t* drow = reinterpret_cast<uint16_t*>(p.d) + (int64_t)(ti.row0 + r) * p.n + f0;
#pragma unroll
          for (int j = 0; j < 8; ++j) store32(drow + 16 * j, reinterpret_cast<uint32_t(&)[8]>(w[8 * j]), p.d_aligned32);
        }
        if (whole) {
          ptx::fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            ptx::tma_store_2d(&tmap_d, out, f0, ti.row0 + q * 32);
            ptx::tma_store_2d(&tmap_d, out + 4096, f0 + 64, ti.row0 + q * 32);
            ptx::bulk_commit();
          }
        }
        __syncwarp();
      }
    }
    if (!kGated && lane == 0) ptx::bulk_wait();
  }

  pdl_trigger();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if (*abort_flag != 0) __nanosleep(20000);
    ptx::tmem_dealloc(tmem_base, 512);
  }
  if (tid == 0 && *abort_flag != 0) report_timeout(p.status);
}

template <bool kWKn, bool kGated>
int launch_fp8t256(const T2TokenMaps& ta, const CUtensorMap& tw, const CUtensorMap& td, TParams& p, int grid, cudaStream_t st) {
  auto kern = grouped_gemm_fp8t256_kernel<kWKn, kGated>;
  const size_t fixed = kT2Fixed + (kGated ? 0 : kT2OutBytes) + tile_walk_bytes(p.num_experts);
  p.stages = fixed + kT2Stages * (size_t)kT2StageBytes <= kMaxSmem ? kT2Stages : 2;
  const size_t smem = fixed + p.stages * (size_t)kT2StageBytes;
  static SmemConfig configured;
  if (int rc = configured.ensure(kern)) return rc;
  B200_LAUNCHED("grouped_gemm_fp8t256_kernel", launch_pdl(p.m <= kEarlyLaunchRows, kern, dim3(grid), dim3(kT2Threads), smem, st, ta, tw, td, p));
  return B200MOE_OK;
}

template <bool kWKn>
int launch_fp8t(const CUtensorMap& ta, const CUtensorMap& tw, const TParams& p, int grid, cudaStream_t st) {
  auto kern = grouped_gemm_fp8t_kernel<kWKn>;
  static SmemConfig configured;
  if (int rc = configured.ensure(kern)) return rc;
  B200_LAUNCHED("grouped_gemm_fp8t_kernel", launch_pdl(p.m <= kEarlyLaunchRows, kern, dim3(grid), dim3(kTThreads), kTSmem, st, ta, tw, p));
  return B200MOE_OK;
}

}  // namespace

// fp8 activations [M,K] (+ fp32 scales [M,K/128]) times block-scaled fp8 weights ([E,N,K] or
// [E,K,N], scales [E,N/128,K/128]); N and K multiples of 128.  Returns
// B200MOE_E_UNSUPPORTED (no launch) for anything else.
int grouped_gemm_tc_fp8t(const b200moe_gemm_args* a, cudaStream_t st) {
  const bool w8b = a->w_format == B200MOE_W_FP8_BLOCK_NK || a->w_format == B200MOE_W_FP8_BLOCK_KN;
  const bool gated = a->epilogue == B200MOE_EPI_SILU_MUL;
  if (!w8b || a->a_dtype != B200MOE_FP8_E4M3 || a->a_scale == nullptr || a->w_scale == nullptr ||
      (a->epilogue != B200MOE_EPI_NONE && !gated))
    return fail(B200MOE_E_UNSUPPORTED, "token-major fp8 grouped GEMM takes fp8 x block-scaled fp8; fused epilogue: SiLU-and-mul");
  if (gated && (a->d_dtype != B200MOE_FP8_E4M3 || a->d_scale == nullptr || a->n % 256 != 0))
    return fail(B200MOE_E_UNSUPPORTED, "token-major fp8 grouped GEMM: the fused SiLU epilogue writes e4m3 + 1x128 scales "
                                       "(d_dtype FP8_E4M3, d_scale) and needs N / 2 divisible by 128");
  if (!gated && a->d_dtype == B200MOE_FP8_E4M3)
    return fail(B200MOE_E_UNSUPPORTED, "token-major fp8 grouped GEMM: e4m3 output only with the fused SiLU epilogue");
  if (a->num_experts > kMaxExperts || a->n % 128 != 0 || a->k % 128 != 0)
    return fail(B200MOE_E_UNSUPPORTED, "token-major fp8 grouped GEMM: N and K must be multiples of 128");
  if (((uintptr_t)a->a & 15) || ((uintptr_t)a->w & 15) || ((uintptr_t)a->d & 15))
    return fail(B200MOE_E_BADARG, "grouped GEMM: A, W and D must be 16-byte aligned");
  if (a->m == 0 || a->n == 0) return B200MOE_OK;
  const bool kn = a->w_format == B200MOE_W_FP8_BLOCK_KN;

  TParams p;
  p.a_scale = reinterpret_cast<const float*>(a->a_scale);
  p.w_scale = reinterpret_cast<const float*>(a->w_scale);
  p.bias = a->bias; p.d = a->d; p.rows_per_expert = a->rows_per_expert; p.status = a->status;
  p.m = a->m; p.n = a->n; p.k = a->k; p.num_experts = a->num_experts;
  p.rows_ready = a->rows_ready == 1 && a->m <= kEarlyLaunchRows;
  const int w_sets = (a->w_experts > 0 && a->w_experts != a->num_experts) ? a->w_experts : a->num_experts;
  p.w_experts = w_sets != a->num_experts ? w_sets : 0;
  p.n_tiles = a->n / kFeat;
  p.num_kb = a->k / 128;
  p.out_f16 = gated ? (a->mid_dtype == B200MOE_F16) : (a->d_dtype == B200MOE_F16);
  p.d_scale = reinterpret_cast<float*>(a->d_scale);
  p.clamp = a->clamp_limit;
  p.d_aligned32 = ((uintptr_t)a->d & 31) == 0;   // (the row pitch is a multiple of 128 bytes)
  // A operand = tokens (K-major), B operand = weights (K-major, or MN-major for [E,K,N])
  p.idesc = ptx::make_idesc(0u, 0u, 0u, kn ? 1u : 0u, kTTok, kFeat);

  const bool wide = a->n >= 256;   // 256-feature tiles; a single 128-feature block takes the narrow kernel
  T2TokenMaps ta;
  CUtensorMap tw, td;
  for (int i = wide ? 0 : 3; i < 4; ++i) {   // (the narrow kernel brings whole boxes)
    cuuint64_t dims[2] = {(cuuint64_t)a->k, (cuuint64_t)a->m};
    cuuint64_t strides[1] = {(cuuint64_t)a->k};
    cuuint32_t box[2] = {128, (cuuint32_t)(32 * (i + 1))};
    int rc = encode_map(&ta.rows[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, a->a, dims, strides, box);
    if (rc) return rc;
  }
  if (!kn) {
    cuuint64_t dims[3] = {(cuuint64_t)a->k, (cuuint64_t)a->n, (cuuint64_t)w_sets};
    cuuint64_t strides[2] = {(cuuint64_t)a->k, (cuuint64_t)a->k * a->n};
    cuuint32_t box[3] = {128, (cuuint32_t)kFeat, 1};
    int rc = encode_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a->w, dims, strides, box);
    if (rc) return rc;
  } else {
    cuuint64_t dims[3] = {(cuuint64_t)a->n, (cuuint64_t)a->k, (cuuint64_t)w_sets};
    cuuint64_t strides[2] = {(cuuint64_t)a->n, (cuuint64_t)a->k * a->n};
    cuuint32_t box[3] = {128, 128, 1};
    int rc = encode_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a->w, dims, strides, box);
    if (rc) return rc;
  }
  int grid = sm_count();
  if (a->max_ctas > 0 && a->max_ctas < grid) grid = a->max_ctas;
  const int64_t tile_bound = ((a->m + kTTok - 1) / kTTok + a->num_experts) * (int64_t)(wide ? (p.n_tiles + 1) / 2 : p.n_tiles);
  if (tile_bound < grid) grid = (int)tile_bound;
  if (grid < 1) grid = 1;
  if (gated) return kn ? launch_fp8t256<true, true>(ta, tw, tw, p, grid, st) : launch_fp8t256<false, true>(ta, tw, tw, p, grid, st);
  if (wide) {
    cuuint64_t dims[2] = {(cuuint64_t)a->n, (cuuint64_t)a->m};
    cuuint64_t strides[1] = {(cuuint64_t)a->n * 2};
    cuuint32_t box[2] = {64, 32};
    const int rc = encode_map(&td, p.out_f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a->d, dims,
                              strides, box);
    if (rc) return rc;
    return kn ? launch_fp8t256<true, false>(ta, tw, td, p, grid, st) : launch_fp8t256<false, false>(ta, tw, td, p, grid, st);
  }
  return kn ? launch_fp8t<true>(ta.rows[3], tw, p, grid, st) : launch_fp8t<false>(ta.rows[3], tw, p, grid, st);
}

}  // namespace b200moe
