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
  int stages;             // 128 x 256 kernel: pipeline stages
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
          if (!ptx::mbar_wait_s(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
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
// Tensor memory holds two accumulator stages of 256 columns.
//
// The promotion sets the rate: a K block's MMAs take 512 cycles, the additions of two warps on a
// scheduler 256 to 300, but a warp that waits for the stage, loads, adds, and reads its scales from
// global memory one after the other took 917 to 1000.  So everything that is not a load or an addition
// is kept off its path: scales (already multiplied, four K blocks per hand-over) and tile coordinates come
// from the preparers through shared memory; a chunk's tensor-memory load is in flight while the chunk
// before it is added up, also from one K block to the next; the next K block's barriers are looked at once,
// before the additions that hide the look, and nothing else in the loop branches.  128 experts of 188 rows,
// N 2048, K 768: 140 -> 110 us; 256 experts of 256 rows on average, N 4096, K 7168: 3.06 -> 2.85 ms.
constexpr int kT2Threads = 384;
// setmaxnreg.inc waits - without any limit - until the CTA's register pool holds what it asks
// for, so the re-balanced total must fit what the CTA got at launch (threads x launch registers)
constexpr int kT2LaunchRegs = 168, kT2LowRegs = 56, kT2HighRegs = 224;
static_assert(128 * kT2LowRegs + 256 * kT2HighRegs <= kT2Threads * kT2LaunchRegs, "setmaxnreg budget");
constexpr int kT2Stages = 4;          // ring: 192 KB in flight per SM (one less beside a walk of many hundred experts)
constexpr int kT2Slots = 2;           // scale groups handed over ahead
// Finished rows leave through per-warp staging tiles of 32 rows x 32 values (64 bytes + 16, conflict-free
// for 16-byte accesses), so that a store instruction writes whole 64-byte pieces of eight rows; straight
// from the registers it would be 16 bytes of 32 rows (4 us per tile that nothing overlaps).  The tile is
// that small so that the ring keeps four stages: with three and whole 256-byte rows the MMA thread
// waited 400 of 1200 cycles per K block for data.
constexpr int kT2RowPitch = 80;
constexpr int kT2StageBytes = 49152;   // weights 2 x 16 KB, tokens 16 KB
constexpr int kT2Acc = 2;

// A group of K blocks' scales as the promotion warps read them.
struct alignas(16) T2Slot {
  float s[2][kTGroup][128];  // [feature block of the tile][K block][token row]: a_scale * w_scale
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
  // The CTA's tile i (first row, valid rows, feature tile, expert) at i % 4, written with its first
  // group of scales: by then every warp has read a group of tile i - 2 or later, so it has finished i - 4.
  int4 tile[4];
};
constexpr size_t kT2XposeBytes = 8 * 32 * kT2RowPitch;
// shared memory: the ring, the staging tiles, T2Ctrl, the tile walk
constexpr size_t kT2Fixed = 1024 + kT2XposeBytes + ((sizeof(T2Ctrl) + 15) & ~(size_t)15);
static_assert(kT2Fixed + 3 * (size_t)kT2StageBytes + tile_walk_bytes(kMaxExperts) <= kMaxSmem, "shared memory");

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
template <bool kWKn, bool kGated>
__global__ void __launch_bounds__(kT2Threads, 1)
grouped_gemm_fp8t256_kernel(const __grid_constant__ CUtensorMap tmap_a,
                            const __grid_constant__ CUtensorMap tmap_w, const TParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int stages = p.stages;
  uint8_t* xpose_base = smem + stages * kT2StageBytes;
  T2Ctrl* ctrl = reinterpret_cast<T2Ctrl*>(xpose_base + kT2XposeBytes);
  uint8_t* walk_mem = reinterpret_cast<uint8_t*>(ctrl) + ((sizeof(T2Ctrl) + 15) & ~(size_t)15);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // 256-feature tiles; gated: one tile per 128 gate features (p.n_tiles counts 128-feature blocks of n)
  const int n_tiles2 = kGated ? p.n_tiles / 2 : (p.n_tiles + 1) / 2;
  const int up_block0 = p.n_tiles / 2;        // gated: first 128-feature block of the up half

  if (warp == 0) {
    pdl_wait();
    build_tile_walk<kTTok>(p.rows_per_expert, p.num_experts, n_tiles2, walk_mem);
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a);
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
      ptx::mbar_init(&ctrl->acc_full[a], 1);
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
  const int n_groups = (p.num_kb + kTGroup - 1) / kTGroup;
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
        for (int kb = 0; kb < p.num_kb; ++kb) {
          const uint32_t full = full0 + 8 * s;
          if (!ptx::mbar_wait_s(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          ptx::mbar_expect_tx_s(full, kT2StageBytes);
          // two 128-feature blocks (the second one is zero-filled past N)
          if (!kWKn) {
            ptx::tma_load_3d_s(st, &tmap_w, full, kb * 128, n0, ti.e);
            ptx::tma_load_3d_s(st + 16384, &tmap_w, full, kb * 128, n1, ti.e);
          } else {
            ptx::tma_load_3d_s(st, &tmap_w, full, n0, kb * 128, ti.e);
            ptx::tma_load_3d_s(st + 16384, &tmap_w, full, n1, kb * 128, ti.e);
          }
          ptx::tma_load_2d_s(st + 32768, &tmap_a, full, kb * 128, ti.row0);
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
      int my_tiles = 0;
      for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) ++my_tiles;
      const int64_t blocks = (int64_t)my_tiles * p.num_kb;   // every tile: same K loop, no tile state needed
      const uint32_t idesc = (p.idesc & ~(0x3fu << 17)) | ((256u >> 3) << 17);
      for (int64_t i = 0; i < blocks; ++i) {
        if (!ptx::mbar_wait_s(full0 + 8 * s, ph, abort_flag)) break;
        if (!ptx::mbar_wait_s(acc_empty0 + 8 * a, aph, abort_flag)) break;
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
      const bool vec4_ok = (kbs % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.a_scale) & 15) == 0);
      uint32_t slot = 0, ph = 1, seq = 0;
      int cursor = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++seq) {
        TileInfo ti;
        locate_tile<kTTok>(walk, t, cursor, ti, p.w_experts);
        const int nb0 = kGated ? ti.n_tile : ti.n_tile * 2, nb1 = kGated ? ti.n_tile + up_block0 : nb0 + 1;
        const float* w0 = p.w_scale + ((int64_t)ti.e * p.n_tiles + nb0) * kbs;
        const float* w1 = w0 + (nb1 < p.n_tiles ? (int64_t)(nb1 - nb0) * kbs : 0);   // past N: any scale, the block's values are zero
        for (int g = 0; g < n_groups; ++g) {
          const int kb0 = g * kTGroup;
          float4 av[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int row = ft + 64 * i;
            const bool live = row < ti.valid;
            const float* src = p.a_scale + (int64_t)(ti.row0 + row) * kbs + kb0;
            if (vec4_ok) {
              av[i] = live ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
              av[i].x = live ? __ldg(src) : 0.f;
              av[i].y = live && kb0 + 1 < kbs ? __ldg(src + 1) : 0.f;
              av[i].z = live && kb0 + 2 < kbs ? __ldg(src + 2) : 0.f;
              av[i].w = live && kb0 + 3 < kbs ? __ldg(src + 3) : 0.f;
            }
          }
          float wv[2][kTGroup];
#pragma unroll
          for (int j = 0; j < kTGroup; ++j) {
            const int kl = min(kb0 + j, kbs - 1);
            wv[0][j] = __ldg(w0 + kl);
            wv[1][j] = __ldg(w1 + kl);
          }
          if (!__all_sync(0xffffffffu, ptx::mbar_wait_inline_s(sf_empty0 + 8 * slot, ph, abort_flag))) { ok = false; break; }
          T2Slot* out = &ctrl->slot[slot];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float rv[kTGroup] = {av[i].x, av[i].y, av[i].z, av[i].w};
#pragma unroll
            for (int j = 0; j < kTGroup; ++j) {
              out->s[0][j][ft + 64 * i] = rv[j] * wv[0][j];
              out->s[1][j][ft + 64 * i] = rv[j] * wv[1][j];
            }
          }
          if (ft == 0 && g == 0) ctrl->tile[seq & 3] = make_int4(ti.row0, ti.valid, ti.n_tile, ti.e);
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_s(sf_full0 + 8 * slot);
          if (++slot == kT2Slots) { slot = 0; ph ^= 1; }
        }
      }
    }
  } else {
    // ------------------------ promotion and epilogue --------------------------
    ptx::setmaxnreg_inc<kT2HighRegs>();
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const int half = (warp - 4) >> 2;                  // which 128-feature block of the tile (gated: which 64 features of both)
    uint32_t a = 0, aph = 0, slot = 0, sph = 0, xpar = 0;
    // one shared address, the rest are constants from there (registers are full)
    const uint32_t cs = ptx::smem_u32(ctrl);
    constexpr uint32_t kAccFull = offsetof(T2Ctrl, acc_full), kAccEmpty = offsetof(T2Ctrl, acc_empty);
    constexpr uint32_t kSfFull = offsetof(T2Ctrl, sf_full), kSfEmpty = offsetof(T2Ctrl, sf_empty), kSlot = offsetof(T2Ctrl, slot);
    bool ok = true;
    const int my_tiles = (int)blockIdx.x < total_tiles ? (total_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    // A K block's scales are read when its first chunk is asked for, without a branch.
    float sc0 = 0.f, sc1 = 0.f;
    uint32_t jb = 0;                                   // position in the slot
    const uint32_t my_scales = cs + kSlot + (kGated ? 0 : half * kTGroup * 512) + r * 4;
    auto read_scales = [&](bool last) {                // `last`: the tile's last K block
      const uint32_t at = my_scales + slot * (uint32_t)sizeof(T2Slot) + jb * 512;
      sc0 = ptx::lds32f(at);
      if (kGated) sc1 = ptx::lds32f(at + kTGroup * 512);
      const bool done = jb == kTGroup - 1 || last;
      __syncwarp();   // lane 0's arrival hands the slot back for all lanes: their reads come first
      ptx::mbar_arrive_if(cs + kSfEmpty + 8 * slot, done && lane == 0);
      jb = done ? 0u : jb + 1;
      slot ^= done ? 1u : 0u;
      sph ^= done && slot == 0 ? 1u : 0u;
    };
    static_assert(kT2Slots == 2, "slot parity");
    auto wait_block = [&]() {                          // the stage and the scales of the next K block
      return __all_sync(0xffffffffu, ptx::mbar_wait_inline_s(cs + kAccFull + 8 * a, aph, abort_flag) &&
                                         ptx::mbar_wait_inline_s(cs + kSfFull + 8 * slot, sph, abort_flag));
    };
    // Chunks of 32 columns (chunk c of a stage -> acc[16 c ..]).  plain: the 128 columns of this warp's
    // block; gated: 64 gate columns, then the 64 up columns of the same features.
    const uint32_t col_base = tmem_base + (kGated ? half * 64 : half * 128) + lane_sel;
    constexpr uint32_t kSecond = kGated ? 128 : 64;
    for (int tile = 0; tile < my_tiles && ok; ++tile) {
      float2 acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = make_float2(0.f, 0.f);
      uint32_t va[32], vb[32];
      if (!wait_block()) { ok = false; break; }
      ptx::tc_fence_after();
      ptx::tmem_ld_32x32(col_base + a * 256, va);
      read_scales(p.num_kb == 1);
#pragma unroll 1
      for (int kb = 0; kb < p.num_kb; ++kb) {
        const uint32_t col = col_base + a * 256, empty = cs + kAccEmpty + 8 * a;
        const bool more = kb + 1 < p.num_kb;
        const float c0 = sc0, c1 = kGated ? sc1 : sc0;
        if (++a == (uint32_t)kT2Acc) { a = 0; aph ^= 1; }
        ptx::tmem_wait_ld_one(va);
        ptx::tmem_ld_32x32(col + 32, vb);
        ptx::fma_f32x2(acc, va, c0);
        ptx::tmem_wait_ld_one(vb);
        ptx::tmem_ld_32x32(col + kSecond, va);
        ptx::fma_f32x2(acc + 16, vb, c0);
        ptx::tmem_wait_ld_one(va);
        ptx::tmem_ld_32x32(col + kSecond + 32, vb);
        const bool ready = ptx::mbar_test_wait_s(cs + kAccFull + 8 * a, aph) & ptx::mbar_test_wait_s(cs + kSfFull + 8 * slot, sph);
        ptx::fma_f32x2(acc + 32, va, c1);
        ptx::tmem_wait_ld_one(vb);
        ptx::tc_fence_before();   // the whole stage is in registers
        __syncwarp();
        ptx::mbar_arrive_if(empty, lane == 0);
        if (more) {
          if (!__all_sync(0xffffffffu, ready) && !wait_block()) { ok = false; break; }
          ptx::tc_fence_after();
          ptx::tmem_ld_32x32(col_base + a * 256, va);
          read_scales(kb + 2 == p.num_kb);
        }
        ptx::fma_f32x2(acc + 48, vb, c1);
      }
      if (!ok) { ptx::tmem_wait_ld(); break; }
      const int4 here = ctrl->tile[tile & 3];
      TileInfo ti;
      ti.row0 = here.x; ti.valid = here.y; ti.n_tile = here.z; ti.e = here.w;
      auto value = [&](int i) -> float& { return (i & 1) ? acc[i >> 1].y : acc[i >> 1].x; };
      if (kGated) {
        // values 0..63 = gate, 64..127 = up of features j0 + half * 64 ..
        const int half_n = p.n >> 1;
        const int j0 = ti.n_tile * 128 + half * 64;
        float amax = 0.f;
        // value(i) becomes the activated value of feature j0 + i (the up half is consumed)
        auto activate = [&](auto round16) {
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            float g = value(i), u = value(64 + i);
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
            value(i) = __fmul_rn(__fdividef(g, 1.0f + __expf(-g)), u);
            amax = fmaxf(amax, fabsf(value(i)));
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
          // 64 codes of this thread's row into the warp's staging tile (rows of 64 + 16 bytes)
          const uint32_t my_row = ptx::smem_u32(xpose_base + (warp - 4) * 32 * kT2RowPitch) + lane * kT2RowPitch;
#pragma unroll
          for (int c = 0; c < 64; c += 16) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              uint32_t x = 0;
#pragma unroll
              for (int b = 0; b < 4; ++b)
                x |= (uint32_t)f32_to_e4m3(fmaxf(-448.0f, fminf(__fdividef(value(c + i + b), scale), 448.0f))) << (8 * b);
              w[i >> 2] = x;
            }
            ptx::sts128(my_row + c, make_uint4(w[0], w[1], w[2], w[3]));
          }
          if (half == 0) p.d_scale[(int64_t)(ti.row0 + r) * (half_n >> 7) + ti.n_tile] = scale;
        }
        __syncwarp();
        if (ok) {
          // eight rows per store: four lanes cover the 64 bytes of a row
          const uint32_t xp = ptx::smem_u32(xpose_base + (warp - 4) * 32 * kT2RowPitch);
          const int piece = lane & 3;
          uint8_t* dbase = reinterpret_cast<uint8_t*>(p.d) + (int64_t)(ti.row0 + q * 32) * half_n + j0 + piece * 16;
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int rr = it * 8 + (lane >> 2);
            if (q * 32 + rr < ti.valid)
              *reinterpret_cast<uint4*>(dbase + (int64_t)rr * half_n) = ptx::lds128(xp + rr * kT2RowPitch + piece * 16);
          }
        }
        __syncwarp();
        continue;
      }
      const int f0 = ti.n_tile * 256 + half * 128;
      if (ok && f0 < p.n) {
        // the 128 finished values of this thread's row, bias added and rounded, as 16 x 16 bytes
        auto packed = [&](int c, uint32_t (&w)[4]) {
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            float x0 = value(c + i), x1 = value(c + i + 1);
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
        };
        const uint32_t xp = ptx::smem_u32(xpose_base + (warp - 4) * 32 * kT2RowPitch);
        const int piece = lane & 3;
        uint16_t* dbase = reinterpret_cast<uint16_t*>(p.d) + (int64_t)(ti.row0 + q * 32) * p.n + f0 + piece * 8;
#pragma unroll
        for (int c0 = 0; c0 < 128; c0 += 32) {
          // 32 values of this thread's row into the warp's staging tile ...
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint32_t w[4];
            packed(c0 + c, w);
            ptx::sts128(xp + lane * kT2RowPitch + c * 2, make_uint4(w[0], w[1], w[2], w[3]));
          }
          __syncwarp();
          // ... and out again eight rows per store: four lanes cover the 64 bytes of a row
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int rr = it * 8 + (lane >> 2);
            if (q * 32 + rr < ti.valid)
              *reinterpret_cast<uint4*>(dbase + (int64_t)rr * p.n + c0) = ptx::lds128(xp + rr * kT2RowPitch + piece * 16);
          }
          __syncwarp();
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
    ptx::tmem_dealloc(tmem_base, 512);
  }
  if (tid == 0 && *abort_flag != 0) report_timeout(p.status);
}

template <bool kWKn, bool kGated>
int launch_fp8t256(const CUtensorMap& ta, const CUtensorMap& tw, TParams& p, int grid, cudaStream_t st) {
  auto kern = grouped_gemm_fp8t256_kernel<kWKn, kGated>;
  const size_t fixed = kT2Fixed + tile_walk_bytes(p.num_experts);
  p.stages = fixed + kT2Stages * (size_t)kT2StageBytes <= kMaxSmem ? kT2Stages : 3;
  const size_t smem = fixed + p.stages * (size_t)kT2StageBytes;
  static SmemConfig configured;
  if (int rc = configured.ensure(kern)) return rc;
  B200_LAUNCHED("grouped_gemm_fp8t256_kernel", launch_pdl(p.m <= kEarlyLaunchRows, kern, dim3(grid), dim3(kT2Threads), smem, st, ta, tw, p));
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
  const int w_sets = (a->w_experts > 0 && a->w_experts != a->num_experts) ? a->w_experts : a->num_experts;
  p.w_experts = w_sets != a->num_experts ? w_sets : 0;
  p.n_tiles = a->n / kFeat;
  p.num_kb = a->k / 128;
  p.out_f16 = gated ? (a->mid_dtype == B200MOE_F16) : (a->d_dtype == B200MOE_F16);
  p.d_scale = reinterpret_cast<float*>(a->d_scale);
  p.clamp = a->clamp_limit;
  // A operand = tokens (K-major), B operand = weights (K-major, or MN-major for [E,K,N])
  p.idesc = ptx::make_idesc(0u, 0u, 0u, kn ? 1u : 0u, kTTok, kFeat);

  CUtensorMap ta, tw;
  {
    cuuint64_t dims[2] = {(cuuint64_t)a->k, (cuuint64_t)a->m};
    cuuint64_t strides[1] = {(cuuint64_t)a->k};
    cuuint32_t box[2] = {128, (cuuint32_t)kTTok};
    int rc = encode_map(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, a->a, dims, strides, box);
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
  const bool wide = a->n >= 256;   // 256-feature tiles; a single 128-feature block takes the narrow kernel
  const int64_t tile_bound = ((a->m + kTTok - 1) / kTTok + a->num_experts) * (int64_t)(wide ? (p.n_tiles + 1) / 2 : p.n_tiles);
  if (tile_bound < grid) grid = (int)tile_bound;
  if (grid < 1) grid = 1;
  if (gated) return kn ? launch_fp8t256<true, true>(ta, tw, p, grid, st) : launch_fp8t256<false, true>(ta, tw, p, grid, st);
  if (wide) return kn ? launch_fp8t256<true, false>(ta, tw, p, grid, st) : launch_fp8t256<false, false>(ta, tw, p, grid, st);
  return kn ? launch_fp8t<true>(ta, tw, p, grid, st) : launch_fp8t<false>(ta, tw, p, grid, st);
}

}  // namespace b200moe
