// Token -> expert bookkeeping: moe_align_block_size, remap_hidden_states,
// init_expert_map and the fused permute + fp8 group quantisation.
//
// Both ops are a stable counting sort of the T*K routed slots by (mapped)
// expert id.  The slots are cut into chunks of 256 handled by one warp each:
//   1. count : every warp builds a histogram of its chunk,
//   2. scan  : per expert an exclusive scan over the chunks (a warp each); every block of the next step
//              then scans the experts itself (padded to block_size for the align op),
//   3. rank  : every warp walks its chunk 32 slots at a time; the rank of a
//              slot among equal ids in the same step comes from
//              __match_any_sync, so slots of one expert keep ascending order.
// Up to 2048 slots all three steps run in one block without any scratch; beyond
// that in one cluster of blocks (row maps) or in three launches (sort.cuh).  The
// result is deterministic: no atomics decide an order.
//
// Semantics follow csrc/moe/moe_align_sum_kernels.cpp:135-273, 1034-1181 and
// csrc/moe/remap_hidden_states.cpp:42-116, 181-330 of vllm-xpu-kernels, which
// leave the order inside an expert unspecified.
#include <atomic>

#include "common.cuh"
#include "mx_quant.cuh"
#include "sort.cuh"

namespace b200moe {
namespace {

// ------------------------- row copies ------------------------------------------
// One block per token: its row is read once and written to its K destinations (`dest` in shared
// memory, negative = none), as it is, quantised to e4m3 per 1x128 group, or as MXFP8 planes.
struct RowJob {
  const void* src;
  void* dst;
  const void* src_s;     // copy: the caller's scale rows, or null
  void* dst_s;           // copy: their destination; fp8: fp32 [rows, H/128]; mx: words [planes][ceil(H/128)][rows]
  int row_bytes;         // copy
  int scale_row_bytes;   // copy
  int H;                 // quantised forms: values per row
  int K;
  int64_t rows;          // mx: rows of a plane (T * K)
  int planes;            // mx: 1 to 3
  int sums;              // mx: fp32 block sums [ceil(H/128)][rows] follow the scale words
  int evens_first;       // mx with sums: the even codes of eight before the odd ones
};

__device__ __forceinline__ void copy_scales(const RowJob& a, int64_t tok, const int* dest) {
  if (a.src_s == nullptr) return;
  const uint8_t* ss = reinterpret_cast<const uint8_t*>(a.src_s) + tok * (int64_t)a.scale_row_bytes;
  uint8_t* dst_s = reinterpret_cast<uint8_t*>(a.dst_s);
  if ((a.scale_row_bytes & 3) == 0) {
    for (int j = threadIdx.x; j < (a.scale_row_bytes >> 2); j += blockDim.x) {
      const uint32_t v = reinterpret_cast<const uint32_t*>(ss)[j];
      for (int k = 0; k < a.K; ++k) {
        const int r = dest[k];
        if (r >= 0) reinterpret_cast<uint32_t*>(dst_s + (int64_t)r * a.scale_row_bytes)[j] = v;
      }
    }
  } else {
    for (int j = threadIdx.x; j < a.scale_row_bytes; j += blockDim.x) {
      const uint8_t v = ss[j];
      for (int k = 0; k < a.K; ++k) {
        const int r = dest[k];
        if (r >= 0) dst_s[(int64_t)r * a.scale_row_bytes + j] = v;
      }
    }
  }
}

// Per-1x128 dynamic e4m3 quantisation of piece j.  A lane holds 8 consecutive elements, 16 lanes
// cover one 128-wide group; all lanes of the warp call it.
template <typename T>
__device__ __forceinline__ void quant_piece_fp8(const RowJob& a, int j, bool in, const vec16& v, const int* dest) {
  const int H = a.H;
  const T* e = reinterpret_cast<const T*>(&v);
  float x[8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) { x[i] = in ? to_f32<T>(e[i]) : 0.f; amax = fmaxf(amax, fabsf(x[i])); }
#pragma unroll
  for (int mask = 8; mask > 0; mask >>= 1)
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, mask));
  amax = fmaxf(amax, 1e-10f);
  const float scale = fmaxf(__fdiv_rn(amax, 448.f), 1.0f / (448.f * 512.f));
  const float inv = __fdiv_rn(1.0f, scale);
  if (!in) return;
  uint32_t c[2] = {0u, 0u};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float q = fminf(fmaxf(__fmul_rn(x[i], inv), -448.f), 448.f);
    c[i >> 2] |= (uint32_t)f32_to_e4m3(q) << (8 * (i & 3));
  }
  uint8_t* dst_q = reinterpret_cast<uint8_t*>(a.dst);
  float* dst_s = reinterpret_cast<float*>(a.dst_s);
  for (int k = 0; k < a.K; ++k) {
    const int r = dest[k];
    if (r >= 0) {
      *reinterpret_cast<uint2*>(dst_q + (int64_t)r * H + (int64_t)j * 8) = make_uint2(c[0], c[1]);
      if ((j & 15) == 0) dst_s[(int64_t)r * (H / 128) + j / 16] = scale;
    }
  }
}

// MXFP8 planes (mx_quant.cuh); sixteen lanes cover a 128-wide K block, whose first lane writes its
// scale word.
template <typename T>
__device__ __forceinline__ void quant_piece_mx(const RowJob& a, int j, bool in, const vec16& x, const int* dest) {
  const int H = a.H, num_kb = (H + 127) / 128;
  const T* e = reinterpret_cast<const T*>(&x);
  uint8_t* dst_q = reinterpret_cast<uint8_t*>(a.dst);
  uint32_t* dst_s = reinterpret_cast<uint32_t*>(a.dst_s);
  float v[8];
  float total = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) { v[i] = in ? to_f32<T>(e[i]) : 0.f; total += v[i]; }
#pragma unroll 1
  for (int p = 0; p < a.planes; ++p) {
    uint2 codes;
    const uint32_t word = mx_quant_lane(v, in, codes, a.sums ? kMxLeastExact : kMxLeast, a.sums || p + 1 < a.planes);
    if (a.evens_first) codes = mx_evens_first(codes);
    uint8_t* q = dst_q + p * a.rows * H + (int64_t)j * 8;
    uint32_t* s = dst_s + ((int64_t)p * num_kb + (j >> 4)) * a.rows;
    for (int k = 0; k < a.K; ++k) {
      const int r = dest[k];
      if (r >= 0) {
        if (in) *reinterpret_cast<uint2*>(q + (int64_t)r * H) = codes;
        if ((j & 15) == 0 && j < num_kb * 16) s[r] = word;
      }
    }
  }
  if (a.sums) {
#pragma unroll
    for (int i = 0; i < 8; ++i) total -= v[i];
    total = mx_block_sum(total);
    if ((j & 15) == 0 && j < num_kb * 16)
      for (int k = 0; k < a.K; ++k)
        if (dest[k] >= 0)
          reinterpret_cast<float*>(dst_s)[((int64_t)a.planes * num_kb + (j >> 4)) * a.rows + dest[k]] = total;
  }
}

enum RowForm { kRowCopy = 0, kRowFp8 = 1, kRowMx = 2 };
// Piece j (16 bytes of the source row; `v` is read only for j < nvec) to its destinations.
template <typename T, int kForm>
__device__ __forceinline__ void place_piece(const RowJob& a, int j, int nvec, const vec16& v, const int* dest) {
  if (kForm == kRowCopy) {
    if (j >= nvec) return;
    for (int k = 0; k < a.K; ++k) {
      const int r = dest[k];
      if (r >= 0) st16(reinterpret_cast<uint8_t*>(a.dst) + (int64_t)r * a.row_bytes + (int64_t)j * 16, v);
    }
  } else if (kForm == kRowFp8) {
    quant_piece_fp8<T>(a, j, j < nvec, v, dest);
  } else {
    quant_piece_mx<T>(a, j, j < nvec, v, dest);
  }
}
template <typename T, int kForm>
__device__ __forceinline__ void place_row(const RowJob& a, int64_t tok, const int* dest) {
  const int nvec = kForm == kRowCopy ? a.row_bytes >> 4 : a.H / 8;
  const int steps = kForm == kRowMx ? ((a.H + 127) / 128) * 16 : nvec;
  const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src) + tok * (int64_t)nvec * 16;
  // full warps iterate together so that the shuffles stay converged
  for (int j0 = (threadIdx.x & ~31); j0 < steps; j0 += blockDim.x) {
    const int j = j0 + (threadIdx.x & 31);
    vec16 v;
    if (j < nvec) v = ld16(src + (int64_t)j * 16);
    place_piece<T, kForm>(a, j, nvec, v, dest);
  }
  if (kForm == kRowCopy) copy_scales(a, tok, dest);
}

template <typename T, int kForm>
__global__ void __launch_bounds__(256)
remap_rows_kernel(const RowJob a, const int32_t* __restrict__ row_map) {
  pdl_trigger();
  pdl_wait();
  __shared__ int dest[32];
  const int64_t tok = blockIdx.x;
  if (threadIdx.x < a.K) dest[threadIdx.x] = row_map[tok * a.K + threadIdx.x];
  __syncthreads();
  place_row<T, kForm>(a, tok, dest);
}

// Up to kBlockSlots routed slots: the bookkeeping and the rows in one launch.  A block finds its
// token's positions by itself: the position of slot i is the number of slots with a smaller bucket
// plus the number of earlier slots with the same one, counted over all slots by the block's threads
// (2048 slots x 8 are 64 comparisons a thread).  One more block counts the rows per expert.  The
// separate sort, a single block that everything waited for, took 6 to 10 us of a decode step and
// its launch.  K up to kSmallK, else the sort.
//
// What remains is latency: the row's loads are issued before the counting, and the code is kept
// small (a kernel that runs for 3 us runs from a cold instruction cache).
constexpr int kSmallK = 8;
// 512 threads with up to two pieces each rather than 256 with four: the quantised forms are unrolled over the
// pieces, and half the code is half the cold instruction fetches.  What the kernel adds to a decode layer's chain,
// MXFP8 planes: one gpt-oss token 4.9 -> 3.6 us, 128 tokens 6.9 -> 5.1, 33 int4 Mixtral tokens 5.8 -> 4.1; plain rows
// and 1x128 fp8 as before (2.7 and 3.4).
constexpr int kSmallThreads = 512;
constexpr int kSmallPre = 2;   // 16-byte pieces of the row a thread holds while the positions are counted
template <typename T, int kForm, typename Id>
__global__ void __launch_bounds__(kSmallThreads)
remap_small_kernel(const Id* __restrict__ ids, const int32_t* __restrict__ map, int numel, int id_limit, int n_buckets,
                   const RowJob a, int32_t* __restrict__ rows_per_expert, int32_t* __restrict__ row_map) {
  __shared__ int dest[kSmallK];
  __shared__ uint32_t part[kSmallThreads / 32][kSmallK / 2];
  __shared__ int hist[kMaxBuckets];
  pdl_trigger();
  pdl_wait();
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, K = a.K;
  auto bucket = [&](int i) {
    const Id e = ids[i];
    if (e < (Id)0 || e >= (Id)id_limit) return -1;
    const int b = map != nullptr ? map[e] : (int)e;
    return b < n_buckets ? b : -1;   // (a negative entry of the map stays negative)
  };
  if (blockIdx.x == gridDim.x - 1) {
    for (int e = t; e < n_buckets; e += kSmallThreads) hist[e] = 0;
    __syncthreads();
    for (int i = t; i < numel; i += kSmallThreads) {
      const int b = bucket(i);
      if (b >= 0) atomicAdd(&hist[b], 1);
    }
    __syncthreads();
    for (int e = t; e < n_buckets; e += kSmallThreads) rows_per_expert[e] = hist[e];
    return;
  }
  const int64_t tok = blockIdx.x;
  const int slot0 = (int)tok * K;
  // (the quantised forms walk whole 128-value groups)
  const int nvec = kForm == kRowCopy ? a.row_bytes >> 4 : a.H / 8;
  const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src) + tok * (int64_t)nvec * 16;
  vec16 pre[kSmallPre];
#pragma unroll
  for (int i = 0; i < kSmallPre; ++i)
    if (t + kSmallThreads * i < nvec) pre[i] = ld16(src + (int64_t)(t + kSmallThreads * i) * 16);
  int own[kSmallK];
#pragma unroll
  for (int k = 0; k < kSmallK; ++k) own[k] = k < K ? bucket(slot0 + k) : -1;
  uint32_t cnt[kSmallK / 2] = {};   // two 16-bit counters a word
#pragma unroll 1
  for (int i = t; i < numel; i += kSmallThreads) {
    const int b = bucket(i);
#pragma unroll
    for (int k = 0; k < kSmallK; ++k)
      if (b >= 0 && (b < own[k] || (b == own[k] && i < slot0 + k))) cnt[k >> 1] += 1u << (16 * (k & 1));
  }
#pragma unroll
  for (int k = 0; k < kSmallK / 2; ++k) {
    cnt[k] = __reduce_add_sync(0xffffffffu, cnt[k]);
    if (lane == 0) part[warp][k] = cnt[k];
  }
  __syncthreads();
  if (t < K) {
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < kSmallThreads / 32; ++w) sum += part[w][t >> 1];
    const int pos = bucket(slot0 + t) < 0 ? -1 : (int)((sum >> (16 * (t & 1))) & 0xffffu);
    dest[t] = pos;
    row_map[slot0 + t] = pos;
  }
  __syncthreads();
  const int steps = kForm == kRowMx ? ((a.H + 127) / 128) * 16 : nvec;
  if (steps <= kSmallThreads * kSmallPre) {
#pragma unroll
    for (int i = 0; i < kSmallPre; ++i)
      if ((t & ~31) + kSmallThreads * i < steps) place_piece<T, kForm>(a, t + kSmallThreads * i, nvec, pre[i], dest);
    if (kForm == kRowCopy) copy_scales(a, tok, dest);
  } else {
    place_row<T, kForm>(a, tok, dest);
  }
}

__global__ void init_expert_map_kernel(int32_t* map, int n_local, int ep_rank, int total) {
  pdl_trigger();
  pdl_wait();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < total) {
    const int lo = ep_rank * n_local;
    map[g] = (g >= lo && g < lo + n_local) ? g - lo : -1;
  }
}

int check_ids_dtype(b200moe_dtype t, const char* name) {
  if (t == B200MOE_I32 || t == B200MOE_I64 || t == B200MOE_U32) return 0;
  return fail(B200MOE_E_BADARG, "%s: topk_ids must be int64 or int32", name);
}

int remap_params(SortParams& p, const int32_t* expert_map, const int32_t* rows_per_expert, const int32_t* row_map,
                 const void* topk_ids, b200moe_dtype ids_dtype, int64_t num_rows, int topk, int total_experts,
                 int local_experts) {
  if (check_ids_dtype(ids_dtype, "remap_hidden_states")) return B200MOE_E_BADARG;
  B200_CHECK_ARG(topk >= 1 && topk <= 32, "Unsupported TopK value");
  B200_CHECK_ARG(local_experts >= 1 && local_experts <= kMaxBuckets,
                 "local_experts_num exceeds the maximum supported number");
  B200_CHECK_ARG(rows_per_expert && row_map && topk_ids, "remap_hidden_states: null pointer");
  p.ids = topk_ids; p.ids_dtype = ids_dtype; p.map = expert_map;
  p.numel = num_rows * topk;
  p.id_limit = expert_map ? total_experts : local_experts;
  p.n_buckets = local_experts;
  p.block_size = 1;
  return B200MOE_OK;
}

// Bookkeeping and rows: one launch where the slots fit one block's count, else the sort and a
// kernel that places the rows.
template <typename T, int kForm>
int remap_rows(const SortParams& p, const RowJob& job, int32_t* rows_per_expert, int32_t* row_map, int64_t num_rows,
               void* workspace, size_t workspace_bytes, cudaStream_t st) {
  const bool early = p.numel <= kEarlyLaunchRows;
  if (p.numel > 0 && p.numel <= kBlockSlots && job.K <= kSmallK) {
    const dim3 grid((unsigned)num_rows + 1);
#define B200_REMAP_SMALL(ID)                                                                                          \
  B200_LAUNCHED("remap_small_kernel", launch_pdl(early, remap_small_kernel<T, kForm, ID>, grid, dim3(kSmallThreads), 0, st, \
                                                 (const ID*)p.ids, p.map, (int)p.numel, p.id_limit, p.n_buckets, job, \
                                                 rows_per_expert, row_map))
    if (p.ids_dtype == B200MOE_I64) B200_REMAP_SMALL(int64_t);
    else if (p.ids_dtype == B200MOE_U32) B200_REMAP_SMALL(uint32_t);
    else B200_REMAP_SMALL(int32_t);
#undef B200_REMAP_SMALL
    return B200MOE_OK;
  }
  AlignOut ao = {};
  RemapOut ro = {rows_per_expert, row_map};
  if (int rc = run_sort<1>(p, ao, ro, workspace, workspace_bytes, st)) return rc;
  if (num_rows == 0) return B200MOE_OK;
  B200_LAUNCHED("remap_rows_kernel", launch_pdl(early, remap_rows_kernel<T, kForm>, dim3((unsigned)num_rows),
                                                dim3(256), 0, st, job, row_map));
  return B200MOE_OK;
}

}  // namespace
}  // namespace b200moe

using namespace b200moe;

extern "C" size_t b200moe_sort_workspace_bytes(int64_t numel, int num_experts) {
  if (numel <= kBlockSlots) return 0;
  const int64_t n_chunks = (numel + kChunk - 1) / kChunk;
  const size_t ints = (size_t)num_experts * n_chunks + num_experts + 1;
  return (ints * sizeof(int) + 255) & ~(size_t)255;
}

extern "C" int b200moe_moe_align_block_size(
    const void* topk_ids, b200moe_dtype ids_dtype, int64_t numel, int num_experts,
    int block_size, int32_t* sorted_token_ids, int64_t sorted_len, int32_t* expert_ids,
    int64_t expert_ids_len, int32_t* num_tokens_post_pad, const int32_t* expert_map,
    void* workspace, size_t workspace_bytes, b200moe_stream stream) {
  B200_CHECK_ARG(ids_dtype == B200MOE_I32 || ids_dtype == B200MOE_I64 || ids_dtype == B200MOE_U32,
                 "moe_align_block_size: topk_ids must be an integer tensor");
  B200_CHECK_ARG(num_experts >= 1 && ((num_experts + 31) / 32) * 32 < 1024,
                 "padded_num_experts must be less than 1024");
  B200_CHECK_ARG(block_size >= 1, "moe_align_block_size: block_size must be positive");
  B200_CHECK_ARG(numel >= 0 && sorted_len >= 0 && expert_ids_len >= 0,
                 "moe_align_block_size: negative size");
  B200_CHECK_ARG((sorted_len == 0 || sorted_token_ids) && (expert_ids_len == 0 || expert_ids) &&
                     num_tokens_post_pad,
                 "moe_align_block_size: null output");
  B200_CHECK_ARG(numel == 0 || topk_ids, "moe_align_block_size: null topk_ids");
  SortParams p;
  p.ids = topk_ids; p.ids_dtype = ids_dtype; p.map = expert_map;
  p.numel = numel; p.id_limit = num_experts; p.n_buckets = num_experts;
  p.block_size = block_size;
  AlignOut ao = {sorted_token_ids, sorted_len, expert_ids, expert_ids_len, num_tokens_post_pad};
  RemapOut ro = {};
  return run_sort<0>(p, ao, ro, workspace, workspace_bytes, as_stream(stream));
}

// ------------------------- legacy prologue ------------------------------------
namespace b200moe {
namespace {

// Tokens per block of the reference's three-step sort; it only enters the size
// of two scratch regions of the packed workspace
// (csrc/moe/fused_moe_prologue.hpp:43-60 of the reference).
int64_t prologue_tokens_per_block(int64_t num_tokens, int64_t experts) {
  for (int64_t n = 32; n <= 1024; n *= 2)
    if ((num_tokens + n - 1) / n * experts <= n) return n;
  return 1024;
}

struct PrologueArgs {
  const unsigned char* input;  unsigned char* permuted;  int64_t row_bytes;
  const unsigned char* scales; unsigned char* permuted_scales; int64_t scale_row_bytes;
  const float* final_scales;   float* permuted_final_scales;
  const int32_t* rows_per_expert;  // [experts]
  const int32_t* row_map;          // [tokens * topk], -1 = not on this rank
  const void* ids; int id_offset;
  int32_t* permuted_to_unpermuted; int32_t* permuted_experts; int32_t* unpermuted_to_permuted;
  int64_t* first_token_offset;     // [experts + 1]
  int64_t num_tokens; int topk; int experts;
};

__device__ __forceinline__ void copy_bytes(unsigned char* dst, const unsigned char* src, int64_t n) {
  if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src) | (uintptr_t)n) & 15) == 0) {
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
    uint4* d4 = reinterpret_cast<uint4*>(dst);
    for (int64_t i = threadIdx.x; i < n / 16; i += blockDim.x) d4[i] = s4[i];
  } else {
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  }
}

// One block per routed slot (grid-stride): copies the token's row, its scale row
// and its routing weight to the slot's permuted position and writes the three
// index maps.  Block 0 first turns the per-expert counts into the int64 offsets.
__global__ void __launch_bounds__(kBlockThreads)
prologue_expand_kernel(PrologueArgs a) {
  pdl_trigger();
  pdl_wait();
  __shared__ int scan[kMaxBuckets + 1];
  __shared__ int warp_tot[kWarps];
  if (blockIdx.x == 0) {
    for (int e = threadIdx.x; e < a.experts; e += kBlockThreads) scan[e] = a.rows_per_expert[e];
    __syncthreads();
    block_exclusive_scan(scan, a.experts, warp_tot);
    for (int e = threadIdx.x; e <= a.experts; e += kBlockThreads) a.first_token_offset[e] = scan[e];
  }
  const int64_t n = a.num_tokens * a.topk;
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int pos = a.row_map[i];
    if (pos < 0) continue;
    const int64_t token = i / a.topk;
    const int k = (int)(i - token * a.topk);
    if (threadIdx.x == 0) {
      const int32_t u = (int32_t)(k * a.num_tokens + token);
      a.permuted_to_unpermuted[pos] = u;
      a.unpermuted_to_permuted[u] = pos;
      a.permuted_experts[pos] = (int32_t)(reinterpret_cast<const int64_t*>(a.ids)[i] - a.id_offset);
      a.permuted_final_scales[pos] = a.final_scales ? a.final_scales[i] : 1.0f;
    }
    copy_bytes(a.permuted + (int64_t)pos * a.row_bytes, a.input + token * a.row_bytes, a.row_bytes);
    if (a.scales != nullptr)
      copy_bytes(a.permuted_scales + (int64_t)pos * a.scale_row_bytes,
                 a.scales + token * a.scale_row_bytes, a.scale_row_bytes);
  }
}

}  // namespace
}  // namespace b200moe

extern "C" int b200moe_fused_moe_prologue_layout(int64_t num_rows, int topk, int num_experts_on_rank,
                                                 int64_t hidden_size, int block_k, int elem_bytes,
                                                 int scale_elem_bytes, size_t offsets[10],
                                                 size_t* total_bytes) {
  B200_CHECK_ARG(num_rows >= 0 && topk >= 1 && num_experts_on_rank >= 1 && hidden_size >= 0 &&
                     block_k >= 1 && elem_bytes >= 1 && scale_elem_bytes >= 0 && offsets && total_bytes,
                 "fused_moe_prologue_layout: bad arguments");
  const size_t n = (size_t)num_rows * topk;
  const int64_t tpb = prologue_tokens_per_block(num_rows, num_experts_on_rank);
  const size_t blocks_per_seq = (size_t)((num_rows + tpb - 1) / tpb);
  const size_t counts = (size_t)num_experts_on_rank * blocks_per_seq * sizeof(int);
  const size_t sizes[10] = {
      n * sizeof(int),                                     // permuted_row_to_unpermuted_row
      n * sizeof(int),                                     // permuted_token_selected_experts
      n * sizeof(int),                                     // unpermuted_row_to_permuted_row
      counts,                                              // blocked_expert_counts (scratch)
      counts,                                              // blocked_expert_counts_cumsum (scratch)
      (size_t)num_experts_on_rank * num_rows * sizeof(int),  // blocked_row_to_unpermuted_row (scratch)
      (size_t)(num_experts_on_rank + 1) * sizeof(int64_t), // expert_first_token_offset
      n * sizeof(float),                                   // permuted_token_final_scales
      n * (size_t)hidden_size * elem_bytes,                // permuted rows
      n * (size_t)hidden_size / block_k * scale_elem_bytes // permuted scale rows
  };
  size_t off = 0;
  for (int i = 0; i < 10; ++i) {
    offsets[i] = off;
    off += (sizes[i] + 255) & ~(size_t)255;
  }
  *total_bytes = off;
  return B200MOE_OK;
}

extern "C" size_t b200moe_fused_moe_prologue_scratch_bytes(int64_t num_rows, int topk,
                                                           int num_experts_on_rank) {
  const size_t n = (size_t)num_rows * topk;
  const size_t maps = ((n + num_experts_on_rank) * sizeof(int32_t) + 255) & ~(size_t)255;
  return maps + b200moe_sort_workspace_bytes((int64_t)n, num_experts_on_rank);
}

extern "C" int b200moe_fused_moe_prologue(
    const void* input, int elem_bytes, const void* input_scales, int scale_elem_bytes,
    const int64_t* token_selected_experts, const float* token_final_scales, void* workspace,
    size_t workspace_bytes, int64_t num_rows, int64_t hidden_size, int block_k, int topk,
    int ep_rank, int ep_size, int num_experts_on_rank, void* scratch, size_t scratch_bytes,
    b200moe_stream stream) {
  B200_CHECK_ARG(ep_size >= 1 && ep_rank >= 0 && ep_rank < ep_size, "fused_moe_prologue: bad ep_rank/ep_size");
  B200_CHECK_ARG(num_experts_on_rank >= 1 && num_experts_on_rank <= kMaxBuckets,
                 "fused_moe_prologue: at most 1024 experts per rank");
  B200_CHECK_ARG(topk >= 1 && topk <= 32 && num_rows >= 0 && hidden_size >= 1 && block_k >= 1,
                 "fused_moe_prologue: bad sizes");
  B200_CHECK_ARG((int64_t)num_rows * topk < (int64_t)1 << 31, "fused_moe_prologue: too many routed rows");
  B200_CHECK_ARG(workspace && (num_rows == 0 || (input && token_selected_experts)),
                 "fused_moe_prologue: null pointer");
  B200_CHECK_ARG(input_scales == nullptr || scale_elem_bytes >= 1, "fused_moe_prologue: scale element size");
  size_t off[10], total = 0;
  if (int rc = b200moe_fused_moe_prologue_layout(num_rows, topk, num_experts_on_rank, hidden_size, block_k,
                                                 elem_bytes, input_scales ? scale_elem_bytes : 0, off, &total))
    return rc;
  if (workspace_bytes < total)
    return fail(B200MOE_E_WORKSPACE, "fused_moe_prologue: workspace of %zu bytes needed, got %zu", total,
                workspace_bytes);
  const size_t need = b200moe_fused_moe_prologue_scratch_bytes(num_rows, topk, num_experts_on_rank);
  if (scratch == nullptr || scratch_bytes < need)
    return fail(B200MOE_E_WORKSPACE, "fused_moe_prologue: scratch of %zu bytes needed, got %zu", need,
                scratch_bytes);
  const size_t n = (size_t)num_rows * topk;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  int32_t* rows = reinterpret_cast<int32_t*>(scratch);
  int32_t* row_map = rows + num_experts_on_rank;
  const size_t maps = ((n + num_experts_on_rank) * sizeof(int32_t) + 255) & ~(size_t)255;
  cudaStream_t st = as_stream(stream);

  SortParams p;
  p.ids = token_selected_experts; p.ids_dtype = B200MOE_I64; p.map = nullptr;
  p.numel = (int64_t)n; p.id_limit = num_experts_on_rank; p.n_buckets = num_experts_on_rank;
  p.block_size = 1; p.topk = topk;
  p.id_offset = num_experts_on_rank * ep_rank; p.first_match_only = true;
  AlignOut ao = {};
  RemapOut ro = {rows, row_map};
  if (int rc = run_sort<1>(p, ao, ro, reinterpret_cast<unsigned char*>(scratch) + maps, scratch_bytes - maps, st))
    return rc;

  PrologueArgs a;
  a.input = reinterpret_cast<const unsigned char*>(input);
  a.permuted = ws + off[8];
  a.row_bytes = hidden_size * elem_bytes;
  a.scales = reinterpret_cast<const unsigned char*>(input_scales);
  a.permuted_scales = ws + off[9];
  a.scale_row_bytes = input_scales ? (hidden_size / block_k) * scale_elem_bytes : 0;
  a.final_scales = token_final_scales;
  a.permuted_final_scales = reinterpret_cast<float*>(ws + off[7]);
  a.rows_per_expert = rows; a.row_map = row_map;
  a.ids = token_selected_experts; a.id_offset = p.id_offset;
  a.permuted_to_unpermuted = reinterpret_cast<int32_t*>(ws + off[0]);
  a.permuted_experts = reinterpret_cast<int32_t*>(ws + off[1]);
  a.unpermuted_to_permuted = reinterpret_cast<int32_t*>(ws + off[2]);
  a.first_token_offset = reinterpret_cast<int64_t*>(ws + off[6]);
  a.num_tokens = num_rows; a.topk = topk; a.experts = num_experts_on_rank;
  const int64_t want = (int64_t)n < 1 ? 1 : (int64_t)n;
  const int64_t most = (int64_t)sm_count() * 8;
  const int grid = (int)(want < most ? want : most);
  B200_LAUNCHED("prologue_expand_kernel", launch_pdl(n <= kEarlyLaunchRows, prologue_expand_kernel, dim3(grid), dim3(kBlockThreads), 0, st,
      a));
  return B200MOE_OK;
}

extern "C" int b200moe_moe_lora_align_block_size(
    const void* topk_ids, b200moe_dtype ids_dtype, int64_t numel, int topk,
    const int32_t* token_lora_mapping, int num_experts, int block_size, int max_loras,
    int max_num_tokens_padded, int max_num_m_blocks, int32_t* sorted_token_ids,
    int32_t* expert_ids, int32_t* num_tokens_post_pad, const int32_t* adapter_enabled,
    const int32_t* lora_ids, const int32_t* expert_map, b200moe_stream stream) {
  B200_CHECK_ARG(ids_dtype == B200MOE_I32 || ids_dtype == B200MOE_I64 || ids_dtype == B200MOE_U32,
                 "moe_lora_align_block_size: topk_ids must be an integer tensor");
  B200_CHECK_ARG(block_size > 0, "block_size should be greater than 0. ");
  B200_CHECK_ARG(num_experts >= 1 && ((num_experts + 31) / 32) * 32 < 1024,
                 "padded_num_experts must be less than 1024");
  B200_CHECK_ARG(topk >= 1 && numel >= 0 && numel % topk == 0 && max_loras >= 0 &&
                     max_num_tokens_padded >= 0 && max_num_m_blocks >= 0,
                 "moe_lora_align_block_size: bad sizes");
  B200_CHECK_ARG(token_lora_mapping && sorted_token_ids && expert_ids && num_tokens_post_pad &&
                     adapter_enabled && lora_ids && (numel == 0 || topk_ids),
                 "moe_lora_align_block_size: null pointer");
  SortParams p;
  p.ids = topk_ids; p.ids_dtype = ids_dtype; p.map = expert_map;
  p.numel = numel; p.id_limit = num_experts; p.n_buckets = num_experts;
  p.block_size = block_size;
  p.token_lora = token_lora_mapping; p.topk = topk;
  LoraAlignArgs a = {adapter_enabled, lora_ids, max_loras, max_num_tokens_padded, max_num_m_blocks,
                     sorted_token_ids, expert_ids, num_tokens_post_pad};
  const size_t smem = (size_t)(kWarps * num_experts + num_experts + 1 + kWarps) * sizeof(int);
  // lora_ids has max_loras + 1 entries: every adapter slot plus a possible -1
  B200_LAUNCHED("lora_align_kernel", launch_pdl(true, lora_align_kernel,
      dim3(max_loras + 1), dim3(kBlockThreads), smem, as_stream(stream),
      p, a));
  return B200MOE_OK;
}

namespace b200moe {
namespace {
// One block; thread b owns batch b (csrc/moe/moe_align_sum_kernels.cpp:61-130 of the
// reference): exclusive scan of the block-padded counts, then each thread
// writes its batch's token slots and block ids.
__global__ void __launch_bounds__(1024)
batched_align_kernel(const int32_t* __restrict__ counts, int B, int max_tokens, int block,
                     int32_t* __restrict__ sorted_ids, int32_t* __restrict__ block_ids,
                     int32_t* __restrict__ num_post_pad) {
  pdl_trigger();
  pdl_wait();
  __shared__ int warp_sums[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blocks_per_batch = (max_tokens + block - 1) / block;
  const int n_sorted = blocks_per_batch * B * block;
  for (int i = tid; i < n_sorted; i += blockDim.x) sorted_ids[i] = B * max_tokens;
  for (int i = tid; i < n_sorted / block; i += blockDim.x) block_ids[i] = -1;
  const int n = tid < B ? counts[tid] : 0;
  const int ceil_n = (n + block - 1) / block * block;
  int incl = ceil_n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();   // also orders the fills above before the writes below
  if (warp == 0) {
    int w = warp_sums[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += o;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  const int start = incl - ceil_n + (warp > 0 ? warp_sums[warp - 1] : 0);
  if (tid == B - 1) *num_post_pad = start + ceil_n;
  if (tid < B) {
    for (int i = 0; i < n; ++i) sorted_ids[start + i] = tid * max_tokens + i;
    for (int i = 0; i < ceil_n / block; ++i) block_ids[start / block + i] = tid;
  }
}
}  // namespace
}  // namespace b200moe

extern "C" int b200moe_batched_moe_align_block_size(int max_tokens_per_batch, int block_size,
                                                    const int32_t* batch_num_tokens, int num_batches,
                                                    int32_t* sorted_ids, int32_t* batch_ids,
                                                    int32_t* num_tokens_post_pad, b200moe_stream stream) {
  B200_CHECK_ARG(num_batches >= 1 && num_batches <= 1024, "batched_moe_align_block_size: at most 1024 batches");
  B200_CHECK_ARG(block_size >= 1 && max_tokens_per_batch >= 0, "batched_moe_align_block_size: bad sizes");
  B200_CHECK_ARG(batch_num_tokens && sorted_ids && batch_ids && num_tokens_post_pad,
                 "batched_moe_align_block_size: null pointer");
  B200_LAUNCHED("batched_align_kernel", launch_pdl(true, batched_align_kernel, dim3(1), dim3(1024), 0, as_stream(stream),
      batch_num_tokens, num_batches, max_tokens_per_batch, block_size, sorted_ids, batch_ids, num_tokens_post_pad));
  return B200MOE_OK;
}

extern "C" int b200moe_init_expert_map(int32_t* expert_map, int num_local_experts,
                                       int ep_rank, int ep_size, b200moe_stream stream) {
  B200_CHECK_ARG(expert_map, "init_expert_map: null pointer");
  B200_CHECK_ARG(num_local_experts >= 1 && ep_size >= 1 && ep_rank >= 0 && ep_rank < ep_size,
                 "init_expert_map: bad ep_rank/ep_size");
  const int total = num_local_experts * ep_size;
  B200_LAUNCHED("init_expert_map_kernel", launch_pdl(true, init_expert_map_kernel,
      dim3((total + 255) / 256), dim3(256), 0, as_stream(stream),
      expert_map, num_local_experts, ep_rank, total));
  return B200MOE_OK;
}

extern "C" int b200moe_remap_hidden_states(
    const void* hidden, const void* scales, void* remapped, void* remapped_scales,
    const int32_t* expert_map, int32_t* rows_per_expert, int32_t* row_map,
    const void* topk_ids, b200moe_dtype ids_dtype, int64_t num_rows, int hidden_size,
    int elem_bytes, int scale_cols, int scale_elem_bytes, int topk, int total_experts,
    int local_experts, void* workspace, size_t workspace_bytes, b200moe_stream stream) {
  B200_CHECK_ARG(elem_bytes == 1 || elem_bytes == 2 || elem_bytes == 4,
                 "Unsupported data type in hidden_states");
  B200_CHECK_ARG((scales == nullptr) == (remapped_scales == nullptr),
                 "if hidden_states_scales is provided, remapped_hidden_states_scales "
                 "must also be provided");
  B200_CHECK_ARG(((int64_t)hidden_size * elem_bytes) % 16 == 0,
                 "hidden_size must be divisible by ElemsPerItem");
  B200_CHECK_ARG(num_rows >= 0, "remap_hidden_states: negative num_rows");
  SortParams p;
  if (int rc = remap_params(p, expert_map, rows_per_expert, row_map, topk_ids, ids_dtype, num_rows, topk,
                            total_experts, local_experts)) return rc;
  B200_CHECK_ARG(num_rows == 0 || (hidden && remapped), "remap_hidden_states: null pointer");
  B200_CHECK_ARG(((uintptr_t)hidden & 15) == 0 && ((uintptr_t)remapped & 15) == 0,
                 "remap_hidden_states: buffers must be 16-byte aligned");
  RowJob job = {};
  job.src = hidden; job.dst = remapped; job.src_s = scales; job.dst_s = remapped_scales;
  job.row_bytes = hidden_size * elem_bytes; job.scale_row_bytes = scale_cols * scale_elem_bytes; job.K = topk;
  return remap_rows<uint8_t, kRowCopy>(p, job, rows_per_expert, row_map, num_rows, workspace, workspace_bytes,
                                       as_stream(stream));
}

extern "C" int b200moe_remap_quant_fp8(
    const void* hidden, b200moe_dtype dtype, void* remapped_q, float* remapped_scales,
    const int32_t* expert_map, int32_t* rows_per_expert, int32_t* row_map,
    const void* topk_ids, b200moe_dtype ids_dtype, int64_t num_rows, int hidden_size,
    int topk, int total_experts, int local_experts, void* workspace,
    size_t workspace_bytes, b200moe_stream stream) {
  B200_CHECK_ARG(dtype == B200MOE_BF16 || dtype == B200MOE_F16,
                 "remap_quant_fp8: activations must be bfloat16 or float16");
  B200_CHECK_ARG(hidden_size % 128 == 0, "remap_quant_fp8: hidden_size must be a multiple of 128");
  SortParams p;
  if (int rc = remap_params(p, expert_map, rows_per_expert, row_map, topk_ids, ids_dtype, num_rows, topk,
                            total_experts, local_experts)) return rc;
  B200_CHECK_ARG(num_rows == 0 || (hidden && remapped_q && remapped_scales), "remap_quant_fp8: null pointer");
  B200_CHECK_ARG(((uintptr_t)hidden & 15) == 0 && ((uintptr_t)remapped_q & 7) == 0,
                 "remap_quant_fp8: buffers must be 16-byte aligned");
  RowJob job = {};
  job.src = hidden; job.dst = remapped_q; job.dst_s = remapped_scales; job.H = hidden_size; job.K = topk;
  auto run = dtype == B200MOE_BF16 ? remap_rows<__nv_bfloat16, kRowFp8> : remap_rows<__half, kRowFp8>;
  return run(p, job, rows_per_expert, row_map, num_rows, workspace, workspace_bytes, as_stream(stream));
}

extern "C" int b200moe_remap_quant_mxfp8(
    const void* hidden, b200moe_dtype dtype, void* remapped_q, void* remapped_scales, int planes, int block_sums,
    const int32_t* expert_map, int32_t* rows_per_expert, int32_t* row_map,
    const void* topk_ids, b200moe_dtype ids_dtype, int64_t num_rows, int hidden_size,
    int topk, int total_experts, int local_experts, void* workspace,
    size_t workspace_bytes, b200moe_stream stream) {
  B200_CHECK_ARG(dtype == B200MOE_BF16 || dtype == B200MOE_F16,
                 "remap_quant_mxfp8: activations must be bfloat16 or float16");
  B200_CHECK_ARG(hidden_size % 32 == 0, "remap_quant_mxfp8: hidden_size must be a multiple of 32");
  const bool evens_first = planes > B200MOE_PLANES_EVENS_FIRST && block_sums;
  if (evens_first) planes -= B200MOE_PLANES_EVENS_FIRST;
  B200_CHECK_ARG(planes >= 1 && planes <= 3, "remap_quant_mxfp8: one to three planes");
  SortParams p;
  if (int rc = remap_params(p, expert_map, rows_per_expert, row_map, topk_ids, ids_dtype, num_rows, topk,
                            total_experts, local_experts)) return rc;
  B200_CHECK_ARG(num_rows == 0 || (hidden && remapped_q && remapped_scales), "remap_quant_mxfp8: null pointer");
  B200_CHECK_ARG(((uintptr_t)hidden & 15) == 0 && ((uintptr_t)remapped_q & 7) == 0,
                 "remap_quant_mxfp8: buffers must be 16-byte aligned");
  RowJob job = {};
  job.src = hidden; job.dst = remapped_q; job.dst_s = remapped_scales; job.H = hidden_size; job.K = topk;
  job.rows = num_rows * topk; job.planes = planes; job.sums = block_sums; job.evens_first = evens_first;
  auto run = dtype == B200MOE_BF16 ? remap_rows<__nv_bfloat16, kRowMx> : remap_rows<__half, kRowMx>;
  return run(p, job, rows_per_expert, row_map, num_rows, workspace, workspace_bytes, as_stream(stream));
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the align op.
//
// Some hosts of this library cannot hand over scratch memory: a cgo / JNI /
// ctypes binding usually receives only the input and output buffers that its
// serving framework allocated and owns no device allocator of its own, and a
// latency-critical serving loop must not call cudaMalloc on its hot path
// (the call serialises the whole device and fails once the framework's pool
// has claimed all memory).  For them the histogram exchange buffer of the
// multi-block sort lives in a fixed array inside the library image.  Every GPU
// that loads the library holds these kNoAllocScratchBytes until the process
// exits.
// ---------------------------------------------------------------------------
namespace b200moe {
namespace {
constexpr size_t kNoAllocScratchBytes = 1u << 20;  // 1 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// device address of the array per device ordinal; written once, read by any thread
std::atomic<void*> g_noalloc_ptr[kMaxDevices];
}  // namespace
}  // namespace b200moe

extern "C" size_t b200moe_noalloc_scratch_capacity(void) { return b200moe::kNoAllocScratchBytes; }

extern "C" int b200moe_moe_align_block_size_noalloc(
    const void* topk_ids, b200moe_dtype ids_dtype, int64_t numel, int num_experts, int block_size,
    int32_t* sorted_token_ids, int64_t sorted_len, int32_t* expert_ids, int64_t expert_ids_len,
    int32_t* num_tokens_post_pad, const int32_t* expert_map, b200moe_stream stream) {
  B200_CHECK_ARG(num_experts >= 1 && numel >= 0, "moe_align_block_size_noalloc: bad sizes");
  const size_t need = b200moe_sort_workspace_bytes(numel, num_experts);
  if (need > kNoAllocScratchBytes)
    return fail(B200MOE_E_WORKSPACE,
                "moe_align_block_size_noalloc: %lld slots over %d experts need %zu bytes of scratch, "
                "the built-in buffer holds %zu; use b200moe_moe_align_block_size with a workspace",
                (long long)numel, num_experts, need, (size_t)kNoAllocScratchBytes);
  int dev = -1;
  B200_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices)
    return fail(B200MOE_E_UNSUPPORTED, "moe_align_block_size_noalloc: device ordinal %d out of range", dev);
  void* scratch = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) {
    // In host code `g_noalloc_scratch` is only a handle for the symbol, not a
    // device address: resolve it once per device, with that device current.
    // (Two threads that race here both look up the same address.)
    B200_CUDA_OK(cudaGetSymbolAddress(&scratch, g_noalloc_scratch));
    if (scratch == nullptr) return fail(B200MOE_E_CUDA, "cudaGetSymbolAddress returned a null address");
    g_noalloc_ptr[dev].store(scratch, std::memory_order_release);
  }
  // Nothing in the buffer has to start at zero: the count pass overwrites every
  // histogram cell it later reads and the scan pass writes the sizes.
  return b200moe_moe_align_block_size(topk_ids, ids_dtype, numel, num_experts, block_size,
                                      sorted_token_ids, sorted_len, expert_ids, expert_ids_len,
                                      num_tokens_post_pad, expert_map, scratch,
                                      kNoAllocScratchBytes, stream);
}
