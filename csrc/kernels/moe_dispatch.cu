// MoE token dispatch / combine as an active-message all-to-all over peer
// memory. The reference has only point-to-point active messages
// (ucx_context/ucx_connection.cpp:353-374: one ucp_am_send_nbx per message);
// here every routed (token, k) row is one active message whose 16-byte header
// {src_token, k_slot | local_expert, gate weight, src_rank} and payload row are
// stored by the sending GPU straight into the destination GPU's receive arena.
//
// Receive arena of a rank: `world` regions (one per source rank) of `capacity`
// rows. Inside a region rows are grouped by local expert, so an expert GEMM can
// consume them as contiguous groups; per-(src, expert) counts travel with the
// arrival flag.
//
// flags block of a rank (uint64 words):
//   [0,W)        arrival sequence written by source rank s
//   [W,2W)       number of rows source rank s sent here
//   [2W,3W)      "expert output ready" sequence written by expert rank e
//   [3W,3W+W*EPR) rows per (source rank, local expert)
//
// Combine is a pull: the source rank reads its rows back from the expert ranks'
// arenas with peer loads and accumulates sum_k w_k * y_k in fp32 registers, so
// the weighted combine is fused into the receive and no intermediate buffer
// exists.
#include <algorithm>

#include "eux_bulk.cuh"
#include "eux_device.cuh"

namespace eux {

constexpr int kMoeThreads = 512;
constexpr int kMaxWorld = 16;
constexpr int kMaxExperts = 4096;

__host__ __device__ __forceinline__ size_t moe_row_bytes(int hidden, int fp8) {
  // fp8 rows: values, then one fp32 scale per 128 values, padded to whole 128-byte lines so that
  // a warp's 512-byte stores into a row never straddle a line (a straddling store costs an extra
  // NVLink packet)
  return fp8 ? (((size_t)hidden + (size_t)(hidden / 128) * 4 + 127) / 128) * 128 : (size_t)hidden * 2;
}

// ---- dispatch: routing, then the transfer -------------------------------------------------------------------
// Every CTA owns a run of tokens and has to know where its rows go: the rows of the experts before each one on the same
// rank, and the rows of the same expert from tokens of the CTAs before it.
//   * Few entries (kRouteSelf): every CTA reads all of them (out of L2) and counts for itself. No CTA waits for another
//     one, so nothing depends on how many of them run at a time.
//   * More: moe_count_kernel in front of the dispatch adds the counts up and gives every entry its place inside its
//     expert's group; the end of that launch is the barrier.
// (A grid barrier inside one cooperative launch needed all CTAs resident at once, which a kernel of another stream can
// prevent for as long as it waits for this dispatch, and a barrier that ran out left its counters behind. Exchange of 128
// tokens of 7168, fp8: 24.8 us with the barrier, 24.1 now; 4096 tokens, bf16: 207.5 and 208.5, 219 with one routing CTA.)
// counters layout: [0,W) unused | [W,W+E) rows per expert | [W+E] done CTAs; zero between launches
__device__ __forceinline__ void moe_ld_v8(const void* p, uint32_t (&v)[8]) {
  asm volatile("ld.global.cg.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(p));
}
__device__ __forceinline__ void moe_st_v8(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
struct MoeRouting {
  int* local;  // [E] rows of this CTA per expert; then rows of all experts before e, whatever their rank
  int* base;   // [E] where this CTA's rows start inside the destination's region
  int* total;  // [E] rows of all CTAs per expert
};
// The tokens [t0, t1) of CTA `b` of `grid`: all shares within one token of one another.
__device__ __forceinline__ int moe_first_token(const eux_moe_desc& d, int b, int grid) {
  return (int)((int64_t)d.n_tokens * b / grid);
}

// Exclusive scan of v over the CTA; `sums`: one int per warp.
__device__ __forceinline__ int cta_exclusive_scan(int v, int* sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sums[warp] = x;
  __syncthreads();
  int before = 0;
#pragma unroll
  for (int w = 0; w < kMoeThreads / 32; ++w) before += w < warp ? sums[w] : 0;
  __syncthreads();
  return before + x - v;
}

constexpr int kRouteSelf = 4096;

// The place of every entry inside its expert's group: a CTA takes a run of entries, ranks them, and adds its counts to the
// global ones, which returns where its rows start. (The additions go out in the order of the experts, a warp's 32 in one
// line; where each expert's first entry made it, 4096 x 7168 took 4 us more.)
__global__ void __launch_bounds__(kMoeThreads) moe_count_kernel(eux_moe_desc d) {
  extern __shared__ int moe_sm[];
  int* const local = moe_sm;
  int* const base = moe_sm + d.n_experts;
  const int E = d.n_experts;
  const int64_t n = (int64_t)d.n_tokens * d.topk;
  const int64_t i0 = n * blockIdx.x / gridDim.x, i1 = n * (blockIdx.x + 1) / gridDim.x;
  const int64_t first = i0 + threadIdx.x;  // all of a thread's entries up to 512 per SM: stays in registers
  int e0 = first < i1 ? __ldg(d.topk_idx + first) : -1, rank0 = -1;
  if (e0 >= E) e0 = -1;
  for (int e = threadIdx.x; e < E; e += blockDim.x) local[e] = 0;
  __syncthreads();
  if (e0 >= 0) rank0 = atomicAdd(&local[e0], 1);
  for (int64_t i = first + blockDim.x; i < i1; i += blockDim.x) {
    const int e = __ldg(d.topk_idx + i);
    d.slot_of[i] = e >= 0 && e < E ? atomicAdd(&local[e], 1) : -1;  // the rank inside this CTA, for now
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) base[e] = local[e] ? atomicAdd(d.counters + d.world + e, local[e]) : 0;
  __syncthreads();
  if (first < i1) d.slot_of[first] = e0 >= 0 ? base[e0] + rank0 : -1;
  for (int64_t i = first + blockDim.x; i < i1; i += blockDim.x) {
    const int rank = d.slot_of[i];
    if (rank >= 0) d.slot_of[i] = rank + base[__ldg(d.topk_idx + i)];
  }
}

// The slots of tokens [t0, t1). `counted`: moe_count_kernel has run. What a thread knows of its entries stays in its
// registers until the slots are known: a trip to memory more costs as much as all of the arithmetic.
__device__ __forceinline__ void moe_route(const eux_moe_desc& d, const MoeRouting& r, int t0, int t1, bool counted) {
  constexpr int PER = kRouteSelf / kMoeThreads;
  const int W = d.world, E = d.n_experts, EPR = E / W, K = d.topk;
  const int64_t lo = (int64_t)t0 * K, hi = (int64_t)t1 * K;
  const int n = counted ? 0 : d.n_tokens * K;  // entries that this CTA counts: at most kRouteSelf
  __shared__ int s_sums[kMoeThreads / 32];
  int expert[PER], rank[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int i = (int)threadIdx.x + j * kMoeThreads;
    expert[j] = i < n ? __ldg(d.topk_idx + i) : -1;
  }
  const int64_t first = lo + threadIdx.x;
  if (counted && first < hi) expert[0] = __ldg(d.topk_idx + first), rank[0] = d.slot_of[first];
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    r.local[e] = 0, r.base[e] = 0;
    r.total[e] = counted ? __ldcg(d.counters + W + e) : 0;
  }
  __syncthreads();
  if (!counted) {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int i = (int)threadIdx.x + j * kMoeThreads, e = expert[j];
      if (e < 0 || e >= E) expert[j] = -1;
      else if (i >= lo && i < hi) rank[j] = atomicAdd(&r.local[e], 1);
      else atomicAdd(i < lo ? &r.base[e] : &r.total[e], 1);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) r.total[e] += r.base[e] + r.local[e];
    __syncthreads();
  }
  // every thread takes a run of consecutive experts
  const int run = (E + (int)blockDim.x - 1) / (int)blockDim.x;
  const int e0 = (int)threadIdx.x * run, e1 = min(e0 + run, E);
  int mine = 0;
  for (int e = e0; e < e1; ++e) mine += r.total[e];
  int sum = cta_exclusive_scan(mine, s_sums);
  for (int e = e0; e < e1; ++e) {
    r.local[e] = sum;
    sum += r.total[e];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) r.base[e] += r.local[e] - r.local[(e / EPR) * EPR];
  __syncthreads();
  auto place = [&](int64_t i, int e, int in_group) {
    const int slot = e >= 0 ? r.base[e] + in_group : -1;
    d.slot_of[i] = slot < d.capacity ? slot : -1;
  };
  if (counted) {
    if (first < hi) place(first, rank[0] >= 0 ? expert[0] : -1, rank[0]);
    for (int64_t i = first + blockDim.x; i < hi; i += blockDim.x) {
      const int in_group = d.slot_of[i];
      place(i, in_group >= 0 ? __ldg(d.topk_idx + i) : -1, in_group);
    }
  } else {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int i = (int)threadIdx.x + j * kMoeThreads;
      if (i >= lo && i < hi) place(i, expert[j], rank[j]);
    }
  }
  __syncthreads();
}

// Every CTA knows all counts after its routing: the first one sends them, in front of its rows.
__device__ __forceinline__ void moe_send_counts(const eux_moe_desc& d, const MoeRouting& r, uint64_t* const* flags) {
  if (blockIdx.x != 0) return;
  const int W = d.world, E = d.n_experts, EPR = E / W;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const int dst = e / EPR, le = e - dst * EPR;
    flags[dst][3 * W + d.rank * EPR + le] = (uint64_t)r.total[e];
  }
  for (int dst = threadIdx.x; dst < W; dst += blockDim.x) {
    const int last = dst * EPR + EPR - 1;
    const int rows = r.local[last] - r.local[dst * EPR] + r.total[last];
    if (rows > d.capacity) set_status(d.status, EUX_ST_OVERFLOW, 10);
    flags[dst][W + d.rank] = (uint64_t)(rows < d.capacity ? rows : d.capacity);
  }
}
// The last CTA sends the arrival flags and leaves the counters at zero. A CTA's fence between its rows and its count is for
// this GPU, where the last CTA sees the counts; that one's fence for everyone stands between them and the flags and covers the
// rows of all CTAs. (System-scope fences queue up at 31 ns each: with one per CTA a dispatch of 128 fp8 tokens of 7168 took
// 12.4 us, 9.0 so, graph replays. With counts and flags both sent here, behind a release each, an exchange of 16 tokens of
// 4096 took 20.4 us, 18.8 without.) Nobody is told of an exchange of which a CTA gave up, as a transfer or a GEMM tells
// nobody: the receivers' own waits run out. Such a CTA sets the top bit of the count before it adds itself.
__device__ __forceinline__ void moe_publish(const eux_moe_desc& d, uint64_t* const* flags, bool ok = true) {
  __syncthreads();
  __shared__ int s_last;
  const int W = d.world, E = d.n_experts;
  if (threadIdx.x == 0) {
    uint32_t* const done = reinterpret_cast<uint32_t*>(d.counters + W + E);
    fence_gpu();
    if (!ok) atomicOr(done, 0x80000000u);
    const uint32_t old = atomicAdd(done, 1u);
    s_last = ((old & 0x7fffffffu) == gridDim.x - 1);
    if (s_last && !(old & 0x80000000u)) {
      fence_sys();
      for (int dst = 0; dst < W; ++dst) st_relaxed_sys(flags[dst] + d.rank, d.seq);
    }
  }
  __syncthreads();
  if (!s_last) return;
  for (int e = threadIdx.x; e < E; e += blockDim.x) d.counters[W + e] = 0;
  if (threadIdx.x == 0) d.counters[W + E] = 0;
}

// The routing entries of a token: lane k (< topk) owns slot k.
struct MoeEntry {
  int dst = -1, slot = -1, expert = -1;
  float w = 0.f;
  __device__ __forceinline__ MoeEntry(const eux_moe_desc& d, int t, int lane, int EPR) {
    if (lane < d.topk) {
      const int64_t i = (int64_t)t * d.topk + lane;
      slot = d.slot_of[i];
      if (slot >= 0) {
        expert = __ldg(d.topk_idx + i);
        dst = expert / EPR;
        w = __ldg(d.topk_w + i);
      }
    }
  }
  __device__ __forceinline__ size_t row(const eux_moe_desc& d) const { return (size_t)d.rank * d.capacity + slot; }
  __device__ __forceinline__ unsigned char* arena_row(const eux_moe_desc& d, size_t row_bytes) const {
    return slot < 0 ? nullptr : reinterpret_cast<unsigned char*>(d.arena_peer[dst]) + row(d) * row_bytes;
  }
  __device__ __forceinline__ void store_header(const eux_moe_desc& d, int t, int lane, int EPR) const {
    if (slot < 0) return;
    uint4 h;
    h.x = (uint32_t)t;
    h.y = (uint32_t)lane | ((uint32_t)(expert - dst * EPR) << 16);
    h.z = __float_as_uint(w);
    h.w = (uint32_t)d.rank;
    st_u4(reinterpret_cast<uint4*>(d.meta_peer[dst]) + row(d), h);
  }
};
__device__ __forceinline__ unsigned char* shfl_ptr(unsigned char* p, int src) {
  return (unsigned char*)__shfl_sync(0xffffffffu, (unsigned long long)p, src);
}

// ---- dispatch, bf16 rows ----------------------------------------------------
// Work unit = (token, 128 consecutive 16-byte chunks): a warp loads 4 chunks per
// lane once and stores them to each of the token's top-k destinations.
__global__ void __launch_bounds__(kMoeThreads) moe_dispatch_bf16_kernel(eux_moe_desc d, int counted) {
  extern __shared__ int moe_sm[];
  const MoeRouting r{moe_sm, moe_sm + d.n_experts, moe_sm + 2 * d.n_experts};
  const int t0 = moe_first_token(d, blockIdx.x, gridDim.x), t1 = moe_first_token(d, blockIdx.x + 1, gridDim.x);
  __shared__ uint64_t* flags[kMaxWorld];
  if ((int)threadIdx.x < d.world) flags[threadIdx.x] = d.flag_peer[threadIdx.x];
  moe_route(d, r, t0, t1, counted != 0);
  moe_send_counts(d, r, flags);
  const int EPR = d.n_experts / d.world, K = d.topk;
  const int chunks = d.hidden / 8;  // uint4 per row
  const int upr = (chunks + 127) / 128;
  const size_t row_bytes = (size_t)d.hidden * 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int units = (t1 - t0) * upr;
  for (int u = warp; u < units; u += nwarps) {
    const int tl = u / upr, t = t0 + tl, part = u - tl * upr;
    const uint4* src = reinterpret_cast<const uint4*>(d.x) + (size_t)t * chunks;
    const int c0 = part * 128 + lane;
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int c = c0 + 32 * j;
      if (c < chunks) v[j] = ld_stream_u4(src + c);
    }
    const MoeEntry my(d, t, lane, EPR);
    unsigned char* const my_out = my.arena_row(d, row_bytes);
    for (int k = 0; k < K; ++k) {
      uint4* out = reinterpret_cast<uint4*>(shfl_ptr(my_out, k));
      if (!out) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int c = c0 + 32 * j;
        if (c < chunks) st_u4(out + c, v[j]);
      }
    }
    if (part == 0) my.store_header(d, t, lane, EPR);
  }
  moe_publish(d, flags);
}

// ---- dispatch, e4m3 rows with one fp32 scale per 128 elements ---------------
// Work unit = (token, 1024 elements): a lane holds 32 elements, four lanes share a scale, and a warp's store into a row
// is 1 KiB. The scales of a batch of tokens are collected in shared memory and leave as one coalesced store per row:
// across NVLink a 4-byte store costs a packet of its own. (One warp per token row, which kept them in registers, left a
// decode batch with a warp per token: 128 tokens of 7168 took 34 us, 20 now. 32-byte stores: with two of 16 bytes per
// lane 4096 tokens took 89 us, 78 now.)
constexpr int kMoeScaleFloats = 4096;  // per buffer; two buffers, so that one barrier per batch is enough
// Tokens per batch; none for rows whose scales do not fit a buffer: those leave one by one.
__host__ __device__ __forceinline__ int moe_scale_batch(int hidden) {
  const int b = kMoeScaleFloats / (hidden / 128);
  return b > 16 ? 16 : b;
}
__host__ __device__ __forceinline__ int moe_scale_stride(int hidden) { return moe_scale_batch(hidden) * (hidden / 128); }

__global__ void __launch_bounds__(kMoeThreads, 2) moe_dispatch_fp8_kernel(eux_moe_desc d, int counted) {
  extern __shared__ int moe_sm[];
  const MoeRouting r{moe_sm, moe_sm + d.n_experts, moe_sm + 2 * d.n_experts};
  float* const scales = reinterpret_cast<float*>(moe_sm + 3 * d.n_experts);
  const int t0 = moe_first_token(d, blockIdx.x, gridDim.x), t1 = moe_first_token(d, blockIdx.x + 1, gridDim.x);
  __shared__ uint64_t* flags[kMaxWorld];
  if ((int)threadIdx.x < d.world) flags[threadIdx.x] = d.flag_peer[threadIdx.x];
  moe_route(d, r, t0, t1, counted != 0);
  moe_send_counts(d, r, flags);
  const int EPR = d.n_experts / d.world, K = d.topk;
  const int upr = (d.hidden + 1023) / 1024;
  const int ngroups = d.hidden / 128;
  const size_t row_bytes = moe_row_bytes(d.hidden, 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int stride = moe_scale_stride(d.hidden);
  const bool collect = stride > 0;
  const int batch = collect ? moe_scale_batch(d.hidden) : 1;
  int buf = 0;
  for (int tb = t0; tb < t1; tb += batch, buf ^= 1) {
    const int nt = min(batch, t1 - tb);
    float* const sc = scales + buf * stride;
    for (int u = warp; u < nt * upr; u += nwarps) {
      const int tl = u / upr, t = tb + tl, part = u - tl * upr;
      const int e0 = part * 1024 + lane * 32;  // first element of this lane
      const bool in = e0 < d.hidden;
      uint4 raw[4];
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(d.x) + (size_t)t * d.hidden + e0);
#pragma unroll
      for (int j = 0; j < 4; ++j) raw[j] = in ? ld_stream_u4(src + j) : make_uint4(0, 0, 0, 0);
      const MoeEntry my(d, t, lane, EPR);
      unsigned char* const my_out = my.arena_row(d, row_bytes);
      const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(raw);
      float amax = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float2 x = __bfloat1622float2(pairs[j]);
        amax = fmaxf(amax, fmaxf(fabsf(x.x), fabsf(x.y)));
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      const float scale = fmaxf(amax, 1e-10f) * (1.0f / 448.0f);
      const float inv = 1.0f / scale;
      uint32_t w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 a = __bfloat1622float2(pairs[2 * j]), b = __bfloat1622float2(pairs[2 * j + 1]);
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a.x * inv, a.y * inv), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(b.x * inv, b.y * inv), __NV_SATFINITE, __NV_E4M3);
        w[j] = lo | (hi << 16);
      }
      const bool keeps = in && (lane & 3) == 0;
      if (keeps && collect) sc[tl * ngroups + (e0 >> 7)] = scale;
      for (int k = 0; k < K; ++k) {
        unsigned char* out = shfl_ptr(my_out, k);
        if (!out || !in) continue;
        if (((uintptr_t)out & 31u) == 0) {
          moe_st_v8(out + e0, w);
        } else {  // an arena has to start on 16 bytes only
          st_u4(out + e0, make_uint4(w[0], w[1], w[2], w[3]));
          st_u4(out + e0 + 16, make_uint4(w[4], w[5], w[6], w[7]));
        }
        if (keeps && !collect) reinterpret_cast<float*>(out + d.hidden)[e0 >> 7] = scale;
      }
      if (part == 0) my.store_header(d, t, lane, EPR);
    }
    if (!collect) continue;
    __syncthreads();
    for (int u = warp; u < nt * K; u += nwarps) {
      const int tl = u / K, k = u - tl * K;
      const MoeEntry my(d, tb + tl, lane, EPR);
      unsigned char* out = shfl_ptr(my.arena_row(d, row_bytes), k);
      if (!out) continue;
      float* so = reinterpret_cast<float*>(out + d.hidden);
      for (int g = lane; g < ngroups; g += 32) so[g] = sc[tl * ngroups + g];
    }
  }
  moe_publish(d, flags);
}

// ---- dispatch, e4m3 rows, two tokens per CTA and more: row images in shared memory, moved by bulk copies -------------------
// Twelve warps quantise units of (token, 1024 elements) into images of whole rows (values, scales, padding) in a ring of
// slots; four warps send the finished images to their top-k rows, a bulk copy each. The kernel above has what its registers
// hold in flight and a barrier in front of the scales: 4096 tokens of 7168 keep the DRAM at 43 % of its peak (ncu, part of
// the rows still in L2 at the end). Dispatches in a loop, above and here: 4096 x 7168 75.1 and 65.0 us, 4096 x 2048 32.6 and 25.9, 1024 x 7168 25.7 and 23.0, 300 x 7168 16.0
// and 15.9, 128 x 7168 13.3 and 14.1 (with one sending warp 65.4, 34.0, 22.8, 15.8: its look-ups are a trip to L2 per token).
// Token tl of the CTA: slot tl % slots, barriers tl % 32, sending warp tl % 4. The number of slots is a multiple of four
// too, so everything about a token belongs to one of four classes, each of which one warp sends in order. A quantising warp
// has a unit of token tl - 12 as well (same class), for which it saw token tl - 12 - slots sent: no wait can meet a barrier
// that is a whole ring behind or ahead.
constexpr int kMoeBars = 32;
constexpr int kMoeSenders = 4;
constexpr int kMoeMinSlots = 8;
constexpr size_t kMoeImageBytes = 112 * 1024;
__host__ __device__ __forceinline__ int moe_image_slots(int hidden) {  // 16, 12 or 8; 0: the rows are too wide
  const int n = (int)(kMoeImageBytes / moe_row_bytes(hidden, 1)) / 4 * 4;
  return n > 16 ? 16 : n < kMoeMinSlots ? 0 : n;
}
// mbar_wait for waits that last microseconds: the clock is read after every failing try (one takes 4 us).
__device__ __forceinline__ bool moe_wait(uint32_t bar, uint32_t parity, volatile int* abort, uint64_t timeout_ns) {
  if (mbar_try(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 0; it < 0x7fffffffu; ++it) {
    if (mbar_try(bar, parity)) return true;
    if (*abort) return false;
    if (globaltimer_ns() - t0 > (timeout_ns ? timeout_ns : 2000000000ull)) break;
  }
  *abort = 1;
  return false;
}
// 16 bf16 values (32 bytes) as e4m3 with the given 1 / scale
__device__ __forceinline__ uint4 moe_quantize16(const uint32_t (&raw)[8], float inv) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[2 * j]));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[2 * j + 1]));
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a.x * inv, a.y * inv), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(b.x * inv, b.y * inv), __NV_SATFINITE, __NV_E4M3);
    w[j] = lo | (hi << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void __launch_bounds__(kMoeThreads) moe_dispatch_fp8_bulk_kernel(eux_moe_desc d, int counted, int slots) {
  extern __shared__ __align__(128) unsigned char moe_image_sm[];
  __shared__ uint64_t bars[2 * kMoeBars];
  __shared__ uint64_t* flags[kMaxWorld];
  __shared__ unsigned char* arenas[kMaxWorld];
  __shared__ uint4* metas[kMaxWorld];
  __shared__ int s_abort;
  const size_t row_bytes = moe_row_bytes(d.hidden, 1);
  unsigned char* const ring = reinterpret_cast<unsigned char*>(((uintptr_t)moe_image_sm + 127) & ~(uintptr_t)127);
  int* const tables = reinterpret_cast<int*>(ring + (size_t)slots * row_bytes);
  const MoeRouting r{tables, tables + d.n_experts, tables + 2 * d.n_experts};
  const int t0 = moe_first_token(d, blockIdx.x, gridDim.x), t1 = moe_first_token(d, blockIdx.x + 1, gridDim.x);
  const int EPR = d.n_experts / d.world;
  const int upr = (d.hidden + 1023) / 1024;
  const int ngroups = d.hidden / 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWorkers = kMoeThreads / 32 - kMoeSenders;
  static_assert(kWorkers % kMoeSenders == 0 && kMoeBars % kMoeSenders == 0, "classes of tokens");
  const uint32_t ring0 = smem_u32(ring), bar0 = smem_u32(bars);
  auto full_bar = [&](int tl) { return bar0 + 8u * (tl % kMoeBars); };
  auto empty_bar = [&](int tl) { return bar0 + 8u * (kMoeBars + tl % kMoeBars); };
  auto phase = [](int tl) { return (uint32_t)(tl / kMoeBars) & 1u; };
  volatile int* abort = &s_abort;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kMoeBars; ++i) {
      mbar_init(full_bar(i), (uint32_t)upr);
      mbar_init(empty_bar(i), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if ((int)threadIdx.x < d.world) {
    flags[threadIdx.x] = d.flag_peer[threadIdx.x];
    arenas[threadIdx.x] = reinterpret_cast<unsigned char*>(d.arena_peer[threadIdx.x]);
    metas[threadIdx.x] = reinterpret_cast<uint4*>(d.meta_peer[threadIdx.x]);
  }
  for (int s = warp; s < slots; s += kMoeThreads / 32)  // the padding behind the scales
    for (int b = d.hidden + ngroups * 4 + lane * 4; b < (int)row_bytes; b += 128) *reinterpret_cast<uint32_t*>(ring + s * row_bytes + b) = 0;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  moe_route(d, r, t0, t1, counted != 0);
  moe_send_counts(d, r, flags);
  const int units = (t1 - t0) * upr;
  if (warp < kWorkers) {
    // a lane has 16 elements of either half of the unit: 32-byte loads, conflict-free stores
    uint32_t v[2][8];
    auto load = [&](int u) {
      const int tl = u / upr, e0 = (u - tl * upr) * 1024 + lane * 16;
      const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(d.x) + (size_t)(t0 + tl) * d.hidden + e0;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (e0 + h * 512 < d.hidden) {
          const uint4 a = ld_stream_u4(src + h * 512), b = ld_stream_u4(src + h * 512 + 8);
          v[h][0] = a.x, v[h][1] = a.y, v[h][2] = a.z, v[h][3] = a.w, v[h][4] = b.x, v[h][5] = b.y, v[h][6] = b.z, v[h][7] = b.w;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[h][j] = 0;
        }
    };
    if (warp < units) load(warp);
    for (int u = warp; u < units; u += kWorkers) {
      const int tl = u / upr, part = u - tl * upr, s = tl % slots;
      uint4 q[2];
      float scale[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v[h][j]));
          amax = fmaxf(amax, fmaxf(fabsf(x.x), fabsf(x.y)));
        }
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
        scale[h] = fmaxf(amax, 1e-10f) * (1.0f / 448.0f);
        q[h] = moe_quantize16(v[h], 1.0f / scale[h]);
      }
      if (u + kWorkers < units) load(u + kWorkers);
      if (tl >= slots && __any_sync(0xffffffffu, !moe_wait(empty_bar(tl - slots), phase(tl - slots), abort, d.wait_timeout_ns))) break;
      unsigned char* const image = ring + (size_t)s * row_bytes;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e0 = part * 1024 + h * 512 + lane * 16;
        if (e0 < d.hidden) {
          *reinterpret_cast<uint4*>(image + e0) = q[h];
          if ((lane & 7) == 0) reinterpret_cast<float*>(image + d.hidden)[e0 >> 7] = scale[h];
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar(tl));
    }
  } else {
    // lane k owns row k; the routing entries of the next token are on their way while this one's image is waited for
    int slot = -1, expert = 0;
    float w = 0.f;
    auto fetch = [&](int t) {
      slot = -1;
      if (lane < d.topk) {
        const int64_t i = (int64_t)t * d.topk + lane;
        slot = d.slot_of[i], expert = __ldg(d.topk_idx + i), w = __ldg(d.topk_w + i);
      }
    };
    const int first = warp - kWorkers;
    if (t0 + first < t1) fetch(t0 + first);
    for (int tl = first; tl < t1 - t0; tl += kMoeSenders) {
      const int t = t0 + tl, s = tl % slots;
      unsigned char* out = nullptr;
      if (slot >= 0) {
        const int dst = expert / EPR;
        const size_t row = (size_t)d.rank * d.capacity + slot;
        out = arenas[dst] + row * row_bytes;
        st_u4(metas[dst] + row, make_uint4((uint32_t)t, (uint32_t)lane | ((uint32_t)(expert - dst * EPR) << 16), __float_as_uint(w), (uint32_t)d.rank));
      }
      if (tl + kMoeSenders < t1 - t0) fetch(t + kMoeSenders);
      if (__any_sync(0xffffffffu, !moe_wait(full_bar(tl), phase(tl), abort, d.wait_timeout_ns))) break;
      if (out) bulk_s2g(out, ring0 + (uint32_t)(s * row_bytes), (uint32_t)row_bytes);
      bulk_commit();
      bulk_wait_read_1();  // the copies of the image before this one have read their slot
      __syncwarp();
      if (lane == 0 && tl >= kMoeSenders) mbar_arrive(empty_bar(tl - kMoeSenders));
    }
    bulk_wait_all();
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  __syncthreads();
  const bool ok = s_abort == 0;
  if (threadIdx.x == 0 && !ok) set_status(d.status, EUX_ST_TIMEOUT, 13);
  moe_publish(d, flags, ok);
}

// ---- expert side: wait for every source, (identity expert), tell the sources -
__global__ void moe_expert_ready_kernel(eux_moe_desc d) {
  const int W = d.world;
  __shared__ int s_ok;
  if (threadIdx.x == 0) s_ok = 1;
  __syncthreads();
  uint64_t* peer = nullptr;
  if ((int)threadIdx.x < W) {
    peer = d.flag_peer[threadIdx.x];  // on its way while the flags are polled
    if (!wait_flag_ge(&d.flag_peer[d.rank][threadIdx.x], d.seq, d.wait_timeout_ns)) {
      set_status(d.status, EUX_ST_TIMEOUT, 11);
      s_ok = 0;
    }
  }
  __syncthreads();
  // identity expert: the rows already are the expert output
  if ((int)threadIdx.x < W && s_ok) st_release_sys(peer + 2 * W + d.rank, d.seq);
}

// The experts' arenas are fetched while the flags are polled.
struct MoeArenas {
  const unsigned char* of[kMaxWorld];
};
__device__ __forceinline__ bool moe_wait_experts(const eux_moe_desc& d, MoeArenas& arenas) {
  __shared__ int s_ok;
  if (threadIdx.x == 0) s_ok = 1;
  __syncthreads();
  if ((int)threadIdx.x < d.world) {
    const void* const arena = d.arena_peer[threadIdx.x];
    if (!wait_flag_ge(&d.flag_peer[d.rank][2 * d.world + threadIdx.x], d.seq, d.wait_timeout_ns)) {
      set_status(d.status, EUX_ST_TIMEOUT, 12);
      s_ok = 0;
    }
    arenas.of[threadIdx.x] = reinterpret_cast<const unsigned char*>(arena);
  }
  __syncthreads();
  return s_ok != 0;
}

// The rows of a token and their weights, lane k (< top-k) row k, for a warp that goes from token to token: the routing entries
// of the next token are on their way while this one's rows are read, a trip to L2 that a warp waited for at every token
// (combines in a loop: 4096 x 7168, top-8, bf16 90.0 and 85.5 us, 1024 x 7168 27.6 and 25.4). Not AHEAD: where the registers
// are short (two CTAs per SM; 4096 x 4096, top-2: 15.2 us, 16.8 ahead).
template <bool AHEAD>
struct MoeRows {
  const eux_moe_desc& d;
  const MoeArenas& arenas;
  const size_t row_bytes;
  const int lane, EPR;
  const unsigned char* row = nullptr;
  float w = 0.f;
  int next_expert = 0, next_slot = -1;
  float next_w = 0.f;
  __device__ __forceinline__ MoeRows(const eux_moe_desc& d_, const MoeArenas& arenas_, size_t row_bytes_, int lane_)
      : d(d_), arenas(arenas_), row_bytes(row_bytes_), lane(lane_), EPR(d_.n_experts / d_.world) {}
  __device__ __forceinline__ void fetch(int t) {
    next_slot = -1;
    if (lane < d.topk && t < d.n_tokens) {
      const int64_t i = (int64_t)t * d.topk + lane;
      next_expert = d.topk_idx[i], next_slot = d.slot_of[i], next_w = d.topk_w[i];
    }
  }
  // token t, which comes behind the one before (or is the first and has been fetched), is the current one now
  __device__ __forceinline__ void enter(int t) {
    row = nullptr, w = 0.f;
    if (AHEAD) {
      if (next_slot >= 0) row = arenas.of[next_expert / EPR] + ((size_t)d.rank * d.capacity + next_slot) * row_bytes, w = next_w;
      fetch(t + 1);
    } else if (lane < d.topk) {
      const int e = d.topk_idx[t * d.topk + lane], slot = d.slot_of[t * d.topk + lane];
      if (slot >= 0) {
        row = reinterpret_cast<const unsigned char*>(d.arena_peer[e / EPR]) + ((size_t)d.rank * d.capacity + slot) * row_bytes;
        w = d.topk_w[t * d.topk + lane];
      }
    }
  }
  __device__ __forceinline__ const unsigned char* of(int k) const {
    return (const unsigned char*)__shfl_sync(0xffffffffu, (unsigned long long)row, k);
  }
};

// ---- combine, bf16: unit = (token, 64 chunks); 16 peer loads in flight per lane
__global__ void __launch_bounds__(kMoeThreads) moe_combine_bf16_kernel(eux_moe_desc d) {
  __shared__ MoeArenas arenas;
  if (!moe_wait_experts(d, arenas)) return;
  const int W = d.world, EPR = d.n_experts / W, K = d.topk;
  const int chunks = d.hidden / 8;
  const int upr = (chunks + 63) / 64;
  const size_t row_bytes = (size_t)d.hidden * 2;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int64_t units = (int64_t)d.n_tokens * upr;
  for (int64_t u = warp; u < units; u += nwarps) {
    const int t = (int)(u / upr), part = (int)(u - (int64_t)t * upr);
    const int c0 = part * 64 + lane, c1 = c0 + 32;
    const unsigned char* my_row = nullptr;
    float my_w = 0.f;
    if (lane < K) {
      int e = d.topk_idx[t * K + lane];
      int slot = d.slot_of[t * K + lane];
      if (slot >= 0) {
        int dst = e / EPR;
        my_row = arenas.of[dst] + ((size_t)d.rank * d.capacity + slot) * row_bytes;
        my_w = d.topk_w[t * K + lane];
      }
    }
    float acc0[8], acc1[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc0[j] = 0.f, acc1[j] = 0.f;
    for (int kb = 0; kb < K; kb += 8) {
      uint4 v0[8], v1[8];
      float w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const unsigned char* row = (const unsigned char*)__shfl_sync(0xffffffffu, (unsigned long long)my_row, (kb + k) & 31);
        w[k] = __shfl_sync(0xffffffffu, my_w, (kb + k) & 31);
        if (kb + k >= K) row = nullptr;
        v0[k] = make_uint4(0, 0, 0, 0);
        v1[k] = make_uint4(0, 0, 0, 0);
        if (row) {
          if (c0 < chunks) v0[k] = ld_cg_u4(reinterpret_cast<const uint4*>(row) + c0);
          if (c1 < chunks) v1[k] = ld_cg_u4(reinterpret_cast<const uint4*>(row) + c1);
        } else {
          w[k] = 0.f;
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const __nv_bfloat162* p0 = reinterpret_cast<const __nv_bfloat162*>(&v0[k]);
        const __nv_bfloat162* p1 = reinterpret_cast<const __nv_bfloat162*>(&v1[k]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 a = __bfloat1622float2(p0[j]), b = __bfloat1622float2(p1[j]);
          acc0[2 * j] = fmaf(w[k], a.x, acc0[2 * j]);
          acc0[2 * j + 1] = fmaf(w[k], a.y, acc0[2 * j + 1]);
          acc1[2 * j] = fmaf(w[k], b.x, acc1[2 * j]);
          acc1[2 * j + 1] = fmaf(w[k], b.y, acc1[2 * j + 1]);
        }
      }
    }
    uint4* out = reinterpret_cast<uint4*>(d.out) + (size_t)t * chunks;
    uint4 o0, o1;
    __nv_bfloat162* q0 = reinterpret_cast<__nv_bfloat162*>(&o0);
    __nv_bfloat162* q1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      q0[j] = __floats2bfloat162_rn(acc0[2 * j], acc0[2 * j + 1]);
      q1[j] = __floats2bfloat162_rn(acc1[2 * j], acc1[2 * j + 1]);
    }
    if (c0 < chunks) st_stream_u4(out + c0, o0);
    if (c1 < chunks) st_stream_u4(out + c1, o1);
  }
}

// ---- combine, bf16, top-k <= 8: a warp streams through a contiguous run of (token, 1 KiB) units. Every load
// is 32 bytes per lane, 1 KiB of one row per warp instruction (measured against 16-byte loads: 132 -> 113 us
// on one GPU, 403 -> 388 us when half the rows cross NVLink). A unit's rows are fetched as G groups of R (eight as two
// groups of four, four and fewer as one, two and fewer as one of two), and the next group is always requested before the
// current one is accumulated, so a warp never sits out a whole memory round trip; the routing entries are read once per
// token. (With eight rows for every top-k, 4096 tokens of 4096 took 25.8 us at top-1, 27.6 at 2, 39.5 at 4; 12.7, 15.0 and 36.3
// so. Groups of two rows for more than two, at 64 registers and two CTAs per SM: 44.7 at top-4, 103 against 93 at 8 x 7168.)
template <int R, int G>
__global__ void __launch_bounds__(kMoeThreads, R < 4 ? 2 : 1) moe_combine_bf16_stream_kernel(eux_moe_desc d) {
  __shared__ MoeArenas arenas;
  if (!moe_wait_experts(d, arenas)) return;
  const int chunks = d.hidden / 16;  // 32-byte pieces per row
  const int upr = (chunks + 31) / 32;
  const size_t row_bytes = (size_t)d.hidden * 2;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int64_t units = (int64_t)d.n_tokens * upr;
  const int64_t per = (units + nwarps - 1) / nwarps;
  const int64_t u0 = (int64_t)warp * per;
  const int64_t u1 = u0 + per < units ? u0 + per : units;
  if (u0 >= u1) return;
  int cur_t = (int)(u0 / upr);
  MoeRows<(R == 4)> rows(d, arenas, row_bytes, lane);
  if (R == 4) rows.fetch(cur_t);
  rows.enter(cur_t);
  auto locate = [&](int64_t u, int& t, int& c) {
    t = (int)(u / upr);
    const int part = (int)(u - (int64_t)t * upr);
    c = part * 32 + lane;
    if (t != cur_t) rows.enter(cur_t = t);
  };
  auto issue = [&](int c, int k0, uint32_t (&v)[R][8]) {
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const unsigned char* row = rows.of(k0 + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[k][j] = 0u;
      if (row && c < chunks) moe_ld_v8(row + (size_t)c * 32, v[k]);
    }
  };
  auto accumulate = [&](const uint32_t (&v)[R][8], float w_lane, int k0, float (&acc)[16]) {
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const float w = __shfl_sync(0xffffffffu, w_lane, k0 + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v[k][j]));
        acc[2 * j] = fmaf(w, a.x, acc[2 * j]);
        acc[2 * j + 1] = fmaf(w, a.y, acc[2 * j + 1]);
      }
    }
  };
  uint32_t a[R][8], b[R][8];
  int t, c;
  int64_t u = u0;
  locate(u, t, c);
  issue(c, 0, a);
  // one unit, whose first group is in x: what comes next is requested into the buffer that is not being accumulated
  auto unit = [&](uint32_t (&x)[R][8], uint32_t (&y)[R][8]) {
    const float w_lane = rows.w;
    const int tu = t, cu = c;
    if (G == 2) issue(cu, R, y);
    float acc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = 0.f;
    if (G == 2) accumulate(x, w_lane, 0, acc);
    if (u + 1 < u1) {
      locate(u + 1, t, c);
      if (G == 2) issue(c, 0, x);
      else issue(c, 0, y);
    }
    if (G == 2) accumulate(y, w_lane, R, acc);
    else accumulate(x, w_lane, 0, acc);
    if (cu < chunks) {
      uint4 o0, o1;
      __nv_bfloat162* q0 = reinterpret_cast<__nv_bfloat162*>(&o0);
      __nv_bfloat162* q1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        q0[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
        q1[j] = __floats2bfloat162_rn(acc[8 + 2 * j], acc[8 + 2 * j + 1]);
      }
      uint4* out = reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(d.out) + (size_t)tu * row_bytes + (size_t)cu * 32);
      st_stream_u4(out, o0);
      st_stream_u4(out + 1, o1);
    }
    return ++u < u1;
  };
  if (G == 2)
    while (unit(a, b)) {
    }
  else
    while (unit(a, b) && unit(b, a)) {
    }
}

// ---- combine, fp8 rows: lane owns 16 elements; dequantise while accumulating --
__global__ void __launch_bounds__(kMoeThreads) moe_combine_fp8_kernel(eux_moe_desc d) {
  __shared__ MoeArenas arenas;
  if (!moe_wait_experts(d, arenas)) return;
  const int W = d.world, EPR = d.n_experts / W, K = d.topk;
  const int upr = (d.hidden + 511) / 512;
  const size_t row_bytes = moe_row_bytes(d.hidden, 1);
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int64_t units = (int64_t)d.n_tokens * upr;
  for (int64_t u = warp; u < units; u += nwarps) {
    const int t = (int)(u / upr), part = (int)(u - (int64_t)t * upr);
    const int e0 = part * 512 + lane * 16;
    const bool in = e0 < d.hidden;
    const unsigned char* my_row = nullptr;
    float my_w = 0.f;
    if (lane < K) {
      int e = d.topk_idx[t * K + lane];
      int slot = d.slot_of[t * K + lane];
      if (slot >= 0) {
        int dst = e / EPR;
        my_row = arenas.of[dst] + ((size_t)d.rank * d.capacity + slot) * row_bytes;
        my_w = d.topk_w[t * K + lane];
      }
    }
    float acc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = 0.f;
    for (int kb = 0; kb < K; kb += 8) {
      uint4 v[8];
      float w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const unsigned char* row = (const unsigned char*)__shfl_sync(0xffffffffu, (unsigned long long)my_row, (kb + k) & 31);
        float wk = __shfl_sync(0xffffffffu, my_w, (kb + k) & 31);
        if (kb + k >= K) row = nullptr;
        v[k] = make_uint4(0, 0, 0, 0);
        w[k] = 0.f;
        if (row && in) {
          v[k] = ld_cg_u4(row + e0);
          w[k] = wk * __ldcg(reinterpret_cast<const float*>(row + d.hidden) + (e0 >> 7));
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(&v[k]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(p[j] & 0xffffu), __NV_E4M3);
          __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(p[j] >> 16), __NV_E4M3);
          float2 a = __half22float2(*reinterpret_cast<__half2*>(&lo));
          float2 b = __half22float2(*reinterpret_cast<__half2*>(&hi));
          acc[4 * j] = fmaf(w[k], a.x, acc[4 * j]);
          acc[4 * j + 1] = fmaf(w[k], a.y, acc[4 * j + 1]);
          acc[4 * j + 2] = fmaf(w[k], b.x, acc[4 * j + 2]);
          acc[4 * j + 3] = fmaf(w[k], b.y, acc[4 * j + 3]);
        }
      }
    }
    if (in) {
      uint4 o0, o1;
      __nv_bfloat162* q0 = reinterpret_cast<__nv_bfloat162*>(&o0);
      __nv_bfloat162* q1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        q0[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
        q1[j] = __floats2bfloat162_rn(acc[8 + 2 * j], acc[8 + 2 * j + 1]);
      }
      uint4* out = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(d.out) + (size_t)t * d.hidden + e0);
      st_stream_u4(out, o0);
      st_stream_u4(out + 1, o1);
    }
  }
}

__device__ __forceinline__ float pick4(const float (&r)[4], int i) {
  return i == 0 ? r[0] : (i == 1 ? r[1] : (i == 2 ? r[2] : r[3]));
}
// ---- combine, fp8 rows, one warp per token (top-k <= 8, hidden <= 16384) -----------------
// The scales of the k rows are fetched once per row (two coalesced loads per row instead of one
// small load per 512 elements), already multiplied by the gate weight.
__global__ void __launch_bounds__(kMoeThreads) moe_combine_fp8_rows_kernel(eux_moe_desc d) {
  __shared__ MoeArenas arenas;
  if (!moe_wait_experts(d, arenas)) return;
  const int W = d.world, EPR = d.n_experts / W, K = d.topk;
  const int upr = (d.hidden + 511) / 512;
  const int ngroups = d.hidden / 128;
  const size_t row_bytes = moe_row_bytes(d.hidden, 1);
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int t = warp; t < d.n_tokens; t += nwarps) {
    const unsigned char* my_row = nullptr;
    float my_w = 0.f;
    if (lane < K) {
      int e = d.topk_idx[t * K + lane];
      int slot = d.slot_of[t * K + lane];
      if (slot >= 0) {
        int dst = e / EPR;
        my_row = arenas.of[dst] + ((size_t)d.rank * d.capacity + slot) * row_bytes;
        my_w = d.topk_w[t * K + lane];
      }
    }
    const unsigned char* rows[8];
    float scw[8][4];  // gate weight x scale, lane L keeps groups L, 32+L, 64+L, 96+L of row k
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      rows[k] = (const unsigned char*)__shfl_sync(0xffffffffu, (unsigned long long)my_row, k);
      const float wk = __shfl_sync(0xffffffffu, my_w, k);
      if (k >= K) rows[k] = nullptr;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int g = r * 32 + lane;
        scw[k][r] = (rows[k] && g < ngroups) ? wk * __ldcg(reinterpret_cast<const float*>(rows[k] + d.hidden) + g) : 0.f;
      }
    }
    __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(d.out) + (size_t)t * d.hidden;
    for (int part = 0; part < upr; ++part) {
      const int e0 = part * 512 + lane * 16;
      const bool in = e0 < d.hidden;
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        v[k] = make_uint4(0, 0, 0, 0);
        if (rows[k] && in) v[k] = ld_cg_u4(rows[k] + e0);
      }
      float acc[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[j] = 0.f;
      const int gi = part * 4 + (lane >> 3);  // scale group of this lane's 16 elements
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float wk = __shfl_sync(0xffffffffu, pick4(scw[k], gi >> 5), gi & 31);
        const uint32_t* p = reinterpret_cast<const uint32_t*>(&v[k]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(p[j] & 0xffffu), __NV_E4M3);
          __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(p[j] >> 16), __NV_E4M3);
          float2 a = __half22float2(*reinterpret_cast<__half2*>(&lo));
          float2 b = __half22float2(*reinterpret_cast<__half2*>(&hi));
          acc[4 * j] = fmaf(wk, a.x, acc[4 * j]);
          acc[4 * j + 1] = fmaf(wk, a.y, acc[4 * j + 1]);
          acc[4 * j + 2] = fmaf(wk, b.x, acc[4 * j + 2]);
          acc[4 * j + 3] = fmaf(wk, b.y, acc[4 * j + 3]);
        }
      }
      if (in) {
        uint4 o0, o1;
        __nv_bfloat162* q0 = reinterpret_cast<__nv_bfloat162*>(&o0);
        __nv_bfloat162* q1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          q0[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
          q1[j] = __floats2bfloat162_rn(acc[8 + 2 * j], acc[8 + 2 * j + 1]);
        }
        uint4* out = reinterpret_cast<uint4*>(orow + e0);
        st_stream_u4(out, o0);
        st_stream_u4(out + 1, o1);
      }
    }
  }
}

static int moe_check(const eux_moe_desc* d) {
  if (!d || d->world < 1 || d->world > kMaxWorld || d->rank < 0 || d->rank >= d->world) return EUX_ERR_BAD_ARG;
  if (d->n_experts % d->world || d->hidden % 128 || d->hidden <= 0 || d->topk < 1 || d->topk > 32) return EUX_ERR_BAD_ARG;
  if (d->n_experts > kMaxExperts || d->capacity < 1 || d->n_tokens < 0) return EUX_ERR_BAD_ARG;
  return 0;
}

}  // namespace eux

using namespace eux;

extern "C" size_t eux_moe_row_bytes(int hidden, int fp8) { return moe_row_bytes(hidden, fp8); }

static int moe_sms(int* dev_out = nullptr) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (dev_out) *dev_out = dev;
  return sms;
}

// The count launch, where there are too many entries for every CTA to count them all, and the dispatch, with the routing
// tables and `extra` bytes of shared memory, at most `most_extra` in any launch of this kernel.
template <auto KERNEL, typename... More>
static int moe_dispatch(const eux_moe_desc* d, int ctas, int dev, int sms, size_t extra, size_t most_extra, cudaStream_t st, More... more) {
  const int grid = std::max(1, std::min(ctas, d->n_tokens));
  const size_t smem = 3 * (size_t)d->n_experts * sizeof(int) + extra;
  if (cudaError_t e = allow_smem<KERNEL>(dev, 3 * (size_t)kMaxExperts * sizeof(int) + most_extra); e != cudaSuccess) return (int)e;
  const int64_t entries = (int64_t)d->n_tokens * d->topk;
  const int counted = entries > kRouteSelf;
  if (counted) {
    const int64_t want = (entries + kMoeThreads - 1) / kMoeThreads;
    moe_count_kernel<<<(int)std::min<int64_t>(want, sms), kMoeThreads, 2 * (size_t)d->n_experts * sizeof(int), st>>>(*d);
  }
  KERNEL<<<grid, kMoeThreads, smem, st>>>(*d, counted, more...);
  return (int)cudaGetLastError();
}

extern "C" int eux_moe_dispatch_launch(const eux_moe_desc* d, int ctas, void* stream) {
  if (int rc = moe_check(d)) return rc;
  const cudaStream_t st = (cudaStream_t)stream;
  int dev = 0;
  const int sms = moe_sms(&dev);
  // A CTA per token, up to one per SM: a second one counts all entries again (256 tokens, fp8: 28.2 us for the exchange
  // with one, 30.2 with two).
  const int one = ctas > 0 ? ctas : sms;
  if (!d->fp8) {
    // Rows for more than twice the L2: six CTAs per SM, the last ones of which begin as SMs become free, so that no SM's share
    // ends late (top-8 of 7168, the exchange with one and with six per SM: 2048 tokens, 235 MB, 104.5 and 104.3 us; 2560
    // 128.7 and 126.6; 4096 197.8 and 192.0; 8192 376.1 and 360.6).
    const bool large = (int64_t)d->n_tokens * d->topk * d->hidden * 2 >= (int64_t(256) << 20) && d->n_tokens >= 12 * sms;
    return moe_dispatch<moe_dispatch_bf16_kernel>(d, ctas > 0 ? ctas : large ? 6 * sms : sms, dev, sms, 0, 0, st);
  }
  if (const int slots = moe_image_slots(d->hidden); slots > 0 && d->n_tokens >= 2 * (int64_t)one)
    return moe_dispatch<moe_dispatch_fp8_bulk_kernel>(d, one, dev, sms, 128 + (size_t)slots * moe_row_bytes(d->hidden, 1), 128 + kMoeImageBytes, st, slots);
  // Rows too wide for images and more than eight tokens per CTA: two per SM, one of which works while the other waits at its
  // barriers.
  if (ctas <= 0) ctas = d->n_tokens > 8 * sms ? 2 * sms : sms;
  return moe_dispatch<moe_dispatch_fp8_kernel>(d, ctas, dev, sms, 2 * (size_t)moe_scale_stride(d->hidden) * sizeof(float),
                                               2 * (size_t)kMoeScaleFloats * sizeof(float), st);
}

extern "C" int eux_moe_expert_ready_launch(const eux_moe_desc* d, void* stream) {
  if (int rc = moe_check(d)) return rc;
  moe_expert_ready_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(*d);
  return (int)cudaGetLastError();
}

// ---- combine, fp8 rows, top-k <= 8, hidden <= 8192: the streaming scheme of the bf16 kernel. A unit is 1024
// elements of a token (32 bytes per lane, 1 KiB of a row per warp instruction); its rows are fetched as G
// groups of two (2 G >= top-k), the next group always requested before the current one is dequantised and
// accumulated. Lane L keeps the scales of groups L and 32 + L of every row, loaded once per token.
// (4096 tokens of 4096, with eight rows for every top-k and so: 25.2 and 18.5 us at top-1, 30.9 and 26.6 at 4, 40.0 and 38.7 at 6.)
template <int G>
__global__ void __launch_bounds__(kMoeThreads) moe_combine_fp8_stream_kernel(eux_moe_desc d) {
  __shared__ MoeArenas arenas;
  if (!moe_wait_experts(d, arenas)) return;
  const int upr = (d.hidden + 1023) / 1024;
  const int ngroups = d.hidden / 128;
  const size_t row_bytes = moe_row_bytes(d.hidden, 1);
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int64_t units = (int64_t)d.n_tokens * upr;
  const int64_t per = (units + nwarps - 1) / nwarps;
  const int64_t u0 = (int64_t)warp * per;
  const int64_t u1 = u0 + per < units ? u0 + per : units;
  if (u0 >= u1) return;
  int cur_t = (int)(u0 / upr);
  MoeRows<true> rows(d, arenas, row_bytes, lane);
  rows.fetch(cur_t);
  rows.enter(cur_t);
  float scw[2 * G][2];
  auto locate = [&](int64_t u, int& t, int& e0) {
    t = (int)(u / upr);
    e0 = (int)(u - (int64_t)t * upr) * 1024 + lane * 32;
  };
  // the scales of the current token's rows, requested behind its first values and multiplied when they are used
  auto scales = [&]() {
#pragma unroll
    for (int k = 0; k < 2 * G; ++k) {
      const unsigned char* row = rows.of(k);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int g = r * 32 + lane;
        scw[k][r] = (row && g < ngroups) ? __ldcg(reinterpret_cast<const float*>(row + d.hidden) + g) : 0.f;
      }
    }
  };
  auto issue = [&](int e0, int k0, uint32_t (&v)[2][8]) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const unsigned char* row = rows.of(k0 + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[k][j] = 0u;
      if (row && e0 < d.hidden) moe_ld_v8(row + e0, v[k]);
    }
  };
  int t, e0;
  int64_t u = u0;
  locate(u, t, e0);
  uint32_t a[2][8], b[2][8];
  issue(e0, 0, a);
  scales();
  // one unit, whose first group is in x; the first group of the next one ends up in x where G is even, in y where it is odd
  auto unit = [&](uint32_t (&x)[2][8], uint32_t (&y)[2][8]) {
    const int tu = t, eu = e0;
    const int gi = eu >> 7;  // scale group of this lane's 32 elements
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0.f;
    // the weights of this unit's token, fetched before the routing entries may move on to the next one
    float wk[2 * G];
#pragma unroll
    for (int k = 0; k < 2 * G; ++k)
      wk[k] = __shfl_sync(0xffffffffu, rows.w, k) * __shfl_sync(0xffffffffu, (gi >> 5) ? scw[k][1] : scw[k][0], gi & 31);
    auto accumulate = [&](const uint32_t (&v)[2][8], float w0, float w1) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float w = k == 0 ? w0 : w1;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v[k][j] & 0xffffu), __NV_E4M3);
          __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v[k][j] >> 16), __NV_E4M3);
          const float2 p = __half22float2(*reinterpret_cast<__half2*>(&lo));
          const float2 q = __half22float2(*reinterpret_cast<__half2*>(&hi));
          acc[4 * j] = fmaf(w, p.x, acc[4 * j]);
          acc[4 * j + 1] = fmaf(w, p.y, acc[4 * j + 1]);
          acc[4 * j + 2] = fmaf(w, q.x, acc[4 * j + 2]);
          acc[4 * j + 3] = fmaf(w, q.y, acc[4 * j + 3]);
        }
      }
    };
#pragma unroll
    for (int g = 0; g < G; ++g) {
      uint32_t (&now)[2][8] = g & 1 ? y : x;
      uint32_t (&then)[2][8] = g & 1 ? x : y;
      if (g + 1 < G) {
        issue(eu, 2 * (g + 1), then);
      } else if (u + 1 < u1) {
        locate(u + 1, t, e0);
        const bool entered = t != cur_t;
        if (entered) rows.enter(cur_t = t);
        issue(e0, 0, then);
        if (entered) scales();
      }
      accumulate(now, wk[2 * g], wk[2 * g + 1]);
    }
    if (eu < d.hidden) {
      uint4* out = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(d.out) + (size_t)tu * d.hidden + eu);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 o;
        __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) p2[j] = __floats2bfloat162_rn(acc[8 * q + 2 * j], acc[8 * q + 2 * j + 1]);
        st_stream_u4(out + q, o);
      }
    }
    return ++u < u1;
  };
  if (G % 2 == 0)
    while (unit(a, b)) {
    }
  else
    while (unit(a, b) && unit(b, a)) {
    }
}

extern "C" int eux_moe_combine_launch(const eux_moe_desc* d, int ctas, void* stream) {
  if (int rc = moe_check(d)) return rc;
  if (ctas <= 0) {
    // As many as are resident: a CTA streams through its share and would start anew in a second wave (calls of 4096 x 7168,
    // top-8, an exchange of bf16 205.3 us with two waves and 202.2 with one, fp8 133.9 and 131.4; 1024 x 7168 62.5 and 59.3).
    // And no CTA without a unit (of at least 512 elements of a token) for some warp: each polls the flags.
    const int64_t units = (int64_t)d->n_tokens * ((d->hidden + 511) / 512);
    const int64_t resident = (int64_t)moe_sms() * (!d->fp8 && d->topk <= 2 ? 2 : 1);
    ctas = (int)std::min<int64_t>(resident, std::max<int64_t>(1, (units + kMoeThreads / 32 - 1) / (kMoeThreads / 32)));
  }
  const cudaStream_t st = (cudaStream_t)stream;
  if (d->fp8 && d->topk <= 8 && d->hidden <= 8192) {
    if (d->topk <= 2) moe_combine_fp8_stream_kernel<1><<<ctas, kMoeThreads, 0, st>>>(*d);
    else if (d->topk <= 4) moe_combine_fp8_stream_kernel<2><<<ctas, kMoeThreads, 0, st>>>(*d);
    else if (d->topk <= 6) moe_combine_fp8_stream_kernel<3><<<ctas, kMoeThreads, 0, st>>>(*d);
    else moe_combine_fp8_stream_kernel<4><<<ctas, kMoeThreads, 0, st>>>(*d);
  } else if (d->fp8 && d->topk <= 8 && d->hidden <= 16384) moe_combine_fp8_rows_kernel<<<ctas, kMoeThreads, 0, st>>>(*d);
  else if (d->fp8) moe_combine_fp8_kernel<<<ctas, kMoeThreads, 0, st>>>(*d);
  else if (d->topk <= 2) moe_combine_bf16_stream_kernel<2, 1><<<ctas, kMoeThreads, 0, st>>>(*d);
  else if (d->topk <= 4) moe_combine_bf16_stream_kernel<4, 1><<<ctas, kMoeThreads, 0, st>>>(*d);
  else if (d->topk <= 8) moe_combine_bf16_stream_kernel<4, 2><<<ctas, kMoeThreads, 0, st>>>(*d);
  else moe_combine_bf16_kernel<<<ctas, kMoeThreads, 0, st>>>(*d);
  return (int)cudaGetLastError();
}


// Loads every kernel of this file (see eux_xfer_preload for why a first launch must not be the one that loads).
extern "C" int eux_moe_preload(void) {
  cudaFuncAttributes attr;
  const void* kernels[] = {(const void*)moe_count_kernel,
                           (const void*)moe_dispatch_bf16_kernel,       (const void*)moe_dispatch_fp8_kernel,
                           (const void*)moe_dispatch_fp8_bulk_kernel,
                           (const void*)moe_expert_ready_kernel,        (const void*)moe_combine_bf16_kernel,
                           (const void*)moe_combine_bf16_stream_kernel<2, 1>, (const void*)moe_combine_bf16_stream_kernel<4, 1>,
                           (const void*)moe_combine_bf16_stream_kernel<4, 2>, (const void*)moe_combine_fp8_kernel,
                           (const void*)moe_combine_fp8_rows_kernel,    (const void*)moe_combine_fp8_stream_kernel<1>,
                           (const void*)moe_combine_fp8_stream_kernel<2>, (const void*)moe_combine_fp8_stream_kernel<3>,
                           (const void*)moe_combine_fp8_stream_kernel<4>};
  for (const void* k : kernels) {
    cudaError_t e = cudaFuncGetAttributes(&attr, k);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}
