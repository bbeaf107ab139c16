// Tensor send/recv data plane (the role UCX's cuda_ipc/cuda_copy transports
// play under ucp_am_send_nbx in the reference, ucx_context/ucx_connection.cpp:353-398,
// and the role of the divide-by-two "handler" kernel in
// ucx_context/ucx_am_context/ucx_am_context_test_cuda_helper.cu:27-78).
//
// One kernel does: (optional bounded acquire-wait on an arrival flag) ->
// strided gather / dense read of the source tensor -> elementwise handler ->
// dtype cast -> dense store into the destination (normally a slot of the
// peer's receive arena, mapped into this process) -> system-scope release of
// a sequence flag. Nothing is staged through the host.
#include "eux_bulk.cuh"
#include "eux_device.cuh"

namespace eux {

constexpr int kXferThreads = 512;

struct XferArgs {
  eux_xfer_desc d;
  uint32_t* counter;
};

template <typename T>
struct Elem;
template <>
struct Elem<float> {
  static __device__ __forceinline__ float to(float v) { return v; }
  static __device__ __forceinline__ float from(float f) { return f; }
};
template <>
struct Elem<__half> {
  static __device__ __forceinline__ float to(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from(float f) { return __float2half_rn(f); }
};
template <>
struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float to(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from(float f) { return __float2bfloat16_rn(f); }
};
template <>
struct Elem<__nv_fp8_e4m3> {
  static __device__ __forceinline__ float to(__nv_fp8_e4m3 v) { return float(v); }
  static __device__ __forceinline__ __nv_fp8_e4m3 from(float f) { return __nv_fp8_e4m3(f); }
};

template <>
struct Elem<uint8_t> {
  static __device__ __forceinline__ uint8_t from(float f) { return (uint8_t)f; }
};

template <int BYTES>
struct PackT;
template <>
struct PackT<8> {
  using type = uint2;
};
template <>
struct PackT<16> {
  using type = uint4;
};

// Wait (bounded) for the arrival flag; every thread of the CTA learns the outcome.
__device__ __forceinline__ bool cta_wait_arrival(const eux_xfer_desc& d) {
  if (d.wait_flag == nullptr) return true;
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    bool ok = wait_flag_ge(d.wait_flag, d.wait_value, d.wait_timeout_ns);
    if (!ok) set_status(d.status, EUX_ST_TIMEOUT, 1);
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// All stores of this CTA are done; the last CTA of the grid publishes the flag, and only if no CTA
// of the grid gave up: every CTA runs its own bounded wait, so near the deadline one can time out (and
// skip its share of the copy) while the last one to arrive succeeded. The scratch word counts arrivals
// in its low 31 bits; a CTA that failed sets the top bit before it counts itself. A CTA's fence before it counts itself is for
// this GPU, where the last CTA sees the counts; that one's fence for everyone then covers what all of them wrote, into a
// peer's memory too. (System-scope fences queue up at 31 ns each: with one per CTA, flagged transfers in a loop took, 16 MiB of
// bytes 10.2 us, of fp32 to bf16 12.5, of bf16 at an odd offset 21.3, 4099 x 4096 fp32 transposed to bf16 29.4; now 7.2, 5.5,
// 8.4 and 20.9.)
__device__ __forceinline__ void cta_publish(const eux_xfer_desc& d, uint32_t* counter, bool ok) {
  if (!d.flag && !d.flag2) return;  // nobody is told: the end of the launch is enough
  __syncthreads();
  if (threadIdx.x != 0) return;
  bool last = true;
  if (gridDim.x > 1) {
    fence_gpu();
    if (!ok) atomicOr(counter, 0x80000000u);
    const uint32_t old = atomicAdd(counter, 1u);
    last = ((old & 0x7fffffffu) == gridDim.x - 1);
    if (old & 0x80000000u) ok = false;
    if (last) {
      *counter = 0;  // leave the scratch word clean for the next launch
    }
  }
  if (last) fence_sys();  // what all CTAs wrote, the others before they counted themselves, comes before the flags
  if (last && ok && d.flag) st_relaxed_sys(d.flag, d.flag_value);
  if (last && ok && d.flag2) st_relaxed_sys(d.flag2, d.flag2_value);
}

// The first and the last thing a transfer kernel does. What follows in the stream may be launched when a CTA has issued its
// last stores, and from the start where the whole takes a few microseconds (a source of up to 32 MiB). It sits on the SMs
// until the transfer ends: let in at the start, a GEMM behind a push of 1 GiB held up a small GEMM of another stream for as
// long as the push and itself took, 0.98 ms instead of 0.34, and large transfers in a loop were no faster for it (4096 x 7168
// fp32 to e4m3 23.8 us and 23.4 from the end on). A push of 640 x 1024 with a GEMM of 640 x 4096 x 1024 behind it takes 11.8 us
// with the GEMM let in at the start and 13.1 at the end, pushes of 16 MiB 4.42 and 4.55 (graph replays).
// Tiles let it in at the end only: several small launches were on the SMs at a time and the later ones of them found room on
// some SMs more than on others (2048 x 2048 e4m3 to bf16 transposed, graph replays, 6.5 us, 4.1 so, 4.5 without early launches;
// bytes 5.3, 3.2 and 3.6).
__device__ __forceinline__ void xfer_begin(const eux_xfer_desc& d) {
  if (d.wait_flag == nullptr && d.n_elems * (uint64_t)dtype_size(d.src_dtype) <= (32u << 20)) allow_next_launch();
  wait_for_launch_before();
}
__device__ __forceinline__ void xfer_end(const eux_xfer_desc& d, uint32_t* counter, bool ok) {
  if (d.wait_flag == nullptr) allow_next_launch();
  cta_publish(d, counter, ok);
}

// Dense byte copy. A CTA works on one contiguous block at a time and the blocks are dealt
// round-robin to the CTAs, so that what a CTA has in flight stays inside a few DRAM pages.
// With 32-byte aligned buffers each thread moves two 32-byte vectors per block (measured best
// on B200: 3.31 TB/s each way for a local copy, above cudaMemcpy's 3.26; four or eight 16-byte
// accesses in flight per thread reach 3.17 and 3.01); otherwise four 16-byte vectors.
__device__ __forceinline__ void ld_v8(const void* p, uint32_t (&v)[8]) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(p));
}
__device__ __forceinline__ void st_v8(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// `cta` of `nctas` CTAs share the copy (the whole grid for one message, a single CTA for one
// descriptor of a batch).
template <bool V32>
__device__ __forceinline__ void copy_bytes_grid(const unsigned char* src, unsigned char* dst, uint64_t nbytes,
                                                uint32_t cta, uint32_t nctas) {
  const uint64_t tid = (uint64_t)cta * blockDim.x + threadIdx.x;
  const uint64_t nthreads = (uint64_t)nctas * blockDim.x;
  uint64_t done = 0;  // bytes handled by the blocked loops
  if (V32) {
    constexpr int U = 2;
    const uint64_t block_bytes = (uint64_t)blockDim.x * U * 32;
    const uint64_t nblocks = nbytes / block_bytes;
    for (uint64_t b = cta; b < nblocks; b += nctas) {
      const uint64_t off = b * block_bytes + (uint64_t)threadIdx.x * 32;
      uint32_t v[U][8];
#pragma unroll
      for (int j = 0; j < U; ++j) ld_v8(src + off + (uint64_t)j * blockDim.x * 32, v[j]);
#pragma unroll
      for (int j = 0; j < U; ++j) st_v8(dst + off + (uint64_t)j * blockDim.x * 32, v[j]);
    }
    done = nblocks * block_bytes;
  } else {
    constexpr int U = 4;
    const uint64_t block_bytes = (uint64_t)blockDim.x * U * 16;
    const uint64_t nblocks = nbytes / block_bytes;
    for (uint64_t b = cta; b < nblocks; b += nctas) {
      const uint64_t off = b * block_bytes + (uint64_t)threadIdx.x * 16;
      uint4 v[U];
#pragma unroll
      for (int j = 0; j < U; ++j) v[j] = ld_cg_u4(src + off + (uint64_t)j * blockDim.x * 16);
#pragma unroll
      for (int j = 0; j < U; ++j) st_u4(dst + off + (uint64_t)j * blockDim.x * 16, v[j]);
    }
    done = nblocks * block_bytes;
  }
  // what is left of the last block: 16-byte vectors, then single bytes
  const uint64_t nvec = (nbytes - done) >> 4;
  for (uint64_t i = tid; i < nvec; i += nthreads) st_u4(dst + done + i * 16, ld_cg_u4(src + done + i * 16));
  for (uint64_t b = done + (nvec << 4) + tid; b < nbytes; b += nthreads) dst[b] = src[b];
}

template <bool V32>
__global__ void __launch_bounds__(kXferThreads) xfer_bytes_kernel(XferArgs a) {
  const eux_xfer_desc& d = a.d;
  xfer_begin(d);
  bool ok = cta_wait_arrival(d);
  if (ok) {
    const uint64_t nbytes = d.n_elems * (uint64_t)dtype_size(d.src_dtype);
    copy_bytes_grid<V32>(reinterpret_cast<const unsigned char*>(d.src), reinterpret_cast<unsigned char*>(d.dst), nbytes,
                         blockIdx.x, gridDim.x);
  }
  xfer_end(d, a.counter, ok);
}

// Dense byte copy on the bulk-copy engine: two threads per CTA drive a ring of shared-memory
// chunks (loads from the source with completion on an mbarrier, stores to the destination in
// bulk groups). The SMs issue almost no instructions, and the bytes in flight per CTA (the whole
// ring) do not depend on how many threads there are, which is what a source across NVLink needs.
constexpr int kBulkChunk = 16384;
constexpr int kBulkStages = 6;  // 96 KiB of ring per CTA: two CTAs per SM
constexpr int kBulkThreads = 128;
constexpr size_t kBulkSmem = (size_t)kBulkChunk * kBulkStages + 128;

__global__ void __launch_bounds__(kBulkThreads) xfer_bulk_kernel(XferArgs a) {
  extern __shared__ unsigned char xb_raw[];
  __shared__ uint64_t xb_bars[2 * kBulkStages];
  __shared__ int xb_abort;
  const eux_xfer_desc& d = a.d;
  bool ok = cta_wait_arrival(d);
  const uint32_t ring0 = smem_u32(reinterpret_cast<unsigned char*>(((uintptr_t)xb_raw + 127) & ~(uintptr_t)127));
  const uint32_t bar0 = smem_u32(xb_bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (kBulkStages + s); };
  if (threadIdx.x == 0) {
    xb_abort = 0;
    for (int s = 0; s < kBulkStages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  volatile int* abort = &xb_abort;
  const uint64_t nbytes = d.n_elems * (uint64_t)dtype_size(d.src_dtype);
  const uint64_t body = nbytes & ~(uint64_t)15;
  const uint64_t nchunks = (body + kBulkChunk - 1) / kBulkChunk;
  const unsigned char* src = reinterpret_cast<const unsigned char*>(d.src);
  unsigned char* dst = reinterpret_cast<unsigned char*>(d.dst);
  if (ok && threadIdx.x == 0) {
    uint32_t c = 0;
    for (uint64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x, ++c) {
      const int st = (int)(c % kBulkStages);
      if (!mbar_wait(empty_bar(st), ((c / kBulkStages) & 1u) ^ 1u, abort, d.wait_timeout_ns)) break;
      const uint64_t off = ch * kBulkChunk;
      const uint32_t n = (uint32_t)min((uint64_t)kBulkChunk, body - off);
      mbar_expect_tx(full_bar(st), n);
      bulk_g2s(ring0 + (uint32_t)st * kBulkChunk, src + off, n, full_bar(st));
    }
    if (*abort) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
  } else if (ok && threadIdx.x == 32) {
    uint32_t c = 0, released = 0;
    for (uint64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x, ++c) {
      const int st = (int)(c % kBulkStages);
      if (!mbar_wait(full_bar(st), (c / kBulkStages) & 1u, abort, d.wait_timeout_ns)) break;
      const uint64_t off = ch * kBulkChunk;
      const uint32_t n = (uint32_t)min((uint64_t)kBulkChunk, body - off);
      bulk_s2g(dst + off, ring0 + (uint32_t)st * kBulkChunk, n);
      bulk_commit();
      bulk_wait_read_1();
      for (; released < c; ++released) mbar_arrive(empty_bar((int)(released % kBulkStages)));
    }
    bulk_wait_all();  // the stores have been performed
    asm volatile("fence.proxy.async;" ::: "memory");
    if (*abort) set_status(d.status, EUX_ST_TIMEOUT, 2);
  } else if (ok && blockIdx.x == 0 && threadIdx.x >= 64 && threadIdx.x < 64 + (nbytes & 15)) {
    const uint64_t b = body + (threadIdx.x - 64);
    dst[b] = src[b];
  }
  __syncthreads();
  cta_publish(d, a.counter, ok && xb_abort == 0);
}

// Eight neighbouring elements as registers: 8 or 16 bytes in one access, 32 bytes (fp32) in one where both buffers start
// on a 32-byte boundary and in two otherwise.
template <typename T>
__device__ __forceinline__ void load8(const T* p, bool wide, T (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    if (wide) {
      ld_v8(p, *reinterpret_cast<uint32_t(*)[8]>(v));
      return;
    }
  }
  using P = typename PackT<(8 * sizeof(T) >= 16 ? 16 : 8)>::type;
#pragma unroll
  for (int k = 0; k < (int)(8 * sizeof(T) / sizeof(P)); ++k) reinterpret_cast<P*>(v)[k] = __ldcg(reinterpret_cast<const P*>(p) + k);
}
template <typename T>
__device__ __forceinline__ void store8(T* p, bool wide, T (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    if (wide) {
      st_v8(p, *reinterpret_cast<uint32_t(*)[8]>(v));
      return;
    }
  }
  using P = typename PackT<(8 * sizeof(T) >= 16 ? 16 : 8)>::type;
#pragma unroll
  for (int k = 0; k < (int)(8 * sizeof(T) / sizeof(P)); ++k) reinterpret_cast<P*>(p)[k] = reinterpret_cast<P*>(v)[k];
}

// Dense typed path: 8 elements per step, two steps in flight, cast + handler fused. Bound by DRAM: what it takes is bytes
// in flight and whole sectors per access (2^26 elements, one step with 16-byte accesses and two CTAs per SM -> now:
// bf16 to e4m3 51 -> 33 us, e4m3 to bf16 52 -> 40, bf16 to fp32 level at 76, fp32 to e4m3 of 4096 x 7168 30 -> 26).
template <typename S, typename D>
__device__ __forceinline__ void typed_body(const eux_xfer_desc& d) {
  const S* src = reinterpret_cast<const S*>(d.src);
  D* dst = reinterpret_cast<D*>(d.dst);
  const uint64_t n8 = d.n_elems >> 3;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
  const int op = d.op;
  const float arg = d.op_arg;
  const bool wide = ((((uintptr_t)src) | ((uintptr_t)dst)) & 31u) == 0;
  for (uint64_t i0 = tid; i0 < n8; i0 += 2 * nthreads) {
    alignas(32) S sv[2][8];
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (i0 + u * nthreads < n8) load8(src + (i0 + u * nthreads) * 8, wide, sv[u]);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (i0 + u * nthreads >= n8) break;
      alignas(32) D dv[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) dv[k] = Elem<D>::from(apply_op(Elem<S>::to(sv[u][k]), op, arg));
      store8(dst + (i0 + u * nthreads) * 8, wide, dv);
    }
  }
  for (uint64_t e = (n8 << 3) + tid; e < d.n_elems; e += nthreads)
    dst[e] = Elem<D>::from(apply_op(Elem<S>::to(src[e]), op, arg));
}

template <typename S, typename D>
__global__ void __launch_bounds__(kXferThreads, sizeof(S) == 4 ? 2 : 4) xfer_typed_kernel(XferArgs a) {
  const eux_xfer_desc& d = a.d;
  xfer_begin(d);
  bool ok = cta_wait_arrival(d);
  if (ok) typed_body<S, D>(d);
  xfer_end(d, a.counter, ok);
}

// One tensor-RPC echo step of a rank in a single launch: push the request into the partner's arena and
// publish its flag; as the partner's server, wait for its request, apply the handler and push the response
// back; as client again, wait for the response. Each phase is what xfer_bytes_kernel / xfer_typed_kernel
// do in a launch of their own. The partner runs the same kernel on its GPU at the same time; no CTA waits
// for a CTA of its own grid (a phase's flag is published by whichever CTA finishes it last), and the grid
// is at most one CTA per SM, so every CTA is resident. All tensors dense, 16-byte aligned, of one dtype.
struct RpcStepArgs {
  eux_xfer_desc req, resp, done;
  uint32_t* counter;  // three words
};
template <typename S>
__device__ __forceinline__ void rpc_phase(const eux_xfer_desc& d, uint32_t* counter) {
  bool ok = cta_wait_arrival(d);
  if (ok && d.n_elems) {
    if (d.op == EUX_OP_NONE) {
      const unsigned char* src = reinterpret_cast<const unsigned char*>(d.src);
      unsigned char* dst = reinterpret_cast<unsigned char*>(d.dst);
      const uint64_t nbytes = d.n_elems * (uint64_t)dtype_size(d.src_dtype);
      if (((((uintptr_t)src) | ((uintptr_t)dst)) & 31u) == 0) copy_bytes_grid<true>(src, dst, nbytes, blockIdx.x, gridDim.x);
      else copy_bytes_grid<false>(src, dst, nbytes, blockIdx.x, gridDim.x);
    } else
      typed_body<S, S>(d);
  }
  cta_publish(d, counter, ok);
}
template <typename S>
__global__ void __launch_bounds__(kXferThreads) xfer_rpc_step_kernel(RpcStepArgs a) {
  rpc_phase<S>(a.req, a.counter);
  rpc_phase<S>(a.resp, a.counter + 1);
  if (blockIdx.x == 0) {  // the completion: one CTA watches the response flag
    const bool ok = cta_wait_arrival(a.done);
    (void)ok;
  }
}

// ---- gathers ---------------------------------------------------------------------------------------
// What the layout is, eux_xfer_launch finds out on the host (size-1 dimensions dropped, dimensions that are
// contiguous with one another merged) and picks one of three kernels:
//   * xfer_gather_kernel: the elements of the innermost dimension are next to one another in the source (row
//     slices, permuted outer dimensions, dense tensors at any offset), or no dimension has stride 1;
//   * xfer_tile_kernel: some other dimension has stride 1 (transposes): tiles through shared memory;
//   * xfer_element_kernel: tensors of up to 2048 elements per SM, and single bytes in short rows.

__device__ __forceinline__ uint64_t div_u64(uint64_t a, uint64_t b) {
  if (((a | b) >> 32) == 0) return (uint32_t)a / (uint32_t)b;  // most tensors; a 64-bit division costs several times as much
  return a / b;
}

// NB bytes from any address, as aligned 16-byte loads of just the granules that hold them, and a byte shift.
template <int NB>
__device__ __forceinline__ void load_span(const unsigned char* p, uint32_t (&out)[NB / 4]) {
  constexpr int NW = NB / 4;
  constexpr int NL = (NB + 15) / 16;  // granules when aligned; one more otherwise
  const uint32_t off = (uint32_t)(uintptr_t)p & 15u;
  const uint4* base = reinterpret_cast<const uint4*>(p - off);
  uint32_t w[4 * (NL + 1)];
#pragma unroll
  for (int i = 0; i <= NL; ++i) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (i < NL ? true : off + NB > 16 * NL) v = base[i];
    w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < NW + 2; ++i) w[i] = (off & 8u) ? (i + 2 < 4 * (NL + 1) ? w[i + 2] : 0u) : w[i];
#pragma unroll
  for (int i = 0; i < NW + 1; ++i) w[i] = (off & 4u) ? w[i + 1] : w[i];
  const uint32_t sh = (off & 3u) * 8u;
#pragma unroll
  for (int i = 0; i < NW; ++i) out[i] = __funnelshift_r(w[i], w[i + 1], sh);
}

// One element of the source as one of the destination: the bits themselves (RAW), or handler and cast.
template <typename S, typename D, bool RAW>
struct Convert;
template <typename S, typename D>
struct Convert<S, D, true> {
  static __device__ __forceinline__ D one(S v, int, float) { return v; }
};
template <typename S, typename D>
struct Convert<S, D, false> {
  static __device__ __forceinline__ D one(S v, int op, float arg) { return Elem<D>::from(apply_op(Elem<S>::to(v), op, arg)); }
};

// Division of any 32-bit number by one that the host knows: a multiplication and shifts (Granlund and Montgomery,
// "Division by invariant integers using multiplication", 1994, figure 4.1).
struct FastDiv {
  uint32_t m, s1, s2;
  __device__ __forceinline__ uint32_t operator()(uint32_t a) const {
    const uint32_t t = __umulhi(a, m);
    return (t + ((a - t) >> s1)) >> s2;
  }
};
struct GatherArgs {
  XferArgs x;
  FastDiv div[EUX_MAX_DIMS];  // by the sizes
  int small;                  // every size, and the number of elements, fits 32 bits: `div` can be used
};

// Offset in the source, in elements, of the row (every dimension but the innermost) and the column of element e.
// (With plain 32-bit divisions a head-major view, four dimensions, was bound by them: 158 us for 16 x 32 x 2048 x 128.)
__device__ __forceinline__ int64_t gather_row(const GatherArgs& a, uint64_t e, uint64_t& col) {
  const eux_xfer_desc& d = a.x.d;
  const int last = d.ndim - 1;
  auto divide = [&](uint64_t v, int k) -> uint64_t { return a.small ? a.div[k]((uint32_t)v) : v / (uint64_t)d.shape[k]; };
  uint64_t rem = divide(e, last);
  col = e - rem * (uint64_t)d.shape[last];
  int64_t off = 0;
  for (int k = last - 1; k >= 0; --k) {
    const uint64_t q = divide(rem, k);
    off += (int64_t)(rem - q * (uint64_t)d.shape[k]) * d.stride[k];
    rem = q;
  }
  return off;
}

// A thread makes 16 (8 for a narrowing cast to one byte, 32 for one to fp32) aligned bytes of the destination per
// chunk, and U chunks per step, whose loads are all in flight together. ALIGNED: every row of the source starts on the
// load's boundary and is a whole number of chunks long, so a chunk is one aligned load (two for fp32 sources).
// Otherwise a chunk takes one or two aligned loads when it lies in one row, and single elements when it straddles rows
// or the innermost stride is not 1. Bound by DRAM and, with rows of a few hundred bytes, by the index computation.
template <typename S, typename D, bool RAW, bool ALIGNED>
__global__ void __launch_bounds__(kXferThreads) xfer_gather_kernel(const __grid_constant__ GatherArgs a) {
  const eux_xfer_desc& d = a.x.d;
  xfer_begin(d);
  bool ok = cta_wait_arrival(d);
  if (ok) {
    constexpr int V = RAW ? 16 / (int)sizeof(D) : 8;
    constexpr int U = ALIGNED ? (V * (int)sizeof(S) > 16 ? 2 : 4) : 1;  // two unaligned chunks spill: 59 -> 70 us on 8192 rows of 5461 bf16
    constexpr int DB = V * (int)sizeof(D);
    constexpr int SB = V * (int)sizeof(S);
    constexpr int VEC = DB >= 16 ? 16 : 8;
    constexpr int SVEC = SB >= 16 ? 16 : 8;
    const S* src = reinterpret_cast<const S*>(d.src);
    D* dst = reinterpret_cast<D*>(d.dst);
    const uint64_t n = d.n_elems;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t cols = (uint64_t)d.shape[d.ndim - 1];
    const int64_t inner = d.stride[d.ndim - 1];
    const int op = d.op;
    const float arg = d.op_arg;
    uint64_t lead = ALIGNED ? 0 : ((VEC - ((uintptr_t)dst & (VEC - 1))) & (VEC - 1)) / sizeof(D);  // elements in front of the first aligned vector
    if (lead > n) lead = n;
    const uint64_t chunks = (n - lead) / V;
    for (uint64_t i0 = tid; i0 < chunks; i0 += U * nthreads) {
      alignas(16) uint32_t w[U][SB / 4];
      uint64_t c[U];
      int64_t row[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t i = i0 + u * nthreads;
        if (i >= chunks) break;
        row[u] = gather_row(a, lead + i * V, c[u]);
        const S* s = src + row[u] + (int64_t)c[u];
        if (ALIGNED) {
#pragma unroll
          for (int k = 0; k < SB / SVEC; ++k)
            reinterpret_cast<typename PackT<SVEC>::type*>(w[u])[k] = reinterpret_cast<const typename PackT<SVEC>::type*>(s)[k];
        } else if (inner == 1 && c[u] + V <= cols) {
          load_span<SB>(reinterpret_cast<const unsigned char*>(s), w[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t i = i0 + u * nthreads;
        if (i >= chunks) break;
        const uint64_t e = lead + i * V;
        alignas(16) D out[V];
        if (ALIGNED || (inner == 1 && c[u] + V <= cols)) {
          const S* sv = reinterpret_cast<const S*>(w[u]);
#pragma unroll
          for (int k = 0; k < V; ++k) out[k] = Convert<S, D, RAW>::one(sv[k], op, arg);
        } else {
          uint64_t col = c[u];
          int64_t r = row[u];
#pragma unroll
          for (int k = 0; k < V; ++k) {
            if (col >= cols) r = gather_row(a, e + k, col);
            out[k] = Convert<S, D, RAW>::one(src[r + (int64_t)col * inner], op, arg);
            ++col;
          }
        }
#pragma unroll
        for (int k = 0; k < DB / VEC; ++k)
          reinterpret_cast<typename PackT<VEC>::type*>(dst + e)[k] = reinterpret_cast<typename PackT<VEC>::type*>(out)[k];
      }
    }
    const uint64_t tail = lead + chunks * V;  // single elements in front of the vectors and behind them
    for (uint64_t i = tid; i < lead + (n - tail); i += nthreads) {
      const uint64_t e = i < lead ? i : tail + (i - lead);
      uint64_t c;
      const int64_t row = gather_row(a, e, c);
      dst[e] = Convert<S, D, RAW>::one(src[row + (int64_t)c * inner], op, arg);
    }
  }
  xfer_end(d, a.x.counter, ok);
}

// Small tensors (a step for every thread of the device, or less), and single bytes in rows of less than a chunk: one
// element per thread at a time, four in flight, neighbouring threads on neighbouring elements. Bound by one trip to memory
// and by the index arithmetic; the chunked kernel's unrolled row crossings are long, cold code to a launch that runs them
// once (1000 matrices of 3 x 3 bytes, transposed: 12.5 us in chunks, 4.1 here; with a 64-bit division per dimension, as
// every strided element once had, 7.0).
template <typename S, typename D, bool RAW>
__global__ void __launch_bounds__(kXferThreads) xfer_element_kernel(const __grid_constant__ GatherArgs a) {
  const eux_xfer_desc& d = a.x.d;
  xfer_begin(d);
  const bool ok = cta_wait_arrival(d);
  if (ok) {
    constexpr int U = 4;
    const S* src = reinterpret_cast<const S*>(d.src);
    D* dst = reinterpret_cast<D*>(d.dst);
    const uint64_t n = d.n_elems;
    const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
    const int64_t inner = d.stride[d.ndim - 1];
    const int op = d.op;
    const float arg = d.op_arg;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += U * nthreads) {
      S v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (i0 + u * nthreads >= n) break;
        uint64_t col;
        const int64_t row = gather_row(a, i0 + u * nthreads, col);
        v[u] = src[row + (int64_t)col * inner];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (i0 + u * nthreads >= n) break;
        dst[i0 + u * nthreads] = Convert<S, D, RAW>::one(v[u], op, arg);
      }
    }
  }
  xfer_end(d, a.x.counter, ok);
}

// Transposes. A tile is `tp` steps of the dimension with stride 1 in the source (P) times `tq` of the innermost
// dimension (Q): it is read along P, with 16-byte loads where the rows' alignment allows them (VECTOR) and element
// by element otherwise, converted, and kept in shared memory as words of G = 4 / sizeof(D) neighbours along Q, so
// that 1- and 2-byte elements are transposed within registers and shared memory only ever moves whole words. The
// row pitch is odd, so reads and writes meet at most two-way bank conflicts. Rows of Q leave as 16-byte stores, or
// element by element where the destination's rows are not 16-byte aligned.
// The usual tile, TP steps by QW words, has its sizes and trip counts at compile time and all its loads in flight at
// once; with sizes read at run time throughout, the index arithmetic alone kept the issue slots two thirds busy
// (8192 x 8192 bf16: 73 us). Tiles at the edges and of other shapes take the general loops.
constexpr int kTileThreads = 256;
template <typename S>
constexpr int tile_p() { return sizeof(S) == 1 ? 128 : 64; }  // every thread has a 16-byte load
// Words of Q: 256 bytes of a destination row where loads are 16 bytes wide (8192 x 8192 bf16: 56 us with 128 bytes, 47
// with 256), 128 otherwise (8191 x 8193 bytes: 64 us; with 256 it took 1.4 times as long).
constexpr int tile_q(bool vector) { return vector ? 64 : 32; }
constexpr int kNarrowBytes = 24576;
constexpr int kTileWords = 64 * 33;  // of a tile of any other shape
struct TileArgs {
  XferArgs x;
  int64_t batch_src[EUX_MAX_DIMS], batch_dst[EUX_MAX_DIMS];  // strides of the other dimensions, in elements
  uint32_t batch_shape[EUX_MAX_DIMS];
  int64_t q_src, p_dst;  // strides, in elements
  uint32_t n_batch, np, nq, tp, tq, tiles_p, tiles_q;
  uint32_t pitch;  // words
  uint32_t vector_store, narrow;
  uint64_t tiles;
};

template <typename S, typename D, bool RAW>
__device__ __forceinline__ uint32_t tile_word(const S* v, int op, float arg) {
  constexpr int G = 4 / (int)sizeof(D);
  alignas(4) D o[G];
#pragma unroll
  for (int g = 0; g < G; ++g) o[g] = Convert<S, D, RAW>::one(v[g], op, arg);
  uint32_t word;
  memcpy(&word, o, 4);
  return word;
}

template <typename S, typename D, bool RAW, bool VECTOR>
__global__ void __launch_bounds__(kTileThreads) xfer_tile_kernel(const __grid_constant__ TileArgs t) {
  constexpr int G = 4 / (int)sizeof(D);
  constexpr int VP = VECTOR ? 16 / (int)sizeof(S) : 1;
  constexpr int TP = tile_p<S>();
  constexpr int QW = tile_q(VECTOR);  // words of Q in a full tile
  constexpr uint32_t PITCH = QW + 1;
  __shared__ uint32_t sm[TP * PITCH > kTileWords ? TP * PITCH : kTileWords];
  const eux_xfer_desc& d = t.x.d;
  wait_for_launch_before();
  const bool ok = cta_wait_arrival(d);
  if (ok) {
    const int op = d.op;
    const float arg = d.op_arg;
    for (uint64_t tile = blockIdx.x; tile < t.tiles; tile += gridDim.x) {
      // neighbouring tiles along P first: they share the source's lines where rows are not aligned to lines
      uint64_t r = div_u64(tile, t.tiles_p);
      const uint32_t p0 = (uint32_t)(tile - r * t.tiles_p) * t.tp;
      uint64_t b = div_u64(r, t.tiles_q);
      const uint32_t q0 = (uint32_t)(r - b * t.tiles_q) * t.tq;
      int64_t so = (int64_t)p0 + (int64_t)q0 * t.q_src;
      int64_t dof = (int64_t)p0 * t.p_dst + (int64_t)q0;
      for (int k = (int)t.n_batch - 1; k >= 0; --k) {
        const uint64_t bq = div_u64(b, t.batch_shape[k]);
        const int64_t ix = (int64_t)(b - bq * t.batch_shape[k]);
        so += ix * t.batch_src[k];
        dof += ix * t.batch_dst[k];
        b = bq;
      }
      const S* src = reinterpret_cast<const S*>(d.src) + so;
      D* dst = reinterpret_cast<D*>(d.dst) + dof;
      const uint32_t pn = min(t.tp, t.np - p0), qn = min(t.tq, t.nq - q0);
      const int64_t q_src = t.q_src;

      // ---- read ----
      if (pn == TP && qn == QW * G) {
        constexpr int PU = TP / VP;                    // units along P
        constexpr int QSTEP = kTileThreads / PU;       // words of Q that one pass of the threads covers
        constexpr int N = QW / QSTEP;                  // passes
        constexpr int B = G * VP * (int)sizeof(S) * N <= 64 ? N : (N > 1 && G * VP * (int)sizeof(S) * N / 2 <= 64 ? N / 2 : 1);  // in flight
        const uint32_t p = (threadIdx.x % PU) * VP, w0 = threadIdx.x / PU;
        const S* s = src + (int64_t)(w0 * G) * q_src + p;
#pragma unroll
        for (int n0 = 0; n0 < N; n0 += B) {
          alignas(16) S v[B][G][VP];
#pragma unroll
          for (int n = 0; n < B; ++n)
#pragma unroll
            for (int g = 0; g < G; ++g) {
              const S* e = s + (int64_t)((n0 + n) * QSTEP * G + g) * q_src;
              if (VECTOR) *reinterpret_cast<uint4*>(v[n][g]) = *reinterpret_cast<const uint4*>(e);
              else v[n][g][0] = *e;
            }
#pragma unroll
          for (int n = 0; n < B; ++n)
#pragma unroll
            for (int i = 0; i < VP; ++i) {
              S col[G];
#pragma unroll
              for (int g = 0; g < G; ++g) col[g] = v[n][g][i];
              sm[(p + i) * PITCH + w0 + (n0 + n) * QSTEP] = tile_word<S, D, RAW>(col, op, arg);
            }
        }
      } else {
        // a unit is VP steps of P by G of Q, B of them in flight; unit indexes are kept split so that no step divides
        constexpr int B = VECTOR ? 1 : 4;
        const uint32_t pu = (pn + VP - 1) / VP, qw = (qn + G - 1) / G, pitch = t.pitch;
        const uint32_t dq = kTileThreads / pu, dp = kTileThreads - dq * pu;
        uint32_t iq = threadIdx.x / pu, ip = threadIdx.x - iq * pu;
        while (iq < qw) {
          alignas(16) S v[B][G][VP];
          uint32_t at[B], steps[B];
#pragma unroll
          for (int n = 0; n < B; ++n) {
            const uint32_t p = ip * VP;
            steps[n] = iq >= qw ? 0 : min((uint32_t)VP, pn - p);
            at[n] = p * pitch + iq;
            const S* s = src + (int64_t)(iq * G) * q_src + p;
#pragma unroll
            for (int g = 0; g < G; ++g) {
              if (VECTOR && iq * G + g < qn && steps[n] == VP) {
                *reinterpret_cast<uint4*>(v[n][g]) = *reinterpret_cast<const uint4*>(s + g * q_src);
              } else {
#pragma unroll
                for (int i = 0; i < VP; ++i) {
                  if (iq * G + g < qn && i < (int)steps[n]) v[n][g][i] = s[g * q_src + i];
                  else memset(&v[n][g][i], 0, sizeof(S));
                }
              }
            }
            ip += dp;
            iq += dq;
            if (ip >= pu) ip -= pu, ++iq;
          }
#pragma unroll
          for (int n = 0; n < B; ++n)
#pragma unroll
            for (int i = 0; i < VP; ++i) {
              S col[G];
#pragma unroll
              for (int g = 0; g < G; ++g) col[g] = v[n][g][i];
              if (i < (int)steps[n]) sm[at[n] + i * pitch] = tile_word<S, D, RAW>(col, op, arg);
            }
        }
      }
      __syncthreads();

      // ---- write ----
      const uint32_t pitch = t.pitch;
      if (t.vector_store && pn == TP && qn == QW * G) {
        constexpr int VR = QW / 4;  // vectors per row
        constexpr int RSTEP = kTileThreads / VR;
        const uint32_t v = threadIdx.x % VR, row0 = threadIdx.x / VR;
        const uint32_t* w = sm + row0 * PITCH + v * 4;
        D* out = dst + (int64_t)row0 * t.p_dst + v * (16 / sizeof(D));
#pragma unroll
        for (int n = 0; n < TP / RSTEP; ++n) {
          const uint32_t* wn = w + n * RSTEP * PITCH;
          *reinterpret_cast<uint4*>(out + (int64_t)(n * RSTEP) * t.p_dst) = make_uint4(wn[0], wn[1], wn[2], wn[3]);
        }
      } else if (t.vector_store) {
        constexpr uint32_t E = 16 / sizeof(D);
        const uint32_t vr = (qn + E - 1) / E;
        const uint32_t dr = kTileThreads / vr, dv = kTileThreads - dr * vr;
        uint32_t row = threadIdx.x / vr, v = threadIdx.x - row * vr;
        while (row < pn) {
          const uint32_t* w = sm + row * pitch + v * 4;
          D* out = dst + (int64_t)row * t.p_dst + v * E;
          if (v * E + E <= qn) {
            *reinterpret_cast<uint4*>(out) = make_uint4(w[0], w[1], w[2], w[3]);
          } else {
            for (uint32_t i = 0; v * E + i < qn; ++i) {
              const uint32_t word = w[i / G] >> (8 * sizeof(D) * (i % G));
              memcpy(out + i, &word, sizeof(D));
            }
          }
          row += dr;
          v += dv;
          if (v >= vr) v -= vr, ++row;
        }
      } else if (pn == TP && qn == QW * G) {
        constexpr int RSTEP = kTileThreads / (QW * G);  // rows that one pass of the threads covers
        const uint32_t q = threadIdx.x % (QW * G), row0 = threadIdx.x / (QW * G);
        const uint32_t* w = sm + row0 * PITCH + q / G;
        const uint32_t shift = 8 * sizeof(D) * (q % G);
        D* out = dst + (int64_t)row0 * t.p_dst + q;
#pragma unroll 8
        for (int n = 0; n < TP / RSTEP; ++n) {
          const uint32_t word = w[n * RSTEP * PITCH] >> shift;
          memcpy(out + (int64_t)(n * RSTEP) * t.p_dst, &word, sizeof(D));
        }
      } else {
        const uint32_t dr = kTileThreads / qn, dq = kTileThreads - dr * qn;
        uint32_t row = threadIdx.x / qn, q = threadIdx.x - row * qn;
#pragma unroll 4
        while (row < pn) {
          const uint32_t word = sm[row * pitch + q / G] >> (8 * sizeof(D) * (q % G));
          memcpy(dst + (int64_t)row * t.p_dst + q, &word, sizeof(D));
          row += dr;
          q += dq;
          if (q >= qn) q -= qn, ++row;
        }
      }
      __syncthreads();
    }
  }
  xfer_end(d, t.x.counter, ok);
}

// Transposes of a dense matrix with few columns (P below 64, rows of the source next to one another): the source of a
// tile, all of P by `tq` of Q, is one contiguous range. It comes in 16 bytes per thread, whatever its alignment, and is
// taken apart on the way out: a thread makes 16 bytes of one row of the destination from elements P apart in shared
// memory. (With element loads, as in the tile kernel, index arithmetic is the bound: 2^24 x 3 bf16 took 119 us.)
template <typename S, typename D, bool RAW>
__global__ void __launch_bounds__(kTileThreads) xfer_narrow_kernel(const __grid_constant__ TileArgs t) {
  __shared__ __align__(16) unsigned char sm[kNarrowBytes];
  const eux_xfer_desc& d = t.x.d;
  wait_for_launch_before();
  const bool ok = cta_wait_arrival(d);
  if (ok) {
    constexpr uint32_t E = 16 / sizeof(D);
    const int op = d.op;
    const float arg = d.op_arg;
    const uint32_t np = t.np;
    const S* el = reinterpret_cast<const S*>(sm);
    for (uint64_t tile = blockIdx.x; tile < t.tiles; tile += gridDim.x) {
      const uint32_t q0 = (uint32_t)tile * t.tq;
      const uint32_t qn = min(t.tq, t.nq - q0);
      const unsigned char* src = reinterpret_cast<const unsigned char*>(reinterpret_cast<const S*>(d.src) + (uint64_t)q0 * np);
      D* dst = reinterpret_cast<D*>(d.dst) + q0;
      const uint32_t bytes = qn * np * (uint32_t)sizeof(S);
#pragma unroll 2
      for (uint32_t o = threadIdx.x * 16; o + 16 <= bytes; o += kTileThreads * 16) {
        uint32_t w[4];
        load_span<16>(src + o, w);
        *reinterpret_cast<uint4*>(sm + o) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      for (uint32_t e = (bytes & ~15u) / sizeof(S) + threadIdx.x; e < qn * np; e += kTileThreads)
        reinterpret_cast<S*>(sm)[e] = reinterpret_cast<const S*>(src)[e];
      __syncthreads();
      if (t.vector_store) {
        // With eight or more rows a warp covers eight of them by 64 bytes: neighbouring rows are neighbours in shared
        // memory, where vectors of one row may be any number of banks apart (2^21 x 20 bf16: 16-way conflicts).
        const uint32_t vr = (qn + E - 1) / E, pb = np >= 8 ? 8 : 1;
        const uint32_t p_groups = (np + pb - 1) / pb, units = p_groups * pb * ((vr + 3) & ~3u);
        for (uint32_t u = threadIdx.x; u < units; u += kTileThreads) {
          uint32_t p, v;
          if (pb == 8) {
            const uint32_t r = u >> 5, g = r / p_groups;
            p = (r - g * p_groups) * 8 + (u & 7), v = g * 4 + ((u >> 3) & 3);
          } else {
            const uint32_t vs = (vr + 3) & ~3u;
            p = u / vs, v = u - p * vs;
          }
          if (p < np && v < vr) {
            const S* s = el + (v * E) * np + p;
            D* out = dst + (int64_t)p * t.p_dst + v * E;
            if (v * E + E <= qn) {
              alignas(16) D o[E];
#pragma unroll
              for (int k = 0; k < (int)E; ++k) o[k] = Convert<S, D, RAW>::one(s[k * np], op, arg);
              *reinterpret_cast<uint4*>(out) = *reinterpret_cast<uint4*>(o);
            } else {
              for (uint32_t k = 0; v * E + k < qn; ++k) out[k] = Convert<S, D, RAW>::one(s[k * np], op, arg);
            }
          }
        }
      } else {
        for (uint32_t p = 0; p < np; ++p)
#pragma unroll 4
          for (uint32_t q = threadIdx.x; q < qn; q += kTileThreads)
            dst[(int64_t)p * t.p_dst + q] = Convert<S, D, RAW>::one(el[q * np + p], op, arg);
      }
      __syncthreads();
    }
  }
  xfer_end(d, t.x.counter, ok);
}

// One CTA per descriptor; meant for many small messages per launch.
__global__ void __launch_bounds__(256) xfer_batch_kernel(const eux_xfer_desc* descs, int n) {
  if ((int)blockIdx.x >= n) return;
  __shared__ eux_xfer_desc d;
  {
    const uint32_t* s = reinterpret_cast<const uint32_t*>(descs + blockIdx.x);
    uint32_t* t = reinterpret_cast<uint32_t*>(&d);
    for (int i = threadIdx.x; i < (int)(sizeof(eux_xfer_desc) / 4); i += blockDim.x) t[i] = s[i];
  }
  __syncthreads();
  bool ok = true;
  if (d.wait_flag) {
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
      bool w = wait_flag_ge(d.wait_flag, d.wait_value, d.wait_timeout_ns);
      if (!w) set_status(d.status, EUX_ST_TIMEOUT, 2);
      s_ok = w;
    }
    __syncthreads();
    ok = s_ok != 0;
  }
  if (ok) {
    const uint64_t esz = (uint64_t)dtype_size(d.src_dtype);
    const bool dense = d.ndim == 0;
    const bool raw = d.src_dtype == d.dst_dtype && d.op == EUX_OP_NONE;
    const bool al16 = ((((uintptr_t)d.src) | ((uintptr_t)d.dst)) & 15u) == 0;
    if (dense && raw && al16) {
      copy_bytes_grid<false>(reinterpret_cast<const unsigned char*>(d.src), reinterpret_cast<unsigned char*>(d.dst),
                             d.n_elems * esz, 0, 1);
    } else if (dense && al16 && d.src_dtype == EUX_DT_F32 && d.dst_dtype == EUX_DT_F32) {
      const float4* s = reinterpret_cast<const float4*>(d.src);
      float4* t = reinterpret_cast<float4*>(d.dst);
      const uint64_t n4 = d.n_elems >> 2;
      for (uint64_t i = threadIdx.x; i < n4; i += blockDim.x) {
        float4 v = __ldcg(s + i);
        v.x = apply_op(v.x, d.op, d.op_arg);
        v.y = apply_op(v.y, d.op, d.op_arg);
        v.z = apply_op(v.z, d.op, d.op_arg);
        v.w = apply_op(v.w, d.op, d.op_arg);
        t[i] = v;
      }
      for (uint64_t e = (n4 << 2) + threadIdx.x; e < d.n_elems; e += blockDim.x)
        reinterpret_cast<float*>(d.dst)[e] = apply_op(reinterpret_cast<const float*>(d.src)[e], d.op, d.op_arg);
    } else {
      for (uint64_t e = threadIdx.x; e < d.n_elems; e += blockDim.x) {
        uint64_t rem = e;
        int64_t off = dense ? (int64_t)e : 0;
        if (!dense)
          for (int k = d.ndim - 1; k >= 0; --k) {
            uint64_t q = rem / (uint64_t)d.shape[k];
            off += (int64_t)(rem - q * (uint64_t)d.shape[k]) * d.stride[k];
            rem = q;
          }
        if (raw) {
          const unsigned char* s = reinterpret_cast<const unsigned char*>(d.src) + off * esz;
          unsigned char* t = reinterpret_cast<unsigned char*>(d.dst) + e * esz;
          for (uint64_t b = 0; b < esz; ++b) t[b] = s[b];
        } else {
          store_from_float(d.dst, e, d.dst_dtype,
                           apply_op(load_as_float(d.src, (uint64_t)off, d.src_dtype), d.op, d.op_arg));
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && ok && d.flag) {
    __threadfence_system();
    st_relaxed_sys(d.flag, d.flag_value);
  }
}

// ---------------------------------------------------------------------------
// Device-driven ping-pong: both GPUs run this kernel at the same time (one
// launch per GPU, never two on the same GPU). The initiator pushes its buffer
// into the peer's buffer and publishes seq; the echo side waits for seq,
// pushes the received bytes back and publishes seq on the initiator.
// initiator == 2 is a single-GPU loopback (no flags, peer_buf is local).
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool grid_barrier(uint32_t* bar, uint32_t& gen, uint64_t timeout_ns) {
  __syncthreads();
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    __threadfence_system();
    gen += 1;
    atomicAdd(bar, 1u);
    s_ok = wait_u32_ge_gpu(bar, gen * gridDim.x, timeout_ns);
  }
  __syncthreads();
  return s_ok != 0;
}

__global__ void __launch_bounds__(kXferThreads) pingpong_kernel(eux_pingpong_desc d) {
  uint32_t gen = 0;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
  __shared__ int s_ok;
  bool alive = true;
  for (int it = 0; it < d.iters && alive; ++it) {
    const uint64_t seq = d.base_seq + 1 + (uint64_t)it;
    if (d.ts_out && tid == 0) d.ts_out[it] = globaltimer_ns();
    if (d.initiator == 0) {
      if (threadIdx.x == 0) s_ok = wait_flag_ge(d.local_flag, seq, d.wait_timeout_ns);
      __syncthreads();
      if (!s_ok) { alive = false; break; }
    }
    copy_bytes_grid<false>(reinterpret_cast<const unsigned char*>(d.local_buf), reinterpret_cast<unsigned char*>(d.peer_buf),
                           d.nbytes, blockIdx.x, gridDim.x);
    if (!grid_barrier(d.grid_bar, gen, d.wait_timeout_ns)) { alive = false; break; }
    if (d.initiator == 2) {
      copy_bytes_grid<false>(reinterpret_cast<const unsigned char*>(d.peer_buf), reinterpret_cast<unsigned char*>(d.local_buf),
                             d.nbytes, blockIdx.x, gridDim.x);
      if (!grid_barrier(d.grid_bar, gen, d.wait_timeout_ns)) { alive = false; break; }
      continue;
    }
    if (tid == 0) st_release_sys(d.peer_flag, seq);
    if (d.initiator == 1) {
      if (threadIdx.x == 0) s_ok = wait_flag_ge(d.local_flag, seq, d.wait_timeout_ns);
      __syncthreads();
      if (!s_ok) { alive = false; break; }
    }
  }
  if (!alive && threadIdx.x == 0) set_status(d.status, EUX_ST_TIMEOUT, 3);
  if (d.ts_out && tid == 0) d.ts_out[d.iters] = globaltimer_ns();
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t old = atomicAdd(d.grid_bar + 1, 1u);
    if (old == gridDim.x - 1) {
      d.grid_bar[0] = 0;
      d.grid_bar[1] = 0;
      __threadfence();
    }
  }
}

static int num_sms() {
  static int sms[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (sms[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    sms[dev] = n;
  }
  return sms[dev];
}

// Transfers are launched while the kernel before them ends (calls in a loop, without that and with it: 4096 x 7168 fp32 to
// e4m3 24.9 and 23.4 us, 4096 x 4096 bf16 to e4m3 8.2 and 7.0). One that waits for an arrival is launched when
// its turn has come: until then it would hold its SMs for nothing.
template <typename A>
static void launch_xfer(void (*kernel)(A), int grid, int threads, cudaStream_t st, const A& a, const eux_xfer_desc& d) {
  if (d.wait_flag) kernel<<<grid, threads, 0, st>>>(a);
  else launch_early(kernel, grid, threads, 0, st, a);
}

template <typename S>
static int launch_typed(const XferArgs& a, int grid, cudaStream_t st) {
  switch (a.d.dst_dtype) {
    case EUX_DT_F32: launch_xfer(xfer_typed_kernel<S, float>, grid, kXferThreads, st, a, a.d); break;
    case EUX_DT_F16: launch_xfer(xfer_typed_kernel<S, __half>, grid, kXferThreads, st, a, a.d); break;
    case EUX_DT_BF16: launch_xfer(xfer_typed_kernel<S, __nv_bfloat16>, grid, kXferThreads, st, a, a.d); break;
    case EUX_DT_F8E4M3: launch_xfer(xfer_typed_kernel<S, __nv_fp8_e4m3>, grid, kXferThreads, st, a, a.d); break;
    default: return EUX_ERR_BAD_ARG;
  }
  return 0;
}

// The layout with as few dimensions as describe it. False: it describes nothing (a size below 1, or a size that
// does not multiply up to the number of elements): the caller's own words are then followed as they stand.
static bool collapse(eux_xfer_desc& d) {
  uint64_t prod = 1;
  for (int i = 0; i < d.ndim; ++i) {
    if (d.shape[i] < 1 || __builtin_mul_overflow(prod, (uint64_t)d.shape[i], &prod)) return false;
  }
  if (prod != d.n_elems || prod >> 62) return false;
  int nd = 0;
  for (int i = 0; i < d.ndim; ++i) {
    if (d.shape[i] == 1) continue;
    int64_t span;
    if (nd > 0 && !__builtin_mul_overflow(d.shape[i], d.stride[i], &span) && d.stride[nd - 1] == span) {
      d.shape[nd - 1] *= d.shape[i];  // the outer one steps over the whole of the inner one: one dimension
      d.stride[nd - 1] = d.stride[i];
    } else {
      d.shape[nd] = d.shape[i];
      d.stride[nd] = d.stride[i];
      ++nd;
    }
  }
  d.ndim = nd;
  if (nd == 0 || (nd == 1 && d.stride[0] == 1)) d.ndim = 0;
  return true;
}

static FastDiv fast_div(uint32_t d) {
  int l = 0;
  while (((uint64_t)1 << l) < d) ++l;
  FastDiv f;
  f.m = (uint32_t)(((uint64_t)1 << 32) * (((uint64_t)1 << l) - d) / d + 1);
  f.s1 = l > 0 ? 1 : 0, f.s2 = l > 0 ? l - 1 : 0;
  return f;
}

enum class Route { kElement, kGather, kGatherAligned, kTile, kTileVector, kNarrow };

template <typename S, typename D, bool RAW>
static void launch_gather(const GatherArgs& a, const TileArgs& t, Route route, int grid, cudaStream_t st) {
  switch (route) {
    case Route::kElement: launch_xfer(xfer_element_kernel<S, D, RAW>, grid, kXferThreads, st, a, a.x.d); break;
    case Route::kGather: launch_xfer(xfer_gather_kernel<S, D, RAW, false>, grid, kXferThreads, st, a, a.x.d); break;
    case Route::kGatherAligned: launch_xfer(xfer_gather_kernel<S, D, RAW, true>, grid, kXferThreads, st, a, a.x.d); break;
    case Route::kTile: launch_xfer(xfer_tile_kernel<S, D, RAW, false>, grid, kTileThreads, st, t, t.x.d); break;
    case Route::kTileVector: launch_xfer(xfer_tile_kernel<S, D, RAW, true>, grid, kTileThreads, st, t, t.x.d); break;
    case Route::kNarrow: launch_xfer(xfer_narrow_kernel<S, D, RAW>, grid, kTileThreads, st, t, t.x.d); break;
  }
}
template <typename S>
static int launch_gather_from(const GatherArgs& a, const TileArgs& t, Route route, int grid, cudaStream_t st) {
  switch (a.x.d.dst_dtype) {
    case EUX_DT_F32: launch_gather<S, float, false>(a, t, route, grid, st); break;
    case EUX_DT_F16: launch_gather<S, __half, false>(a, t, route, grid, st); break;
    case EUX_DT_BF16: launch_gather<S, __nv_bfloat16, false>(a, t, route, grid, st); break;
    case EUX_DT_F8E4M3: launch_gather<S, __nv_fp8_e4m3, false>(a, t, route, grid, st); break;
    case EUX_DT_BYTES: launch_xfer(xfer_element_kernel<S, uint8_t, false>, grid, kXferThreads, st, a, a.x.d); break;  // truncated
    default: return EUX_ERR_BAD_ARG;
  }
  return 0;
}

// Fills `t` when the layout is a transpose the tile kernel takes: the innermost dimension is strided and another one
// has stride 1. (Without such a dimension every element has a line of its own and tiles would gain nothing.)
static bool plan_tiles(const eux_xfer_desc& d, TileArgs& t, bool& vector) {
  const int last = d.ndim - 1;
  if (d.ndim < 2 || d.stride[last] == 1) return false;
  int p = -1;
  for (int k = 0; k < last; ++k)
    if (d.stride[k] == 1) p = k;
  if (p < 0) return false;
  for (int k = 0; k < d.ndim; ++k)
    if (d.shape[k] > 0x7fffffff) return false;
  const int ssz = dtype_size(d.src_dtype), dsz = dtype_size(d.dst_dtype), g = 4 / dsz;
  t.np = (uint32_t)d.shape[p], t.nq = (uint32_t)d.shape[last];
  t.q_src = d.stride[last];
  bool store16 = ((uintptr_t)d.dst & 15u) == 0;
  vector = (((uintptr_t)d.src | (uint64_t)(t.q_src * ssz)) & 15u) == 0;
  uint64_t inner = 1, batch = 1;
  int64_t dst_stride[EUX_MAX_DIMS];
  for (int k = last; k >= 0; --k) {
    dst_stride[k] = (int64_t)inner;
    inner *= (uint64_t)d.shape[k];
  }
  t.n_batch = 0;
  for (int k = 0; k < last; ++k) {
    if ((dst_stride[k] * dsz) & 15) store16 = false;
    if (k == p) continue;
    if ((d.stride[k] * ssz) & 15) vector = false;
    t.batch_src[t.n_batch] = d.stride[k], t.batch_dst[t.n_batch] = dst_stride[k];
    t.batch_shape[t.n_batch++] = (uint32_t)d.shape[k];
    batch *= (uint64_t)d.shape[k];
  }
  t.p_dst = dst_stride[p];
  // TP steps of P by 128 or 256 bytes of Q; where one of the two is shorter the tile is as much longer in the other
  uint32_t qw_all = (t.nq + g - 1) / g, qw = tile_q(vector), tp = ssz == 1 ? tile_p<uint8_t>() : tile_p<uint16_t>();
  if (t.np < 64) {
    tp = t.np;
    qw = (uint32_t)(kTileWords / tp - 1) & ~3u;
    if (qw > qw_all) qw = qw_all;
  } else if (qw_all < qw) {
    qw = qw_all;
    tp = ((uint32_t)kTileWords / (qw | 1u)) & ~15u;  // whole vectors of P
    if (tp > t.np) tp = t.np;
  }
  t.pitch = qw | 1u;
  t.tp = tp, t.tq = qw * g < t.nq ? qw * g : t.nq;
  t.tiles_p = (t.np + tp - 1) / tp, t.tiles_q = (t.nq + t.tq - 1) / t.tq;
  t.narrow = d.ndim == 2 && t.np < 64 && t.q_src == (int64_t)t.np && t.nq >= 1024;
  if (t.narrow) {
    t.tq = (uint32_t)(kNarrowBytes / (t.np * ssz)) & ~15u;  // whole vectors of Q
    if (t.tq > 2048) t.tq = 2048;
    t.tiles_q = (t.nq + t.tq - 1) / t.tq;
  }
  t.tiles = batch * t.tiles_p * t.tiles_q;
  t.vector_store = store16;
  // A tile costs a CTA two barriers and its index set-up however small it is. In tiles and in chunks, bf16: 2^20 matrices of
  // 3 x 3 2821 and 45 us, 2^14 of 32 x 32 52 and 25, 2^12 of 64 x 64 21 and 25 (fp32: 60 and 45, 25 and 50).
  return batch == 1 || (uint64_t)t.np * t.nq >= 1280;
}

// Whether every chunk of `chunk` elements is one aligned load of the source and one aligned store.
static bool rows_aligned(const eux_xfer_desc& d, bool whole, int chunk, int ssz, int dsz) {
  if (!whole || d.stride[d.ndim - 1] != 1 || d.shape[d.ndim - 1] % chunk) return false;
  const uint64_t load = chunk * ssz >= 16 ? 16 : 8, store = chunk * dsz >= 16 ? 16 : 8;
  if ((uintptr_t)d.src % load || (uintptr_t)d.dst % store) return false;
  for (int k = 0; k + 1 < d.ndim; ++k)
    if ((uint64_t)(d.stride[k] * ssz) % load) return false;
  return true;
}

}  // namespace eux

using namespace eux;

extern "C" int eux_xfer_launch(const eux_xfer_desc* d, uint32_t* scratch_counter, int max_ctas, void* stream) {
  if (!d || !d->src || !d->dst || d->ndim < 0 || d->ndim > EUX_MAX_DIMS) return EUX_ERR_BAD_ARG;
  if (d->src_dtype == EUX_DT_BYTES && (d->dst_dtype != EUX_DT_BYTES || d->op != EUX_OP_NONE)) return EUX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  XferArgs a{*d, scratch_counter};
  const int sms = num_sms();
  const bool ctas_given = max_ctas > 0;
  if (!ctas_given) max_ctas = 2 * sms;
  const bool raw = d->src_dtype == d->dst_dtype && d->op == EUX_OP_NONE;
  const bool whole = collapse(a.d);
  const int ssz = dtype_size(d->src_dtype), dsz = dtype_size(d->dst_dtype);
  const uintptr_t al = ((uintptr_t)d->src) | ((uintptr_t)d->dst);
  auto limit = [&](uint64_t want) { return (int)(want < 1 ? 1 : (want > (uint64_t)max_ctas ? max_ctas : want)); };
  // Floating-point elements as bytes: an unaligned source or one described by a layout is taken, an aligned dense one is not.
  const bool to_bytes = d->dst_dtype == EUX_DT_BYTES && !raw;
  if (d->ndim > 0 && !scratch_counter && d->n_elems > (uint64_t)kXferThreads * 4 && max_ctas > 1) return EUX_ERR_BAD_ARG;
  int grid;
  if (a.d.ndim == 0 && raw && (al & 15u) == 0) {
    // 64 B per thread per step, one CTA per SM; small messages stay on one CTA (no counter traffic)
    if (!ctas_given) max_ctas = sms;
    grid = limit((d->n_elems * (uint64_t)ssz + (uint64_t)kXferThreads * 64 - 1) / ((uint64_t)kXferThreads * 64));
    if (grid > 1 && !scratch_counter) return EUX_ERR_BAD_ARG;
    if ((al & 31u) == 0) launch_xfer(xfer_bytes_kernel<true>, grid, kXferThreads, st, a, a.d);
    else launch_xfer(xfer_bytes_kernel<false>, grid, kXferThreads, st, a, a.d);
  } else if (a.d.ndim == 0 && d->src_dtype != EUX_DT_BYTES && (al & 15u) == 0 && !(to_bytes && d->ndim > 0)) {
    // two CTAs per SM carry enough bytes when the source is fp32 (4096 x 7168 to e4m3: 25 us, 29 with four), narrower ones take four
    // (narrow sources have 32 registers, fp32 ones up to 58). One that waits for its arrival keeps to half of an SM: kernels
    // of other streams, the one that it waits for perhaps among them, find room.
    if (!ctas_given) max_ctas = (d->wait_flag ? 1 : 2) * (ssz == 4 ? 1 : 2) * sms;
    grid = limit((d->n_elems / 8 + kXferThreads - 1) / kXferThreads);
    if (grid > 1 && !scratch_counter) return EUX_ERR_BAD_ARG;
    int rc = 0;
    switch (d->src_dtype) {
      case EUX_DT_F32: rc = launch_typed<float>(a, grid, st); break;
      case EUX_DT_F16: rc = launch_typed<__half>(a, grid, st); break;
      case EUX_DT_BF16: rc = launch_typed<__nv_bfloat16>(a, grid, st); break;
      case EUX_DT_F8E4M3: rc = launch_typed<__nv_fp8_e4m3>(a, grid, st); break;
      default: rc = EUX_ERR_BAD_ARG;
    }
    if (rc) return rc;
  } else {
    bool as_bytes = false;
    if (a.d.ndim == 0) {  // dense, but not on a 16-byte boundary: one row
      as_bytes = raw;
      if (as_bytes) a.d.n_elems *= (uint64_t)ssz;
      a.d.ndim = 1;
      a.d.shape[0] = a.d.n_elems ? (int64_t)a.d.n_elems : 1;
      a.d.stride[0] = 1;
    }
    if (!as_bytes && d->n_elems && (((uintptr_t)d->src % ssz) || ((uintptr_t)d->dst % dsz))) return EUX_ERR_BAD_ARG;  // would fault
    for (int k = 0; k < a.d.ndim; ++k)
      if (a.d.shape[k] < 1 && a.d.n_elems) return EUX_ERR_BAD_ARG;
    TileArgs t;
    bool vector = false;
    const int chunk = raw ? 16 / (as_bytes ? 1 : dsz) : 8;  // elements per chunk of the gather kernel
    const bool few = a.d.n_elems <= (uint64_t)sms * 2048;   // less than a step of four elements for every thread of the device
    Route route = Route::kElement;
    if (to_bytes) {
      // one kernel
    } else if (whole && !as_bytes && plan_tiles(a.d, t, vector) && (vector || !few)) {
      route = t.narrow ? Route::kNarrow : vector ? Route::kTileVector : Route::kTile;
      t.x = a;
    } else if (!as_bytes && rows_aligned(a.d, whole, chunk, ssz, dsz)) {
      route = Route::kGatherAligned;
    } else if (as_bytes || !(few || (ssz * dsz == 1 && a.d.ndim > 2 && a.d.shape[a.d.ndim - 1] < chunk))) {
      route = Route::kGather;
    }
    const bool tiled = route >= Route::kTile;
    // Four gather CTAs fill an SM's threads. Tiles: a CTA each, whose loads then overlap other CTAs' stores (47 us against
    // 51 on 8192 x 8192 bf16).
    // With a flag: five tile CTAs per SM, which are resident at once, and two gather CTAs, fewer CTAs that have to be counted
    // (4099 x 4096 fp32 to bf16 transposed 20.9 us, 22.5 with eight; 16 MiB of bf16 at an odd offset 8.4, 9.6 with four).
    // One that waits keeps to half of an SM (gathers have 64 registers and 512 threads), and all its CTAs wait at once, so
    // that a limit passes once.
    const bool flagged = d->flag || d->flag2;
    if (!ctas_given) max_ctas = d->wait_flag ? (tiled ? 2 : 1) * sms : !tiled ? (flagged ? 2 : 4) * sms : flagged ? 5 * sms : 0x7fffffff;
    const uint64_t per_cta = (uint64_t)kXferThreads * (route == Route::kElement ? 2 : chunk);
    grid = limit(tiled ? t.tiles : (a.d.n_elems + per_cta - 1) / per_cta);
    if (!scratch_counter) {  // up to 2048 elements, or when told to, one CTA does without
      if (d->n_elems > (uint64_t)kXferThreads * 4 && max_ctas > 1) return EUX_ERR_BAD_ARG;
      grid = 1;
    }
    GatherArgs ga{a, {}, a.d.n_elems >> 32 == 0};
    for (int k = 0; k < a.d.ndim; ++k) {
      if (a.d.shape[k] >> 32) ga.small = 0;
      else if (a.d.shape[k] > 0) ga.div[k] = fast_div((uint32_t)a.d.shape[k]);
    }
    int rc = 0;
    if (raw) {
      const int esz = as_bytes ? 1 : ssz;
      if (esz == 4) launch_gather<uint32_t, uint32_t, true>(ga, t, route, grid, st);
      else if (esz == 2) launch_gather<uint16_t, uint16_t, true>(ga, t, route, grid, st);
      else launch_gather<uint8_t, uint8_t, true>(ga, t, route, grid, st);
    } else {
      switch (d->src_dtype) {
        case EUX_DT_F32: rc = launch_gather_from<float>(ga, t, route, grid, st); break;
        case EUX_DT_F16: rc = launch_gather_from<__half>(ga, t, route, grid, st); break;
        case EUX_DT_BF16: rc = launch_gather_from<__nv_bfloat16>(ga, t, route, grid, st); break;
        case EUX_DT_F8E4M3: rc = launch_gather_from<__nv_fp8_e4m3>(ga, t, route, grid, st); break;
        default: rc = EUX_ERR_BAD_ARG;
      }
    }
    if (rc) return rc;
  }
  return (int)cudaGetLastError();
}

extern "C" int eux_xfer_rpc_step_launch(const eux_xfer_desc* req, const eux_xfer_desc* resp, const eux_xfer_desc* done,
                                        uint32_t* scratch3, int max_ctas, void* stream) {
  if (!req || !resp || !done || !scratch3 || !req->src || !req->dst || !resp->src || !resp->dst) return EUX_ERR_BAD_ARG;
  const eux_xfer_desc* ds[2] = {req, resp};
  for (const eux_xfer_desc* d : ds) {
    if (d->ndim != 0 || d->src_dtype != d->dst_dtype) return EUX_ERR_BAD_ARG;
    if ((((uintptr_t)d->src) | ((uintptr_t)d->dst)) & 15u) return EUX_ERR_BAD_ARG;
    if (d->op != EUX_OP_NONE && d->src_dtype == EUX_DT_BYTES) return EUX_ERR_BAD_ARG;
  }
  if (req->src_dtype != resp->src_dtype) return EUX_ERR_BAD_ARG;
  const int sms = num_sms();
  if (max_ctas <= 0 || max_ctas > sms) max_ctas = sms;  // every CTA resident: see the kernel
  const uint64_t bytes = req->n_elems * (uint64_t)dtype_size(req->src_dtype);
  const uint64_t want = (bytes + (uint64_t)kXferThreads * 64 - 1) / ((uint64_t)kXferThreads * 64);
  const int grid = (int)(want < 1 ? 1 : (want > (uint64_t)max_ctas ? max_ctas : want));
  RpcStepArgs a{*req, *resp, *done, scratch3};
  a.done.n_elems = 0;
  cudaStream_t st = (cudaStream_t)stream;
  switch (req->src_dtype) {
    case EUX_DT_F32: xfer_rpc_step_kernel<float><<<grid, kXferThreads, 0, st>>>(a); break;
    case EUX_DT_F16: xfer_rpc_step_kernel<__half><<<grid, kXferThreads, 0, st>>>(a); break;
    case EUX_DT_BF16: xfer_rpc_step_kernel<__nv_bfloat16><<<grid, kXferThreads, 0, st>>>(a); break;
    case EUX_DT_F8E4M3: xfer_rpc_step_kernel<__nv_fp8_e4m3><<<grid, kXferThreads, 0, st>>>(a); break;
    case EUX_DT_BYTES: xfer_rpc_step_kernel<float><<<grid, kXferThreads, 0, st>>>(a); break;  // no handler: bytes only
    default: return EUX_ERR_BAD_ARG;
  }
  return (int)cudaGetLastError();
}

extern "C" int eux_xfer_bulk_launch(const eux_xfer_desc* d, uint32_t* scratch_counter, int max_ctas, void* stream) {
  if (!d || !d->src || !d->dst || d->ndim != 0) return EUX_ERR_BAD_ARG;
  if (d->src_dtype != d->dst_dtype || d->op != EUX_OP_NONE) return EUX_ERR_BAD_ARG;
  if ((((uintptr_t)d->src) | ((uintptr_t)d->dst)) & 15u) return EUX_ERR_BAD_ARG;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return EUX_ERR_BAD_ARG;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(xfer_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBulkSmem);
    if (e != cudaSuccess) return (int)e;
    attr_set[dev] = true;
  }
  const uint64_t bytes = d->n_elems * (uint64_t)dtype_size(d->src_dtype);
  if (max_ctas <= 0) max_ctas = 2 * num_sms();
  uint64_t want = (bytes + kBulkChunk - 1) / kBulkChunk;
  int grid = (int)(want < 1 ? 1 : (want > (uint64_t)max_ctas ? max_ctas : want));
  if (grid > 1 && !scratch_counter) return EUX_ERR_BAD_ARG;
  XferArgs a{*d, scratch_counter};
  xfer_bulk_kernel<<<grid, kBulkThreads, kBulkSmem, (cudaStream_t)stream>>>(a);
  return (int)cudaGetLastError();
}

// One CTA per item, the items in the launch parameters.
struct PullBatchArgs {
  eux_pull_item it[EUX_PULL_BATCH_MAX];
};
// 1024 threads: a 64 KiB message is in flight at once (four 16-byte vectors per thread), so its CTA needs one
// memory round trip for it and not four; the launch is as long as its largest item.
constexpr int kPullBatchThreads = 1024;
__global__ void __launch_bounds__(kPullBatchThreads) xfer_pull_batch_kernel(const __grid_constant__ PullBatchArgs a) {
  const eux_pull_item& d = a.it[blockIdx.x];
  const unsigned char* src = reinterpret_cast<const unsigned char*>(d.src);
  unsigned char* dst = reinterpret_cast<unsigned char*>(d.dst);
  if (((((uintptr_t)src) | ((uintptr_t)dst)) & 15u) == 0) {
    copy_bytes_grid<false>(src, dst, d.nbytes, 0, 1);
  } else {
    for (uint64_t b = threadIdx.x; b < d.nbytes; b += blockDim.x) dst[b] = src[b];
  }
  __syncthreads();
  if (threadIdx.x == 0 && (d.flag || d.flag2)) {
    __threadfence_system();
    if (d.flag) st_relaxed_sys(d.flag, d.flag_value);
    if (d.flag2) st_relaxed_sys(d.flag2, d.flag2_value);
  }
}

extern "C" int eux_xfer_pull_batch_launch(const eux_pull_item* items, int n, void* stream) {
  if (n <= 0) return 0;
  if (!items || n > EUX_PULL_BATCH_MAX) return EUX_ERR_BAD_ARG;
  PullBatchArgs a;
  for (int i = 0; i < n; ++i) {
    if (!items[i].src || !items[i].dst) return EUX_ERR_BAD_ARG;
    a.it[i] = items[i];
  }
  for (int i = n; i < EUX_PULL_BATCH_MAX; ++i) a.it[i] = eux_pull_item{};
  xfer_pull_batch_kernel<<<n, kPullBatchThreads, 0, (cudaStream_t)stream>>>(a);
  return (int)cudaGetLastError();
}

extern "C" int eux_xfer_batch_launch(const eux_xfer_desc* descs_dev, int n, void* stream) {
  if (n <= 0) return 0;
  if (!descs_dev) return EUX_ERR_BAD_ARG;
  xfer_batch_kernel<<<n, 256, 0, (cudaStream_t)stream>>>(descs_dev, n);
  return (int)cudaGetLastError();
}

extern "C" int eux_pingpong_launch(const eux_pingpong_desc* d, int ctas, void* stream) {
  if (!d || !d->local_buf || !d->peer_buf || !d->grid_bar || (d->nbytes & 15u)) return EUX_ERR_BAD_ARG;
  if (d->initiator != 2 && (!d->local_flag || !d->peer_flag)) return EUX_ERR_BAD_ARG;
  const int sms = num_sms();
  if (ctas <= 0 || ctas > sms) ctas = sms;  // every CTA must be resident: they wait on one another
  uint64_t want = (d->nbytes + (uint64_t)kXferThreads * 64 - 1) / ((uint64_t)kXferThreads * 64);
  if ((uint64_t)ctas > want) ctas = (int)(want < 1 ? 1 : want);
  eux_pingpong_desc dd = *d;
  void* args[] = {&dd};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)pingpong_kernel, dim3(ctas), dim3(kXferThreads), args, 0,
                                              (cudaStream_t)stream);
  return (int)e;
}

extern "C" int eux_ipc_export(void* dev_ptr, unsigned char handle_out[64]) {
  static_assert(sizeof(cudaIpcMemHandle_t) == 64, "handle size");
  cudaIpcMemHandle_t h;
  cudaError_t e = cudaIpcGetMemHandle(&h, dev_ptr);
  if (e == cudaSuccess) memcpy(handle_out, &h, 64);
  return (int)e;
}
extern "C" int eux_ipc_open(const unsigned char handle[64], void** dev_ptr_out) {
  cudaIpcMemHandle_t h;
  memcpy(&h, handle, 64);
  return (int)cudaIpcOpenMemHandle(dev_ptr_out, h, cudaIpcMemLazyEnablePeerAccess);
}
extern "C" int eux_ipc_close(void* dev_ptr) { return (int)cudaIpcCloseMemHandle(dev_ptr); }
extern "C" int eux_memcpy_peer_async(void* dst, int dst_device, const void* src, int src_device, size_t bytes, void* stream) {
  return (int)cudaMemcpyPeerAsync(dst, dst_device, src, src_device, bytes, (cudaStream_t)stream);
}
extern "C" int eux_enable_peer_access(int this_dev, int peer_dev) {
  int can = 0;
  cudaError_t e = cudaDeviceCanAccessPeer(&can, this_dev, peer_dev);
  if (e != cudaSuccess) return (int)e;
  if (!can) return EUX_ERR_UNSUPPORTED;
  int cur = 0;
  cudaGetDevice(&cur);
  cudaSetDevice(this_dev);
  e = cudaDeviceEnablePeerAccess(peer_dev, 0);
  if (e == cudaErrorPeerAccessAlreadyEnabled) {
    cudaGetLastError();
    e = cudaSuccess;
  }
  cudaSetDevice(cur);
  return (int)e;
}
extern "C" int eux_device_malloc(void** p, size_t bytes) { return (int)cudaMalloc(p, bytes); }
extern "C" int eux_device_free(void* p) { return (int)cudaFree(p); }
extern "C" int eux_host_alloc_mapped(void** host_ptr, void** dev_ptr, size_t bytes) {
  cudaError_t e = cudaHostAlloc(host_ptr, bytes, cudaHostAllocMapped | cudaHostAllocPortable);
  if (e != cudaSuccess) return (int)e;
  memset(*host_ptr, 0, bytes);
  return (int)cudaHostGetDevicePointer(dev_ptr, *host_ptr, 0);
}
extern "C" int eux_host_free(void* host_ptr) { return (int)cudaFreeHost(host_ptr); }
extern "C" const char* eux_error_string(int err) {
  switch (err) {
    case EUX_ERR_BAD_ARG: return "eux: bad argument";
    case EUX_ERR_TOO_LARGE: return "eux: size beyond the supported maximum";
    case EUX_ERR_UNSUPPORTED: return "eux: unsupported on this device";
    default: return cudaGetErrorString((cudaError_t)err);
  }
}


// ---------------------------------------------------------------------------
// Loading every kernel of this file up front. With lazy module loading (the default of the driver) the
// first launch of a kernel loads it, and loading may have to wait for kernels that are running on the
// device. A kernel of some other library that spins until a peer does something (a collective's barrier,
// say) while that peer waits for the reply to a call whose handler launches one of these kernels for the
// first time is then a deadlock. Everything that launches on behalf of a peer loads its kernels first.
// ---------------------------------------------------------------------------
namespace {
template <class K>
int preload_one(K kernel) {
  cudaFuncAttributes attr;
  return (int)cudaFuncGetAttributes(&attr, reinterpret_cast<const void*>(kernel));
}
template <typename S, typename D, bool RAW>
int preload_gather() {
  int rc = preload_one(xfer_element_kernel<S, D, RAW>);
  if (!rc) rc = preload_one(xfer_gather_kernel<S, D, RAW, true>);
  if (!rc) rc = preload_one(xfer_gather_kernel<S, D, RAW, false>);
  if (!rc) rc = preload_one(xfer_narrow_kernel<S, D, RAW>);
  if (!rc) rc = preload_one(xfer_tile_kernel<S, D, RAW, true>);
  if (!rc) rc = preload_one(xfer_tile_kernel<S, D, RAW, false>);
  return rc;
}
template <typename S>
int preload_typed() {
  int rc = preload_one(xfer_typed_kernel<S, float>);
  if (!rc) rc = preload_one(xfer_typed_kernel<S, __half>);
  if (!rc) rc = preload_one(xfer_typed_kernel<S, __nv_bfloat16>);
  if (!rc) rc = preload_one(xfer_typed_kernel<S, __nv_fp8_e4m3>);
  if (!rc) rc = preload_one(xfer_rpc_step_kernel<S>);
  if (!rc) rc = preload_one(xfer_element_kernel<S, uint8_t, false>);
  if (!rc) rc = preload_gather<S, float, false>();
  if (!rc) rc = preload_gather<S, __half, false>();
  if (!rc) rc = preload_gather<S, __nv_bfloat16, false>();
  if (!rc) rc = preload_gather<S, __nv_fp8_e4m3, false>();
  return rc;
}
}  // namespace

extern "C" int eux_xfer_preload(void) {
  int rc = preload_one(xfer_bytes_kernel<true>);
  if (!rc) rc = preload_one(xfer_bytes_kernel<false>);
  if (!rc) rc = preload_one(xfer_bulk_kernel);
  if (!rc) rc = preload_gather<uint8_t, uint8_t, true>();
  if (!rc) rc = preload_gather<uint16_t, uint16_t, true>();
  if (!rc) rc = preload_gather<uint32_t, uint32_t, true>();
  if (!rc) rc = preload_one(xfer_batch_kernel);
  if (!rc) rc = preload_one(pingpong_kernel);
  if (!rc) rc = preload_one(xfer_pull_batch_kernel);
  if (!rc) rc = preload_typed<float>();
  if (!rc) rc = preload_typed<__half>();
  if (!rc) rc = preload_typed<__nv_bfloat16>();
  if (!rc) rc = preload_typed<__nv_fp8_e4m3>();
  return rc;
}
