// Residual add + RMSNorm of a rank's own rows (no communication): y = rmsnorm(x + residual) * weight.
//
// Bound by memory: x and the residual are read once, y and the new residual written once, and nothing is reused but the
// norm weight.  Two kernels:
//   * many long rows: a CTA walks rows b, b + G, ...; rows arrive through a ring of bulk copies (cp.async.bulk, one thread
//     issues them), so the loads of the next rows are in flight while a row is summed, scaled and written.  The old form (plain
//     loads, three block barriers per row, loads of a row issued only when the row before was done) kept too little in
//     flight.  One block barrier per row: it publishes the warps' partial sums (two sets, alternating) and
//     frees the row's buffer at the same time.  A wait that runs out costs the ring, not the rows: from there on the block
//     reads rows with plain loads, and leaves when its copies have landed.
//   * few rows (a decode step), or short ones: one row per CTA, all loads issued at once; what counts is latency.
// fp32 sums; the normalisation sees the residual stream as it is stored (rounded).
// Measured on B200, bf16 with residual: 16384 x 8192 in 182.5 us (5.9 TB/s; 280.4 us before), 4096 x 8192 in 47.6 us,
// 1024 x 8192 in 11.0 us, 16 rows in 2.2 us as a link of a chain of launches.
//
// Capability parity: the reference's stand-alone RMSNorm (src/rmsnorm/rmsnorm.cuh:11-121).
#include <cuda_runtime.h>

#include <atomic>

#include "../device/reduce.cuh"
#include "collectives.h"

namespace oob {
namespace {

constexpr int kThreadsN = 256;
constexpr int kWarpsN = kThreadsN / 32;
constexpr int kMaxStagesN = 4;
constexpr int kSmPerGpu = 148;

struct LocalNorm {
  const char* x;
  const char* res;  // null: no residual
  const char* w;
  char* y;
  char* ro;         // null: the sum is not stored (and not rounded)
  int rows, hidden;
  float eps;
  int stages;
  uint32_t polls;  // of a wait for a row
};

// Rows are read once.  In a call that moves more than L2 holds they leave it first: what is written instead of them is read next (residual + norm of 16384 x 8192
// 182.6 us, 181.5 so; 6000 x 5120 45.3, 43.3; 6144 x 8192 without residual 40.5, 38.2).  In smaller calls rows may be in L2 the next time, and what they
// came from may be read again: 3072 x 4096 with residual, the same rows again and again, 11.5, 13.6; 6144 x 4096 without 15.8, 17.6.
constexpr long long kOnceBytesN = 160ll << 20;  // rows read and written
// A kernel of its own: chosen row by row, by the thread that asks for the rows, 32768 x 1024 with residual took 51.5 us and not 49.9.
template <bool ONCE>
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  if constexpr (ONCE) {
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                 :
                 : "r"(ptx::smem_u32(smem_dst)), "l"(src), "r"(bytes), "r"(ptx::smem_u32(bar)), "l"(policy)
                 : "memory");
  } else {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :
                 : "r"(ptx::smem_u32(smem_dst)), "l"(src), "r"(bytes), "r"(ptx::smem_u32(bar))
                 : "memory");
  }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One pack of the residual stream: adds, rounds and stores it where asked; returns its share of the sum of squares.
template <typename T>
__device__ __forceinline__ float take_pack(const LocalNorm& a, const uint4& xv, const uint4& rv, size_t off, float (&v)[8]) {
  using PT = PackTraits<T>;
  PT::unpack(xv, v);
  if (a.res != nullptr) {
    float r[8];
    PT::unpack(rv, r);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] += r[i];
  }
  if (a.ro != nullptr) {
    const uint4 o = PT::pack(v);
    PT::unpack(o, v);
    ptx::st_v4(a.ro + off, o);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
  return ss;
}

// The rows `row`, row + G, ... of a block whose ring was given up, with plain loads.  `summed`: this thread has seen the first of
// them land, and has stored its packs of the sum where a.ro asks for it (in place, over an input), before the block learned
// that others have not.  One pack at a time and two passes, so that it asks for no more registers than the streaming loop.
template <typename T>
__device__ __forceinline__ void finish_rows(const LocalNorm& a, int row, bool summed, float (*part)[kWarpsN]) {
  using PT = PackTraits<T>;
  const int packs = a.hidden / 8;
  int set = 0;
#pragma unroll 1
  for (; row < a.rows; row += gridDim.x, set ^= 1, summed = false) {
    const size_t off = size_t(row) * a.hidden * 2;
    float v[8], ss = 0.f;
#pragma unroll 1
    for (int p = threadIdx.x; p < packs; p += kThreadsN) {
      const size_t at = off + size_t(p) * 16;
      LocalNorm from = a;
      if (summed && a.ro != nullptr) {
        from.x = a.ro;
        from.res = nullptr;
      }
      const uint4 xv = ptx::ld_v4(from.x + at);
      ss += take_pack<T>(from, xv, from.res != nullptr ? ptx::ld_v4(from.res + at) : xv, at, v);
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) part[set][threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < kWarpsN; ++i) total += part[set][i];
    const float scale = rsqrtf(total / float(a.hidden) + a.eps);
#pragma unroll 1
    for (int p = threadIdx.x; p < packs; p += kThreadsN) {
      const size_t at = off + size_t(p) * 16;
      float w[8];
      PT::unpack(ptx::ld_v4(a.w + size_t(p) * 16), w);
      PT::unpack(ptx::ld_v4((a.ro != nullptr ? a.ro : a.x) + at), v);
      if (a.ro == nullptr && a.res != nullptr) {
        float r[8];
        PT::unpack(ptx::ld_v4(a.res + at), r);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += r[i];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = v[i] * scale * w[i];
      ptx::st_v4(a.y + at, PT::pack(v));
    }
  }
}

// PPT: 16-byte packs per thread and row.  ONCE: see kOnceBytesN.
template <typename T, int PPT, bool ONCE>
__global__ void __launch_bounds__(kThreadsN, PPT <= 2 ? 5 : PPT <= 4 ? 3 : 1) norm_stream_kernel(const __grid_constant__ LocalNorm a) {
  using PT = PackTraits<T>;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t full[kMaxStagesN];
  __shared__ float part[2][kWarpsN];
  __shared__ int abort_word;
  const int packs = a.hidden / 8;
  const uint32_t row_bytes = uint32_t(a.hidden) * 2;
  const uint32_t stage_bytes = row_bytes * (a.res != nullptr ? 2 : 1);
  const int warp = threadIdx.x >> 5;
  volatile int* abort = &abort_word;
  auto issue = [&](int row, int stage) {
    uint8_t* dst = smem + size_t(stage) * stage_bytes;
    ptx::mbar_arrive_expect_tx(&full[stage], stage_bytes);
    bulk_load<ONCE>(dst, a.x + size_t(row) * row_bytes, row_bytes, &full[stage]);
    if (a.res != nullptr) bulk_load<ONCE>(dst + row_bytes, a.res + size_t(row) * row_bytes, row_bytes, &full[stage]);
  };
  if (threadIdx.x == 0) {
    abort_word = 0;
    for (int s = 0; s < a.stages; ++s) ptx::mbar_init(&full[s], 1);
    ptx::mbar_fence_init();
  }
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      const int row = blockIdx.x + s * gridDim.x;
      if (row < a.rows) issue(row, s);
    }
  }
  uint4 w[PPT];
#pragma unroll
  for (int j = 0; j < PPT; ++j) {
    const int p = threadIdx.x + j * kThreadsN;
    if (p < packs) w[j] = ptx::ld_v4(a.w + size_t(p) * 16);
  }
  __syncthreads();
  int stage = 0, set = 0;
  uint32_t phase = 0;
  int row = blockIdx.x;
  bool landed = true;
  for (; row < a.rows; row += gridDim.x) {
    landed = ptx::mbar_wait(&full[stage], phase, abort, a.polls);
    const uint8_t* src = smem + size_t(stage) * stage_bytes;
    const size_t off = size_t(row) * row_bytes;
    float v[PPT][8];
    float ss = 0.f;
    if (landed) {
#pragma unroll
      for (int j = 0; j < PPT; ++j) {
        const int p = threadIdx.x + j * kThreadsN;
        if (p < packs) {
          const uint4 xv = *reinterpret_cast<const uint4*>(src + size_t(p) * 16);
          uint4 rv = xv;
          if (a.res != nullptr) rv = *reinterpret_cast<const uint4*>(src + row_bytes + size_t(p) * 16);
          ss += take_pack<T>(a, xv, rv, off + size_t(p) * 16, v[j]);
        }
      }
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) part[set][warp] = ss;
    if (!__syncthreads_and(landed)) break;  // a copy did not land in time: the same in every thread
    if (threadIdx.x == 0) {
      const int next = row + a.stages * int(gridDim.x);
      if (next < a.rows) issue(next, stage);
    }
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < kWarpsN; ++i) total += part[set][i];
    const float scale = rsqrtf(total / float(a.hidden) + a.eps);
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
      const int p = threadIdx.x + j * kThreadsN;
      if (p < packs) {
        float wf[8], o[8];
        PT::unpack(w[j], wf);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = v[j][i] * scale * wf[i];
        ptx::st_v4(a.y + off + size_t(p) * 16, PT::pack(o));
      }
    }
    set ^= 1;
    if (++stage == a.stages) {
      stage = 0;
      phase ^= 1;
    }
  }
  if (row < a.rows) {
    finish_rows<T>(a, row, landed, part);
    if (threadIdx.x == 0) {  // copies in flight (this row's and the next rows') land before shared memory is released
      int gave_up = 0;
      for (int s = 0; s < a.stages && row < a.rows; ++s, row += gridDim.x) {
        ptx::mbar_wait(&full[stage], phase, &gave_up);
        if (++stage == a.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  }
}

// One row per CTA (rows b, b + G, ... when the caller caps the grid).
template <typename T, int THREADS, int PPT>
__global__ void __launch_bounds__(THREADS) norm_rows_kernel(const __grid_constant__ LocalNorm a) {
  using PT = PackTraits<T>;
  __shared__ float part[2][THREADS / 32];
  const int packs = a.hidden / 8;
  const size_t row_bytes = size_t(a.hidden) * 2;
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  int set = 0;
  for (int row = blockIdx.x; row < a.rows; row += gridDim.x, set ^= 1) {
    const size_t off = size_t(row) * row_bytes;
    uint4 xv[PPT], rv[PPT], w[PPT];
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
      const int p = threadIdx.x + j * THREADS;
      if (p < packs) {
        xv[j] = *reinterpret_cast<const uint4*>(a.x + off + size_t(p) * 16);
        rv[j] = a.res != nullptr ? *reinterpret_cast<const uint4*>(a.res + off + size_t(p) * 16) : xv[j];
        w[j] = ptx::ld_v4(a.w + size_t(p) * 16);
      }
    }
    float v[PPT][8];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
      const int p = threadIdx.x + j * THREADS;
      if (p < packs) ss += take_pack<T>(a, xv[j], rv[j], off + size_t(p) * 16, v[j]);
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) part[set][threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < THREADS / 32; ++i) total += part[set][i];
    const float scale = rsqrtf(total / float(a.hidden) + a.eps);
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
      const int p = threadIdx.x + j * THREADS;
      if (p < packs) {
        float wf[8], o[8];
        PT::unpack(w[j], wf);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = v[j][i] * scale * wf[i];
        ptx::st_v4(a.y + off + size_t(p) * 16, PT::pack(o));
      }
    }
  }
}

cudaError_t launch(void (*kernel)(LocalNorm), int grid, int threads, int smem, const LocalNorm& n, cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, n);
}

template <typename T, int PPT, bool ONCE>
cudaError_t launch_stream_of(LocalNorm n, int max_ctas, cudaStream_t stream) {
  auto kernel = norm_stream_kernel<T, PPT, ONCE>;
  static std::atomic<uint64_t> attr_set{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_set.load(std::memory_order_relaxed) >> (dev & 63) & 1)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    attr_set.fetch_or(uint64_t(1) << (dev & 63), std::memory_order_relaxed);
  }
  const int stage_bytes = n.hidden * 2 * (n.res != nullptr ? 2 : 1);
  // Three rows of the ring, or two, in at most 110 KiB, so that two CTAs share an SM.  Two rows it is in any case: from 13832
  // elements with a residual on they leave room for one CTA only.
  n.stages = 110 * 1024 / stage_bytes;
  if (n.stages > 3) n.stages = 3;
  if (n.stages < 2) n.stages = 2;
  const int smem = n.stages * stage_bytes;
  int per_sm = 220 * 1024 / (smem + 2048);
  if (per_sm > 8) per_sm = 8;
  if (per_sm < 1) per_sm = 1;
  int grid = kSmPerGpu * per_sm;
  if (grid > max_ctas) grid = max_ctas;
  if (grid > n.rows) grid = n.rows;
  return launch(kernel, grid, kThreadsN, smem, n, stream);
}

template <typename T, int PPT>
cudaError_t launch_stream(const LocalNorm& n, int max_ctas, cudaStream_t stream) {
  const long long bytes = 2ll * n.rows * n.hidden * (2 + (n.res != nullptr ? 1 : 0) + (n.ro != nullptr ? 1 : 0));
  return bytes >= kOnceBytesN ? launch_stream_of<T, PPT, true>(n, max_ctas, stream) : launch_stream_of<T, PPT, false>(n, max_ctas, stream);
}

template <typename T>
cudaError_t dispatch(const LocalNorm& n, int max_ctas, cudaStream_t stream) {
  const int packs = n.hidden / 8;
  // Up to two rows per SM nothing is gained by a ring: every row is in flight at once (256 x 8192: 3.6 us).  Nor is it, however
  // many rows there are, where a row is at most one pack per thread: what a row costs then is the wait, the barrier and the
  // copies' set-up of the ring, while CTAs of one row each overlap freely.  With and without residual, one row per CTA
  // against the ring: 4096 x 1024 7.2 and 4.4 against 9.2 and 7.9 us, 16384 x 128 14.3 and 9.4 against 23.4 and
  // 21.7, 16384 x 2048 44.1 and 25.5 against 45.1 and 27.6; at 16384 x 2560 the ring is ahead, 62.9 and 32.5 against 67.3 and 41.9.
  // With a residual and very many rows of 513 - 1024 elements eight CTAs of 128 threads per SM have too little in flight: 16384 x
  // 1024 29.7 against 27.1 (4096 x 1000 still 7.4 against 9.2).
  const bool few_in_flight = n.res != nullptr && packs > 64 && packs <= 128 && n.rows > 8192;
  if (n.rows <= 2 * kSmPerGpu || (packs <= kThreadsN && !few_in_flight)) {
    const int grid = n.rows < max_ctas ? n.rows : max_ctas;
    if (packs <= 128) return launch(norm_rows_kernel<T, 128, 1>, grid, 128, 0, n, stream);
    if (packs <= 256) return launch(norm_rows_kernel<T, 256, 1>, grid, 256, 0, n, stream);
    if (packs <= 512) return launch(norm_rows_kernel<T, 512, 1>, grid, 512, 0, n, stream);
    if (packs <= 1024) return launch(norm_rows_kernel<T, 512, 2>, grid, 512, 0, n, stream);
    return launch(norm_rows_kernel<T, 512, 4>, grid, 512, 0, n, stream);
  }
  const int ppt = (packs + kThreadsN - 1) / kThreadsN;
  if (ppt <= 1) return launch_stream<T, 1>(n, max_ctas, stream);
  if (ppt <= 2) return launch_stream<T, 2>(n, max_ctas, stream);
  if (ppt <= 4) return launch_stream<T, 4>(n, max_ctas, stream);
  return launch_stream<T, 8>(n, max_ctas, stream);
}

}  // namespace

cudaError_t launch_norm_local(int rank, const NormArgs& a, int max_ctas, cudaStream_t stream, uint32_t polls) {
  if (a.hidden > 8 * 8 * kThreadsN) return cudaErrorInvalidValue;  // 16384
  LocalNorm n{};
  n.x = static_cast<const char*>(a.x.p[rank]);
  n.res = static_cast<const char*>(a.residual);
  n.w = static_cast<const char*>(a.weight);
  n.y = static_cast<char*>(a.y_local);
  n.ro = static_cast<char*>(a.res_out_local);
  n.rows = a.rows;
  n.hidden = a.hidden;
  n.eps = a.eps;
  n.polls = polls;
  if (a.rows == 0) return cudaSuccess;
  if (max_ctas < 1) max_ctas = 1;
  return a.dtype == kF16 ? dispatch<__half>(n, max_ctas, stream) : dispatch<__nv_bfloat16>(n, max_ctas, stream);
}

}  // namespace oob
