// Decode-path kernels of the tensor-parallel model runner (sm_100a): rotary embedding + KV-cache write, SwiGLU,
// and grouped-query decode attention over a static cache.
//
// The attention kernel is bound by reading the cache once: a CTA handles one (sequence, KV head, key chunk); its
// four warps take 16-key tiles in turn (cp.async, three stages or six, per-warp buffers, XOR-swizzled rows), compute
// scores for all query heads of the KV group at once on the tensor cores (m16n8k16: up to eight query heads are its columns and the
// keys its rows, nine to sixteen are its rows -- too few for a tcgen05 tile, which needs 64), keep an online softmax per head and
// accumulate P*V in fp32.  The warps' partial results are merged through shared memory, those of the up to eight CTAs of a cluster
// through distributed shared memory; only few long sequences are cut further, and a second small kernel then merges.
//
// Capability parity: none of these exist in the reference (it delegates the model to vLLM,
// patches/vllm/v0.25.0/vllm/model_executor/models/qwen2.py); they make this library's own serving path a fixed
// sequence of kernels per layer.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "../api/oob.h"
#include "../api/oob_model.h"
#include "../device/activation.cuh"
#include "../device/ptx.cuh"
#include "../runtime/errors.h"

namespace oob {
namespace model {

// ---------------------------------------------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------------------------------------------
template <typename T>
struct Cvt;
template <>
struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
};
template <>
struct Cvt<__half> {
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
};

// Launches with programmatic stream serialization: the kernel's launch overlaps the tail of the one before it.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream, int cluster, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// ---------------------------------------------------------------------------------------------------------------
// RoPE + KV-cache write
// ---------------------------------------------------------------------------------------------------------------
// One thread per 16-byte unit (8 elements = 4 rotation pairs) of one head of one token.
template <typename T>
__global__ void rope_kv_write_kernel(oob_rope_args_t a, long long units) {
  const int upr = a.hd / 8;  // units per head
  const int heads = a.H + 2 * a.KV;
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  const long long pos_base = a.pos_dev != nullptr ? *a.pos_dev : static_cast<long long>(a.pos0);
  for (long long u = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; u < units;
       u += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(u % upr);
    const long long th = u / upr;
    const int hh = static_cast<int>(th % heads);
    const long long token = th / heads;
    const int b = static_cast<int>(token / a.T), t = static_cast<int>(token % a.T);
    long long p = pos_base + t;
    if (p < 0) p = 0;
    if (p > a.max_len - 1) p = a.max_len - 1;  // the host checks the range; never index outside the tables / cache
    const uint4 in = *reinterpret_cast<const uint4*>(static_cast<const T*>(a.qkv) + (token * heads + hh) * a.hd + c * 8);
    uint4 out = in;
    if (hh < a.H + a.KV) {
      const float4 cs = *reinterpret_cast<const float4*>(a.cos_table + p * (a.hd / 2) + c * 4);
      const float4 sn = *reinterpret_cast<const float4*>(a.sin_table + p * (a.hd / 2) + c * 4);
      const float cc[4] = {cs.x, cs.y, cs.z, cs.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
      const uint32_t w[4] = {in.x, in.y, in.z, in.w};
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = Cvt<T>::unpack(w[i]);
        o[i] = Cvt<T>::pack(x.x * cc[i] - x.y * ss[i], x.x * ss[i] + x.y * cc[i]);
      }
      out = make_uint4(o[0], o[1], o[2], o[3]);
    }
    T* dst;
    if (hh < a.H) {
      dst = static_cast<T*>(a.q_out) + (token * a.H + hh) * a.hd + c * 8;
    } else {
      const int kvh = hh < a.H + a.KV ? hh - a.H : hh - a.H - a.KV;
      T* cache = static_cast<T*>(hh < a.H + a.KV ? a.k_cache : a.v_cache);
      dst = cache + (a.batch0 + b) * a.cache_batch_stride + (static_cast<long long>(kvh) * a.max_len + p) * a.hd + c * 8;
    }
    *reinterpret_cast<uint4*>(dst) = out;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// SwiGLU
// ---------------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void silu_mul_kernel(const T* gu, long long ld, T* out, long long units, int F) {
  const int upr = F / 8;
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  for (long long u = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; u < units;
       u += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = u / upr;
    const int c = static_cast<int>(u % upr);
    const uint4 g = *reinterpret_cast<const uint4*>(gu + r * ld + c * 8);
    const uint4 v = *reinterpret_cast<const uint4*>(gu + r * ld + F + c * 8);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, vw[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = Cvt<T>::unpack(gw[i]), y = Cvt<T>::unpack(vw[i]);
      o[i] = Cvt<T>::pack(swiglu_f32(x.x, y.x), swiglu_f32(x.y, y.y));
    }
    *reinterpret_cast<uint4*>(out + r * static_cast<long long>(F) + c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Decode attention
// ---------------------------------------------------------------------------------------------------------------
constexpr int kHD = 128;
constexpr int kTileKeys = 16;                      // keys per warp tile: one K = 16 step of the P V product
constexpr int kAttnWarps = 4;
constexpr int kAttnThreads = kAttnWarps * 32;
constexpr int kRowBytes = kHD * 2;                 // 256
constexpr int kKvTileBytes = kTileKeys * kRowBytes;  // 4 KiB
// Keys and values are read once; those that the next call will not find in L2 leave it first.  A cache that is read again and again is found there up to 100 MB, so
// that this is for the live keys of a call from here on: 256 x 1024 keys (128 MB) 23.4 -> 22.8 us, 256 x 1900 40.7 -> 40.3; but 80 MB of them, 256 x 640,
// 10.35 -> 12.3, and in a cache of five times the length 10.5 -> 13.9.  The host knows a bound of the length and takes a kernel of its own by it (the
// policy in a register costs short contexts 1 - 4 %), which looks at the length and has loads of both kinds (a normal policy for the short ones instead: up to
// 5 % slower).  Not with more than eight heads a KV head: no gain (40 x 6553 keys 26.7, 27.0).
constexpr long long kOnceBytes = 128ll << 20;
constexpr int kMaxAttnCluster = 8;                 // portable cluster size
constexpr int kAttnStages = 3;                     // tiles of K and V in flight or in use per warp (96 KiB per CTA, two per SM)
// Where no SM gets two CTAs anyway, and CTAs alone or in pairs (64 x 300 keys 5.5 -> 5.15 us; clusters of eight gain nothing, fewer of
// them fit the device, and they start later: 1 x 4000 keys 6.9 and 7.15).
constexpr int kAttnDeepStages = 6;
__host__ __device__ constexpr int attn_warp_bytes(int stages) { return stages * 2 * kKvTileBytes; }
__host__ __device__ constexpr int attn_smem_bytes(int stages) { return kAttnWarps * attn_warp_bytes(stages); }
// fp32 words of a head's row of a warp's result: the rows that are stored together start in different banks.
__host__ __device__ constexpr int merge_stride(bool few) { return few ? kHD + 4 : kHD + 8; }
constexpr int kPartialStride = kHD + 2;            // fp32 words of one partial result: 128 values, max, sum

template <typename T>
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// Rows and columns of an 8 x 8 matrix of 16-bit values change places.
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
template <bool ONCE>
__device__ __forceinline__ void cp_async_16(uint32_t smem_addr, const void* gptr, uint64_t policy) {
  if constexpr (ONCE) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(smem_addr), "l"(gptr), "l"(policy) : "memory");
  } else {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr), "l"(gptr) : "memory");
  }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Byte offset of 16-byte unit `c` of key row `r` inside a tile (rows of 256 bytes, units XOR-swizzled by the row so
// that the eight rows of an ldmatrix hit different banks).
__device__ __forceinline__ uint32_t kv_off(int r, int c) { return uint32_t(r) * kRowBytes + (uint32_t(c ^ (r & 7)) << 4); }

struct AttnParams {
  const void* q;
  const void* k;
  const void* v;
  void* out;
  float* ws;
  bool ws_pairs;  // the workspace, which is on four bytes, stands on eight (and with it every part, of 65 pairs): two floats an access
  const long long* pos_dev;
  int len;
  int B, H, KV, G;
  long long batch_stride;
  int max_len, batch0;
  int splits;
  int once_len;  // of the kernel with ONCE: the length from which on keys and values leave L2 first (see kOnceBytes)
  float scale_log2;
  float nan;   // see the merge over the cluster
  bool ahead;  // the position and the keys and values before the newest may be read before the kernels this one depends on are done
};

template <typename T>
__device__ __forceinline__ T to_out(float y) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    return __float2bfloat16_rn(y);
  } else {
    return __float2half_rn(y);
  }
}

__device__ __forceinline__ void attn_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The two halves of attn_cluster_sync.
__device__ __forceinline__ void attn_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void attn_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  float2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// Grid: (splits * S, KV, B) in clusters of S along x.  The keys of one (sequence, KV head) are dealt out in 16-key tiles
// to the splits * S CTAs from the length the kernel finds on the device, so that a cache that is mostly empty, or a
// length just past a multiple of anything, leaves no CTA with more than one tile per warp over its share.
//
// What bounds a warp is the chain of a tile: with eight tiles a warp and nothing else on its SM a tile of 16 keys took 0.53 us, as long as with
// twice as many loads in flight.  So all fragments of a tile are read before the first instruction that needs one, and the maximum
// over the warp is taken, and values rescaled, only for a tile that has a new one.  FEW, up to eight heads a KV head: the keys are the 16
// rows of the instruction and the heads its eight columns, half the instructions, exponentials and accumulators of the layout with
// heads as rows, of which half would be zero; the probabilities are transposed in registers.  Microseconds before, after: 1 x 4000 keys
// 7.65, 7.25; 16 x 2000 7.3, 6.9; 64 x 300 6.0, 5.2; 2 x 8000 with 8 KV heads 15.9, 14.9; 256 x 1900 41.5, 40.9; 16 heads a KV head,
// 20 x 3000 11.35, 11.2.  (A maximum raised only by scores that exceed it by eight was another 2 % faster, and 10 % further from 64-bit
// results: the largest probabilities are then no longer exactly one.)
template <typename T, int S, int STAGES, bool FEW, bool ONCE>
__global__ void __launch_bounds__(kAttnThreads, 2) attn_decode_kernel(AttnParams p) {
  static_assert(attn_smem_bytes(STAGES) >= (kAttnWarps * 16 * merge_stride(FEW) + 16 * (kHD + 2)) * 4, "merge buffers");
  extern __shared__ __align__(128) uint8_t attn_smem[];
  constexpr int kMergeStride = merge_stride(FEW);
  const int part = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.G;
  ptx::griddep_launch_dependents();
  if (!p.ahead) ptx::griddep_wait();
  int L = p.pos_dev != nullptr ? static_cast<int>(*p.pos_dev) + 1 : p.len;
  if (L > p.max_len) L = p.max_len;
  if (L < 1) L = 1;
  const long long nt = (L + kTileKeys - 1) / kTileKeys;
  const int parts = p.splits * S;
  const int t0 = static_cast<int>(nt * part / parts), t1 = static_cast<int>(nt * (part + 1) / parts);
  const int h0 = kvh * G;

  const T* kbase = static_cast<const T*>(p.k) + (p.batch0 + b) * p.batch_stride + static_cast<long long>(kvh) * p.max_len * kHD;
  const T* vbase = static_cast<const T*>(p.v) + (p.batch0 + b) * p.batch_stride + static_cast<long long>(kvh) * p.max_len * kHD;
  const uint32_t wbuf_u32 = static_cast<uint32_t>(__cvta_generic_to_shared(attn_smem + warp * attn_warp_bytes(STAGES)));
  // The warps take the CTA's tiles in turn.
  const int my_tiles = t1 - t0 > warp ? (t1 - t0 - warp + kAttnWarps - 1) / kAttnWarps : 0;

  [[maybe_unused]] uint64_t policy = 0;
  [[maybe_unused]] const bool first = ONCE && L >= p.once_len;
  if constexpr (ONCE) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  auto issue_tile = [&](int i, int stage) {
    const int key0 = (t0 + warp + i * kAttnWarps) * kTileKeys;
    const uint32_t ks = wbuf_u32 + stage * 2 * kKvTileBytes, vs = ks + kKvTileBytes;
    auto copy = [&](auto leaves_first) {
      constexpr bool H = decltype(leaves_first)::value;
#pragma unroll
      for (int j = 0; j < kKvTileBytes / 512; ++j) {
        const int r = j * 2 + (lane >> 4), c = lane & 15;  // 16 units of 16 bytes per key row
        const int key = min(key0 + r, L - 1);  // masked later; the address stays inside the written part of the cache
        cp_async_16<H>(ks + kv_off(r, c), kbase + static_cast<long long>(key) * kHD + c * 8, policy);
        cp_async_16<H>(vs + kv_off(r, c), vbase + static_cast<long long>(key) * kHD + c * 8, policy);
      }
    };
    if constexpr (ONCE) {
      if (first) {
        copy(std::true_type{});
      } else {
        copy(std::false_type{});
      }
    } else {
      copy(std::false_type{});
    }
  };

  constexpr int kAcc = FEW ? 8 : 16;
  float o[kAcc][4];
#pragma unroll
  for (int i = 0; i < kAcc; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};

  // One commit group per tile slot, empty when there is no tile: the group count is then the same for every warp
  // and wait<STAGES - 1> always means "tile i has landed".  Ahead of the kernel before: all but the tile with the newest key, which is
  // a warp's last one.
  bool waited = !p.ahead;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < my_tiles) {
      if (!waited && (t0 + warp + s * kAttnWarps + 1) * kTileKeys >= L) {
        ptx::griddep_wait();
        waited = true;
      }
      issue_tile(s, s);
    }
    cp_async_commit();
  }
  if (!waited) ptx::griddep_wait();

  // ---- Q fragments (16 x 128, the A operand; FEW: 128 x 8, the B operand; heads >= G are zero) ----
  const int row0 = lane >> 2, colp = (lane & 3) * 2;
  uint32_t qa[8][FEW ? 2 : 4];
  if constexpr (FEW) {
    const T* qb = static_cast<const T*>(p.q) + (static_cast<long long>(b) * p.H + h0) * kHD;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      qa[ks][0] = row0 < G ? *reinterpret_cast<const uint32_t*>(qb + row0 * kHD + ks * 16 + colp) : 0u;
      qa[ks][1] = row0 < G ? *reinterpret_cast<const uint32_t*>(qb + row0 * kHD + ks * 16 + colp + 8) : 0u;
    }
  } else {
    const T* qb = static_cast<const T*>(p.q) + (static_cast<long long>(b) * p.H + h0) * kHD;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const int c0 = ks * 16 + colp;
      qa[ks][0] = row0 < G ? *reinterpret_cast<const uint32_t*>(qb + row0 * kHD + c0) : 0u;
      qa[ks][1] = row0 + 8 < G ? *reinterpret_cast<const uint32_t*>(qb + (row0 + 8) * kHD + c0) : 0u;
      qa[ks][2] = row0 < G ? *reinterpret_cast<const uint32_t*>(qb + row0 * kHD + c0 + 8) : 0u;
      qa[ks][3] = row0 + 8 < G ? *reinterpret_cast<const uint32_t*>(qb + (row0 + 8) * kHD + c0 + 8) : 0u;
    }
  }
  int stage = 0, fill = STAGES - 1;
  for (int i = 0; i < my_tiles; ++i) {
    if (i + STAGES - 1 < my_tiles) issue_tile(i + STAGES - 1, fill);
    if (++fill == STAGES) fill = 0;
    cp_async_commit();
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    const int key0 = (t0 + warp + i * kAttnWarps) * kTileKeys;
    const uint32_t ks = wbuf_u32 + stage * 2 * kKvTileBytes, vs = ks + kKvTileBytes;
    if (++stage == STAGES) stage = 0;

    if constexpr (FEW) {
      // ---- S^T = K Q^T: 16 keys x 8 heads, in two sums (each instruction waits for the one before it) ----
      float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
      const int mat = lane >> 3;
      uint32_t kf[8][4], vf[8][4];
#pragma unroll
      for (int kp = 0; kp < 8; ++kp) ldmatrix_x4(kf[kp], ks + kv_off((mat & 1) * 8 + (lane & 7), kp * 2 + (mat >> 1)));
#pragma unroll
      for (int dt = 0; dt < 8; ++dt) ldmatrix_x4_trans(vf[dt], vs + kv_off((mat >> 1) * 8 + (lane & 7), dt * 2 + (mat & 1)));
#pragma unroll
      for (int kp = 0; kp < 8; kp += 2) {
        mma_16816<T>(sa, kf[kp], qa[kp][0], qa[kp][1]);
        mma_16816<T>(sb, kf[kp + 1], qa[kp + 1][0], qa[kp + 1][1]);
      }
      // ---- mask, online softmax: a thread has keys row0 and row0 + 8 of heads colp and colp + 1 ----
      float s[4], m_use[2];
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = key0 + row0 + (e >> 1) * 8 < L ? (sa[e] + sb[e]) * p.scale_log2 : -INFINITY;
      if (__any_sync(0xffffffffu, fmaxf(s[0], s[2]) > m_run[0] || fmaxf(s[1], s[3]) > m_run[1])) {
        float tmax[2] = {fmaxf(s[0], s[2]), fmaxf(s[1], s[3])}, corr[2];
#pragma unroll
        for (int x = 4; x < 32; x <<= 1)
#pragma unroll
          for (int h = 0; h < 2; ++h) tmax[h] = fmaxf(tmax[h], __shfl_xor_sync(0xffffffffu, tmax[h], x));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float m_new = fmaxf(m_run[h], tmax[h]);
          corr[h] = exp2f(m_run[h] - (m_new == -INFINITY ? 0.f : m_new));  // 0 when nothing has been seen yet
          m_run[h] = m_new;
          l_run[h] *= corr[h];
        }
#pragma unroll
        for (int i2 = 0; i2 < kAcc; ++i2) {
          o[i2][0] *= corr[0];
          o[i2][1] *= corr[1];
          o[i2][2] *= corr[0];
          o[i2][3] *= corr[1];
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        m_use[h] = m_run[h] == -INFINITY ? 0.f : m_run[h];
        s[h] = exp2f(s[h] - m_use[h]);
        s[h + 2] = exp2f(s[h + 2] - m_use[h]);
        l_run[h] += s[h] + s[h + 2];
      }
      // ---- O^T += V^T P^T ----
      const uint32_t p0 = transpose_8x8(Cvt<T>::pack(s[0], s[1])), p1 = transpose_8x8(Cvt<T>::pack(s[2], s[3]));
#pragma unroll
      for (int dt = 0; dt < 8; ++dt) mma_16816<T>(o[dt], vf[dt], p0, p1);
    } else {
      // ---- S = Q K^T for 16 keys ----
      float s[2][4];
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) s[nb][0] = s[nb][1] = s[nb][2] = s[nb][3] = 0.f;
      uint32_t f[8][4];
#pragma unroll
      for (int i2 = 0; i2 < 8; ++i2) ldmatrix_x4(f[i2], ks + kv_off((i2 & 1) * 8 + (lane & 7), (i2 >> 1) * 4 + (lane >> 3)));
#pragma unroll
      for (int kp = 0; kp < 4; ++kp) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) mma_16816<T>(s[nb], qa[2 * kp + h], f[kp * 2 + nb][h * 2], f[kp * 2 + nb][h * 2 + 1]);
      }
#pragma unroll
      for (int dp = 0; dp < 8; ++dp) ldmatrix_x4_trans(f[dp], vs + kv_off(((lane >> 3) & 1) * 8 + (lane & 7), dp * 2 + (lane >> 4)));
      // ---- mask, online softmax ----
      float tmax[2] = {-INFINITY, -INFINITY}, m_use[2];
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int key = key0 + nb * 8 + colp + (e & 1);
          const float v = key < L ? s[nb][e] * p.scale_log2 : -INFINITY;
          s[nb][e] = v;
          tmax[e >> 1] = fmaxf(tmax[e >> 1], v);
        }
      }
      if (__any_sync(0xffffffffu, tmax[0] > m_run[0] || tmax[1] > m_run[1])) {
        float corr[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tmax[h] = fmaxf(tmax[h], __shfl_xor_sync(0xffffffffu, tmax[h], 1));
          tmax[h] = fmaxf(tmax[h], __shfl_xor_sync(0xffffffffu, tmax[h], 2));
          const float m_new = fmaxf(m_run[h], tmax[h]);
          corr[h] = exp2f(m_run[h] - (m_new == -INFINITY ? 0.f : m_new));  // 0 when nothing has been seen yet
          m_run[h] = m_new;
          l_run[h] *= corr[h];
        }
#pragma unroll
        for (int i2 = 0; i2 < kAcc; ++i2) {
          o[i2][0] *= corr[0];
          o[i2][1] *= corr[0];
          o[i2][2] *= corr[1];
          o[i2][3] *= corr[1];
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) m_use[h] = m_run[h] == -INFINITY ? 0.f : m_run[h];
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float pv = exp2f(s[nb][e] - m_use[e >> 1]);
          s[nb][e] = pv;
          l_run[e >> 1] += pv;
        }
      }
      // ---- O += P V ----
      uint32_t pa[4];
      pa[0] = Cvt<T>::pack(s[0][0], s[0][1]);
      pa[1] = Cvt<T>::pack(s[0][2], s[0][3]);
      pa[2] = Cvt<T>::pack(s[1][0], s[1][1]);
      pa[3] = Cvt<T>::pack(s[1][2], s[1][3]);
#pragma unroll
      for (int dp = 0; dp < 8; ++dp) {
        mma_16816<T>(o[2 * dp], pa, f[dp][0], f[dp][1]);
        mma_16816<T>(o[2 * dp + 1], pa, f[dp][2], f[dp][3]);
      }
    }
    __syncwarp();  // every lane is done with this stage before the next iteration's copies overwrite it
  }
  cp_async_wait<0>();
  // A thread's two heads, and whether it speaks for them.
  const int head0 = FEW ? colp : row0, head_step = FEW ? 1 : 8;
  const bool speaks = FEW ? lane < 4 : (lane & 3) == 0;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int x = FEW ? 4 : 1; x < (FEW ? 32 : 4); x <<= 1) l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], x);

  // ---- merge over the warps.  Every warp scales its own values to the largest maximum of a head before it stores them, so that what is
  // left is a sum.  A warp or CTA without keys has max = -inf and contributes nothing.  What bounds a short context is this tail: 3 - 4 us of
  // 5 - 9 when one thread a dimension went through the heads one by one, 8-way bank conflicts in front (1 sequence, 500 keys
  // 4.7 -> 4.1 us, 16 x 2000 keys 8.4 -> 7.3, 20 x 3000 keys with 16 heads 14.2 -> 11.3).
  __shared__ float warp_max[kAttnWarps * 16], warp_sum[kAttnWarps * 16];
  if (speaks) {
    warp_max[warp * 16 + head0] = m_run[0];
    warp_max[warp * 16 + head0 + head_step] = m_run[1];
  }
  __syncthreads();  // all warps are done with their tile buffers: shared memory is reused from here on
  float* mo = reinterpret_cast<float*>(attn_smem);   // [warp][16][kMergeStride]
  float* co = mo + kAttnWarps * 16 * kMergeStride;   // the CTA's result: [16][kHD], then (max, sum) of each head
  float* cml = co + 16 * kHD;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = head0 + h * head_step;
    float m_tot = warp_max[row];
#pragma unroll
    for (int w = 1; w < kAttnWarps; ++w) m_tot = fmaxf(m_tot, warp_max[w * 16 + row]);
    const float f = m_run[h] == -INFINITY ? 0.f : exp2f(m_run[h] - m_tot);
    if (speaks) warp_sum[warp * 16 + row] = f * l_run[h];
    if constexpr (FEW) {
      if (row < G) {
        float* dst = mo + (warp * 16 + row) * kMergeStride + row0;
#pragma unroll
        for (int dt = 0; dt < 8; ++dt) {
          dst[dt * 16] = f * o[dt][h];
          dst[dt * 16 + 8] = f * o[dt][h + 2];
        }
      }
    } else if (row < G) {
      float* dst = mo + (warp * 16 + row) * kMergeStride + colp;
#pragma unroll
      for (int nb = 0; nb < 16; ++nb) *reinterpret_cast<float2*>(dst + nb * 8) = make_float2(f * o[nb][2 * h], f * o[nb][2 * h + 1]);
    }
  }
  __syncthreads();
  // A unit is four dimensions of a head.
  auto deliver = [&](int u, const float4& acc, float m_tot, float l_tot) {
    const int g = u >> 5, d = (u & 31) * 4;
    const long long hrow = static_cast<long long>(b) * p.H + h0 + g;
    if (p.splits == 1) {
      *reinterpret_cast<uint2*>(static_cast<T*>(p.out) + hrow * kHD + d) =
          make_uint2(Cvt<T>::pack(acc.x / l_tot, acc.y / l_tot), Cvt<T>::pack(acc.z / l_tot, acc.w / l_tot));
    } else {
      float* w = p.ws + (hrow * p.splits + part / S) * kPartialStride;
      if (p.ws_pairs) {
        *reinterpret_cast<float2*>(w + d) = make_float2(acc.x, acc.y);
        *reinterpret_cast<float2*>(w + d + 2) = make_float2(acc.z, acc.w);
        if (d == 0) *reinterpret_cast<float2*>(w + kHD) = make_float2(m_tot, l_tot);
      } else {
        w[d] = acc.x;
        w[d + 1] = acc.y;
        w[d + 2] = acc.z;
        w[d + 3] = acc.w;
        if (d == 0) {
          w[kHD] = m_tot;
          w[kHD + 1] = l_tot;
        }
      }
    }
  };
  for (int u = threadIdx.x; u < G * 32; u += kAttnThreads) {
    const int g = u >> 5;
    const float* src = mo + g * kMergeStride + (u & 31) * 4;
    float4 acc = *reinterpret_cast<const float4*>(src);
    float l_tot = warp_sum[g], m_tot = warp_max[g];
#pragma unroll
    for (int w = 1; w < kAttnWarps; ++w) {
      const float4 v = *reinterpret_cast<const float4*>(src + w * 16 * kMergeStride);
      acc = make_float4(acc.x + v.x, acc.y + v.y, acc.z + v.z, acc.w + v.w);
      l_tot += warp_sum[w * 16 + g];
      m_tot = fmaxf(m_tot, warp_max[w * 16 + g]);
    }
    if constexpr (S == 1) {
      deliver(u, acc, m_tot, l_tot);
    } else {
      *reinterpret_cast<float4*>(co + u * 4) = acc;
      if ((u & 31) == 0) *reinterpret_cast<float2*>(cml + g * 2) = make_float2(m_tot, l_tot);
    }
  }
  if constexpr (S > 1) {
    // ---- merge over the cluster through distributed shared memory: the units are dealt out to its CTAs ----
    const int rank = part % S;
    const uint32_t co_a = static_cast<uint32_t>(__cvta_generic_to_shared(co)), cml_a = static_cast<uint32_t>(__cvta_generic_to_shared(cml));
    attn_cluster_sync();
    const int u1 = G * 32 * (rank + 1) / S, u_first = G * 32 * rank / S;
    const int turns = (u1 - u_first + kAttnThreads - 1) / kAttnThreads;  // at least one: G >= 1, S <= 8
    for (int turn = 0; turn < turns; ++turn) {
      const int u = u_first + turn * kAttnThreads + int(threadIdx.x);
      const bool live = u < u1;
      float4 v[S], acc = make_float4(0.f, 0.f, 0.f, 0.f);
      float2 ml[S];
      float m_tot = -INFINITY, l_tot = 0.f;
      if (live) {
#pragma unroll
        for (int r = 0; r < S; ++r) {
          ml[r] = ld_cluster_f2(cml_a + (u >> 5) * 8, r);
          v[r] = ld_cluster_f4(co_a + u * 16, r);
        }
#pragma unroll
        for (int r = 0; r < S; ++r) m_tot = fmaxf(m_tot, ml[r].x);
#pragma unroll
        for (int r = 0; r < S; ++r) {
          const float f = ml[r].x == -INFINITY ? 0.f : exp2f(ml[r].x - m_tot);
          acc = make_float4(acc.x + f * v[r].x, acc.y + f * v[r].y, acc.z + f * v[r].z, acc.w + f * v[r].w);
          l_tot += f * ml[r].y;
        }
      }
      // All parts are read: the barrier need not wait for the stores of the last result.  A peer may end behind it, and a load from it
      // that is still under way then faults; what makes an instruction wait for a load is its use.  No value equals the NaN, which is
      // no constant to the compiler: the stores never happen.
      if (turn + 1 == turns) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.f32 p, %0, %2;\n\t@p st.shared.f32 [%3], %0;\n\tsetp.eq.f32 p, %1, %2;\n\t@p st.shared.f32 [%3], %1;\n\t}" ::"f"(acc.x), "f"(l_tot), "f"(p.nan), "r"(cml_a) : "memory");
        __syncwarp();
        attn_cluster_arrive();
      }
      if (live) deliver(u, acc, m_tot, l_tot);
    }
    __syncwarp();
    attn_cluster_wait();  // the peers have read this CTA's part
  }
}

// Merges the key chunks of one (sequence, head): grid = B * H, 128 threads.  PAIRS: see AttnParams::ws_pairs.
template <typename T, bool PAIRS>
__global__ void attn_combine_kernel(const float* ws, void* out, int splits) {
  const long long hrow = blockIdx.x;
  const int d = threadIdx.x;
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  // A lane a part: all maxima and sums are on their way at once, as are the values, eight parts at a time (a thread that went through the
  // parts one by one: 1 x 32000 keys in seven parts 12.2 us, 10.2 so; 8 x 9000 keys 17.7, 17.1).
  const float* w = ws + hrow * splits * kPartialStride;
  const int lane = threadIdx.x & 31;
  float m_tot = -INFINITY, acc = 0.f, l_tot = 0.f;
  for (int s0 = 0; s0 < splits; s0 += 32) {
    const int n = min(splits - s0, 32);
    float2 ml = make_float2(-INFINITY, 0.f);
    if (lane < n) {
      const float* p = w + (s0 + lane) * kPartialStride + kHD;
      if constexpr (PAIRS) {
        ml = *reinterpret_cast<const float2*>(p);
      } else {
        ml = make_float2(p[0], p[1]);
      }
    }
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < n ? w[(s0 + i) * kPartialStride + d] : 0.f;
    float m_new = fmaxf(m_tot, ml.x);
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, x));
    // A part without keys may hold anything; one whose factor underflows has values, and a NaN or infinity among them is passed on.
    const unsigned some = __ballot_sync(0xffffffffu, ml.x != -INFINITY);
    const float f = ml.x == -INFINITY ? 0.f : exp2f(ml.x - m_new);
    float l = ml.x == -INFINITY ? 0.f : f * ml.y;
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
    if (s0 > 0) {
      const float corr = m_tot == -INFINITY ? 0.f : exp2f(m_tot - m_new);
      acc *= corr;
      l_tot *= corr;
    }
    for (int i0 = 0; i0 < n; i0 += 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float fi = __shfl_sync(0xffffffffu, f, (i0 + i) & 31);
        if (i0 + i < n && (some >> ((i0 + i) & 31) & 1)) acc += fi * v[i];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = i0 + 8 + i < n ? w[(s0 + i0 + 8 + i) * kPartialStride + d] : 0.f;
    }
    l_tot += l;
    m_tot = m_new;
  }
  static_cast<T*>(out)[hrow * kHD + d] = to_out<T>(acc / l_tot);
}

template <typename T, int S, int STAGES, bool FEW, bool ONCE>
cudaError_t launch_attn_s(const AttnParams& p, cudaStream_t stream) {
  static std::atomic<uint64_t> attr_done{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_done.load(std::memory_order_relaxed) >> (dev & 63) & 1)) {
    cudaError_t e = cudaFuncSetAttribute(attn_decode_kernel<T, S, STAGES, FEW, ONCE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         attn_smem_bytes(STAGES));
    if (e != cudaSuccess) return e;
    attr_done.fetch_or(uint64_t(1) << (dev & 63), std::memory_order_relaxed);
  }
  return launch_pdl(attn_decode_kernel<T, S, STAGES, FEW, ONCE>, dim3(p.splits * S, p.KV, p.B), kAttnThreads, attn_smem_bytes(STAGES), stream, S, p);
}

template <typename T>
cudaError_t launch_attn(const AttnParams& p, int cluster, bool deep, bool once, cudaStream_t stream) {
  constexpr int A = kAttnStages, D = kAttnDeepStages;
  auto size = [&](auto few, auto read_once) {
    constexpr bool F = decltype(few)::value, O = decltype(read_once)::value;
    switch (cluster) {
      case 1: return deep ? launch_attn_s<T, 1, D, F, O>(p, stream) : launch_attn_s<T, 1, A, F, O>(p, stream);
      case 2: return deep ? launch_attn_s<T, 2, D, F, O>(p, stream) : launch_attn_s<T, 2, A, F, O>(p, stream);
      case 4: return launch_attn_s<T, 4, A, F, O>(p, stream);
      default: return launch_attn_s<T, 8, A, F, O>(p, stream);
    }
  };
  cudaError_t e = p.G > 8 ? size(std::false_type{}, std::false_type{})
                  : once  ? size(std::true_type{}, std::true_type{})
                          : size(std::true_type{}, std::false_type{});
  if (e != cudaSuccess) return e;
  if (p.splits > 1) e = launch_pdl(p.ws_pairs ? attn_combine_kernel<T, true> : attn_combine_kernel<T, false>, dim3(p.B * p.H), kHD, 0, stream, 1, p.ws, p.out, p.splits);
  return e;
}

// CTAs that run at once in clusters of 1, 2, 4 and 8.  Two fit an SM, but a cluster lives in one GPC, and how many SMs a GPC has
// may differ from one GPU to the next: the device is asked.
struct AttnSlots {
  int n[4];
  int deep[2];  // of the kernel with kAttnDeepStages, alone and in pairs
};

template <typename T, int S, int STAGES, bool FEW = true, bool ONCE = false>
int attn_slots_of() {
  if (cudaFuncSetAttribute(attn_decode_kernel<T, S, STAGES, FEW, ONCE>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_smem_bytes(STAGES)) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(S * 2 * 148);
  cfg.blockDim = dim3(kAttnThreads);
  cfg.dynamicSmemBytes = attn_smem_bytes(STAGES);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, attn_decode_kernel<T, S, STAGES, FEW, ONCE>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return clusters * S;
}

// The same kernel shape for both types: one answer per device.
AttnSlots attn_slots() {
  static std::mutex mu;
  static AttnSlots cached[64];
  static bool have[64];
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> g(mu);
  AttnSlots& s = cached[dev & 63];
  if (!have[dev & 63]) {
    s.n[0] = 2 * 148;
    s.n[1] = attn_slots_of<__nv_bfloat16, 2, kAttnStages>();
    s.n[2] = attn_slots_of<__nv_bfloat16, 4, kAttnStages>();
    s.n[3] = attn_slots_of<__nv_bfloat16, 8, kAttnStages>();
    s.deep[0] = 148;
    s.deep[1] = attn_slots_of<__nv_bfloat16, 2, kAttnDeepStages>();
    have[dev & 63] = true;
  }
  return s;
}

// Nanoseconds for `items` (sequence, KV head) pairs of `len` keys with s CTAs each, `slots` of which run at once.  A key takes a
// CTA 8 ns where its own loads in flight are the limit and 23 ns where 296 CTAs share the memory's rate; the limits blend.
// Starting a CTA and merging takes 2.6 us, 4.2 us in a cluster.
double attn_cost_ns(long long items, int s, int slots, double len) {
  slots -= slots % s;
  const long long rounds = items * s / slots, rest = items * s % slots;
  const double keys = len / s, fixed = s > 1 ? 4200.0 : 2600.0;
  auto ns_key = [](double ctas) {
    const double shared = 23.0 * ctas / 296;
    return std::cbrt(512.0 + shared * shared * shared);
  };
  return rounds * (ns_key(slots) * keys + fixed) + (rest > 0 ? ns_key(double(rest)) * keys + fixed : 0.0);
}

// CTAs of a cluster that share the keys of one (sequence, KV head).  The host knows a bound of the length, not the length, so a
// size is weighed at the bound and at a third of it, each against one CTA: a cluster that gains little on a full cache loses
// several times over on a short context, where all it adds is CTAs.  The constants of attn_cost_ns were fitted to the kernel before this one,
// whose merges took 0.5 - 3 us longer (0.3 % off the best size at full caches).  With this one, every size timed over 171 combinations of batch, heads,
// bound and length on B200, the choice is 2.9 % off the best size at full caches (11 of 57 more than 3 %, most of them of less than 500 keys, where more CTAs
// would pay), 0.7 % at a third and 14 % at a thirtieth of the bound (20 sequences with 16 heads, 59 of 1974 keys 5.9 us, 3.8 without clusters).  The rule that
// looked at whole rounds at the bound only took four CTAs for 300 items of a 2048-key cache with 16 keys in it (20.3 us, 5.6 with
// one) and for 600 items with 500 keys in it (68.5, 33.5).
int attn_cluster_size(long long items, int len_bound, const AttnSlots& slots) {
  // With a CTA for every SM the memory is busy: clusters gained 8 % at most on full caches (192 items of 8192 keys 119 us in fours, 129)
  // and lost up to 2.5 times on short contexts (150 items, 100 of 8192 keys 11.4 in pairs, 6.1).
  if (items > 148) return 1;
  const double third = len_bound / 3.0;
  const double one = attn_cost_ns(items, 1, slots.n[0], len_bound), one_third = attn_cost_ns(items, 1, slots.n[0], third);
  int best = 1;
  double best_cost = 2.0;
  for (int i = 1; i < 4; ++i) {
    const int s = 1 << i;
    if (slots.n[i] < s || len_bound < s * kTileKeys * kAttnWarps) continue;
    const double cost = attn_cost_ns(items, s, slots.n[i], len_bound) / one + attn_cost_ns(items, s, slots.n[i], third) / one_third;
    if (cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace model
}  // namespace oob

using namespace oob;
using namespace oob::model;

extern "C" {

int oob_rope_kv_write(const oob_rope_args_t* a, void* stream) {
  if (a == nullptr) return set_error(OOB_ERR_INVALID, "null argument");
  if (a->dtype != OOB_F16 && a->dtype != OOB_BF16) return set_error(OOB_ERR_INVALID, "dtype must be fp16 or bf16");
  if (a->B <= 0 || a->T <= 0 || a->H <= 0 || a->KV <= 0 || a->hd <= 0 || a->hd % 8 != 0)
    return set_error(OOB_ERR_INVALID, "bad RoPE shape");
  if (a->qkv == nullptr || a->q_out == nullptr || a->k_cache == nullptr || a->v_cache == nullptr ||
      a->cos_table == nullptr || a->sin_table == nullptr)
    return set_error(OOB_ERR_INVALID, "null pointer");
  if (a->batch0 < 0 || a->max_len <= 0 || a->cache_batch_stride < int64_t(a->KV) * a->max_len * a->hd)
    return set_error(OOB_ERR_INVALID, "bad cache geometry");
  if (a->pos_dev == nullptr && (a->pos0 < 0 || a->pos0 + a->T > a->max_len))
    return set_error(OOB_ERR_INVALID, "positions outside the cache");
  const uintptr_t align = reinterpret_cast<uintptr_t>(a->qkv) | reinterpret_cast<uintptr_t>(a->q_out) |
                          reinterpret_cast<uintptr_t>(a->k_cache) | reinterpret_cast<uintptr_t>(a->v_cache) |
                          reinterpret_cast<uintptr_t>(a->cos_table) | reinterpret_cast<uintptr_t>(a->sin_table);
  if (align & 15) return set_error(OOB_ERR_INVALID, "pointers must be 16-byte aligned");
  if ((a->cache_batch_stride % 8) != 0) return set_error(OOB_ERR_INVALID, "cache stride must be a multiple of 8 elements");
  const long long units = static_cast<long long>(a->B) * a->T * (a->H + 2 * a->KV) * (a->hd / 8);
  const int threads = 256;
  long long blocks = (units + threads - 1) / threads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = launch_pdl(a->dtype == OOB_BF16 ? rope_kv_write_kernel<__nv_bfloat16> : rope_kv_write_kernel<__half>,
                                   dim3(static_cast<int>(blocks)), threads, 0, s, 1, *a, units);
  if (e != cudaSuccess) return cuda_fail(e, "rope_kv_write launch");
  return OOB_OK;
}

int oob_silu_mul(int dtype, const void* gu, int64_t ld_gu, void* out, int rows, int F, void* stream) {
  if (dtype != OOB_F16 && dtype != OOB_BF16) return set_error(OOB_ERR_INVALID, "dtype must be fp16 or bf16");
  if (gu == nullptr || out == nullptr || rows <= 0 || F <= 0 || F % 8 != 0 || ld_gu < 2 * int64_t(F) || ld_gu % 8 != 0)
    return set_error(OOB_ERR_INVALID, "bad SwiGLU arguments");
  if ((reinterpret_cast<uintptr_t>(gu) | reinterpret_cast<uintptr_t>(out)) & 15)
    return set_error(OOB_ERR_INVALID, "pointers must be 16-byte aligned");
  const long long units = static_cast<long long>(rows) * (F / 8);
  const int threads = 256;
  long long blocks = (units + threads - 1) / threads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const dim3 grid(static_cast<int>(blocks));
  const cudaError_t e =
      dtype == OOB_BF16 ? launch_pdl(silu_mul_kernel<__nv_bfloat16>, grid, threads, 0, s, 1, static_cast<const __nv_bfloat16*>(gu),
                                     ld_gu, static_cast<__nv_bfloat16*>(out), units, F)
                        : launch_pdl(silu_mul_kernel<__half>, grid, threads, 0, s, 1, static_cast<const __half*>(gu), ld_gu,
                                     static_cast<__half*>(out), units, F);
  if (e != cudaSuccess) return cuda_fail(e, "silu_mul launch");
  return OOB_OK;
}

int oob_attn_decode_auto_splits(int B, int KV, int len_bound) {
  if (B <= 0 || KV <= 0 || len_bound <= 0) return 1;
  // A cluster of eight CTAs shares the keys of one (sequence, KV head) without touching memory; more CTAs are only worth
  // the round trip of their partial results, and a second kernel, when few sequences are long.
  const long long ctas = static_cast<long long>(B) * KV * kMaxAttnCluster;
  long long s = (148 + ctas - 1) / ctas;
  const int max_by_len = len_bound / (kMaxAttnCluster * 512);
  if (s > max_by_len) s = max_by_len;
  if (s > 32) s = 32;
  if (s < 1) s = 1;
  return static_cast<int>(s);
}

int oob_test_attn_cluster_size(long long items, int len_bound, int slots2, int slots4, int slots8) {
  if (items <= 0 || len_bound <= 0) return -1;
  return oob::model::attn_cluster_size(items, len_bound, {{2 * 148, slots2, slots4, slots8}});
}

uint64_t oob_attn_decode_workspace_bytes(int B, int H, int splits) {
  if (splits <= 1) return 0;
  return uint64_t(B) * H * splits * kPartialStride * sizeof(float);
}

int oob_attn_decode(const oob_attn_decode_args_t* a, void* stream) {
  if (a == nullptr) return set_error(OOB_ERR_INVALID, "null argument");
  if (a->dtype != OOB_F16 && a->dtype != OOB_BF16) return set_error(OOB_ERR_INVALID, "dtype must be fp16 or bf16");
  if (a->B <= 0 || a->H <= 0 || a->KV <= 0 || a->H % a->KV != 0 || a->H / a->KV > 16)
    return set_error(OOB_ERR_INVALID, "bad head counts (at most 16 query heads per KV head)");
  if (a->q == nullptr || a->k_cache == nullptr || a->v_cache == nullptr || a->out == nullptr)
    return set_error(OOB_ERR_INVALID, "null pointer");
  if (a->max_len <= 0 || a->batch0 < 0 || a->cache_batch_stride < int64_t(a->KV) * a->max_len * kHD ||
      a->cache_batch_stride % 8 != 0)
    return set_error(OOB_ERR_INVALID, "bad cache geometry");
  if (a->pos_dev == nullptr && (a->len < 1 || a->len > a->max_len)) return set_error(OOB_ERR_INVALID, "bad context length");
  if ((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k_cache) |
       reinterpret_cast<uintptr_t>(a->v_cache) | reinterpret_cast<uintptr_t>(a->out)) & 15)
    return set_error(OOB_ERR_INVALID, "pointers must be 16-byte aligned");
  int bound = a->len_bound > 0 ? a->len_bound : a->max_len;
  if (bound > a->max_len) bound = a->max_len;
  if (a->pos_dev == nullptr && a->len > bound) bound = a->len;
  int splits = a->splits > 0 ? a->splits : oob_attn_decode_auto_splits(a->B, a->KV, bound);
  if (splits > 65535) return set_error(OOB_ERR_INVALID, "too many splits");
  if (splits > 1 && a->workspace == nullptr) return set_error(OOB_ERR_INVALID, "splits > 1 need a workspace");
  if (splits > 1 && (reinterpret_cast<uintptr_t>(a->workspace) & 3)) return set_error(OOB_ERR_INVALID, "the workspace holds floats: four-byte aligned");
  AttnParams p{};
  p.q = a->q;
  p.k = a->k_cache;
  p.v = a->v_cache;
  p.out = a->out;
  p.ws = a->workspace;
  p.ws_pairs = (reinterpret_cast<uintptr_t>(a->workspace) & 7) == 0;
  p.pos_dev = reinterpret_cast<const long long*>(a->pos_dev);
  p.len = a->len;
  p.B = a->B;
  p.H = a->H;
  p.KV = a->KV;
  p.G = a->H / a->KV;
  p.batch_stride = a->cache_batch_stride;
  p.max_len = a->max_len;
  p.batch0 = a->batch0;
  p.splits = splits;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.nan = NAN;
  p.ahead = a->ahead != 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  AttnSlots slots = attn_slots();
  // Behind a split launch waits the kernel that merges, and calls follow one another: clusters of eight that need every slot of
  // the GPU then wait for the last ones (2 x 30000 keys on 8 KV heads 48 - 55 us in eights, 45 in fours; alone both 44).
  if (splits > 1) slots.n[3] -= slots.n[3] / 4;
  const int cluster = attn_cluster_size(static_cast<long long>(a->B) * a->KV * splits, (bound + splits - 1) / splits, slots);
  const long long key_bytes = static_cast<long long>(a->B) * a->KV * (4 * kHD);  // of one key and value of all sequences
  const bool once = key_bytes * bound >= kOnceBytes;
  p.once_len = static_cast<int>((kOnceBytes + key_bytes - 1) / key_bytes);
  const bool deep = cluster <= 2 && static_cast<long long>(a->B) * a->KV * splits * cluster <= slots.deep[cluster - 1];
  cudaError_t e = a->dtype == OOB_BF16 ? launch_attn<__nv_bfloat16>(p, cluster, deep, once, s) : launch_attn<__half>(p, cluster, deep, once, s);
  if (e != cudaSuccess) return cuda_fail(e, "attn_decode launch");
  return OOB_OK;
}

}  // extern "C"
