// Weight-streaming tcgen05 GEMM for few rows: C[M, N] = A[M, K] * B[N, K]^T is computed as C^T = B * A^T, so the WEIGHT rows
// fill the 128-row dimension of the tensor-core instruction and the tokens are its N dimension (16 .. 256).  This is the GEMM
// of a decode step or of a short mixed batch: what bounds it is the time to read B once, plus whatever happens before the
// first and after the last byte.
//
// A CTA goes through 64 elements of K in 0.11 - 0.15 us (the chain load - multiply - release of its issuing threads), so that
// neither few CTAs nor long K ranges reach the memory's rate.  128-row weight tiles are therefore computed by S CTAs, each over 1/S
// of K; a cost model on the host picks S and the token blocks.
//
// Split over K inside a thread-block cluster (S = 1 .. 8).  When a CTA has its partial sums it drains them from TMEM into its
// own shared memory (the pipeline buffers, idle by then) as [token][128] fp32; after one cluster barrier each CTA reads its share
// of the tokens from all S copies through distributed shared memory, adds them in rank order (deterministic) and writes
// the 16-bit result.  Nothing goes through global memory and no second kernel has to be launched.
//
// PAIR: two CTAs of the cluster form a tensor-core pair (cta_group::2) on 256 weight rows.  Each stages its own 128 weight
// rows and HALF of the tokens, and keeps the sums of its own rows.  From about 128 tokens on the activations, which every
// weight tile reads again, rival the weights on the way from L2 to the SMs; a pair halves them.
//
// RMSNorm around it (a decode step, ParamsC::row_ssq and the Add epilogue): the GEMM in front of a norm adds the residual, writes the
// new residual stream h and h * norm weight, and each tile the sum of h^2 of its columns; the GEMM behind the norm multiplies its sums
// by 1 / rms of their row.  No norm kernel stands between the two.
//
// Epilogues applied to the fp32 sums before the only rounding:
//   SwiGLU     a tile is 64 gate rows + 64 up rows of the [gate | up] weight; out = silu(gate) * up
//   RoPE + KV  query and key heads are rotated, queries go to q_out, keys and values into the layer's cache
//
// Measured on B200, bf16, in a chain of launches (before: fp32 partial tiles through memory and a second kernel that sums
// them): 16 x 7168 x 8192 20.6 us (26.5), 32 x 8192 x 3584 12.2 (18.2 with 16 rows), 8 x 8192 x 1024 6.1 (10.6), 8 x 1280 x 8192 7.4 (14.3),
// 128 x 7168 x 8192 24.0 (27.5), 64 x 7168 x 8192 22.9 (29.6), 128 x 4096 x 4096 12.2, 512 x 1280 x 8192 17.5 (21.6).
//
// Roles: warp 0 loads weights, warp 1 issues the MMAs, warp 2 loads activations (one thread each), warps 2-5 drain TMEM; all six
// warps take part in the reduction.  A cluster handles tiles c, c + G, ... one after the other; normally the grid covers all tiles, a CTA
// budget (max_ctas) makes G smaller.  All waits are bounded, and a CTA that gives up still meets its cluster's barriers.
//
// Capability parity with the reference: its stream-K GEMM instances (src/gemm/gemm_with_signal_sm90.h:238-292) and the
// small-M end of its plain-GEMM dispatch table (src/gemm/gemm_plain_sm90_dispatch.h:19-46).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <limits>
#include <type_traits>

#include "../api/oob.h"
#include "../api/oob_model.h"
#include "gemm_kernel.cuh"
#include "gemm_pair.h"

namespace oob {
namespace gemm_cluster {

using namespace gemm_detail;

constexpr int kRowsW = 128;                  // weight rows of a CTA (the instruction's M)
constexpr int kRowBytes = kTileK * 2;        // 128: one row of a stage
constexpr int kMaxTokens = 256;              // per instruction (its N)
constexpr int kMaxTileTokens = 384;          // per tile: what its fp32 sums leave of an SM's shared memory; more rows are cut into blocks
// Up to this many tokens a stage holds 128 elements of K: half the waits and commits per byte (one CTA, 16 tokens: 0.107 us per
// 64 elements, 128 tokens with 64 elements a stage 0.142).  With more tokens it would leave too few stages
// (128 x 7168 x 8192 27.1 us with 64 elements and 27.6 with 128, 128 x 8192 x 3584 split four ways 17.6 and 22.8).
constexpr int kWideTokens = 64;
// The first stage of a CTA's weights is fetched into L2 while the kernel before this one ends (0.7 us from its end to the return of the wait for
// it, then 1.4 us to weights from memory and 0.8 to weights from L2), where the weight is large enough not to be in L2 as a matter of course and
// its rows start on a line.  One stage: over 728 shapes of 1 - 64 rows in a chain of calls on weights from memory 0.984 of the time, 3 of 330 more than
// 2 % slower, on weights from L2 1.002.  All of up to eight stages: 0.973 and 1.018, 43 and 130 shapes slower, by up to 13 %: many CTAs' loads wait behind
// what is fetched.  Weights of less than kFetchBytes are slower by up to 6 % where they are in L2 (1024 x 2048, 16 rows 4.26 -> 4.48 us); rows off a
// line, whose boxes are two lines a row, are slower from memory as well (40 x 2736 x 1880 6.7 -> 7.3, 54 x 4800 x 3032 with SwiGLU 10.7 -> 11.9) but for
// weights that leave L2 first (three weights of 99 - 119 MB, 3 - 100 rows: 0.95 - 0.99 of the time).
// From kFetchTwoBytes on two stages: 16 x 8192 x 4096 13.5 -> 13.3 us, 64 x 8192 x 4096 14.0 -> 13.8; 16 x 7168 x 8192 21.3 -> 20.95.
constexpr long long kFetchBytes = 8ll << 20, kFetchTwoBytes = 32ll << 20;
// With one token block a launch reads every weight once, and weights that will not be in L2 the next time leave it first: they then drive out neither
// what is read again nor what has just been written.  One weight used again and again is in L2 up to some 70 MB (more than half of it: both dies hold
// some lines).  Time with such loads to time without, 3 - 64 rows, K of 4096 and 8192, one weight in repeated calls / two / three in turn: 40 MB 1.00 / 1.08 /
// 0.95, 56 MB 1.03 / 0.95 / 0.96, 72 MB 1.03 / 0.93 / 0.95, 80 MB 0.99 / 0.97 / 0.95, 96 MB 0.97 / 0.97 / 0.97, 112 MB 0.94 / 0.95 / 0.95.  So from kOnceBytes on for a
// single call, and below only where the caller says that the weights are part of a chain that L2 does not hold (a layer of a decode step of 32 sequences
// 60.1 -> 55.0 us; but four weights of 32 MB in turn 8.25 -> 8.9): weights of kOnceChainBytes and more, smaller ones gain nothing.
constexpr long long kOnceBytes = 80ll << 20, kOnceChainBytes = 8ll << 20;
constexpr int kThreadsC = 192;
constexpr int kMaxStagesC = 12;
constexpr int kSpreadRows = 32, kSpreadMost = 1500;  // rows between which blocks of fewer tokens than 128 are weighed, down to the first
constexpr int kSpreadBlocks = 10;            // as far as they were timed
constexpr double kSpreadGain[2] = {0.82, 0.943};  // up to 128 rows and above, see planned
constexpr double kSpreadTwoSm = 1.235;       // see gemm_cluster_preferred
constexpr int kMaxCluster = 8;               // portable cluster size
constexpr int kMaxScaledRows = 128;           // rows that may carry a sum of squares (ParamsC::row_ssq)
constexpr int kCtlBytes = 256 + kMaxScaledRows * 4;
constexpr int kSmemLimit = 227 * 1024;

enum { kEpiPlain = 0, kEpiSwiglu = 1, kEpiRopeKv = 2, kEpiAdd = 3 };

// The fetch is paid for in registers of the sums, 4 - 6 a thread.  Where four CTAs share an SM they would be spilled, 12 - 28 bytes of 80; in the SwiGLU kernels they
// cost what it gives (1 - 32 rows, weights in L2 1.02, from memory 1.00) but for weights that leave L2 first (16 x 7168 x 8192 21.8 -> 20.9 us, 16 x 28672 x 4096
// 40.0 -> 37.7).
constexpr bool fetches(int epi, int res, bool once) { return res < 4 && (epi != kEpiSwiglu || once); }

struct CtlC {
  uint64_t full[kMaxStagesC];
  uint64_t empty[kMaxStagesC];
  uint64_t tmem_full;
  uint32_t tmem_base;
  int abort;
  float scale[kMaxScaledRows];  // 1 / rms of the rows of A
};
static_assert(sizeof(CtlC) <= kCtlBytes, "control block");

struct ParamsC {
  int M, N, Mp;  // Mp: tokens of a tile = n_mma * nj
  int n_mma, nj;  // instructions per K step and their N, a multiple of 16
  int m_blocks;  // token blocks; tile t is block t % m_blocks of weight tile t / m_blocks
  int F;         // SwiGLU: gate rows (N = 2F)
  void* C;
  int ldc;
  int num_kb, num_tiles, clusters;  // num_kb: pipeline stages' worth of K (sub * 64 elements each)
  int sub;
  int S;  // CTAs (pairs) that share the K range of a tile
  int per_sm;  // CTAs of an SM (the host's)
  int stages, stage_bytes, work_bytes;  // work_bytes: pipeline buffers or partial sums, whichever is larger
  int smem_bytes;
  uint32_t tmem_cols;
  bool vec_ok;  // 8-byte stores into C are aligned
  bool w_static;  // the weights may be loaded before the kernels this one depends on are done
  oob_rope_args_t rope;
  // Rows of A that are still to be divided by their rms: its sums of squares in `row_parts` pieces, [part][M]; null: none.
  const float* row_ssq;
  int row_parts;
  float row_eps, inv_k;
  float nan;  // see settle
  bool once;  // which kernel the host takes
  int fetch;  // stages of weights, at most two, that a CTA fetches into L2 before the wait for earlier kernels (see kFetchBytes)
  oob_gemm_epilogue_add_t add;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The two halves of cluster_sync.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
// Waits for the loads that `x` comes from.  A CTA may end when its peers have arrived at the last cluster barrier, and a load from it that
// is still under way then faults; nothing but its use makes an instruction wait for a load, and one whose result goes nowhere (past the
// last column) is not waited for.  `nan` is no constant to the compiler, and equal to nothing: the store never happens.
__device__ __forceinline__ void settle(float x, float nan, uint32_t smem_addr) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.f32 p, %0, %1;\n\t@p st.shared.f32 [%2], %0;\n\t}" ::"f"(x), "f"(nan), "r"(smem_addr) : "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The cta_group::2 forms.  A load goes into THIS CTA's shared memory and counts its bytes on the leader's barrier.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar_cluster_addr, int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(ptx::smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in every CTA of `mask` once all MMAs issued so far are complete.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(ptx::smem_u32(bar)),
      "h"(mask)
      : "memory");
}

// ONCE: `policy` says how the box is kept in L2.
template <bool PAIR, bool ONCE = false>
__device__ __forceinline__ void load_box(void* smem_dst, const void* tmap, uint32_t bar, int32_t x, int32_t y, uint64_t policy = 0) {
  if constexpr (ONCE) {
    static_assert(!PAIR, "a pair's weights are read by every token block");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
        :
        : "r"(ptx::smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y), "l"(policy)
        : "memory");
  } else if constexpr (PAIR) {
    tma_load_2d_pair(smem_dst, tmap, bar, x, y);
  } else {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        :
        : "r"(ptx::smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y)
        : "memory");
  }
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (PackTraits<T>::kDType == kBF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}

template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (PackTraits<T>::kDType == kBF16) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  } else {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
}

// Where a unit of a query, key or value head goes, and the rotation it gets.
struct RopeUnit {
  float2 cs, sn;
  long long pos;
  int hh, c, b;
};
__device__ __forceinline__ RopeUnit rope_unit(const ParamsC& p, int m, int n, long long pos_base) {
  const oob_rope_args_t& a = p.rope;
  RopeUnit r;
  r.hh = n / a.hd;
  r.c = n - r.hh * a.hd;
  r.b = m / a.T;
  r.pos = pos_base + (m - r.b * a.T);
  if (r.pos < 0) r.pos = 0;
  if (r.pos > a.max_len - 1) r.pos = a.max_len - 1;  // the host checks the range; never index outside the tables / cache
  r.cs = r.sn = make_float2(0.f, 0.f);
  if (r.hh < a.H + a.KV) {
    r.cs = *reinterpret_cast<const float2*>(a.cos_table + r.pos * (a.hd / 2) + r.c / 2);
    r.sn = *reinterpret_cast<const float2*>(a.sin_table + r.pos * (a.hd / 2) + r.c / 2);
  }
  return r;
}

// Writes token `m`, output columns n .. n + 3 (SwiGLU: `v` gate sums, `u` up sums).
template <typename T, int EPI>
__device__ __forceinline__ void emit(const ParamsC& p, int m, int n, const float4& v, const float4& u, const RopeUnit& r) {
  if constexpr (EPI == kEpiSwiglu) {
    if (n >= p.F) return;  // F % 8 == 0: the four columns are in or out together
    uint32_t g[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
    const uint32_t up[4] = {__float_as_uint(u.x), __float_as_uint(u.y), __float_as_uint(u.z), __float_as_uint(u.w)};
    swiglu_n(g, up);
    *reinterpret_cast<uint2*>(static_cast<T*>(p.C) + size_t(m) * p.ldc + n) =
        make_uint2(pack2<T>(__uint_as_float(g[0]), __uint_as_float(g[1])), pack2<T>(__uint_as_float(g[2]), __uint_as_float(g[3])));
  } else if constexpr (EPI == kEpiRopeKv) {
    const oob_rope_args_t& a = p.rope;
    if (n >= p.N) return;  // N is a multiple of 8
    float4 x = v;
    if (r.hh < a.H + a.KV)
      x = make_float4(v.x * r.cs.x - v.y * r.sn.x, v.x * r.sn.x + v.y * r.cs.x, v.z * r.cs.y - v.w * r.sn.y,
                      v.z * r.sn.y + v.w * r.cs.y);
    T* dst;
    if (r.hh < a.H) {
      dst = static_cast<T*>(a.q_out) + (static_cast<long long>(m) * a.H + r.hh) * a.hd + r.c;
    } else {
      const int kvh = r.hh < a.H + a.KV ? r.hh - a.H : r.hh - a.H - a.KV;
      T* cache = static_cast<T*>(r.hh < a.H + a.KV ? a.k_cache : a.v_cache);
      dst = cache + (a.batch0 + r.b) * a.cache_batch_stride + (static_cast<long long>(kvh) * a.max_len + r.pos) * a.hd + r.c;
    }
    *reinterpret_cast<uint2*>(dst) = make_uint2(pack2<T>(x.x, x.y), pack2<T>(x.z, x.w));
  } else {
    T* dst = static_cast<T*>(p.C) + size_t(m) * p.ldc + n;
    if (p.vec_ok && n + 4 <= p.N) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack2<T>(v.x, v.y), pack2<T>(v.z, v.w));
    } else {
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n + i < p.N) dst[i] = PackTraits<T>::from_float(f[i]);
    }
  }
}

// Sums the S partial copies of this CTA's share of a tile and writes them.  A unit is four output columns of a token; the
// units are dealt out over the CTAs of the cluster, then over the threads, and TB units x S copies of independent loads are
// in flight per thread.  `n_first`: first output column of the tile.
// All threads of the CTA call `read_done` together, once, when the last copies have been read (each turn waits for its loads).  Where one
// turn reads them all that is before the results are written: the cluster barrier behind it would otherwise wait for those stores
// (35 x 2304 x 1536 5.4 us, 5.8 behind them).  Not so where a plain or SwiGLU launch takes several turns: inside the loop it keeps a turn's
// loads from being issued among the stores of the turn before (250 x 8192 x 3584 20.7 us, 20.4 behind the loop; 128 x 3896 x 608 7.8 and 7.4).
template <typename T, int EPI, int S, bool PAIR, typename F>
__device__ __forceinline__ void reduce_tile(const ParamsC& p, uint32_t smem_base, int rank, int m_first, int n_first, int rows,
                                            long long pos_base, const float* scale, F read_done) {
  constexpr int kParts = EPI == kEpiSwiglu ? 2 : 1;  // gate and up columns
  constexpr int TB = S * kParts >= 8 ? 1 : (S * kParts >= 4 ? 2 : 4);
  uint32_t base[S];
#pragma unroll
  for (int r = 0; r < S; ++r) base[r] = S == 1 ? smem_base : map_to_cta(smem_base, PAIR ? r * 2 + (cluster_ctarank() & 1) : r);
  constexpr int upt = kRowsW / 4 / kParts;  // units of a token
  const int units = rows * upt;
  // The Add epilogue sums the squares of a token's columns in a warp: whole tokens for each CTA.
  const int u_first = EPI == kEpiAdd ? rows * rank / S * upt : units * rank / S;
  const int u1 = EPI == kEpiAdd ? rows * (rank + 1) / S * upt : units * (rank + 1) / S;
  const int turns = (u1 - u_first + kThreadsC * TB - 1) / (kThreadsC * TB);  // the same for all threads
  auto take = [&](int turn, auto last) {
    const int u0 = u_first + turn * kThreadsC * TB + int(threadIdx.x);
    float4 v[TB][kParts][S];
    RopeUnit rope[TB];
    uint2 res[TB], nw[TB];
    int m[TB], c[TB];
#pragma unroll
    for (int i = 0; i < TB; ++i) {
      const bool live = u0 + i * kThreadsC < u1;
      const int u = live ? u0 + i * kThreadsC : u_first;
      m[i] = u / upt;
      c[i] = (u - m[i] * upt) * 4;
      if constexpr (EPI == kEpiRopeKv) rope[i] = rope_unit(p, m_first + m[i], n_first + c[i], pos_base);
      if constexpr (EPI == kEpiAdd) {
        res[i] = nw[i] = make_uint2(0u, 0u);
        if (n_first + c[i] < p.N) {  // N is a multiple of 8
          res[i] = *reinterpret_cast<const uint2*>(static_cast<const T*>(p.add.residual) + size_t(m_first + m[i]) * p.add.ld_residual + n_first + c[i]);
          nw[i] = *reinterpret_cast<const uint2*>(static_cast<const T*>(p.add.norm_weight) + n_first + c[i]);
        }
      }
#pragma unroll
      for (int h = 0; h < kParts; ++h)
#pragma unroll
        for (int r = 0; r < S; ++r) {
          v[i][h][r] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (live) v[i][h][r] = ld_cluster_f4(base[r] + uint32_t(m[i] * kRowsW + h * (kRowsW / 2) + c[i]) * 4u);
        }
    }
    float4 s[TB][kParts];
#pragma unroll
    for (int i = 0; i < TB; ++i) {
#pragma unroll
      for (int h = 0; h < kParts; ++h) {
        s[i][h] = v[i][h][0];
#pragma unroll
        for (int r = 1; r < S; ++r) {
          s[i][h].x += v[i][h][r].x;
          s[i][h].y += v[i][h][r].y;
          s[i][h].z += v[i][h][r].z;
          s[i][h].w += v[i][h][r].w;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < TB; ++i)
#pragma unroll
      for (int h = 0; h < kParts; ++h) settle(s[i][h].x, p.nan, smem_base);
    if (last) read_done();
    if (p.row_ssq != nullptr) {
#pragma unroll
      for (int i = 0; i < TB; ++i) {
        const float f = scale[m[i]];
#pragma unroll
        for (int h = 0; h < kParts; ++h) s[i][h] = make_float4(s[i][h].x * f, s[i][h].y * f, s[i][h].z * f, s[i][h].w * f);
      }
    }
    if constexpr (EPI == kEpiAdd) {
#pragma unroll
      for (int i = 0; i < TB; ++i) {
        if (u0 + i * kThreadsC >= u1) continue;  // all lanes of a warp together
        const int row = m_first + m[i], n = n_first + c[i];
        float ss = 0.f;
        if (n < p.N) {
          // The product is rounded before the sum, as the norm kernel would read it.
          const float2 o0 = unpack2<T>(pack2<T>(s[i][0].x, s[i][0].y)), o1 = unpack2<T>(pack2<T>(s[i][0].z, s[i][0].w));
          const float2 r0 = unpack2<T>(res[i].x), r1 = unpack2<T>(res[i].y), w0 = unpack2<T>(nw[i].x), w1 = unpack2<T>(nw[i].y);
          const uint2 hw = make_uint2(pack2<T>(o0.x + r0.x, o0.y + r0.y), pack2<T>(o1.x + r1.x, o1.y + r1.y));
          const float2 h0 = unpack2<T>(hw.x), h1 = unpack2<T>(hw.y);
          *reinterpret_cast<uint2*>(static_cast<T*>(p.C) + size_t(row) * p.ldc + n) = hw;
          *reinterpret_cast<uint2*>(static_cast<T*>(p.add.scaled_out) + size_t(row) * p.N + n) =
              make_uint2(pack2<T>(h0.x * w0.x, h0.y * w0.y), pack2<T>(h1.x * w1.x, h1.y * w1.y));
          ss = h0.x * h0.x + h0.y * h0.y + h1.x * h1.x + h1.y * h1.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if ((threadIdx.x & 31) == 0) p.add.ssq[size_t(n_first / kRowsW) * p.M + row] = ss;
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < TB; ++i)
      if (u0 + i * kThreadsC < u1) emit<T, EPI>(p, m_first + m[i], n_first + c[i], s[i][0], s[i][kParts - 1], rope[i]);
  };
  if constexpr (EPI == kEpiRopeKv || EPI == kEpiAdd) {
    for (int turn = 0; turn < turns; ++turn) take(turn, turn + 1 == turns);
    if (turns == 0) read_done();
  } else if (turns == 1) {
    take(0, std::true_type{});
  } else {
    for (int turn = 0; turn < turns; ++turn) take(turn, std::false_type{});
    read_done();
  }
}

// SUB: 64-element boxes of K in a pipeline stage.  RES: CTAs of an SM that the registers leave room for, 0 = what the compiler makes of it.
// For a plain launch's sums that is so few registers (50) that the loads of a turn wait for each other; with three CTAs 80 - 96
// (256 x 3456 x 4544 18.8 us, 17.9), with four 70 - 80 (143 x 1024 x 7680 17.7 us, 16.4 with three), which only the plans take that
// place four on an SM (16 x 64000 x 512 14.4 us, 16.8 on three).
// ONCE: see kOnceBytes (a kernel of its own: the policy beside the loop costs small launches 1 - 5 %).
template <typename T, int EPI, bool PAIR, int SUB, int RES, bool ONCE>
__global__ void __launch_bounds__(kThreadsC, RES)
    gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                        const __grid_constant__ ParamsC p, DeviceStatus* status) {
  constexpr int FMT = PackTraits<T>::kDType == kBF16 ? 1 : 0;
  extern __shared__ uint8_t smem_raw[];
  // The same offset in every CTA of the cluster (same kernel, same dynamic shared memory base).
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  CtlC* ctl = reinterpret_cast<CtlC*>(smem + p.work_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int P = PAIR ? 2 : 1;
  const int S = p.S;
  const int cluster = blockIdx.x / (S * P), in_cluster = blockIdx.x - cluster * (S * P);
  const int rank = in_cluster / P;                    // share of the K range
  const int member = PAIR ? (in_cluster & 1) : 0;      // CTA of the pair: 0 = leader
  const int kb0 = static_cast<int>(static_cast<long long>(p.num_kb) * rank / S);
  const int kb1 = static_cast<int>(static_cast<long long>(p.num_kb) * (rank + 1) / S);

  if (threadIdx.x == 0) {
    ptx::prefetch_tmap(&tmap_w);
    ptx::prefetch_tmap(&tmap_x);
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(&ctl->full[s], 2);  // two producers
      ptx::mbar_init(&ctl->empty[s], 1);
    }
    ptx::mbar_init(&ctl->tmem_full, 1);
    ctl->abort = 0;
    ptx::mbar_fence_init();
  }
  if constexpr (PAIR) {
    __syncthreads();
    cluster_sync();  // both CTAs' barriers exist before anything can signal them
    if (warp == 1) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(&ctl->tmem_base)),
                   "r"(p.tmem_cols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
  } else if (warp == 1) {
    ptx::tmem_alloc(&ctl->tmem_base, p.tmem_cols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if constexpr (PAIR) cluster_sync();  // both CTAs hold their TMEM before the first MMA writes into it
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abort = &ctl->abort;
  // This CTA holds its TMEM: the next kernel may be set up beside it.  Everything below touches memory that earlier
  // kernels wrote or still read.
  ptx::griddep_launch_dependents();
  // Static weights are not behind that wait: their warp fills the ring at once, and waits when it has loaded its first tile.
  bool waited = !(p.w_static && warp == 0);
  uint64_t once_policy = 0;
  if constexpr (ONCE) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once_policy));
  // Other weights may still be written by the kernel before: they are fetched into L2, which keeps up with such a write, and no further.
  if constexpr (fetches(EPI, RES, ONCE)) {
    if (warp == 0 && p.fetch > 0 && ptx::elect_one()) {
      const int w_row = (cluster / p.m_blocks * P + member) * (EPI == kEpiSwiglu ? kRowsW / 2 : kRowsW);
      for (int kb = kb0; kb < min(kb1, kb0 + p.fetch); ++kb)
#pragma unroll
        for (int h = 0; h < SUB; ++h) {
          ptx::tma_prefetch_2d(&tmap_w, (kb * SUB + h) * kTileK, w_row);
          if constexpr (EPI == kEpiSwiglu) ptx::tma_prefetch_2d(&tmap_w, (kb * SUB + h) * kTileK, p.F + w_row);
        }
    }
  }
  __syncwarp();
  if (waited) ptx::griddep_wait();
  long long pos_base = 0;
  auto load_pos = [&]() { return p.rope.pos_dev != nullptr ? *p.rope.pos_dev : static_cast<long long>(p.rope.pos0); };
  if constexpr (EPI == kEpiRopeKv) {
    if (waited) pos_base = load_pos();
  }

  if (warp >= 3 && p.row_ssq != nullptr) {  // at most kMaxScaledRows rows: one token block
    for (int m = threadIdx.x - 96; m < p.M; m += 96) {
      float ss = 0.f;
#pragma unroll 8
      for (int i = 0; i < p.row_parts; ++i) ss += p.row_ssq[size_t(i) * p.M + m];
      ctl->scale[m] = rsqrtf(ss * p.inv_k + p.row_eps);
    }
  }

  int stage = 0;          // producer's / MMA issuer's position in the ring, carried from tile to tile
  uint32_t phase = 0;
  uint32_t tile_phase = 0;
  constexpr int w_bytes = kRowsW * kRowBytes;       // a stage holds SUB boxes of weights, then SUB of activations
  const int x_bytes = SUB * (p.Mp / P) * kRowBytes;
  for (int t = cluster; t < p.num_tiles; t += p.clusters, tile_phase ^= 1) {
    const int wide_tile = t / p.m_blocks, m_first = (t - wide_tile * p.m_blocks) * p.Mp;
    const int tile = wide_tile * P + member;  // this CTA's 128 weight rows
    const int w_row = EPI == kEpiSwiglu ? tile * (kRowsW / 2) : tile * kRowsW;
    const int rows = min(p.Mp, p.M - m_first);
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    // ------------------------- TMA producers: warp 0 the weights, warp 2 the activations -------------------------
    // Straight-line copies of the loops here and below: where the compiler cannot see which tensor map a thread takes or how
    // many instructions it issues, 64 elements of K take a CTA 0.16 us (16 tokens) and 0.26 (128) instead of 0.107 and 0.142.
    auto produce = [&](auto weights, auto instructions) {
      constexpr bool W = decltype(weights)::value;
      constexpr int NM = decltype(instructions)::value;
      const uint32_t bytes = P * (W ? SUB * w_bytes : x_bytes);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!ptx::mbar_wait(&ctl->empty[stage], phase ^ 1, abort)) break;
        uint8_t* sw = smem + stage * p.stage_bytes;
        // The bytes of both CTAs of a pair are counted on the leader's barrier.
        if (!PAIR || member == 0) ptx::mbar_arrive_expect_tx(&ctl->full[stage], bytes);
        uint32_t full = ptx::smem_u32(&ctl->full[stage]);
        if constexpr (PAIR) full = map_to_cta(full, in_cluster & ~1);
#pragma unroll
        for (int h = 0; h < SUB; ++h) {
          const int k = (kb * SUB + h) * kTileK;  // past K: the box is filled with zeros
          if constexpr (W) {
            load_box<PAIR, ONCE>(sw + h * w_bytes, &tmap_w, full, k, w_row, once_policy);
            if constexpr (EPI == kEpiSwiglu) load_box<PAIR, ONCE>(sw + h * w_bytes + w_bytes / 2, &tmap_w, full, k, p.F + w_row, once_policy);
          } else {
            uint8_t* sx = sw + SUB * w_bytes + h * (x_bytes / SUB);
#pragma unroll
            for (int j = 0; j < NM; ++j)
              load_box<PAIR>(sx + j * (p.nj / P) * kRowBytes, &tmap_x, full, k, m_first + j * p.nj + member * (p.nj / P));
          }
        }
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    };
    if (warp == 0) {
      if (ptx::elect_one()) produce(std::true_type{}, One{});
    } else if (warp == 2) {
      if (ptx::elect_one()) {
        if (SUB == 1 && p.n_mma == 2) {  // a wide stage holds one instruction's tokens
          produce(std::false_type{}, Two{});
        } else {
          produce(std::false_type{}, One{});
        }
      }
    }
    if (warp == 0 || warp == 2) {
      __syncwarp();
      if (!waited) {  // the results below go where earlier kernels may still read
        ptx::griddep_wait();
        waited = true;
        if constexpr (EPI == kEpiRopeKv) pos_base = load_pos();
      }
    }
    if (warp == 1) {
      if (member == 0 && ptx::elect_one()) {
        // ------------------------- MMA issuer (of the pair: the leader's) ---------------------------
        const uint32_t idesc = ptx::umma_idesc_f16(FMT, P * kRowsW, p.nj);
        [[maybe_unused]] const uint16_t mask = static_cast<uint16_t>(3u << in_cluster);  // both CTAs of the pair
        bool ok = true;
        auto multiply = [&](auto instructions) {
          constexpr int NM = decltype(instructions)::value;
          bool ready = false;  // seen while the stage before was worked on
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!ready && !ptx::mbar_wait(&ctl->full[stage], phase, abort)) {
              ok = false;
              break;
            }
            ptx::tc_fence_after_sync();
            const uint32_t sw = ptx::smem_u32(smem + stage * p.stage_bytes);
            uint64_t* empty = &ctl->empty[stage];
            if (++stage == p.stages) {
              stage = 0;
              phase ^= 1;
            }
            ready = kb + 1 < kb1 && ptx::mbar_test_wait(&ctl->full[stage], phase);
#pragma unroll
            for (int h = 0; h < SUB; ++h) {
              const uint64_t da = ptx::umma_desc_kmajor_sw128(sw + h * w_bytes);
#pragma unroll
              for (int j = 0; j < NM; ++j) {
                const uint64_t db = ptx::umma_desc_kmajor_sw128(sw + SUB * w_bytes + h * (x_bytes / SUB) + j * (p.nj / P) * kRowBytes);
                const uint32_t d_tmem = tmem_base + j * p.nj;
#pragma unroll
                for (int k = 0; k < kTileK / 16; ++k) {
                  const uint32_t add = (kb > kb0 || h > 0 || k > 0) ? 1u : 0u;
                  if constexpr (PAIR) {
                    umma_f16_pair(d_tmem, da + uint64_t(k * 2), db + uint64_t(k * 2), idesc, add);
                  } else {
                    ptx::umma_f16(d_tmem, da + uint64_t(k * 2), db + uint64_t(k * 2), idesc, add);
                  }
                }
              }
            }
            if constexpr (PAIR) {
              umma_commit_pair(empty, mask);
            } else {
              ptx::umma_commit(empty);
            }
          }
        };
        if (SUB == 1 && p.n_mma == 2) {
          multiply(Two{});
        } else {
          multiply(One{});
        }
        if (ok) {
          if constexpr (PAIR) {
            umma_commit_pair(&ctl->tmem_full, mask);
          } else {
            ptx::umma_commit(&ctl->tmem_full);
          }
        }
      }
    } else if (warp >= 2) {
      // ------------------- TMEM -> own shared memory, [token][128] fp32 -------------------
      const int q = warp & 3;  // TMEM lane quadrant this warp may read: weight rows q * 32 ..
      if (ptx::mbar_wait(&ctl->tmem_full, tile_phase, abort)) {
        ptx::tc_fence_after_sync();
        const uint32_t t_addr = tmem_base + (uint32_t(q * 32) << 16);
        float* dst = reinterpret_cast<float*>(smem) + q * 32 + lane;
        for (int c = 0; c * 16 < rows; ++c) {
          uint32_t r[16];
          ptx::tmem_ld_32x32b_x16(t_addr + c * 16, r);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[(c * 16 + j) * kRowsW] = __uint_as_float(r[j]);
        }
      }
    }
    __syncwarp();
    ptx::tc_fence_before_sync();
    if (S * P > 1) {
      cluster_sync();
    } else {
      __syncthreads();
    }
    const uint32_t own = ptx::smem_u32(smem);
    // Nobody reads this CTA's copy any more: the buffers belong to the pipeline again (or to the next kernel).
    const bool last_tile = t + p.clusters >= p.num_tiles;
    auto read_done = [&]() {
      if (!last_tile) ptx::fence_proxy_async_all();
      __syncwarp();
      if (S * P > 1) cluster_arrive();
    };
#define OOB_REDUCE(SS) \
  case SS: reduce_tile<T, EPI, SS, PAIR>(p, own, rank, m_first, w_row, rows, pos_base, ctl->scale, read_done); break;
    switch (S) {
      OOB_REDUCE(1) OOB_REDUCE(2) OOB_REDUCE(3) OOB_REDUCE(4)
      default:
        if constexpr (!PAIR) {
          switch (S) { OOB_REDUCE(5) OOB_REDUCE(6) OOB_REDUCE(7) OOB_REDUCE(8) }
        }
    }
#undef OOB_REDUCE
    __syncwarp();
    if (S * P > 1) {
      cluster_wait();
    } else {
      __syncthreads();
    }
    ptx::tc_fence_after_sync();
  }

  // ---- teardown -----------------------------------------------------------
  if (*abort != 0) {
    if (threadIdx.x == 0) {
      gemm_report(status, 0, kDevTimeoutMbarrier, 95);
      const uint64_t t0 = ptx::globaltimer_ns();
      while (ptx::globaltimer_ns() - t0 < 200000) __nanosleep(1000);  // copies in flight land before smem is released
    }
  }
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    if constexpr (PAIR) {
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
    } else {
      ptx::tmem_dealloc(tmem_base, p.tmem_cols);
    }
  }
}

template <typename T, int EPI, bool PAIR, int SUB, int RES, bool ONCE = false>
cudaError_t launch_pair(const GemmArgs& a, ParamsC& p, DeviceStatus* status, cudaStream_t stream, TmapFn make_tmap) {
  auto kernel = gemm_cluster_kernel<T, EPI, PAIR, SUB, RES, ONCE>;
  const int size = PAIR ? 2 * p.S : p.S;  // CTAs of a cluster
  static std::atomic<uint64_t> attr_set_mask{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_set_mask.load(std::memory_order_relaxed) >> (dev & 63) & 1)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return e;
    attr_set_mask.fetch_or(uint64_t(1) << (dev & 63), std::memory_order_relaxed);
  }
  p.clusters = p.num_tiles;
  if (a.max_ctas > 0 && p.clusters > a.max_ctas / size) p.clusters = a.max_ctas / size;
  if (p.clusters < 1) p.clusters = 1;
  CUtensorMap tw, tx;
  if (!make_tmap(&tw, a.B, a.N, a.K, a.ldb, EPI == kEpiSwiglu ? kRowsW / 2 : kRowsW)) return cudaErrorInvalidValue;
  if (!make_tmap(&tx, a.A, a.M, a.K, a.lda, PAIR ? p.nj / 2 : p.nj)) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(p.clusters * size);
  cfg.blockDim = dim3(kThreadsC);
  cfg.dynamicSmemBytes = p.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = size;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = size > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, tw, tx, p, status);
}

// RES of the kernels that are not asked for four CTAs an SM.  The Add epilogue holds a turn's loads in 132 - 141 registers; with three CTAs it spills 250 - 350
// bytes and takes 1.066 times as long, 72 shapes of 1 - 128 rows.
constexpr int residents(int epi) { return epi == kEpiPlain || epi == kEpiSwiglu ? 3 : epi == kEpiAdd ? 2 : 0; }

template <typename T, int EPI>
cudaError_t launch_epi(const GemmArgs& a, ParamsC& p, bool pair, DeviceStatus* status, cudaStream_t stream, TmapFn make_tmap) {
  constexpr bool kBound = EPI == kEpiPlain || EPI == kEpiSwiglu;  // the others read more, of weights with at most two tiles for every SM
  constexpr int kRes = residents(EPI);
  if constexpr (EPI == kEpiAdd) {  // at most 128 rows, which no pair takes; a pair's second tile may lie past N, and has no sums to write
    if (pair) return cudaErrorInvalidValue;
  } else {
    if (pair) return launch_pair<T, EPI, true, 1, kRes>(a, p, status, stream, make_tmap);
  }
  auto launch = [&](auto once) {
    constexpr bool O = decltype(once)::value;
    if constexpr (kBound) {
      if (p.per_sm > kRes)
        return p.sub == 2 ? launch_pair<T, EPI, false, 2, 4, O>(a, p, status, stream, make_tmap)
                          : launch_pair<T, EPI, false, 1, 4, O>(a, p, status, stream, make_tmap);
    }
    return p.sub == 2 ? launch_pair<T, EPI, false, 2, kRes, O>(a, p, status, stream, make_tmap)
                      : launch_pair<T, EPI, false, 1, kRes, O>(a, p, status, stream, make_tmap);
  };
  return p.once ? launch(std::true_type{}) : launch(std::false_type{});
}

template <typename T>
cudaError_t launch_fmt(const GemmArgs& a, ParamsC& p, bool pair, DeviceStatus* status, cudaStream_t stream, TmapFn make_tmap) {
  switch (a.epilogue) {
    case kEpiSwiglu:
    case kGemmEpilogueSwigluTile: return launch_epi<T, kEpiSwiglu>(a, p, pair, status, stream, make_tmap);
    case kEpiRopeKv: return launch_epi<T, kEpiRopeKv>(a, p, pair, status, stream, make_tmap);
    case kGemmEpilogueAdd: return launch_epi<T, kEpiAdd>(a, p, pair, status, stream, make_tmap);
    default: return launch_epi<T, kEpiPlain>(a, p, pair, status, stream, make_tmap);
  }
}

// The most bytes of local memory (spilled registers) that a thread of any of the kernels has on the current device, -1 on an error.
template <typename T, int EPI>
int local_bytes() {
  int most = 0;
  auto look = [&](auto kernel) {
    cudaFuncAttributes attr{};
    if (most < 0 || cudaFuncGetAttributes(&attr, kernel) != cudaSuccess) {
      (void)cudaGetLastError();
      most = -1;
    } else {
      most = std::max(most, static_cast<int>(attr.localSizeBytes));
    }
  };
  constexpr int R = residents(EPI);
  look(gemm_cluster_kernel<T, EPI, false, 1, R, false>);
  look(gemm_cluster_kernel<T, EPI, false, 2, R, false>);
  look(gemm_cluster_kernel<T, EPI, false, 1, R, true>);
  look(gemm_cluster_kernel<T, EPI, false, 2, R, true>);
  if constexpr (EPI != kEpiAdd) look(gemm_cluster_kernel<T, EPI, true, 1, R, false>);
  if constexpr (EPI == kEpiPlain || EPI == kEpiSwiglu) {
    look(gemm_cluster_kernel<T, EPI, false, 1, 4, false>);
    look(gemm_cluster_kernel<T, EPI, false, 2, 4, false>);
    look(gemm_cluster_kernel<T, EPI, false, 1, 4, true>);
    look(gemm_cluster_kernel<T, EPI, false, 2, 4, true>);
  }
  return most;
}

}  // namespace gemm_cluster

namespace gemm_cluster {

// How a problem is cut: token blocks, pairs, K splits.
struct PlanC {
  int m_blocks, n_mma, nj;
  int sub;  // 64-element boxes of K in a stage
  bool pair;
  int S;
  int stages, smem, per_sm;  // pipeline stages, shared memory of a CTA, CTAs that share an SM
};

// Tokens of a tile when M rows are cut into `blocks`: n_mma instructions of nj.
void token_tile(int M, int blocks, PlanC* pl) {
  const int rows = (M + blocks - 1) / blocks;
  pl->n_mma = (rows + kMaxTokens - 1) / kMaxTokens;
  pl->nj = ((rows + pl->n_mma - 1) / pl->n_mma + 15) / 16 * 16;
  pl->m_blocks = (M + pl->n_mma * pl->nj - 1) / (pl->n_mma * pl->nj);
}

int tile_count(int N, const PlanC& pl) {
  const int wtiles = (N + kRowsW - 1) / kRowsW;  // SwiGLU too: N / 2 columns in steps of 64
  return (pl.pair ? (wtiles + 1) / 2 : wtiles) * pl.m_blocks;
}

uint32_t tmem_columns(int Mp) {
  uint32_t cols = 32;
  while (cols < uint32_t(Mp)) cols <<= 1;
  return cols;
}

// Shared memory: as many stages as fit when the CTAs of the launch are spread over the SMs; fails when the work of one CTA
// alone does not fit.
bool size_cta(int N, int num_kb, int sms, PlanC* pl) {
  const int P = pl->pair ? 2 : 1, Mp = pl->n_mma * pl->nj;
  const int stage_bytes = pl->sub * (kRowsW + Mp / P) * kRowBytes;
  const int fixed = 1024 + kCtlBytes;
  const int partial = Mp * kRowsW * 4 + fixed;
  const int steps = (num_kb + pl->sub - 1) / pl->sub;
  if (steps < pl->S) return false;
  const int kb_per = (steps + pl->S - 1) / pl->S;
  const int tmem = int(tmem_columns(Mp));
  // A CTA takes at least the share of an SM's shared memory that its TMEM columns are of the 512 (456 bytes a column; the
  // other TMEM kernels of this library take all of both).  CTAs that fit an SM then always find their columns free:
  // were one to wait for columns while its cluster waits for it, two clusters could wait for each other.
  const int least = tmem * 456 < kSmemLimit ? tmem * 456 : kSmemLimit;
  const int ctas = tile_count(N, *pl) * P * pl->S;
  int k = (ctas + sms - 1) / sms;
  const int most = 512 / tmem < 4 ? 512 / tmem : 4;
  if (k > most) k = most;
  for (; k >= 1; --k) {
    const int share = 228 * 1024 / k - 1024;
    const int budget = share < kSmemLimit ? share : kSmemLimit;
    int stages = (budget - fixed) / stage_bytes;
    if (stages > kMaxStagesC) stages = kMaxStagesC;
    if (stages > kb_per) stages = kb_per;
    if (stages < 2 && stages < kb_per && k > 1) continue;
    if (stages < 1) stages = 1;
    int smem = stages * stage_bytes + fixed;
    if (smem < partial) smem = partial;
    if (smem < least) smem = least;
    if (smem > kSmemLimit || k * (smem + 1024) > 228 * 1024) continue;
    pl->stages = stages;
    pl->smem = smem;
    pl->per_sm = k;
    return true;
  }
  return false;
}

// Clusters of `size` CTAs that run at once with `per_sm` CTAs on an SM, as a B200 answers (cudaOccupancyMaxActiveClusters).  A cluster lives
// in one GPC, about 18 SMs on this part, some have fewer, and not the same on every GPU.  One cluster too many is a second round of them
// (SwiGLU 116 x 1024 x 5624 on 16 clusters of seven, of which 15 run at once: 17.9 us, 11.0).  A table all the same, and not a question to the
// device: a plan has the K split in it, and with that the order of the sums, so that a call has the same bits on every GPU of a group, and
// plans can be kept by sizes alone.
int cluster_slots(int size, int per_sm) {
  static const int b200[4][kMaxCluster + 1] = {{0, 148, 74, 45, 33, 26, 22, 15, 15}, {0, 296, 148, 93, 71, 56, 45, 37, 33},
                                               {0, 444, 222, 142, 104, 82, 71, 56, 48}, {0, 592, 296, 187, 142, 112, 93, 78, 71}};
  return b200[per_sm - 1][size];
}
// What the plans of few rows were fitted with.
int rough_slots(int sms, int size, int per_sm) {
  if (size <= 2) return sms * per_sm / size;
  if (size > 4 && per_sm == 1) return size == 8 ? 12 : 16;
  return 8 * (18 * per_sm / size);
}

// Microseconds a plan takes: rounds of clusters, each as long as its K blocks at the pace of one CTA or of the tensor cores of an
// SM (cycles a block grow with the tokens), at the memory's rate for the weights or at L2's for all operands, whichever is
// slowest; then draining the sums, reading the other CTAs' sums, writing a CTA's share of C, and the fixed cost of a launch.  A
// row of a box that starts off a 128-byte line touches two (`line`), one that starts off a 32-byte sector one more of these
// (`sector`); the pace of one CTA with stages of many tokens suffers most (`pace_sector`: 103 x 5504 x 6728 split two ways 28.2 us,
// three ways 21.1, which were taken for the slower).
// The constants are fitted to timings for the choice they make, so that one need not be the rate that it stands for; kNone takes a limit
// out.  kFewRows (up to 128 rows): 16000 timings of every K split (1930 shapes of 3 - 128 rows, N and K of 512 - 8192), 3.3 % off the best plan on
// average; `write`, `alone`, the paces and `pace_sector` once more to 461 shapes.  kMoreRows: the set against which the two-SM kernel is weighed.
// Both were fitted to blocks of 128 tokens and more.
// kSpreadSome (33 - 128 rows) and kSpreadMore (129 - 1500) tell where blocks of 32 tokens and more beat these, see planned: only the quotient of two
// estimates of one set is used, and its constants are no rates.  Fitted to 1223 and 867 timed shapes, every split of up to ten blocks.
struct CostC {
  double wide, wide_tokens, pace, pace_tokens, mma, l2, hbm, drain, write, reduce, round, alone, cluster, eight, split, five, line, sector,
      pace_sector;
};
constexpr double kNone = 1e30;
constexpr CostC kFewRows = {0.153, 0.00061, 0.18, 0.0004, 1140.0, 11.8e6, 6.4e6, 0.0117, 0.01, 2.84e6, 1.85, 3.1, 3.06, 2.6, 0.105, 0.0, 1.29, 1.29, 1.6};
constexpr CostC kMoreRows = {0.165, 0.0005, 0.235, 0.0002, 1850.0, 11.5e6, 6.4e6, 0.015, 0.0, 3.0e6, 2.0, 3.4, 3.8, 2.0, 0.08, 0.0, 1.16, 1.45, 1.45};
constexpr CostC kSpreadSome = {0.185, 0.00294, 0.0018, 0.0038, kNone, 7.92e6, 6.69e6, 0.0, 0.066, 0.381e6, 2.95, 0.27, 0.054, 0.0, 0.188, 0.036, 2.21, 2.70, 2.52};
constexpr CostC kSpreadMore = {0.0036, 0.0026, 0.082, 0.000745, 2080.0, 17.8e6, kNone, 0.0, 0.0303, 1.415e6, 22.6, 0.574, 0.715, 0.095, 0.0, 0.01, 2.04, 2.81, 2.79};

// Blocks of fewer tokens than 128 are weighed in the range that they were timed in (150 shapes of 1501 - 4096 rows: 0.995 of the time with them, as many
// faster as slower), where the rows may be cut: row sums and the Add epilogue need one block, and static weights of few rows are
// planned for what their rings hold.
bool spread_rows(int M, bool ahead, bool one_block) { return M > kSpreadRows && M <= kSpreadMost && !one_block && (M > kTileM || !ahead); }

double plan_cost(const CostC& c, int N, int num_kb, RowStart start, const PlanC& pl, int slots, int sms) {
  const int P = pl.pair ? 2 : 1, Mp = pl.n_mma * pl.nj, size = P * pl.S;
  const int clusters = tile_count(N, pl);
  const int rounds = (clusters + slots - 1) / slots;
  const double live = double(clusters < slots ? clusters : slots) * size;  // CTAs at once
  const double share = live > sms ? live / sms : 1.0;
  const double kb = double((num_kb + pl.S - 1) / pl.S);
  const double w = kRowsW * kRowBytes, x = double(Mp) / P * kRowBytes;
  const double lines = start == kOnLine ? 1.0 : start == kOnSector ? c.line : c.sector;
  double t = (start == kOffSector && Mp > kWideTokens ? c.pace_sector : lines) * kb * (pl.sub == 2 ? c.wide + c.wide_tokens * Mp : c.pace + c.pace_tokens * Mp);
  const double mma = share * kb * 2.0 * Mp / c.mma, l2 = lines * live * kb * (w + x) / c.l2, hbm = live * kb * w / pl.m_blocks / c.hbm;
  if (mma > t) t = mma;
  if (l2 > t) t = l2;
  if (hbm > t) t = hbm;
  t += c.drain * Mp + c.write * Mp / pl.S + live * Mp * kRowsW * 4.0 * (pl.S - 1) / pl.S / c.reduce;
  return rounds * t + (rounds - 1) * c.round + (size > 1 ? c.cluster : c.alone) + (size == 8 && Mp > 128 ? c.eight : 0.0) +
         c.split * (pl.S - 1) + (pl.S >= 5 ? c.five : 0.0);
}
// With blocks of 128 tokens and more.
double whole_cost(int M, int N, int K, RowStart start, int sms, const PlanC& pl) {
  const int num_kb = (K + kTileK - 1) / kTileK, size = (pl.pair ? 2 : 1) * pl.S;
  return plan_cost(M <= kTileM ? kFewRows : kMoreRows, N, num_kb, start, pl, rough_slots(sms, size, pl.per_sm), sms);
}
// With blocks of any size.
double spread_cost(int M, int N, int K, int sms, const PlanC& pl) {
  const int num_kb = (K + kTileK - 1) / kTileK, size = (pl.pair ? 2 : 1) * pl.S;
  return plan_cost(M <= kTileM ? kSpreadSome : kSpreadMore, N, num_kb, row_start(K), pl, cluster_slots(size, pl.per_sm), sms);
}

// What static weights save: the rings are filled while the kernel before ends.  Plans with more CTAs hold more (32 x 8192 x 3584 in a
// decode step 13.3 us on 128 CTAs, 14.3 on 64, which were taken for faster).
double ring_us(int N, int num_kb, int sms, const PlanC& pl) {
  const int clusters = tile_count(N, pl), size = (pl.pair ? 2 : 1) * pl.S, slots = rough_slots(sms, size, pl.per_sm);
  const double live = double(clusters < slots ? clusters : slots) * size;
  return live * pl.stages * pl.sub * kRowsW * kRowBytes / 6.05e6;
}

// The cheapest cut of a problem into blocks of 128 tokens and more, or of any size (`spread`).  `fix_s` > 0 fixes the K split, `pair` is as
// in GemmArgs; `ahead`: static weights.
bool plan(int M, int N, int K, int sms, int pair, int fix_s, bool ahead, bool spread, PlanC* out, double* cost) {
  const int num_kb = (K + kTileK - 1) / kTileK;
  if (N <= kRowsW) pair = -1;  // one weight tile is no pair
  bool found = false;
  int last = 0;
  int most_blocks = (M + 127) / 128;
  if (spread) most_blocks = std::max(most_blocks, std::min((M + kSpreadRows - 1) / kSpreadRows, kSpreadBlocks));
  for (int blocks = (M + kMaxTileTokens - 1) / kMaxTileTokens; blocks <= most_blocks; ++blocks) {
    PlanC pl{};
    token_tile(M, blocks, &pl);
    const int Mp = pl.n_mma * pl.nj;
    if (Mp == last) continue;
    last = Mp;
    for (int two = 0; two < 2; ++two) {
      pl.pair = two != 0;
      if (two ? pair < 0 || (pair == 0 && Mp <= 128) : pair > 0) continue;
      pl.sub = !two && Mp <= kWideTokens && num_kb >= 2 * kMaxCluster ? 2 : 1;
      for (pl.S = 1; pl.S <= kMaxCluster / (two ? 2 : 1); ++pl.S) {
        if (fix_s > 0 ? pl.S != fix_s : (num_kb < 4 * pl.S && pl.S > 1)) continue;
        if (!size_cta(N, num_kb, sms, &pl)) continue;
        // (with more rows the plans of whole blocks are compared as if rows started on a line: the set was fitted so)
        double c = spread ? spread_cost(M, N, K, sms, pl) : whole_cost(M, N, K, M <= kTileM ? row_start(K) : kOnLine, sms, pl);
        if (ahead) c -= ring_us(N, num_kb, sms, pl);
        if (!found || c < *cost) {
          found = true;
          *out = pl;
          *cost = c;
        }
      }
    }
  }
  return found;
}

// Whether the weights are loaded so that they leave L2 first.
bool read_once(int N, int K, const PlanC& pl, int b_static) {
  return pl.m_blocks == 1 && 2ll * N * K >= (b_static == 2 ? kOnceChainBytes : kOnceBytes);
}

// Plans depend on sizes alone; the last ones of a thread are kept (a model's layers repeat a handful of shapes).
struct Planned {
  int M, N, K, flags;
  bool ok, spread;  // spread: cut into blocks of any size
  PlanC pl;
  double whole_us, spread_us;  // estimates (without what static weights save): of the cut into whole blocks, of the spread one
};
// A spread cut is taken where its estimate is kSpreadGain of that of whole blocks, which the sets were fitted with: first of all to be no slower.
// Over the 2090 timed shapes 0.952 of the time of whole blocks, 15 more than 3 % slower (a fit to the smallest mean time, where the cheaper estimate is
// taken: 0.946, and 98 slower, 432 x 4048 x 4136 21.5 -> 24.6 us among them).
// 340 other shapes of 33 - 1500 rows, against the code with whole blocks alone: plain 0.955, SwiGLU 0.93, QKV with rotation and cache write 0.97 of
// the time, 16 more than 3 % slower (46 with the cheaper estimate).
const Planned& planned(int M, int N, int K, int pair, int fix_s, bool ahead, bool one_block) {
  static thread_local Planned cache[64];
  const int flags = 1 | (pair > 0 ? 2 : pair < 0 ? 1 : 0) << 1 | (ahead ? 1 : 0) << 3 | fix_s << 4 | (one_block ? 1 : 0) << 12;
  Planned& c = cache[(static_cast<unsigned>(M) * 2654435761u ^ static_cast<unsigned>(N) * 40503u ^ static_cast<unsigned>(K) * 97u ^
                      static_cast<unsigned>(flags) * 7u) >> 8 & 63u];
  if (c.M != M || c.N != N || c.K != K || c.flags != flags) {
    c.M = M;
    c.N = N;
    c.K = K;
    c.flags = flags;
    const int sms = sm_count();
    double us;
    c.spread = false;
    c.ok = plan(M, N, K, sms, pair, fix_s, ahead, false, &c.pl, &us);
    c.whole_us = c.ok ? whole_cost(M, N, K, row_start(K), sms, c.pl) : kNone;
    PlanC other;
    if (spread_rows(M, ahead, one_block) && plan(M, N, K, sms, pair, fix_s, ahead, true, &other, &us)) {
      c.spread_us = spread_cost(M, N, K, sms, other);
      if (!c.ok || c.spread_us < kSpreadGain[M > kTileM] * spread_cost(M, N, K, sms, c.pl)) {
        c.ok = c.spread = true;
        c.pl = other;
      }
    }
  }
  return c;
}

}  // namespace gemm_cluster

bool gemm_cluster_supported(const GemmArgs& a) {
  return a.mode == kGemmPlain && a.M >= 1 && a.M <= kGemmClusterMaxRows && a.epilogue <= kGemmEpilogueAdd &&
         ((a.row_ssq == nullptr && a.epilogue != kGemmEpilogueAdd) || a.M <= gemm_cluster::kMaxScaledRows);
}

// Whether this kernel is expected to be faster than the persistent two-SM kernel, which overlaps a tile's epilogue with the next
// tile and needs no sum of parts, but deals out 256-row tiles: with fewer than three rounds of those, what they leave
// idle or compute on padding is often more than this kernel's fixed cost.  The estimate of whole blocks is taken a tenth lower, which
// fits its present pace (over 467 shapes of more than 128 rows the choice is then 0.9 % slower than the best one on average), that of a spread
// cut times kSpreadTwoSm, as it was when its constants were fitted.
// Both sides measured, bf16 on B200: 512 x 1280 x 8192 17.5 here and 26.6 us there, 200 x 4096 x 4096 12.6 and 16.4, 512 x 2048 x 2048
// 9.4 and 10.3; 1037 x 4104 x 2056 24.3 and 22.2, 768 x 7168 x 8192 70.5 and 63.6, 512 x 8192 x 8192 61.9 and 50.9, 2048 x 2048 x 2048
// 25.6 and 16.8.
bool gemm_cluster_preferred(const GemmArgs& a) {
  using namespace gemm_cluster;
  // Up to 128 rows the alternative is the one-SM kernel, persistent from the first tile to the last, on 256 weight rows a tile.
  // It is the better one where there are more than two CTAs of 128 weight rows for every SM, from 49 rows on (128 x 57344 x 1024 27.9
  // and 37.4 here, 80 x 64000 x 2048 47.3 and 61.5, 128 x 128256 x 4096 183 and 214) and, where K is long, from nine (16 x 57344 x
  // 8192 155 and 172, 16 x 128256 x 4096 171 and 185; but 32 x 57344 x 1024 28.2 and 25.9, 16 x 64000 x 2048 62.6 and 58.9, 4 x 57344 x
  // 8192 193 and 164).  With fewer tiles it is the worse one or equal (128 x 32768 x 4096 50.4 and 50.7, 64 x 24000 x 4096 40.2 and
  // 38.4).  SwiGLU would need a kernel of its own behind it.
  if (a.M <= kTileM)
    return a.epilogue != 0 || a.M <= (a.K >= 4096 ? 8 : 48) || (a.N + kRowsW - 1) / kRowsW <= 2 * sm_count();
  const bool swiglu = a.epilogue == kEpiSwiglu || a.epilogue == kGemmEpilogueSwigluTile;
  const int pairs = sm_count() / 2;
  if (static_cast<long long>((a.M + 2 * kTileM - 1) / (2 * kTileM)) * ((a.N + kTileN - 1) / kTileN) > 3ll * pairs) return false;
  const double two_sm = pair_cut(kGemmPlain, a.M, a.N, a.K, pairs, a.stream_k, swiglu, false, false).us;
  const Planned& c = planned(a.M, a.N, a.K, a.pair, 0, false, false);
  return c.ok && (0.9 * c.whole_us < two_sm || (c.spread && kSpreadTwoSm * c.spread_us < two_sm));
}

int gemm_cluster_local_bytes(int epilogue, int fmt) {
  using namespace gemm_cluster;
  auto of = [&](auto t) {
    using T = decltype(t);
    switch (epilogue) {
      case kEpiPlain: return local_bytes<T, kEpiPlain>();
      case kEpiSwiglu: return local_bytes<T, kEpiSwiglu>();
      case kEpiRopeKv: return local_bytes<T, kEpiRopeKv>();
      default: return local_bytes<T, kEpiAdd>();
    }
  };
  return fmt == 1 ? of(__nv_bfloat16()) : of(__half());
}

bool gemm_cluster_plan(int M, int N, int K, int pair, int splits, int b_static, bool one_block, int out[6]) {
  const gemm_cluster::Planned& c = gemm_cluster::planned(M, N, K, pair, splits, b_static != 0, one_block);
  if (!c.ok) return false;
  out[0] = c.pl.m_blocks;
  out[1] = c.pl.n_mma * c.pl.nj;
  out[2] = c.pl.pair;
  out[3] = c.pl.S;
  out[4] = c.pl.per_sm;
  out[5] = gemm_cluster::read_once(N, K, c.pl, b_static);
  return true;
}

cudaError_t launch_gemm_cluster(const GemmArgs& a, DeviceStatus* status, cudaStream_t stream, gemm_detail::TmapFn make_tmap) {
  using namespace gemm_cluster;
  const bool swiglu = a.epilogue == kEpiSwiglu || a.epilogue == kGemmEpilogueSwigluTile;
  const int num_kb = (a.K + kTileK - 1) / kTileK;
  int fix_s = a.splits;
  const int most = a.pair > 0 ? kMaxCluster / 2 : kMaxCluster;
  if (fix_s > most) fix_s = most;
  if (fix_s > num_kb) fix_s = num_kb;
  if (a.max_ctas > 0) {  // a budget: K is split as far as asked for
    if (fix_s == 0) fix_s = 1;
    if (fix_s > a.max_ctas) fix_s = a.max_ctas;
  }
  const Planned& chosen = planned(a.M, a.N, a.K, a.max_ctas > 0 ? -1 : a.pair, fix_s, a.b_static != 0,
                                  a.row_ssq != nullptr || a.epilogue == kGemmEpilogueAdd);
  if (!chosen.ok) return cudaErrorInvalidValue;
  const PlanC pl = chosen.pl;
  const int P = pl.pair ? 2 : 1;
  ParamsC p{};
  p.M = a.M;
  p.N = a.N;
  p.C = a.C;
  p.ldc = a.ldc;
  p.w_static = a.b_static != 0;
  p.vec_ok = a.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(a.C) & 7) == 0;
  p.sub = pl.sub;
  p.num_kb = (num_kb + pl.sub - 1) / pl.sub;
  if (swiglu) p.F = static_cast<const oob_gemm_epilogue_swiglu_t*>(a.epilogue_args)->F;
  if (a.epilogue == kGemmEpilogueAdd) p.add = *static_cast<const oob_gemm_epilogue_add_t*>(a.epilogue_args);
  p.row_ssq = a.row_ssq;
  p.row_parts = a.row_parts;
  p.row_eps = a.row_eps;
  p.inv_k = 1.f / static_cast<float>(a.K);
  p.nan = std::numeric_limits<float>::quiet_NaN();
  if (a.epilogue == kEpiRopeKv) p.rope = *static_cast<const oob_rope_args_t*>(a.epilogue_args);
  p.once = read_once(a.N, a.K, pl, a.b_static);
  const long long weights = 2ll * a.N * a.K;
  const bool on_line = a.ldb % kTileK == 0 && (reinterpret_cast<uintptr_t>(a.B) & 127) == 0;
  p.fetch = a.b_static || weights < (on_line ? kFetchBytes : kOnceBytes) ? 0 : weights < kFetchTwoBytes ? 1 : 2;
  p.n_mma = pl.n_mma;
  p.nj = pl.nj;
  p.Mp = pl.n_mma * pl.nj;
  p.m_blocks = pl.m_blocks;
  p.S = pl.S;
  p.per_sm = pl.per_sm;
  p.num_tiles = tile_count(a.N, pl);
  p.stage_bytes = pl.sub * (kRowsW + p.Mp / P) * kRowBytes;
  p.stages = pl.stages;
  p.smem_bytes = pl.smem;
  p.work_bytes = pl.smem - 1024 - kCtlBytes;
  p.work_bytes -= p.work_bytes % 16;
  p.tmem_cols = tmem_columns(p.Mp);
  return a.fmt == 1 ? gemm_cluster::launch_fmt<__nv_bfloat16>(a, p, pl.pair, status, stream, make_tmap)
                    : gemm_cluster::launch_fmt<__half>(a, p, pl.pair, status, stream, make_tmap);
}

}  // namespace oob
