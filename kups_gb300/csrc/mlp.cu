// Tensor-core (tcgen05) GEMM and the learned insertion-proposal MLP.
//
// The learned proposal has no counterpart in the reference; it plugs into the
// ChangesFn log-ratio hook of the insertion move (src/kups/mcmc/moves.py:92-98,
// src/kups/core/propagator.py:330-334).
//
// GEMM: C[M, N] = act(alpha * A[M, K] . B[N, K]^T + bias[N]) with arbitrary
// element strides for A, B and C (so transposed operands need no copies);
// split-K (grid z) for products with a long K.
// One CTA computes a 128 x BN tile.  Bfloat16 operands with K contiguous are
// loaded by TMA (cp.async.bulk.tensor, 128-byte swizzle) into a ring of
// stages (gemm_tma_kernel); other layouts are staged by the threads with
// 16-byte copies or element-wise into the canonical no-swizzle K-major layout
// (8-row x 16-byte core matrices, gemm_tcgen05_kernel).  One thread issues
// tcgen05.mma.cta_group::1.kind::f16 (BF16 inputs, FP32 accumulation in
// tensor memory) and tcgen05.commit to an mbarrier, and the epilogue reads
// the accumulator back with tcgen05.ld.32x32b.  Every mbarrier wait is
// bounded; on time-out the kernel records KUPS_ERR_UNSUPPORTED, frees its
// tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "common.cuh"
#include "proposal.cuh"

namespace kups {
namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kGemmThreads = 256;  // 8 warps: warps w and w + 4 share TMEM lanes 32 (w % 4) ..
constexpr long long kWaitLimit = 1LL << 26;

__device__ inline uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor (no swizzle, K-major): start >> 4 in
// [0, 14), leading byte offset >> 4 in [16, 30) (next core matrix along K),
// stride byte offset >> 4 in [32, 46) (next 8-row group), descriptor version
// 1 in [46, 48), swizzle mode 0 in [61, 64).
__device__ inline uint64_t make_sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor, kind::f16: D = F32 (bits 4-5 = 1), A = B = BF16
// (bits 7-9 = 1, 10-12 = 1), both K-major, N >> 3 in [17, 23), M >> 4 in [24, 29).
__device__ inline uint32_t make_idesc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ inline void mbar_init(uint32_t addr, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr), "r"(count));
}

__device__ inline bool mbar_wait(uint32_t addr, uint32_t phase) {
  for (long long i = 0; i < kWaitLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(addr), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// 2^x and log2 x by one SFU instruction each, subnormal values flushed to zero.  PTX gives ex2.approx a
// relative error of 2^-22 and lg2.approx an absolute one of 2^-22 between 1/2 and 2.
__device__ inline float exp2_sfu(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ inline float log2_sfu(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// softplus(x) = ln(1 + e^x) in base 2, max(x, 0) + ln 2 log2(1 + 2^(-|x| log2 e)): no overflow, t =
// 2^(-|x| log2 e) in [0, 1] (a t below 2^-126 is nothing beside the 1), the logarithm's argument in [1, 2].
// Its error is below 4e-7 + 2^-24 |x|: 1.7e-7 of the logarithm, 1.2e-7 of t, 4.4e-8 of the exponent's
// rounding and 6e-8 of 1 + t's, and the rounding of the result.
constexpr float kLog2E = 1.44269504088896341f, kLn2 = 0.69314718055994531f;
__device__ inline float softplus_fast(float x) {
  const float t = exp2_sfu(__fmul_rn(-kLog2E, fabsf(x)));
  return fmaf(log2_sfu(1.0f + t), kLn2, fmaxf(x, 0.f));
}

// One 32-byte store (a whole L2 sector) of eight 32-bit values.
__device__ inline void st_v8(void *p, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

__device__ inline void red_add_v4(float *p, float a, float b, float c, float d) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

__device__ inline float act_fn(float x, int act) {
  if (act == 1) return fmaxf(x, 0.f);                      // ReLU
  if (act == 2) return x > 20.f ? x : log1pf(__expf(x));  // softplus (SFU exp)
  return x;
}

// Strided element access: element (r, c) of a matrix at p + r * sr + c * sc.
template <typename T>
__device__ inline float ld_el(const T *p, int64_t r, int64_t c, int64_t sr, int64_t sc) {
  return (float)p[r * sr + c * sc];
}
template <>
__device__ inline float ld_el<__nv_bfloat16>(const __nv_bfloat16 *p, int64_t r, int64_t c, int64_t sr, int64_t sc) {
  return __bfloat162float(p[r * sr + c * sc]);
}

struct GemmArgs {
  const void *a;
  const void *b;
  void *c;
  void *c2;           // optional second output (same tile, its own strides)
  const float *bias;  // [N] or null
  const float *gate;  // optional: C *= act'(pre) mask source (same layout as c, fp32) or null
  int64_t sar, sac, sbr, sbc, scr, scc, sc2r, sc2c, sgr, sgc;
  int m, n, k;
  float alpha, beta;  // C = alpha * AB^T (+ beta * C)
  int act;            // 0 none, 1 relu, 2 softplus
  int a_bf16, b_bf16, c_bf16, c2_bf16;
  int gate_kind;      // 0 none, 1: multiply by relu'(gate) (gate > 0), 2: by softplus'(gate) = sigmoid,
                      // 3: by softplus' expressed through its output h = softplus(z): 1 - exp(-h)
  int split_k;        // > 1: blockIdx.z takes a slice of K and atomically adds alpha * partial to C
  int row_epi;        // set by dispatch_gemm: the register (lane = row) epilogue applies
  int row_v8;         // ... and C (and c2) rows are 32-byte aligned: whole-sector 32-byte stores
};

__device__ inline void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ inline void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Stages rows [r0, r0 + ROWS) x columns [k0, k0 + 64) of an operand into the
// no-swizzle K-major core-matrix layout: element (r, kk) at
//   ((r / 8) * 8 + kk / 8) * 64 + (r % 8) * 8 + kk % 8.
// Fast path (bfloat16, unit K stride, 16-byte rows): one 16-byte cp.async per
// core-matrix row; thread e copies row (e / 64) * 8 + e % 8, K group (e / 8) % 8,
// whose shared-memory destination is element 8 e (a warp fills 512 contiguous
// bytes and reads 64 contiguous bytes of each of 8 rows).  Rows past the end
// are zero-filled (source size 0).  Otherwise every element is loaded,
// converted and stored.
template <int ROWS>
__device__ inline void stage_operand(__nv_bfloat16 *s, const void *p, int is_bf16, int64_t sr, int64_t sc, bool fast,
                                     int r0, int nrows, int k0, int k, int tid) {
  if (fast) {
    const __nv_bfloat16 *base = (const __nv_bfloat16 *)p;
    const uint32_t s0 = smem_u32(s);
    for (int e = tid; e < ROWS * (kBK / 8); e += kGemmThreads) {
      const int r = (e >> 6) * 8 + (e & 7), kg = (e >> 3) & 7;
      const int gr = r0 + r, gk = k0 + kg * 8;
      const bool in = gr < nrows && gk < k;
      const __nv_bfloat16 *src = in ? base + (int64_t)gr * sr + gk : base;
      cp_async16(s0 + (uint32_t)e * 16u, src, in ? 16u : 0u);
    }
  } else {
    const bool rows_fast = sr == 1 && sc != 1;  // walk along the unit-stride index
    for (int e = tid; e < ROWS * kBK; e += kGemmThreads) {
      const int r = rows_fast ? e % ROWS : e / kBK, kk = rows_fast ? e / ROWS : e % kBK;
      const int gr = r0 + r, gk = k0 + kk;
      float v = 0.f;
      if (gr < nrows && gk < k)
        v = is_bf16 ? ld_el((const __nv_bfloat16 *)p, gr, gk, sr, sc) : ld_el((const float *)p, gr, gk, sr, sc);
      s[((r >> 3) * (kBK / 8) + (kk >> 3)) * 64 + (r & 7) * 8 + (kk & 7)] = __float2bfloat16(v);
    }
  }
}

__device__ inline bool fast_operand(const void *p, int is_bf16, int64_t sr, int64_t sc, int k) {
  return is_bf16 && sc == 1 && (sr % 8) == 0 && (k % 8) == 0 && (((uintptr_t)p) & 15) == 0;
}

// Register epilogue of a 128 x BN accumulator tile in tensor memory (row-major float32 C with
// 16-byte aligned rows, N a multiple of 32, beta = 0 or split K): warp w reads TMEM lanes
// 32 (w % 4) .. + 31, so lane l holds row m0 + 32 (w % 4) + l, 32 columns at a time of the
// column half w / 4, and applies every term in registers: 16-byte loads of bias and gate,
// 16-byte stores of C and of the bfloat16 copy (c2), vector reductions for split K.
template <int BN>
__device__ inline void register_epilogue(const GemmArgs &g, uint32_t tmem, int m0, int n0, int warp, int lane) {
  const int quarter = warp & 3, half = warp >> 2;
  const int row = m0 + quarter * 32 + lane;
  const bool rin = row < g.m;
  for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
    uint32_t r[32];
    const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    const int col0 = n0 + c0;
    if (col0 >= g.n) continue;  // N is a multiple of 32: the chunk is wholly in or out
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = g.alpha * __uint_as_float(r[i]);
    if (g.split_k > 1) {
      if (rin) {
        float *dst = (float *)g.c + (int64_t)row * g.scr + col0;
#pragma unroll
        for (int q = 0; q < 8; ++q) red_add_v4(dst + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
      continue;
    }
    if (g.bias != nullptr) {
      const float4 *b4 = reinterpret_cast<const float4 *>(g.bias + col0);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 b = __ldg(b4 + q);
        v[4 * q] += b.x;
        v[4 * q + 1] += b.y;
        v[4 * q + 2] += b.z;
        v[4 * q + 3] += b.w;
      }
    }
    if (g.gate_kind != 0 && rin) {
      const float4 *g4 = reinterpret_cast<const float4 *>(g.gate + (int64_t)row * g.sgr + col0);
      const int kind = g.gate_kind;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 t = g4[q];
        const float pre[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = pre[e];
          float f;
          if (kind == 1) f = x > 0.f ? 1.f : 0.f;
          else if (kind == 2) f = 1.f / (1.f + expf(-x));
          else f = -expm1f(-x);
          v[4 * q + e] *= f;
        }
      }
    }
    if (g.act == 1) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.f);
    } else if (g.act == 2) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = act_fn(v[i], 2);
    }
    if (rin) {
      float *cr = (float *)g.c + (int64_t)row * g.scr + col0;
      if (g.row_v8) {  // each lane writes whole 32-byte sectors of its row
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(v[8 * q + e]);
          st_v8(cr + 8 * q, w);
        }
      } else {
        float4 *cp = reinterpret_cast<float4 *>(cr);
#pragma unroll
        for (int q = 0; q < 8; ++q) cp[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
      if (g.c2 != nullptr) {
        __nv_bfloat16 *c2r = (__nv_bfloat16 *)g.c2 + (int64_t)row * g.sc2r + col0;
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
          w[e] = *reinterpret_cast<const uint32_t *>(&h);
        }
        if (g.row_v8) {
          st_v8(c2r, *reinterpret_cast<const uint32_t(*)[8]>(&w[0]));
          st_v8(c2r + 16, *reinterpret_cast<const uint32_t(*)[8]>(&w[8]));
        } else {
          uint4 *c2p = reinterpret_cast<uint4 *>(c2r);
#pragma unroll
          for (int q = 0; q < 4; ++q) c2p[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        }
      }
    }
  }
}

// Two-stage pipeline: the 16-byte copies of K chunk c + 1 are in flight while
// the tensor cores work on chunk c; a stage is refilled only after the
// mbarrier of the MMAs that read it has completed.
template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 4) gemm_tcgen05_kernel(GemmArgs g, kups_status *status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int kStageBytes = (kBM + BN) * kBK * 2;
  uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + 2 * kStageBytes);  // [2]
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbar + 2);
  auto sa = [&](int st) { return reinterpret_cast<__nv_bfloat16 *>(smem + st * kStageBytes); };
  auto sb = [&](int st) { return reinterpret_cast<__nv_bfloat16 *>(smem + st * kStageBytes + kBM * kBK * 2); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
  if (warp == 0) {
    const uint32_t cols = BN < 32 ? 32 : BN;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    mbar_init(smem_u32(&mbar[0]), 1);
    mbar_init(smem_u32(&mbar[1]), 1);
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t idesc = make_idesc(kBM, BN);
  const int nk_all = (g.k + kBK - 1) / kBK;
  const int per_split = (nk_all + g.split_k - 1) / g.split_k;
  const int kc_begin = blockIdx.z * per_split;
  const int kc_end = min(nk_all, kc_begin + per_split);
  const bool fa = fast_operand(g.a, g.a_bf16, g.sar, g.sac, g.k);
  const bool fb = fast_operand(g.b, g.b_bf16, g.sbr, g.sbc, g.k);
  // per stage (bit st): parity of the next completion to wait for, and whether MMAs reading it are
  // in flight (bit fields, not arrays: the stage index is dynamic)
  uint32_t phase = 0u, pending = 0u;
  bool ok = true;
  if (kc_begin < kc_end) {
    stage_operand<kBM>(sa(0), g.a, g.a_bf16, g.sar, g.sac, fa, m0, g.m, kc_begin * kBK, g.k, tid);
    stage_operand<BN>(sb(0), g.b, g.b_bf16, g.sbr, g.sbc, fb, n0, g.n, kc_begin * kBK, g.k, tid);
    cp_async_commit();
  }
  for (int kc = kc_begin; kc < kc_end; ++kc) {
    const int st = (kc - kc_begin) & 1, nx = st ^ 1;
    if (kc + 1 < kc_end) {
      if ((pending >> nx) & 1u) {  // the MMAs of chunk kc - 1 read stage nx
        ok = mbar_wait(smem_u32(&mbar[nx]), (phase >> nx) & 1u);
        if (ok) {  // after a time-out the clean-up below waits for these MMAs again
          phase ^= 1u << nx;
          pending &= ~(1u << nx);
        }
      }
      if (!__syncthreads_and(ok)) {
        ok = false;
        break;
      }
      stage_operand<kBM>(sa(nx), g.a, g.a_bf16, g.sar, g.sac, fa, m0, g.m, (kc + 1) * kBK, g.k, tid);
      stage_operand<BN>(sb(nx), g.b, g.b_bf16, g.sbr, g.sbc, fb, n0, g.n, (kc + 1) * kBK, g.k, tid);
      cp_async_commit();
      cp_async_wait<1>();  // chunk kc has landed (this thread's copies)
    } else {
      cp_async_wait<0>();
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int ks = 0; ks < kBK / 16; ++ks) {
        // K step of 16 = two core matrices along K = 256 bytes
        const uint64_t ad = make_sdesc(smem_u32(sa(st)) + ks * 256, 128, (kBK / 8) * 128);
        const uint64_t bd = make_sdesc(smem_u32(sb(st)) + ks * 256, 128, (kBK / 8) * 128);
        const uint32_t accumulate = (kc > kc_begin || ks > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&mbar[st]))
                   : "memory");
    }
    pending |= 1u << st;
  }
  cp_async_wait<0>();
  // every MMA in flight completes (bounded waits) before the accumulator is read or freed
  for (int st = 0; st < 2; ++st)
    if ((pending >> st) & 1u) ok = mbar_wait(smem_u32(&mbar[st]), (phase >> st) & 1u) && ok;
  ok = __syncthreads_and(ok);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok) {
    if (tid == 0) status_error(status, KUPS_ERR_UNSUPPORTED, blockIdx.x);
  } else if (kc_begin < kc_end && g.row_epi) {
    register_epilogue<BN>(g, tmem, m0, n0, warp, lane);
  } else if (kc_begin < kc_end) {  // an empty K slice holds no accumulator
    // epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (rows) and the column half
    // w / 4, 32 columns at a time, into a padded 32 x 33 shared-memory block.  The
    // elementwise terms run with lane = column (coalesced bias / gate / C loads and
    // row-major stores, 128 contiguous bytes of one row per instruction).
    const int quarter = warp & 3, half = warp >> 2;
    const int rbase = m0 + quarter * 32;
    float *blk = reinterpret_cast<float *>(smem) + warp * 32 * 33;  // pipeline stages are free now
    for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
      uint32_t r[32];
      const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
          "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
            "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
            "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
          : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int i = 0; i < 32; ++i) blk[lane * 33 + i] = __uint_as_float(r[i]);
      __syncwarp();
      const int col = n0 + c0 + lane;
      if (col < g.n) {
        const float bias = g.bias ? g.bias[col] : 0.f;
        // unrolled so that the gate loads of several rows are in flight together
#pragma unroll 8
        for (int rr = 0; rr < 32; ++rr) {
          const int row = rbase + rr;
          if (row >= g.m) continue;
          float v = g.alpha * blk[rr * 33 + lane];
          const int64_t o = (int64_t)row * g.scr + (int64_t)col * g.scc;
          if (g.split_k > 1) {
            atomicAdd((float *)g.c + o, v);
            continue;
          }
          if (g.beta != 0.f) v += g.beta * (g.c_bf16 ? __bfloat162float(((__nv_bfloat16 *)g.c)[o]) : ((float *)g.c)[o]);
          v += bias;
          if (g.gate_kind) {
            const float pre = g.gate[(int64_t)row * g.sgr + (int64_t)col * g.sgc];
            v *= g.gate_kind == 1 ? (pre > 0.f ? 1.f : 0.f)
                 : g.gate_kind == 2 ? 1.f / (1.f + expf(-pre))
                                    : -expm1f(-pre);
          }
          v = act_fn(v, g.act);
          if (g.c_bf16) ((__nv_bfloat16 *)g.c)[o] = __float2bfloat16(v);
          else ((float *)g.c)[o] = v;
          if (g.c2) {
            const int64_t o2 = (int64_t)row * g.sc2r + (int64_t)col * g.sc2c;
            if (g.c2_bf16) ((__nv_bfloat16 *)g.c2)[o2] = __float2bfloat16(v);
            else ((float *)g.c2)[o2] = v;
          }
        }
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    const uint32_t cols = BN < 32 ? 32 : BN;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
  }
}

template <int BN>
int32_t launch_gemm(const GemmArgs &g, kups_status *status, cudaStream_t stream) {
  const size_t smem = (size_t)2 * (kBM + BN) * kBK * 2 + 64;
  KUPS_CUDA_TRY(cudaFuncSetAttribute(gemm_tcgen05_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((g.m + kBM - 1) / kBM, (g.n + BN - 1) / BN, g.split_k);
  gemm_tcgen05_kernel<BN><<<grid, kGemmThreads, smem, stream>>>(g, status);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// TMA-fed variant for bfloat16 operands with K contiguous: one thread issues
// cp.async.bulk.tensor loads of 64-wide K chunks (128-byte rows, 128-byte swizzle) into a
// ring of STAGES stages, each completing on its mbarrier, and the MMAs of a chunk as soon as
// it has landed; the ring holds a K of up to 256 whole, so every load of such a tile is in
// flight at once.  A stage is refilled only after the commit of the MMAs that read it.  The other threads wait at the
// block barrier, then all run the register epilogue.  Every wait is bounded; on time-out the
// thread waits (bounded) for the loads and MMAs it issued, records KUPS_ERR_UNSUPPORTED, and
// the tile frees its tensor memory without writing C.

// Shared-memory matrix descriptor, K-major with 128-byte swizzle: 8-row groups of 128-byte
// rows 1024 bytes apart (stride byte offset), leading byte offset unused (1), version 1,
// layout type 2 (128-byte swizzle) in [61, 64).  The tile base is 1024-byte aligned; a K step
// of 16 elements advances the start address by 32 bytes.
__device__ inline uint64_t make_sdesc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__device__ inline void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

// 2-D tiled load of the box at (x = c0 along K, y = c1 along rows) into shared memory.
__device__ inline void tma_load_2d(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(mbar)
      : "memory");
}

template <int BN, int STAGES, int MINB>
__global__ void __launch_bounds__(kGemmThreads, MINB)
    gemm_tma_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, GemmArgs g,
                    kups_status *status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                          ~uintptr_t(1023));
  constexpr uint32_t kABytes = kBM * kBK * 2, kBBytes = BN * kBK * 2, kStage = kABytes + kBBytes;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * kStage);  // [STAGES]: chunk landed
  uint64_t *freed = full + STAGES;                                        // [STAGES]: its MMAs done
  uint64_t *done = freed + STAGES;                                        // every MMA of the tile done
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
  int *ok_flag = reinterpret_cast<int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int st = 0; st < STAGES; ++st) {
      mbar_init(smem_u32(&full[st]), 1);
      mbar_init(smem_u32(&freed[st]), 1);
    }
    mbar_init(smem_u32(done), 1);
    *ok_flag = 1;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const int nk_all = (g.k + kBK - 1) / kBK;
  const int per_split = (nk_all + g.split_k - 1) / g.split_k;
  const int kc_begin = blockIdx.z * per_split;
  const int kc_end = min(nk_all, kc_begin + per_split);
  const int nk = max(0, kc_end - kc_begin);
  if (tid == 0) {
    const uint32_t idesc = make_idesc(kBM, BN);
    auto sa = [&](int st) { return smem_u32(smem + st * kStage); };
    auto sb = [&](int st) { return smem_u32(smem + st * kStage + kABytes); };
    auto load = [&](int j) {  // chunk j of this tile's K range into stage j % STAGES
      const int st = j % STAGES, k0 = (kc_begin + j) * kBK;
      mbar_expect_tx(smem_u32(&full[st]), kStage);
      tma_load_2d(sa(st), &ta, k0, m0, smem_u32(&full[st]));
      tma_load_2d(sb(st), &tb, k0, n0, smem_u32(&full[st]));
    };
    bool ok = true;
    int issued = 0, consumed = 0;
    for (; issued < min(STAGES, nk); ++issued) load(issued);
    for (int i = 0; i < nk && ok; ++i) {
      const int st = i % STAGES;
      const uint32_t par = (uint32_t)(i / STAGES) & 1u;
      ok = mbar_wait(smem_u32(&full[st]), par);
      if (!ok) break;
      consumed = i + 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int ks = 0; ks < kBK / 16; ++ks) {
        const uint64_t ad = make_sdesc_sw128(sa(st) + ks * 32);
        const uint64_t bd = make_sdesc_sw128(sb(st) + ks * 32);
        const uint32_t accumulate = (i > 0 || ks > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&freed[st]))
                   : "memory");
      if (issued < nk) {  // refill this stage once its MMAs are done
        ok = mbar_wait(smem_u32(&freed[st]), par);
        if (!ok) break;
        load(issued++);
      }
    }
    // every MMA issued so far completes before the accumulator is read or freed
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(done))
                 : "memory");
    const bool mma_done = mbar_wait(smem_u32(done), 0u);
    if (!ok) {  // loads still in flight land before the tile exits
      for (int j = consumed; j < issued; ++j)
        mbar_wait(smem_u32(&full[j % STAGES]), (uint32_t)(j / STAGES) & 1u);
    }
    *ok_flag = (ok && mma_done) ? 1 : 0;
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!*ok_flag) {
    if (tid == 0) status_error(status, KUPS_ERR_UNSUPPORTED, blockIdx.x);
  } else if (nk > 0) {
    register_epilogue<BN>(g, tmem, m0, n0, warp, lane);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN));
}

bool encode_operand_map(PFN_cuTensorMapEncodeTiled_v12000 enc, CUtensorMap *m, const void *p, int64_t rows,
                        int64_t k, int64_t sr, int box_rows);

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// Tensor map of a bfloat16 [rows, k] operand with row stride sr elements (K contiguous), boxes
// of 64 x box_rows, 128-byte swizzle; out-of-range elements read as zero.  The last maps made
// are kept (a training step passes the same weights and rows every step), so encoding runs
// once per distinct operand; the cache is per host thread.
bool operand_map(CUtensorMap *m, const void *p, int64_t rows, int64_t k, int64_t sr, int box_rows) {
  struct Entry {
    const void *p;
    int64_t rows, k, sr;
    int box;
    CUtensorMap map;
  };
  constexpr int kCache = 32;
  static thread_local Entry cache[kCache];
  static thread_local int next = 0;
  for (int i = 0; i < kCache; ++i) {
    const Entry &e = cache[i];
    if (e.p == p && e.rows == rows && e.k == k && e.sr == sr && e.box == box_rows) {
      *m = e.map;
      return true;
    }
  }
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (enc == nullptr || !encode_operand_map(enc, m, p, rows, k, sr, box_rows)) return false;
  cache[next] = Entry{p, rows, k, sr, box_rows, *m};
  next = (next + 1) % kCache;
  return true;
}

bool encode_operand_map(PFN_cuTensorMapEncodeTiled_v12000 enc, CUtensorMap *m, const void *p, int64_t rows,
                        int64_t k, int64_t sr, int box_rows) {
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)sr * 2};
  cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(p), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whether the TMA-fed kernel applies: both operands bfloat16 with K contiguous, 16-byte aligned
// bases and row strides of at least K elements that are multiples of 8, and the register epilogue.
bool tma_operands(const GemmArgs &g) {
  auto al16 = [](const void *q) { return (((uintptr_t)q) & 15) == 0; };
  return g.a_bf16 && g.b_bf16 && g.sac == 1 && g.sbc == 1 && g.sar % 8 == 0 && g.sbr % 8 == 0 && g.sar >= g.k &&
         g.sbr >= g.k && al16(g.a) && al16(g.b) && g.row_epi;
}

template <int BN, int STAGES, int MINB>
int32_t launch_gemm_tma(const GemmArgs &g, kups_status *status, cudaStream_t stream, bool &launched) {
  launched = false;
  CUtensorMap ta, tb;
  if (!operand_map(&ta, g.a, g.m, g.k, g.sar, kBM) || !operand_map(&tb, g.b, g.n, g.k, g.sbr, BN)) return KUPS_OK;
  const size_t smem = (size_t)STAGES * (kBM + BN) * kBK * 2 + 1024 + 256;
  static int set_device = -1;  // the attribute is per device: set it once for each device in turn
  int dev = 0;
  KUPS_CUDA_TRY(cudaGetDevice(&dev));
  if (set_device != dev) {
    KUPS_CUDA_TRY(cudaFuncSetAttribute(gemm_tma_kernel<BN, STAGES, MINB>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set_device = dev;
  }
  dim3 grid((g.m + kBM - 1) / kBM, (g.n + BN - 1) / BN, g.split_k);
  gemm_tma_kernel<BN, STAGES, MINB><<<grid, kGemmThreads, smem, stream>>>(ta, tb, g, status);
  launched = true;
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

// Whether the register epilogue of gemm_tcgen05_kernel applies: float32 C (and the optional
// bias, gate and bfloat16 copy) row-major with unit column stride and 16-byte aligned rows,
// N a multiple of 32, no beta term.
bool row_epilogue(const GemmArgs &g) {
  auto al16 = [](const void *q) { return (((uintptr_t)q) & 15) == 0; };
  if (g.c_bf16 || g.scc != 1 || g.scr % 4 != 0 || !al16(g.c) || g.n % 32 != 0) return false;
  if (g.split_k > 1) return true;  // alpha * partial added into C
  if (g.beta != 0.f) return false;
  if (g.bias != nullptr && !al16(g.bias)) return false;
  if (g.gate_kind != 0 && (g.sgc != 1 || g.sgr % 4 != 0 || !al16(g.gate))) return false;
  if (g.c2 != nullptr && (!g.c2_bf16 || g.sc2c != 1 || g.sc2r % 8 != 0 || !al16(g.c2))) return false;
  return true;
}

int32_t dispatch_gemm(const GemmArgs &g0, kups_status *status, cudaStream_t st) {
  GemmArgs g = g0;
  g.row_epi = row_epilogue(g) ? 1 : 0;
  auto al32 = [](const void *q) { return (((uintptr_t)q) & 31) == 0; };
  g.row_v8 = g.row_epi && g.scr % 8 == 0 && al32(g.c) &&
             (g.c2 == nullptr || (g.sc2r % 16 == 0 && al32(g.c2)));
  if (tma_operands(g)) {  // one tile column per 256 of N; the tile ring holds K <= 256 whole
    // tiles as wide as N (up to 256, one CTA per SM) with a four-stage ring: measured against
    // 128 x 128 and 128 x 64 tiles with two stages (three and four CTAs per SM) and with four
    // stages, it was the fastest on a network step by separate products, 16384 x 256 x 256 and their
    // gradients (0.194 against 0.196-0.214 ms)
    bool launched = false;
    const int32_t rc = g.n <= 64    ? launch_gemm_tma<64, 4, 1>(g, status, st, launched)
                       : g.n <= 128 ? launch_gemm_tma<128, 4, 1>(g, status, st, launched)
                                    : launch_gemm_tma<256, 4, 1>(g, status, st, launched);
    if (launched || rc != KUPS_OK) return rc;
  }
  // Tile width: 128 (64 for N <= 64), narrowed to 64 while the grid would leave SMs idle (fewer than
  // two CTAs per SM of 148).
  const int64_t rows = ((int64_t)g.m + kBM - 1) / kBM * g.split_k;
  int bn = g.n <= 64 ? 64 : 128;
  while (bn > 64 && rows * ((g.n + bn - 1) / bn) < 2 * 148) bn >>= 1;
  return bn == 64 ? launch_gemm<64>(g, status, st) : launch_gemm<128>(g, status, st);
}

// ============================================================================
// Learned insertion proposal: network, training and grid density.
//
// Fixed architecture: 64 Fourier features of the fractional position f,
// (sin, cos)(2 pi m_j . f) for 32 integer vectors m_j, three softplus layers of
// width 256 (tensor-core products, bfloat16 operands, float32 accumulation) and
// a linear output g(f).  Parameters are one flat float32 array at the kOff*
// offsets plus a bfloat16 copy that the matrix products read.  Training minimises
// the noise-contrastive loss with equal halves of data and uniform points,
//   L = (1/n) [sum_data softplus(-g) + sum_uniform softplus(g)],
// whose minimiser is g(f) = ln p_data(f) for f uniform on the unit cube.
constexpr int kFreq = 32, kIn = 2 * kFreq, kHid = 256;
constexpr int64_t kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
                  kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kHid, kOffW4 = kOffB3 + kHid,
                  kOffB4 = kOffW4 + kHid, kParams = kOffB4 + 1;
static_assert(kParams == KUPS_MLP_PARAMS, "parameter layout");
constexpr int64_t kChunk = 65536;  // points of the largest training batch, and that a workspace is sized for

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Rows of c points that the weight gradients read, bfloat16: features, h1, h2 and dL/dz of the three
// layers; h1 in float32 (its gate in the backward pass); scratch of the grid normaliser.
struct MlpWork {
  __nv_bfloat16 *feat, *h1b, *h2b, *dz1, *dz2, *dz3;
  float *h1;
  double *partial;
  __nv_bfloat16 *weights;  // aligned copy of the weights, if the network's own are not
};

constexpr int64_t kWeightCopy = (kParams + 7) / 8 * 8 + 2 * kHid * kHid;

constexpr int kNormBlocks = 152, kNormThreads = 1024;

MlpWork carve(void *ws, int64_t c) {
  char *p = (char *)(((uintptr_t)ws + 255) & ~uintptr_t(255));
  MlpWork w;
  auto take = [&](size_t bytes) {
    char *q = p;
    p += align256(bytes);
    return (void *)q;
  };
  w.feat = (__nv_bfloat16 *)take(2 * (size_t)c * kIn);
  w.h1b = (__nv_bfloat16 *)take(2 * (size_t)c * kHid);
  w.h2b = (__nv_bfloat16 *)take(2 * (size_t)c * kHid);
  w.dz1 = (__nv_bfloat16 *)take(2 * (size_t)c * kHid);
  w.dz2 = (__nv_bfloat16 *)take(2 * (size_t)c * kHid);
  w.dz3 = (__nv_bfloat16 *)take(2 * (size_t)c * kHid);
  w.h1 = (float *)take(4 * (size_t)c * kHid);
  w.partial = (double *)take(8 * (size_t)3 * kNormBlocks);
  w.weights = (__nv_bfloat16 *)take(2 * (size_t)kWeightCopy);
  return w;
}

size_t work_bytes(int64_t c) {
  return align256(2 * (size_t)c * kIn) + 5 * align256(2 * (size_t)c * kHid) + align256(4 * (size_t)c * kHid) +
         align256(8 * (size_t)3 * kNormBlocks) + align256(2 * (size_t)kWeightCopy) + 256;
}

__device__ inline float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ inline float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// sin and cos of 2 pi (m . f) for a point whose coordinates, reduced to [-0.5, 0.5), are the
// float pairs fh + fl.  The phase is carried as a float pair (the products' rounding errors
// recovered by fma, the sums' by two-sum) and reduced modulo one before its single rounding
// to float, so the phase reaching sincospi is within 3e-8 of a turn of the float64 phase and
// the features round to the same bfloat16 values as the float64 features almost always.
__device__ inline void phase_sincos(const int32_t *m, const float fh[3], const float fl[3], float &sn, float &cs) {
  const float m0 = (float)m[0], m1 = (float)m[1], m2 = (float)m[2];
  const float p0 = __fmul_rn(m0, fh[0]), p1 = __fmul_rn(m1, fh[1]), p2 = __fmul_rn(m2, fh[2]);
  float lo = __fadd_rn(__fadd_rn(fmaf(m0, fh[0], -p0), fmaf(m1, fh[1], -p1)), fmaf(m2, fh[2], -p2));
  lo = fmaf(m0, fl[0], fmaf(m1, fl[1], fmaf(m2, fl[2], lo)));
  const float s1 = __fadd_rn(p0, p1);
  float b = __fsub_rn(s1, p0);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(p0, __fsub_rn(s1, b)), __fsub_rn(p1, b)));
  const float s2 = __fadd_rn(s1, p2);
  b = __fsub_rn(s2, s1);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(s1, __fsub_rn(s2, b)), __fsub_rn(p2, b)));
  float t = __fadd_rn(__fsub_rn(s2, rintf(s2)), lo);
  t = __fsub_rn(t, rintf(t));
  sincospif(2.0f * t, &sn, &cs);
}

// Equal halves: rows [0, batch/2) are data points drawn with replacement,
// rows [batch/2, batch) uniform points; Philox keyed by (seed, step, row).
__global__ void nce_batch_kernel(const double *data, int64_t n_data, int64_t batch, uint64_t seed, uint64_t step,
                                 double *x, float *label) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= batch) return;
  const U4 c{(uint32_t)r, (uint32_t)(r >> 32), (uint32_t)step, (uint32_t)(step >> 32)};
  const U4 w = philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  if (r < batch / 2) {
    const uint64_t idx = ((((uint64_t)w.x) << 32) | w.y) % (uint64_t)n_data;
    for (int a = 0; a < 3; ++a) x[3 * r + a] = data[3 * idx + a];
    label[r] = 1.f;
  } else {
    x[3 * r] = w.x * (1.0 / 4294967296.0);
    x[3 * r + 1] = w.y * (1.0 / 4294967296.0);
    x[3 * r + 2] = w.z * (1.0 / 4294967296.0);
    label[r] = 0.f;
  }
}

// Adam (Kingma & Ba 2015) with bias corrections c1 = 1 / (1 - beta1^t),
// c2 = 1 / (1 - beta2^t); refreshes the bfloat16 copy and zeroes the gradient.
// bfloat16 copies of a parameter: the flat copy, and for W2 / W3 the transposed copy
// (W^T[in][out]) that the training kernel multiplies the next layer's gradients by.
__device__ inline void store_bf16(__nv_bfloat16 *pb, __nv_bfloat16 *pbt, int64_t i, float v) {
  const __nv_bfloat16 b = __float2bfloat16(v);
  pb[i] = b;
  if (i >= kOffW2 && i < kOffB2) {
    const int64_t l = i - kOffW2;
    pbt[(l % kHid) * kHid + l / kHid] = b;
  } else if (i >= kOffW3 && i < kOffB3) {
    const int64_t l = i - kOffW3;
    pbt[kHid * kHid + (l % kHid) * kHid + l / kHid] = b;
  }
}

__global__ void adam_kernel(float *p, __nv_bfloat16 *pb, __nv_bfloat16 *pbt, float *g, float *m, float *v, int64_t n,
                            float lr, float b1, float b2, float eps, float c1, float c2) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  p[i] = pi;
  store_bf16(pb, pbt, i, pi);
  g[i] = 0.f;
}

// Weights uniform with variance 1 / fan_in (Philox keyed by (seed, index)),
// biases zero; optimiser state and gradients zero.
__global__ void init_kernel(float *p, __nv_bfloat16 *pb, __nv_bfloat16 *pbt, float *g, float *m, float *v,
                            uint64_t seed) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  float fan = 0.f;
  if (i < kOffB1) fan = kIn;
  else if ((i >= kOffW2 && i < kOffB2) || (i >= kOffW3 && i < kOffB3) || (i >= kOffW4 && i < kOffB4)) fan = kHid;
  float val = 0.f;
  if (fan > 0.f) {
    const U4 c{(uint32_t)i, (uint32_t)(i >> 32), 0x6d6c70u, 0u};
    const U4 w = philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    const float u = (float)(w.x >> 8) * (1.0f / 16777216.0f);
    val = (2.f * u - 1.f) * sqrtf(3.f / fan);
  }
  p[i] = val;
  store_bf16(pb, pbt, i, val);
  g[i] = 0.f;
  m[i] = 0.f;
  v[i] = 0.f;
}

__device__ inline float block_max1024(float v, float *red) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    float w = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : -INFINITY;
    for (int o = 16; o > 0; o >>= 1) w = fmaxf(w, __shfl_xor_sync(0xffffffffu, w, o));
    if (threadIdx.x == 0) red[0] = w;
  }
  __syncthreads();
  const float r = red[0];
  __syncthreads();
  return r;
}

__device__ inline double block_sum_d(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double w = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (threadIdx.x == 0) red[0] = w;
  }
  __syncthreads();
  const double r = red[0];
  __syncthreads();
  return r;
}

// node holds g on entry; on exit d = exp(temper (g - max g)) + floor_frac * mean(exp(temper (g - max g))).
// Two launches over the whole GPU: each block of grid_partials_kernel reduces a grid-stride
// share of the nodes to (its max m_b, sum exp(temper (g - m_b)) in float64, a non-finite flag);
// every block of grid_apply_kernel combines the partials (M = max m_b,
// Z = sum_b s_b exp(temper (m_b - M))) and rewrites its share of the nodes.
__global__ void __launch_bounds__(kNormThreads) grid_partials_kernel(const float *node, int64_t n, float temper,
                                                                     double *partial, kups_status *status) {
  __shared__ float redf[32];
  __shared__ double redd[32];
  float mx = -INFINITY;
  int bad = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float v = node[i];
    if (!isfinite(v)) bad = 1;
    mx = fmaxf(mx, v);
  }
  bad = __syncthreads_or(bad);
  mx = block_max1024(mx, redf);
  double s = 0.0;
  if (!bad && mx > -INFINITY)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
      s += expf(temper * (node[i] - mx));
  s = block_sum_d(s, redd);
  if (threadIdx.x == 0) {
    partial[3 * blockIdx.x] = (double)mx;
    partial[3 * blockIdx.x + 1] = s;
    partial[3 * blockIdx.x + 2] = bad ? 1.0 : 0.0;
    if (bad) status_error(status, KUPS_ERR_NONFINITE, -1);
  }
}

__global__ void __launch_bounds__(256) grid_apply_kernel(float *node, int64_t n, float temper, float floor_frac,
                                                         const double *partial, int n_partial) {
  // thread b < n_partial (<= 256) holds partial b: block max, then the rescaled sums
  __shared__ float redf[32];
  __shared__ double redd[32];
  const int b = threadIdx.x;
  const bool has = b < n_partial;
  const float mb = has ? (float)partial[3 * b] : -INFINITY;
  const int bad = __syncthreads_or(has && partial[3 * b + 2] != 0.0);
  if (bad) return;
  const float M = block_max1024(mb, redf);
  const double zb = has && mb > -INFINITY ? partial[3 * b + 1] * (double)expf(temper * (mb - M)) : 0.0;
  const float fl = (float)(floor_frac * (block_sum_d(zb, redd) / (double)n));
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    node[i] = expf(temper * (node[i] - M)) + fl;
}

// cdf[c] = sum_{c' < c} mass(c'), mass = mean of the cell's 8 corners (float64),
// in three passes: each block of 256 threads scans kCdfPerBlock cells (8 per thread)
// and records its total, one block scans the totals, and the block offsets are added.
constexpr int kCdfThreads = 256, kCdfPerThread = 8, kCdfPerBlock = kCdfThreads * kCdfPerThread;

__device__ inline double cell_mass(const float *node, int g, int64_t c) {
  const int i = (int)(c / ((int64_t)g * g)), j = (int)((c / g) % g), k = (int)(c % g);
  double d[8];
  grid_corners(node, g, i, j, k, d);
  double s = 0.0;
  for (int b = 0; b < 8; ++b) s += d[b];
  return s * 0.125;
}

// inclusive scan of one double per thread over a block of kCdfThreads threads
__device__ inline double block_inclusive_scan(double v, double *sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < kCdfThreads; o <<= 1) {
    const double add = threadIdx.x >= (unsigned)o ? sh[threadIdx.x - o] : 0.0;
    __syncthreads();
    sh[threadIdx.x] += add;
    __syncthreads();
  }
  const double r = sh[threadIdx.x];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kCdfThreads) grid_cdf_local_kernel(const float *node, int g, double *cdf,
                                                                      double *block_total) {
  __shared__ double sh[kCdfThreads];
  const int64_t n = (int64_t)g * g * g;
  const int64_t c0 = (int64_t)blockIdx.x * kCdfPerBlock + (int64_t)threadIdx.x * kCdfPerThread;
  double m[kCdfPerThread], local = 0.0;
  for (int t = 0; t < kCdfPerThread; ++t) {
    m[t] = c0 + t < n ? cell_mass(node, g, c0 + t) : 0.0;
    local += m[t];
  }
  double run = block_inclusive_scan(local, sh) - local;
  for (int t = 0; t < kCdfPerThread; ++t) {
    if (c0 + t < n) cdf[c0 + t] = run;
    run += m[t];
  }
  if (threadIdx.x == kCdfThreads - 1) block_total[blockIdx.x] = run;
}

// exclusive scan of the block totals (one block; offsets written in place), cdf[n] = total
__global__ void __launch_bounds__(kCdfThreads) grid_cdf_totals_kernel(double *block_total, int n_blocks, double *cdf,
                                                                       int64_t n) {
  __shared__ double sh[kCdfThreads];
  __shared__ double round_total;
  double carry = 0.0;
  for (int b0 = 0; b0 < n_blocks; b0 += kCdfThreads) {
    const int b = b0 + threadIdx.x;
    const double v = b < n_blocks ? block_total[b] : 0.0;
    const double inc = block_inclusive_scan(v, sh);
    if (b < n_blocks) block_total[b] = carry + inc - v;
    if (threadIdx.x == kCdfThreads - 1) round_total = inc;
    __syncthreads();
    carry += round_total;
    __syncthreads();
  }
  if (threadIdx.x == 0) cdf[n] = carry;
}

__global__ void grid_cdf_offset_kernel(double *cdf, int64_t n, const double *block_offset) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c < n) cdf[c] += block_offset[c / kCdfPerBlock];
}

__global__ void proposal_sample_kernel(const float *node, const double *cdf, int g, int64_t n, uint64_t seed,
                                       double *f, double *lnq) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const U4 a = philox4x32_10(U4{(uint32_t)i, (uint32_t)(i >> 32), 1u, 0u}, (uint32_t)seed, (uint32_t)(seed >> 32));
  const U4 b = philox4x32_10(U4{(uint32_t)i, (uint32_t)(i >> 32), 2u, 0u}, (uint32_t)seed, (uint32_t)(seed >> 32));
  const double ua[3] = {u32_open0(b.x), u32_open0(b.y), u32_open0(b.z)};
  double x[3];
  const double l = grid_sample(node, cdf, g, u53(a.x, a.y), u53(a.z, a.w), ua, x);
  for (int k = 0; k < 3; ++k) f[3 * i + k] = x[k];
  lnq[i] = l;
}

__global__ void proposal_density_kernel(const float *node, const double *cdf, int g, const double *f, int64_t n,
                                        double *lnq) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x[3] = {f[3 * i], f[3 * i + 1], f[3 * i + 2]};
  lnq[i] = grid_log_q(node, cdf, g, x);
}

// ============================================================================
// Fused forward pass (inference: kups_mlp_fwd and the grid refresh).  A persistent CTA works on two
// tiles of 128 points at a time, each with its own A operand in shared memory and its own 256-column
// accumulator in tensor memory, by three kinds of warps that meet only at mbarriers:
//   * sixteen epilogue warps, all on one tile and then on the other: features of the tile's points
//     (coordinates reduced to [-0.5, 0.5) once in float64 and split into float pairs, the 32 phases as
//     float pairs, phase_sincos) written as the first layer's A operand (bfloat16, no-swizzle K-major
//     core matrices); after each layer tcgen05.ld, bias, softplus, and the next layer's A operand, or
//     after the last the head (w4 . h3 + b4);
//   * one warp loading the weights by TMA, 64 columns of W (256 rows, 128-byte swizzle, 32 KB) at a
//     time, through a ring of two stages, in the order the MMAs take them;
//   * one warp issuing tcgen05.mma (128 x 256 x 16, BF16 in, FP32 accumulate): the layers of the two
//     tiles in turn, so that one tile's MMAs run under the other tile's epilogue.
// What bounds it is the epilogue's issue slots and SFU operations (about ten instructions per
// activation, two of them on the SFU) with the hand-overs between layers: 54 % issue, tensor pipe 25 %.
// 3e5 points: 152 us (158 with eight epilogue warps for each tile, which idle together while its MMAs
// run; 162 without the next 16 columns on their way during the epilogue's work); 292 us with one tile of
// 256 points whose MMAs and epilogue took turns, block barriers at every weight chunk and 16-byte
// copies by all threads.
// Every mbarrier wait is bounded; the one that runs out raises a flag that ends the others, the
// kernel records KUPS_ERR_UNSUPPORTED, waits (bounded) for its copies and MMAs, frees its tensor
// memory and returns.
constexpr int kFwdTile = 128, kFwdEpiWarps = 16, kFwdThreads = 32 * (kFwdEpiWarps + 2), kFwdKc = 64;
constexpr uint32_t kFwdStage = kHid * kFwdKc * 2;  // 32 KB: one weight chunk
constexpr size_t kFwdA = (size_t)kFwdTile * kHid * 2;  // 64 KB: a tile's A operand, K up to 256
// shared memory: weight stages | A operands | head partials [2][4][128] | coordinates [2][6][128] |
// biases b1 b2 b3 and head weights w4 [4][256] | frequencies [32][3] | b4 | mbarriers, TMEM slot, flag
constexpr size_t kFwdOffA = 2 * (size_t)kFwdStage;
constexpr size_t kFwdOffPart = kFwdOffA + 2 * kFwdA;
constexpr size_t kFwdOffFr = kFwdOffPart + 2 * 4 * kFwdTile * 4;
constexpr size_t kFwdOffPar = kFwdOffFr + 2 * 6 * kFwdTile * 4;
constexpr size_t kFwdOffFreq = kFwdOffPar + 4 * kHid * 4;
constexpr size_t kFwdOffB4 = kFwdOffFreq + 3 * kFreq * 4;
constexpr size_t kFwdOffBar = kFwdOffB4 + 16;
constexpr size_t kFwdSmem = kFwdOffBar + 128 + 1024;  // the stages start on 1024 bytes
static_assert(kFwdOffBar % 8 == 0, "mbarriers are 8-byte aligned");
static_assert(kFwdSmem <= 227 * 1024, "forward pass shared memory above the per-CTA limit");

__device__ inline int fwd_core(int r, int kk, int K) {
  return ((r >> 3) * (K / 8) + (kk >> 3)) * 64 + (r & 7) * 8 + (kk & 7);
}

// mbar_wait that also ends when another wait of the CTA has run out (*stop), and raises it itself.
__device__ inline bool mbar_wait_or_stop(uint32_t addr, uint32_t phase, volatile int *stop) {
  for (long long i = 0; i < kWaitLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(addr), "r"(phase)
        : "memory");
    if (done) return true;
    if (*stop) return false;
  }
  *stop = 1;
  return false;
}

__device__ inline void mbar_arrive(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(addr) : "memory");
}

__device__ inline void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ inline void mma_f16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate ? 1u : 0u));
}

__device__ inline void tmem_load16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__global__ void __launch_bounds__(kFwdThreads, 1)
mlp_forward_kernel(const __grid_constant__ CUtensorMap w1, const __grid_constant__ CUtensorMap w2,
                   const __grid_constant__ CUtensorMap w3, const float *p, const int32_t *freq, const double *x,
                   int64_t n, int grid, float *g_out, kups_status *status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                          ~uintptr_t(1023));
  float *spar = reinterpret_cast<float *>(smem + kFwdOffPar);  // [4][256] b1, b2, b3, w4
  int32_t *sfreq = reinterpret_cast<int32_t *>(smem + kFwdOffFreq);
  float *sb4 = reinterpret_cast<float *>(smem + kFwdOffB4);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kFwdOffBar);
  uint64_t *full = bars, *freed = bars + 2;        // [2] weight stage landed / its MMAs done
  uint64_t *ready = bars + 4, *acc = bars + 6;     // [2] tile's A operand written / accumulator complete
  uint64_t *meet = bars + 8;                       // the epilogue threads meet
  uint64_t *drained = bars + 10;                   // every MMA done (after a stop)
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 11);
  volatile int *stop = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int e = tid; e < 4 * kHid; e += kFwdThreads) {
    const int which = e / kHid;
    const int64_t off = which == 0 ? kOffB1 : which == 1 ? kOffB2 : which == 2 ? kOffB3 : kOffW4;
    spar[e] = p[off + e % kHid];
  }
  for (int e = tid; e < 3 * kFreq; e += kFwdThreads) sfreq[e] = freq[e];
  if (tid == 0) sb4[0] = p[kOffB4];
  if (warp == kFwdEpiWarps) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * kHid));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int k = 0; k < 2; ++k) {
      mbar_init(smem_u32(&full[k]), 1);
      mbar_init(smem_u32(&freed[k]), 1);
      mbar_init(smem_u32(&ready[k]), 32 * kFwdEpiWarps);
      mbar_init(smem_u32(&acc[k]), 1);
    }
    mbar_init(smem_u32(meet), 32 * kFwdEpiWarps);
    mbar_init(smem_u32(drained), 1);
    *stop = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // tiles u = blockIdx + gridDim (2 t + h) go to slot h of this CTA: the first gridDim tiles to every
  // CTA's slot 0, so that few points still spread over the chip
  const int64_t n_tiles = (n + kFwdTile - 1) / kFwdTile;
  auto tiles_of = [&](int h) {
    const int64_t first = blockIdx.x + (int64_t)gridDim.x * h;
    return first < n_tiles ? (n_tiles - 1 - first) / (2 * (int64_t)gridDim.x) + 1 : (int64_t)0;
  };
  const int64_t count[2] = {tiles_of(0), tiles_of(1)};  // count[0] >= count[1]
  if (warp < kFwdEpiWarps) {
    const int quarter = warp & 3, cq = warp >> 2, row = quarter * 32 + lane, cb = cq * 64;  // TMEM lanes, columns
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    __nv_bfloat16 *const sA0 = reinterpret_cast<__nv_bfloat16 *>(smem + kFwdOffA);
    float *part = reinterpret_cast<float *>(smem + kFwdOffPart), *fr = reinterpret_cast<float *>(smem + kFwdOffFr);
    const float *w4 = spar + 3 * kHid;
    bool ok = true;
    uint32_t parity[2] = {0u, 0u}, met = 0u;  // of the slots' next accumulators and of the next meeting
    // waits end alike for a whole warp (tcgen05.ld is a warp's operation)
    auto wait = [&](uint64_t *bar, uint32_t &phase) {
      const bool done = __all_sync(0xffffffffu, mbar_wait_or_stop(smem_u32(bar), phase, stop));
      phase ^= 1u;
      return done;
    };
    auto meeting = [&]() {
      mbar_arrive(smem_u32(meet));
      return wait(meet, met);
    };
    // slot h's A operand is visible to the tensor cores and its accumulator read: its next layer may start
    auto start_layer = [&](int h) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(smem_u32(&ready[h]));
    };
    for (int64_t t = 0; t < count[0]; ++t) {
      const int slots = t < count[1] ? 2 : 1;
      auto first_row = [&](int h) { return (blockIdx.x + (int64_t)gridDim.x * (2 * t + h)) * kFwdTile; };
      if (tid < slots * kFwdTile) {  // coordinates reduced to [-0.5, 0.5) in float64, kept as float pairs
        const int h = tid / kFwdTile, ht = tid % kFwdTile;
        const int64_t pt = first_row(h) + ht;
        double f[3] = {0.0, 0.0, 0.0};
        if (pt < n) {
          if (x != nullptr) {
            for (int a = 0; a < 3; ++a) f[a] = x[3 * pt + a];
          } else {
            const int64_t g2 = (int64_t)grid * grid;
            f[0] = (double)(pt / g2) / grid;
            f[1] = (double)((pt / grid) % grid) / grid;
            f[2] = (double)(pt % grid) / grid;
          }
        }
        for (int a = 0; a < 3; ++a) {
          const double red = f[a] - rint(f[a]);
          const float hi = (float)red;
          fr[(6 * h + a) * kFwdTile + ht] = hi;
          fr[(6 * h + 3 + a) * kFwdTile + ht] = (float)(red - (double)hi);
        }
      }
      ok = meeting();
      if (!ok) break;
      for (int h = 0; h < slots; ++h) {  // 8 of the 32 phases of a row
        const float *c = fr + 6 * h * kFwdTile + row;
        const bool in = first_row(h) + row < n;
        const float fh[3] = {c[0], c[kFwdTile], c[2 * kFwdTile]};
        const float fl[3] = {c[3 * kFwdTile], c[4 * kFwdTile], c[5 * kFwdTile]};
        __nv_bfloat16 *sA = sA0 + h * (kFwdA / 2);
#pragma unroll 2
        for (int j = 8 * cq; j < 8 * cq + 8; ++j) {
          float sn = 0.f, cs = 0.f;
          if (in) phase_sincos(sfreq + 3 * j, fh, fl, sn, cs);
          *reinterpret_cast<__nv_bfloat162 *>(sA + fwd_core(row, 2 * j, kIn)) = __floats2bfloat162_rn(sn, cs);
        }
        start_layer(h);
      }
      for (int layer = 0; layer < 3 && ok; ++layer)
        for (int h = 0; h < slots; ++h) {
          ok = wait(&acc[h], parity[h]);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const float *bias = spar + layer * kHid;
          __nv_bfloat16 *sA = sA0 + h * (kFwdA / 2);
          float head = 0.f;
          // 16 columns at a time, the next 16 on their way from tensor memory meanwhile
          uint32_t next[16];
          const uint32_t t0 = lanes + (uint32_t)(h * kHid + cb);
          tmem_load16(t0, next);
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const int c0 = cb + 16 * s;
            uint32_t r[16];
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i] = next[i];
            if (s < 3) tmem_load16(t0 + 16 * (s + 1), next);
            const float4 *b4 = reinterpret_cast<const float4 *>(bias + c0);
            float v[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 b = b4[q];
              v[4 * q] = softplus_fast(__uint_as_float(r[4 * q]) + b.x);
              v[4 * q + 1] = softplus_fast(__uint_as_float(r[4 * q + 1]) + b.y);
              v[4 * q + 2] = softplus_fast(__uint_as_float(r[4 * q + 2]) + b.z);
              v[4 * q + 3] = softplus_fast(__uint_as_float(r[4 * q + 3]) + b.w);
            }
            if (layer < 2) {
              // next layer's A operand: 2 core-matrix rows of 8 bfloat16 (16 bytes each)
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                __nv_bfloat162 hv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) hv[u] = __floats2bfloat162_rn(v[q * 8 + 2 * u], v[q * 8 + 2 * u + 1]);
                *reinterpret_cast<uint4 *>(sA + fwd_core(row, c0 + q * 8, kHid)) = *reinterpret_cast<uint4 *>(hv);
              }
            } else {
              const float4 *h4 = reinterpret_cast<const float4 *>(w4 + c0);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const float4 w = h4[q];
                head = fmaf(v[4 * q], w.x, head);
                head = fmaf(v[4 * q + 1], w.y, head);
                head = fmaf(v[4 * q + 2], w.z, head);
                head = fmaf(v[4 * q + 3], w.w, head);
              }
            }
          }
          if (layer < 2) start_layer(h);
          else part[(4 * h + cq) * kFwdTile + row] = head;  // of 64 columns
        }
      if (!ok) break;
      ok = meeting();
      if (!ok) break;
      if (tid < slots * kFwdTile) {
        const int h = tid / kFwdTile, ht = tid % kFwdTile;
        const float *g = part + 4 * h * kFwdTile + ht;
        if (first_row(h) + ht < n)
          g_out[first_row(h) + ht] = ((g[0] + g[kFwdTile]) + (g[2 * kFwdTile] + g[3 * kFwdTile])) + sb4[0];
      }
    }
  } else if (warp == kFwdEpiWarps) {
    if (lane == 0) {  // weights, in the order of the MMAs
      int64_t q = 0;
      bool ok = true;
      for (int64_t t = 0; t < count[0] && ok; ++t)
        for (int layer = 0; layer < 3 && ok; ++layer)
          for (int h = 0; h < 2 && ok; ++h) {
            if (t >= count[h]) continue;
            const CUtensorMap *map = layer == 0 ? &w1 : layer == 1 ? &w2 : &w3;
            for (int c = 0; c < (layer == 0 ? kIn : kHid) / kFwdKc; ++c, ++q) {
              const int st = (int)(q & 1);
              if (q >= 2) ok = mbar_wait_or_stop(smem_u32(&freed[st]), (uint32_t)((q >> 1) - 1) & 1u, stop);
              if (!ok) break;
              mbar_expect_tx(smem_u32(&full[st]), kFwdStage);
              tma_load_2d(smem_u32(smem + st * kFwdStage), map, c * kFwdKc, 0, smem_u32(&full[st]));
            }
          }
      if (*stop)  // copies in flight land before the CTA ends
        for (int64_t k = q > 2 ? q - 2 : 0; k < q; ++k) mbar_wait(smem_u32(&full[k & 1]), (uint32_t)(k >> 1) & 1u);
    }
  } else if (lane == 0) {
    const uint32_t idesc = make_idesc(kFwdTile, kHid);
    int64_t q = 0;
    uint32_t parity[2] = {0u, 0u};
    bool ok = true;
    for (int64_t t = 0; t < count[0] && ok; ++t)
      for (int layer = 0; layer < 3 && ok; ++layer)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!ok || t >= count[h]) continue;
          ok = mbar_wait_or_stop(smem_u32(&ready[h]), parity[h], stop);
          if (!ok) continue;
          parity[h] ^= 1u;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int K = layer == 0 ? kIn : kHid;
          const uint32_t a0 = smem_u32(smem + kFwdOffA + h * kFwdA);
          for (int c = 0; c < K / kFwdKc; ++c, ++q) {
            const int st = (int)(q & 1);
            ok = mbar_wait_or_stop(smem_u32(&full[st]), (uint32_t)(q >> 1) & 1u, stop);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t b0 = smem_u32(smem + st * kFwdStage);
            for (int ks = 0; ks < kFwdKc / 16; ++ks)
              mma_f16(tmem + (uint32_t)(h * kHid), make_sdesc(a0 + (c * 4 + ks) * 256, 128, (K / 8) * 128),
                      make_sdesc_sw128(b0 + ks * 32), idesc, c > 0 || ks > 0);
            mma_commit(smem_u32(&freed[st]));
          }
          if (ok) mma_commit(smem_u32(&acc[h]));
        }
    if (*stop) {  // MMAs in flight end before the tensor memory is freed
      mma_commit(smem_u32(drained));
      mbar_wait(smem_u32(drained), 0u);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && *stop) status_error(status, KUPS_ERR_UNSUPPORTED, blockIdx.x);
  if (warp == kFwdEpiWarps) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kHid));
  }
}

// copy: room for the weights, taken where theirs do not start on a 16-byte boundary (TMA reads from those)
int32_t fused_forward(const kups_mlp *net, const double *x, int64_t n, int grid, float *g, __nv_bfloat16 *copy,
                      kups_status *status, cudaStream_t st) {
  if (n <= 0) return KUPS_OK;
  const __nv_bfloat16 *pb = (const __nv_bfloat16 *)net->param_bf16;
  if (((uintptr_t)pb & 15) != 0) {
    KUPS_CUDA_TRY(cudaMemcpyAsync(copy, pb, 2 * kParams, cudaMemcpyDeviceToDevice, st));
    pb = copy;
  }
  CUtensorMap w1, w2, w3;
  if (!operand_map(&w1, pb + kOffW1, kHid, kIn, kIn, kHid) || !operand_map(&w2, pb + kOffW2, kHid, kHid, kHid, kHid) ||
      !operand_map(&w3, pb + kOffW3, kHid, kHid, kHid, kHid))
    return KUPS_ERR_CUDA;
  KUPS_CUDA_TRY(cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem));
  const int64_t tiles = (n + kFwdTile - 1) / kFwdTile;
  const unsigned ctas = (unsigned)std::min<int64_t>(tiles, device_sm_count());
  mlp_forward_kernel<<<ctas, kFwdThreads, kFwdSmem, st>>>(w1, w2, w3, net->param, net->freq, x, n, grid, g, status);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

inline unsigned blocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// ============================================================================
// Training step.  One kernel runs forward, loss and backward of a tile of 128 points from its
// coordinates to the three layers' dL/dz, everything between the layers on chip, by the same three
// kinds of warps as the forward pass: sixteen epilogue warps (warp w: TMEM lanes 32 (w % 4) ..,
// columns 64 (w / 4) ..), one loading weights, one issuing MMAs:
//   h1 = softplus(F W1^T + b1), h2 = softplus(h1 W2^T + b2), h3 = softplus(h2 W3^T + b3),
//   g = h3 . w4 + b4, dL/dg = (sigmoid(g) - y) / n,
//   dz3 = dL/dg w4 (1 - e^-h3), dz2 = (dz3 W3) (1 - e^-h2), dz1 = (dz2 W2) (1 - e^-h1)
// (softplus' through its output).  h3 and h2 stay in tensor memory in float32, h1 goes to the
// workspace in float32 and comes back to the thread that wrote it; bias and head gradients are
// float32 column sums.  What the weight gradients read (F, h1, h2 and the dz, bfloat16 row-major) is
// the kernel's only other traffic, 2.7 KB per point.  A second kernel forms all three weight
// gradients dz^T h from those rows (points along K, both operands MN-major), so no transposed copy is
// written.  Sixteen launches with float32 activations, transposed copies and column sums in memory
// took 172 us of device time for 16384 points and 199 us with their enqueueing; three with Adam now take
// 64 us, enqueueing included (46 + 18 + 4, overlapping at their ends; 70 us one after the other).
constexpr int kTrainStages = 4, kTrainEpi = 512, kTrainThreads = kTrainEpi + 64;
// shared memory: weight stages | A operand | head partials [4][128] | coordinates [6][128] | biases
// b1 b2 b3 and head weights w4 [4][256] | column sums of dz1, dz2, dz3 and of dL/dg h3 [4][256] |
// frequencies [32][3] | mbarriers, TMEM slot, flag
constexpr size_t kTrainOffA = (size_t)kTrainStages * kFwdStage;
constexpr size_t kTrainOffPart = kTrainOffA + kFwdA;
constexpr size_t kTrainOffFr = kTrainOffPart + 4 * kFwdTile * 4;
constexpr size_t kTrainOffPar = kTrainOffFr + 6 * kFwdTile * 4;
constexpr size_t kTrainOffSum = kTrainOffPar + 4 * kHid * 4;
constexpr size_t kTrainOffFreq = kTrainOffSum + 4 * kHid * 4;
constexpr size_t kTrainOffBar = kTrainOffFreq + 3 * kFreq * 4;
constexpr size_t kTrainSmem = kTrainOffBar + 128 + 1024;
static_assert(kTrainOffBar % 8 == 0, "mbarriers are 8-byte aligned");
static_assert(kTrainSmem <= 227 * 1024, "training shared memory above the per-CTA limit");

struct TrainMaps {
  CUtensorMap w[5];  // W1, W2, W3, W3^T, W2^T in the order a tile takes them
};

struct TrainRows {  // row-major outputs of n points
  __nv_bfloat16 *feat, *h1b, *h2b, *dz1, *dz2, *dz3;
  float *h1;
};

__device__ inline void tmem_store16(uint32_t taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16};" ::"r"(taddr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
      "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
      "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])),
      "r"(__float_as_uint(v[11])), "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])),
      "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])));
}

__device__ inline void tmem_get16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  tmem_load16(taddr, r);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// softplus' through the output h = softplus(z) >= 0: 1 - e^-h = 1 - 2^(-h log2 e), to 4e-7 (2.4e-7 of the
// power, 4.4e-8 of the exponent's rounding, 6e-8 of the difference's)
__device__ inline float softplus_gate(float h) { return 1.f - exp2_sfu(__fmul_rn(-kLog2E, h)); }

// Sum over the warp's 32 lanes (rows) of 16 columns: lane l returns the sum of column l / 2.  Each
// step halves the columns a lane keeps: 16 shuffles instead of five per column.
__device__ inline float column_sums16(const float (&v)[16], int lane) {
  float a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float keep = lane & 16 ? v[8 + i] : v[i], send = lane & 16 ? v[i] : v[8 + i];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int o = 8, w = 4; o >= 2; o >>= 1, w >>= 1)
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float keep = lane & o ? a[w + i] : a[i], send = lane & o ? a[i] : a[w + i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1);
}

__device__ inline void add_columns16(float *sums, const float (&v)[16], int lane) {
  const float t = column_sums16(v, lane);
  if (!(lane & 1)) atomicAdd(&sums[lane >> 1], t);
}

// 16 columns of a row in bfloat16: two core-matrix rows of the next A operand and 32 bytes of global
// memory (whole sectors).
__device__ inline void store_row16(__nv_bfloat16 *sA, int row, int c0, int K, __nv_bfloat16 *out, bool in,
                                   const float (&v)[16]) {
  uint32_t w[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
    w[q] = *reinterpret_cast<const uint32_t *>(&h);
  }
  if (sA != nullptr) {
    *reinterpret_cast<uint4 *>(sA + fwd_core(row, c0, K)) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4 *>(sA + fwd_core(row, c0 + 8, K)) = make_uint4(w[4], w[5], w[6], w[7]);
  }
  if (in) st_v8(out, w);
}

__global__ void __launch_bounds__(kTrainThreads, 1)
mlp_train_kernel(const __grid_constant__ TrainMaps maps, const float *p, const int32_t *freq, const double *x,
                 const float *label, int64_t n, TrainRows out, float *grad, float *loss, kups_status *status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                          ~uintptr_t(1023));
  __nv_bfloat16 *sA = reinterpret_cast<__nv_bfloat16 *>(smem + kTrainOffA);
  float *part = reinterpret_cast<float *>(smem + kTrainOffPart);
  float *fr = reinterpret_cast<float *>(smem + kTrainOffFr);
  float *spar = reinterpret_cast<float *>(smem + kTrainOffPar);
  float *sums = reinterpret_cast<float *>(smem + kTrainOffSum);
  int32_t *sfreq = reinterpret_cast<int32_t *>(smem + kTrainOffFreq);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kTrainOffBar);
  uint64_t *full = bars, *freed = bars + kTrainStages;
  uint64_t *ready = bars + 2 * kTrainStages, *acc = ready + 1, *meet = ready + 2, *drained = ready + 3;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(ready + 4);
  volatile int *stop = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == kTrainEpi / 32) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * kHid));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int k = 0; k < kTrainStages; ++k) {
      mbar_init(smem_u32(&full[k]), 1);
      mbar_init(smem_u32(&freed[k]), 1);
    }
    mbar_init(smem_u32(ready), kTrainEpi);
    mbar_init(smem_u32(acc), 1);
    mbar_init(smem_u32(meet), kTrainEpi);
    mbar_init(smem_u32(drained), 1);
    *stop = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("fence.proxy.async;" ::: "memory");
  for (int e = tid; e < 4 * kHid; e += kTrainThreads) {
    const int which = e / kHid;
    const int64_t off = which == 0 ? kOffB1 : which == 1 ? kOffB2 : which == 2 ? kOffB3 : kOffW4;
    spar[e] = p[off + e % kHid];
    sums[e] = 0.f;
  }
  for (int e = tid; e < 3 * kFreq; e += kTrainThreads) sfreq[e] = freq[e];
  __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;");  // tensor memory is held: the next grid cannot take it away
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const int64_t n_tiles = (n + kFwdTile - 1) / kFwdTile;
  if (warp < kTrainEpi / 32) {
    const int quarter = warp & 3, cq = warp >> 2, row = quarter * 32 + lane, cb = cq * 64;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);  // accumulator columns; h2 at + 256
    const float *w4 = spar + 3 * kHid;
    const float b4 = p[kOffB4], inv_n = 1.f / (float)n;
    float db4 = 0.f, ls = 0.f;
    uint32_t parity = 0u, met = 0u;
    auto wait = [&](uint64_t *bar, uint32_t &phase) {
      const bool done = __all_sync(0xffffffffu, mbar_wait_or_stop(smem_u32(bar), phase, stop));
      phase ^= 1u;
      return done;
    };
    auto meeting = [&]() {
      mbar_arrive(smem_u32(meet));
      return wait(meet, met);
    };
    auto next_layer = [&]() {  // A operand written and accumulator read: run the MMAs, wait for them
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(smem_u32(ready));
      const bool done = wait(acc, parity);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return done;
    };
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
      const int64_t row0 = tile * kFwdTile, pt = row0 + row;
      const bool in = pt < n;
      const float y = in ? label[pt] : 0.f;
      if (tid < kFwdTile) {  // coordinates reduced to [-0.5, 0.5) in float64, kept as float pairs
        for (int a = 0; a < 3; ++a) {
          const double f = row0 + tid < n ? x[3 * (row0 + tid) + a] : 0.0, red = f - rint(f);
          const float hi = (float)red;
          fr[a * kFwdTile + tid] = hi;
          fr[(3 + a) * kFwdTile + tid] = (float)(red - (double)hi);
        }
      }
      if (!meeting()) break;
      {  // 8 of the 32 phases of a row: 16 columns of the first A operand
        const float fh[3] = {fr[row], fr[kFwdTile + row], fr[2 * kFwdTile + row]};
        const float fl[3] = {fr[3 * kFwdTile + row], fr[4 * kFwdTile + row], fr[5 * kFwdTile + row]};
        float v[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[2 * j] = v[2 * j + 1] = 0.f;
          if (in) phase_sincos(sfreq + 3 * (8 * cq + j), fh, fl, v[2 * j], v[2 * j + 1]);
        }
        store_row16(sA, row, 16 * cq, kIn, out.feat + pt * kIn + 16 * cq, in, v);
      }
      if (!next_layer()) break;
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {  // h1: float32 to memory, bfloat16 to the A operand and to memory
        const int c0 = cb + 16 * s;
        float v[16];
        tmem_get16(lanes + c0, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = softplus_fast(v[i] + spar[c0 + i]);
        if (in) {
          uint32_t w[8];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(v[8 * q + e]);
            st_v8(out.h1 + pt * kHid + c0 + 8 * q, w);
          }
        }
        store_row16(sA, row, c0, kHid, out.h1b + pt * kHid + c0, in, v);
      }
      if (!next_layer()) break;
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {  // h2: float32 to the spare tensor memory
        const int c0 = cb + 16 * s;
        float v[16];
        tmem_get16(lanes + c0, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = softplus_fast(v[i] + spar[kHid + c0 + i]);
        tmem_store16(lanes + kHid + c0, v);
        store_row16(sA, row, c0, kHid, out.h2b + pt * kHid + c0, in, v);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      if (!next_layer()) break;
      // h3 in place of its accumulator, and g = h3 . w4 + b4: four interleaved sums per thread of 64
      // columns, then a tree, the same whatever the timing
      float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {
        const int c0 = cb + 16 * s;
        float v[16];
        tmem_get16(lanes + c0, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          v[i] = softplus_fast(v[i] + spar[2 * kHid + c0 + i]);
          dot[i & 3] = fmaf(v[i], w4[c0 + i], dot[i & 3]);
        }
        tmem_store16(lanes + c0, v);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      part[cq * kFwdTile + row] = (dot[0] + dot[1]) + (dot[2] + dot[3]);
      if (!meeting()) break;
      float dg = 0.f;
      if (in) {
        const float gg = ((part[row] + part[kFwdTile + row]) + (part[2 * kFwdTile + row] + part[3 * kFwdTile + row])) + b4;
        dg = (1.f / (1.f + expf(-gg)) - y) * inv_n;
        if (cq == 0) {
          ls += y > 0.5f ? softplus(-gg) : softplus(gg);
          db4 += dg;
        }
      }
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {  // dz3, and the head's gradient dL/dg h3
        const int c0 = cb + 16 * s;
        float h[16], v[16];
        tmem_get16(lanes + c0, h);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = dg * w4[c0 + i] * softplus_gate(h[i]);
        store_row16(sA, row, c0, kHid, out.dz3 + pt * kHid + c0, in, v);
        add_columns16(sums + 2 * kHid + c0, v, lane);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = dg * h[i];
        add_columns16(sums + 3 * kHid + c0, v, lane);
      }
      if (!next_layer()) break;
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {  // dz2
        const int c0 = cb + 16 * s;
        float h[16], v[16];
        tmem_get16(lanes + kHid + c0, h);
        tmem_get16(lanes + c0, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] *= softplus_gate(h[i]);
        store_row16(sA, row, c0, kHid, out.dz2 + pt * kHid + c0, in, v);
        add_columns16(sums + kHid + c0, v, lane);
      }
      float4 h1v[4];  // this thread's h1 of the first 16 columns, on its way during the MMAs
      const float4 *h1p = reinterpret_cast<const float4 *>(out.h1 + (in ? pt : 0) * kHid + cb);
#pragma unroll
      for (int q = 0; q < 4; ++q) h1v[q] = h1p[q];
      if (!next_layer()) break;
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {  // dz1 (no gradient into the features)
        const int c0 = cb + 16 * s;
        float v[16];
        const float h[16] = {h1v[0].x, h1v[0].y, h1v[0].z, h1v[0].w, h1v[1].x, h1v[1].y, h1v[1].z, h1v[1].w,
                             h1v[2].x, h1v[2].y, h1v[2].z, h1v[2].w, h1v[3].x, h1v[3].y, h1v[3].z, h1v[3].w};
        if (s < 3)
#pragma unroll
          for (int q = 0; q < 4; ++q) h1v[q] = h1p[4 * (s + 1) + q];
        tmem_get16(lanes + c0, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = in ? v[i] * softplus_gate(h[i]) : 0.f;
        store_row16(nullptr, row, c0, kHid, out.dz1 + pt * kHid + c0, in, v);
        add_columns16(sums + c0, v, lane);
      }
    }
    if (cq == 0) {
      db4 = warp_sum(db4);
      ls = warp_sum(ls);
      if (lane == 0) {
        atomicAdd(&grad[kOffB4], db4);
        if (loss != nullptr) atomicAdd(loss, ls * inv_n);
      }
    }
  } else if (warp == kTrainEpi / 32) {
    if (lane == 0) {  // weights, in the order of the MMAs
      int64_t q = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x)
        for (int layer = 0; layer < 5 && ok; ++layer)
          for (int c = 0; c < (layer == 0 ? kIn : kHid) / kFwdKc; ++c, ++q) {
            const int st = (int)(q % kTrainStages);
            if (q >= kTrainStages)
              ok = mbar_wait_or_stop(smem_u32(&freed[st]), (uint32_t)(q / kTrainStages - 1) & 1u, stop);
            if (!ok) break;
            mbar_expect_tx(smem_u32(&full[st]), kFwdStage);
            tma_load_2d(smem_u32(smem + st * kFwdStage), &maps.w[layer], c * kFwdKc, 0, smem_u32(&full[st]));
          }
      if (*stop)  // copies in flight land before the CTA ends
        for (int64_t k = q > kTrainStages ? q - kTrainStages : 0; k < q; ++k)
          mbar_wait(smem_u32(&full[k % kTrainStages]), (uint32_t)(k / kTrainStages) & 1u);
    }
  } else if (lane == 0) {
    const uint32_t idesc = make_idesc(kFwdTile, kHid), a0 = smem_u32(sA);
    int64_t q = 0;
    uint32_t parity = 0u;
    bool ok = true;
    for (int64_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x)
      for (int layer = 0; layer < 5 && ok; ++layer) {
        ok = mbar_wait_or_stop(smem_u32(ready), parity, stop);
        if (!ok) break;
        parity ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int K = layer == 0 ? kIn : kHid;
        for (int c = 0; c < K / kFwdKc; ++c, ++q) {
          const int st = (int)(q % kTrainStages);
          ok = mbar_wait_or_stop(smem_u32(&full[st]), (uint32_t)(q / kTrainStages) & 1u, stop);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t b0 = smem_u32(smem + st * kFwdStage);
          for (int ks = 0; ks < kFwdKc / 16; ++ks)
            mma_f16(tmem, make_sdesc(a0 + (c * 4 + ks) * 256, 128, (K / 8) * 128), make_sdesc_sw128(b0 + ks * 32),
                    idesc, c > 0 || ks > 0);
          mma_commit(smem_u32(&freed[st]));
        }
        if (ok) mma_commit(smem_u32(acc));
      }
    if (*stop) {  // MMAs in flight end before the tensor memory is freed
      mma_commit(smem_u32(drained));
      mbar_wait(smem_u32(drained), 0u);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && *stop) status_error(status, KUPS_ERR_UNSUPPORTED, blockIdx.x);
  for (int e = tid; e < 4 * kHid; e += kTrainThreads) {
    const int which = e / kHid;
    const int64_t off = which == 0 ? kOffB1 : which == 1 ? kOffB2 : which == 2 ? kOffB3 : kOffW4;
    atomicAdd(&grad[off + e % kHid], sums[e]);
  }
  if (warp == kTrainEpi / 32) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kHid));
  }
}

// Weight gradients dW[o, i] += sum over points of dz[p, o] h[p, i] of the three layers in one launch.
// Both operands are row-major in points (K), so they are MN-major to the tensor cores: a TMA box of 64
// columns x 64 points (128-byte rows, 128-byte swizzle) holds 64 of M or N for four K steps of 16, with
// 8-point groups 1024 bytes apart (stride offset) and the next 64 columns one box further (leading
// offset).  A CTA forms one 128 x 128 tile (128 x 64 for the first layer) over a share of the points
// and adds it to the gradient with 16-byte reductions; sixteen shares per tile fill the chip while the
// reductions stay at 8 MB (64 shares of 128 x 256 tiles moved 34 MB and took 39 us in three launches).
constexpr int kWgStages = 6, kWgThreads = 256;
constexpr uint32_t kWgBox = 64 * 64 * 2;  // 8 KB
constexpr size_t kWgSmem = (size_t)kWgStages * 4 * kWgBox + 1024 + 256;

struct GradMaps {
  CUtensorMap dz[3], h[3];  // layers 3, 2, 1
};

__device__ inline uint64_t make_sdesc_sw128_mn(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)(kWgBox >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__global__ void __launch_bounds__(kWgThreads, 1)
mlp_weight_grad_kernel(const __grid_constant__ GradMaps maps, int64_t n, int shares, int shares1, float *grad,
                       int aligned, kups_status *status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                          ~uintptr_t(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)kWgStages * 4 * kWgBox);
  uint64_t *freed = full + kWgStages, *done = freed + kWgStages;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
  int *ok_flag = reinterpret_cast<int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // unit: layers 3 and 2: 2 x 2 tiles x shares, then layer 1: 2 tiles x shares1
  int u = blockIdx.x, which, m0, n0, share, total;
  if (u < 8 * shares) {
    which = u / (4 * shares);
    u -= which * 4 * shares;
    share = u >> 2;
    m0 = ((u >> 1) & 1) * 128;
    n0 = (u & 1) * 128;
    total = shares;
  } else {
    u -= 8 * shares;
    which = 2;
    share = u >> 1;
    m0 = (u & 1) * 128;
    n0 = 0;
    total = shares1;
  }
  const int bn = which == 2 ? 64 : 128;
  const int64_t chunks = (n + 63) / 64;
  const int64_t c_begin = chunks * share / total, nc = chunks * (share + 1) / total - c_begin;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(128));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int k = 0; k < kWgStages; ++k) {
      mbar_init(smem_u32(&full[k]), 1);
      mbar_init(smem_u32(&freed[k]), 1);
    }
    mbar_init(smem_u32(done), 1);
    *ok_flag = 1;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  // the rows are whole when the training kernel has ended; every thread waits, so this grid ends after it
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("fence.proxy.async;" ::: "memory");
  __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  if (tid == 0) {
    const uint32_t idesc = make_idesc(128, bn) | (1u << 15) | (1u << 16);  // A and B MN-major
    const CUtensorMap *ma = &maps.dz[which], *mb = &maps.h[which];
    const uint32_t bytes = (2 + bn / 64) * kWgBox;
    auto box = [&](int st, int k) { return smem_u32(smem + ((size_t)st * 4 + k) * kWgBox); };
    auto load = [&](int64_t j) {
      const int st = (int)(j % kWgStages), p0 = (int)((c_begin + j) * 64);
      const uint32_t bar = smem_u32(&full[st]);
      mbar_expect_tx(bar, bytes);
      tma_load_2d(box(st, 0), ma, m0, p0, bar);
      tma_load_2d(box(st, 1), ma, m0 + 64, p0, bar);
      tma_load_2d(box(st, 2), mb, n0, p0, bar);
      if (bn == 128) tma_load_2d(box(st, 3), mb, n0 + 64, p0, bar);
    };
    bool ok = true;
    int64_t issued = 0, consumed = 0;
    for (; issued < kWgStages && issued < nc; ++issued) load(issued);
    for (int64_t i = 0; i < nc && ok; ++i) {
      const int st = (int)(i % kWgStages);
      ok = mbar_wait(smem_u32(&full[st]), (uint32_t)(i / kWgStages) & 1u);
      if (!ok) break;
      consumed = i + 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int ks = 0; ks < 4; ++ks)
        mma_f16(tmem, make_sdesc_sw128_mn(box(st, 0) + ks * 2048), make_sdesc_sw128_mn(box(st, 2) + ks * 2048), idesc,
                i > 0 || ks > 0);
      mma_commit(smem_u32(&freed[st]));
      // refill the stage of the chunk before this one, whose MMAs end first
      if (i > 0 && issued < nc) {
        const int64_t k = i - 1;
        ok = mbar_wait(smem_u32(&freed[k % kWgStages]), (uint32_t)(k / kWgStages) & 1u);
        if (ok) load(issued++);
      }
    }
    mma_commit(smem_u32(done));
    const bool mma_done = mbar_wait(smem_u32(done), 0u);
    if (!ok)  // loads still in flight land before the tile ends
      for (int64_t j = consumed; j < issued; ++j)
        mbar_wait(smem_u32(&full[j % kWgStages]), (uint32_t)(j / kWgStages) & 1u);
    *ok_flag = ok && mma_done ? 1 : 0;
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!*ok_flag) {
    if (tid == 0) status_error(status, KUPS_ERR_UNSUPPORTED, blockIdx.x);
  } else if (nc > 0) {
    const int quarter = warp & 3, half = warp >> 2, row = m0 + quarter * 32 + lane;
    const int width = which == 2 ? kIn : kHid;
    float *c = grad + (which == 0 ? kOffW3 : which == 1 ? kOffW2 : kOffW1) + (int64_t)row * width + n0;
    for (int c0 = half * (bn / 2); c0 < (half + 1) * (bn / 2); c0 += 16) {
      float v[16];
      tmem_get16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
      if (aligned) {
#pragma unroll
        for (int q = 0; q < 4; ++q) red_add_v4(c + c0 + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) atomicAdd(c + c0 + i, v[i]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128));
}

// Launches a kernel that may start while its predecessor on the stream still runs: it sets up (barriers,
// tensor memory), and every one of its threads waits (griddepcontrol.wait) before it reads or writes
// memory of others, so it also ends after all that came before.  A kernel lets its successor start only
// once it holds its tensor memory, which the successor could otherwise take while waiting for it.
// Training step of 16384 points: 63.7 us (69.8 with each kernel set up after the last had drained; 68.2
// with the weight gradients alone started early).  A captured launch keeps its full dependency.
template <typename... P, typename... A>
int32_t launch_early(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  KUPS_CUDA_TRY(cudaStreamIsCapturing(st, &capture));
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &early;
  cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
  KUPS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
  return KUPS_OK;
}

}  // namespace
}  // namespace kups

using namespace kups;

extern "C" int32_t kups_gemm_bf16(const void *a, int32_t a_bf16, int64_t sa_row, int64_t sa_col,
                                  const void *b, int32_t b_bf16, int64_t sb_row, int64_t sb_col,
                                  void *c, int32_t c_bf16, int64_t sc_row, int64_t sc_col, void *c2,
                                  int32_t c2_bf16, int64_t sc2_row, int64_t sc2_col, const float *bias,
                                  const float *gate, int32_t gate_kind, int64_t sg_row, int64_t sg_col,
                                  int32_t m, int32_t n, int32_t k, float alpha, float beta, int32_t act,
                                  int32_t split_k, kups_status *status, void *stream) {
  if (m <= 0 || n <= 0 || k <= 0 || act < 0 || act > 2 || gate_kind < 0 || gate_kind > 3 || split_k < 1 ||
      split_k > 65535)
    return KUPS_ERR_INVALID;
  // split-K accumulates into float32 C with atomics: no epilogue terms but alpha
  if (split_k > 1 && (c_bf16 || c2 || bias || gate_kind || act || beta != 1.f)) return KUPS_ERR_INVALID;
  GemmArgs g;
  g.a = a; g.b = b; g.c = c; g.c2 = c2; g.bias = bias; g.gate = gate;
  g.sar = sa_row; g.sac = sa_col; g.sbr = sb_row; g.sbc = sb_col; g.scr = sc_row; g.scc = sc_col;
  g.sc2r = sc2_row; g.sc2c = sc2_col; g.sgr = sg_row; g.sgc = sg_col;
  g.m = m; g.n = n; g.k = k; g.alpha = alpha; g.beta = beta; g.act = act;
  g.a_bf16 = a_bf16; g.b_bf16 = b_bf16; g.c_bf16 = c_bf16; g.c2_bf16 = c2_bf16; g.gate_kind = gate_kind;
  g.split_k = split_k;
  return dispatch_gemm(g, status, (cudaStream_t)stream);
}

extern "C" size_t kups_mlp_workspace_bytes(int64_t n_points) {
  return work_bytes(std::max<int64_t>(1, std::min<int64_t>(n_points, kChunk)));
}

extern "C" int32_t kups_mlp_init(const kups_mlp *net, uint64_t seed, void *stream) {
  if (net == nullptr) return KUPS_ERR_INVALID;
  init_kernel<<<blocks(kParams, 256), 256, 0, (cudaStream_t)stream>>>(
      net->param, (__nv_bfloat16 *)net->param_bf16, (__nv_bfloat16 *)net->param_bf16_t, net->grad, net->adam_m,
      net->adam_v, seed);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_mlp_fwd(const kups_mlp *net, const double *x, int64_t n, float *g, void *workspace,
                                size_t workspace_bytes, kups_status *status, void *stream) {
  if (net == nullptr || n < 0 || (n > 0 && (x == nullptr || g == nullptr))) return KUPS_ERR_INVALID;
  if (workspace_bytes < kups_mlp_workspace_bytes(n)) return KUPS_ERR_INVALID;
  const MlpWork w = carve(workspace, std::min<int64_t>(n, kChunk));
  return fused_forward(net, x, n, 0, g, w.weights, status, (cudaStream_t)stream);
}

extern "C" int32_t kups_mlp_nce_batch(const double *data, int64_t n_data, int32_t batch, uint64_t seed,
                                      uint64_t step, double *x, float *label, void *stream) {
  if (n_data <= 0 || batch <= 0 || (batch & 1)) return KUPS_ERR_INVALID;
  nce_batch_kernel<<<blocks(batch, 256), 256, 0, (cudaStream_t)stream>>>(data, n_data, batch, seed, step, x, label);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_mlp_bwd(const kups_mlp *net, const double *x, const float *label, int32_t n, float *loss,
                                void *workspace, size_t workspace_bytes, kups_status *status, void *stream) {
  if (net == nullptr || n <= 0 || n > kChunk) return KUPS_ERR_INVALID;
  if (workspace_bytes < kups_mlp_workspace_bytes(n)) return KUPS_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  const MlpWork w = carve(workspace, n);
  const __nv_bfloat16 *pb = (const __nv_bfloat16 *)net->param_bf16, *pbt = (const __nv_bfloat16 *)net->param_bf16_t;
  if ((((uintptr_t)pb | (uintptr_t)pbt) & 15) != 0) {  // TMA reads from 16-byte boundaries
    KUPS_CUDA_TRY(cudaMemcpyAsync(w.weights, pb, 2 * kParams, cudaMemcpyDeviceToDevice, st));
    __nv_bfloat16 *t = w.weights + kWeightCopy - 2 * kHid * kHid;
    KUPS_CUDA_TRY(cudaMemcpyAsync(t, pbt, 2 * 2 * kHid * kHid, cudaMemcpyDeviceToDevice, st));
    pb = w.weights;
    pbt = t;
  }
  TrainMaps tm;
  GradMaps gm;
  const __nv_bfloat16 *weights[5] = {pb + kOffW1, pb + kOffW2, pb + kOffW3, pbt + kHid * kHid, pbt};
  for (int k = 0; k < 5; ++k) {
    const int64_t cols = k == 0 ? kIn : kHid;
    if (!operand_map(&tm.w[k], weights[k], kHid, cols, cols, kHid)) return KUPS_ERR_CUDA;
  }
  const __nv_bfloat16 *dz[3] = {w.dz3, w.dz2, w.dz1}, *h[3] = {w.h2b, w.h1b, w.feat};
  for (int k = 0; k < 3; ++k) {
    const int64_t cols = k == 2 ? kIn : kHid;
    if (!operand_map(&gm.dz[k], dz[k], n, kHid, kHid, 64) || !operand_map(&gm.h[k], h[k], n, cols, cols, 64))
      return KUPS_ERR_CUDA;
  }
  KUPS_CUDA_TRY(cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem));
  KUPS_CUDA_TRY(cudaFuncSetAttribute(mlp_weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kWgSmem));
  const int64_t tiles = (n + kFwdTile - 1) / kFwdTile, chunks = (n + 63) / 64;
  const TrainRows rows{w.feat, w.h1b, w.h2b, w.dz1, w.dz2, w.dz3, w.h1};
  const int32_t rc = launch_early(mlp_train_kernel, (int)std::min<int64_t>(tiles, device_sm_count()), kTrainThreads,
                                  kTrainSmem, st, tm, net->param, net->freq, x, label, n, rows, net->grad, loss, status);
  if (rc != KUPS_OK) return rc;
  // shares of the points: 8 x 16 + 2 x 10 CTAs for a batch that gives each at least two chunks of 64
  const int shares = (int)std::min<int64_t>(16, std::max<int64_t>(1, chunks / 2));
  const int shares1 = (int)std::min<int64_t>(10, std::max<int64_t>(1, chunks / 2));
  const int aligned = ((uintptr_t)net->grad & 15) == 0;
  return launch_early(mlp_weight_grad_kernel, 8 * shares + 2 * shares1, kWgThreads, kWgSmem, st, gm, n, shares, shares1,
                      net->grad, aligned, status);
}

extern "C" int32_t kups_mlp_adam(const kups_mlp *net, int64_t t, float lr, float beta1, float beta2, float eps,
                                 void *stream) {
  if (net == nullptr || t < 1) return KUPS_ERR_INVALID;
  const float c1 = (float)(1.0 / (1.0 - pow((double)beta1, (double)t)));
  const float c2 = (float)(1.0 / (1.0 - pow((double)beta2, (double)t)));
  return launch_early(adam_kernel, (int)blocks(kParams, 256), 256, 0, (cudaStream_t)stream, net->param,
                      (__nv_bfloat16 *)net->param_bf16, (__nv_bfloat16 *)net->param_bf16_t, net->grad, net->adam_m,
                      net->adam_v, kParams, lr, beta1, beta2, eps, c1, c2);
}

extern "C" int32_t kups_mlp_grid_norm(const kups_mlp *net, int32_t grid, float temper, float floor_frac,
                                      float *node, double *cdf, void *workspace, size_t workspace_bytes,
                                      kups_status *status, void *stream) {
  if (net == nullptr || grid < 2 || grid > 256 || !(floor_frac > 0.f) || !(temper > 0.f)) return KUPS_ERR_INVALID;
  const int64_t n = (int64_t)grid * grid * grid;
  if (workspace_bytes < kups_mlp_workspace_bytes(n)) return KUPS_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  const MlpWork w = carve(workspace, std::min<int64_t>(n, kChunk));
  const int32_t rc = fused_forward(net, nullptr, n, grid, node, w.weights, status, st);
  if (rc) return rc;
  double *partial = w.partial;
  const int n_norm = (int)std::min<int64_t>(kNormBlocks, (n + kNormThreads - 1) / kNormThreads);
  grid_partials_kernel<<<n_norm, kNormThreads, 0, st>>>(node, n, temper, partial, status);
  grid_apply_kernel<<<4 * kNormBlocks, 256, 0, st>>>(node, n, temper, floor_frac, partial, n_norm);
  // three-pass scan
  const int n_blocks = (int)((n + kCdfPerBlock - 1) / kCdfPerBlock);
  double *totals = reinterpret_cast<double *>(w.h1);  // unused here: at least a double per 2048 nodes
  grid_cdf_local_kernel<<<n_blocks, kCdfThreads, 0, st>>>(node, grid, cdf, totals);
  grid_cdf_totals_kernel<<<1, kCdfThreads, 0, st>>>(totals, n_blocks, cdf, n);
  grid_cdf_offset_kernel<<<blocks(n, 256), 256, 0, st>>>(cdf, n, totals);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_proposal_sample(const float *node, const double *cdf, int32_t grid, int64_t n,
                                        uint64_t seed, double *f, double *log_q, void *stream) {
  if (grid < 2 || n < 0) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  proposal_sample_kernel<<<blocks(n, 128), 128, 0, (cudaStream_t)stream>>>(node, cdf, grid, n, seed, f, log_q);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_proposal_log_density(const float *node, const double *cdf, int32_t grid, const double *f,
                                             int64_t n, double *log_q, void *stream) {
  if (grid < 2 || n < 0) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  proposal_density_kernel<<<blocks(n, 128), 128, 0, (cudaStream_t)stream>>>(node, cdf, grid, f, n, log_q);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
