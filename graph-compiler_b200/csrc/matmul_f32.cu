// Exact-order f32 matmul: every output element accumulates k ascending with a separate multiply and add, the arithmetic
// of the reference's scalar loops (BrgemmNaive.cpp:46-99), so an f32 graph returns the reference's bits.
//
// Two instructions per term on the FMA pipe (no contraction, no K split: the order is part of the result), so the floor
// is 2 M N K / (128 lanes x SMs x clock).  A thread owns TM x TN outputs as packed pairs (f32x2 arithmetic: one issue
// slot for two terms, which leaves slots for the shared-memory loads); the next K slab travels from global memory to
// registers while the current one is computed, two shared buffers, one barrier per slab.
// Measured at 512 x 1024 x 1024: 151 us with 64 x 64 tiles, scalar arithmetic and one buffer; 50 us in this form.
#include "runtime.h"
#include "sm100_ptx.cuh"

namespace gcb {

namespace {

__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
// The product and the sum of a term are rounded separately: fma with a neutral third operand (a b + -0, and acc 1 + t).
// The neutral operands come from the host, because the assembler joins a packed mul and add into one fma (.rn or not) and
// sees through constants.
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
constexpr int kSlab = 16;   // K values per shared-memory buffer

// One operand's share of a K slab: T x kSlab values, PER per thread, held in registers between the global load and the
// shared store.  k_inner: consecutive memory runs along k (row-major A, transposed B), otherwise along the tile's rows.
// vec: rows of a whole number of 16 bytes - four consecutive values per load; otherwise single values.
template <int T, int THREADS> struct SlabLoader {
  static constexpr int kValues = T * kSlab / THREADS;
  static_assert(kValues == 4 || kValues == 2 || kValues == 1, "values per thread");
  float r[kValues];
  __device__ __forceinline__ void load(const float *base, int64_t ld, bool k_inner, bool vec, int row0, int rows, int k0, int K) {
    if (kValues == 4 && vec) {
      const int t = threadIdx.x;
      const int mn = k_inner ? t / (kSlab / 4) : (t % (T / 4)) * 4, k = k_inner ? (t % (kSlab / 4)) * 4 : t / (T / 4);
      const bool in = row0 + mn < rows && k0 + k < K;   // four values at a time: rows or K are a multiple of 4
      const float4 v = in ? *reinterpret_cast<const float4 *>(base + (k_inner ? int64_t(row0 + mn) * ld + k0 + k : int64_t(k0 + k) * ld + row0 + mn))
                          : make_float4(0.f, 0.f, 0.f, 0.f);
      r[0] = v.x; r[kValues > 1 ? 1 : 0] = v.y; r[kValues > 2 ? 2 : 0] = v.z; r[kValues > 3 ? 3 : 0] = v.w;
      return;
    }
#pragma unroll
    for (int i = 0; i < kValues; ++i) {
      const int e = threadIdx.x + i * THREADS;
      const int mn = k_inner ? e / kSlab : e % T, k = k_inner ? e % kSlab : e / T;
      const bool in = row0 + mn < rows && k0 + k < K;
      r[i] = in ? base[k_inner ? int64_t(row0 + mn) * ld + k0 + k : int64_t(k0 + k) * ld + row0 + mn] : 0.f;
    }
  }
  template <int P> __device__ __forceinline__ void store(float (*dst)[P], bool k_inner, bool vec) const {
    if (kValues == 4 && vec) {
      const int t = threadIdx.x;
      if (k_inner) {
        const int mn = t / (kSlab / 4), k = (t % (kSlab / 4)) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[k + i][mn] = r[kValues > i ? i : 0];
      } else {
        const int mn = (t % (T / 4)) * 4, k = t / (T / 4);
        *reinterpret_cast<float4 *>(&dst[k][mn]) = make_float4(r[0], r[kValues > 1 ? 1 : 0], r[kValues > 2 ? 2 : 0], r[kValues > 3 ? 3 : 0]);
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < kValues; ++i) {
      const int e = threadIdx.x + i * THREADS;
      if (k_inner) dst[e % kSlab][e / kSlab] = r[i];
      else         dst[e / T][e % T] = r[i];
    }
  }
};

template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
matmul_f32_kernel(const float *A, const float *B, const float *bias, float *out, int M, int N, int K, int ta, int tb, int relu,
                  int vec_a, int vec_b, int vec_o, uint64_t minus_zero, uint64_t one) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  __shared__ __align__(16) float As[2][kSlab][BM + 4];
  __shared__ __align__(16) float Bs[2][kSlab][BN + 4];
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  const int blocks_n = (N + BN - 1) / BN;
  const int m0 = int(blockIdx.x / unsigned(blocks_n)) * BM, n0 = int(blockIdx.x % unsigned(blocks_n)) * BN;
  const int64_t lda = ta ? M : K, ldb = tb ? K : N;
  SlabLoader<BM, THREADS> la;
  SlabLoader<BN, THREADS> lb;
  uint64_t acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;   // (+0, +0)
  pdl_launch_dependents();
  pdl_wait();   // operands may come from the kernel ahead in the stream
  la.load(A, lda, !ta, vec_a, m0, M, 0, K);
  lb.load(B, ldb, tb, vec_b, n0, N, 0, K);
  la.store(As[0], !ta, vec_a);
  lb.store(Bs[0], tb, vec_b);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += kSlab, buf ^= 1) {
    const bool more = k0 + kSlab < K;
    if (more) {
      la.load(A, lda, !ta, vec_a, m0, M, k0 + kSlab, K);
      lb.load(B, ldb, tb, vec_b, n0, N, k0 + kSlab, K);
    }
    auto term = [&](int kk) {
      float a[TM];
      uint64_t b[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) b[j] = *reinterpret_cast<const uint64_t *>(&Bs[buf][kk][tx * TN + 2 * j]);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const uint64_t aa = pack_f32x2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma_f32x2(acc[i][j], one, fma_f32x2(aa, b[j], minus_zero));
      }
    };
    // terms beyond K would add +0 (and turn a sum of -0 into +0), so the last slab stops at K
    if (K - k0 >= kSlab) {
#pragma unroll
      for (int kk = 0; kk < kSlab; ++kk) term(kk);
    } else {
      for (int kk = 0; kk < K - k0; ++kk) term(kk);
    }
    if (more) {
      la.store(As[buf ^ 1], !ta, vec_a);
      lb.store(Bs[buf ^ 1], tb, vec_b);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
    float v[TN];
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      const float2 f = unpack_f32x2(acc[i][j]);
      v[2 * j] = f.x;
      v[2 * j + 1] = f.y;
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (bias && n < N) v[j] = __fadd_rn(v[j], bias[n]);
      if (relu) v[j] = (v[j] != v[j]) ? v[j] : (v[j] > 0.f ? v[j] : 0.f);
    }
    float *dst = out + int64_t(m) * N + n0 + tx * TN;
    if (TN == 4 && vec_o && n0 + tx * TN + TN <= N) {
      *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[TN > 2 ? 2 : 0], v[TN > 3 ? 3 : 0]);
    } else {
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (n0 + tx * TN + j < N) dst[j] = v[j];
    }
  }
}

template <int BM, int BN, int TM, int TN>
void launch(const float *A, const float *B, const float *bias, float *out, int M, int N, int K, int ta, int tb, int relu,
            cudaStream_t stream) {
  auto al = [](const void *q, int64_t ld) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0 && ld % 4 == 0; };
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned((N + BN - 1) / BN) * unsigned((M + BM - 1) / BM));
  cfg.blockDim = dim3((BM / TM) * (BN / TN));
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  GCB_CUDA(cudaLaunchKernelEx(&cfg, matmul_f32_kernel<BM, BN, TM, TN>, A, B, bias, out, M, N, K, ta, tb, relu,
                              int(al(A, ta ? M : K)), int(al(B, tb ? K : N)), int(al(out, N)),
                              uint64_t(0x8000000080000000ull), uint64_t(0x3F8000003F800000ull)));
  count_launch();
}

} // namespace

void matmul_f32(const float *A, const float *B, const float *bias, float *out, int64_t M, int64_t N, int64_t K, int trans_a,
                int trans_b, int relu, cudaStream_t stream) {
  const int sms = device_state().sm_count;
  // Issue cycles a block spends per k: 64 for a 64 x 64 tile (FMA pipe), 22 for 32 x 32 and 14 for 16 x 32 (shared-memory
  // reads per term grow as the tile shrinks).  The cheapest sum over the waves wins: large tiles once they fill the SMs
  // (up to four small blocks share an SM's pipes, which is the same work again), small ones where they would not.
  auto cost = [&](int64_t bm, int64_t bn, double per_k) {
    const int64_t blocks = ((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    return double((blocks + sms - 1) / sms) * per_k;
  };
  const double c0 = cost(64, 64, 64), c1 = cost(32, 32, 22), c2 = cost(16, 32, 14);
  if (c0 <= c1 && c0 <= c2) launch<64, 64, 4, 4>(A, B, bias, out, int(M), int(N), int(K), trans_a, trans_b, relu, stream);
  else if (c1 <= c2)        launch<32, 32, 2, 2>(A, B, bias, out, int(M), int(N), int(K), trans_a, trans_b, relu, stream);
  else                      launch<16, 32, 1, 2>(A, B, bias, out, int(M), int(N), int(K), trans_a, trans_b, relu, stream);
}

} // namespace gcb
