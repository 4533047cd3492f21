// Exact-order f32 matmul: every output element accumulates k ascending with a separate multiply and add, the arithmetic
// of the reference's scalar loops (BrgemmNaive.cpp:46-99), so an f32 graph returns the reference's bits.
//
// Two instructions per term on the FMA pipe (no contraction, no K split: the order is part of the result), so the floor
// is 2 M N K / (128 lanes x SMs x clock): 37 us at 512 x 1024 x 1024 on the 128 blocks that 64 x 64 tiles give.  A thread owns
// TM x TN outputs; two K slabs are on their way from global memory in registers while one is computed from shared memory
// (two buffers, one barrier per slab), and the next term's operands are read while one is multiplied.  Packed f32x2
// arithmetic is no faster (the pipe is the limit, and a packed mul + add would be joined into an fma).
// Measured at 512 x 1024 x 1024: 151 us (one buffer, 16-wide slabs, no read-ahead) -> 64 us; slabs of 16: 68 us, 8 x 4
// outputs per thread: 71 us.
#include <algorithm>

#include "runtime.h"

namespace gcb {

namespace {

constexpr int kSlab = 32;   // K values per shared-memory buffer
constexpr int kDepth = 2;   // slabs in registers

// One operand's share of a K slab, held in registers between the global load and the shared store.  k_inner: consecutive
// memory runs along k (row-major A, transposed B), otherwise along the tile's rows.  vec: rows of whole 16-byte groups -
// four consecutive values per load; otherwise single values.
template <int T, int THREADS> struct SlabLoader {
  static constexpr int N = T * kSlab / THREADS;   // values per thread
  float r[N];
  __device__ __forceinline__ void load(const float *base, int64_t ld, bool k_inner, bool vec, int row0, int rows, int k0, int K) {
    if (N % 4 == 0 && vec) {
#pragma unroll
      for (int i = 0; i < N / 4; ++i) {
        const int t = threadIdx.x + i * THREADS;
        const int mn = k_inner ? t / (kSlab / 4) : (t % (T / 4)) * 4, k = k_inner ? (t % (kSlab / 4)) * 4 : t / (T / 4);
        const bool in = row0 + mn < rows && k0 + k < K;
        const float4 v = in ? *reinterpret_cast<const float4 *>(base + (k_inner ? int64_t(row0 + mn) * ld + k0 + k : int64_t(k0 + k) * ld + row0 + mn)) : make_float4(0.f, 0.f, 0.f, 0.f);
        r[(4 * i) % N] = v.x; r[(4 * i + 1) % N] = v.y; r[(4 * i + 2) % N] = v.z; r[(4 * i + 3) % N] = v.w;
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = threadIdx.x + i * THREADS;
      const int mn = k_inner ? e / kSlab : e % T, k = k_inner ? e % kSlab : e / T;
      const bool in = row0 + mn < rows && k0 + k < K;
      r[i] = in ? base[k_inner ? int64_t(row0 + mn) * ld + k0 + k : int64_t(k0 + k) * ld + row0 + mn] : 0.f;
    }
  }
  template <int P> __device__ __forceinline__ void store(float (*dst)[P], bool k_inner, bool vec) const {
    if (N % 4 == 0 && vec) {
#pragma unroll
      for (int i = 0; i < N / 4; ++i) {
        const int t = threadIdx.x + i * THREADS;
        if (k_inner) {
          const int mn = t / (kSlab / 4), k = (t % (kSlab / 4)) * 4;
#pragma unroll
          for (int j = 0; j < 4; ++j) dst[k + j][mn] = r[(4 * i + j) % N];
        } else {
          const int mn = (t % (T / 4)) * 4, k = t / (T / 4);
          *reinterpret_cast<float4 *>(&dst[k][mn]) = make_float4(r[(4 * i) % N], r[(4 * i + 1) % N], r[(4 * i + 2) % N], r[(4 * i + 3) % N]);
        }
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = threadIdx.x + i * THREADS;
      if (k_inner) dst[e % kSlab][e / kSlab] = r[i];
      else         dst[e / T][e % T] = r[i];
    }
  }
};
template <int TM> __device__ __forceinline__ void read_frag(const float *s, float (&r)[TM]) {
  if (TM % 4 == 0) {
#pragma unroll
    for (int i = 0; i < TM / 4; ++i) { const float4 v = reinterpret_cast<const float4 *>(s)[i]; r[(4*i)%TM] = v.x; r[(4*i+1)%TM] = v.y; r[(4*i+2)%TM] = v.z; r[(4*i+3)%TM] = v.w; }
  } else if (TM == 2) { const float2 v = *reinterpret_cast<const float2 *>(s); r[0] = v.x; r[1 % TM] = v.y; }
  else {
#pragma unroll
    for (int i = 0; i < TM; ++i) r[i] = s[i];
  }
}
template <int BM, int BN, int TM, int TN, int UNROLL>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
matmul_f32_kernel(const float *A, const float *B, const float *bias, float *out, int M, int N, int K, int ta, int tb, int relu, int vec_a, int vec_b, int vec_o) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  __shared__ __align__(16) float As[2][kSlab][BM + 4];
  __shared__ __align__(16) float Bs[2][kSlab][BN + 4];
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  const int blocks_n = (N + BN - 1) / BN;
  const int m0 = int(blockIdx.x / unsigned(blocks_n)) * BM, n0 = int(blockIdx.x % unsigned(blocks_n)) * BN;
  const int64_t lda = ta ? M : K, ldb = tb ? K : N;
  SlabLoader<BM, THREADS> la[kDepth];
  SlabLoader<BN, THREADS> lb[kDepth];
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int d = 0; d < kDepth; ++d) { la[d].load(A, lda, !ta, vec_a, m0, M, d * kSlab, K); lb[d].load(B, ldb, tb, vec_b, n0, N, d * kSlab, K); }
  la[0].store(As[0], !ta, vec_a); lb[0].store(Bs[0], tb, vec_b);
  __syncthreads();
  const int slabs = (K + kSlab - 1) / kSlab;
  for (int s0 = 0; s0 < slabs; s0 += kDepth) {
#pragma unroll
    for (int d = 0; d < kDepth; ++d) {
      const int slab = s0 + d;
      if (slab >= slabs) break;
      la[d].load(A, lda, !ta, vec_a, m0, M, (slab + kDepth) * kSlab, K);
      lb[d].load(B, ldb, tb, vec_b, n0, N, (slab + kDepth) * kSlab, K);
      const int buf = slab & 1;
      const int left = K - slab * kSlab;
      auto term = [&](const float (&a)[TM], const float (&b)[TN]) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(a[i], b[j]));
      };
      // terms beyond K would add +0 (and turn a sum of -0 into +0), so the last slab stops at K
      if (left >= kSlab) {
        float a[2][TM], b[2][TN];
        read_frag<TM>(&As[buf][0][ty * TM], a[0]); read_frag<TN>(&Bs[buf][0][tx * TN], b[0]);
#pragma unroll UNROLL
        for (int kk = 0; kk < kSlab; ++kk) {
          if (kk + 1 < kSlab) { read_frag<TM>(&As[buf][kk + 1][ty * TM], a[(kk + 1) & 1]); read_frag<TN>(&Bs[buf][kk + 1][tx * TN], b[(kk + 1) & 1]); }
          term(a[kk & 1], b[kk & 1]);
        }
      } else {
        for (int kk = 0; kk < left; ++kk) {
          float a[TM], b[TN];
          read_frag<TM>(&As[buf][kk][ty * TM], a); read_frag<TN>(&Bs[buf][kk][tx * TN], b);
          term(a, b);
        }
      }
      if (slab + 1 < slabs) {
        la[(d + 1) % kDepth].store(As[buf ^ 1], !ta, vec_a); lb[(d + 1) % kDepth].store(Bs[buf ^ 1], tb, vec_b);
        __syncthreads();
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
    float (&v)[TN] = acc[i];
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (bias && n < N) v[j] = __fadd_rn(v[j], bias[n]);
      if (relu) v[j] = (v[j] != v[j]) ? v[j] : (v[j] > 0.f ? v[j] : 0.f);
    }
    float *dst = out + int64_t(m) * N + n0 + tx * TN;
    if (TN == 4 && vec_o && n0 + tx * TN + TN <= N) {
      *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1 % TN], v[2 % TN], v[3 % TN]);
    } else {
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (n0 + tx * TN + j < N) dst[j] = v[j];
    }
  }
}

template <int BM, int BN, int TM, int TN, int UNROLL>
void launch(const float *A, const float *B, const float *bias, float *out, int M, int N, int K, int ta, int tb, int relu,
            cudaStream_t stream) {
  auto al = [](const void *q, int64_t ld) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0 && ld % 4 == 0; };
  // An ordinary launch: as a dependent one its blocks would be placed while the kernel ahead still holds most SMs, several
  // to each idle SM, and stay there (512 x 1024 x 1024 back to back: 103 us instead of 64).
  const unsigned blocks = unsigned((N + BN - 1) / BN) * unsigned((M + BM - 1) / BM);
  matmul_f32_kernel<BM, BN, TM, TN, UNROLL><<<blocks, (BM / TM) * (BN / TN), 0, stream>>>(
      A, B, bias, out, M, N, K, ta, tb, relu, int(al(A, ta ? M : K)), int(al(B, tb ? K : N)), int(al(out, N)));
  GCB_CUDA(cudaGetLastError());
  count_launch();
}

} // namespace

void matmul_f32(const float *A, const float *B, const float *bias, float *out, int64_t M, int64_t N, int64_t K, int trans_a,
                int trans_b, int relu, cudaStream_t stream) {
  const int sms = device_state().sm_count;
  // Time of a tile alone on its SM and of one among many, in us per 1024 k, measured: 64 x 64 60 / 53, 32 x 32 29 / 21,
  // 16 x 16 23 / 8.2.  Large tiles once there are enough of them to occupy the SMs, small ones where there are not.
  auto cost = [&](int64_t tile, double alone, double among) {
    return std::max(alone, double((M + tile - 1) / tile) * double((N + tile - 1) / tile) / sms * among);
  };
  const double c0 = cost(64, 60, 53), c1 = cost(32, 29, 21), c2 = cost(16, 23, 8.2);
  if (c0 <= c1 && c0 <= c2) launch<64, 64, 4, 4, 4>(A, B, bias, out, int(M), int(N), int(K), trans_a, trans_b, relu, stream);
  else if (c1 <= c2)        launch<32, 32, 2, 2, 8>(A, B, bias, out, int(M), int(N), int(K), trans_a, trans_b, relu, stream);
  else                      launch<16, 16, 2, 1, 4>(A, B, bias, out, int(M), int(N), int(K), trans_a, trans_b, relu, stream);
}

} // namespace gcb
