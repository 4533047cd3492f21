// bf16 matmuls whose operands the copy engine cannot address.
//
// cp.async.bulk.tensor needs a 16-byte aligned base and row pitch; a row of 1001 bf16 values has neither.  One pass copies
// such an operand to rows padded to whole 128-byte groups (padding zero, so that it may take part in a product) and the
// tensor-core kernels run on the copy.  The pass is bound by memory (2 bytes read, 2 written per element); an exact-order
// loop on the FMA pipes took 28 times as long as both together at 1000 x 1001 x 2048.
#include <algorithm>
#include <mutex>

#include "runtime.h"
#include "sm100_ptx.cuh"

namespace gcb {

namespace {

// One thread writes 16 bytes (eight elements).  The source address has no alignment beyond two bytes: five aligned words
// are loaded and shifted by half a word where needed; words that lie partly outside the matrix are put together from
// single elements.
__global__ void __launch_bounds__(256) pack_rows_kernel(const uint16_t *src, uint4 *dst, long long rows, int cols, int chunks) {
  pdl_wait();
  pdl_launch_dependents();
  const long long total = rows * chunks;
  const uintptr_t first = reinterpret_cast<uintptr_t>(src), last = reinterpret_cast<uintptr_t>(src + rows * cols);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const long long row = i / chunks;
    const int col = int(i - row * chunks) * 8;
    const uint16_t *s = src + row * cols + col;
    uint32_t w[4] = {0, 0, 0, 0};
    const int n = min(8, cols - col);
    const uintptr_t at = reinterpret_cast<uintptr_t>(s) & ~uintptr_t(3);
    if (n == 8 && at >= first && at + 20 <= last) {
      const uint32_t *q = reinterpret_cast<const uint32_t *>(at);
      uint32_t v[5];
#pragma unroll
      for (int e = 0; e < 5; ++e) v[e] = __ldg(q + e);
      const uint32_t shift = (reinterpret_cast<uintptr_t>(s) & 2) * 8;
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = __funnelshift_r(v[e], v[e + 1], shift);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (e < n) w[e >> 1] |= uint32_t(s[e]) << ((e & 1) * 16);
    }
    dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

struct Operand {
  const void *ptr;
  int64_t rows, cols;
  bool pack;
  int64_t pitch() const { return (cols + 63) / 64 * 64; }
  size_t bytes() const { return pack ? size_t(rows) * size_t(pitch()) * 2 : 0; }
};
void operands(const MatmulArgs &a, Operand (&o)[2]) {
  o[0] = {a.A, a.trans_a ? a.K : a.M, a.trans_a ? a.M : a.K, false};
  o[1] = {a.B, a.trans_b ? a.N : a.K, a.trans_b ? a.K : a.N, false};
  for (Operand &x : o) x.pack = !tma_compatible(x.ptr, x.cols, 2);
}

// Stream-ordered memory for the copies of the direct launchers.  Up to kKeep bytes stay with the pool between calls
// (more is given back to the device at the next synchronisation), so that a repeated call does not map memory again.
constexpr uint64_t kKeep = uint64_t(256) << 20;
cudaMemPool_t pack_pool() {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  GCB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(mu);
  cudaMemPool_t &p = pools[dev & 63];
  if (!p) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    GCB_CUDA(cudaMemPoolCreate(&p, &props));
    uint64_t keep = kKeep;
    GCB_CUDA(cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep));
  }
  return p;
}

} // namespace

size_t matmul_pack_bytes(const MatmulArgs &a) {
  Operand o[2];
  operands(a, o);
  return o[0].bytes() + o[1].bytes();
}

void matmul_bf16_packed(const MatmulArgs &a, void *pack, cudaStream_t stream) {
  DeviceState &dev = device_state();
  Operand o[2];
  operands(a, o);
  MatmulArgs m = a;
  // pack_rows lets the matmul start while it still writes: a packed operand is not complete until its wait is over
  m.early_inputs = 0;
  if (o[1].pack) m.early_weights = 0;
  uint8_t *at = static_cast<uint8_t *>(pack);
  for (int i = 0; i < 2; ++i) {
    if (!o[i].pack) continue;
    const int chunks = int(o[i].pitch() / 8);
    const long long total = o[i].rows * (long long)chunks;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(std::min<long long>((total + 255) / 256, (long long)dev.sm_count * 8)));
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GCB_CUDA(cudaLaunchKernelEx(&cfg, pack_rows_kernel, static_cast<const uint16_t *>(o[i].ptr), reinterpret_cast<uint4 *>(at),
                                (long long)o[i].rows, int(o[i].cols), chunks));
    count_launch();
    (i == 0 ? m.A : m.B) = at;
    (i == 0 ? m.lda : m.ldb) = o[i].pitch();
    at += o[i].bytes();
  }
  matmul_tc(m, stream);
}

void matmul_bf16_any_layout(const MatmulArgs &a, cudaStream_t stream) {
  const size_t bytes = matmul_pack_bytes(a);
  if (!bytes) {
    matmul_tc(a, stream);
    return;
  }
  void *pack = nullptr;
  GCB_CUDA(cudaMallocFromPoolAsync(&pack, bytes, pack_pool(), stream));
  try {
    matmul_bf16_packed(a, pack, stream);
  } catch (...) {
    cudaFreeAsync(pack, stream);
    throw;
  }
  GCB_CUDA(cudaFreeAsync(pack, stream));
}

} // namespace gcb
