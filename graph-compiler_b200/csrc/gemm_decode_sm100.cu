// Matmuls of a few rows (M <= 64) against a large weight matrix: the weights take the MMA M side, 128 output columns per
// tile, and are streamed through the SMs once.
//
// Bound by HBM: 2 N K bytes of weights for 2 M N K operations.  What a launch costs beyond that stream is fixed time
// (launch, set-up, the first loads' latency, the tail) and SMs without work because there are too few tiles, so
//  * a tile's K range is shared by a cluster of 1 to 8 CTAs, which exchange their f32 partial sums through distributed
//    shared memory: each finishes its share of the rows, adding the parts in K order.  No workspace, no second launch.
//  * a CTA has an SM to itself and a ring of two-K-block stages (32 KB of weights and their activations; 192 KB under way
//    with 16 rows): a stage's hand-shake takes 0.3 us whatever it holds, so one K block a stage held a CTA to 63 GB/s, and
//    two CTAs to an SM made the SMs with two of them the last to finish.  Measured against that form: 16 x 28672 x 8192
//    91 -> 76 us (6.2 TB/s), 64 x 28672 x 8192 118 -> 82, 32 x 4096 x 11008 24.8 -> 21, 16 x 1024 x 8192 14.3 -> 8.9 us.
//  * where the caller knows that nothing in flight writes the weights, the ring is filled with them while the kernel ahead
//    ends.
// A variant that shared the K blocks of all tiles out evenly over the SMs (partial sums in global memory, finished by the
// last warp to arrive) took 95 us instead of 14 at 32 x 4096 x 4096: one warp per tile cannot hide the latency of the sums.
#include "gemm_decode.h"

#include <mutex>

#include "sm100_ptx.cuh"

namespace gcb {

namespace {

constexpr int kDecThreads = 224;
constexpr int kDecMaxStages = 12;
constexpr size_t kDecSmem = 226 * 1024;   // all but 1 KB of what a CTA may have

struct DecBars {
  uint64_t full[kDecMaxStages], empty[kDecMaxStages], tmem_full[2], tmem_empty[2];
  uint64_t parts_in, parts_out;   // every CTA's partial sums lie in shared memory / have been read by everyone
  uint32_t tmem_base, abort_flag;
};

// Finishes one element of the result: f32 (or s32) sum -> output type with its post-ops.
template <int KIND>
__device__ __forceinline__ void finish(const DecodeParams &p, uint32_t acc, int orow, int ocol, uint32_t bias_bits, float bias_f, float scale_f,
                                       int32_t comp_i) {
  const size_t idx = size_t(orow) * size_t(p.ld_out) + size_t(ocol);
  if (p.out_kind == OUT_BF16) {
    uint32_t y = f32_to_bf16_bits(__uint_as_float(acc));
    if (p.bias_kind == BIAS_BF16) y = f32_to_bf16_bits(__fadd_rn(bf16_bits_to_f32(y), bf16_bits_to_f32(bias_bits)));
    if (p.relu) {
      const float f = bf16_bits_to_f32(y);
      y = (f != f) ? y : (f > 0.f ? y : 0u);
    }
    reinterpret_cast<uint16_t *>(p.out)[idx] = uint16_t(y);
  } else if (p.out_kind == OUT_DEQUANT_F32) {
    float f = __fmul_rn(float(int32_t(acc) - comp_i), scale_f);
    if (p.bias_kind == BIAS_F32) f = __fadd_rn(f, bias_f);
    if (p.relu) f = (f != f) ? f : (f > 0.f ? f : 0.f);
    reinterpret_cast<float *>(p.out)[idx] = f;
    if (p.acc_dump) p.acc_dump[size_t(orow) * size_t(p.ld_dump) + size_t(ocol)] = int32_t(acc);
  } else if (p.out_kind == OUT_F32) {
    float f = __uint_as_float(acc);
    if (p.bias_kind == BIAS_F32) f = __fadd_rn(f, bias_f);
    if (p.relu) f = (f != f) ? f : (f > 0.f ? f : 0.f);
    reinterpret_cast<float *>(p.out)[idx] = f;
  } else {
    reinterpret_cast<uint32_t *>(p.out)[idx] = acc;
  }
}

template <int KIND>
__global__ void __launch_bounds__(kDecThreads, 1)
gemm_decode_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ DecodeParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);
  const uint32_t stage_bytes = p.w.bytes + p.x.bytes;
  float *parts = reinterpret_cast<float *>(smem + size_t(p.stages) * stage_bytes);   // [row][128 columns], clusters only
  DecBars *bars = reinterpret_cast<DecBars *>(smem + size_t(p.stages) * stage_bytes + p.parts_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int stages = p.stages, kbs = p.k_blocks;
  const int split = p.split, rank = split > 1 ? int(cluster_ctarank()) : 0;
  const int kpb = p.kpb, per = ((kbs + split - 1) / split + kpb - 1) / kpb * kpb, kb0 = min(kbs, rank * per), kb1 = min(kbs, kb0 + per);   // this CTA's K blocks
  const int first = int(blockIdx.x) / split, stride = int(gridDim.x) / split;                         // its cluster's tiles

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&bars->full[s]), 2);   // one expect-tx arrive per producer warp
      mbar_init(smem_u32(&bars->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bars->tmem_full[b]), 1);
      mbar_init(smem_u32(&bars->tmem_empty[b]), 4);
    }
    mbar_init(smem_u32(&bars->parts_in), uint32_t(4 * split));
    mbar_init(smem_u32(&bars->parts_out), uint32_t(4 * split));
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&bars->tmem_base), p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  if (split > 1) cluster_sync_all();   // every CTA's barriers are there before another one signals them
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(&bars->tmem_base);

  if (warp == 0 || warp == 6) {
    // ------------------------------------------------------------------ TMA producers: weights (0), activations (6)
    const bool is_w = warp == 0;
    const CUtensorMap *tm = is_w ? &tmW : &tmX;
    const OperandGeom &g = is_w ? p.w : p.x;
    const uint32_t my_bytes = g.bytes, my_off = is_w ? 0u : p.w.bytes, boxes = g.boxes, box_bytes = g.box_bytes, box_mn = g.box_mn;
    const bool mn = g.mn_major != 0, one = g.one_load != 0, k3d = g.k3d != 0;
    // Weights may be fetched before the kernel ahead has finished when nothing in flight writes them; everything else
    // (activations, results, and weights of unknown origin) waits for it.
    if (!(is_w && p.early_weights)) {
      if (is_w && elect_one()) {   // the first ring of weights at least comes to L2 meanwhile
        for (int kb = kb0; kb < min(kb1, kb0 + stages * kpb); kb += kpb) {
          if (!mn && k3d) tma_prefetch_3d(tm, 0, first * 128, kb);
          else if (!mn)
            for (uint32_t i = 0; i < boxes; ++i) tma_prefetch_2d(tm, (kb + int(i)) * p.bk_elems, first * 128);
          else if (one) tma_prefetch_3d(tm, 0, kb * p.bk_elems, first * 128 / int(box_mn));
          else
            for (uint32_t i = 0; i < boxes; ++i) tma_prefetch_2d(tm, first * 128 + int(i * box_mn), kb * p.bk_elems);
        }
      }
      __syncwarp();
      pdl_wait();
    }
    bool behind = !(is_w && p.early_weights);
    if (!is_w) pdl_launch_dependents();   // behind the wait: whoever starts after this finds all work before the kernel ahead done
    int s = 0, err = 0;
    uint32_t ph = 0, issued = 0;
    for (int t = first; t < p.tiles && !err; t += stride) {
      const int mn_off = is_w ? t * 128 : 0;
      const int grp = mn_off / int(box_mn ? box_mn : 1u);
      for (int kb = kb0; kb < kb1; kb += kpb, ++issued) {
        if (!behind && issued == uint32_t(stages)) {   // the ring is full: its first release is behind the kernel ahead
          pdl_wait();
          behind = true;
        }
        if (!mbar_wait_warp(smem_u32(&bars->empty[s]), ph ^ 1u)) { err = ERR_WAIT_EMPTY; break; }
        if (elect_one()) {
          const uint32_t full = smem_u32(&bars->full[s]);
          const uint32_t dst = base + uint32_t(s) * stage_bytes + my_off;
          const int k_off = kb * p.bk_elems;
          mbar_expect_tx(full, my_bytes);
          if (!mn && k3d) tma_load_3d(dst, tm, full, 0, mn_off, kb);
          else if (!mn)
            for (uint32_t i = 0; i < boxes; ++i) tma_load_2d(dst + i * box_bytes, tm, full, k_off + int(i) * p.bk_elems, mn_off);
          else if (one) tma_load_3d(dst, tm, full, 0, k_off, grp);
          else
            for (uint32_t i = 0; i < boxes; ++i) tma_load_2d(dst + i * box_bytes, tm, full, mn_off + int(i * box_mn), k_off);
        }
        __syncwarp();
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
    }
    if (err && lane == 0) { atomicExch(p.error, err); bars->abort_flag = 1; }
    // every copy issued here must have landed before the CTA may exit; in the normal path the MMA warp has consumed them
    if (__any_sync(0xFFFFFFFFu, *reinterpret_cast<volatile uint32_t *>(&bars->abort_flag) != 0)) {
      const uint32_t n = issued < uint32_t(stages) ? issued : uint32_t(stages);
      for (uint32_t j = 0; j < n; ++j) {
        const uint32_t i2 = issued - 1 - j;
        if (!mbar_wait_warp(smem_u32(&bars->full[i2 % uint32_t(stages)]), (i2 / uint32_t(stages)) & 1u) && lane == 0) atomicExch(p.error, ERR_WAIT_DRAIN);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (see elect_one)
    const uint64_t wd = umma_smem_desc(base, p.w.lbo, p.w.sbo), xd = umma_smem_desc(base + p.w.bytes, p.x.lbo, p.x.sbo);
    const uint32_t w_hi = uint32_t(wd >> 32), x_hi = uint32_t(xd >> 32), w_lo0 = uint32_t(wd), x_lo0 = uint32_t(xd);
    const uint32_t step = stage_bytes >> 4, w_k = p.w.kstep >> 4, x_k = p.x.kstep >> 4, idesc = p.idesc;
    const uint32_t w_sub = p.w.sub_step >> 4, x_sub = p.x.sub_step >> 4;   // next K block of a stage
    auto desc = [](uint32_t lo, uint32_t hi) { return (uint64_t(hi) << 32) | uint64_t(lo); };
    int s = 0, err = 0;
    uint32_t ph = 0, seg = 0;
    pdl_wait();   // so that no bounded wait runs while the kernel ahead does
    for (int t = first; t < p.tiles && !err; t += stride, ++seg) {
      const uint32_t acc = seg & 1u, acc_ph = (seg >> 1) & 1u;
      if (!mbar_wait_warp(smem_u32(&bars->tmem_empty[acc]), acc_ph ^ 1u)) { err = ERR_WAIT_TMEM_EMPTY; break; }
      tc_fence_after();
      const uint32_t d = tmem_base + acc * uint32_t(p.BN);
      for (int kb = kb0; kb < kb1; kb += kpb) {
        if (!mbar_wait_warp(smem_u32(&bars->full[s]), ph)) { err = ERR_WAIT_FULL; break; }
        tc_fence_after();
        uint32_t wl = w_lo0 + uint32_t(s) * step, xl = x_lo0 + uint32_t(s) * step;
        if (elect_one()) {
#pragma unroll 1
          for (int i = 0; i < kpb; ++i, wl += w_sub, xl += x_sub) {
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
              if (KIND == 0) umma_f16(d, desc(wl + k * w_k, w_hi), desc(xl + k * x_k, x_hi), idesc, (kb + i > kb0 || k > 0) ? 1u : 0u);
              else           umma_i8(d, desc(wl + k * w_k, w_hi), desc(xl + k * x_k, x_hi), idesc, (kb + i > kb0 || k > 0) ? 1u : 0u);
            }
          }
          umma_commit(smem_u32(&bars->empty[s]));
          if (kb + kpb >= kb1) umma_commit(smem_u32(&bars->tmem_full[acc]));
        }
        __syncwarp();
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
    }
    if (err && lane == 0) { atomicExch(p.error, err); bars->abort_flag = 1; }
  } else {
    // ------------------------------------------------------------------ epilogue: this warp's 32 output columns of a tile
    const int q = warp & 3;
    pdl_wait();
    uint32_t seg = 0;
    for (int t = first; t < p.tiles; t += stride, ++seg) {
      const uint32_t acc = seg & 1u, acc_ph = (seg >> 1) & 1u;
      const int ocol = t * 128 + q * 32 + lane;
      const bool col_in = ocol < p.out_cols;
      uint32_t bias_bits = 0;
      float bias_f = 0.f, scale_f = 1.f;
      int32_t comp_i = 0;
      if (col_in) {
        if (p.bias_kind == BIAS_BF16) bias_bits = reinterpret_cast<const uint16_t *>(p.bias)[ocol];
        if (p.bias_kind == BIAS_F32) bias_f = reinterpret_cast<const float *>(p.bias)[ocol];
        if (p.out_kind == OUT_DEQUANT_F32) { scale_f = p.scale[ocol]; comp_i = p.comp ? p.comp[ocol] : 0; }
      }
      if (!mbar_wait_warp(smem_u32(&bars->tmem_full[acc]), acc_ph)) {
        if (lane == 0) atomicExch(p.error, ERR_WAIT_TMEM_FULL);
        break;
      }
      tc_fence_after();
      const uint32_t ta = tmem_base + acc * uint32_t(p.BN) + (uint32_t(q * 32) << 16);
      // the parts of the tile before have been read by every CTA of the cluster
      if (split > 1 && seg > 0 && !mbar_wait_warp_cluster(smem_u32(&bars->parts_out), (seg - 1) & 1u)) {
        if (lane == 0) atomicExch(p.error, ERR_WAIT_PARTS);
        break;
      }
      for (int c0 = 0; c0 < p.out_rows; c0 += 16) {
        uint32_t v[16];
        tmem_ld_x16(ta + c0, v);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int orow = c0 + j;
          if (orow >= p.out_rows) continue;
          if (split > 1) parts[orow * 128 + q * 32 + lane] = __uint_as_float(v[j]);
          else if (col_in) finish<KIND>(p, v[j], orow, ocol, bias_bits, bias_f, scale_f, comp_i);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars->tmem_empty[acc]));
      if (split == 1) continue;
      // hand the part to everyone, wait for everyone's, finish rows rank, rank + split, ... of these 32 columns
      if (lane < split) mbar_arrive_cluster(mapa_shared(smem_u32(&bars->parts_in), uint32_t(lane)));
      if (!mbar_wait_warp_cluster(smem_u32(&bars->parts_in), seg & 1u)) {
        if (lane == 0) atomicExch(p.error, ERR_WAIT_PARTS);
        break;
      }
      const uint32_t mine = smem_u32(parts + q * 32 + lane);
      // four rows' parts are on their way at a time: fetched row by row, 32 rows took 4 us
      for (int row0 = rank; row0 < p.out_rows; row0 += 4 * split) {
        uint32_t w[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 8; ++c)
            if (c < split && row0 + i * split < p.out_rows) w[i][c] = ld_shared_cluster(mapa_shared(mine + uint32_t(row0 + i * split) * 512u, uint32_t(c)));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int orow = row0 + i * split;
          if (orow >= p.out_rows) break;
          uint32_t sum = w[i][0];
#pragma unroll
          for (int c = 1; c < 8; ++c)
            if (c < split) sum = KIND == 0 ? __float_as_uint(__fadd_rn(__uint_as_float(sum), __uint_as_float(w[i][c]))) : sum + w[i][c];
          if (col_in) finish<KIND>(p, sum, orow, ocol, bias_bits, bias_f, scale_f, comp_i);
        }
      }
      __syncwarp();
      if (lane < split) mbar_arrive_cluster(mapa_shared(smem_u32(&bars->parts_out), uint32_t(lane)));
    }
  }

  // ---------------------------------------------------------------------- tear-down
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
  if (split > 1) cluster_sync_all();   // no CTA leaves while another may read its parts or signal it
}

} // namespace

int decode_stages(const DecodeParams &p) {
  const size_t stage = size_t(p.w.bytes) + p.x.bytes;
  return int(std::min<size_t>(kDecMaxStages, (kDecSmem - 1024 - p.parts_bytes - sizeof(DecBars)) / stage));
}

static size_t decode_smem(const DecodeParams &p) {
  return 1024 + size_t(p.stages) * (size_t(p.w.bytes) + p.x.bytes) + p.parts_bytes + sizeof(DecBars);
}

static void configure(cudaLaunchConfig_t &cfg, cudaLaunchAttribute (&at)[2], int grid, int split, size_t smem, cudaStream_t stream) {
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = unsigned(split);
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = split > 1 ? 2 : 1;
}

// Once per device: shared memory beyond the default, and how many clusters of each size run at the same time.
template <int KIND> static const int *decode_device(int dev) {
  struct State {
    std::once_flag once;
    int at_once[9];
  };
  static State states[64];
  State &st = states[dev & 63];
  std::call_once(st.once, [&] {
    cudaFuncSetAttribute(gemm_decode_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kDecSmem));
    for (int split = 1; split <= 8; ++split) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[2];
      configure(cfg, at, split, split, kDecSmem, nullptr);
      cfg.numAttrs = 2;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_decode_kernel<KIND>, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
      st.at_once[split] = n;
    }
  });
  return st.at_once;
}

int decode_clusters_at_once(bool int8, int device, int split) { return (int8 ? decode_device<1>(device) : decode_device<0>(device))[split]; }

template <int KIND>
cudaError_t launch_gemm_decode(const CUtensorMap &tmW, const CUtensorMap &tmX, const DecodeParams &p, int grid, int device, cudaStream_t stream) {
  decode_device<KIND>(device);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  configure(cfg, at, grid, p.split, decode_smem(p), stream);
  return cudaLaunchKernelEx(&cfg, gemm_decode_kernel<KIND>, tmW, tmX, p);
}

template cudaError_t launch_gemm_decode<0>(const CUtensorMap &, const CUtensorMap &, const DecodeParams &, int, int, cudaStream_t);
template cudaError_t launch_gemm_decode<1>(const CUtensorMap &, const CUtensorMap &, const DecodeParams &, int, int, cudaStream_t);

} // namespace gcb
