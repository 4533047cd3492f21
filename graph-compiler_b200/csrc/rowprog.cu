#include "rowprog.h"

#include <algorithm>
#include <mutex>
#include <stdexcept>
#include <unordered_map>

#include "elementwise.cuh"
#include "runtime.h"

namespace gcb {

// ----------------------------------------------------------------------------- kernel
namespace {

__device__ __forceinline__ void load8(const void *p, long long i, int dt, float (&x)[kProgVec]) {
  if (dt == 0) {
    const float4 *q = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p) + i);
    const float4 a = q[0], b = q[1];
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    return;
  }
  const uint4 q = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(p) + i);
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const uint32_t h = (e & 1) ? w[e >> 1] >> 16 : w[e >> 1] & 0xFFFFu;
    x[e] = dt == 1 ? bf16_bits_to_f32(h) : __half2float(__ushort_as_half((unsigned short)h));
  }
}
__device__ __forceinline__ void store8(void *p, long long i, int dt, const float (&x)[kProgVec]) {
  if (dt == 0) {
    float4 *q = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p) + i);
    q[0] = make_float4(x[0], x[1], x[2], x[3]);
    q[1] = make_float4(x[4], x[5], x[6], x[7]);
    return;
  }
  uint32_t w[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t lo = dt == 1 ? f32_to_bf16_bits(x[2 * e]) : uint32_t(__half_as_ushort(__float2half_rn(x[2 * e])));
    const uint32_t hi = dt == 1 ? f32_to_bf16_bits(x[2 * e + 1]) : uint32_t(__half_as_ushort(__float2half_rn(x[2 * e + 1])));
    w[e] = lo | (hi << 16);
  }
  *reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(p) + i) = make_uint4(w[0], w[1], w[2], w[3]);
}

// One choice for all eight values: chosen value by value, the branches were most of an operation.
template <class F> __device__ __forceinline__ void each(float (&r)[kProgVec], F f) {
#pragma unroll
  for (int e = 0; e < kProgVec; ++e) r[e] = f(e);
}
__device__ __forceinline__ void binary8(int fn, const float (&x)[kProgVec], const float (&y)[kProgVec], float (&r)[kProgVec]) {
  switch (fn) {
  case 0: each(r, [&](int e) { return ew_binary(0, x[e], y[e]); }); break;
  case 1: each(r, [&](int e) { return ew_binary(1, x[e], y[e]); }); break;
  case 2: each(r, [&](int e) { return ew_binary(2, x[e], y[e]); }); break;
  default: each(r, [&](int e) { return ew_binary(3, x[e], y[e]); }); break;
  }
}
__device__ __forceinline__ void unary8(int fn, float beta, const float (&x)[kProgVec], float (&r)[kProgVec]) {
  switch (fn) {
  case 0: each(r, [&](int e) { return ew_unary(0, beta, x[e]); }); break;
  case 1: each(r, [&](int e) { return ew_unary(1, beta, x[e]); }); break;
  case 2:
    if (beta == 2.f) each(r, [&](int e) { return ew_unary(2, 2.f, x[e]); });
    else each(r, [&](int e) { return ew_unary(2, beta, x[e]); });
    break;
  case 4: each(r, [&](int e) { return ew_unary(4, beta, x[e]); }); break;
  case 5: each(r, [&](int e) { return ew_unary(5, beta, x[e]); }); break;
  default: each(r, [&](int e) { return x[e]; }); break;
  }
}
__device__ __forceinline__ void round8(float (&r)[kProgVec], int dt) {
  if (dt == 1) each(r, [&](int e) { return ew_round(r[e], 1); });
  else if (dt == 2) each(r, [&](int e) { return ew_round(r[e], 2); });
}

// A thread's registers lie in shared memory, where the program can index them.  Picked from real registers by comparisons,
// with a branch per value for the operation, one operation took a block some 2000 cycles, and at 128 registers a thread an SM
// held one block of wide rows: x^2, mean, x * m^-0.5 * v over 2368 x 3072 bf16 134.8 us, where the steps one by one take 99;
// in this form 40.0 (1.1 TB/s in and out).  9472 x 4096 560 -> 195 (steps: 571), add + relu over 16384 x 4096 421 -> 206, the
// decoder block's runs with 32 tokens together 29 -> 11 us, with 512 tokens the block 354 -> 239.
struct Registers {
  float4 *v;   // [register][half][thread]
  float *s;    // [register][thread]
  __device__ __forceinline__ void get(int r, float (&x)[kProgVec]) const {
    if (r >= 16) {
      const float f = s[(r - 16) * blockDim.x];
      each(x, [&](int) { return f; });
      return;
    }
    const float4 a = v[(2 * r) * blockDim.x], b = v[(2 * r + 1) * blockDim.x];
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  }
  __device__ __forceinline__ void set(int r, const float (&x)[kProgVec]) const {
    v[(2 * r) * blockDim.x] = make_float4(x[0], x[1], x[2], x[3]);
    v[(2 * r + 1) * blockDim.x] = make_float4(x[4], x[5], x[6], x[7]);
  }
  __device__ __forceinline__ float &row(int r) const { return s[(r - 16) * blockDim.x]; }
};
constexpr size_t kRegisterBytes = kProgRegs * kProgVec * 4 + kProgRowRegs * 4;   // of a thread

// Each thread has eight consecutive values of a row in every vector register and a copy of the row's values in the row
// registers.  With a reduction a block owns one row; without, blocks walk the tensor in 8-value chunks.
// Measured on the decoder block with 32 rows: 21 launches in 79 us before, 3 in 10 us.
constexpr int kRowThreads = 512, kFlatThreads = 128;
template <bool REDUCE>
__global__ void __launch_bounds__(REDUCE ? kRowThreads : kFlatThreads, REDUCE ? 2 : 8) row_program_kernel(const __grid_constant__ RowProgram p) {
  extern __shared__ float4 registers[];
  __shared__ float part[32];
  const Registers reg = {registers + threadIdx.x, reinterpret_cast<float *>(registers + kProgRegs * 2 * blockDim.x) + threadIdx.x};
  pdl_wait();
  pdl_launch_dependents();
  const int chunks = p.cols / kProgVec;
  const long long total = REDUCE ? p.rows : p.rows * chunks;
  for (long long it = REDUCE ? blockIdx.x : blockIdx.x * (long long)blockDim.x + threadIdx.x; it < total;
       it += REDUCE ? gridDim.x : (long long)gridDim.x * blockDim.x) {
    const long long row = REDUCE ? it : it / chunks;
    const int chunk = REDUCE ? int(threadIdx.x) : int(it - row * chunks);
    const bool in = !REDUCE || chunk < chunks;
    const int col = chunk * kProgVec;
    const long long at = row * p.cols + col;
    for (int i = 0; i < p.n; ++i) {
      const RowOp o = p.op[i];
      float x[kProgVec], y[kProgVec], r[kProgVec];
      if (o.row) {
        float f = 0.f;
        if (o.kind == RowOp::LOAD) {
          f = ew_load(p.ptr[o.ptr], o.mode == 4 ? row : 0, o.dtype);
        } else if (o.kind == RowOp::STORE) {
          if (col == 0) ew_store(p.ptr[o.ptr], row, o.dtype, reg.row(o.a));
          continue;
        } else if (o.kind == RowOp::REDUCE) {
          if (REDUCE) {
            float sum = 0.f;
            if (in) {
              reg.get(o.a, x);
#pragma unroll
              for (int e = 0; e < kProgVec; ++e) sum = __fadd_rn(sum, x[e]);
            }
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xFFFFFFFFu, sum, w));
            __syncthreads();   // the shared sums of an earlier reduction have been read
            if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
            __syncthreads();
            const int warps = blockDim.x / 32;
            for (int w = 0; w < warps; ++w) f = w == 0 ? part[0] : __fadd_rn(f, part[w]);
            if (o.fn) f = __fdiv_rn(f, float(p.cols));
          }
        } else {
          f = o.kind == RowOp::BINARY ? ew_binary(o.fn, reg.row(o.a), reg.row(o.b)) : ew_unary(o.fn, o.beta, reg.row(o.a));
        }
        if (o.kind != RowOp::LOAD) f = ew_round(f, o.dtype);
        reg.row(o.dst) = f;
        continue;
      }
      if (!in) continue;
      if (o.kind == RowOp::STORE) {
        reg.get(o.a, r);
        store8(p.ptr[o.ptr], at, o.dtype, r);
        continue;
      }
      if (o.kind == RowOp::LOAD || (o.kind == RowOp::LOAD_PLANES && p.planes[o.ptr] == 0)) {
        load8(p.ptr[o.ptr], o.mode == 3 ? col : at, o.dtype, r);
      } else if (o.kind == RowOp::LOAD_PLANES) {
        // a matmul's K-split partial sums: added in split order, rounded once
        const float *base = reinterpret_cast<const float *>(p.ptr[o.ptr]);
        load8(base, at, 0, r);
        for (int k = 1; k < p.planes[o.ptr]; ++k) {
          load8(base + (long long)k * p.plane_stride[o.ptr], at, 0, x);
#pragma unroll
          for (int e = 0; e < kProgVec; ++e) r[e] = __fadd_rn(r[e], x[e]);
        }
        round8(r, 1);
      } else if (o.kind == RowOp::BINARY) {
        reg.get(o.a, x);
        reg.get(o.b, y);
        binary8(o.fn, x, y, r);
        round8(r, o.dtype);
      } else {
        reg.get(o.a, x);
        unary8(o.fn, o.beta, x, r);
        round8(r, o.dtype);
      }
      reg.set(o.dst, r);
    }
  }
}

} // namespace

void launch_row_program(const RowProgram &p, cudaStream_t stream) {
  const int chunks = p.cols / kProgVec;
  cudaLaunchConfig_t cfg = {};
  if (p.has_reduce) {
    cfg.blockDim = dim3(unsigned((chunks + 31) / 32 * 32));
    cfg.gridDim = dim3(unsigned(std::min<long long>(p.rows, 65535)));
  } else {
    const long long total = p.rows * chunks;
    cfg.blockDim = dim3(kFlatThreads);
    cfg.gridDim = dim3(unsigned(std::min<long long>((total + kFlatThreads - 1) / kFlatThreads, (long long)device_state().sm_count * 16)));
  }
  cfg.dynamicSmemBytes = cfg.blockDim.x * kRegisterBytes;
  cfg.stream = stream;
  if (p.has_reduce) {   // rows of more than 2700 columns need more shared memory than a block has without asking
    static std::once_flag configured[64];
    std::call_once(configured[device_state().device & 63], [] {
      GCB_CUDA(cudaFuncSetAttribute(row_program_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kRowThreads * kRegisterBytes)));
    });
  }
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  GCB_CUDA(cudaLaunchKernelEx(&cfg, p.has_reduce ? row_program_kernel<true> : row_program_kernel<false>, p));
  count_launch();
}

// ----------------------------------------------------------------------------- planner
namespace {

bool float_type(DType t) { return t == DType::F32 || t == DType::BF16 || t == DType::F16; }
uint8_t type_code(DType t) { return t == DType::F32 ? 0 : t == DType::BF16 ? 1 : 2; }

std::vector<int64_t> stripped(const std::vector<int64_t> &s) {   // without leading ones
  size_t i = 0;
  while (i + 1 < s.size() && s[i] == 1) ++i;
  return std::vector<int64_t>(s.begin() + long(i), s.end());
}
bool dense(const LogicalTensor &t) {
  if (!t.strided || t.stride.size() != t.shape.size()) return true;
  int64_t expect = 1;
  for (int d = int(t.shape.size()) - 1; d >= 0; --d) {
    if (t.shape[size_t(d)] != 1 && t.stride[size_t(d)] != expect) return false;
    expect *= t.shape[size_t(d)];
  }
  return true;
}
bool fusable_kind(const Step &st) { return st.kind == StepKind::BINARY || st.kind == StepKind::UNARY || st.kind == StepKind::REDUCE; }

enum class Form { FULL, VECTOR, ROW, ONE, OTHER };

struct Compiler {
  const Plan &plan;
  int first, last;
  RowGroup g;
  std::vector<int64_t> full, lead;   // the run's shape and the same with one value per row, leading ones stripped
  std::unordered_map<size_t, int> reg;     // tensor -> register, while it is needed
  std::unordered_map<size_t, uint8_t> slot;
  std::vector<size_t> loaded, stored;
  bool used[kProgRegs] = {}, used_row[kProgRowRegs] = {};

  Compiler(const Plan &p, int f, int l) : plan(p), first(f), last(l) {}
  const LogicalTensor &tensor(size_t id) const { return plan.part.tensors.at(id); }
  const Step &step(int i) const { return plan.steps[size_t(i)]; }

  Form form(const LogicalTensor &t) const {
    if (!dense(t) || !float_type(t.dtype) || t.numel() == 0) return Form::OTHER;
    const auto s = stripped(t.shape);
    if (s == full) return Form::FULL;
    if (t.numel() == 1) return Form::ONE;
    if (s == lead) return Form::ROW;
    if (s.size() == 1 && s[0] == full.back()) return Form::VECTOR;
    return Form::OTHER;
  }
  bool needed_after(size_t id, int i) const {   // read by a later step of the run
    for (int k = i + 1; k <= last; ++k)
      if (std::find(step(k).in.begin(), step(k).in.end(), id) != step(k).in.end()) return true;
    return false;
  }
  bool leaves(size_t id) const {
    if (std::find(plan.part.output_ids.begin(), plan.part.output_ids.end(), id) != plan.part.output_ids.end()) return true;
    for (size_t k = size_t(last) + 1; k < plan.steps.size(); ++k)
      if (std::find(plan.steps[k].in.begin(), plan.steps[k].in.end(), id) != plan.steps[k].in.end()) return true;
    return false;
  }
  int take(bool row) {
    bool *u = row ? used_row : used;
    for (int k = 0; k < (row ? kProgRowRegs : kProgRegs); ++k)
      if (!u[k]) {
        u[k] = true;
        return row ? 16 + k : k;
      }
    return -1;
  }
  void drop(size_t id) {
    auto it = reg.find(id);
    if (it == reg.end()) return;
    (it->second >= 16 ? used_row[it->second - 16] : used[it->second]) = false;
    reg.erase(it);
  }
  int pointer(size_t id) {
    auto it = slot.find(id);
    if (it != slot.end()) return it->second;
    if (g.ids.size() == size_t(kProgPtrs)) return -1;
    g.ids.push_back(id);
    g.bytes.push_back(plan.slots.at(id).bytes);
    g.stored.push_back(0);
    g.whole.push_back(form(tensor(id)) == Form::FULL);
    return slot[id] = uint8_t(g.ids.size() - 1);
  }
  bool emit(const RowOp &o) {
    if (g.prog.n == kProgOps) return false;
    g.prog.op[g.prog.n++] = o;
    return true;
  }
  // The matmul step whose K-split planes may be summed here: a bf16 result that only this run reads (its own memory is
  // then never written, so no step before or after the run may look there).
  int deferrable(size_t id) const {
    if (leaves(id)) return -1;
    int producer = -1;
    for (int k = 0; k < first; ++k) {
      const Step &st = step(k);
      if (std::find(st.in.begin(), st.in.end(), id) != st.in.end()) return -1;
      if (st.out.size() == 1 && st.out[0] == id)
        producer = st.kind == StepKind::MATMUL && !st.has_bias && !st.relu && tensor(id).dtype == DType::BF16 ? k : -1;
    }
    return producer;
  }
  bool load(size_t id) {   // brings an operand into a register
    if (reg.count(id)) return true;
    const LogicalTensor &t = tensor(id);
    const Form f = form(t);
    for (int k = first; k <= last; ++k)   // produced inside the run: must still be in a register
      if (std::find(step(k).out.begin(), step(k).out.end(), id) != step(k).out.end()) return false;
    RowOp o{};
    o.kind = RowOp::LOAD;
    o.dtype = type_code(t.dtype);
    o.row = f == Form::ROW || f == Form::ONE;
    o.mode = f == Form::FULL ? 1 : f == Form::ONE ? 2 : f == Form::VECTOR ? 3 : 4;
    if (f == Form::OTHER) return false;
    if (f == Form::FULL) {
      const int m = deferrable(id);
      if (m >= 0) {
        o.kind = RowOp::LOAD_PLANES;
        g.deferred.push_back(m);
      }
    }
    const int p = pointer(id), r = take(o.row);
    if (p < 0 || r < 0) return false;
    o.ptr = uint8_t(p);
    o.dst = uint8_t(r);
    reg[id] = r;
    loaded.push_back(id);
    return emit(o);
  }

  bool run() {
    // the run's shape: the widest tensor it produces or reduces
    const std::vector<int64_t> *widest = nullptr;
    int64_t most = 0;
    for (int i = first; i <= last; ++i) {
      for (const auto *list : {&step(i).in, &step(i).out})
        for (size_t id : *list)
          if (tensor(id).numel() > most) {
            most = tensor(id).numel();
            widest = &tensor(id).shape;
          }
    }
    if (!widest || widest->empty()) return false;
    full = stripped(*widest);
    lead = full;
    lead.back() = 1;
    lead = stripped(lead);
    const int64_t cols = full.back();
    if (cols % kProgVec || cols > (int64_t(1) << 30)) return false;
    g.first = first;
    g.last = last;
    g.prog.cols = int(cols);
    g.prog.rows = most / cols;
    for (int i = first; i <= last; ++i) {
      const Step &st = step(i);
      if (st.out.size() != 1) return false;
      const LogicalTensor &O = tensor(st.out[0]);
      if (!float_type(O.dtype) || !dense(O)) return false;
      for (size_t id : st.in)
        if (!load(id)) return false;
      RowOp o{};
      o.dtype = type_code(O.dtype);
      o.a = uint8_t(reg.at(st.in[0]));
      bool row = false;
      if (st.kind == StepKind::REDUCE) {
        // over the last axis, rows long enough that a kernel of its own would not sum in plain ascending order either
        const LogicalTensor &A = tensor(st.in[0]);
        if (form(A) != Form::FULL || st.axes.size() != 1 || st.axes[0] != int64_t(A.shape.size()) - 1) return false;
        if (cols < 512 || cols > kRowThreads * kProgVec || O.numel() != g.prog.rows) return false;
        const bool keeps = O.shape.size() == A.shape.size();
        if (!keeps && needed_after(st.out[0], i)) return false;   // without its last axis it broadcasts as another shape
        g.prog.has_reduce = 1;
        o.kind = RowOp::REDUCE;
        o.fn = st.mean ? 1 : 0;
        row = true;
      } else {
        o.kind = st.kind == StepKind::BINARY ? RowOp::BINARY : RowOp::UNARY;
        o.fn = uint8_t(st.fn);
        o.beta = st.beta;
        if (st.kind == StepKind::BINARY) o.b = uint8_t(reg.at(st.in[1]));
        const Form f = form(O);
        row = f == Form::ROW || (f == Form::ONE && g.prog.rows == 1);
        if (!row && f != Form::FULL) return false;
        bool any_full = false;
        for (size_t id : st.in) any_full |= reg.at(id) < 16;
        if (any_full == row) return false;   // a row value comes from row values, a full tensor from at least one vector
        if (f == Form::FULL) {
          bool whole = false;   // two [cols] vectors would make a [cols] tensor
          for (size_t id : st.in) whole |= form(tensor(id)) == Form::FULL || (form(tensor(id)) == Form::ROW && st.in.size() == 2);
          if (!whole) return false;
        }
      }
      for (size_t id : st.in)
        if (!needed_after(id, i)) drop(id);
      const int r = take(row);
      if (r < 0) return false;
      o.row = row;
      o.dst = uint8_t(r);
      reg[st.out[0]] = r;
      if (!emit(o)) return false;
      if (leaves(st.out[0])) {
        RowOp w{};
        w.kind = RowOp::STORE;
        w.row = row;
        w.a = uint8_t(r);
        w.dtype = type_code(O.dtype);
        const int p = pointer(st.out[0]);
        if (p < 0) return false;
        w.ptr = uint8_t(p);
        g.stored[size_t(p)] = 1;
        stored.push_back(st.out[0]);
        if (!emit(w)) return false;
      }
      if (!needed_after(st.out[0], i)) drop(st.out[0]);
    }
    // blocks run at their own pace: nothing may be stored over memory that another block has still to read
    for (size_t w : stored)
      for (size_t l : loaded) {
        const TensorSlot &a = plan.slots.at(w), &b = plan.slots.at(l);
        if (a.where == TensorSlot::ARENA && b.where == TensorSlot::ARENA && a.offset < b.offset + b.bytes && b.offset < a.offset + a.bytes) return false;
      }
    return true;
  }
};

} // namespace

bool row_program_fits(const RowGroup &g, void *const *ptr) {
  auto at = [&](size_t i) { return reinterpret_cast<uintptr_t>(ptr[i]); };
  for (size_t i = 0; i < g.ids.size(); ++i) {
    if (at(i) & 15) return false;
    if (!g.stored[i]) continue;
    for (size_t k = 0; k < g.ids.size(); ++k) {
      if (k == i || at(i) >= at(k) + g.bytes[k] || at(k) >= at(i) + g.bytes[i]) continue;
      if (!(at(i) == at(k) && g.whole[i] && g.whole[k] && g.bytes[i] == g.bytes[k])) return false;
    }
  }
  return true;
}

std::vector<RowGroup> plan_row_groups(const Plan &plan) {
  std::vector<RowGroup> groups;
  const int n = int(plan.steps.size());
  for (int i = 0; i < n; ++i) {
    if (!fusable_kind(plan.steps[size_t(i)])) continue;
    int end = i;
    while (end + 1 < n && fusable_kind(plan.steps[size_t(end) + 1])) ++end;
    for (int e = end; e > i; --e) {   // the longest run that one program holds: mostly the first try
      Compiler c(plan, i, e);
      if (!c.run()) continue;
      groups.push_back(std::move(c.g));
      i = e;
      break;
    }
  }
  return groups;
}

} // namespace gcb
