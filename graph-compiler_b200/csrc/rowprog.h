// Elementwise runs of a partition as one kernel.
//
// A run of consecutive Add / Multiply / Pow / Typecast / ReduceMean / ... steps over tensors of one [rows][cols] shape is
// compiled, when the executable is built, into a short program that one kernel interprets: every value of the run stays
// in registers, only what later steps or the caller need is stored.  Each operation rounds to its own result type, so
// the bits are those of the step-by-step kernels (a row reduction sums in another order than a kernel of its own would).
#pragma once
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "graph.h"

namespace gcb {

constexpr int kProgOps = 40, kProgPtrs = 16, kProgRegs = 4, kProgRowRegs = 4, kProgVec = 8;

struct RowOp {
  enum Kind : uint8_t { LOAD, LOAD_PLANES, STORE, BINARY, UNARY, REDUCE };
  uint8_t kind;
  uint8_t row;       // 1: one value per row (registers s0..), 0: a vector of the row (registers v0..)
  uint8_t fn;        // BINARY / UNARY function (Step::fn); REDUCE: 1 = mean
  uint8_t dst, a, b; // registers: 0..kProgRegs-1 vectors, 16 + i row values
  uint8_t dtype;     // LOAD / STORE: element type in memory; otherwise the type the result is rounded to (0 f32, 1 bf16, 2 f16)
  uint8_t ptr;       // LOAD / STORE: pointer slot
  uint8_t mode;      // LOAD: 1 the run's own layout, 2 one value, 3 a vector of cols values, 4 one value per row
  float beta;
};
struct RowProgram {
  int n = 0, cols = 0, has_reduce = 0;
  long long rows = 0;
  RowOp op[kProgOps];
  void *ptr[kProgPtrs];
  int planes[kProgPtrs];             // LOAD_PLANES: partial planes to sum, in order, before the value is rounded to bf16
  long long plane_stride[kProgPtrs]; // elements
};

// A fused run: steps [first, last] of the plan.
struct RowGroup {
  int first = 0, last = 0;
  RowProgram prog;
  std::vector<size_t> ids;     // tensor behind each pointer slot
  std::vector<size_t> bytes;   // its size
  std::vector<char> stored, whole;   // the program writes it; it has the run's shape (a thread touches its own elements only)
  std::vector<int> deferred;   // matmul steps whose K-split planes the program may sum itself (their result has no other reader)
};

// Runs worth fusing (two steps or more).  Host logic; steps that do not fit are left out.
std::vector<RowGroup> plan_row_groups(const Plan &plan);

// Whether the tensors lie where the program may run on them: 16-byte aligned, and nothing is stored over memory that
// another thread has still to load - a caller may hand in buffers that overlap, and one after the other the steps allow it.
// The one overlap that is fine is a result in the place of an operand of the same shape and element size.
bool row_program_fits(const RowGroup &g, void *const *ptr);

// The caller runs the steps one by one where row_program_fits says no.
void launch_row_program(const RowProgram &p, cudaStream_t stream);

} // namespace gcb
