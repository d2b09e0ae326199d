// SSOR sweeps as a dataflow of rows (ssorflow.cu).
#pragma once
#include "linalg.cuh"

namespace rsg {

// Forward and backward sweeps of SSOR over one pattern, rows in the order of
// their level (the sweep plans of precond.cu).
struct SsorFlow {
  // A, its sweep plans (entries: the row without its diagonal) and which
  // kernels run (see ssorflow.cu) are the pattern's; the values are set by
  // values() and stay until it is called again.
  void plan(Csr& A, const SweepPlan& fwd, const SweepPlan& bwd);
  void values(const double* csr);
  // whether a sweep in this precision reads its sweep plan's values
  bool reads_plan(bool backward, bool f32) const { return f32 ? slices : levels[backward ? 1 : 0]; }
  // One sweep over `old`: out_i = old_i + omega (sigma_i - old_i), sigma_i from
  // out's values at lower (backward: higher) columns and old's elsewhere.
  template <typename T>
  void sweep(bool backward, const T* b, const T* old, T* out, T omega, const int* active);

 private:
  Context* ctx = nullptr;
  Csr* A = nullptr;
  const SweepPlan* plans[2] = {nullptr, nullptr};
  bool slices = false;                    // FP32: a warp per slice (else by rows)
  bool levels[2] = {false, false};        // FP64: a launch per level
  bool few[2] = {false, false};           // FP64: by rows in one CTA (else over all SMs)
  DeviceBuffer<int> order[2], newest[2];
  DeviceBuffer<double> val;  // by CSR position, where the rows kernel runs
  DeviceBuffer<float> valf;
  DeviceBuffer<unsigned> ticket;
};

}  // namespace rsg
