// SSOR sweeps as a dataflow of rows (ssorflow.cu).
#pragma once
#include "linalg.cuh"

namespace rsg {

// Forward and backward sweeps of SSOR over one pattern, rows in the order of
// their level (the sweep plans of precond.cu).
struct SsorFlow {
  // A, its sweep plans (entries: the row without its diagonal) and whether
  // the rows kernel runs (see plan()) are the pattern's; the values are set
  // by values() and stay until it is called again.
  void plan(Csr& A, const SweepPlan& fwd, const SweepPlan& bwd);
  void values(const double* csr);
  // One sweep over `old`: out_i = old_i + omega (sigma_i - old_i), sigma_i from
  // out's values at lower (backward: higher) columns and old's elsewhere.
  template <typename T>
  void sweep(bool backward, const T* b, const T* old, T* out, T omega, const int* active);

 private:
  Context* ctx = nullptr;
  Csr* A = nullptr;
  const SweepPlan* plans[2] = {nullptr, nullptr};
  int widest = 0;  // longest row, without its diagonal
  DeviceBuffer<int> order[2], newest[2];
  DeviceBuffer<double> val;  // by CSR position, where the rows kernel runs
  DeviceBuffer<float> valf;
  DeviceBuffer<unsigned> ticket;
  template <typename T>
  bool by_slices() const;
};

}  // namespace rsg
