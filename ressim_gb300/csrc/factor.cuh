// ILU(0) factorisation as a dataflow of rows (factor.cu).
#pragma once
#include "linalg.cuh"

namespace rsg {

constexpr int FACTOR_LANES = 32;  // rows up to this many entries: a lane per entry

struct RowFactor {
  bool planned = false;
  DeviceBuffer<int> order, lptr;
  DeviceBuffer<unsigned char> match;  // per strictly lower entry and lane
  DeviceBuffer<double> rinv;          // reciprocal of each finished row's diagonal
  DeviceBuffer<unsigned> ticket;
  // order: the rows by level of the lower triangle.  False (and not planned)
  // when a row is longer than a warp.
  bool plan(Csr& A, const std::vector<int>& order);
  // LU := the factors of A; flag: 1 + the position of a lower entry whose
  // pivot is zero.
  void run(Csr& A, double* LU, int* flag);
};

}  // namespace rsg
