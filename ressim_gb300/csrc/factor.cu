// ILU(0) factorisation (mtj/src/no/uib/cipr/matrix/sparse/ILU.java:98-125),
// one warp per row, rows in the order of their level, each started as soon as
// the values it reads are there.
//
// Row k's lane l holds entry l.  For every strictly lower entry i in
// ascending order LU_ki = v_i / U_ii is formed and LU_ki U_ij subtracted from
// the entries whose column U's row i has, product and sum rounded apart as in
// the Java loop, so the factors equal its bit for bit.  Which entry of row i
// a lane needs is a byte per lower entry and lane, matched once per pattern
// on the GPU.
//
// What bounds it: double precision.  A warp instruction of it costs 19 cycles
// of an SM (64 of its sub-partition), and a row of a 27-point pattern takes
// 13 x (5 for the quotient + 2) + the reciprocal of its diagonal.  The quotient
// is therefore not the library's division (560 cycles of dependent steps)
// but two corrections from the diagonal's reciprocal, which its row's warp
// computes once.  A row waits for its neighbours only where it reads them:
// the neighbour finished last is the last one read.  128x128x32 (13.7M
// entries): 3.5 ms, against 51 ms level by level on an 8-CTA cluster with a
// thread per row; 64x64x16: 0.77 against 20.7 ms; 32x32x8: 0.21 against 5.3.
#include <cmath>

#include "dataflow.cuh"
#include "factor.cuh"

namespace rsg {

namespace {

struct RowFactorArgs {
  int n;
  const int* order;
  const int* rowptr;
  const int* col;
  const int* diag;
  const int* lptr;
  const unsigned char* match;
  const double* val;
  double* LU;
  double* rinv;
  unsigned* ticket;
  int* flag;
  int* err;
};

__device__ __forceinline__ bool mid_range(double x) {  // 2^-800 <= |x| <= 2^800
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  return e > 1023 - 800 && e < 1023 + 800;
}

// a / d, rounded as IEEE division rounds it, given r = RN(1 / d): a first
// quotient, one correction that brings it within an ulp, and a second whose
// remainder is exact and whose result is the correctly rounded quotient
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990, theorem 8.2).  Away from
// over- and underflow only; elsewhere, and for zeros, plain division.
__device__ __forceinline__ double quotient(double a, double d, double r) {
  const double q0 = __dmul_rn(a, r);
  if (mid_range(a) && mid_range(d) && mid_range(q0)) {
    const double q1 = __fma_rn(__fma_rn(-q0, d, a), r, q0);
    return __fma_rn(__fma_rn(-q1, d, a), r, q1);
  }
  return a / d;
}

constexpr int FACTOR_CHUNK = 8;  // lower entries whose operands are loaded together

__global__ void __launch_bounds__(256) k_factor_rows(RowFactorArgs g) {
  using S = Sentinel<double>;
  constexpr unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  auto draw = [&] { return lane == 0 ? atomicAdd(g.ticket, 1u) : 0u; };
  // Rows in order, from a counter: the row of the smallest ticket not yet
  // finished reads finished rows only, so some warp always goes on.
  unsigned next = draw();
  for (;;) {
    const unsigned t = __shfl_sync(ALL, next, 0);
    if (t >= (unsigned)g.n) break;
    next = draw();  // the counter's latency passes behind this row
    const int k = g.order[t];
    const int r0 = g.rowptr[k], len = g.rowptr[k + 1] - r0, nl = g.diag[k] - r0;
    const unsigned char* match = g.match + (size_t)g.lptr[k] * FACTOR_LANES + lane;
    double v = lane < len ? g.val[r0 + lane] : 0.0;
    // lane i < nl: the pivot of lower entry i and its reciprocal
    const int index = lane < nl ? g.col[r0 + lane] : 0;
    const int piv = lane < nl ? g.diag[index] : 0;
    S::Bits d = 0, r = 0;
    if (lane < nl) {
      d = S::load(g.LU + piv);
      r = S::load(g.rinv + index);
    }
    for (int c = 0; c < nl; c += FACTOR_CHUNK) {
      int at[FACTOR_CHUNK];
      S::Bits u[FACTOR_CHUNK];
#pragma unroll
      for (int q = 0; q < FACTOR_CHUNK; ++q) {
        const int m = c + q < nl ? match[(size_t)(c + q) * FACTOR_LANES] : 0;
        const int p = __shfl_sync(ALL, piv, (c + q) & 31);
        at[q] = m ? p + m : -1;
      }
#pragma unroll
      for (int q = 0; q < FACTOR_CHUNK; ++q) u[q] = at[q] >= 0 ? S::load(g.LU + at[q]) : 0;
#pragma unroll
      for (int q = 0; q < FACTOR_CHUNK; ++q) {
        const int i = c + q;
        if (i >= nl) break;
        unsigned long long start = 0;
        for (int w = 1; __any_sync(ALL, u[q] == S::bits || (lane == i && (d == S::bits || r == S::bits))); ++w) {
          if (u[q] == S::bits) u[q] = S::load(g.LU + at[q]);
          if (lane == i && d == S::bits) d = S::load(g.LU + piv);
          if (lane == i && r == S::bits) r = S::load(g.rinv + index);
          if ((w & 255) == 0 && __any_sync(ALL, wait_over(start, g.err))) {
            atomicCAS(g.err, 0, 1 + k);
            break;
          }
        }
        const double dd = __shfl_sync(ALL, S::value(d), i), rr = __shfl_sync(ALL, S::value(r), i);
        if (dd == 0 && lane == 0) atomicCAS(g.flag, 0, r0 + i + 1);
        const double f = quotient(__shfl_sync(ALL, v, i), dd, rr);
        if (lane == i) v = f;
        if (at[q] >= 0) v = __dsub_rn(v, __dmul_rn(f, S::value(u[q])));
      }
    }
    if (lane < len) S::store(g.LU + r0 + lane, S::guard(v));
    if (lane == nl) S::store(g.rinv + k, S::guard(1.0 / v));
  }
}

// For every strictly lower entry i of every row: the lane's entry in U's row
// col_i, as its distance from that row's diagonal (0: it has none).
__global__ void k_factor_match(int n, const int* __restrict__ rowptr, const int* __restrict__ col,
                               const int* __restrict__ diag, const int* __restrict__ lptr,
                               unsigned char* __restrict__ match) {
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= n) return;
  const int r0 = rowptr[k], len = rowptr[k + 1] - r0, nl = diag[k] - r0;
  const int c = lane < len ? col[r0 + lane] : -1;
  for (int i = 0; i < nl; ++i) {
    const int index = col[r0 + i], d = diag[index];
    int m = 0;
    for (int j = d + 1; j < rowptr[index + 1]; ++j)
      if (col[j] == c) m = j - d;
    match[((size_t)lptr[k] + i) * FACTOR_LANES + lane] = (unsigned char)m;
  }
}

}  // namespace

bool RowFactor::plan(Csr& A, const std::vector<int>& rows) {
  planned = false;
  for (int k = 0; k < A.n; ++k)
    if (A.h_rowptr[k + 1] - A.h_rowptr[k] > FACTOR_LANES) return false;
  Context& ctx = *A.ctx;
  std::vector<int> lp(A.n + 1, 0);
  for (int k = 0; k < A.n; ++k) lp[k + 1] = lp[k] + A.h_diag[k] - A.h_rowptr[k];
  order.resize(A.n);
  lptr.resize(A.n + 1);
  match.resize(std::max<size_t>((size_t)lp[A.n] * FACTOR_LANES, 1));
  rinv.resize(A.n);
  ticket.resize(1);
  RSG_CUDA(cudaMemcpyAsync(order.get(), rows.data(), sizeof(int) * A.n, cudaMemcpyHostToDevice, ctx.stream));
  RSG_CUDA(cudaMemcpyAsync(lptr.get(), lp.data(), sizeof(int) * (A.n + 1), cudaMemcpyHostToDevice, ctx.stream));
  RSG_LAUNCH(ctx, "factor_match", k_factor_match, blocks_for((int64_t)A.n * 32, 256), 256, 0, A.n, A.rowptr.get(),
             A.col.get(), A.diag.get(), lptr.get(), match.get());
  ctx.sync();  // lp goes out of scope
  planned = true;
  return true;
}

void RowFactor::run(Csr& A, double* LU, int* flag) {
  Context& ctx = *A.ctx;
  RSG_LAUNCH(ctx, "factor_fill", k_sentinel<double>, blocks_for(A.nnz, 256), 256, 0, (int64_t)A.nnz, LU);
  RSG_LAUNCH(ctx, "factor_fill", k_sentinel<double>, blocks_for(A.n, 256), 256, 0, (int64_t)A.n, rinv.get());
  RSG_CUDA(cudaMemsetAsync(ticket.get(), 0, sizeof(unsigned), ctx.stream));
  const RowFactorArgs g{A.n,         order.get(),   A.rowptr.get(), A.col.get(), A.diag.get(), lptr.get(), match.get(),
                        A.val.get(), LU,            rinv.get(),     ticket.get(), flag,        ctx.dev_err.get()};
  // two CTAs of eight warps per SM keep its double-precision pipe busy
  const int grid = std::min(2 * ctx.num_sms, blocks_for((int64_t)A.n * 32, 256));
  RSG_LAUNCH(ctx, "ilu_factor", k_factor_rows, grid, 256, 0, g);
}

}  // namespace rsg
