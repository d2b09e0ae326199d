// SSOR sweeps (mtj/src/no/uib/cipr/matrix/sparse/SSOR.java:143-194) as a
// dataflow of rows: a row starts as soon as the values it reads are there,
// polling the values themselves (dataflow.cuh).  Rows are summed in CSR order,
// products and sums rounded apart, as the Java loop does.
//
// What bounds a sweep is its chain of dependent rows (about 160 on a 40 x 36 x
// 12 grid, and nearly as many rows on the narrow coarse levels of an AMG
// hierarchy), or, where many rows are independent, the double-precision pipe,
// which a warp instruction holds for 64 cycles whatever its active lanes.
//
// FP64, times of one sweep:
//  * Rows over all SMs, a warp per row, a lane per entry, the lanes' products
//    summed in order through shuffles; values polled through L2.  40x36x12
//    0.34 ms, 96x96x24 1.0, against 1.5 and 7.2 level by level on an 8-CTA
//    cluster.
//  * Rows in one CTA, values polled in shared memory: a shorter hop, one SM.
//    Where a level has at most four rows on average: tridiagonal 20,000 rows
//    15.5 ms against 20.0 over all SMs, 1,000 rows in 697 levels 1.63 against
//    1.82; at eleven rows a level the one SM takes twice as long.  Rows of more
//    than 128 entries wait for their sums rather than for hops.
//  * Level by level, a launch each, a thread per row: a thirty-second of the
//    pipe's time.  Where a level has 10,000 rows or more, or there are two at
//    most: red-black order, 1,000,000 rows of 24 entries 0.15 ms against 2.3;
//    at 3,300 rows a level (128x128x64, seven points) rows take 1.4 ms and
//    levels 3.3.
//
// FP32 sweeps are the mixed-precision solver's own:
//  * Patterns whose vector fits shared memory and whose rows have at most 32
//    entries: one CTA, a thread per row, a warp per slice of 32 rows of one
//    level (the sweep plan's SELL slices).  A hop is a poll of shared memory.
//    A warp's slices are far apart in the order, so the loads of one pass
//    behind the chain of the slices before it.
//  * Wider rows (Galerkin products): a warp per row as above, one CTA while the
//    rows are few.  No order is owed to the Java loop: a row leaves the operand
//    that comes last (of the highest level) out of the sum, adds the others by
//    a tree while it waits for it, and has one multiply-add left when it is
//    there.
// The V-cycle sweeps of a 40 x 36 x 12 system in FP32: 26 us on the 17,280
// rows (slices) and 20 us on average on the three coarse levels (a warp per
// row; 34 us with the ordered sum), against 245 us on average on one 8-CTA
// cluster with a barrier per level.  That solve with its setup takes 45 ms, 287
// with the cluster's sweeps; chained launches, where a sweep readies its shared
// memory beside the end of the kernel before, are a sixth of what is left.
#include "dataflow.cuh"
#include "ssorflow.cuh"

namespace rsg {

namespace {

constexpr int FLOW_WIDTH = 32;               // entries of a row held in registers (slices)
constexpr int FLOW_GROUP = 8;                // operands polled together
constexpr int FLOW_CHUNKS = 4;               // 32 entries each held in registers (rows)
constexpr int FLOW_ROWS_MAX = 4096;          // FP32 rows one CTA takes a warp each: 100 instructions a row
constexpr int FLOW_FEW = 4;                  // rows a level, on average, that one CTA takes in FP64
constexpr int FLOW_MANY = 10000;             // rows a level, on average, from which levels are launched
constexpr size_t FLOW_SMEM = 200 * 1024;
constexpr int FLOW_SLICE_THREADS = 512;
constexpr int FLOW_ROW_THREADS = 512;

// The values being computed, in the CTA's shared memory or in global memory.
template <typename T, bool SMEM>
struct Fresh;
template <bool SMEM>
struct Fresh<double, SMEM> {
  using S = Sentinel<double>;
  static __device__ __forceinline__ S::Bits load(const double* p) {
    if (!SMEM) return S::load(p);
    S::Bits v;
    asm volatile("ld.relaxed.cta.shared.u64 %0, [%1];" : "=l"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(double* p, S::Bits v) {
    if (!SMEM) return S::store(p, v);
    asm volatile("st.relaxed.cta.shared.u64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "l"(v) : "memory");
  }
};
template <bool SMEM>
struct Fresh<float, SMEM> {
  using S = Sentinel<float>;
  static __device__ __forceinline__ S::Bits load(const float* p) {
    if (!SMEM) return S::load(p);
    S::Bits v;
    asm volatile("ld.relaxed.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(float* p, S::Bits v) {
    if (!SMEM) return S::store(p, v);
    asm volatile("st.relaxed.cta.shared.u32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v) : "memory");
  }
};

__device__ __forceinline__ double from_bits(unsigned long long b) { return Sentinel<double>::value(b); }
__device__ __forceinline__ float from_bits(unsigned b) { return Sentinel<float>::value(b); }

template <typename T>
struct SsorArgs {
  int n;
  const T* val;
  const T* b;
  const T* old;
  T* out;
  T omega;
  const int* active;
  int* err;
  // slices
  int nslices;
  const int *slice_base, *row, *len, *scol;
  const T* diag;
  // rows
  const int *order, *rowptr, *col, *dpos;
  const int* newest;  // entry of the row that is computed last, -1 none
  unsigned* ticket;
};

// Waits until none of a lane's operands u[k] with at[k] >= 0 is missing, the
// warp together.  A wait given up goes on with what is there.
template <typename T, bool SMEM, int N>
__device__ __forceinline__ void await(typename Sentinel<T>::Bits (&u)[N], const int* at, const T* fresh, int row,
                                      int* err) {
  using S = Sentinel<T>;
  unsigned long long start = 0;
  for (int w = 1;; ++w) {
    bool missing = false;
#pragma unroll
    for (int k = 0; k < N; ++k) missing |= at[k] >= 0 && u[k] == S::bits;
    if (!__any_sync(0xffffffffu, missing)) return;
    if ((w & 255) == 0 && __any_sync(0xffffffffu, wait_over(start, err))) {
      atomicCAS(err, 0, 1 + max(row, 0));
      return;
    }
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (at[k] >= 0 && u[k] == S::bits) u[k] = Fresh<T, SMEM>::load(fresh + at[k]);
  }
}

template <typename T, bool BWD>
__global__ void __launch_bounds__(FLOW_SLICE_THREADS, 1) k_ssor_slices(SsorArgs<T> a) {
  using S = Sentinel<T>;
  extern __shared__ __align__(16) unsigned char smem[];
  T* fresh = reinterpret_cast<T*>(smem);
  for (int i = threadIdx.x; i < a.n; i += blockDim.x) fresh[i] = S::value(S::bits);
  chain_begin();
  if (a.active && *a.active != 0) return;
  __syncthreads();
  const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  // Slices in order, every nwarps-th a warp's: the first one not finished
  // reads finished ones only, and its warp has no earlier one left.
  struct Meta {
    int row, len, base;
  };
  auto meta = [&](int s) {
    Meta m{-1, 0, 0};
    if (s < a.nslices) {
      m.row = a.row[s * 32 + lane];
      m.len = m.row >= 0 ? a.len[s * 32 + lane] : 0;
      m.base = a.slice_base[s] + lane;
    }
    return m;
  };
  Meta next = meta(threadIdx.x >> 5);
  for (int s = threadIdx.x >> 5; s < a.nslices; s += nwarps) {
    const Meta m = next;
    T v[FLOW_WIDTH];
    int at[FLOW_WIDTH];
    typename S::Bits u[FLOW_WIDTH / FLOW_GROUP][FLOW_GROUP];
#pragma unroll
    for (int k = 0; k < FLOW_WIDTH; ++k) {
      at[k] = -1;
      v[k] = 0;
      if (k < m.len) {
        at[k] = a.scol[m.base + 32 * k];
        v[k] = a.val[m.base + 32 * k];
      }
    }
    T d = 1, bi = 0, self = 0;
    if (m.row >= 0) {
      d = a.diag[s * 32 + lane];
      bi = a.b[m.row];
      self = a.old[m.row];
    }
    next = meta(s + nwarps);
#pragma unroll
    for (int k = 0; k < FLOW_WIDTH; ++k) {
      auto& w = u[k / FLOW_GROUP][k % FLOW_GROUP];
      w = 0;
      if (k < m.len && !(BWD ? at[k] > m.row : at[k] < m.row)) {
        w = S::of(a.old[at[k]]);
        at[k] = -1;  // there already
      }
    }
    T sum = 0;
#pragma unroll
    for (int g = 0; g < FLOW_WIDTH / FLOW_GROUP; ++g) {
#pragma unroll
      for (int k = 0; k < FLOW_GROUP; ++k)
        if (at[g * FLOW_GROUP + k] >= 0) u[g][k] = Fresh<T, true>::load(fresh + at[g * FLOW_GROUP + k]);
      await<T, true>(u[g], at + g * FLOW_GROUP, fresh, m.row, a.err);
#pragma unroll
      for (int k = 0; k < FLOW_GROUP; ++k)
        if (g * FLOW_GROUP + k < m.len) sum += v[g * FLOW_GROUP + k] * from_bits(u[g][k]);
    }
    if (m.row >= 0) {
      const T sigma = (bi - sum) / d;
      const typename S::Bits r = S::guard(self + a.omega * (sigma - self));
      Fresh<T, true>::store(fresh + m.row, r);
      a.out[m.row] = S::value(r);
    }
    __syncwarp();
  }
}

template <typename T, bool BWD, bool SMEM>
__global__ void __launch_bounds__(FLOW_ROW_THREADS, 1) k_ssor_rows(SsorArgs<T> a) {
  using S = Sentinel<T>;
  constexpr unsigned ALL = 0xffffffffu;
  constexpr bool TREE = sizeof(T) == 4;
  extern __shared__ __align__(16) unsigned char smem[];
  T* fresh = SMEM ? reinterpret_cast<T*>(smem) : a.out;
  if (SMEM)
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) fresh[i] = S::value(S::bits);
  chain_begin();
  if (a.active && *a.active != 0) return;
  if (SMEM) __syncthreads();
  const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  // Rows in order: in one CTA every nwarps-th is a warp's, else from a
  // counter.  Either way the first row not finished reads finished rows only,
  // and its warp is at it.
  struct Meta {
    int row, r0, len, d, newest;
  };
  unsigned drawn = SMEM ? threadIdx.x >> 5 : lane == 0 ? atomicAdd(a.ticket, 1u) : 0u;
  auto take = [&] {
    const unsigned t = SMEM ? drawn : __shfl_sync(ALL, drawn, 0);
    Meta m{-1, 0, 0, 0, -1};
    if (t < (unsigned)a.n) {
      m.row = a.order[t];
      m.r0 = a.rowptr[m.row];
      m.len = a.rowptr[m.row + 1] - m.r0;
      m.d = a.dpos[m.row] - m.r0;
      if (TREE) m.newest = a.newest[m.row];
      if (SMEM) drawn += nwarps;
    }
    return m;
  };
  Meta next = take();
  while (next.row >= 0) {
    const Meta m = next;
    if (!SMEM) drawn = lane == 0 ? atomicAdd(a.ticket, 1u) : 0u;
    T v[FLOW_CHUNKS];
    int at[FLOW_CHUNKS];
    typename S::Bits u[FLOW_CHUNKS][1];
    // a chunk's entries: coefficient, and the operand or (at >= 0) where it will be
    auto load = [&](int q0, T& vk, int& ak, typename S::Bits& uk) {
      const int e = q0 + lane;
      vk = 0;
      ak = -1;
      uk = 0;
      if (e >= m.len || e == m.d || e == m.newest) return;
      const int c = a.col[m.r0 + e];
      vk = a.val[m.r0 + e];
      if (BWD ? c > m.row : c < m.row) {
        ak = c;
        uk = S::bits;
      } else {
        if constexpr (sizeof(T) == 8) uk = (typename S::Bits)__double_as_longlong(a.old[c]);
        else uk = __float_as_uint(a.old[c]);
      }
    };
#pragma unroll
    for (int c = 0; c < FLOW_CHUNKS; ++c) load(32 * c, v[c], at[c], u[c][0]);
    const T d = a.val[m.r0 + m.d], bi = a.b[m.row], self = a.old[m.row];
    next = take();
    T sum = 0;
    if constexpr (TREE) {
      const int nq = m.r0 + max(m.newest, 0);
      const T nv = m.newest >= 0 ? a.val[nq] : (T)0;
      const int nc = m.newest >= 0 ? a.col[nq] : -1;
      const T w = a.omega / d;
#pragma unroll
      for (int c = 0; c < FLOW_CHUNKS; ++c) {
        await<T, SMEM>(u[c], &at[c], fresh, m.row, a.err);
        sum = fmaf(v[c], from_bits(u[c][0]), sum);
      }
      for (int q0 = 32 * FLOW_CHUNKS; q0 < m.len; q0 += 32) {
        load(q0, v[0], at[0], u[0][0]);
        await<T, SMEM>(u[0], &at[0], fresh, m.row, a.err);
        sum = fmaf(v[0], from_bits(u[0][0]), sum);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(ALL, sum, o);
      const T rest = fmaf(w, bi - sum, self - a.omega * self);
      typename S::Bits last[1] = {nc >= 0 ? S::bits : 0};
      await<T, SMEM>(last, &nc, fresh, m.row, a.err);
      const typename S::Bits r = S::guard(fmaf(-(w * nv), from_bits(last[0]), rest));
      if (lane == 0) {
        Fresh<T, SMEM>::store(fresh + m.row, r);
        if (SMEM) a.out[m.row] = S::value(r);
      }
      __syncwarp();
      continue;
    }
    // a lane without an entry adds +0, which changes no sum (none is -0)
    auto add = [&](int q0, T vk, const int& ak, typename S::Bits (&uk)[1]) {
      await<T, SMEM>(uk, &ak, fresh, m.row, a.err);
      const T p = vk * from_bits(uk[0]);
      const T q = q0 + lane >= m.len || q0 + lane == m.d ? (T)0 : p;
      const int cnt = min(32, m.len - q0);
#pragma unroll 8
      for (int j = 0; j < cnt; ++j) sum += __shfl_sync(ALL, q, j);
    };
#pragma unroll
    for (int c = 0; c < FLOW_CHUNKS; ++c)
      if (32 * c < m.len) add(32 * c, v[c], at[c], u[c]);
    for (int q0 = 32 * FLOW_CHUNKS; q0 < m.len; q0 += 32) {
      load(q0, v[0], at[0], u[0][0]);
      add(q0, v[0], at[0], u[0]);
    }
    const T sigma = (bi - sum) / d;
    const typename S::Bits r = S::guard(self + a.omega * (sigma - self));
    if (lane == 0) {
      Fresh<T, SMEM>::store(fresh + m.row, r);
      if (SMEM) a.out[m.row] = S::value(r);
    }
    __syncwarp();
  }
}

// One level of a sweep, a thread per row.
template <bool BWD>
__global__ void __launch_bounds__(256) k_ssor_level(SsorArgs<double> a, int slice0, int slices) {
  chain_begin();
  if (a.active && *a.active != 0) return;
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
  if (q >= slices) return;
  const int s = slice0 + q, slot = s * 32 + lane, row = a.row[slot];
  if (row < 0) return;
  const int base = a.slice_base[s] + lane, len = a.len[slot];
  double sum = 0;
#pragma unroll 8
  for (int k = 0; k < len; ++k) {
    const int c = a.scol[base + 32 * k];
    sum += a.val[base + 32 * k] * ((BWD ? c > row : c < row) ? a.out[c] : a.old[c]);
  }
  const double sigma = (a.b[row] - sum) / a.diag[slot], self = a.old[row];
  a.out[row] = self + a.omega * (sigma - self);
}

template <typename T>
__global__ void k_flow_reset(int n, T* out, unsigned* ticket, const int* active) {
  chain_begin();
  if (active && *active != 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = Sentinel<T>::value(Sentinel<T>::bits);
  if (i == 0) *ticket = 0;
}

__global__ void k_flow_f32(int nnz, const double* __restrict__ a, float* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nnz) b[i] = (float)a[i];
}

// The slices of a sweep plan.
template <typename T>
void slice_args(SsorArgs<T>& a, const SweepPlan& P) {
  if constexpr (sizeof(T) == 8) {
    a.val = P.val.get();
    a.diag = P.diag.get();
  } else {
    a.val = P.valf.get();
    a.diag = P.diagf.get();
  }
  a.nslices = P.nslices;
  a.slice_base = P.slice_base.get();
  a.row = P.row.get();
  a.len = P.len.get();
  a.scol = P.col.get();
}

template <bool BWD>
void launch_slices(Context& ctx, const char* name, const SsorArgs<float>& a) {
  static PerDevice allowed;
  allow_smem(allowed, ctx, k_ssor_slices<float, BWD>, FLOW_SMEM);
  launch_chained(ctx, name, k_ssor_slices<float, BWD>, 1, FLOW_SLICE_THREADS, sizeof(float) * a.n, a);
}

template <bool BWD>
void launch_levels(Context& ctx, const char* name, const SsorArgs<double>& a, const SweepPlan& P) {
  for (int l = 0; l < P.nlev; ++l) {
    const int s0 = P.h_level_slices[l], slices = P.h_level_slices[l + 1] - s0;
    launch_chained(ctx, name, k_ssor_level<BWD>, blocks_for(slices, 8), 256, 0, a, s0, slices);
  }
}

template <typename T, bool BWD>
void launch_rows(Context& ctx, const char* name, const SsorArgs<T>& a, bool one) {
  if (one) {
    static PerDevice allowed;
    allow_smem(allowed, ctx, k_ssor_rows<T, BWD, true>, FLOW_SMEM);
    launch_chained(ctx, name, k_ssor_rows<T, BWD, true>, 1, FLOW_ROW_THREADS, sizeof(T) * a.n, a);
    return;
  }
  launch_chained(ctx, name, k_flow_reset<T>, blocks_for(a.n, 256), 256, 0, a.n, a.out, a.ticket, a.active);
  const int grid = std::min(ctx.num_sms, blocks_for((int64_t)a.n * 32, FLOW_ROW_THREADS));
  launch_chained(ctx, name, k_ssor_rows<T, BWD, false>, grid, FLOW_ROW_THREADS, 0, a);
}

}  // namespace

void SsorFlow::plan(Csr& M, const SweepPlan& fwd, const SweepPlan& bwd) {
  ctx = M.ctx;
  A = &M;
  plans[0] = &fwd;
  plans[1] = &bwd;
  int widest = 0;  // longest row, without its diagonal
  for (int k = 0; k < M.n; ++k) widest = std::max(widest, M.h_rowptr[k + 1] - M.h_rowptr[k] - 1);
  slices = widest <= FLOW_WIDTH && sizeof(float) * (size_t)M.n <= FLOW_SMEM;
  const bool wide = widest > 32 * FLOW_CHUNKS;
  for (int u = 0; u < 2; ++u) {
    const int64_t nlev = plans[u]->nlev;
    levels[u] = !wide && (nlev <= 2 || M.n >= FLOW_MANY * nlev);
    few[u] = !wide && M.n <= FLOW_FEW * nlev && sizeof(double) * (size_t)M.n <= FLOW_SMEM;
    if (levels[u] && slices) continue;  // no sweep by rows
    const std::vector<int>& o = plans[u]->h_order;
    order[u].resize(std::max<size_t>(o.size(), 1));
    RSG_CUDA(cudaMemcpyAsync(order[u].get(), o.data(), sizeof(int) * o.size(), cudaMemcpyHostToDevice, ctx->stream));
    if (slices) continue;
    // the entry of the highest level of each row, of several the one nearest
    // the diagonal (on a grid it is computed last)
    std::vector<int> lev(M.n, 0), entry(std::max(M.n, 1), -1);
    for (int row : o) {
      const int r0 = M.h_rowptr[row], d = M.h_diag[row], r1 = M.h_rowptr[row + 1];
      int top = -1;
      for (int q = u ? r1 - 1 : r0; u ? q > d : q < d; u ? --q : ++q)
        if (lev[M.h_col[q]] >= top) {
          top = lev[M.h_col[q]];
          entry[row] = q - r0;
        }
      lev[row] = top + 1;
    }
    newest[u].resize(entry.size());
    RSG_CUDA(cudaMemcpyAsync(newest[u].get(), entry.data(), sizeof(int) * entry.size(), cudaMemcpyHostToDevice,
                             ctx->stream));
    ctx->sync();  // entry goes out of scope
  }
  ticket.resize(1);
}

void SsorFlow::values(const double* csr) {
  const size_t size = std::max(A->nnz, 1);
  if (!levels[0] || !levels[1]) {
    val.resize(size);
    RSG_CUDA(cudaMemcpyAsync(val.get(), csr, sizeof(double) * A->nnz, cudaMemcpyDeviceToDevice, ctx->stream));
  }
  if (!slices) {
    valf.resize(size);
    RSG_LAUNCH(*ctx, "flow_f32", k_flow_f32, blocks_for(A->nnz, 256), 256, 0, A->nnz, csr, valf.get());
  }
}

template <typename T>
void SsorFlow::sweep(bool backward, const T* b, const T* old, T* out, T omega, const int* active) {
  const int u = backward ? 1 : 0;
  const SweepPlan& P = *plans[u];
  const bool f32 = sizeof(T) == 4;
  const char* name = backward ? (f32 ? "ssor_bwd_f32" : "ssor_bwd") : (f32 ? "ssor_fwd_f32" : "ssor_fwd");
  SsorArgs<T> a{};
  a.n = A->n;
  a.b = b;
  a.old = old;
  a.out = out;
  a.omega = omega;
  a.active = active;
  a.err = ctx->dev_err.get();
  if (f32 ? slices : levels[u]) {
    slice_args(a, P);
    if constexpr (sizeof(T) == 4) {
      if (backward) launch_slices<true>(*ctx, name, a);
      else launch_slices<false>(*ctx, name, a);
    } else {
      if (backward) launch_levels<true>(*ctx, name, a, P);
      else launch_levels<false>(*ctx, name, a, P);
    }
    return;
  }
  if constexpr (sizeof(T) == 8) a.val = val.get();
  else a.val = valf.get();
  a.order = order[u].get();
  a.newest = newest[u].get();
  a.rowptr = A->rowptr.get();
  a.col = A->col.get();
  a.dpos = A->diag.get();
  a.ticket = ticket.get();
  const bool one = f32 ? a.n <= FLOW_ROWS_MAX : few[u];
  if (backward) launch_rows<T, true>(*ctx, name, a, one);
  else launch_rows<T, false>(*ctx, name, a, one);
}

template void SsorFlow::sweep<double>(bool, const double*, const double*, double*, double, const int*);
template void SsorFlow::sweep<float>(bool, const float*, const float*, float*, float, const int*);

}  // namespace rsg
