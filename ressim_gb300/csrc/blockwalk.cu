// Block walks (see blockwalk.cuh): planner, host check, kernel.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <random>
#include <unordered_map>

#include "blockwalk.cuh"
#include "dataflow.cuh"

namespace rsg {

// ---------------------------------------------------------------- planning --
namespace {

// Line length and plane size of a grid in natural order, from the offsets
// most rows have: {1}, {line - 1 .. line + 1}, {plane - ... .. plane + ...}.
// Zero when the pattern is not one.
void grid_shape(int n, const std::vector<int>& rp, const std::vector<int>& cl, int& line, int& plane) {
  line = plane = 0;
  // Candidates: offsets that a tenth of 512 rows have, taken at random (an
  // offset of three in ten rows is missed by none of 10^20 draws); then counted
  // in all rows.  Patterns of scattered columns have none and end here.
  constexpr int SAMPLE = 512;
  std::unordered_map<int, int> seen;
  std::mt19937 draw(1);
  for (int k = 0; k < SAMPLE; ++k) {
    const int i = (int)(draw() % (unsigned)n);
    for (int q = rp[i]; q < rp[i + 1] && cl[q] < i; ++q) seen[i - cl[q]]++;
  }
  std::vector<int> off;
  for (auto& f : seen)
    if (f.second >= SAMPLE / 10) off.push_back(f.first);
  std::sort(off.begin(), off.end());
  std::vector<int> freq(off.size(), 0);
  if (!off.empty())
    for (int i = 0; i < n; ++i) {
      size_t k = off.size();  // columns ascend: offsets descend
      for (int q = rp[i]; q < rp[i + 1] && cl[q] < i; ++q) {
        const int o = i - cl[q];
        while (k > 0 && off[k - 1] > o) --k;
        if (k > 0 && off[k - 1] == o) freq[--k]++;
      }
    }
  size_t kept = 0;
  for (size_t k = 0; k < off.size(); ++k)
    if (freq[k] >= 0.3 * n) off[kept++] = off[k];
  off.resize(kept);
  if (off.empty() || off[0] != 1) return;
  size_t q = 1;
  if (q >= off.size()) return;
  size_t e = q;
  while (e + 1 < off.size() && off[e + 1] - off[e] <= 2) ++e;
  const int l = (off[q] + off[e]) / 2;
  if (l < 4 || off[q] <= 2 || n % l) return;
  if (e + 1 == off.size()) {  // two dimensions
    line = l;
    plane = n;
    return;
  }
  const int p = (off[e + 1] + off.back()) / 2;
  if (p % l || n % p) return;
  line = l;
  plane = p;
}

// Block boundaries in positions of the solve order.  On a grid a block is up
// to 32 lines of one plane (a lane per line).  Planes of more lines are cut
// at lines j with j + k (k the plane) a multiple of the block's lines: line j
// reads line j + 1 of the plane before, which with cuts at the same j in
// every plane would lie in a block that itself waits for this block's
// predecessor, two hops between blocks per plane instead of one.
std::vector<int> block_bounds(int n, const std::vector<int>& rp, const std::vector<int>& cl) {
  std::vector<int> b{0};
  int line, plane;
  grid_shape(n, rp, cl, line, plane);
  if (line) {
    const int nj = plane / line, nk = n / plane;
    const int span = nj <= BW_LANES ? nj : nj + nk - 1;
    const int parts = (span + BW_LANES - 1) / BW_LANES, lines = (span + parts - 1) / parts;
    for (int k = 0; k < nk; ++k) {
      if (nj > BW_LANES)
        for (int m = 1; m * lines - k < nj; ++m)
          if (m * lines - k > 0) b.push_back(k * plane + (m * lines - k) * line);
      b.push_back((k + 1) * plane);
    }
    return b;
  }
  // no grid: about as many blocks as SMs, none smaller than 512 rows
  const int parts = std::max(1, std::min(144, n / 512));
  for (int s = 1; s <= parts; ++s) b.push_back((int)((int64_t)n * s / parts));
  return b;
}

}  // namespace

bool plan_block_walk(int n, const std::vector<int>& rp, const std::vector<int>& cl, const std::vector<int>& dg,
                     bool upper, HostBlockWalk& H) {
  if (n <= 0) return false;
  // positions run in solve order: row = position (lower) or n - 1 - position (upper)
  auto row_of = [&](int pos) { return upper ? n - 1 - pos : pos; };
  auto q0_of = [&](int r) { return upper ? dg[r] + 1 : rp[r]; };
  auto q1_of = [&](int r) { return upper ? rp[r + 1] : dg[r]; };
  const std::vector<int> bounds = block_bounds(n, rp, cl);
  const int nblk = (int)bounds.size() - 1;
  int64_t nnz = 0;
  int wmax = 0;
  for (int r = 0; r < n; ++r) {
    nnz += q1_of(r) - q0_of(r);
    wmax = std::max(wmax, q1_of(r) - q0_of(r));
  }
  if (wmax > BW_WIDTH_MAX) return false;
  // a block's rows in the order of their dependency depth
  std::vector<int> blk(n), t(n);
  for (int b = 0; b < nblk; ++b)
    for (int p = bounds[b]; p < bounds[b + 1]; ++p) blk[p] = b;
  for (int p = 0; p < n; ++p) {
    const int r = row_of(p);
    int L = 0;
    for (int q = q0_of(r); q < q1_of(r); ++q) L = std::max(L, t[row_of(cl[q])] + 1);  // the map is its own inverse
    t[p] = L;
  }
  // steps
  std::vector<int> order(n), step(n), lane(n);
  H.nblk = nblk;
  H.blk_step.assign(nblk + 1, 0);
  int ns = 0;
  for (int b = 0; b < nblk; ++b) {
    const int p0 = bounds[b], p1 = bounds[b + 1];
    for (int p = p0; p < p1; ++p) order[p] = p;
    std::stable_sort(order.begin() + p0, order.begin() + p1, [&](int x, int y) { return t[x] < t[y]; });
    int fill = 0;
    for (int k = p0; k < p1; ++k) {
      if (k == p0) fill = 0;
      else if (fill == BW_LANES || t[order[k]] != t[order[k - 1]]) {
        ++ns;
        fill = 0;
      }
      step[order[k]] = ns;
      lane[order[k]] = fill++;
    }
    ++ns;
    H.blk_step[b + 1] = ns;
    if ((int64_t)ns * BW_LANES > 4 * (int64_t)n + (int64_t)8 * 1024 * 1024) return false;
  }
  // values of other blocks (or own ones older than the own window): fetched
  // at the step that first needs them, kept for AGE steps
  for (int age : {24, 12, 6, 3, 0}) {
    H.hptr.assign(ns + 1, 0);
    H.hsrc.clear();
    std::vector<int> at(n, -1), at_step(n, -1), at_blk(n, -1);
    std::vector<int> hidx(nnz), age_of(nnz);  // halo position (in its block) of each term, -1: own window; age in steps
    std::vector<int> rows_at((size_t)ns * BW_LANES, -1);
    for (int p = 0; p < n; ++p) rows_at[(size_t)step[p] * BW_LANES + lane[p]] = p;
    std::vector<int64_t> base(n + 1, 0);
    for (int p = 0; p < n; ++p) base[p + 1] = base[p] + q1_of(row_of(p)) - q0_of(row_of(p));
    int need = 1;
    for (int b = 0; b < nblk; ++b) {
      const size_t h0 = H.hsrc.size();
      for (int s = H.blk_step[b]; s < H.blk_step[b + 1]; ++s) {
        for (int l = 0; l < BW_LANES; ++l) {
          const int p = rows_at[(size_t)s * BW_LANES + l];
          if (p < 0) continue;
          const int r = row_of(p), q0 = q0_of(r), q1 = q1_of(r);
          for (int q = q0; q < q1; ++q) {
            const int d = row_of(cl[q]);
            if (blk[d] == b && s - step[d] < BW_OWN) {
              hidx[base[p] + q - q0] = -1;
              age_of[base[p] + q - q0] = s - step[d];
              continue;
            }
            if (at_blk[d] != b || s - at_step[d] > age) {
              at_blk[d] = b;
              at_step[d] = s;
              at[d] = (int)(H.hsrc.size() - h0);
              H.hsrc.push_back(step[d] * BW_LANES + lane[d]);
            }
            hidx[base[p] + q - q0] = at[d];
            age_of[base[p] + q - q0] = s - at_step[d];
          }
        }
        H.hptr[s + 1] = (int)H.hsrc.size();
      }
      // values alive at step s: those of steps s - age .. s + stages - 1
      for (int s = H.blk_step[b]; s < H.blk_step[b + 1]; ++s) {
        const int lo = std::max(H.blk_step[b], s - age), hi = std::min(H.blk_step[b + 1], s + BW_STAGES_MAX);
        need = std::max(need, H.hptr[hi] - H.hptr[lo]);
      }
    }
    int cap = 32;
    while (cap < need) cap *= 2;
    if (cap > BW_HALO_MAX) continue;
    H.halo = cap;
    // Phases (see BwWidths).  Each is as long as the longest row of a step,
    // so a row with more early terms than most (a block's first line, whose
    // neighbouring line is another block's) has some of them in the room its
    // later phases leave.
    auto phase = [&](int64_t e) {
      if (hidx[e] >= 0) return age_of[e] >= BW_NEW ? 0 : 1;
      return age_of[e] >= BW_OLD ? 0 : age_of[e] >= 2 ? 2 : 3;
    };
    int cmax[4] = {0, 0, 0, 1}, longest = 1;
    auto count = [&](int p, int* c) {
      c[0] = c[1] = c[2] = c[3] = 0;
      for (int64_t e = base[p]; e < base[p + 1]; ++e) c[phase(e)]++;
    };
    int c[4];
    for (int p = 0; p < n; ++p) {
      count(p, c);
      cmax[2] = std::max(cmax[2], c[2]);
      cmax[3] = std::max(cmax[3], c[3]);
      longest = std::max(longest, (int)(base[p + 1] - base[p]));
    }
    for (int p = 0; p < n; ++p) {
      count(p, c);
      cmax[1] = std::max(cmax[1], c[1] - (cmax[2] - c[2]) - (cmax[3] - c[3]));
    }
    H.w.last = cmax[3];
    H.w.pre = cmax[2];
    H.w.fresh = cmax[1];
    H.w.old = std::max(0, longest - cmax[1] - cmax[2] - cmax[3]);
    const int W = H.w.total();
    if (W > BW_WIDTH_MAX) return false;
    if ((int64_t)ns * BW_LANES * W > 4 * nnz + (int64_t)8 * 1024 * 1024) return false;
    if ((int64_t)ns * BW_LANES * W > INT32_MAX) return false;
    const int IB = H.w.index_bytes(), zero = BW_OWN * BW_LANES + H.halo;
    const size_t per = IB + 256 + (size_t)(W + 1) * 256 + 512, fixed = (size_t)(zero + 2) * 8;
    H.stages = BW_STAGES_MAX * per + fixed <= BW_SMEM_MAX ? BW_STAGES_MAX : BW_STAGES_MIN;
    if (H.stages * per + fixed > BW_SMEM_MAX) return false;
    H.idx.assign((size_t)ns * IB / 2, (unsigned short)zero);
    H.rows.assign((size_t)ns * BW_LANES, -1);
    H.src.assign((size_t)ns * BW_LANES * W, -1);
    H.own_old = false;
    const int first[5] = {0, H.w.old, H.w.old + H.w.fresh, W - H.w.last, W};
    std::vector<std::pair<int, int>> terms[4];  // (-age, position)
    for (int s = 0; s < ns; ++s) {
      unsigned short* idx = H.idx.data() + (size_t)s * IB / 2;
      int* rows = H.rows.data() + (size_t)s * BW_LANES;
      for (int l = 0; l < BW_LANES; ++l) {
        const int p = rows_at[(size_t)s * BW_LANES + l];
        if (p < 0) continue;
        rows[l] = row_of(p);
        const int r = row_of(p), q0 = q0_of(r), q1 = q1_of(r);
        for (auto& t : terms) t.clear();
        for (int u = 0; u < q1 - q0; ++u) {
          const int q = upper ? q1 - 1 - u : q0 + u;  // both triangles sum far columns first
          terms[phase(base[p] + q - q0)].push_back({-age_of[base[p] + q - q0], q});
        }
        // oldest operands first within a phase; what exceeds a phase moves to
        // a later one with room, oldest first
        for (int f = 0; f < 4; ++f) {
          std::stable_sort(terms[f].begin(), terms[f].end(), [](auto& x, auto& y) { return x.first < y.first; });
          const int room = first[f + 1] - first[f];
          for (int to = f + 1; to < 4 && (int)terms[f].size() > room; ++to)
            while ((int)terms[f].size() > room && (int)terms[to].size() < first[to + 1] - first[to]) {
              terms[to].insert(terms[to].begin(), {-(1 << 20), terms[f].front().second});
              terms[f].erase(terms[f].begin());
            }
          if ((int)terms[f].size() > room) return false;
          for (int u = 0; u < (int)terms[f].size(); ++u) {
            const int q = terms[f][u].second, k = first[f] + u;
            const int64_t e = base[p] + q - q0;
            const int d = row_of(cl[q]);
            if (f < 2 && hidx[e] < 0) H.own_old = true;
            idx[H.w.index_at(k, l)] =
                (unsigned short)(hidx[e] >= 0 ? BW_OWN * BW_LANES + (hidx[e] & (H.halo - 1))
                                              : ((step[d] - H.blk_step[blk[p]]) & (BW_OWN - 1)) * BW_LANES + lane[d]);
            H.src[((size_t)s * W + k) * BW_LANES + l] = q;
          }
        }
      }
    }
    return true;
  }
  return false;
}

std::string check_block_walk(int n, const std::vector<int>& rp, const std::vector<int>& cl,
                             const std::vector<int>& dg, bool upper, const HostBlockWalk& H) {
  // synthetic coefficients and right-hand side, exact in double
  auto coef = [](int q) { return (double)(q % 5 - 2); };
  auto rhs = [](int r) { return (double)(r % 7 + 1); };
  const double STALE = std::nan("");
  auto mod = [](double v) { return std::fmod(v, 1021.0); };  // keeps every value a small whole number
  std::vector<double> ref(n), x(H.steps() * (size_t)BW_LANES, STALE);  // x: the exchange array
  for (int p = 0; p < n; ++p) {
    const int r = upper ? n - 1 - p : p;
    double v = rhs(r);
    for (int q = upper ? dg[r] + 1 : rp[r]; q < (upper ? rp[r + 1] : dg[r]); ++q) v -= coef(q) * ref[cl[q]];
    ref[r] = mod(v);
  }
  const int ns = H.steps(), W = H.w.total();
  if ((int)H.blk_step.size() != H.nblk + 1 || (int)H.hptr.size() != ns + 1) return "step arrays";
  if (H.hptr[ns] != (int)H.hsrc.size()) return "halo arrays";
  const int IB = H.w.index_bytes(), zero = BW_OWN * BW_LANES + H.halo;
  if (H.idx.size() != (size_t)ns * IB / 2 || H.rows.size() != (size_t)ns * BW_LANES) return "index arrays";
  if (H.src.size() < (size_t)ns * W * BW_LANES) return "source array";
  if (H.halo & (H.halo - 1) || H.halo > BW_HALO_MAX || (H.stages != BW_STAGES_MIN && H.stages != BW_STAGES_MAX))
    return "window sizes";
  std::vector<double> own(BW_OWN * BW_LANES), halo(H.halo);
  std::vector<int> halo_step(H.halo, -1);
  std::vector<int> own_step(BW_OWN * BW_LANES);
  std::vector<char> seen(n, 0);
  for (int b = 0; b < H.nblk; ++b) {
    const int s0 = H.blk_step[b], s1 = H.blk_step[b + 1];
    if (s1 < s0) return "step order";
    std::fill(own.begin(), own.end(), STALE);
    std::fill(own_step.begin(), own_step.end(), -1);
    std::fill(halo.begin(), halo.end(), STALE);
    int fetched = s0;
    for (int s = s0; s < s1; ++s) {
      // the fetch warps may be `stages` steps ahead; a value that does not
      // exist yet is polled and lands by the time of its own step
      for (; fetched < std::min(s1, s + H.stages); ++fetched)
        for (int e = H.hptr[fetched]; e < H.hptr[fetched + 1]; ++e) {
          if (H.hsrc[e] < 0 || H.hsrc[e] >= s1 * BW_LANES) return "halo slot out of range";
          halo[(e - H.hptr[s0]) & (H.halo - 1)] = x[H.hsrc[e]];
        }
      for (int e = H.hptr[s]; e < H.hptr[s + 1]; ++e) {
        if (std::isnan(x[H.hsrc[e]])) return "value needed before it exists";
        halo[(e - H.hptr[s0]) & (H.halo - 1)] = x[H.hsrc[e]];
        halo_step[(e - H.hptr[s0]) & (H.halo - 1)] = s;
      }
      const unsigned short* idx = H.idx.data() + (size_t)s * IB / 2;
      const int* rows = H.rows.data() + (size_t)s * BW_LANES;
      double out[BW_LANES];
      for (int l = 0; l < BW_LANES; ++l) {
        const int r = rows[l];
        if (r < -1 || r >= n) return "row out of range";
        if (r >= 0) {
          if (seen[r]) return "row placed twice";
          seen[r] = 1;
        }
        const int q0 = r < 0 ? 0 : upper ? dg[r] + 1 : rp[r], q1 = r < 0 ? 0 : upper ? rp[r + 1] : dg[r];
        int terms = 0;
        double v = r < 0 ? 0 : rhs(r);
        for (int k = 0; k < W; ++k) {
          const int i = idx[H.w.index_at(k, l)], q = H.src[((size_t)s * W + k) * BW_LANES + l];
          if (i > zero) return "index out of range";
          if ((i == zero) != (q < 0)) return "term without an operand";
          if (q < 0) continue;
          if (q < q0 || q >= q1) return "term of another row";
          ++terms;
          double xv;
          if (i < BW_OWN * BW_LANES) {
            xv = own[i];
            const int age = s - own_step[i];
            if (age < 1 || age >= BW_OWN) return "own value outside its window";
            if (k < H.w.old + H.w.fresh ? !H.own_old || age < BW_OLD : k < W - H.w.last && age < 2)
              return "operand too young for its phase";
          } else {
            xv = halo[i - BW_OWN * BW_LANES];
            if (k < H.w.old && s - halo_step[i - BW_OWN * BW_LANES] < BW_NEW) return "value too new for its phase";
          }
          if (!(xv == ref[cl[q]])) return "operand is not the column's value";
          v -= coef(q) * xv;
        }
        if (terms != q1 - q0) return "row length";
        if (r < 0) continue;
        out[l] = mod(v);
        if (out[l] != ref[r]) return "row value";
      }
      for (int l = 0; l < BW_LANES; ++l) {
        const int i = ((s - s0) & (BW_OWN - 1)) * BW_LANES + l;
        own_step[i] = s;
        own[i] = STALE;
        if (rows[l] >= 0) own[i] = x[(size_t)s * BW_LANES + l] = out[l];
      }
    }
  }
  for (int i = 0; i < n; ++i)
    if (!seen[i]) return "row missing";
  return "";
}

// ----------------------------------------------------------------- kernel --
namespace {

// Warps of a CTA.  The chain's warp has sub-partition 0 (warp % 4) to itself:
// its loop is bound by its own instructions, and other warps would take its
// issue slots (warps 4, 8, ... end at once).  The others by their number
// among the remaining ones: early warps, some that stage coefficients, the
// ones that fetch other blocks' values (a fetch takes about 700 cycles, so
// that many are in flight).
constexpr int BW_EARLY = 6;
constexpr int BW_STREAM = 4;
constexpr int BW_FETCH = 8;
constexpr int BW_THREADS = 32 * (BW_EARLY + BW_STREAM + BW_FETCH) / 3 * 4;

struct BlockWalkArgs {
  const int* blk_step;
  const int* hptr;
  const int* hsrc;
  const unsigned char* ints;
  const int* bsrc;  // per slot: where the right-hand side is (lower: the row, upper: the lower walk's exchange slot)
  BwWidths w;
  int nblk, halo, own_old;
  unsigned* ticket;
  int* err;
};

__device__ __forceinline__ unsigned bw_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// One thread's copy of a contiguous piece (16-byte aligned and sized), counted
// in bytes on the barrier.
__device__ __forceinline__ void cp_bulk(void* dst, const void* src, int bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   bw_addr(dst)),
               "l"(src), "r"(bytes), "r"(bw_addr(bar))
               : "memory");
}

__device__ __forceinline__ void cp_value(double* dst, const double* src, bool have) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(bw_addr(dst)), "l"(src), "r"(have ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_value(float* dst, const float* src, bool have) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(bw_addr(dst)), "l"(src), "r"(have ? 4 : 0) : "memory");
}

// Barriers between the warps of a CTA, one of each kind per stage: a step's
// coefficients are staged, so are the values it reads (and those of every
// step before), its early sums are there, it is done.  The phase of
// step s at its stage is s / stages.  A wait tells one phase from the one
// before only, so none may miss a phase: the next one at the stage must need
// the waiting warp first.  (That is why a stage is refilled BW_NEW steps
// later than it could be: an early warp at step s still asks for full[s -
// BW_NEW].)
struct BwBars {
  unsigned long long coef[BW_STAGES_MAX], full[BW_STAGES_MAX], part[BW_STAGES_MAX], done[BW_STAGES_MAX];
};

// try_wait wakes a waiting warp 173 cycles after the other side's arrival,
// spinning on test_wait 260, on a flag in shared memory 364.
__device__ __forceinline__ bool bw_test(const unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bw_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool bw_try(const unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bw_addr(bar)), "r"(parity)
      : "memory");
  return __all_sync(0xffffffffu, ok);
}
// Waits for a phase, the whole warp together.  False when the wait is given
// up: the walk has then failed, and the warp ends at once, because what it
// waited for (staged indices among it) is not there to be used.  The warps
// that wait for this one in turn give up by the error that is set.
__device__ __forceinline__ bool bw_wait(const unsigned long long* bar, unsigned parity, int* err) {
  unsigned long long start = 0;
  for (int i = 1;; ++i) {
    if (bw_try(bar, parity)) return true;
    if ((i & 255) == 0 && __any_sync(0xffffffffu, wait_over(start, err))) {
      atomicCAS(err, 0, 1);
      return false;
    }
  }
}
// Publishes the calling warp's shared-memory accesses to the waiters.  Lane
// 0's arrival is predicated rather than branched on: lanes running ahead of a
// branch into a wait that depends on this very arrival could starve it.
__device__ __forceinline__ void bw_arrive(unsigned long long* bar, int lane) {
  __syncwarp();
  asm volatile(
      "{\n .reg .pred p;\n setp.eq.s32 p, %1, 0;\n @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(bw_addr(bar)),
      "r"(lane)
      : "memory");
}

// Term offsets of a lane: four indices at a time.
struct alignas(8) BwIdx {
  unsigned short i[4];
};

// v - the sum of N terms: coefficients val[0], val[32], ..., operands by index.
template <int N, typename T>
__device__ __forceinline__ T bw_sub(T v, const T* val, const BwIdx& ix, const T* xs) {
  T a[N], x[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    a[q] = val[q * 32];
    x[q] = xs[ix.i[q]];
  }
#pragma unroll
  for (int q = 0; q < N; ++q) v = fma(-a[q], x[q], v);
  return v;
}

// v - the sum of n terms, in groups of four; lanes with fewer terms hold
// zeros (times the zero slot), and the groups' lengths follow n exactly: a
// term costs its pipe time with or without active lanes.
template <typename T>
__device__ __forceinline__ T bw_terms(T v, const T* val, const BwIdx* idx, const T* xs, int n) {
  if (n <= 0) return v;
  BwIdx ix = idx[0];
#pragma unroll 1
  for (; n > 4; n -= 4) {
    const BwIdx nx = idx[32];
    v = bw_sub<4>(v, val, ix, xs);
    ix = nx;
    idx += 32;
    val += 4 * 32;
  }
  if (n == 4) return bw_sub<4>(v, val, ix, xs);
  if (n == 3) return bw_sub<3>(v, val, ix, xs);
  if (n == 2) return bw_sub<2>(v, val, ix, xs);
  return bw_sub<1>(v, val, ix, xs);
}

// The staged step in shared memory: integers (operand indices, the
// right-hand-side indices of the step BW_BACK later, upper: rows),
// coefficients, right-hand side, early sums.
__host__ __device__ inline int bw_int_bytes(const BwWidths& w, bool upper) { return w.index_bytes() + (upper ? 256 : 128); }
template <typename T>
struct BwStage {
  int IS, VS, SS;
  __device__ __forceinline__ BwStage(const BwWidths& w, bool upper)
      : IS(bw_int_bytes(w, upper)),
        VS((w.total() + (upper ? 1 : 0)) * 32 * (int)sizeof(T)),
        SS(IS + VS + 64 * (int)sizeof(T)) {}
};

// The chain.  NP pre and NL last terms (both at most two).  A step's early
// sum, indices and coefficients come into registers two steps ahead, if they
// are there by then.  A double-precision term holds the pipe for 64 cycles,
// as long as the next dependent one waits for it, so the pre terms of the
// next step go between the last terms of this one and under its exchange
// through shared memory.
template <typename T, int NP, int NL>
struct BwTerms {
  T v, ap[NP ? NP : 1], al[NL];
  BwIdx ix;
};

template <typename T, int NP, int NL, int D>
__device__ __forceinline__ void bw_chain(const BlockWalkArgs& g, const BwStage<T>& z, unsigned char* smem, T* xs,
                                         BwBars& bars, T* ex, int nst, int lane) {
  using S = Sentinel<T>;
  static_assert(NP <= 2 && NL >= 1 && NL <= 2, "one index group");
  using Terms = BwTerms<T, NP, NL>;
  const int io = g.w.early_groups() * 256 + lane * 8, vo = z.IS + ((g.w.old + g.w.fresh) * 32 + lane) * (int)sizeof(T),
            po = z.IS + z.VS + (32 + lane) * (int)sizeof(T);
  auto load = [&](Terms& t, int s) {
    const unsigned char* sp = smem + (s & (D - 1)) * z.SS;
    t.v = *reinterpret_cast<const T*>(sp + po);
    t.ix = *reinterpret_cast<const BwIdx*>(sp + io);
    const T* val = reinterpret_cast<const T*>(sp + vo);
#pragma unroll
    for (int q = 0; q < NP; ++q) t.ap[q] = val[q * 32];
#pragma unroll
    for (int q = 0; q < NL; ++q) t.al[q] = val[(NP + q) * 32];
  };
  auto there = [&](int s) {
    return (bool)__all_sync(0xffffffffu, bw_test(&bars.part[s & (D - 1)], s / D & 1));
  };
  auto publish = [&](int s, T v) {
    bw_arrive(&bars.done[s & (D - 1)], lane);
    S::store(ex + s * BW_LANES, S::guard(v));  // idle lanes' slots are never read
  };
  // A's last step alone
  auto finish = [&](const Terms& A, int s) {
    T v = A.v;
#pragma unroll
    for (int q = 0; q < NL; ++q) v = fma(-A.al[q], xs[A.ix.i[NP + q]], v);
    xs[(s & (BW_OWN - 1)) * BW_LANES + lane] = v;
    publish(s, v);
  };
  // step s from A (its pre terms done), the pre terms of B (step s + 1), and
  // C for step s + 2 if it is there.  The three trade places from step to
  // step instead of being copied: a copy of a sum would wait for its term.
  auto step = [&](const Terms& A, Terms& B, Terms& C, int s) {
    T x[NL], xp[NP ? NP : 1];
#pragma unroll
    for (int q = 0; q < NL; ++q) x[q] = xs[A.ix.i[NP + q]];
#pragma unroll
    for (int q = 0; q < NP; ++q) xp[q] = xs[B.ix.i[q]];
    const bool more = there(s + 2);
    if (more) load(C, s + 2);
    T v = fma(-A.al[0], x[0], A.v);
    if (NP > 0) B.v = fma(-B.ap[0], xp[0], B.v);
    if (NL > 1) v = fma(-A.al[NL - 1], x[NL - 1], v);
    xs[(s & (BW_OWN - 1)) * BW_LANES + lane] = v;
    if (NP > 1) B.v = fma(-B.ap[NP - 1], xp[NP - 1], B.v);
    publish(s, v);
    return more;
  };
  Terms a, b, c;
#pragma unroll 1
  for (int s = 0; s < nst;) {
    if (!bw_wait(&bars.part[s & (D - 1)], s / D & 1, g.err)) return;
    load(a, s);
#pragma unroll
    for (int q = 0; q < NP; ++q) a.v = fma(-a.ap[q], xs[a.ix.i[q]], a.v);
    if (!there(s + 1)) {
      finish(a, s++);
      continue;
    }
    load(b, s + 1);
#pragma unroll 1
    for (;;) {
      if (!step(a, b, c, s++)) {
        finish(b, s++);
        break;
      }
      if (!step(b, c, a, s++)) {
        finish(c, s++);
        break;
      }
      if (!step(c, a, b, s++)) {
        finish(a, s++);
        break;
      }
    }
  }
}

// The chain of patterns with more terms of recent operands.
template <typename T, int D>
__device__ __forceinline__ void bw_chain_wide(const BlockWalkArgs& g, const BwStage<T>& z, unsigned char* smem, T* xs,
                                              BwBars& bars, T* ex, int nst, int lane) {
  using S = Sentinel<T>;
#pragma unroll 1
  for (int s = 0; s < nst; ++s) {
    unsigned char* sp = smem + (s & (D - 1)) * z.SS;
    if (!bw_wait(&bars.part[s & (D - 1)], s / D & 1, g.err)) return;
    const T v = bw_terms(reinterpret_cast<const T*>(sp + z.IS + z.VS)[32 + lane],
                         reinterpret_cast<const T*>(sp + z.IS) + (g.w.old + g.w.fresh) * 32 + lane,
                         reinterpret_cast<const BwIdx*>(sp) + g.w.early_groups() * 32 + lane, xs, g.w.pre + g.w.last);
    xs[(s & (BW_OWN - 1)) * BW_LANES + lane] = v;
    bw_arrive(&bars.done[s & (D - 1)], lane);
    S::store(ex + s * BW_LANES, S::guard(v));
  }
}

// What the walks read and write.  The lower walk solves for b into one of the
// two arrays lex (the ticket's high bit says which) and readies uex; the
// upper one takes that array as its right-hand side, exchanges through uex,
// writes x and readies the other lower array.
template <typename T>
struct BlockWalkIo {
  const T* vals;
  const T* b;
  T* lex[2];
  T* uex;
  T* x;
  int lower_slots, upper_slots;
  const int* active;
};

template <typename T, bool UPPER, int D>
__global__ void __launch_bounds__(BW_THREADS, 1) k_block_walk(BlockWalkArgs g, BlockWalkIo<T> io) {
  chain_begin();
  if (io.active && *io.active != 0) return;
  using S = Sentinel<T>;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ BwBars bars;
  __shared__ unsigned sh_ticket;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const BwStage<T> z(g.w, UPPER);
  T* xs = reinterpret_cast<T*>(smem + (size_t)D * z.SS);
  T* hs = xs + BW_OWN * BW_LANES;
  if (threadIdx.x == 0) {
    // blocks in order; the launch's last ticket returns the counter to zero
    // and flips the lower exchange array in use (bit 31)
    const unsigned t = atomicAdd(g.ticket, 1u);
    if ((t & 0x7fffffffu) == (unsigned)g.nblk - 1) atomicExch(g.ticket, (t & 0x80000000u) ^ 0x80000000u);
    sh_ticket = t;
    hs[g.halo] = 0;  // the zero slot
  }
  if (threadIdx.x >= 32 && threadIdx.x < 32 + (int)(sizeof(BwBars) / 8))
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bw_addr(&bars) + 8 * (threadIdx.x - 32)),
                 "r"(threadIdx.x - 32 < BW_STAGES_MAX ? 33 : 1)  // coef: the bulk copies' issuer and every lane's own copy
                 : "memory");
  // the barriers' initialisation is visible to the bulk copies
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const int blk = (int)(sh_ticket & 0x7fffffffu), which = (int)(sh_ticket >> 31);
  const int s0 = g.blk_step[blk], nst = g.blk_step[blk + 1] - s0;
  T* lex = which ? io.lex[1] : io.lex[0];
  T* ex = UPPER ? io.uex : lex;
  if (warp == 0) {
    T* mine = ex + (size_t)s0 * BW_LANES + lane;
    if (g.w.pre == 2 && g.w.last == 2) bw_chain<T, 2, 2, D>(g, z, smem, xs, bars, mine, nst, lane);
    else if (g.w.pre == 0 && g.w.last == 2) bw_chain<T, 0, 2, D>(g, z, smem, xs, bars, mine, nst, lane);
    else if (g.w.pre == 0 && g.w.last == 1) bw_chain<T, 0, 1, D>(g, z, smem, xs, bars, mine, nst, lane);
    else bw_chain_wide<T, D>(g, z, smem, xs, bars, mine, nst, lane);
    return;
  }
  if ((warp & 3) == 0) return;
  const int role = warp - 1 - (warp >> 2);
  auto wait_done = [&](int s) { return bw_wait(&bars.done[s & (D - 1)], s / D & 1, g.err); };
  auto wait_coef = [&](int s) { return bw_wait(&bars.coef[s & (D - 1)], s / D & 1, g.err); };
  auto wait_full = [&](int s) { return bw_wait(&bars.full[s & (D - 1)], s / D & 1, g.err); };
  if (role < BW_EARLY) {
    for (int s = role; s < nst; s += BW_EARLY) {
      unsigned char* sp = smem + (s & (D - 1)) * z.SS;
      if (!wait_coef(s)) return;
      const T* val = reinterpret_cast<const T*>(sp + z.IS) + lane;
      const BwIdx* idx = reinterpret_cast<const BwIdx*>(sp) + lane;
      T* bp = reinterpret_cast<T*>(sp + z.IS + z.VS) + lane;
      T v = bp[0];
      if (UPPER) v *= val[g.w.total() * 32];
      if (s >= BW_NEW && !wait_full(s - BW_NEW)) return;
      if (g.own_old && s >= BW_OLD && !wait_done(s - BW_OLD)) return;
      v = bw_terms(v, val, idx, xs, g.w.old);
      if (!wait_full(s)) return;
      v = bw_terms(v, val + g.w.old * 32, idx + g.w.old_groups() * 32, xs, g.w.fresh);
      bp[32] = v;
      bw_arrive(&bars.part[s & (D - 1)], lane);
    }
  } else if (role < BW_EARLY + BW_STREAM) {
    const int f = role - BW_EARLY;
    // this block's share of the exchange array to ready for a later walk
    T* reset = UPPER ? (which ? io.lex[0] : io.lex[1]) : io.uex;
    const int64_t rn = UPPER ? io.lower_slots : io.upper_slots;
    const int r0 = (int)(rn * blk / g.nblk), r1 = (int)(rn * (blk + 1) / g.nblk), rs = (r1 - r0 + nst - 1) / max(nst, 1);
    const T* b = UPPER ? lex : io.b;
    // upper: the values of a step that is done go to x before its stage is refilled
    auto retire = [&](int s) {
      if (!UPPER) return;
      const int row = reinterpret_cast<const int*>(smem + (s & (D - 1)) * z.SS + g.w.index_bytes() + 128)[lane];
      const T v = xs[(s & (BW_OWN - 1)) * BW_LANES + lane];
      if (row >= 0) io.x[row] = v;
      __syncwarp();
    };
    bool ok = true;
    int s = f, issued = -1;
    for (; s < nst; s += BW_STREAM) {
      if (s >= D - BW_NEW && !(ok = wait_done(s - D + BW_NEW))) break;
      if (s >= D) retire(s - D);
      // Indices of the right-hand side: a load from global memory here, even
      // of several steps ahead, would have each step wait for it (loads of
      // one scoreboard are waited for together).
      int bi;
      if (s < BW_BACK) bi = g.bsrc[(size_t)(s0 + s) * BW_LANES + lane];
      else {
        if (!(ok = wait_coef(s - BW_BACK))) break;
        bi = reinterpret_cast<const int*>(smem + ((s - BW_BACK) & (D - 1)) * z.SS + g.w.index_bytes())[lane];
      }
      unsigned char* sp = smem + (s & (D - 1)) * z.SS;
      unsigned long long* bar = &bars.coef[s & (D - 1)];
      cp_value(reinterpret_cast<T*>(sp + z.IS + z.VS) + lane, b + max(bi, 0), bi >= 0);
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bw_addr(bar)) : "memory");
      __syncwarp();
      if (lane == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bw_addr(bar)), "r"(z.IS + z.VS)
                     : "memory");
        cp_bulk(sp, g.ints + (size_t)(s0 + s) * z.IS, z.IS, bar);
        cp_bulk(sp + z.IS, reinterpret_cast<const unsigned char*>(io.vals) + (size_t)(s0 + s) * z.VS, z.VS, bar);
      }
      issued = s;
      for (int r = r0 + s * rs + lane; r < min(r1, r0 + (s + 1) * rs); r += 32) S::store(reset + r, S::bits);
    }
    if (UPPER)
      for (; ok && s - D < nst; s += BW_STREAM)
        if (s >= D && (ok = wait_done(s - D))) retire(s - D);
    // The copies land before the CTA may end, also when the warps that use
    // them have given up.  Their barriers take this warp's arrivals alone, so
    // the wait has an end.
    for (int q = issued; q >= 0 && q > issued - D; q -= BW_STREAM)
      for (unsigned long long start = 0;;) {
        if (bw_try(&bars.coef[q & (D - 1)], q / D & 1)) break;
        if (__any_sync(0xffffffffu, time_over(start))) break;
      }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    const int f = role - BW_EARLY - BW_STREAM;
    const int hbase = g.hptr[s0];
    // indices of the next step are loaded ahead
    int h0_n = 0, h1_n = 0, hr_n[2] = {0, 0};
    auto ahead = [&](int s) {
      if (s >= nst) return;
      h0_n = g.hptr[s0 + s];
      h1_n = g.hptr[s0 + s + 1];
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (h0_n + lane + 32 * q < h1_n) hr_n[q] = g.hsrc[h0_n + lane + 32 * q];
    };
    ahead(f);
    for (int s = f; s < nst; s += BW_FETCH) {
      const int h0 = h0_n, h1 = h1_n;
      const int hr[2] = {hr_n[0], hr_n[1]};
      ahead(s + BW_FETCH);
      if (!wait_coef(s)) return;  // not ahead of the coefficients: the window is bounded
      for (int q = 0; h0 + 32 * q < h1; ++q) {
        const int h = h0 + lane + 32 * q;
        const bool mine = h < h1;
        const T* p = ex;
        if (mine) p += q == 0 ? hr[0] : q == 1 ? hr[1] : g.hsrc[h];
        typename S::Bits v = 0;
        if (mine) v = S::load(p);
        // the whole warp polls together: lanes that are done must not spin elsewhere
        unsigned long long start = 0;
        for (int i = 1; __any_sync(0xffffffffu, mine && v == S::bits); ++i) {
          if (mine && v == S::bits) v = S::load(p);
          if ((i & 255) == 0 && __any_sync(0xffffffffu, wait_over(start, g.err))) {
            atomicCAS(g.err, 0, 1 + s);
            return;
          }
        }
        if (mine) hs[(h - hbase) & (g.halo - 1)] = S::value(v);
      }
      // released in order: a step's operands may have been staged with an earlier step
      if (s > 0 && !wait_full(s - 1)) return;
      bw_arrive(&bars.full[s & (D - 1)], lane);
    }
  }
}

// One thread per slot of the walk: coefficients (upper: divided by the
// diagonal, with its reciprocal behind them), zeros on empty slots.  flag: bit
// 0 a scaled coefficient is not finite, bit 1 not finite in single precision.
template <typename T, bool UPPER>
__global__ void k_block_walk_values(int nslots, int W, const int* __restrict__ rows, const int* __restrict__ src, const double* __restrict__ lu,
                                    const int* __restrict__ diag, T* __restrict__ out, int* __restrict__ flag,
                                    const int* __restrict__ failed, const int* __restrict__ err) {
  if ((failed && *failed) || *err) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nslots) return;
  const int s = t >> 5, lane = t & 31;
  const int row = rows[t];
  T* o = out + (size_t)s * (W + (UPPER ? 1 : 0)) * 32 + lane;
  double scale = 1.0;
  int bad = 0;
  if (UPPER) {
    scale = row >= 0 ? 1.0 / lu[diag[row]] : 0.0;
    o[W * 32] = (T)scale;
    bad = (isfinite(scale) ? 0 : 1) | (isfinite((float)scale) ? 0 : 2);
  }
  for (int k = 0; k < W; ++k) {
    const int q = src[((size_t)s * W + k) * 32 + lane];
    double v = 0;
    if (q >= 0) {
      v = UPPER ? lu[q] * scale : lu[q];
      if (UPPER) bad |= (isfinite(v) ? 0 : 1) | (isfinite((float)v) ? 0 : 2);
    }
    o[k * 32] = (T)v;
  }
  if (UPPER && bad && flag) atomicOr(flag, bad);
}

void upload(Context& ctx, BlockWalk& P, const HostBlockWalk& H, const HostBlockWalk* lower, int n) {
  P.upper = lower != nullptr;
  P.nblk = H.nblk;
  P.w = H.w;
  P.halo = H.halo;
  P.stages = H.stages;
  P.nsteps = H.steps();
  P.own_old = H.own_old;
  auto up = [&](auto& dst, const auto& v) {
    dst.resize(std::max<size_t>(v.size(), 1));
    if (!v.empty())
      RSG_CUDA(cudaMemcpyAsync(dst.get(), v.data(), sizeof(v[0]) * v.size(), cudaMemcpyHostToDevice, ctx.stream));
  };
  std::vector<int> bsrc = H.rows;
  if (lower) {  // where the lower walk leaves each row's value
    std::vector<int> slot(n, -1);
    for (size_t q = 0; q < lower->rows.size(); ++q)
      if (lower->rows[q] >= 0) slot[lower->rows[q]] = (int)q;
    for (int& v : bsrc)
      if (v >= 0) v = slot[v];
  }
  // a step's integers as they are staged
  const int IB = P.w.index_bytes(), IS = bw_int_bytes(P.w, P.upper);
  std::vector<unsigned char> ints((size_t)P.nsteps * IS, 0xff);
  for (int b = 0; b < P.nblk; ++b)
    for (int s = H.blk_step[b]; s < H.blk_step[b + 1]; ++s) {
      unsigned char* o = ints.data() + (size_t)s * IS;
      std::memcpy(o, H.idx.data() + (size_t)s * IB / 2, IB);
      if (s + BW_BACK < H.blk_step[b + 1]) std::memcpy(o + IB, &bsrc[(size_t)(s + BW_BACK) * BW_LANES], 128);
      if (P.upper) std::memcpy(o + IB + 128, &H.rows[(size_t)s * BW_LANES], 128);
    }
  up(P.bsrc, bsrc);
  up(P.rows, H.rows);
  up(P.ints, ints);
  up(P.blk_step, H.blk_step);
  up(P.hptr, H.hptr);
  up(P.hsrc, H.hsrc);
  up(P.src, H.src);
  P.ticket.resize(1);
  ctx.sync();
}

template <typename T, bool UPPER, int D>
void launch(Context& ctx, const char* name, const BlockWalk& P, const BlockWalkIo<T>& io) {
  const size_t stage = bw_int_bytes(P.w, UPPER) + (size_t)(P.w.total() + (UPPER ? 1 : 0)) * 32 * sizeof(T) + 64 * sizeof(T);
  const size_t smem = D * stage + (size_t)(BW_OWN * BW_LANES + P.halo + 2) * sizeof(T);
  auto kern = k_block_walk<T, UPPER, D>;
  static PerDevice allowed;
  allow_smem(allowed, ctx, kern, BW_SMEM_MAX);
  const BlockWalkArgs g{P.blk_step.get(), P.hptr.get(), P.hsrc.get(), P.ints.get(), P.bsrc.get(), P.w, P.nblk, P.halo,
                        (int)P.own_old, P.ticket.get(), ctx.dev_err.get()};
  launch_chained(ctx, name, kern, P.nblk, BW_THREADS, smem, g, io);
}

}  // namespace

static std::atomic<bool> g_used{false};
bool block_walks_used() { return g_used.load(std::memory_order_relaxed); }

void BlockWalkPair::plan(Context* c, int n, const HostBlockWalk& hl, const HostBlockWalk& hu) {
  ctx = c;
  planned = false;
  if (!hl.nblk || !hu.nblk) return;
  upload(*ctx, L, hl, nullptr, n);
  upload(*ctx, U, hu, &hl, n);
  planned = true;
}

template <>
BlockWalkData<double>& BlockWalkPair::data<double>() { return d64; }
template <>
BlockWalkData<float>& BlockWalkPair::data<float>() { return d32; }

template <typename T>
void BlockWalkPair::values(const double* lu, const int* diag, int* flag, const int* failed) {
  BlockWalkData<T>& d = data<T>();
  d.lval.resize(std::max<size_t>(L.slots() * L.w.total(), 1));
  d.uval.resize(U.slots() * (U.w.total() + 1));
  RSG_LAUNCH(*ctx, "walk_values", (k_block_walk_values<T, false>), blocks_for(L.slots(), 256), 256, 0, (int)L.slots(),
             L.w.total(), L.rows.get(), L.src.get(), lu, diag, d.lval.get(), flag, failed, ctx->dev_err.get());
  RSG_LAUNCH(*ctx, "walk_values", (k_block_walk_values<T, true>), blocks_for(U.slots(), 256), 256, 0, (int)U.slots(),
             U.w.total(), U.rows.get(), U.src.get(), lu, diag, d.uval.get(), flag, failed, ctx->dev_err.get());
}

template <typename T>
void BlockWalkPair::begin() {
  BlockWalkData<T>& d = data<T>();
  auto fill = [&](DeviceBuffer<T>& x, size_t n) {
    x.resize(n);
    RSG_LAUNCH(*ctx, "walk_fill", k_sentinel<T>, blocks_for(n, 256), 256, 0, (int64_t)n, x.get());
  };
  fill(d.lex[0], L.slots());
  fill(d.lex[1], L.slots());
  fill(d.uex, U.slots());
  for (BlockWalk* w : {&L, &U}) RSG_CUDA(cudaMemsetAsync(w->ticket.get(), 0, sizeof(unsigned), ctx->stream));
}

template <typename T>
void BlockWalkPair::apply(const T* b, T* x, const int* active) {
  BlockWalkData<T>& d = data<T>();
  BlockWalkIo<T> io{d.lval.get(), b, {d.lex[0].get(), d.lex[1].get()}, d.uex.get(), x, (int)L.slots(), (int)U.slots(),
                    active};
  if (!block_walks_used()) g_used = true;
  const bool f32 = sizeof(T) == 4;
  const char *lname = f32 ? "ilu_lower_f32" : "ilu_lower", *uname = f32 ? "ilu_upper_f32" : "ilu_upper";
  if (L.stages == BW_STAGES_MAX) launch<T, false, BW_STAGES_MAX>(*ctx, lname, L, io);
  else launch<T, false, BW_STAGES_MIN>(*ctx, lname, L, io);
  io.vals = d.uval.get();
  if (U.stages == BW_STAGES_MAX) launch<T, true, BW_STAGES_MAX>(*ctx, uname, U, io);
  else launch<T, true, BW_STAGES_MIN>(*ctx, uname, U, io);
}

template void BlockWalkPair::values<double>(const double*, const int*, int*, const int*);
template void BlockWalkPair::values<float>(const double*, const int*, int*, const int*);
template void BlockWalkPair::begin<double>();
template void BlockWalkPair::begin<float>();
template void BlockWalkPair::apply<double>(const double*, double*, const int*);
template void BlockWalkPair::apply<float>(const float*, float*, const int*);

}  // namespace rsg

// Plans the block walk of one ILU(0) sweep of a pattern on the host and
// walks the plan there.  Needs no GPU.
extern "C" rsg_status rsg_block_walk_check(int32_t n, const int32_t* row_ptr, const int32_t* col, int32_t sweep,
                                           int64_t* stats, char* msg, int32_t msg_len) {
  auto say = [&](const std::string& m) {
    if (msg && msg_len > 0) {
      std::strncpy(msg, m.c_str(), (size_t)msg_len - 1);
      msg[msg_len - 1] = 0;
    }
  };
  if (n <= 0 || !row_ptr || !col || (sweep != 0 && sweep != 1) || row_ptr[0] != 0) return RSG_BAD_ARG;
  try {
    for (int i = 0; i < n; ++i)
      if (row_ptr[i + 1] < row_ptr[i]) return RSG_BAD_ARG;
    std::vector<int> rp(row_ptr, row_ptr + n + 1), cl(col, col + row_ptr[n]), dg(n, -1);
    for (int i = 0; i < n; ++i)
      for (int q = rp[i]; q < rp[i + 1]; ++q) {
        if (cl[q] < 0 || cl[q] >= n || (q > rp[i] && cl[q] <= cl[q - 1])) return RSG_BAD_ARG;
        if (cl[q] == i) dg[i] = q;
      }
    for (int i = 0; i < n; ++i)
      if (dg[i] < 0) return RSG_MISSING_DIAGONAL;
    rsg::HostBlockWalk H;
    if (!rsg::plan_block_walk(n, rp, cl, dg, sweep == 1, H)) {
      say("no block walk");
      return RSG_UNSUPPORTED;
    }
    if (stats) {
      stats[0] = H.nblk;
      stats[1] = H.steps();
      stats[2] = 0;
      for (int b = 0; b < H.nblk; ++b) stats[2] = std::max<int64_t>(stats[2], H.blk_step[b + 1] - H.blk_step[b]);
      stats[3] = H.w.total();
    }
    const std::string err = rsg::check_block_walk(n, rp, cl, dg, sweep == 1, H);
    say(err);
    return err.empty() ? RSG_OK : RSG_OUT_OF_PATTERN;
  } catch (const std::exception& e) {
    say(e.what());
    return RSG_CUDA_ERROR;
  }
}
