// Block walks: triangular solves of ILU(0) factors as a dataflow of row
// blocks over the whole GPU (blockwalk.cu).
//
// Rows are cut into contiguous blocks (on a grid in natural order: up to 32
// grid lines of one plane), one CTA per block.  A block's rows form steps of
// at most 32 mutually independent rows, one per lane, in the order of their
// dependency depth (on a grid: a wavefront across the lines).  Within a CTA
// the work of a step is spread over warps of different SM sub-partitions,
// because a double-precision warp instruction occupies its sub-partition for
// 64 cycles whatever its active lanes (19 cycles per SM with all four busy),
// and a dependent one waits as long:
//   * fetch warps stage a step's coefficients, right-hand side and the
//     values of other blocks it reads into shared memory, several steps
//     ahead;
//   * early warps sum the terms whose operands are not recent values of the
//     block itself (on a 27-point grid pattern: the neighbouring plane's nine);
//   * one warp adds the remaining terms (the neighbouring line's three and the
//     line's own), oldest operands first, and publishes the values.  Its chain
//     is all that separates two steps: handing values to another warp and back
//     costs more (170 cycles each way) than the terms it could take over.
// Blocks exchange values through an array in global memory laid out by step
// and lane, so that a step's values are a contiguous 256 bytes for the writer
// and for the readers.  It is filled with a sentinel (a NaN no arithmetic
// yields) beforehand, and readers poll until the value is there.  A block
// reads only earlier blocks, and CTAs take blocks in order from a counter, so
// a running CTA never waits for one that has not started, whatever else
// occupies the GPU.
//
// What bounds it: the chain of steps and the hops between blocks, ni + 2 nj
// steps and nk hops on a grid.  A step takes 208 ns in double precision (four
// terms of about 100 cycles each, one after the other on the sub-partition; a
// single block of 2048 x 32 rows never waits for anything else) and 110 in
// single, a hop 2.2 and 1.5 us.  A walk, chained to the kernels around it,
// double and single: 2048 x 32 x 1 445 and 239 us, 32 x 32 x 8 40 and 25, 64 x
// 64 x 16 87 and 54, 128 x 128 x 32 190 and 128.  The level walk on one 16-CTA
// cluster (ring.cuh), whose levels each wait for a CTA barrier and a load from
// memory, took 700 to 780 and 480 us on the last, about 300 and 190 on the one
// before.  Measured and not kept: handing the chain's newest operands on by
// shuffles (204 ns a step: the terms bound it, not their exchange), staging
// further ahead, more or fewer warps of a kind, fetch warps that take two steps
// in a row (a quarter slower in three dimensions) or release steps together.
//
// A row's sum starts from the right-hand side and subtracts fused products;
// upper factors are stored divided by their row's diagonal (with its
// reciprocal for the right-hand side), which takes the division out of the
// chain.
#pragma once
#include "linalg.cuh"

namespace rsg {

constexpr int BW_LANES = 32;
constexpr int BW_OWN = 16;                // steps of the block's own values kept in shared memory
constexpr int BW_HALO_MAX = 4096;         // values of other blocks kept in shared memory
constexpr int BW_STAGES_MAX = 16;         // steps staged ahead: 16, or 8 for wide rows
constexpr int BW_STAGES_MIN = 8;
constexpr int BW_WIDTH_MAX = 48;          // terms per row
constexpr int BW_OLD = 8;                 // own operands younger than this are the chain's
constexpr int BW_NEW = 2;                 // others' values fetched less than this many steps ago are summed last
constexpr int BW_BACK = 8;                // a step's right-hand-side indices are staged with the step this many before
constexpr size_t BW_SMEM_MAX = 200 * 1024;

// A row's terms by phase, and the most any row has of each: early warps sum
// the old ones before the step's newest values of other blocks are there and
// the new ones after; the chain subtracts pre (own operands at least two
// steps old) ahead of its turn and last (one step old) in it.
struct BwWidths {
  int old = 0, fresh = 0, pre = 0, last = 0;
  __host__ __device__ int total() const { return old + fresh + pre + last; }
  // groups of four operand indices: early phases padded separately, the chain's together
  __host__ __device__ int old_groups() const { return (old + 3) / 4; }
  __host__ __device__ int early_groups() const { return old_groups() + (fresh + 3) / 4; }
  __host__ __device__ int groups() const { return early_groups() + (pre + last + 3) / 4; }
  // bytes of a step's operand indices (u16, a lane's four together)
  __host__ __device__ int index_bytes() const { return groups() * 256; }
  // place of the index of term k (in the order old, fresh, pre, last) of a lane, in u16 units
  int index_at(int k, int lane) const {
    const int g0 = k < old ? 0 : k < old + fresh ? old_groups() : early_groups();
    const int k0 = k < old ? 0 : k < old + fresh ? old : old + fresh;
    return ((g0 + (k - k0) / 4) * 32 + lane) * 4 + (k - k0) % 4;
  }
};

// Host form of a block walk of one triangle.
struct HostBlockWalk {
  int nblk = 0, halo = 0, stages = 0;
  BwWidths w;
  bool own_old = false;        // some early operand is the block's own
  std::vector<int> blk_step;   // nblk + 1: first step of each block
  std::vector<int> hptr;       // steps + 1: halo entries of each step
  std::vector<int> hsrc;       // halo entry: exchange slot (step * 32 + lane) fetched
  std::vector<unsigned short> idx;  // per step: w.index_bytes() of operand indices
  std::vector<int> rows;       // per step: rows[32], -1 on idle lanes
  std::vector<int> src;        // per step: CSR position of each term [w.total()][32], -1 none (a zero times the zero slot)
  int steps() const { return blk_step.empty() ? 0 : blk_step.back(); }
};

// Plans the walk of the strictly lower (upper = false) or upper triangle.
// False when the pattern does not suit it (a row too wide, too many values
// of other blocks alive at once, too much padding).
bool plan_block_walk(int n, const std::vector<int>& rp, const std::vector<int>& cl, const std::vector<int>& dg,
                     bool upper, HostBlockWalk& H);
// Walks a plan on the host, with every staged value overwritten as early as
// the device may overwrite it, against the sequential solve.  Empty when sound.
std::string check_block_walk(int n, const std::vector<int>& rp, const std::vector<int>& cl,
                             const std::vector<int>& dg, bool upper, const HostBlockWalk& H);

// Whether this process has launched a block walk.
bool block_walks_used();

struct BlockWalk {
  bool upper = false;
  int nblk = 0, halo = 0, stages = 0, nsteps = 0;
  BwWidths w;
  bool own_old = false;
  DeviceBuffer<int> blk_step, hptr, hsrc, src, rows, bsrc;
  DeviceBuffer<unsigned char> ints;
  DeviceBuffer<unsigned> ticket;
  size_t slots() const { return (size_t)nsteps * BW_LANES; }
};

// What the walks hold per precision: coefficients and exchange arrays (the
// lower walk's twice: an apply uses one while its upper walk readies the other).
template <typename T>
struct BlockWalkData {
  DeviceBuffer<T> lval, uval, lex[2], uex;
};

// x = U^-1 L^-1 b with both triangles' block walks.
struct BlockWalkPair {
  Context* ctx = nullptr;
  bool planned = false;
  BlockWalk L, U;
  BlockWalkData<double> d64;
  BlockWalkData<float> d32;
  // takes both triangles' plans (nblk == 0: none)
  void plan(Context* c, int n, const HostBlockWalk& lower, const HostBlockWalk& upper);
  // Gathers the coefficients from the factor values.  flag (may be null): bit
  // 0 is set when a scaled upper coefficient is not finite, bit 1 when it is
  // not in single precision.  The earlier coefficients stay when the
  // factorisation has set *failed (may be null) or a wait of it ran out.
  template <typename T>
  void values(const double* lu, const int* diag, int* flag, const int* failed = nullptr);
  // Readies the exchange arrays; once before a solve's applies (an apply
  // leaves them ready for the next one, unless it was given up).
  template <typename T>
  void begin();
  template <typename T>
  void apply(const T* b, T* x, const int* active);

 private:
  template <typename T>
  BlockWalkData<T>& data();
};

}  // namespace rsg
