// A block walk whose wait runs out: its second block is made to read, for an
// early row, the value of its own last row.  Every access stays in bounds (the
// slot exists), and each wait ends by its limit.  Exit code 0: the walk ended,
// the timeout is reported, nothing outside x was written, and the mended plan
// gives the bits of before once the walk is begun anew.
#include <cstdio>
#include <cstring>

#include "../../ressim_gb300/csrc/blockwalk.cuh"

#define CHECK(x)                                          \
  do {                                                    \
    if (!(x)) {                                           \
      std::printf("line %d: %s\n", __LINE__, #x);         \
      return 1;                                           \
    }                                                     \
  } while (0)

// the 27-point pattern of a grid, rows in natural order
static void pattern(int ni, int nj, int nk, std::vector<int>& rp, std::vector<int>& cl, std::vector<int>& dg) {
  rp.assign(1, 0);
  for (int k = 0; k < nk; ++k)
    for (int j = 0; j < nj; ++j)
      for (int i = 0; i < ni; ++i) {
        for (int c = std::max(0, k - 1); c <= std::min(nk - 1, k + 1); ++c)
          for (int b = std::max(0, j - 1); b <= std::min(nj - 1, j + 1); ++b)
            for (int a = std::max(0, i - 1); a <= std::min(ni - 1, i + 1); ++a) {
              if (a == i && b == j && c == k) dg.push_back((int)cl.size());
              cl.push_back(a + ni * (b + nj * c));
            }
        rp.push_back((int)cl.size());
      }
}

template <typename T>
static int run(rsg::Context& ctx, int n, rsg::BlockWalkPair& walk, const rsg::HostBlockWalk& L, const double* lu,
               const int* diag) {
  const int entry = L.hptr[L.blk_step[1]], last = (L.blk_step[2] - 1) * rsg::BW_LANES;
  CHECK(entry < L.hptr[L.blk_step[2]] && last / rsg::BW_LANES > L.blk_step[1] + 1);
  auto read_from = [&](int slot) {
    RSG_CUDA(cudaMemcpyAsync(walk.L.hsrc.get() + entry, &slot, sizeof(slot), cudaMemcpyHostToDevice, ctx.stream));
    ctx.sync();
  };
  constexpr int PAD = 4096;
  std::vector<T> hb(n), x0(n), x1(n + 2 * PAD);
  for (int i = 0; i < n; ++i) hb[i] = (T)(1 + i % 7);
  rsg::DeviceBuffer<T> b(n), x(n + 2 * PAD);
  RSG_CUDA(cudaMemcpyAsync(b.get(), hb.data(), sizeof(T) * n, cudaMemcpyHostToDevice, ctx.stream));
  RSG_CUDA(cudaMemsetAsync(x.get(), 0x5a, sizeof(T) * x.size(), ctx.stream));
  walk.values<T>(lu, diag, nullptr);
  walk.begin<T>();
  walk.apply<T>(b.get(), x.get() + PAD, nullptr);
  RSG_CUDA(cudaMemcpyAsync(x0.data(), x.get() + PAD, sizeof(T) * n, cudaMemcpyDeviceToHost, ctx.stream));
  ctx.check_device_error();
  for (int i = 0; i < n; ++i) CHECK(x0[i] == x0[i]);
  for (int again = 0; again < 2; ++again) {
    walk.begin<T>();
    read_from(last);
    for (int q = 0; q < 3; ++q) walk.apply<T>(b.get(), x.get() + PAD, nullptr);
    rsg_status st = RSG_OK;
    try {
      ctx.check_device_error();
    } catch (const rsg::Error& e) {
      st = e.status;
      std::printf("%s\n", e.what());
    }
    CHECK(st == RSG_TIMEOUT);
    read_from(L.hsrc[entry]);
    walk.begin<T>();
    walk.apply<T>(b.get(), x.get() + PAD, nullptr);
    RSG_CUDA(cudaMemcpyAsync(x1.data(), x.get(), sizeof(T) * x1.size(), cudaMemcpyDeviceToHost, ctx.stream));
    ctx.check_device_error();
    CHECK(!std::memcmp(x0.data(), x1.data() + PAD, sizeof(T) * n));
    for (size_t q = 0; q < sizeof(T) * PAD; ++q) {
      CHECK(reinterpret_cast<unsigned char*>(x1.data())[q] == 0x5a);
      CHECK(reinterpret_cast<unsigned char*>(x1.data() + PAD + n)[q] == 0x5a);
    }
  }
  return 0;
}

int main() {
  rsg_ctx* h = nullptr;
  CHECK(rsg_context_create(0, &h) == RSG_OK);
  rsg::Context& ctx = h->c;
  // 33 lines a plane: blocks that read each other along both directions; the
  // second pattern has 48 terms a row, the widest there are (8 stages)
  for (int wide = 0; wide < 2; ++wide) {
    std::vector<int> rp, cl, dg;
    if (!wide) pattern(20, 33, 6, rp, cl, dg);
    else {
      rp.assign(1, 0);
      const int n = 4000;
      for (int i = 0; i < n; ++i) {
        for (int c = std::max(0, i - 48); c <= std::min(n - 1, i + 48); ++c) {
          if (c == i) dg.push_back((int)cl.size());
          cl.push_back(c);
        }
        rp.push_back((int)cl.size());
      }
    }
    const int n = (int)rp.size() - 1;
    std::vector<double> lu(cl.size());
    for (size_t q = 0; q < lu.size(); ++q) lu[q] = ((int)(q * 7919 % 13) - 6) / 300.0;
    for (int i = 0; i < n; ++i) lu[dg[i]] = 1 + i % 3;
    rsg::DeviceBuffer<double> dlu(lu.size());
    rsg::DeviceBuffer<int> ddg(n);
    RSG_CUDA(cudaMemcpyAsync(dlu.get(), lu.data(), sizeof(double) * lu.size(), cudaMemcpyHostToDevice, ctx.stream));
    RSG_CUDA(cudaMemcpyAsync(ddg.get(), dg.data(), sizeof(int) * n, cudaMemcpyHostToDevice, ctx.stream));
    rsg::HostBlockWalk L, U;
    CHECK(rsg::plan_block_walk(n, rp, cl, dg, false, L) && rsg::plan_block_walk(n, rp, cl, dg, true, U));
    CHECK(L.nblk > 2 && L.stages == (wide ? rsg::BW_STAGES_MIN : rsg::BW_STAGES_MAX));
    rsg::BlockWalkPair walk;
    walk.plan(&ctx, n, L, U);
    if (run<double>(ctx, n, walk, L, dlu.get(), ddg.get()) || run<float>(ctx, n, walk, L, dlu.get(), ddg.get())) return 1;
  }
  CHECK(rsg_context_destroy(h) == RSG_OK);
  std::printf("ended\n");
  return 0;
}
