// The affine solve's LU (dice_b200/csrc/dg_lu.cuh) on the CPU: 32 lanes, each a
// context of its own, run one after the other from one warp-synchronous call to
// the next, in several orders.  A read that another lane's write may overtake
// then gives another factorisation.  Compared bit for bit with the same steps
// done by one thread.  Prints LU PASSED.
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#define __device__
#define __forceinline__ inline

namespace warp {
constexpr int W = 32;
ucontext_t home, ctx[W];
std::vector<char> stack[W];
bool done[W];
int me;              // the lane that runs
unsigned in[W];      // what each lane brings to a synchronising call
unsigned maxv, ballot;

void meet(unsigned v) {
  in[me] = v;
  const int lane = me;
  swapcontext(&ctx[lane], &home);
}
}  // namespace warp

static unsigned __reduce_max_sync(unsigned, unsigned v) { warp::meet(v); return warp::maxv; }
static unsigned __ballot_sync(unsigned, int v) { warp::meet(v ? 1u : 0u); return warp::ballot; }
static void __syncwarp() { warp::meet(0u); }
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
static long long __double_as_longlong(double d) {
  long long r;
  std::memcpy(&r, &d, 8);
  return r;
}

#include "../../dice_b200/csrc/dg_lu.cuh"

static double H[36];
static int N, pos[warp::W], info[warp::W];

static void lane_main(int lane) {
  info[lane] = dg::lu_affine(H, N, lane, pos[lane]);
  warp::done[lane] = true;
  swapcontext(&warp::ctx[lane], &warp::home);
}

static void run(const int* order) {
  using namespace warp;
  for (int l = 0; l < W; ++l) {
    getcontext(&ctx[l]);
    stack[l].resize(64 * 1024);
    ctx[l].uc_stack.ss_sp = stack[l].data();
    ctx[l].uc_stack.ss_size = stack[l].size();
    ctx[l].uc_link = &home;
    done[l] = false;
    makecontext(&ctx[l], (void (*)())lane_main, 1, l);
  }
  for (;;) {
    bool any = false;
    for (int k = 0; k < W; ++k) {
      const int l = order[k];
      if (done[l]) continue;
      any = true;
      me = l;
      swapcontext(&home, &ctx[l]);
    }
    if (!any) return;
    maxv = *std::max_element(in, in + W);
    ballot = 0u;
    for (int l = 0; l < W; ++l)
      if (in[l]) ballot |= 1u << l;
  }
}

// the same steps by one thread
static int plain(double* A, int n, int* where) {
  int inf = 0;
  for (int l = 0; l < warp::W; ++l) where[l] = l;
  for (int j = 0; j < n; ++j) {
    int p = j;
    double best = std::fabs(A[j * n + j]);
    for (int i = j + 1; i < n; ++i)
      if (std::fabs(A[i * n + j]) > best) { best = std::fabs(A[i * n + j]); p = i; }
    for (int l = 0; l < warp::W; ++l) {
      if (where[l] == j) where[l] = p;
      else if (where[l] == p) where[l] = j;
    }
    const double pv = A[p * n + j];
    if (pv != 0.0) {
      const double r = 1.0 / pv;
      for (int k = 0; k < n; ++k) std::swap(A[j * n + k], A[p * n + k]);
      for (int i = j + 1; i < n; ++i) A[i * n + j] = A[i * n + j] * r;
    } else if (inf == 0) {
      inf = j + 1;
    }
    for (int i = j + 1; i < n; ++i)
      for (int k = j + 1; k < n; ++k) A[i * n + k] = A[i * n + k] - A[i * n + j] * A[j * n + k];
  }
  return inf;
}

static bool same(double a, double b) { return std::memcmp(&a, &b, 8) == 0 || (std::isnan(a) && std::isnan(b)); }

int main() {
  std::mt19937 rng(3);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  const double special[] = {0.0, -0.0, 1.0, -1.0, std::numeric_limits<double>::infinity(),
                            std::numeric_limits<double>::quiet_NaN(), 5e-324, 1e300};
  std::vector<std::vector<int>> orders;
  for (int o = 0; o < 4; ++o) {
    std::vector<int> v(warp::W);
    for (int l = 0; l < warp::W; ++l) v[l] = o == 1 ? warp::W - 1 - l : l;
    if (o > 1) std::shuffle(v.begin(), v.end(), rng);
    orders.push_back(v);
  }
  int swaps = 0;
  for (N = 2; N <= 6; ++N)
    for (int t = 0; t < 300; ++t) {
      double A[36], want[36];
      for (int k = 0; k < N * N; ++k) A[k] = t % 3 == 2 && rng() % 4 == 0 ? special[rng() % 8] : u(rng) * std::pow(10.0, 4.0 * u(rng));
      if (t % 3 == 0)   // symmetric, as a Hessian
        for (int i = 0; i < N; ++i)
          for (int k = 0; k < i; ++k) A[i * N + k] = A[k * N + i];
      std::memcpy(want, A, sizeof(A));
      int where[warp::W];
      const int inf = plain(want, N, where);
      for (int l = 0; l < N; ++l) swaps += where[l] != l;
      for (const auto& o : orders) {
        std::memcpy(H, A, sizeof(A));
        run(o.data());
        for (int l = 0; l < warp::W; ++l)
          if (info[l] != inf || pos[l] != where[l]) {
            std::printf("N %d matrix %d: lane %d has info %d row %d, not %d and %d\n", N, t, l, info[l], pos[l], inf, where[l]);
            return 1;
          }
        for (int k = 0; k < N * N; ++k)
          if (!same(H[k], want[k])) {
            std::printf("N %d matrix %d: entry %d is %.17g, not %.17g\n", N, t, k, H[k], want[k]);
            return 1;
          }
      }
    }
  if (swaps < 1000) return 2;
  std::printf("LU PASSED\n");
  return 0;
}
