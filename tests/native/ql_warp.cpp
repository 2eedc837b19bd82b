// The warp form of ql_first_row with its 32 lanes as coroutines that are switched
// at random between any two loads or stores, as a GPU may do. Prints the number of
// matrices whose result differs from the single-thread form's in any bit.
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace {

constexpr int kLanes = 32;
ucontext_t g_main, g_lane[kLanes];
int g_cur = -1;  // running lane, -1: none
enum State { kRun, kBarrier, kDone };
State g_state[kLanes];
unsigned g_vote[kLanes], g_ballot;
uint64_t g_rng = 1;

unsigned rnd() {
  g_rng ^= g_rng << 13;
  g_rng ^= g_rng >> 7;
  g_rng ^= g_rng << 17;
  return static_cast<unsigned>(g_rng >> 33);
}

int g_burst = 0;
void maybe_switch() {
  if (g_cur < 0 || --g_burst > 0) return;
  swapcontext(&g_lane[g_cur], &g_main);
}
unsigned meet(unsigned vote) {
  g_vote[g_cur] = vote;
  g_state[g_cur] = kBarrier;
  swapcontext(&g_lane[g_cur], &g_main);
  return g_ballot;
}

struct Idx {
  struct X {
    operator unsigned() const { return g_cur < 0 ? 0u : static_cast<unsigned>(g_cur); }
  } x;
} threadIdx;

unsigned __ballot_sync(unsigned, bool p) { return meet(p ? 1u : 0u); }
void __syncwarp() { meet(0); }
int __ffs(unsigned v) { return __builtin_ffs(static_cast<int>(v)); }
double rsqrt(double x) { return 1.0 / std::sqrt(x); }

// Array whose every load and store is a place where another lane may run.
struct Ref {
  double* p;
  operator double() const {
    maybe_switch();
    return *p;
  }
  Ref& operator=(double v) {
    maybe_switch();
    *p = v;
    return *this;
  }
  Ref& operator=(const Ref& o) { return *this = static_cast<double>(o); }
};
struct View {
  double* p;
  Ref operator[](int i) const { return Ref{p + i}; }
};

}  // namespace

#define __device__
#define __forceinline__ inline
#include QL_HEADER

namespace {

int g_n;
std::vector<double> g_d, g_z, g_e;
bool g_ok[kLanes];

void lane_main(int lane) {
  g_ok[lane] = ftlm::ql_first_row<true>(g_n, View{g_d.data()}, View{g_z.data()}, View{g_e.data()});
  g_state[lane] = kDone;
  swapcontext(&g_lane[lane], &g_main);
}

// False when the lanes do not all arrive at the same barriers or do not finish.
bool run_warp() {
  static std::vector<char> stacks(static_cast<size_t>(kLanes) << 16);
  for (int l = 0; l < kLanes; ++l) {
    getcontext(&g_lane[l]);
    g_lane[l].uc_stack.ss_sp = stacks.data() + (static_cast<size_t>(l) << 16);
    g_lane[l].uc_stack.ss_size = size_t(1) << 16;
    g_lane[l].uc_link = &g_main;
    makecontext(&g_lane[l], reinterpret_cast<void (*)()>(lane_main), 1, l);
    g_state[l] = kRun;
  }
  for (int64_t turn = 0; turn < 50000000; ++turn) {
    int ready[kLanes], nr = 0, done = 0;
    for (int l = 0; l < kLanes; ++l) {
      if (g_state[l] == kRun) ready[nr++] = l;
      done += g_state[l] == kDone;
    }
    if (done == kLanes) return true;
    if (nr == 0) {
      if (done) return false;  // some wait for lanes that have left
      g_ballot = 0;
      for (int l = 0; l < kLanes; ++l) g_ballot |= g_vote[l] << l;
      for (int l = 0; l < kLanes; ++l) g_state[l] = kRun;
      continue;
    }
    g_cur = ready[rnd() % static_cast<unsigned>(nr)];
    g_burst = 1 + static_cast<int>(rnd() % 400);
    swapcontext(&g_main, &g_lane[g_cur]);
    g_cur = -1;
  }
  return false;
}

}  // namespace

int main(int argc, char** argv) {
  const int matrices = argc > 1 ? std::atoi(argv[1]) : 10;
  int bad = 0;
  for (int t = 0; t < matrices; ++t) {
    g_rng = 0x9E3779B97F4A7C15ull * static_cast<uint64_t>(t + 1);
    const int n = 1 + static_cast<int>(rnd() % 70);
    std::vector<double> d0(n), e0(n), z0(n, 0.0);
    for (int i = 0; i < n; ++i) {
      d0[i] = rnd() / 2147483648.0 * 20.0 - 10.0;
      e0[i] = i + 1 < n ? rnd() / 2147483648.0 * 4.0 : 0.0;
    }
    if (n > 8) e0[n / 3] = 0.0;  // a matrix that falls apart
    z0[0] = 1.0;
    std::vector<double> d = d0, z = z0, e = e0;
    const bool ok = ftlm::ql_first_row<false>(n, d.data(), z.data(), e.data());
    g_n = n;
    g_d = d0;
    g_z = z0;
    g_e = e0;
    bool same = run_warp();
    for (int l = 0; l < kLanes; ++l) same = same && g_ok[l] == ok;
    same = same && !std::memcmp(d.data(), g_d.data(), sizeof(double) * n) &&
           !std::memcmp(z.data(), g_z.data(), sizeof(double) * n);
    bad += !same;
  }
  std::printf("%d\n", bad);
  return 0;
}
