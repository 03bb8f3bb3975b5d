// Runs the kernels' warp roles on the CPU, one coroutine per warp, under many schedules: random priorities,
// re-drawn now and then, decide which warp, copy or tensor-pipe arrival goes on at every barrier
// operation, so one or the other is held back for as long as the rest can go on without it.  A schedule
// fails when nothing can go on (deadlock), when a warp arrives twice in one phase of a barrier (it has
// stood in for another one), when a wait returns on a phase its warp has already seen, or when a warp
// starts a copy from global memory before it has waited for the kernel before its own.  One CTA runs at a
// time, one lane of each warp; data does not exist.  With `giveup` one wait of a launch, drawn at random, runs into
// its time limit: the CTA must come to its end and leave the forward's work counter at zero.  The lanes of a warp may
// part in a wait without a vote that returns while the CTA gives up (some have seen their barrier, others the
// abort flag), so that warp must not wait with a vote before all of its lanes have met.
#include "cuda_runtime.h"
#include <ucontext.h>
#include <unistd.h>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>
#include <memory>
#include <random>
#include <set>
#include <vector>

dim3 threadIdx, blockIdx, gridDim;
namespace fa2 { namespace { alignas(1024) uint8_t smem[232448]; } }
uint8_t* sim_smem = fa2::smem;

namespace {
struct Barrier {
  unsigned count = 0, pending = 0, completed = 0;
  std::map<int, unsigned> seen;  // warp -> completed phases at its last successful wait, plus one
  std::set<int> arrived;         // in the current phase
};
std::map<uint32_t, Barrier> barriers;
struct Arrival { uint32_t bar; int warp; };
std::vector<Arrival> copies;
std::deque<Arrival> pipe_queue;
struct Warp {
  ucontext_t ctx;
  std::unique_ptr<char[]> stack;
  bool done = false, at_sync = false, waited_previous = false, parted = false;
  uint32_t bar = 0, parity = 0;
  int site = -1;  // >= 0: waiting
};
std::vector<Warp> warps;
ucontext_t scheduler;
int current;
std::mt19937 rng;
long waits, give_up = -1;  // waits of the launch so far; the one that runs into its limit
volatile int* abort_flag;  // of the CTA, once a warp has waited
std::vector<int> stored;  // first rows of the output boxes of the launch, in the order of their stores
bool aborted() { return abort_flag && *abort_flag; }

[[noreturn]] void fail(const char* what, uint32_t bar, int warp, int site) {
  printf("%s: block %u, hardware warp %d, barrier +%u, wait site %d\n", what, blockIdx.x, warp, bar, site);
  fflush(stdout);
  _exit(1);
}
void arrive(Arrival a) {
  Barrier& b = barriers[a.bar];
  if (!b.arrived.insert(a.warp).second && !aborted()) fail("second arrival in one phase", a.bar, a.warp, -1);
  if (--b.pending == 0) b.pending = b.count, ++b.completed, b.arrived.clear();
}
bool passes(uint32_t bar, uint32_t parity) { return (barriers[bar].completed & 1u) != parity; }
void yield() { swapcontext(&warps[current].ctx, &scheduler); }
void (*body_fn)(void*);
void* body_arg;
void entry() {
  body_fn(body_arg);
  warps[current].done = true;
  yield();
}
}  // namespace

void sim_init(uint32_t bar, uint32_t count) { barriers[bar] = Barrier{count, count, 0, {}, {}}; }
void sim_arrive(uint32_t bar) { yield(); arrive({bar, current}); }
void sim_arrive_later(uint32_t bar) { yield(); copies.push_back({bar, current}); }
void sim_arrive_after_mma(uint32_t bar) { yield(); pipe_queue.push_back({bar, current}); }
bool sim_wait(uint32_t bar, uint32_t parity, int site, volatile int* flag, bool vote) {
  Warp& w = warps[current];
  abort_flag = flag;
  if (vote && w.parted) fail("vote of a warp whose lanes may have parted", bar, current, site);
  if (waits++ == give_up) {
    *flag = 1, w.parted = !vote;
    return false;
  }
  w.bar = bar, w.parity = parity, w.site = site;
  yield();  // resumed only when the wait passes, or when the CTA gives up
  w.site = -1;
  if (aborted()) {
    w.parted |= !vote;
    return passes(bar, parity);
  }
  Barrier& b = barriers[bar];
  unsigned& seen = b.seen[current];
  if (seen >= b.completed + 1) fail("wait returned on a phase already seen", bar, current, site);
  seen = b.completed + 1;
  return true;
}
void sim_wait_previous() { warps[current].waited_previous = true; }
void sim_access() {
  if (!warps[current].waited_previous) fail("access before the wait for the previous kernel", 0, current, -1);
}
bool sim_meet(bool x) {
  const bool parted = warps[current].parted;
  warps[current].parted = false;
  return x && !parted;
}
void sim_stored(int row) { stored.push_back(row); }
void __syncthreads() {
  warps[current].at_sync = true;
  yield();
}
void sim_run(unsigned n, void (*body)(void*), void* arg) {
  body_fn = body, body_arg = arg;
  barriers.clear(), copies.clear(), pipe_queue.clear();
  abort_flag = nullptr;
  warps = std::vector<Warp>(n);
  for (unsigned i = 0; i < n; ++i) {
    Warp& w = warps[i];
    w.stack.reset(new char[1 << 17]);
    getcontext(&w.ctx);
    w.ctx.uc_stack.ss_sp = w.stack.get(), w.ctx.uc_stack.ss_size = 1 << 17, w.ctx.uc_link = nullptr;
    makecontext(&w.ctx, entry, 0);
  }
  std::vector<unsigned> priority(n + 2);  // warps, copies, tensor pipe
  auto draw = [&] { for (auto& p : priority) p = rng(); };
  draw();
  for (;;) {
    if (rng() % 64 == 0) draw();
    int best = -1;
    auto offer = [&](int i) { if (best < 0 || priority[i] > priority[best]) best = i; };
    unsigned done = 0, synced = 0;
    for (unsigned i = 0; i < n; ++i) {
      done += warps[i].done, synced += warps[i].at_sync;
      if (!warps[i].done && !warps[i].at_sync && (warps[i].site < 0 || aborted() || passes(warps[i].bar, warps[i].parity))) offer(i);
    }
    if (done == n) return;
    if (done + synced == n) {
      for (auto& w : warps) w.at_sync = false;
      continue;
    }
    if (!copies.empty()) offer(n);
    if (!pipe_queue.empty()) offer(n + 1);
    if (best < 0)
      for (unsigned i = 0; i < n; ++i)
        if (warps[i].site >= 0) fail("deadlock", warps[i].bar, i, warps[i].site);
    if (best == int(n)) {
      const size_t k = rng() % copies.size();
      const Arrival a = copies[k];
      copies.erase(copies.begin() + k);
      arrive(a);
    } else if (best == int(n) + 1) {
      const Arrival a = pipe_queue.front();
      pipe_queue.pop_front();
      arrive(a);
    } else {
      current = best;
      threadIdx = dim3(32 * best, 0, 0);
      swapcontext(&scheduler, &warps[best].ctx);
    }
  }
}

#include "bwd.cu"
#include "fwd.cu"

// main <kernel> <head dim> <rows> <keys> <schedules> <rows of a step> [<SMs> [giveup | order]]
int main(int argc, char** argv) {
  using namespace fa2;
  const std::string kernel = argv[1];
  const int d = atoi(argv[2]), n = atoi(argv[3]), nk = atoi(argv[4]);
  const AttnShape s{1, 1, n, padded_head_dim(d), 1, 1.f, d, nk};
  std::vector<unsigned> amax((n + 127) / 128);
  std::vector<float> scratch(dstile_pairs(n, nk) * 16384), lse(n), stats(amax.size() * 256);
  CUtensorMap m{};
  const F32Out none{nullptr, {}};
  const RowStats rs{stats.data(), amax.data()};
  int status = 0;
  unsigned counter = 0;
  LaunchCtx ctx{&status, &counter, 1};
  const int step = atoi(argv[6]);
  auto launch = [&] {
    waits = 0, stored.clear();
    if (kernel == "fwd") launch_fwd(s, step, m, m, m, m, none, lse.data(), ctx, nullptr);
    if (kernel == "dkdv") launch_bwd_dkdv(s, m, m, m, m, m, m, none, none, rs, nullptr, 0, step, &status, nullptr);
    if (kernel == "dkdv_atomic") launch_bwd_dkdv(s, m, m, m, m, m, m, none, none, rs, scratch.data(), 1, step, &status, nullptr);
    if (kernel == "dkdv_spill") launch_bwd_dkdv(s, m, m, m, m, m, m, none, none, rs, scratch.data(), 2, step, &status, nullptr);
    if (kernel == "dq") launch_bwd_dq(s, m, m, m, m, m, none, rs, step, &status, nullptr);
    if (kernel == "scores") launch_bwd_scores_wide(s, m, m, m, m, m, none, rs, scratch.data(), &status, nullptr);
    for (int form = 1; form < 3; ++form) {
      if (kernel == "consume" && (d > 128 || form == 2)) launch_bwd_consume(s, form, scratch.data(), m, m, none, rs, false, &status, nullptr);
      if (kernel == "consume_pair") launch_bwd_consume(s, form, scratch.data(), m, m, none, rs, true, &status, nullptr);
    }
    if (counter) fail("work counter not left at zero", 0, -1, -1);
  };
  for (int seed = 0; seed < atoi(argv[5]); ++seed) {
    rng.seed(seed);
    ctx.num_sms = argc > 7 ? atoi(argv[7]) : 1 + seed % 2 * 63;  // work items of two Q tiles and of one
    launch();
    if (argc <= 8) continue;
    if (argv[8] == std::string("order")) {
      for (int row : stored) printf("%d ", row);
      puts("");
      continue;
    }
    give_up = rng() % waits;
    launch();
    give_up = -1;
  }
  return 0;
}
