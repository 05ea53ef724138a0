// The hand-over ring (csrc/ring.cuh) under arbitrary interleavings of its memory
// operations: agents on coroutines take values from a ring of `entries` slots and put
// them back, and the scheduler switches between them before every operation. A value
// must be held by one agent at a time, and none may be lost.
#include <ucontext.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "ring.cuh"

using rapt::RingWord;

static ucontext_t main_ctx;
static std::vector<ucontext_t> agents;
static int current = 0;
static void yield() { swapcontext(&agents[current], &main_ctx); }

struct Mem {
  static RingWord get(const RingWord* p) { yield(); return *p; }
  static void put(RingWord* p, RingWord v) { yield(); *p = v; }
  static RingWord add(RingWord* p, RingWord v) { yield(); const RingWord o = *p; *p += v; return o; }
  static RingWord cas(RingWord* p, RingWord was, RingWord v) {
    yield();
    const RingWord o = *p;
    if (o == was) *p = v;
    return o;
  }
};

static RingWord head, tail;
static std::vector<RingWord> ring;
static std::vector<int> holder;
static bool doubled;
static std::vector<char> over;

static void agent(int me, int turns) {
  for (int i = 0; i < turns; ++i) {
    const int64_t v = rapt::ring_take<Mem>(ring.data(), ring.size(), &head);
    if (v < 0) continue;
    if (v >= (int64_t)holder.size() || holder[v] != -1) { doubled = true; break; }
    holder[v] = me;
    yield();
    holder[v] = -1;
    rapt::ring_put<Mem>(ring.data(), ring.size(), &tail, (int32_t)v);
  }
  over[me] = 1;
  swapcontext(&agents[me], &main_ctx);
}

int main(int argc, char** argv) {
  const int values = atoi(argv[1]), n_agents = atoi(argv[2]), runs = atoi(argv[3]);
  constexpr size_t kStack = 64 << 10;
  std::vector<std::vector<char>> stacks(n_agents, std::vector<char>(kStack));
  unsigned long long x = 88172645463325252ull;
  long taken = 0;
  for (int run = 0; run < runs; ++run) {
    ring.assign(values, 0);
    head = tail = 0;
    holder.assign(values, -1);
    over.assign(n_agents, 0);
    doubled = false;
    agents.assign(n_agents, ucontext_t());
    for (int v = 0; v < values; ++v) ring[tail % values] = (tail + 1) << 32 | (RingWord)v, ++tail;
    for (int a = 0; a < n_agents; ++a) {
      getcontext(&agents[a]);
      agents[a].uc_stack.ss_sp = stacks[a].data();
      agents[a].uc_stack.ss_size = kStack;
      agents[a].uc_link = nullptr;
      makecontext(&agents[a], (void (*)())agent, 2, a, 24);
    }
    int left = n_agents;
    while (left) {
      x ^= x << 13; x ^= x >> 7; x ^= x << 17;
      current = (int)(x % n_agents);
      if (over[current]) continue;
      // now and then an agent stands still while another runs for many operations
      int ops = (x >> 32) % 8 ? 1 : 1 + (int)((x >> 40) % 40);
      while (ops-- && !over[current]) swapcontext(&main_ctx, &agents[current]);
      left -= over[current];
    }
    taken += (long)head;
    // every value is in the ring once
    std::vector<int> seen(values, 0);
    if (tail - head != (RingWord)values) { printf("lost or doubled: run %d\n", run); return 1; }
    for (RingWord at = head; at < tail; ++at) {
      const RingWord e = ring[at % values];
      if ((e >> 32) != at + 1 || seen[(uint32_t)e]++) doubled = true;
    }
    if (doubled) { printf("taken twice: run %d\n", run); return 1; }
  }
  printf("ok %ld\n", taken);
  return 0;
}
