// build_jumps (newman_gb300/csrc/jump.hpp) on a given number of threads: never more
// than that at once, the same tables for any number, and the same again where no
// thread can be started.
//
//   jump_threads re im step nr nc N
//
// Prints "differing-tables threads-beyond-the-limit threads-started".
#include <dlfcn.h>
#include <pthread.h>

#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../newman_gb300/csrc/jump.hpp"

using namespace nmg;

static std::atomic<int> live{0}, most{0}, started{0};
static std::atomic<bool> refuse{false};

struct Call {
  void* (*run)(void*);
  void* arg;
};
static void* counted(void* p) {
  const Call c = *(Call*)p;
  delete (Call*)p;
  void* r = c.run(c.arg);
  live--;
  return r;
}
// in place of the C library's
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*run)(void*), void* arg) {
  using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Create create = (Create)dlsym(RTLD_NEXT, "pthread_create");
  if (refuse) return EAGAIN;
  started++;
  const int now = ++live;
  for (int m = most; now > m && !most.compare_exchange_weak(m, now);) {
  }
  return create(t, a, counted, new Call{run, arg});
}

int main(int argc, char** argv) {
  if (argc != 7) return 2;
  MPView v(std::atoi(argv[4]), std::atoi(argv[5]));
  if (v.set_view(argv[1], argv[2], argv[3], argv[3], std::atoi(argv[6]), 1e-10, 0)) return 3;
  OrbitData od;
  if (v.precompute(1, od, REFERENCE_CENTER, false, nullptr, nullptr)) return 4;
  std::vector<RFE> er, ei;
  v.eps_tables_fe(er, ei);
  const EpsRange range = eps_range(er, ei);
  JumpTables one;
  int differ = 0, beyond = 0, all = 0;
  const int limits[] = {1, 2, 3, 16, 16};
  for (int k = 0; k < 5; k++) {
    refuse = k == 4;
    live = most = started = 0;
    JumpTables t;
    build_jumps(od, range.norm(), range.e, limits[k], t);
    beyond += most > limits[k] - 1 ? most - (limits[k] - 1) : 0;
    all += started;
    if (k == 0) one = t;
    auto same = [](const std::vector<JumpRec>& a, const std::vector<JumpRec>& b) {
      return a.size() == b.size() && !std::memcmp(a.data(), b.data(), a.size() * sizeof(JumpRec));
    };
    if (!same(t.start, one.start) || !same(t.chain, one.chain) || t.start_index != one.start_index)
      differ++;
  }
  std::printf("%d %d %d\n", differ, beyond, all);
  return differ || beyond ? 1 : 0;
}
