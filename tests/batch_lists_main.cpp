// Sorts a large job's batches into their lists with memory running out, in the
// helper threads (argument "helpers") or in the calling one ("caller").  The
// caller gets std::bad_alloc, the process lives on, and a second try succeeds.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>

#include "engine.h"

static std::thread::id g_main;
static int g_fail = 0;  // 1: large allocations of other threads fail, 2: of this one

void* operator new(size_t n) {
  const bool mine = std::this_thread::get_id() == g_main;
  if (n >= 4096 && g_fail == (mine ? 2 : 1)) throw std::bad_alloc();
  void* p = std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main(int argc, char** argv) {
  if (argc != 2) return 2;
  g_main = std::this_thread::get_id();
  const int32_t N = 200000;
  sbp::Job job;
  job.N = N;
  job.h_optr.resize(N + 1);
  job.h_iptr.resize(N + 1);
  for (int32_t v = 0; v <= N; ++v) job.h_optr[v] = job.h_iptr[v] = 10 * v;
  sbp::Run run;
  run.J = &job;
  run.o.num_batches = 4;
  bool caught = false;
  g_fail = std::strcmp(argv[1], "helpers") == 0 ? 1 : 2;
  try {
    run.setup_batches();
  } catch (const std::bad_alloc&) {
    caught = true;
  }
  g_fail = 0;
  run.setup_batches();
  std::printf("caught %d lists %zu\n", (int)caught, run.lists_all.size());
  return caught && run.lists_all.size() == (size_t)N ? 0 : 1;
}
