// Host-only exercise of host_stage.h: the CUDA calls it makes are answered by the fakes below.
//   host_stage_test <name>   runs one check; exit code 0 = passed
#include "host_stage.h"

#include <dlfcn.h>
#include <sys/wait.h>
#include <unistd.h>

#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <string>

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
  *p = std::malloc(bytes);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
static int g_waits = 0;
static bool g_held = true;  // the buffers were all in use whenever a stream was waited for
cudaError_t cudaStreamSynchronize(cudaStream_t);
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
}

// the process is at its limit of threads after so many more
static std::atomic<int> g_threads_left{1 << 30};
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* attr, void* (*f)(void*), void* arg) {
  if (g_threads_left-- <= 0) return EAGAIN;
  using Real = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Real real = reinterpret_cast<Real>(dlsym(RTLD_NEXT, "pthread_create"));
  return real(t, attr, f, arg);
}

using hnsw::HostStage;

cudaError_t cudaStreamSynchronize(cudaStream_t) {
  ++g_waits;
  void* p = HostStage::Get().Acquire();
  if (p) g_held = false;
  HostStage::Get().Release(p);
  return cudaSuccess;
}

namespace {
#define EXPECT(x)                                                  \
  do {                                                             \
    if (!(x)) {                                                    \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #x);         \
      std::exit(1);                                                \
    }                                                              \
  } while (0)

// a parallel loop gives every part exactly one turn
void Loop(int n) {
  std::vector<int> turns((size_t)n, 0);
  HostStage::Get().ParallelFor(n, [&](int i) { ++turns[(size_t)i]; });
  for (int t : turns) EXPECT(t == 1);
}

// the last user goes, and while its threads are on their way out another one comes and goes: nobody waits for good
void Users() {
  for (int i = 0; i < 3000; ++i) {
    HostStage::Get().AddUser();
    Loop(6);
    std::atomic<bool> go{false};
    std::thread other([&go, i] {
      while (!go) {
      }
      for (volatile int spin = 0; spin < i % 60 * 50; ++spin) {
      }
      HostStage::Get().AddUser();
      HostStage::Get().DropUser();
    });
    go = true;
    HostStage::Get().DropUser();
    other.join();
  }
}

// a buffer that a stream works on goes back behind that work, also when an exception takes its scope down
void Unwinding() {
  HostStage::Get().AddUser();
  void* others[HostStage::kMaxBuffers - 1];
  for (void*& p : others) EXPECT((p = HostStage::Get().Acquire()) != nullptr);
  try {
    hnsw::StreamBuffer b;
    EXPECT(b.Open());
    b.Use(nullptr);
    throw std::bad_alloc();
  } catch (const std::bad_alloc&) {
  }
  EXPECT(g_waits == 1 && g_held);
  {
    hnsw::StreamBuffer b;
    EXPECT(b.Open());
    EXPECT(!hnsw::StreamBuffer().Open());
    b.Use(nullptr);
    EXPECT(b.Wait() == cudaSuccess && b.Wait() == cudaSuccess);
  }
  EXPECT(g_waits == 2 && g_held);
  for (void* p : others) HostStage::Get().Release(p);
  HostStage::Get().DropUser();
}

// no thread, or fewer than asked for, can be started: the work is done all the same
void ThreadLimit() {
  for (int left : {0, 1, 3}) {
    HostStage::Get().AddUser();
    g_threads_left = left;
    for (int i = 0; i < 3; ++i) Loop(9);
    std::vector<char> from(5u << 20, 'x'), to(from.size());
    HostStage::Get().Copy(to.data(), from.data(), from.size());
    EXPECT(from == to);
    HostStage::Get().DropUser();
  }
}

// a forked child, which has none of the threads, can use what it inherited and give it back
void Fork() {
  HostStage::Get().AddUser();
  Loop(9);
  const pid_t child = fork();
  if (child == 0) {
    alarm(20);
    Loop(9);
    HostStage::Get().DropUser();
    _exit(0);
  }
  int status = -1;
  EXPECT(waitpid(child, &status, 0) == child && status == 0);
  HostStage::Get().DropUser();
}
}  // namespace

int main(int argc, char** argv) {
  const std::string name = argc > 1 ? argv[1] : "";
  if (name == "users") Users();
  else if (name == "thread-limit") ThreadLimit();
  else if (name == "fork") Fork();
  else if (name == "unwinding") Unwinding();
  else return 2;
  return 0;
}
