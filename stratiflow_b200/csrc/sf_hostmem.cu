// Host memory for results (sf_host_alloc). A result of megabytes arrives by one
// direct copy only in page-locked memory (10.5 MB: 0.2 ms, 0.64 through the
// driver's staging, 1.3 with the first touch of new pages). But page-locked
// memory in a caller's hands changes what the caller's own calls do: a copy to
// the device is no longer staged, so it still reads the array after it was
// changed or dropped; cudaHostAlloc's memory goes with the device's context;
// and a forked child shares it. So a block is mapped twice: the library's view
// is registered with the driver and takes the copies, the caller's view of the
// same pages is not, and counts as ordinary memory. A fork waits until the
// child has moved its views to pages of its own.
#include <cuda_runtime.h>
#include <fcntl.h>
#include <pthread.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cerrno>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>

#include "../../include/stratiflow_b200.h"

extern void sf_set_error_message(const std::string& msg);

namespace {

struct Block {
  void* dma;
  size_t bytes;   // whole pages
};
struct Blocks {
  std::mutex mu;
  std::map<void*, Block> by_view;   // the caller's view -> the library's
  int pipe[2] = {-1, -1};           // of a fork in progress
};
Blocks& blocks() {
  static Blocks* b = new Blocks;   // outlives the exit handlers, which may still free arrays
  return *b;
}

// cudaHostRegister is refused while another thread captures a stream, and
// would spoil its capture, unless this thread's mode is relaxed
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

void before_fork() {
  Blocks& b = blocks();
  b.mu.lock();
  if (b.by_view.empty() || pipe2(b.pipe, O_CLOEXEC) != 0) b.pipe[0] = b.pipe[1] = -1;
}
// returns when the child has its own pages (or is gone: the pipe's other end closes)
void after_fork_parent() {
  Blocks& b = blocks();
  if (b.pipe[0] >= 0) {
    close(b.pipe[1]);
    char c;
    while (read(b.pipe[0], &c, 1) < 0 && errno == EINTR) {
    }
    close(b.pipe[0]);
  }
  b.mu.unlock();
}
void after_fork_child() {
  Blocks& b = blocks();
  for (auto& v : b.by_view) {
    void* p = mmap(nullptr, v.second.bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) continue;
    std::memcpy(p, v.first, v.second.bytes);
    if (mremap(p, v.second.bytes, v.second.bytes, MREMAP_MAYMOVE | MREMAP_FIXED, v.first) == MAP_FAILED)
      munmap(p, v.second.bytes);
    munmap(v.second.dma, v.second.bytes);
  }
  b.by_view.clear();
  if (b.pipe[0] >= 0) {
    close(b.pipe[0]);
    close(b.pipe[1]);
  }
  b.mu.unlock();
}

}  // namespace

// where the library's copies to and from p go: the registered view of a block that holds p
void* sf_host_dma(const void* p) {
  Blocks& b = blocks();
  char* c = static_cast<char*>(const_cast<void*>(p));
  std::lock_guard<std::mutex> lock(b.mu);
  auto it = b.by_view.upper_bound(c);
  if (it == b.by_view.begin()) return c;
  --it;
  const size_t off = (size_t)(c - static_cast<char*>(it->first));
  return off < it->second.bytes ? static_cast<char*>(it->second.dma) + off : c;
}

extern "C" {

int sf_host_alloc(size_t bytes, void** ptr) {
  if (!ptr || bytes == 0) {
    sf_set_error_message("bad argument");
    return SF_EINVAL;
  }
  static const int hooked = pthread_atfork(before_fork, after_fork_parent, after_fork_child);
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = (bytes + page - 1) / page * page;
  void *dma = MAP_FAILED, *view = MAP_FAILED;
  const int fd = hooked == 0 ? memfd_create("stratiflow results", MFD_CLOEXEC) : -1;
  if (fd >= 0 && ftruncate(fd, (off_t)n) == 0) {
    dma = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_SHARED | MAP_POPULATE, fd, 0);
    view = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_SHARED | MAP_POPULATE, fd, 0);
  }
  if (fd >= 0) close(fd);
  if (dma == MAP_FAILED || view == MAP_FAILED) {
    if (dma != MAP_FAILED) munmap(dma, n);
    if (view != MAP_FAILED) munmap(view, n);
    sf_set_error_message("sf_host_alloc: no memory");
    return SF_ENOMEM;
  }
  {
    RelaxedCapture relaxed;
    if (cudaHostRegister(dma, n, cudaHostRegisterPortable) != cudaSuccess) cudaGetLastError();   // slower copies
  }
  try {
    Blocks& b = blocks();
    std::lock_guard<std::mutex> lock(b.mu);
    b.by_view[view] = Block{dma, n};
  } catch (const std::bad_alloc&) {
    RelaxedCapture relaxed;
    if (cudaHostUnregister(dma) != cudaSuccess) cudaGetLastError();
    munmap(dma, n);
    munmap(view, n);
    sf_set_error_message("sf_host_alloc: no memory");
    return SF_ENOMEM;
  }
  *ptr = view;
  return SF_OK;
}

int sf_host_free(void* ptr) {
  if (!ptr) return SF_OK;
  Blocks& b = blocks();
  Block k;
  {
    std::lock_guard<std::mutex> lock(b.mu);
    const auto it = b.by_view.find(ptr);
    if (it == b.by_view.end()) {
      sf_set_error_message("sf_host_free: not a block of sf_host_alloc");
      return SF_EINVAL;
    }
    k = it->second;
    b.by_view.erase(it);
  }
  {
    RelaxedCapture relaxed;
    if (cudaHostUnregister(k.dma) != cudaSuccess) cudaGetLastError();   // after a reset of the device
  }
  munmap(k.dma, k.bytes);
  munmap(ptr, k.bytes);
  return SF_OK;
}

}  // extern "C"
