// Pageable host <-> device copies over several threads (hostcopy.cuh).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <thread>

#include "hostcopy.cuh"

namespace cq {

namespace {

constexpr size_t kPiece = 1 << 20;   // bytes of one staging buffer
constexpr int kMaxThreads = 8;
constexpr int kMaxStageSets = 4;     // concurrent large copies of one process; others go direct
// Below this the threads' start costs more than they save.
constexpr size_t kMinBytes = 8 << 20;

struct StageSet {
  int dev = 0;
  unsigned char* p = nullptr;  // kMaxThreads x 2 buffers
  cudaEvent_t ev[kMaxThreads][2] = {};
};

std::mutex g_mu;
int g_users = 0, g_sets = 0;            // live users; sets in use or free
StageSet* g_free[kMaxStageSets];        // the first g_nfree
int g_nfree = 0;

void destroy(StageSet* s) {
  for (auto& t : s->ev)
    for (cudaEvent_t e : t)
      if (e) cudaEventDestroy(e);
  if (s->p) cudaFreeHost(s->p);
  cudaGetLastError();
  delete s;
}

// a staging set of the current device, or nullptr (none to spare: copy directly)
StageSet* take() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (int i = 0; i < g_nfree; ++i)
      if (g_free[i]->dev == dev) {
        StageSet* s = g_free[i];
        g_free[i] = g_free[--g_nfree];
        return s;
      }
    if (g_users == 0 || g_sets >= kMaxStageSets) return nullptr;
    ++g_sets;
  }
  StageSet* s = new (std::nothrow) StageSet();
  bool ok = s && cudaHostAlloc((void**)&s->p, kMaxThreads * 2 * kPiece, cudaHostAllocDefault) == cudaSuccess;
  if (ok) {
    s->dev = dev;
    for (auto& t : s->ev)
      for (cudaEvent_t& e : t)
        ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) {
    if (s) destroy(s);
    std::lock_guard<std::mutex> lk(g_mu);
    --g_sets;
    return nullptr;
  }
  return s;
}

void give_back(StageSet* s) {
  std::unique_lock<std::mutex> lk(g_mu);
  if (g_users > 0) {
    g_free[g_nfree++] = s;
    return;
  }
  --g_sets;
  lk.unlock();
  destroy(s);
}

int thread_count(size_t bytes) {
  const unsigned hc = std::thread::hardware_concurrency();
  const size_t most = std::min<size_t>(kMaxThreads, std::max(1u, hc / 2));
  return (int)std::max<size_t>(1, std::min(most, bytes / (2 * kPiece)));
}

// work(t) on n threads, this one included; a thread that cannot be started has its share done
// here.  Nothing is thrown while threads run.
template <typename F> void parallel(int n, F&& work) {
  std::thread th[kMaxThreads];
  int started = 1;
  try {
    for (; started < n; ++started) th[started] = std::thread(work, started);
  } catch (const std::exception&) {
  }
  work(0);
  for (int t = started; t < n; ++t) work(t);
  for (int t = 1; t < started; ++t) th[t].join();
}

// Moves `bytes` through the staging set: thread t takes the pieces t, t + n, ...
template <bool TO_DEVICE>
cudaError_t staged(StageSet* set, unsigned char* dst, const unsigned char* src, size_t bytes,
                   cudaStream_t s) {
  const int n = thread_count(bytes);
  const size_t pieces = (bytes + kPiece - 1) / kPiece;
  std::atomic<int> err{cudaSuccess};
  auto check = [&](cudaError_t e) {
    if (e != cudaSuccess) err.store(e);
    return e == cudaSuccess;
  };
  parallel(n, [&](int t) {
    if (!check(cudaSetDevice(set->dev))) return;
    unsigned char* buf[2] = {set->p + (size_t)(2 * t) * kPiece, set->p + (size_t)(2 * t + 1) * kPiece};
    auto size = [&](size_t i) { return std::min(kPiece, bytes - i * kPiece); };
    auto fetch = [&](size_t i, int b) {  // device -> buffer
      return check(cudaMemcpyAsync(buf[b], src + i * kPiece, size(i), cudaMemcpyDeviceToHost, s)) &&
             check(cudaEventRecord(set->ev[t][b], s));
    };
    int b = 0;
    if (TO_DEVICE) {
      for (size_t i = t, k = 0; i < pieces && err.load() == cudaSuccess; i += n, ++k, b ^= 1) {
        if (k >= 2 && !check(cudaEventSynchronize(set->ev[t][b]))) break;
        std::memcpy(buf[b], src + i * kPiece, size(i));
        if (!check(cudaMemcpyAsync(dst + i * kPiece, buf[b], size(i), cudaMemcpyHostToDevice, s)) ||
            !check(cudaEventRecord(set->ev[t][b], s)))
          break;
      }
    } else {
      if ((size_t)t < pieces) fetch(t, 0);
      for (size_t i = t; i < pieces && err.load() == cudaSuccess; i += n, b ^= 1) {
        if (i + n < pieces && !fetch(i + n, b ^ 1)) break;
        if (!check(cudaEventSynchronize(set->ev[t][b]))) break;
        std::memcpy(dst + i * kPiece, buf[b], size(i));
      }
    }
  });
  // every piece has left its buffer before the set is used again, also after an error
  const cudaError_t e = cudaStreamSynchronize(s);
  return err.load() != cudaSuccess ? (cudaError_t)err.load() : e;
}

}  // namespace

namespace {
bool memory_is(const void* p, cudaMemoryType type) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == type;
}
// A staging set for a copy from or to host memory at p that the threads may read and write
// themselves: ordinary memory only.  Page-locked, managed and device memory go to the driver.
StageSet* take_for(const void* p, size_t bytes) {
  return bytes >= kMinBytes && memory_is(p, cudaMemoryTypeUnregistered) ? take() : nullptr;
}
}  // namespace

bool host_is_pinned(const void* p) { return memory_is(p, cudaMemoryTypeHost); }

void copy_to_device(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  StageSet* set = take_for(src, bytes);
  if (!set) {
    CQ_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
    return;
  }
  const cudaError_t e = staged<true>(set, (unsigned char*)dst, (const unsigned char*)src, bytes, s);
  give_back(set);
  CQ_CHECK_CUDA(e);
}

void copy_from_device(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  StageSet* set = take_for(dst, bytes);
  if (!set) {
    CQ_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
    return;
  }
  const cudaError_t e = staged<false>(set, (unsigned char*)dst, (const unsigned char*)src, bytes, s);
  give_back(set);
  CQ_CHECK_CUDA(e);
}

StageUser::StageUser() {
  std::lock_guard<std::mutex> lk(g_mu);
  ++g_users;
}

StageUser::~StageUser() {
  StageSet* gone[kMaxStageSets];
  int n = 0;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (--g_users == 0) {
      n = g_nfree;
      std::copy(g_free, g_free + n, gone);
      g_nfree = 0;
      g_sets -= n;
    }
  }
  for (int i = 0; i < n; ++i) destroy(gone[i]);
}

}  // namespace cq
