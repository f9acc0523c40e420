// The pool behind scratch.hpp: one CUDA memory pool per context, found by
// the context's ID (unique for the life of the process, never reused), so a
// pool that went with its context -- cudaDeviceReset -- is never touched
// again.  Allocation is ordered by the caller's stream: calls on several
// streams and threads get memory of their own.
#include "scratch.hpp"

#include <mutex>

namespace chucky {

namespace {

// cuCtxGetCurrent and cuCtxGetId, fetched through the runtime so that the
// library does not link libcuda itself (CUresult is an int-sized enum,
// CUcontext a pointer).
using CtxGetCurrentFn = int (*)(void**);
using CtxGetIdFn = int (*)(void*, unsigned long long*);

void* driver_entry(const char* name)
{
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q{};
  if (cudaGetDriverEntryPointByVersion(name, &fn, 12000, cudaEnableDefault, &q) !=
        cudaSuccess ||
      q != cudaDriverEntryPointSuccess) {
    cudaGetLastError(); // clear a failed lookup
    return nullptr;
  }
  return fn;
}

struct Pool
{
  unsigned long long ctx_id;
  cudaMemPool_t pool;
};

// While another stream is being captured (by this thread, or by any in the
// global mode), making a pool, allocating from it and freeing count as unsafe
// and would invalidate that capture.  Neither touches it: this thread says so
// for the time of the call.
struct CaptureRelaxed
{
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  CaptureRelaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~CaptureRelaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

constexpr int kMaxPools = 64;
std::mutex g_mutex;
Pool g_pools[kMaxPools];
int g_used = 0;

// The current context's pool (nullptr: none and `create` is off, or it
// cannot be made).
cudaMemPool_t pool_of_context(bool create)
{
  std::lock_guard<std::mutex> lock(g_mutex);
  const unsigned long long id = current_context_id();
  for (int i = 0; id && i < g_used; ++i)
    if (g_pools[i].ctx_id == id)
      return g_pools[i].pool;
  int dev = -1;
  if (!id || !create || g_used == kMaxPools || cudaGetDevice(&dev) != cudaSuccess)
    return nullptr;
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  unsigned long long keep = kScratchKept;
  cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  g_pools[g_used++] = Pool{ id, pool };
  return pool;
}

} // namespace

unsigned long long current_context_id()
{
  static const CtxGetCurrentFn get_current =
    reinterpret_cast<CtxGetCurrentFn>(driver_entry("cuCtxGetCurrent"));
  static const CtxGetIdFn get_id = reinterpret_cast<CtxGetIdFn>(driver_entry("cuCtxGetId"));
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0)
    return 0;
  return id;
}

void* scratch_acquire(size_t bytes, cudaStream_t st)
{
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (cs != cudaStreamCaptureStatusNone)
    return nullptr;
  const CaptureRelaxed relaxed;
  const cudaMemPool_t pool = pool_of_context(true);
  void* p = nullptr;
  if (!pool)
    return nullptr;
  if (cudaMallocFromPoolAsync(&p, bytes, pool, st) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}

void scratch_release(void* p, cudaStream_t st)
{
  if (!p)
    return;
  const CaptureRelaxed relaxed;
  cudaFreeAsync(p, st);
}

void scratch_trim()
{
  const CaptureRelaxed relaxed;
  const cudaMemPool_t pool = pool_of_context(false);
  if (pool && cudaMemPoolTrimTo(pool, 0) != cudaSuccess)
    cudaGetLastError();
}

} // namespace chucky
