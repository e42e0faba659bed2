// Status strings, stream-ordered allocation and the device-wide prefix sum used by the
// rulebook builders.
#include <stdarg.h>

#include <array>
#include <atomic>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "common.cuh"

namespace scn {
void pinned_trim();  // host_keys.cu

static thread_local char g_last_error[512] = "";
static std::atomic<long long> g_launches{0};

void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
static std::atomic<long long> g_host_waits{0};
void note_host_wait() { g_host_waits.fetch_add(1, std::memory_order_relaxed); }

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
}

// The library's memory (site tables, rulebooks, prepared weight images, scratch) comes from a CUDA memory pool of its
// own per device, behind a cache of idle blocks per stream.  A forward pass takes and gives back some 200 blocks of
// the same sizes as the pass before; from the cache that is 0.1 us each instead of 1 to 2 us of driver call, and it
// never has to wait or grow because the pool cannot prove that another stream's free has executed (single passes of
// 18 to 75 ms among 4 to 13 ms ones came from there).
//   * A block freed on a stream is only handed out again to allocations on the same stream (by cudaStreamGetId, which
//     is not reused as handles are), so stream order alone makes the reuse safe, as for cudaFreeAsync.
//   * Sizes are rounded up to four steps per power of two, and a request takes a block up to two steps larger.
//   * While a stream is being captured its blocks come from the pool itself and go back to it, as memory nodes of the graph:
//     an idle block that a graph has been recorded with would be handed out again and written by every replay.
//   * Idle blocks are bounded by an eighth of the device's memory; what comes back beyond that goes to the pool, and
//     the pool returns it to the driver (release threshold 64 MB).  A failing allocation first gives back every idle
//     block, and so does scn_trim_memory; if the rounded size still does not fit, the size itself is tried.
namespace {
constexpr int kSteps = 4 * 40;
int size_step(size_t bytes) {  // the smallest step that holds `bytes`
  if (bytes <= 512) return 0;
  int e = 63 - __builtin_clzll((unsigned long long)bytes - 1);  // 2^e <= bytes - 1 < 2^(e+1)
  const int q = (int)(((bytes - 1) >> (e - 2)) & 3) + 1;        // quarters above 2^e, rounded up
  return (e - 9) * 4 + q;
}
size_t step_bytes(int step) { return ((size_t)512 << (step / 4)) / 4 * (4 + step % 4); }

struct DeviceCache {
  std::mutex mu;
  cudaMemPool_t pool = nullptr;
  size_t idle = 0, used = 0, idle_limit = 0;
  struct Block {
    size_t bytes;
    int step;  // -1: goes back to the pool, not to the idle lists
  };
  std::unordered_map<void *, Block> live;
  std::unordered_map<unsigned long long, std::array<std::vector<void *>, kSteps>> idle_blocks;  // per stream id
};
DeviceCache *const g_cache = new DeviceCache[64];  // never destroyed: objects may be released while the process ends

int device_cache(DeviceCache **out) {
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev >= 0 && dev < 64, SCN_ERR_UNSUPPORTED, "device index %d unsupported", dev);
  *out = &g_cache[dev];
  return SCN_OK;
}

int make_pool(DeviceCache &c) {  // c.mu held
  if (c.pool) return SCN_OK;
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  size_t free_bytes = 0, total = 0;
  SCN_CUDA_CHECK(cudaMemGetInfo(&free_bytes, &total));
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t p = nullptr;
  SCN_CUDA_CHECK(cudaMemPoolCreate(&p, &props));
  unsigned long long keep = 64ull << 20;
  SCN_CUDA_CHECK(cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep));
  c.idle_limit = total / 8;
  c.pool = p;
  return SCN_OK;
}

// Is `stream` being captured?  Otherwise its id, which a stream under capture must not be asked for (the question ends the
// capture).  The legacy stream is never captured, and must not be asked either while a stream it waits for is.
int stream_state(cudaStream_t stream, bool *capture, unsigned long long *id) {
  *capture = false;
  *id = ~0ull;
  if (stream == nullptr || stream == cudaStreamLegacy) return SCN_OK;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  SCN_CUDA_CHECK(cudaStreamIsCapturing(stream, &status));
  *capture = status != cudaStreamCaptureStatusNone;
  if (!*capture) SCN_CUDA_CHECK(cudaStreamGetId(stream, id));
  return SCN_OK;
}

// Gives idle blocks back to the pool until at most `keep` bytes are idle (c.mu held).  They may belong to streams that
// no longer exist, so the device is waited for first.
int release_idle(DeviceCache &c, size_t keep) {
  if (c.idle <= keep) return SCN_OK;
  SCN_CUDA_CHECK(cudaDeviceSynchronize());
  for (auto it = c.idle_blocks.begin(); it != c.idle_blocks.end();) {
    bool empty = true;
    for (int s = kSteps - 1; s >= 0; --s) {
      auto &list = it->second[s];
      while (!list.empty() && c.idle > keep) {
        void *p = list.back();
        list.pop_back();
        c.idle -= step_bytes(s);
        c.live.erase(p);
        SCN_CUDA_CHECK(cudaFreeAsync(p, nullptr));
      }
      empty &= list.empty();
    }
    it = empty ? c.idle_blocks.erase(it) : std::next(it);
  }
  SCN_CUDA_CHECK(cudaStreamSynchronize(nullptr));
  return SCN_OK;
}
}  // namespace

// scn_test_fail_allocation: does the allocation that is being asked for fail?
static thread_local int g_fail_in = 0;
int test_allocation() {
  SCN_REQUIRE(!g_fail_in || --g_fail_in, SCN_ERR_CUDA, "out of memory (asked for by scn_test_fail_allocation)");
  return SCN_OK;
}

int device_alloc(void **p, size_t bytes, cudaStream_t stream) {
  *p = nullptr;
  SCN_TRY(test_allocation());
  DeviceCache *c = nullptr;
  SCN_TRY(device_cache(&c));
  unsigned long long id = 0;
  bool capture = false;
  SCN_TRY(stream_state(stream, &capture, &id));
  const int step = size_step(bytes);
  SCN_REQUIRE(step < kSteps, SCN_ERR_UNSUPPORTED, "allocation of %zu bytes", bytes);
  std::lock_guard<std::mutex> lock(c->mu);
  auto mine = capture ? c->idle_blocks.end() : c->idle_blocks.find(id);
  if (mine != c->idle_blocks.end())
    for (int s = step; s <= step + 2 && s < kSteps; ++s) {
      auto &list = mine->second[s];
      if (list.empty()) continue;
      *p = list.back();
      list.pop_back();
      c->idle -= step_bytes(s);
      c->used += step_bytes(s);
      return SCN_OK;
    }
  SCN_TRY(make_pool(*c));
  DeviceCache::Block block{step_bytes(step), capture ? -1 : step};
  cudaError_t e = cudaMallocFromPoolAsync(p, block.bytes, c->pool, stream);
  if (e == cudaErrorMemoryAllocation && !capture) {
    cudaGetLastError();
    SCN_TRY(release_idle(*c, 0));
    SCN_CUDA_CHECK(cudaMemPoolTrimTo(c->pool, 0));
    e = cudaMallocFromPoolAsync(p, block.bytes, c->pool, stream);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      block = {bytes ? bytes : 1, -1};
      e = cudaMallocFromPoolAsync(p, block.bytes, c->pool, stream);
    }
  }
  SCN_CUDA_CHECK(e);
  c->live[*p] = block;
  c->used += block.bytes;
  return SCN_OK;
}

int device_free(void *p, cudaStream_t stream) {
  if (!p) return SCN_OK;
  DeviceCache *c = nullptr;
  SCN_TRY(device_cache(&c));
  unsigned long long id = 0;
  bool capture = false;
  SCN_TRY(stream_state(stream, &capture, &id));
  std::lock_guard<std::mutex> lock(c->mu);
  auto it = c->live.find(p);
  SCN_REQUIRE(it != c->live.end(), SCN_ERR_BAD_ARG, "freed memory is not a block of the current device");
  const size_t bytes = it->second.bytes;
  // (nobody may write it any more, the graph reads it at every replay: it stays taken)
  SCN_REQUIRE(it->second.step < 0 || !capture, SCN_ERR_UNSUPPORTED, "memory taken before a stream capture cannot be given back inside it");
  c->used -= bytes;
  if (it->second.step < 0 || c->idle + bytes > c->idle_limit) {
    c->live.erase(it);
    SCN_CUDA_CHECK(cudaFreeAsync(p, stream));
    return SCN_OK;
  }
  c->idle += bytes;
  c->idle_blocks[id][it->second.step].push_back(p);
  return SCN_OK;
}

// ---- exclusive scan -----------------------------------------------------------------------
// Three passes over tiles of 4096 values: per-tile sums, a recursive scan of those sums, and
// a per-tile scan seeded with the tile's base.  All int32; callers keep totals below 2^31.

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ inline int block_exclusive_scan(int v, int &block_total) {
  __shared__ int warp_sums[32];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = warp_sums[lane];
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_sums[lane] = wi - w;  // exclusive offset of each warp
    if (lane == 31) block_total = wi;
  }
  __syncthreads();
  int base = warp_sums[warp];
  return base + incl - v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tile_sums(const int *in, int *tile_sums,
                                                                 long long n) {
  SCN_GRID_WAIT();
  __shared__ int total;
  long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i)
    if (base + i < n) s += in[base + i];
  block_exclusive_scan(s, total);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const int *in, int *out,
                                                             const int *tile_base, long long n,
                                                             int *total_dev) {
  SCN_GRID_WAIT();
  __shared__ int total;
  long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = (base + i < n) ? in[base + i] : 0;
    s += v[i];
  }
  int excl = block_exclusive_scan(s, total) + (tile_base ? tile_base[blockIdx.x] : 0);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) out[base + i] = excl;
    excl += v[i];
  }
  if (total_dev && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
    *total_dev = total + (tile_base ? tile_base[blockIdx.x] : 0);
}

__global__ void k_set_zero(int *p) {
  SCN_GRID_WAIT(); *p = 0; }

int exclusive_scan_i32(const int *in, int *out, long long n, int *total_dev, cudaStream_t stream) {
  if (n <= 0) {
    if (total_dev) SCN_LAUNCH(k_set_zero, 1, 1, 0, stream, total_dev);
    return SCN_OK;
  }
  long long tiles = ceil_div(n, kScanTile);
  if (tiles == 1) {
    SCN_LAUNCH(k_scan_tiles, 1, kScanThreads, 0, stream, in, out, nullptr, n, total_dev);
    SCN_CUDA_CHECK(cudaGetLastError());
    return SCN_OK;
  }
  int *sums = nullptr;
  SCN_TRY(device_alloc((void **)&sums, sizeof(int) * (size_t)tiles, stream));
  SCN_LAUNCH(k_scan_tile_sums, (unsigned)tiles, kScanThreads, 0, stream, in, sums, n);
  SCN_CUDA_CHECK(cudaGetLastError());
  SCN_TRY(exclusive_scan_i32(sums, sums, tiles, nullptr, stream));
  SCN_LAUNCH(k_scan_tiles, (unsigned)tiles, kScanThreads, 0, stream, in, out, sums, n, total_dev);
  SCN_CUDA_CHECK(cudaGetLastError());
  return device_free(sums, stream);
}

}  // namespace scn

extern "C" {

int scn_abi_version(void) { return SCN_ABI_VERSION; }

long long scn_launch_count(void) { return scn::g_launches.load(std::memory_order_relaxed); }
long long scn_host_wait_count(void) { return scn::g_host_waits.load(std::memory_order_relaxed); }

int scn_memory_usage(uint64_t *reserved_bytes, uint64_t *used_bytes) {
  using namespace scn;
  SCN_REQUIRE(reserved_bytes && used_bytes, SCN_ERR_BAD_ARG, "null argument");
  *reserved_bytes = *used_bytes = 0;
  DeviceCache *c = nullptr;
  SCN_TRY(device_cache(&c));
  std::lock_guard<std::mutex> lock(c->mu);
  if (c->pool) {
    unsigned long long r = 0;
    SCN_CUDA_CHECK(cudaMemPoolGetAttribute(c->pool, cudaMemPoolAttrReservedMemCurrent, &r));
    *reserved_bytes = r;
    *used_bytes = c->used;
  }
  return SCN_OK;
}

int scn_test_fail_allocation(int which) {
  const int left = scn::g_fail_in;
  scn::g_fail_in = which > 0 ? which : 0;
  return left;
}

int scn_trim_memory(uint64_t keep_bytes) {
  using namespace scn;
  pinned_trim();
  DeviceCache *c = nullptr;
  SCN_TRY(device_cache(&c));
  std::lock_guard<std::mutex> lock(c->mu);
  if (!c->pool) return SCN_OK;
  SCN_TRY(release_idle(*c, keep_bytes > c->used ? (size_t)(keep_bytes - c->used) : 0));
  SCN_CUDA_CHECK(cudaMemPoolTrimTo(c->pool, (size_t)keep_bytes));
  return SCN_OK;
}

const char *scn_last_error(void) { return scn::g_last_error; }

const char *scn_status_string(int status) {
  switch (status) {
    case SCN_OK: return "ok";
    case SCN_ERR_BAD_ARG: return "bad argument";
    case SCN_ERR_CUDA: return "CUDA runtime error";
    case SCN_ERR_COORD_RANGE: return "coordinate or batch index out of range";
    case SCN_ERR_KEY_BITS: return "spatial size x batch does not fit a 63-bit site key";
    case SCN_ERR_NO_GRID: return "no grid for that spatial size";
    case SCN_ERR_TABLE_FULL: return "site hash probe limit reached";
    case SCN_ERR_UNSUPPORTED: return "unsupported shape";
    case SCN_ERR_SIZE_MISMATCH: return "size mismatch";
    default: return "unknown status";
  }
}
}
