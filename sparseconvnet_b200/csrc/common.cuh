// Shared definitions of the sm_100a sparse-convolution library: status handling, the packed
// site key, and the open-addressing site hash used by every rulebook kernel.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <string>

#include "../../include/scn_b200.h"

namespace scn {

// ---- status -----------------------------------------------------------------------------

void set_error(const char *fmt, ...);

#define SCN_CUDA_CHECK(expr)                                                                   \
  do {                                                                                         \
    cudaError_t _e = (expr);                                                                   \
    if (_e != cudaSuccess) {                                                                   \
      scn::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__,         \
                     __LINE__);                                                                \
      return SCN_ERR_CUDA;                                                                     \
    }                                                                                          \
  } while (0)

#define SCN_TRY(expr)                                                                          \
  do {                                                                                         \
    int _s = (expr);                                                                           \
    if (_s != SCN_OK) return _s;                                                               \
  } while (0)

#define SCN_REQUIRE(cond, code, ...)                                                           \
  do {                                                                                         \
    if (!(cond)) {                                                                             \
      scn::set_error(__VA_ARGS__);                                                             \
      return (code);                                                                           \
    }                                                                                          \
  } while (0)

// Every kernel launch of the library goes through this macro so that the number of launches
// can be read back (scn_launch_count), e.g. to state how many kernels a timed region ran.
void note_launch();
// Every place where the library makes the calling thread wait for the GPU (a stream or event
// synchronisation) notes it; scn_host_wait_count reads the total.
void note_host_wait();
// A pass is a chain of up to 250 short kernels on one stream, and each used to start 1 to 2 us after the one before it had
// ended.  They are launched with programmatic stream serialisation: the next kernel's blocks are put in place as the last
// blocks of the one before leave, and wait at their first instruction (SCN_GRID_WAIT).  U-Net on eight rooms (186 launches
// then, 147 since) 6511 -> 6158 us, on one room (178, 139) 2288 -> 1972, one layer on 267 k sites (15, 12) 281 -> 255.  No
// kernel asks for its successor any earlier (griddepcontrol.launch_dependents): blocks that wait in the last wave's free
// places are handed out to whichever SM has room first instead of evenly, 6499, 2079 and 277 us.
#define SCN_LAUNCH(kernel, grid, block, smem, stream, ...)                                      \
  do {                                                                                         \
    scn::note_launch();                                                                        \
    scn::launch_behind(kernel, dim3(grid), dim3(block), (smem), (stream), __VA_ARGS__);        \
  } while (0)
#ifdef __CUDACC__
template <typename... P, typename... A>
inline void launch_behind(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = &attr;
  config.numAttrs = 1;
  cudaLaunchKernelEx(&config, kernel, static_cast<A &&>(args)...);  // (the callers look at cudaGetLastError)
}
#endif
// The first statement of every kernel that SCN_LAUNCH launches, run by all its threads: waits until the kernel before it has
// ended and what it wrote can be seen.  Because every kernel waits here for the one before it, the end of a kernel is also
// the end of all before it.  The branch that is never taken keeps loads that the compiler takes for independent of
// everything (__ldg, const __restrict__) behind the wait.
#define SCN_GRID_WAIT()                                                                        \
  do {                                                                                         \
    unsigned never_;                                                                           \
    asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(never_)::"memory");            \
    if (never_) return;                                                                        \
  } while (0)

// Kernels report problems by OR-ing a bit into a device word; the host reads it at the next
// point where it waits for the stream anyway.  Nothing on the device traps.
enum DeviceFlag : int {
  FLAG_COORD_RANGE = 1,
  FLAG_TABLE_FULL = 2,
  FLAG_BAD_ROW = 4,
  FLAG_TC_TIMEOUT = 8,
};

// ---- packed site key ----------------------------------------------------------------------
//
// A site (batch index, x_0 .. x_{D-1}) is packed into one 64-bit word: coordinate d occupies
// bits [shift[d], shift[d] + bits[d]), the batch index the bits above batch_shift.  Because
// every coordinate is range-checked against its field before packing, the key of a neighbour
// is the site's key plus a precomputed signed delta.  The all-ones word is the empty marker.

constexpr int kMaxDim = SCN_MAX_DIMENSION;
constexpr unsigned long long kEmptyKey = 0xFFFFFFFFFFFFFFFFull;

struct KeyLayout {
  int dim;
  int shift[kMaxDim];
  int bits[kMaxDim];
  int size[kMaxDim];  // spatial size per dimension
  int batch_shift;
  int batch_bits;
};

__host__ __device__ inline unsigned long long pack_key(const KeyLayout &L, const int *x, int b) {
  unsigned long long k = (unsigned long long)(unsigned)b << L.batch_shift;
  for (int d = 0; d < L.dim; ++d) k |= (unsigned long long)(unsigned)x[d] << L.shift[d];
  return k;
}
__host__ __device__ inline void unpack_key(const KeyLayout &L, unsigned long long k, int *x,
                                           int &b) {
  for (int d = 0; d < L.dim; ++d) x[d] = (int)((k >> L.shift[d]) & ((1ull << L.bits[d]) - 1));
  b = (int)(k >> L.batch_shift);
}

// ---- site hash ----------------------------------------------------------------------------
//
// Open addressing over 32-byte buckets of two 16-byte slots, so one probe is one aligned
// 32-byte sector: both slots of a bucket arrive with two 128-bit loads of the same sector.
// Inserts claim the first free slot of the home bucket, then walk to the next bucket.
// Nothing is ever deleted, so a lookup can stop at the first bucket with a free slot.

struct __align__(16) Slot {
  unsigned long long key;  // kEmptyKey when free
  int row;                 // feature-row index of the site (-1 until numbered)
  unsigned aux;            // build-time scratch: smallest id that touched the site
};

struct HashTable {
  Slot *slots;            // 2 * n_buckets slots
  unsigned long long n_buckets;  // power of two
};

__host__ __device__ inline unsigned long long mix64(unsigned long long k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return k;
}

#ifdef __CUDACC__
// The slot of `key`, claimed if it is not there yet, or -1 if the bounded walk gave up.  LAST: the slot's row becomes the
// largest id that named the key; otherwise its aux becomes the smallest.  A free slot is claimed and its id written by one
// 16-byte compare-and-swap (a compare-and-swap on the key and an atomic on the id were two trips to L2).  LOOK: read the
// slot first, where most calls find their key there, named by a smaller id, and need no atomic at all.
// The look is two relaxed 64-bit loads, the key one of them: a key changes once, from free to its value, and is seen as one
// or the other, never half of each (four 32-bit accesses could show half, and the walk would claim the key a second time).
// The id beside it may be older than the key; an old one is larger (LAST: smaller) than the present one and costs an atomic
// that changes nothing.  The 32-bit atomics on row and aux only ever touch slots that are claimed, where the 16-byte
// compare-and-swap fails on the key whatever half it sees of them.
template <bool LAST, bool LOOK>
__device__ inline long long hash_claim(const HashTable &T, unsigned long long key, unsigned id) {
  const unsigned long long mask = T.n_buckets - 1;
  unsigned long long b = mix64(key) & mask;
  const unsigned long long limit = T.n_buckets < 4096 ? T.n_buckets : 4096;
  const Slot vacant{kEmptyKey, -1, 0xFFFFFFFFu}, mine{key, LAST ? (int)id : -1, LAST ? 0xFFFFFFFFu : id};
  for (unsigned long long p = 0; p < limit; ++p) {
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      Slot *at = T.slots + 2 * b + s;
      Slot was = vacant;
      if (LOOK) {
        unsigned long long ids;
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(was.key), "=l"(ids) : "l"(at) : "memory");
        was.row = (int)(unsigned)ids;
        was.aux = (unsigned)(ids >> 32);
      }
      if (was.key == kEmptyKey) was = atomicCAS(at, vacant, mine);
      if (was.key == kEmptyKey) return (long long)(at - T.slots);
      if (was.key == key) {
        if (LAST) {
          if (was.row < (int)id) atomicMax(&at->row, (int)id);
        } else if (was.aux > id) {
          atomicMin(&at->aux, id);
        }
        return (long long)(at - T.slots);
      }
    }
    b = (b + 1) & mask;
  }
  return -1;
}

// Returns the slot index of `key` or -1 when absent.  Read-only tables only.
__device__ inline long long hash_find_slot(const HashTable &T, unsigned long long key) {
  unsigned long long mask = T.n_buckets - 1;
  unsigned long long b = mix64(key) & mask;
  unsigned long long limit = T.n_buckets < 4096 ? T.n_buckets : 4096;
  for (unsigned long long p = 0; p < limit; ++p) {
    const uint4 *q = reinterpret_cast<const uint4 *>(T.slots + 2 * b);
    uint4 s0 = __ldg(q);
    uint4 s1 = __ldg(q + 1);
    unsigned long long k0 = ((unsigned long long)s0.y << 32) | s0.x;
    unsigned long long k1 = ((unsigned long long)s1.y << 32) | s1.x;
    if (k0 == key) return (long long)(2 * b);
    if (k1 == key) return (long long)(2 * b + 1);
    if (k0 == kEmptyKey || k1 == kEmptyKey) return -1;
    b = (b + 1) & mask;
  }
  return -1;
}

// Returns the feature row of `key` or -1 when absent.
__device__ inline int hash_find_row(const HashTable &T, unsigned long long key) {
  unsigned long long mask = T.n_buckets - 1;
  unsigned long long b = mix64(key) & mask;
  unsigned long long limit = T.n_buckets < 4096 ? T.n_buckets : 4096;
  for (unsigned long long p = 0; p < limit; ++p) {
    const uint4 *q = reinterpret_cast<const uint4 *>(T.slots + 2 * b);
    uint4 s0 = __ldg(q);
    uint4 s1 = __ldg(q + 1);
    unsigned long long k0 = ((unsigned long long)s0.y << 32) | s0.x;
    unsigned long long k1 = ((unsigned long long)s1.y << 32) | s1.x;
    if (k0 == key) return (int)s0.z;
    if (k1 == key) return (int)s1.z;
    if (k0 == kEmptyKey || k1 == kEmptyKey) return -1;
    b = (b + 1) & mask;
  }
  return -1;
}
#endif  // __CUDACC__

// ---- small host helpers -------------------------------------------------------------------

inline unsigned long long next_pow2(unsigned long long v) {
  unsigned long long p = 1;
  while (p < v) p <<= 1;
  return p;
}
inline int bit_length(unsigned long long v) {
  int n = 0;
  while (v) {
    ++n;
    v >>= 1;
  }
  return n;
}
inline long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

// Stream-ordered device allocation (cudaMallocAsync on the current device's default pool,
// whose release threshold is raised once so freed blocks are reused instead of returned).
int device_alloc(void **p, size_t bytes, cudaStream_t stream);
int device_free(void *p, cudaStream_t stream);
int test_allocation();  // the test hook of device_alloc, for the pinned buffers too

// Blocks that go back, stream-ordered, on every way out of a function.
class Scratch {
 public:
  explicit Scratch(cudaStream_t stream) : stream_(stream) {}
  Scratch(const Scratch &) = delete;
  ~Scratch() {
    for (int i = 0; i < n_; ++i) device_free(p_[i], stream_);
  }
  template <typename T>
  int get(T **p, size_t bytes) {
    SCN_REQUIRE(n_ < kMost, SCN_ERR_UNSUPPORTED, "more than %d scratch blocks", kMost);
    void *q = nullptr;
    SCN_TRY(device_alloc(&q, bytes, stream_));
    *p = (T *)(p_[n_++] = q);
    return SCN_OK;
  }

 private:
  static constexpr int kMost = 8;
  void *p_[kMost];
  int n_ = 0;
  cudaStream_t stream_;
};

// Exclusive prefix sum of n int32 values (out may alias in).  total_dev (may be null)
// receives the sum of all inputs as int32.
int exclusive_scan_i32(const int *in, int *out, long long n, int *total_dev, cudaStream_t stream);

}  // namespace scn
