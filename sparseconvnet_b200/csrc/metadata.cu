// The Metadata object: GPU site hash per spatial scale and the rulebook builders.
//
// Replaces, with device kernels and no host round trip for the rules themselves,
//   Metadata<D>::inputLayer / inputLayerRules     (Metadata.cpp:413-425, IOLayersRules.h:18-121)
//   Metadata<D>::getSubmanifoldRuleBook           (Metadata.cpp:437-451,
//                                                  SubmanifoldConvolutionRules.h:11-87)
//   Metadata<D>::getRuleBook                      (Metadata.cpp:492-518, ConvolutionRules.h:11-105,
//                                                  RectangularRegions.h:94-119)
//   Metadata<D>::getSpatialLocations              (Metadata.cpp:149-170)
// of the reference.  Only counts (active sites, rules per offset) ever travel to the host.
#include <stdlib.h>

#include <algorithm>
#include <climits>

#include <atomic>
#include <mutex>

#include "metadata.cuh"

namespace scn {

static std::atomic<long long> g_rulebook_builds{0};  // rulebooks constructed (not served from a cache)

// ------------------------------------------------------------------------------------------
// key layout
// ------------------------------------------------------------------------------------------

static int make_layout(int dim, const int64_t *size, KeyLayout &L) {
  L = KeyLayout{};
  L.dim = dim;
  int sh = 0;
  for (int d = dim - 1; d >= 0; --d) {  // last dimension in the lowest bits
    SCN_REQUIRE(size[d] >= 1 && size[d] <= INT_MAX, SCN_ERR_BAD_ARG,
                "spatial size[%d]=%lld out of range", d, (long long)size[d]);
    int bits = std::max(1, bit_length((unsigned long long)size[d] - 1));
    L.shift[d] = sh;
    L.bits[d] = bits;
    L.size[d] = (int)size[d];
    sh += bits;
  }
  SCN_REQUIRE(sh <= 62, SCN_ERR_KEY_BITS, "spatial size needs %d key bits (max 62)", sh);
  L.batch_shift = sh;
  L.batch_bits = std::min(31, 63 - sh);
  return SCN_OK;
}

std::vector<int64_t> make_key(int dim, const int64_t *a, const int64_t *b, const int64_t *c) {
  std::vector<int64_t> k(a, a + dim);
  if (b) k.insert(k.end(), b, b + dim);
  if (c) k.insert(k.end(), c, c + dim);
  return k;
}

int md_touch(scn_metadata *md, cudaStream_t stream) {
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  if (md->device < 0) md->device = dev;
  SCN_REQUIRE(md->device == dev, SCN_ERR_BAD_ARG, "metadata object lives on device %d, current device is %d",
              md->device, dev);
  md->last_stream = stream;
  return SCN_OK;
}

static int chain_finalize(scn_metadata *md, cudaStream_t stream, int *n_built, bool on_host = false);
static void chain_abandon(scn_metadata *md, cudaStream_t stream);

static Grid *find_grid_now(scn_metadata *md, const int64_t *spatial_size) {  // no pending chain is waited for
  auto it = md->grids.find(make_key(md->dim, spatial_size));
  return it == md->grids.end() ? nullptr : &it->second;
}

Grid *find_grid(scn_metadata *md, const int64_t *spatial_size) {
  Grid *g = find_grid_now(md, spatial_size);
  if (!g && md->pending) {
    // the grid may be one of a chain that was started on the side stream: take the chain over, then look again.  Nobody
    // says which stream will read the grid (a caller that can takes the chain over itself, before), so the host waits
    // until the tables are finished.
    if (chain_finalize(md, md->last_stream, nullptr, true) != SCN_OK) return nullptr;
    g = find_grid_now(md, spatial_size);
  }
  return g;
}

static int alloc_table(HashTable &T, long long expected_sites, cudaStream_t stream) {
  unsigned long long slots = next_pow2((unsigned long long)std::max<long long>(64, 2 * expected_sites));
  SCN_REQUIRE(slots < (1ull << 31), SCN_ERR_UNSUPPORTED, "site table too large (%llu slots)", slots);
  T.n_buckets = slots / 2;
  return device_alloc((void **)&T.slots, slots * sizeof(Slot), stream);
}

// ---- what the builders start from ------------------------------------------------------------------
// Site tables and rule tables all ones (a free key, no row), counters zero: up to kMaxFills arrays in ONE launch, for a
// whole chain of levels at once.  (One memset each was three calls of 3 to 10 us on the host per level.)
constexpr int kMaxFills = 48;
struct Fills {
  int *p[kMaxFills];
  long long n[kMaxFills];  // 4-byte words
  unsigned ones;           // no: zeros
  unsigned ones_hi;
  int count;
};
static void fill_add(Fills &f, void *p, size_t bytes, bool ones) {
  if (!bytes) return;
  f.p[f.count] = (int *)p;
  f.n[f.count] = (long long)(bytes / 4);
  if (ones) (f.count < 32 ? f.ones : f.ones_hi) |= 1u << (f.count & 31);
  ++f.count;
}

__global__ void __launch_bounds__(256) k_fill(const __grid_constant__ Fills f) {
  SCN_GRID_WAIT();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  for (int a = 0; a < f.count; ++a) {
    const int v = (((a < 32 ? f.ones : f.ones_hi) >> (a & 31)) & 1u) ? -1 : 0;
    int *p = f.p[a];
    const long long n = f.n[a];
    const bool wide = (uintptr_t)p % 16 == 0;
    const long long n4 = wide ? n / 4 : 0;
    for (long long j = i; j < n4; j += step) reinterpret_cast<int4 *>(p)[j] = make_int4(v, v, v, v);
    for (long long j = n4 * 4 + i; j < n; j += step) p[j] = v;
  }
}

static int fill_launch(const Fills &f, cudaStream_t stream) {
  long long most = 0;
  for (int a = 0; a < f.count; ++a) most = std::max(most, f.n[a]);
  if (!most) return SCN_OK;
  SCN_LAUNCH(k_fill, (unsigned)std::min<long long>(148 * 8, ceil_div(most, 4 * 256)), 256, 0, stream, f);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

static void free_grid(Grid &g, cudaStream_t stream) {
  device_free(g.row_keys, stream);
  device_free(g.table.slots, stream);
  g = Grid{};
}
static void free_rulebook(Rulebook &r, cudaStream_t stream) {
  count_ticket_release(r.ticket);
  device_free(r.nbr, stream);
  device_free(r.tnbr, stream);
  device_free(r.counts_dev, stream);
  device_free(r.masks, stream);
  free_row_order(r.order, stream);
  free_row_order(r.torder, stream);
  r = Rulebook{};
}

static int ensure_scratch(scn_metadata *md, cudaStream_t stream) {
  if (!md->flags_dev) {
    SCN_TRY(device_alloc((void **)&md->flags_dev, sizeof(int), stream));
    SCN_CUDA_CHECK(cudaMemsetAsync(md->flags_dev, 0, sizeof(int), stream));
  }
  if (!md->scalars_dev) SCN_TRY(device_alloc((void **)&md->scalars_dev, 4 * sizeof(int), stream));
  return SCN_OK;
}

// ---- host mailboxes -------------------------------------------------------------------------------
// The few integers the host has to wait for (flag word, site counts) are written by a one-thread
// kernel into pinned host memory that is mapped into the device's address space, not copied by
// cudaMemcpy: a device-to-host copy queues on the copy engine behind whatever the application is
// copying at the time (a previous batch's 127 MB of results held every such read-back up for 2 ms,
// once per strided level of a U-Net forward).  Slots of 256 bytes from slabs that are never given back.
constexpr int kMailboxBytes = 256;  // 64 integers: flag word + the counts of a whole chain of levels
namespace {
struct MailboxPool {
  std::mutex mu;
  std::vector<int *> free_slots;
};
MailboxPool &mailbox_pool() {
  static MailboxPool *p = new MailboxPool();
  return *p;
}
}  // namespace

static int mailbox_acquire(int **slot) {
  MailboxPool &P = mailbox_pool();
  std::lock_guard<std::mutex> lock(P.mu);
  if (P.free_slots.empty()) {
    int *slab = nullptr;
    SCN_CUDA_CHECK(cudaHostAlloc((void **)&slab, 4096, cudaHostAllocMapped | cudaHostAllocPortable));
    for (int i = 0; i < 4096 / kMailboxBytes; ++i) P.free_slots.push_back(slab + i * (kMailboxBytes / 4));
  }
  *slot = P.free_slots.back();
  P.free_slots.pop_back();
  return SCN_OK;
}

static void mailbox_release(int *slot) {
  if (!slot) return;
  MailboxPool &P = mailbox_pool();
  std::lock_guard<std::mutex> lock(P.mu);
  P.free_slots.push_back(slot);
}

// ---- rule counts: pinned chunks are pooled per device and never given back to the driver -----------------------
namespace {
constexpr int kTicketValues = 256;  // filter volumes up to 256 offsets
struct TicketPool {
  std::mutex mu;
  std::vector<unsigned long long *> chunks[64];  // kTicketValues values each
  std::vector<CountTicket *> dropped[64];        // released before the device had written their counts (or just now)
};
TicketPool &ticket_pool() {
  static TicketPool *p = new TicketPool();  // leaked on purpose: tickets may be released at exit
  return *p;
}
}  // namespace

static bool counts_landed(const CountTicket *t);

// A ticket for a rulebook that is about to be built (none above kTicketValues offsets).
static int count_ticket_new(Rulebook &rb) {
  if (rb.ticket || rb.n_offsets > kTicketValues) return SCN_OK;
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev < 64, SCN_ERR_UNSUPPORTED, "device %d", dev);
  unsigned long long *host = nullptr;
  CountTicket *t = nullptr;
  TicketPool &P = ticket_pool();
  {
    std::lock_guard<std::mutex> lock(P.mu);
    auto &dropped = P.dropped[dev];
    for (size_t i = 0; i < dropped.size() && !host; ++i)
      if (counts_landed(dropped[i])) {
        t = dropped[i];
        host = (unsigned long long *)t->host;
        dropped[i] = dropped.back();
        dropped.pop_back();
      }
    if (!host && !P.chunks[dev].empty()) {
      host = P.chunks[dev].back();
      P.chunks[dev].pop_back();
    }
    if (!host) {  // a slab of 256 chunks (512 KB of pinned memory) at a time
      unsigned long long *slab = nullptr;
      if (cudaHostAlloc((void **)&slab, sizeof(unsigned long long) * kTicketValues * 256,
                        cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        SCN_REQUIRE(false, SCN_ERR_CUDA, "pinned allocation failed");
      }
      host = slab;
      for (int i = 1; i < 256; ++i) P.chunks[dev].push_back(slab + (size_t)i * kTicketValues);
    }
  }
  unsigned long long *host_dev = t ? t->dev : nullptr;
  if (!t) {
    t = new CountTicket();
    if (cudaHostGetDevicePointer((void **)&host_dev, host, 0) != cudaSuccess) {
      cudaGetLastError();
      delete t;
      std::lock_guard<std::mutex> lock(P.mu);
      P.chunks[dev].push_back(host);
      SCN_REQUIRE(false, SCN_ERR_CUDA, "pinned memory is not mapped");
    }
  }
  t->host = host;
  t->dev = host_dev;
  t->n = rb.n_offsets;
  t->device = dev;
  t->refs.store(1);
  for (int k = 0; k < t->n; ++k) t->host[k] = kCountPending;
  rb.ticket = t;
  return SCN_OK;
}
static unsigned long long *ticket_dev(const Rulebook &rb) { return rb.ticket ? rb.ticket->dev : nullptr; }
static void count_ticket_zero(Rulebook &rb) {  // nothing will be launched: no rules
  if (rb.ticket)
    for (int k = 0; k < rb.ticket->n; ++k) rb.ticket->host[k] = 0;
}

__global__ void k_post_flags(int *flags_dev, volatile int *mailbox) {
  SCN_GRID_WAIT();
  mailbox[0] = *flags_dev;
  *flags_dev = 0;
  __threadfence_system();
}

// Where the last block of a pass leaves what the host waits for: pinned, device-mapped words.  `ready` is written last.
constexpr int kNotPosted = INT_MIN;
struct HostPost {
  volatile int *ready, *flags, *total, *extra;  // each may be null
};
__device__ __forceinline__ void post_to_host(const HostPost &h, int *flags_dev, bool clear_flags, int total, const int *extra) {
  if (h.flags) *h.flags = clear_flags ? atomicExch(flags_dev, 0) : *(volatile int *)flags_dev;
  if (h.total) *h.total = total;
  if (h.extra) *h.extra = *(const volatile int *)extra;
  if (h.ready) {
    __threadfence_system();
    *h.ready = 0;
  }
  __threadfence_system();
}

// Waits for a post.  The word itself is looked at for a while (it arrives a few us before cudaStreamSynchronize would
// return, and the stream may still be working on what follows); then the host sleeps on the stream.
static inline void cpu_relax() {
#if defined(__x86_64__)
  asm volatile("pause");
#elif defined(__aarch64__)
  asm volatile("yield");
#endif
}
static int wait_posted(const volatile int *ready, cudaStream_t stream) {
  note_host_wait();
  for (int i = 0; i < 20000; ++i) {
    if (*ready != kNotPosted) {
      std::atomic_thread_fence(std::memory_order_acquire);
      return SCN_OK;
    }
    cpu_relax();
  }
  SCN_CUDA_CHECK(cudaStreamSynchronize(stream));
  SCN_REQUIRE(*ready != kNotPosted, SCN_ERR_CUDA, "a site count did not arrive");
  return SCN_OK;
}

// Reads (and clears) the device flag word; waits for the stream.
static int fetch_flags(scn_metadata *md, cudaStream_t stream, int *flags) {
  if (!md->mailbox) SCN_TRY(mailbox_acquire(&md->mailbox));
  int *mailbox_dev = nullptr;
  SCN_CUDA_CHECK(cudaHostGetDevicePointer((void **)&mailbox_dev, md->mailbox, 0));
  SCN_LAUNCH(k_post_flags, 1, 1, 0, stream, md->flags_dev, mailbox_dev);
  SCN_CUDA_CHECK(cudaGetLastError());
  note_host_wait();
  SCN_CUDA_CHECK(cudaStreamSynchronize(stream));
  *flags = *(const volatile int *)md->mailbox;
  return SCN_OK;
}

// A mailbox whose first word is "not posted", and the device's view of it: [0] ready, [1] flags, [2] total, [3] extra.
static int post_begin(scn_metadata *md, HostPost &h) {
  if (!md->mailbox) SCN_TRY(mailbox_acquire(&md->mailbox));
  int *dev = nullptr;
  SCN_CUDA_CHECK(cudaHostGetDevicePointer((void **)&dev, md->mailbox, 0));
  *(volatile int *)md->mailbox = kNotPosted;
  h.ready = dev;
  h.flags = dev + 1;
  h.total = dev + 2;
  h.extra = dev + 3;
  return SCN_OK;
}

static int flags_to_status(int flags) {
  if (flags & FLAG_COORD_RANGE) {
    set_error("a coordinate or batch index lies outside the spatial size");
    return SCN_ERR_COORD_RANGE;
  }
  if (flags & FLAG_TABLE_FULL) {
    set_error("site hash probe limit reached");
    return SCN_ERR_TABLE_FULL;
  }
  if (flags & FLAG_TC_TIMEOUT) {
    set_error("a bounded wait inside the tensor-core convolution kernel expired");
    return SCN_ERR_CUDA;
  }
  if (flags & FLAG_BAD_ROW) {
    set_error("a rulebook entry points outside the feature matrix");
    return SCN_ERR_SIZE_MISMATCH;
  }
  return SCN_OK;
}

// The site kernels are compiled for 1 to 4 dimensions (and once for any number): with the number of dimensions known only
// at run time a site's coordinates lived in local memory, 5 M sectors each way beside the 6 M of the table for 400 k sites.
template <int DIM>
__device__ __forceinline__ void unpack_site(const KeyLayout &L, unsigned long long k, int (&x)[DIM ? DIM : kMaxDim], int &b) {
  const int dim = DIM ? DIM : L.dim;
#pragma unroll
  for (int d = 0; d < dim; ++d) x[d] = (int)(k >> L.shift[d]) & (int)((1u << L.bits[d]) - 1u);
  b = (int)(k >> L.batch_shift);
}
template <int DIM>
__device__ __forceinline__ unsigned long long pack_site(const KeyLayout &L, const int (&x)[DIM ? DIM : kMaxDim], int b) {
  const int dim = DIM ? DIM : L.dim;
  unsigned long long k = (unsigned long long)(unsigned)b << L.batch_shift;
#pragma unroll
  for (int d = 0; d < dim; ++d) k |= (unsigned long long)(unsigned)x[d] << L.shift[d];
  return k;
}
#define SCN_LAUNCH_DIM(dim, kernel, ...)                                     \
  do {                                                                       \
    switch (dim) {                                                           \
      case 1: SCN_LAUNCH(kernel<1>, __VA_ARGS__); break;                     \
      case 2: SCN_LAUNCH(kernel<2>, __VA_ARGS__); break;                     \
      case 3: SCN_LAUNCH(kernel<3>, __VA_ARGS__); break;                     \
      case 4: SCN_LAUNCH(kernel<4>, __VA_ARGS__); break;                     \
      default: SCN_LAUNCH(kernel<0>, __VA_ARGS__);                           \
    }                                                                        \
  } while (0)

// ------------------------------------------------------------------------------------------
// input layer
// ------------------------------------------------------------------------------------------

// One thread per input row: range-check, pack, insert.  mode 0 keeps the largest row index
// per site (the reference's serial `mp[p] = i` leaves the last writer, IOLayersRules.h:41,55);
// the other modes record the first row that touched the site.
// bl_length > 0: coords are [batch, bl_length, dim] (BLInputLayer, IOLayersRules.h:134-288):
// the sample index is i / bl_length and a point whose first coordinate is negative is empty.
// packed (coordinates that came from the host): the checked keys, the empty key for an empty slot.
template <int DIM>
__global__ void k_insert_input(KeyLayout L, HashTable T, const long long *__restrict__ coords,
                               const unsigned long long *__restrict__ packed,
                               long long n, int ncols, int mode, long long bl_length,
                               unsigned long long *__restrict__ row_keys, int *__restrict__ slot_of,
                               int *flags, int *n_samples) {
  SCN_GRID_WAIT();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long key = kEmptyKey;
  long long bl = -1;
  if (packed) {
    key = packed[i];
  } else {
    const long long *c = coords + i * ncols;
    if (!(bl_length > 0 && c[0] < 0)) {  // otherwise an empty slot of the batch x length array: in no map, in no rule
      constexpr int kDim = DIM ? DIM : kMaxDim;
      const int dim = DIM ? DIM : L.dim;
      int x[kDim];
      bool ok = true;
#pragma unroll
      for (int d = 0; d < dim; ++d) {
        long long v = c[d];
        ok &= (v >= 0 && v < L.size[d]);
        x[d] = (int)v;
      }
      bl = bl_length > 0 ? i / bl_length : ((ncols > L.dim) ? c[L.dim] : 0);
      ok &= (bl >= 0 && bl < (1ll << L.batch_bits));
      if (ok)
        key = pack_site<DIM>(L, x, (int)bl);
      else
        atomicOr(flags, FLAG_COORD_RANGE);
    }
  }
  if (key == kEmptyKey) {
    if (mode == 0) row_keys[i] = kEmptyKey;
    slot_of[i] = -1;
    return;
  }
  const long long s = mode == 0 ? hash_claim<true, false>(T, key, (unsigned)i) : hash_claim<false, false>(T, key, (unsigned)i);
  if (s < 0) {
    atomicOr(flags, FLAG_TABLE_FULL);
    if (mode == 0) row_keys[i] = kEmptyKey;
    slot_of[i] = -1;
    return;
  }
  // batch indices in use: one atomic per warp, and none once the word already holds the value
  if (!packed) {
    const unsigned peers = __activemask();
    const int warp_max = __reduce_max_sync(peers, (int)bl + 1);
    if ((threadIdx.x & 31) == __ffs(peers) - 1 && warp_max > *(volatile int *)n_samples) atomicMax(n_samples, warp_max);
  }
  slot_of[i] = (int)s;
  if (mode == 0) row_keys[i] = key;
}

// The same for the checked keys of coordinates that came from the host, in pinned memory: bits 0 to 31 of every key, bits 32 to
// 39 and 40 to 47 in bytes of their own (null: no key has them).  Bound by the bus: as 8-byte keys 93 k points of 21 bits took 54 us,
// 32 now, 400 k of 37 bits 190, 115.  (Four points a thread, so that the bytes are requests of 128 too: 48 and 110.)
__global__ void __launch_bounds__(256)
k_insert_narrow(HashTable T, const unsigned *__restrict__ low, const unsigned char *__restrict__ high0,
                const unsigned char *__restrict__ high1, long long n, int mode, unsigned long long *__restrict__ row_keys,
                int *__restrict__ slot_of, int *flags) {
  SCN_GRID_WAIT();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long key = low[i];
  if (high0) key |= (unsigned long long)high0[i] << 32;
  if (high1) key |= (unsigned long long)high1[i] << 40;
  const long long s = mode == 0 ? hash_claim<true, false>(T, key, (unsigned)i) : hash_claim<false, false>(T, key, (unsigned)i);
  if (s < 0) atomicOr(flags, FLAG_TABLE_FULL);
  slot_of[i] = s < 0 ? -1 : (int)s;
  if (mode == 0) row_keys[i] = s < 0 ? kEmptyKey : key;
}

// Input mode 0 with repeated coordinates: the site belongs to the last row that named it.
// Earlier rows keep their feature row but are in no map of the reference, so no rule ever
// touches them and getSpatialLocations leaves them zero; here their key is blanked.
// Block 0 tells the host what the inserts found.
__global__ void __launch_bounds__(256)
k_blank_overwritten(const Slot *__restrict__ slots, const int *__restrict__ slot_of, long long n,
                    unsigned long long *__restrict__ row_keys, int *flags, const int *n_samples, HostPost post) {
  SCN_GRID_WAIT();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) post_to_host(post, flags, true, 0, n_samples);
  if (i >= n) return;
  const int s = slot_of[i];
  if (s >= 0 && slots[s].row != (int)i) row_keys[i] = kEmptyKey;
}

// ---- row numbers in the order of first touch --------------------------------------------------------
// A candidate (input row; pair of a site and an output it feeds) is the first of its site if the site's slot holds its
// id.  The site's row is the number of such candidates before it: a bit per candidate, 32 of them with the count before
// them in their run of kRankTile candidates (`words`), and the count before the run (`base`), which the block that
// finishes last sums up.  Whoever needs a row reads the 8-byte word and the base, both in L2: no array of ranks, no flags,
// and one pass where there were a flag pass, a scan of two or three kernels and a pass over all slots of the table.
constexpr int kRankTile = 1024;

__device__ __forceinline__ int row_of_first(const uint2 *__restrict__ words, const int *__restrict__ base, unsigned id) {
  const uint2 w = words[id >> 5];
  return base[id / kRankTile] + (int)w.y + __popc(w.x & ((1u << (id & 31)) - 1u));
}

// The number of input sites comes from the host (`n_in`, n_in_dev null) or, inside a chain of levels whose counts the host
// has not seen yet, from the device, with `n_in` the bound that sized the launch and the arrays.  A level that did not
// fit its arrays hands nothing on: it will be built again, and so will what is below it.
__device__ __forceinline__ long long sites_here(const int *n_dev, long long bound) {
  if (!n_dev) return bound;
  const long long n = *n_dev;
  return n <= bound ? n : 0;
}

__global__ void __launch_bounds__(256)
k_first_ranks(const Slot *__restrict__ slots, const int *__restrict__ slot_of, long long n_in, const int *__restrict__ n_in_dev,
              int per_site, uint2 *__restrict__ words, int *base, int *done, int *total_dev, int *flags, bool clear_flags,
              const int *extra, HostPost post) {
  SCN_GRID_WAIT();
  __shared__ unsigned sh_bits[32];
  __shared__ int sh_sum[8];
  __shared__ bool last;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const long long n = sites_here(n_in_dev, n_in) * per_site, at = (long long)blockIdx.x * kRankTile;
  if (at < n) {
    int s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long id = at + j * 256 + t;
      s[j] = id < n ? slot_of[id] : -1;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const unsigned id = (unsigned)(at + j * 256 + t);
      const unsigned bits = __ballot_sync(0xffffffffu, s[j] >= 0 && slots[s[j] < 0 ? 0 : s[j]].aux == id);
      if (lane == 0) sh_bits[j * 8 + warp] = bits;
    }
  } else if (t < 32) {
    sh_bits[t] = 0;
  }
  __syncthreads();
  if (warp == 0) {
    const unsigned bits = sh_bits[lane];
    int incl = __popc(bits);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (at < n) words[(at >> 5) + lane] = make_uint2(bits, (unsigned)(incl - __popc(bits)));
    if (lane == 31) {
      base[blockIdx.x] = incl;
      __threadfence();
      last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  int run = 0;
  for (long long b0 = 0; b0 < gridDim.x; b0 += 1024) {  // four per thread and round
    int v[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long b = b0 + t * 4 + j;
      v[j] = b < gridDim.x ? __ldcg(base + b) : 0;
      sum += v[j];
    }
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    if (lane == 31) sh_sum[warp] = incl;
    __syncthreads();
    int before = run, all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      if (w < warp) before += sh_sum[w];
      all += sh_sum[w];
    }
    int excl = before + incl - sum;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long b = b0 + t * 4 + j;
      if (b < gridDim.x) base[b] = excl;
      excl += v[j];
    }
    run += all;
    __syncthreads();
  }
  if (t == 0) {
    if (total_dev) *total_dev = run;
    post_to_host(post, flags, clear_flags, run, extra);
  }
}

// The row that touched a site first gives the site its row number: its rank among such rows in input
// order, which is the numbering of the reference (one counter over the whole input,
// IOLayersRules.h:69-72,84-87; one per output grid, ConvolutionRules.h:24-30).  One thread per table
// SLOT, not per candidate: the table is read and written front to back, and what is reached at random
// (the rank of the slot's first toucher, the row -> key array) is a few MB that stay in L2.  The
// candidate-order form of this pass (a random read-modify-write of a slot per numbered site) was bound by
// the DRAM's random-access rate: 198 us against 142 us for the inserts themselves at 1.6 M sites.
__global__ void k_number_slots(Slot *slots, long long n_slots, const uint2 *__restrict__ words,
                               const int *__restrict__ base, unsigned long long *__restrict__ row_keys) {
  SCN_GRID_WAIT();
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_slots) return;
  const uint4 v = *reinterpret_cast<const uint4 *>(slots + idx);
  const unsigned long long key = ((unsigned long long)v.y << 32) | v.x;
  if (key == kEmptyKey || v.w == 0xFFFFFFFFu) return;
  const int r = row_of_first(words, base, v.w);
  slots[idx].row = r;
  row_keys[r] = key;
}

__global__ void k_count_per_site(const Slot *__restrict__ slots, const int *__restrict__ slot_of,
                                 long long n, int *cnt) {
  SCN_GRID_WAIT();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s = slot_of[i];
  if (s >= 0) atomicAdd(&cnt[slots[s].row], 1);
}

__global__ void k_fill_per_site(const Slot *__restrict__ slots, const int *__restrict__ slot_of,
                                long long n, const int *__restrict__ start, int *cursor,
                                int *__restrict__ csr_rows) {
  SCN_GRID_WAIT();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s = slot_of[i];
  if (s < 0) return;
  int r = slots[s].row;
  int p = atomicAdd(&cursor[r], 1);
  csr_rows[start[r] + p] = (int)i;
}

// Puts the input rows of every site in ascending order (heap sort, in place, one thread per
// site; sites with duplicates hold a handful of rows).
__global__ void k_sort_segments(const int *__restrict__ start, long long n_sites, int *csr_rows) {
  SCN_GRID_WAIT();
  long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_sites) return;
  int *a = csr_rows + start[r];
  int m = start[r + 1] - start[r];
  if (m < 2) return;
  if (m <= 16) {
    for (int i = 1; i < m; ++i) {
      int v = a[i], j = i - 1;
      while (j >= 0 && a[j] > v) {
        a[j + 1] = a[j];
        --j;
      }
      a[j + 1] = v;
    }
    return;
  }
  for (int root0 = m / 2 - 1; root0 >= 0; --root0) {
    int root = root0;
    for (;;) {
      int child = 2 * root + 1;
      if (child >= m) break;
      if (child + 1 < m && a[child] < a[child + 1]) ++child;
      if (a[root] >= a[child]) break;
      int t = a[root]; a[root] = a[child]; a[child] = t;
      root = child;
    }
  }
  for (int end = m - 1; end > 0; --end) {
    int t = a[0]; a[0] = a[end]; a[end] = t;
    int root = 0;
    for (;;) {
      int child = 2 * root + 1;
      if (child >= end) break;
      if (child + 1 < end && a[child] < a[child + 1]) ++child;
      if (a[root] >= a[child]) break;
      int u = a[root]; a[root] = a[child]; a[child] = u;
      root = child;
    }
  }
}

static void clear_input_rules(scn_metadata *md, cudaStream_t stream) {
  device_free(md->input_csr_start, stream);
  device_free(md->input_csr_rows, stream);
  md->input_csr_start = md->input_csr_rows = nullptr;
  md->input_mode = -1;
  md->input_n_rows = md->input_n_active = 0;
}

static int md_clear(scn_metadata *md, cudaStream_t stream) {
  chain_abandon(md, stream);
  for (auto &g : md->grids) free_grid(g.second, stream);
  for (auto &r : md->sub_rules) free_rulebook(r.second, stream);
  for (auto &r : md->strided_rules) free_rulebook(r.second, stream);
  md->grids.clear();
  md->sub_rules.clear();
  md->strided_rules.clear();
  clear_input_rules(md, stream);
  return SCN_OK;
}

constexpr int64_t kPackRows = 4 << 20;  // host coordinates: packed by the host up to here (32 MB of pinned memory)

// Packed keys of host coordinates; given back unless a kernel may still be reading them (after an error nobody knows).
struct PinnedKeys {
  unsigned long long *p = nullptr;
  size_t bytes = 0;
  bool in_use = false;
  ~PinnedKeys() {
    if (p && !in_use) pinned_release(p, bytes);
  }
};

// Will some key have bits from 48 on?  The batch index lies above the coordinates: 16 points are looked at, the last one among them (a batch
// is mostly in order).  Where they say no and another point says yes, the host pass is made twice: 400 k points 430 -> 600 us.
static bool wide_keys(const KeyLayout &L, const long long *coords, int64_t n, int ncols, int64_t bl_length) {
  if (bl_length > 0 || L.batch_shift >= 48) return true;  // (an empty slot's key has all its bits)
  if (ncols <= L.dim) return false;
  for (int64_t i = n - 1, step = std::max<int64_t>(1, n / 16); i >= 0; i -= step)
    if ((unsigned long long)coords[i * ncols + L.dim] >> (48 - L.batch_shift)) return true;
  return false;
}

// The site table `g` and the input rules of `coords`; what it leaves behind when it fails is the caller's to free.
static int build_input(scn_metadata *md, const int64_t *coords, int coords_on_device, int64_t n, int ncols,
                       int64_t batch_size, int mode, int64_t bl_length, cudaStream_t stream, Grid &g) {
  SCN_TRY(alloc_table(g.table, n, stream));
  SCN_TRY(device_alloc((void **)&g.row_keys, sizeof(unsigned long long) * (size_t)std::max<int64_t>(n, 1), stream));
  const unsigned tiles = (unsigned)ceil_div(std::max<int64_t>(n, 1), kRankTile);
  Scratch tmp(stream);
  int *slot_of = nullptr, *base = nullptr, *cursor = nullptr;
  uint2 *words = nullptr;
  SCN_TRY(tmp.get(&slot_of, sizeof(int) * (size_t)std::max<int64_t>(n, 1)));
  if (mode != 0) {
    SCN_TRY(tmp.get(&words, sizeof(uint2) * (kRankTile / 32) * (size_t)tiles));
    SCN_TRY(tmp.get(&base, sizeof(int) * (size_t)tiles));
  }

  const long long *coords_dev = (const long long *)coords;
  PinnedKeys packed;
  unsigned long long *packed_dev = nullptr;
  int packed_samples = 0;
  NarrowKeys narrow{};
  bool narrow_keys = false;
  if (!coords_on_device && n > 0 && n <= kPackRows) {
    SCN_TRY(pinned_acquire(sizeof(unsigned long long) * (size_t)n, (void **)&packed.p, &packed.bytes));
    bool bad = false;
    unsigned long long any = ~0ull;
    if (!wide_keys(g.layout, coords_dev, n, ncols, bl_length)) {
      narrow.low = (unsigned *)packed.p;
      narrow.high[0] = (unsigned char *)(narrow.low + n), narrow.high[1] = narrow.high[0] + n;
      pack_keys(g.layout, coords_dev, n, ncols, narrow, &packed_samples, &bad, &any);
      narrow_keys = (any >> 48) == 0;
      for (int h = 0; h < 2; ++h)
        if ((any >> (32 + 8 * h) & (h ? 0xFFull : 0xFFFFull)) == 0) narrow.high[h] = nullptr;
    }
    if (!narrow_keys) pack_keys(g.layout, coords_dev, n, ncols, bl_length, packed.p, &packed_samples, &bad);
    if (bad) return flags_to_status(FLAG_COORD_RANGE);
    // (copied to the device first, 400 k keys took 240 us longer: the bus is what the insert kernel waits for either way)
    SCN_CUDA_CHECK(cudaHostGetDevicePointer((void **)&packed_dev, packed.p, 0));
    const auto on_device = [&](auto *q) { return q ? (decltype(q))((unsigned char *)packed_dev + ((unsigned char *)q - (unsigned char *)packed.p)) : nullptr; };
    narrow = NarrowKeys{on_device(narrow.low), {on_device(narrow.high[0]), on_device(narrow.high[1])}};
  } else if (!coords_on_device && n > 0) {
    const size_t bytes = sizeof(long long) * (size_t)n * ncols;
    long long *staged = nullptr;
    SCN_TRY(tmp.get(&staged, bytes));
    SCN_CUDA_CHECK(cudaMemcpyAsync(staged, coords, bytes, cudaMemcpyHostToDevice, stream));
    coords_dev = staged;
  }

  const int threads = 256;
  unsigned blocks = (unsigned)ceil_div(std::max<int64_t>(n, 1), threads);
  int *n_samples = md->scalars_dev, *done = md->scalars_dev + 1;  // batch indices in use; finished blocks
  Fills fills{};
  fill_add(fills, g.table.slots, 2 * g.table.n_buckets * sizeof(Slot), true);
  fill_add(fills, n_samples, 2 * sizeof(int), false);
  SCN_TRY(fill_launch(fills, stream));
  HostPost post{};
  SCN_TRY(post_begin(md, post));
  if (n > 0) {
    packed.in_use = true;
    if (narrow_keys)
      SCN_LAUNCH(k_insert_narrow, blocks, threads, 0, stream, g.table, narrow.low, narrow.high[0], narrow.high[1], (long long)n, mode, g.row_keys, slot_of, md->flags_dev);
    else
      SCN_LAUNCH_DIM(md->dim, k_insert_input, blocks, threads, 0, stream, g.layout, g.table, coords_dev, packed_dev, n, ncols, mode, (long long)bl_length, g.row_keys, slot_of, md->flags_dev, n_samples);
    if (mode == 0)
      SCN_LAUNCH(k_blank_overwritten, blocks, threads, 0, stream, g.table.slots, slot_of, n, g.row_keys, md->flags_dev, n_samples, post);
    SCN_CUDA_CHECK(cudaGetLastError());
  }
  if (mode != 0 && n > 0) {
    SCN_LAUNCH(k_first_ranks, tiles, 256, 0, stream, g.table.slots, slot_of, (long long)n, nullptr, 1, words, base, done, nullptr, md->flags_dev, true, n_samples, post);
    const long long n_slots = 2 * (long long)g.table.n_buckets;
    SCN_LAUNCH(k_number_slots, (unsigned)ceil_div(n_slots, threads), threads, 0, stream, g.table.slots, n_slots, words, base, g.row_keys);
    SCN_CUDA_CHECK(cudaGetLastError());
  }

  int flags = 0, total = 0, samples = 0;
  if (n > 0) {
    SCN_TRY(wait_posted(md->mailbox, stream));
    packed.in_use = false;
    const volatile int *host = md->mailbox;
    flags = host[1];
    total = host[2];
    samples = packed.p ? packed_samples : host[3];
  }
  SCN_TRY(flags_to_status(flags));
  long long active = (mode == 0) ? n : total;
  // Every point has a site of its own (no repeated coordinates, no empty slots): rows are numbered in
  // order of first occurrence, so row i is point i and the rule table is the identity -- the feature
  // pass is then the plain copy of mode 0 and no table is built.  Otherwise: CSR of the input rows of
  // every site, each site's rows ascending (the order the reference sums them in).
  const bool identity = mode != 0 && active == n;
  if (mode != 0 && n > 0 && active > 0 && !identity) {
    SCN_TRY(device_alloc((void **)&md->input_csr_start, sizeof(int) * (size_t)(n + 1), stream));
    SCN_TRY(device_alloc((void **)&md->input_csr_rows, sizeof(int) * (size_t)n, stream));
    SCN_TRY(tmp.get(&cursor, sizeof(int) * (size_t)(n + 1)));
    SCN_CUDA_CHECK(cudaMemsetAsync(cursor, 0, sizeof(int) * (size_t)(n + 1), stream));
    SCN_LAUNCH(k_count_per_site, blocks, threads, 0, stream, g.table.slots, slot_of, n, cursor);
    SCN_TRY(exclusive_scan_i32(cursor, md->input_csr_start, n + 1, nullptr, stream));
    SCN_CUDA_CHECK(cudaMemsetAsync(cursor, 0, sizeof(int) * (size_t)(n + 1), stream));
    SCN_LAUNCH(k_fill_per_site, blocks, threads, 0, stream, g.table.slots, slot_of, n, md->input_csr_start, cursor, md->input_csr_rows);
    unsigned sblocks = (unsigned)ceil_div(active, threads);
    SCN_LAUNCH(k_sort_segments, sblocks, threads, 0, stream, md->input_csr_start, active, md->input_csr_rows);
    SCN_CUDA_CHECK(cudaGetLastError());
  }
  g.n_active = active;
  g.may_have_blank_rows = (mode == 0);
  // batch size: IOLayersRules.h:25,35,52-53 -- one sample when there is no batch column,
  // otherwise max(requested, largest index + 1)
  if (bl_length > 0)
    g.batch_size = batch_size;
  else if (ncols == md->dim)
    g.batch_size = 1;
  else
    g.batch_size = std::max<long long>(batch_size, samples);
  md->input_mode = identity ? 0 : mode;  // what the feature passes do (a copy when the table is the identity)
  return SCN_OK;
}

static int md_input_layer(scn_metadata *md, const int64_t *spatial_size, const int64_t *coords,
                          int coords_on_device, int64_t n, int ncols, int64_t batch_size, int mode,
                          int64_t bl_length, cudaStream_t stream, int64_t *n_active) {
  SCN_REQUIRE(md && spatial_size && n_active, SCN_ERR_BAD_ARG, "null argument");
  SCN_REQUIRE(mode >= 0 && mode <= 4, SCN_ERR_BAD_ARG, "input layer mode %d not in 0..4", mode);
  SCN_REQUIRE(ncols == md->dim || ncols == md->dim + 1, SCN_ERR_BAD_ARG,
              "coords must have %d or %d columns, got %d", md->dim, md->dim + 1, ncols);
  SCN_REQUIRE(n >= 0 && n < (1ll << 30), SCN_ERR_UNSUPPORTED, "row count %lld unsupported", (long long)n);
  SCN_REQUIRE(n == 0 || coords, SCN_ERR_BAD_ARG, "null coords");
  SCN_TRY(md_touch(md, stream));
  SCN_TRY(ensure_scratch(md, stream));

  // A new input replaces everything the object knew: grids of other scales and rulebooks built from
  // the old input would otherwise stay cached with the old row counts.  (The reference asserts that
  // the object is empty, IOLayersRules.h:22-24.)
  SCN_TRY(md_clear(md, stream));

  Grid g;
  SCN_TRY(make_layout(md->dim, spatial_size, g.layout));
  const int st = build_input(md, coords, coords_on_device, n, ncols, batch_size, mode, bl_length, stream, g);
  if (st != SCN_OK) {
    free_grid(g, stream);
    clear_input_rules(md, stream);
    return st;
  }
  md->input_n_rows = n;
  md->input_n_active = g.n_active;
  md->grids[make_key(md->dim, spatial_size)] = g;
  *n_active = g.n_active;
  return SCN_OK;
}

// ------------------------------------------------------------------------------------------
// spatial locations
// ------------------------------------------------------------------------------------------

// Row r -> (x_0..x_{D-1}, batch).  A row with a blank key (an earlier duplicate under input
// mode 0) is reported as zeros, as the reference leaves it (Metadata.cpp:154-168 writes only
// rows reachable from the maps).
__global__ void k_spatial_locations(KeyLayout L, const unsigned long long *__restrict__ row_keys,
                                    long long n, long long *__restrict__ out) {
  SCN_GRID_WAIT();
  long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  unsigned long long key = row_keys[r];
  long long *o = out + r * (L.dim + 1);
  bool live = (key != kEmptyKey);
  int x[kMaxDim], b = 0;
  if (live) unpack_key(L, key, x, b);
  for (int d = 0; d < L.dim; ++d) o[d] = live ? x[d] : 0;
  o[L.dim] = live ? b : 0;
}

// ------------------------------------------------------------------------------------------
// submanifold rulebook
// ------------------------------------------------------------------------------------------

struct FilterDesc {
  int f[kMaxDim];  // filter size
  int s[kMaxDim];  // stride (strided rules only)
  int out_size[kMaxDim];
  int tdim[kMaxDim];  // outputs an input can feed per dimension: ceil(f / s)
  int tmax;
};

// Called by every block of a rulebook builder after it has added to the rule counts: the block that finishes last hands
// them to the host (counts_host: pinned, device-mapped; null: nobody wants them).  counts[K] counts finished blocks.
__device__ __forceinline__ void post_counts(unsigned long long *counts, int K, volatile unsigned long long *counts_host) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&counts[K], 1ull) == (unsigned long long)gridDim.x * gridDim.y - 1;
  }
  __syncthreads();
  if (!last || !counts_host) return;
  for (int k = threadIdx.x; k < K; k += blockDim.x) counts_host[k] = atomicAdd(&counts[k], 0ull);
  __threadfence_system();
}

// One thread per output site, looping over this block's range of at most 32 filter offsets.  Offset k
// (row-major over the filter, last dimension fastest, RectangularRegions.h:30-38) looks at
// input = output + delta_k with delta = k_d - f_d / 2 (SubmanifoldConvolutionRules.h:15-19).
// The neighbour's key is the site's key plus a per-offset constant, so a probe is a bounds
// check, one 64-bit add and one 32-byte bucket read; the buckets of kAhead offsets are read before the first is looked at.
// Bound by instruction issue and the latency of the bucket reads, which threads hide better than reads ahead do, whose
// registers cost threads (400 k sites, 27 offsets: 76, 81, 91, 104 us with 1, 2, 3, 5 ahead, 101 with coordinates in local
// memory; 1.5 M sites, 81 offsets: 758, 714, 796 us with 1, 2, 3).
template <int DIM>
__global__ void __launch_bounds__(256)
k_submanifold_rules(KeyLayout L, HashTable T, const unsigned long long *__restrict__ row_keys,
                    long long n, int K, FilterDesc F, int k_chunk, int *__restrict__ nbr,
                    unsigned long long *counts, int mirrored, unsigned *__restrict__ masks, int mask_words,
                    volatile unsigned long long *counts_host) {
  SCN_GRID_WAIT();
  constexpr int kDim = DIM ? DIM : kMaxDim, kAhead = DIM == 4 ? 2 : 1;
  __shared__ long long sh_keydelta[32];
  __shared__ int sh_count[32];
  __shared__ signed char sh_delta[32][kDim];
  const int dim = DIM ? DIM : L.dim, lane = threadIdx.x & 31;
  // mirrored (all filter sizes odd): offset K-1-k is offset k seen from the neighbour, so only the
  // offsets up to the centre are looked up; a hit also fills the neighbour's entry at the mirrored
  // offset (pre-set to -1 by the caller), and the centre is the site itself.
  const int k_end = mirrored ? K / 2 + 1 : K;
  const int k0 = blockIdx.y * k_chunk, k1 = min(k_end, k0 + k_chunk);
  if (k0 + (int)threadIdx.x < k1) {
    int rem = k0 + threadIdx.x;
    long long kd = 0;
    for (int d = dim - 1; d >= 0; --d) {
      const int delta = rem % F.f[d] - F.f[d] / 2;
      rem /= F.f[d];
      sh_delta[threadIdx.x][d] = (signed char)delta;
      kd += (long long)delta * (1ll << L.shift[d]);
    }
    sh_keydelta[threadIdx.x] = kd;
    sh_count[threadIdx.x] = 0;
  }
  __syncthreads();
  const unsigned long long bucket_mask = T.n_buckets - 1;
  int my_count = 0;  // of offset k0 + lane, by this warp
  // at most a few blocks per SM, each over several runs of sites: the counts below are atomics on K addresses per block
  for (long long site0 = (long long)blockIdx.x * blockDim.x; site0 < n; site0 += (long long)gridDim.x * blockDim.x) {
    const long long site = site0 + threadIdx.x;
    unsigned long long key = site < n ? row_keys[site] : kEmptyKey;
    const bool active = key != kEmptyKey;  // blank key: overwritten duplicate, in no map
    int x[kDim], b = 0;
    unpack_site<DIM>(L, key, x, b);
    // masks (optional, zeroed by the caller): the offsets of every site as bits, both ends of a hit OR theirs in.  Six
    // million of these at 1.6 M sites disappear beside the lookups; reading the finished table back took 109 us.
    unsigned bits = 0;
    int word = k0 >> 5;
    int *out = nbr + (long long)k0 * n + site, *back = nbr + (long long)(K - 1 - k0) * n;  // offset kk, and its mirror
    for (int kb = k0; kb < k1; kb += kAhead) {
      unsigned long long want[kAhead];
      uint4 s0[kAhead], s1[kAhead];
      bool look[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int i = kb + u - k0;
        look[u] = active && kb + u < k1 && !(mirrored && kb + u == K / 2);
        if (kb + u < k1) {
#pragma unroll
          for (int d = 0; d < dim; ++d) look[u] &= (unsigned)(x[d] + sh_delta[i][d]) < (unsigned)L.size[d];
          want[u] = key + (unsigned long long)sh_keydelta[i];
        }
        if (look[u]) {
          const uint4 *q = reinterpret_cast<const uint4 *>(T.slots + 2 * (mix64(want[u]) & bucket_mask));
          s0[u] = __ldg(q);
          s1[u] = __ldg(q + 1);
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int kk = kb + u;
        if (kk >= k1) break;
        int row = -1;
        if (look[u]) {
          const unsigned long long e0 = ((unsigned long long)s0[u].y << 32) | s0[u].x;
          const unsigned long long e1 = ((unsigned long long)s1[u].y << 32) | s1[u].x;
          if (e0 == want[u]) row = (int)s0[u].z;
          else if (e1 == want[u]) row = (int)s1[u].z;
          else if (e0 != kEmptyKey && e1 != kEmptyKey) row = hash_find_row(T, want[u]);  // a full bucket: walk on
        }
        if (mirrored && kk == K / 2 && active) row = (int)site;
        if (masks && (kk >> 5) != word) {
          if (bits) atomicOr(&masks[site * mask_words + word], bits);
          bits = 0;
          word = kk >> 5;
        }
        if (site < n) *out = row;
        if (masks && row >= 0) bits |= 1u << (kk & 31);
        if (mirrored && kk < K / 2 && row >= 0) {
          back[row] = (int)site;
          const int kr = K - 1 - kk;
          if (masks) atomicOr(&masks[(long long)row * mask_words + (kr >> 5)], 1u << (kr & 31));
        }
        out += n;
        back -= n;
        const unsigned hits = __ballot_sync(0xffffffffu, row >= 0);
        if (lane == kk - k0) my_count += __popc(hits);
      }
    }
    if (masks && bits) atomicOr(&masks[site * mask_words + word], bits);
  }
  if (my_count) atomicAdd(&sh_count[lane], my_count);
  __syncthreads();
  if (k0 + (int)threadIdx.x < k1 && sh_count[threadIdx.x]) {
    const int kk = k0 + threadIdx.x;
    atomicAdd(&counts[kk], (unsigned long long)sh_count[threadIdx.x]);
    if (mirrored && kk < K / 2) atomicAdd(&counts[K - 1 - kk], (unsigned long long)sh_count[threadIdx.x]);
  }
  post_counts(counts, K, counts_host);
}

// What a submanifold rulebook starts from, in one launch: counts and masks zero, the mirrored half of the table empty.
__global__ void __launch_bounds__(256)
k_rules_init(unsigned long long *counts, int n_counts, unsigned *masks, long long n_masks, int *nbr, long long n_nbr) {
  SCN_GRID_WAIT();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  for (long long j = i; j < n_counts; j += step) counts[j] = 0;
  for (long long j = i; j < n_masks; j += step) masks[j] = 0;
  if ((uintptr_t)nbr % 16 == 0) {
    for (long long j = i; j < n_nbr / 4; j += step) reinterpret_cast<int4 *>(nbr)[j] = make_int4(-1, -1, -1, -1);
    for (long long j = n_nbr / 4 * 4 + i; j < n_nbr; j += step) nbr[j] = -1;
  } else {
    for (long long j = i; j < n_nbr; j += step) nbr[j] = -1;
  }
}

// (what it leaves in `rb` when it fails is the caller's to free)
static int build_submanifold(scn_metadata *md, Grid *g, const int64_t *filter_size, cudaStream_t stream, Rulebook &rb) {
  long long K = 1;
  FilterDesc F{};
  for (int d = 0; d < md->dim; ++d) {
    SCN_REQUIRE(filter_size[d] >= 1 && filter_size[d] <= 127, SCN_ERR_UNSUPPORTED,
                "filter size %lld unsupported", (long long)filter_size[d]);
    F.f[d] = (int)filter_size[d];
    K *= filter_size[d];
  }
  SCN_REQUIRE(K <= 4096, SCN_ERR_UNSUPPORTED, "filter volume %lld unsupported", K);
  long long n = g->n_active;
  SCN_REQUIRE(K * std::max<long long>(n, 1) < (1ll << 40), SCN_ERR_UNSUPPORTED, "rulebook too large");
  rb.n_offsets = (int)K;
  rb.dim = md->dim;
  rb.symmetric = true;
  for (int d = 0; d < md->dim; ++d) {
    rb.filter[d] = filter_size[d];
    rb.symmetric &= filter_size[d] % 2 == 1;
  }
  rb.n_in = rb.n_out = n;
  SCN_TRY(device_alloc((void **)&rb.nbr, sizeof(int) * (size_t)(K * std::max<long long>(n, 1)), stream));
  SCN_TRY(device_alloc((void **)&rb.counts_dev, sizeof(unsigned long long) * (size_t)(K + 1), stream));
  SCN_TRY(count_ticket_new(rb));
  if (n == 0) {
    SCN_CUDA_CHECK(cudaMemsetAsync(rb.counts_dev, 0, sizeof(unsigned long long) * (size_t)(K + 1), stream));
    count_ticket_zero(rb);
  } else {
    const int threads = 256;
    long long bx = ceil_div(n, threads);
    bool mirrored = K > 1 && !(getenv("SCN_RULES_MIRROR") && atoi(getenv("SCN_RULES_MIRROR")) == 0);
    for (int d = 0; d < md->dim; ++d) mirrored &= (filter_size[d] % 2 == 1);
    const long long k_end = mirrored ? K / 2 + 1 : K;  // offsets that are looked up
    const int words = mask_words((int)K);
    if (K <= kOrderMaxOffsets) SCN_TRY(device_alloc((void **)&rb.masks, sizeof(unsigned) * words * (size_t)n, stream));
    const long long n_back = mirrored ? (K - k_end) * n : 0;
    SCN_LAUNCH(k_rules_init, (unsigned)std::min<long long>(148 * 8, ceil_div(std::max(n_back / 4, n * words), 256)), 256, 0, stream, rb.counts_dev, (int)K + 1, rb.masks, rb.masks ? n * words : 0, rb.nbr + k_end * n, n_back);
    // enough blocks to fill the machine even for few sites: split the offsets over grid.y
    long long want_y = std::max<long long>(1, std::min<long long>(k_end, ceil_div(148 * 16, bx)));
    const int k_chunk = (int)ceil_div(k_end, std::max(want_y, ceil_div(k_end, 32)));  // at most 32: a lane counts an offset
    int gy = (int)ceil_div(k_end, k_chunk);
    SCN_LAUNCH_DIM(md->dim, k_submanifold_rules, dim3((unsigned)std::min<long long>(bx, 148 * 16), (unsigned)gy), threads, 0, stream, g->layout, g->table, g->row_keys, n, (int)K, F, k_chunk, rb.nbr, rb.counts_dev, mirrored ? 1 : 0, rb.masks, words, ticket_dev(rb));
    SCN_CUDA_CHECK(cudaGetLastError());
  }
  rb.built = true;
  g_rulebook_builds.fetch_add(1);
  return SCN_OK;
}

int get_submanifold_rulebook(scn_metadata *md, const int64_t *spatial_size,
                             const int64_t *filter_size, cudaStream_t stream, Rulebook **out) {
  SCN_TRY(md_touch(md, stream));
  auto key = make_key(md->dim, spatial_size, filter_size);
  auto have = md->sub_rules.find(key);
  if (have != md->sub_rules.end()) {
    *out = &have->second;
    return SCN_OK;
  }
  if (md->pending && !find_grid_now(md, spatial_size)) SCN_TRY(chain_finalize(md, stream, nullptr));
  Grid *g = find_grid_now(md, spatial_size);
  SCN_REQUIRE(g, SCN_ERR_NO_GRID, "submanifold rulebook: no grid for that spatial size");
  Rulebook rb;
  const int st = build_submanifold(md, g, filter_size, stream, rb);
  if (st != SCN_OK) {
    free_rulebook(rb, stream);
    return st;
  }
  *out = &(md->sub_rules[key] = rb);
  return SCN_OK;
}

// ------------------------------------------------------------------------------------------
// strided rulebook (Convolution / MaxPooling; Deconvolution reads it transposed)
// ------------------------------------------------------------------------------------------

// For input site x and candidate t in [0, tmax): the t-th output (row-major over the output
// region, last dimension fastest) that x feeds, and the filter offset it feeds it through.
// Output region per dimension: lb = max(0, (x - f + s) / s), ub = min(out - 1, x / s)
// (RectangularRegions.h:108-119); offset = sum (x_d - o_d * s_d) * prod_{j>d} f_j
// (RectangularRegions.h:30-38,94-105).
template <int DIM>
__device__ __forceinline__ bool strided_target(const KeyLayout &L, const FilterDesc &F, const int (&x)[DIM ? DIM : kMaxDim],
                                               int t, int (&o)[DIM ? DIM : kMaxDim], int &k) {
  const int dim = DIM ? DIM : L.dim;
  k = 0;
  int mult = 1;
#pragma unroll
  for (int d = dim - 1; d >= 0; --d) {
    int lb, ub, j = 0;
    if (F.tmax == 1) {  // windows side by side
      lb = ub = (int)((unsigned)x[d] / (unsigned)F.s[d]);
    } else {
      const int num = x[d] - F.f[d] + F.s[d];
      lb = num > 0 ? (int)((unsigned)num / (unsigned)F.s[d]) : 0;
      ub = (int)((unsigned)x[d] / (unsigned)F.s[d]);
      j = (int)((unsigned)t % (unsigned)F.tdim[d]);
      t = (int)((unsigned)t / (unsigned)F.tdim[d]);
    }
    const int od = lb + j;
    if (od > min(F.out_size[d] - 1, ub)) return false;
    o[d] = od;
    const int kd = x[d] - od * F.s[d];
    if (kd >= F.f[d]) return false;  // (a window narrower than the stride)
    k += kd * mult;
    mult *= F.f[d];
  }
  return true;
}

template <int DIM>
__global__ void __launch_bounds__(256)
k_strided_insert(KeyLayout Lin, KeyLayout Lout, FilterDesc F, HashTable Tout, const unsigned long long *__restrict__ in_keys,
                 long long n_in, const int *__restrict__ n_in_dev, int *__restrict__ slot_of, int *flags) {
  SCN_GRID_WAIT();
  const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;  // (fewer than 2^31 candidates)
  if (id >= sites_here(n_in_dev, n_in) * F.tmax) return;
  const unsigned i = F.tmax == 1 ? id : id / (unsigned)F.tmax;
  const int t = (int)(id - i * (unsigned)F.tmax);
  const unsigned long long key = in_keys[i];
  unsigned long long okey = kEmptyKey;
  if (key != kEmptyKey) {
    int x[DIM ? DIM : kMaxDim], o[DIM ? DIM : kMaxDim], b, k;
    unpack_site<DIM>(Lin, key, x, b);
    if (strided_target<DIM>(Lin, F, x, t, o, k)) okey = pack_site<DIM>(Lout, o, b);
  }
  // Candidates of one warp that name the same output site (neighbouring input rows usually do) insert
  // it once: the lowest lane of the group, which also holds the group's smallest id, does the insert
  // and hands the slot to the others.
  const unsigned peers = __match_any_sync(__activemask(), okey);
  const int leader = __ffs(peers) - 1;
  int s_out = -1;
  if (okey != kEmptyKey && (int)(threadIdx.x & 31) == leader) {
    const long long s = hash_claim<false, true>(Tout, okey, id);
    if (s < 0)
      atomicOr(flags, FLAG_TABLE_FULL);
    else
      s_out = (int)s;
  }
  slot_of[id] = __shfl_sync(peers, s_out, leader);
}

// A few blocks per SM, each over several runs of candidates, with the rule counts of up to kFillCounts offsets summed in
// shared memory first: counted in global memory per warp, a 3 / 2 layer's eight rules per candidate were 370 us of
// atomics on 27 addresses for 184 k sites.
constexpr int kFillCounts = 1024;
template <int DIM>
__global__ void __launch_bounds__(256)
k_strided_fill(KeyLayout Lin, KeyLayout Lout, FilterDesc F, Slot *slots, const unsigned long long *__restrict__ in_keys,
               const int *__restrict__ slot_of, long long n_in, const int *__restrict__ n_in_dev, long long n_out,
               const int *__restrict__ n_out_dev, long long capacity, const uint2 *__restrict__ words,
               const int *__restrict__ base, unsigned long long *__restrict__ row_keys, int *__restrict__ nbr,
               unsigned long long *counts, int K, volatile unsigned long long *counts_host) {
  SCN_GRID_WAIT();
  __shared__ int sh_count[kFillCounts];
  const bool shared = K <= kFillCounts;
  if (shared)
    for (int k = threadIdx.x; k < K; k += blockDim.x) sh_count[k] = 0;
  __syncthreads();
  if (n_out_dev) n_out = *n_out_dev;  // inside a chain: the level's row count is on the device only
  const long long n_ids = sites_here(n_in_dev, n_in) * F.tmax;
  if (n_out <= capacity)  // otherwise the level overflowed its arrays and will be rebuilt
    for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < n_ids; id += (long long)gridDim.x * blockDim.x) {
      const int s = slot_of[id];
      if (s < 0) continue;
      const unsigned i = F.tmax == 1 ? (unsigned)id : (unsigned)id / (unsigned)F.tmax;
      const int t = (int)((unsigned)id - i * (unsigned)F.tmax);
      int x[DIM ? DIM : kMaxDim], o[DIM ? DIM : kMaxDim], b, k;
      unpack_site<DIM>(Lin, in_keys[i], x, b);
      strided_target<DIM>(Lin, F, x, t, o, k);
      // one look at the slot per group of lanes that share it; the site's first candidate, always the lowest lane of its
      // group, leaves the row in the slot and the site's key in its row
      const unsigned act = __activemask();
      const unsigned same = __match_any_sync(act, s);
      const int first = __ffs(same) - 1;
      int orow = 0;
      if ((int)(threadIdx.x & 31) == first) {
        const unsigned toucher = slots[s].aux;
        orow = row_of_first(words, base, toucher);
        if (toucher == (unsigned)id) {
          slots[s].row = orow;
          row_keys[orow] = pack_site<DIM>(Lout, o, b);
        }
      }
      orow = __shfl_sync(same, orow, first);
      nbr[(long long)k * n_out + orow] = (int)i;
      // one counter update per distinct offset in the warp
      const unsigned peers = __match_any_sync(act, k);
      if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) {
        if (shared) atomicAdd(&sh_count[k], __popc(peers));
        else atomicAdd(&counts[k], (unsigned long long)__popc(peers));
      }
    }
  __syncthreads();
  if (shared)
    for (int k = threadIdx.x; k < K; k += blockDim.x)
      if (sh_count[k]) atomicAdd(&counts[k], (unsigned long long)sh_count[k]);
  post_counts(counts, K, counts_host);
}

// (what it leaves in `gout` and `rb` when it fails is the caller's to free)
// Does every site of a fine grid have exactly one rule in the rulebook of F?  Filter = stride: the children of different
// coarse sites and offsets never coincide, and none is left out where the coarse grid covers the fine one.  (Rows in no map,
// earlier duplicates under input mode 0, have none.)
static bool one_rule_per_row(const KeyLayout &fine, bool may_have_blank_rows, const FilterDesc &F) {
  for (int d = 0; d < fine.dim; ++d)
    if (F.f[d] != F.s[d] || (long long)F.out_size[d] * F.s[d] < fine.size[d]) return false;
  return !may_have_blank_rows;
}

static int build_strided(scn_metadata *md, Grid *gin, const int64_t *output_size, const int64_t *filter_size,
                         const int64_t *filter_stride, cudaStream_t stream, Grid &gout, Rulebook &rb) {
  SCN_TRY(ensure_scratch(md, stream));
  FilterDesc F{};
  long long K = 1;
  F.tmax = 1;
  for (int d = 0; d < md->dim; ++d) {
    SCN_REQUIRE(filter_size[d] >= 1 && filter_size[d] <= 127 && filter_stride[d] >= 1 &&
                    filter_stride[d] <= 127 && output_size[d] >= 1 && output_size[d] <= INT_MAX,
                SCN_ERR_UNSUPPORTED, "filter/stride/output size unsupported");
    F.f[d] = (int)filter_size[d];
    F.s[d] = (int)filter_stride[d];
    F.out_size[d] = (int)output_size[d];
    F.tdim[d] = (int)ceil_div(filter_size[d], filter_stride[d]);
    F.tmax *= F.tdim[d];
    K *= filter_size[d];
  }
  SCN_REQUIRE(K <= 4096 && F.tmax <= 4096, SCN_ERR_UNSUPPORTED, "filter volume unsupported");
  long long n_in = gin->n_active;
  long long n_ids = n_in * F.tmax;
  SCN_REQUIRE(n_ids < (1ll << 31), SCN_ERR_UNSUPPORTED, "too many (site, output) candidates");

  SCN_TRY(make_layout(md->dim, output_size, gout.layout));
  SCN_REQUIRE(gout.layout.batch_bits >= gin->layout.batch_bits ||
                  gin->batch_size <= (1ll << gout.layout.batch_bits),
              SCN_ERR_KEY_BITS, "batch index does not fit the output key");
  gout.batch_size = gin->batch_size;

  const int threads = 256;
  Scratch tmp(stream);
  int *slot_of = nullptr, *base = nullptr;
  uint2 *words = nullptr;
  long long n_out = 0;
  if (n_ids > 0) {
    SCN_TRY(tmp.get(&slot_of, sizeof(int) * (size_t)n_ids));
    const unsigned tiles = (unsigned)ceil_div(n_ids, kRankTile);
    SCN_TRY(tmp.get(&words, sizeof(uint2) * (kRankTile / 32) * (size_t)tiles));
    SCN_TRY(tmp.get(&base, sizeof(int) * (size_t)tiles));
    unsigned blocks = (unsigned)ceil_div(n_ids, threads);
    long long expect = n_in;
    for (int attempt = 0;; ++attempt) {
      SCN_TRY(alloc_table(gout.table, expect, stream));
      int *done = md->scalars_dev;
      Fills fills{};
      fill_add(fills, gout.table.slots, 2 * gout.table.n_buckets * sizeof(Slot), true);
      fill_add(fills, done, sizeof(int), false);
      SCN_TRY(fill_launch(fills, stream));
      HostPost post{};
      SCN_TRY(post_begin(md, post));
      post.extra = nullptr;
      SCN_LAUNCH_DIM(md->dim, k_strided_insert, blocks, threads, 0, stream, gin->layout, gout.layout, F, gout.table, gin->row_keys, n_in, nullptr, slot_of, md->flags_dev);
      SCN_LAUNCH(k_first_ranks, tiles, 256, 0, stream, gout.table.slots, slot_of, n_in, nullptr, F.tmax, words, base, done, nullptr, md->flags_dev, true, nullptr, post);
      SCN_CUDA_CHECK(cudaGetLastError());
      SCN_TRY(wait_posted(md->mailbox, stream));
      const int flags = ((const volatile int *)md->mailbox)[1];
      if ((flags & FLAG_TABLE_FULL) && attempt < 3) {  // more coarse sites than guessed: grow
        device_free(gout.table.slots, stream);
        gout.table = HashTable{};
        expect *= 4;
        continue;
      }
      SCN_TRY(flags_to_status(flags));
      n_out = ((const volatile int *)md->mailbox)[2];
      break;
    }
  } else {
    SCN_TRY(alloc_table(gout.table, 0, stream));
  }
  gout.n_active = n_out;
  SCN_TRY(device_alloc((void **)&gout.row_keys, sizeof(unsigned long long) * (size_t)std::max<long long>(n_out, 1), stream));
  rb.n_offsets = (int)K;
  rb.dim = md->dim;
  for (int d = 0; d < md->dim; ++d) rb.filter[d] = filter_size[d];
  rb.n_in = n_in;
  rb.n_out = n_out;
  rb.disjoint = F.tmax == 1;
  rb.one_parent = one_rule_per_row(gin->layout, gin->may_have_blank_rows, F);
  size_t nbr_bytes = sizeof(int) * (size_t)(K * std::max<long long>(n_out, 1));
  SCN_TRY(device_alloc((void **)&rb.nbr, nbr_bytes, stream));
  SCN_TRY(device_alloc((void **)&rb.counts_dev, sizeof(unsigned long long) * (size_t)(2 * K + 2), stream));
  SCN_TRY(count_ticket_new(rb));
  Fills fills{};
  fill_add(fills, rb.nbr, nbr_bytes, true);
  fill_add(fills, rb.counts_dev, sizeof(unsigned long long) * (size_t)(2 * K + 2), false);
  if (n_ids == 0) {
    fill_add(fills, gout.table.slots, 2 * gout.table.n_buckets * sizeof(Slot), true);
    count_ticket_zero(rb);
  }
  SCN_TRY(fill_launch(fills, stream));
  if (n_ids > 0) {
    unsigned blocks = (unsigned)ceil_div(n_ids, threads);
    SCN_LAUNCH_DIM(md->dim, k_strided_fill, std::min(blocks, 148u * 8u), threads, 0, stream, gin->layout, gout.layout, F, gout.table.slots, gin->row_keys, slot_of, n_in, nullptr, n_out, nullptr, n_out, words, base, gout.row_keys, rb.nbr, rb.counts_dev, (int)K, ticket_dev(rb));
    SCN_CUDA_CHECK(cudaGetLastError());
  }
  rb.built = true;
  g_rulebook_builds.fetch_add(1);
  return SCN_OK;
}

int get_strided_rulebook(scn_metadata *md, const int64_t *input_size, const int64_t *output_size,
                         const int64_t *filter_size, const int64_t *filter_stride,
                         cudaStream_t stream, Rulebook **out) {
  SCN_TRY(md_touch(md, stream));
  auto key = make_key(md->dim, input_size, filter_size, filter_stride);
  auto have = md->strided_rules.find(key);
  if (have == md->strided_rules.end() && md->pending) {  // it may be one of a chain that was started on the side stream
    SCN_TRY(chain_finalize(md, stream, nullptr));
    have = md->strided_rules.find(key);
  }
  if (have != md->strided_rules.end()) {
    *out = &have->second;
    return SCN_OK;
  }
  Grid *gin = find_grid_now(md, input_size);
  SCN_REQUIRE(gin, SCN_ERR_NO_GRID, "strided rulebook: no grid for the input spatial size");
  Grid gout;
  Rulebook rb;
  const int st = build_strided(md, gin, output_size, filter_size, filter_stride, stream, gout, rb);
  if (st != SCN_OK) {
    free_grid(gout, stream);
    free_rulebook(rb, stream);
    return st;
  }
  // (the grid of that size that was there goes only now: with filter and stride 1 it is the one that has been read)
  Grid &place = md->grids[make_key(md->dim, output_size)];
  free_grid(place, stream);
  place = gout;
  *out = &(md->strided_rules[key] = rb);
  return SCN_OK;
}

// ---- a chain of strided levels ---------------------------------------------------------------
// An encoder asks for the same (filter, stride) rulebook at every level (2/2 in a U-Net, 3/2 in a ResNet),
// each level's input being the last level's output.  Built one call at a time, every level ends with the host waiting for its row count
// (the next level's arrays and launches are sized by it), the GPU idling through each round trip.
// Here the whole chain is enqueued at once: level l reads its number of input sites from the device
// (`lev[l]`), its launches and arrays are sized by a bound the host knows, and one mailbox read at the
// end fetches every level's count.  With disjoint windows (filter == stride) a level has at most as
// many sites as its input; the arrays are sized for half of the input bound (surfaces and volumes
// shrink by 2.5x to 8x per level in 3-D); with overlapping windows they are sized for as many sites as
// the input has.  A level that needs more raises its own flag, after which that level and the deeper
// ones are enqueued again with the safe bound (one site per candidate).  Same kernels, same numbering
// (first touch in input-row order) as one call per level.
constexpr int kMaxChain = 16;

struct ChainLevel {
  std::vector<int64_t> in_size, out_size;
  FilterDesc F{};
  long long K = 1;
  Grid gout;
  Rulebook rb;
  long long bound_in = 0, cap_out = 0;
  int *slot_of = nullptr, *base = nullptr;  // scratch of the level's build
  uint2 *words = nullptr;
};

static void chain_free_level(ChainLevel &lv, bool keep_result, cudaStream_t stream) {
  device_free(lv.slot_of, stream);
  device_free(lv.words, stream);
  device_free(lv.base, stream);
  lv.slot_of = lv.base = nullptr;
  lv.words = nullptr;
  if (!keep_result) {
    free_grid(lv.gout, stream);
    free_rulebook(lv.rb, stream);
  }
}

// Memory first, work second.  Everything the chain needs is allocated on `alloc_stream` (stream-ordered
// allocation: the blocks may be ones that earlier work of THAT stream is still using), and only then are the
// memsets and kernels enqueued on `stream`.  With two different streams the caller orders `stream` behind
// `alloc_stream` between the two calls and frees the scratch later, on a stream that is ordered behind `stream`.
static int chain_allocate(std::vector<ChainLevel> &plan, cudaStream_t alloc_stream) {
  for (auto &lv : plan) {
    const size_t n_ids = (size_t)std::max<long long>(lv.bound_in * lv.F.tmax, 1), cap = (size_t)std::max<long long>(lv.cap_out, 1);
    SCN_TRY(device_alloc((void **)&lv.slot_of, sizeof(int) * n_ids, alloc_stream));
    const size_t tiles = (size_t)ceil_div((long long)n_ids, kRankTile);
    SCN_TRY(device_alloc((void **)&lv.words, sizeof(uint2) * (kRankTile / 32) * tiles, alloc_stream));
    SCN_TRY(device_alloc((void **)&lv.base, sizeof(int) * tiles, alloc_stream));
    const unsigned long long slots = next_pow2((unsigned long long)std::max<long long>(64, 2 * lv.cap_out));
    SCN_REQUIRE(slots < (1ull << 31), SCN_ERR_UNSUPPORTED, "site table too large (%llu slots)", slots);
    lv.gout.table.n_buckets = slots / 2;
    SCN_TRY(device_alloc((void **)&lv.gout.table.slots, slots * sizeof(Slot), alloc_stream));
    SCN_TRY(device_alloc((void **)&lv.gout.row_keys, sizeof(unsigned long long) * cap, alloc_stream));
    SCN_TRY(device_alloc((void **)&lv.rb.nbr, sizeof(int) * (size_t)lv.K * cap, alloc_stream));
    SCN_TRY(device_alloc((void **)&lv.rb.counts_dev, sizeof(unsigned long long) * (size_t)(2 * lv.K + 2), alloc_stream));
    lv.rb.n_offsets = (int)lv.K;
    SCN_TRY(count_ticket_new(lv.rb));
    if (lv.bound_in == 0) count_ticket_zero(lv.rb);
  }
  return SCN_OK;
}

// lev: [0, L) row counts of the levels, [L, 2 L) their flags, [2 L, 3 L) finished blocks of their numbering.
// mailbox: [0] ready, [1, L] the counts, [L + 1, 2 L] the flags -- each level's numbering posts its own, the last one
// the ready word (the rule tables are finished a little later: the reader is ordered behind the chain's stream).
static int chain_enqueue(scn_metadata *md, const Grid *gin, std::vector<ChainLevel> &plan, int *lev, int *mailbox,
                         cudaStream_t stream) {
  const int L = (int)plan.size(), threads = 256;
  int *mailbox_dev = nullptr;
  SCN_CUDA_CHECK(cudaHostGetDevicePointer((void **)&mailbox_dev, mailbox, 0));
  for (int i = 1; i <= 2 * L; ++i) ((volatile int *)mailbox)[i] = 0;
  *(volatile int *)mailbox = plan[L - 1].bound_in > 0 ? kNotPosted : 0;
  Fills fills{};
  fill_add(fills, lev, sizeof(int) * 3 * L, false);
  for (auto &lv : plan) {
    if (fills.count + 3 > kMaxFills) {
      SCN_TRY(fill_launch(fills, stream));
      fills = Fills{};
    }
    const size_t cap = (size_t)std::max<long long>(lv.cap_out, 1);
    fill_add(fills, lv.gout.table.slots, 2 * lv.gout.table.n_buckets * sizeof(Slot), true);
    fill_add(fills, lv.rb.nbr, sizeof(int) * (size_t)lv.K * cap, true);
    fill_add(fills, lv.rb.counts_dev, sizeof(unsigned long long) * (size_t)(2 * lv.K + 2), false);
  }
  SCN_TRY(fill_launch(fills, stream));
  const unsigned long long *in_keys = gin->row_keys;
  KeyLayout Lin = gin->layout;
  for (int l = 0; l < L; ++l) {
    ChainLevel &lv = plan[l];
    if (lv.bound_in > 0) {
      const long long n_ids = lv.bound_in * lv.F.tmax;  // (site, output it may feed) candidates
      const unsigned blocks = (unsigned)ceil_div(n_ids, threads);
      const int *n_in_dev = l ? lev + l - 1 : nullptr;
      int *level_flags = lev + L + l;
      HostPost post{};
      post.total = mailbox_dev + 1 + l;
      post.flags = mailbox_dev + 1 + L + l;
      post.ready = l == L - 1 ? mailbox_dev : nullptr;
      SCN_LAUNCH_DIM(md->dim, k_strided_insert, blocks, threads, 0, stream, Lin, lv.gout.layout, lv.F, lv.gout.table, in_keys, lv.bound_in, n_in_dev, lv.slot_of, level_flags);
      SCN_LAUNCH(k_first_ranks, (unsigned)ceil_div(n_ids, kRankTile), 256, 0, stream, lv.gout.table.slots, lv.slot_of, lv.bound_in, n_in_dev, lv.F.tmax, lv.words, lv.base, lev + 2 * L + l, lev + l, level_flags, false, nullptr, post);
      SCN_LAUNCH_DIM(md->dim, k_strided_fill, std::min(blocks, 148u * 8u), threads, 0, stream, Lin, lv.gout.layout, lv.F, lv.gout.table.slots, in_keys, lv.slot_of, lv.bound_in, n_in_dev, 0ll, lev + l, lv.cap_out, lv.words, lv.base, lv.gout.row_keys, lv.rb.nbr, lv.rb.counts_dev, (int)lv.K, ticket_dev(lv.rb));
      SCN_CUDA_CHECK(cudaGetLastError());
    }
    in_keys = lv.gout.row_keys;
    Lin = lv.gout.layout;
  }
  return SCN_OK;
}

// ---- plan / enqueue / collect: the three parts of a chain -----------------------------------------------------
// plan: sizes, layouts and bounds of the levels below `start` that can be chained (stops at the first level that
// is already there, does not divide, or does not fit the key)
static void chain_plan(scn_metadata *md, const Grid *gin, const std::vector<int64_t> &start, const int64_t *filter,
                       const int64_t *stride, int levels, bool safe, std::vector<ChainLevel> &plan) {
  const int dim = md->dim;
  std::vector<int64_t> cur = start;
  long long bound = gin->n_active;
  for (int l = 0; l < levels; ++l) {
    ChainLevel lv;
    lv.in_size = cur;
    lv.out_size.resize(dim);
    bool ok = true;
    lv.F.tmax = 1;
    long long out_volume = gin->batch_size;
    for (int d = 0; d < dim; ++d) {
      const int64_t f = filter[d], st = stride[d];
      if (cur[d] < f || (cur[d] - f) % st != 0) ok = false;
      lv.out_size[d] = ok ? (cur[d] - f) / st + 1 : 1;
      if (lv.out_size[d] > INT_MAX) ok = false;
      lv.F.f[d] = (int)f;
      lv.F.s[d] = (int)st;
      lv.F.out_size[d] = (int)lv.out_size[d];
      lv.F.tdim[d] = (int)ceil_div(f, st);
      lv.F.tmax *= lv.F.tdim[d];
      lv.K *= f;
      out_volume = out_volume > (1ll << 40) ? out_volume : out_volume * lv.out_size[d];
    }
    if (!ok || lv.K > 4096 || lv.F.tmax > 4096 || bound * lv.F.tmax >= (1ll << 31)) break;
    auto found = md->strided_rules.find(make_key(dim, cur.data(), filter, stride));
    if (found != md->strided_rules.end() && found->second.built) break;
    if (md->grids.count(make_key(dim, lv.out_size.data()))) break;
    if (make_layout(dim, lv.out_size.data(), lv.gout.layout) != SCN_OK) break;
    if (!(lv.gout.layout.batch_bits >= gin->layout.batch_bits || gin->batch_size <= (1ll << lv.gout.layout.batch_bits)))
      break;
    lv.rb.disjoint = lv.F.tmax == 1;
    lv.rb.one_parent = plan.empty() ? one_rule_per_row(gin->layout, gin->may_have_blank_rows, lv.F)
                                    : one_rule_per_row(plan.back().gout.layout, false, lv.F);
    lv.bound_in = bound;
    // Sites of the level: at most one per candidate (and no more than the output volume).  Disjoint windows
    // (filter == stride) give at most one site per input site, and the arrays are first sized for half of that;
    // overlapping windows are first sized for as many sites as the input has.  A level that needs more raises its
    // flag and is built again from the safe bound.
    const long long most = std::min(bound * lv.F.tmax, std::max<long long>(out_volume, 1));
    if (safe)
      lv.cap_out = most;
    else if (lv.F.tmax == 1)
      lv.cap_out = std::max((bound + 1) / 2, std::min<long long>(bound, 4096));
    else
      lv.cap_out = std::min(most, std::max<long long>(bound, 4096));
    if (lv.cap_out >= (1ll << 30)) break;
    bound = lv.cap_out;
    cur = lv.out_size;
    plan.push_back(std::move(lv));
  }
}

// collect (after the host has seen the mailbox): the levels up to the first that overflowed its arrays become
// grids and rulebooks of the object, the others are freed.  Returns the number of good levels.
static int chain_collect(scn_metadata *md, long long n_in, long long batch_size, std::vector<ChainLevel> &plan,
                         const int64_t *filter, const int64_t *stride, const volatile int *host, cudaStream_t stream,
                         int *n_built) {
  const int dim = md->dim, L = (int)plan.size();
  int good = 0;
  while (good < L && host[L + 1 + good] == 0 && host[good + 1] <= plan[good].cap_out) ++good;
  for (int l = 0; l < L; ++l) {
    ChainLevel &lv = plan[l];
    if (l < good) {
      const long long n_out = host[l + 1];
      lv.gout.n_active = n_out;
      lv.gout.batch_size = batch_size;
      lv.rb.n_offsets = (int)lv.K;
      lv.rb.dim = dim;
      for (int d = 0; d < dim; ++d) lv.rb.filter[d] = filter[d];
      lv.rb.n_in = n_in;
      lv.rb.n_out = n_out;
      lv.rb.built = true;
      chain_free_level(lv, true, stream);
      md->grids[make_key(dim, lv.out_size.data())] = lv.gout;
      md->strided_rules[make_key(dim, lv.in_size.data(), filter, stride)] = lv.rb;
      g_rulebook_builds.fetch_add(1);
      if (n_built) ++*n_built;
      n_in = n_out;
    } else {
      chain_free_level(lv, false, stream);
    }
  }
  return good;
}

static bool chain_applies(int dim, const int64_t *filter_size, const int64_t *filter_stride) {
  for (int d = 0; d < dim; ++d)
    if (filter_size[d] < 1 || filter_size[d] > 127 || filter_stride[d] < 1 || filter_stride[d] > 127) return false;
  return true;
}

// A chain that was started on the side stream and whose counts the host has not looked at yet.
struct PendingChain {
  std::vector<ChainLevel> plan;
  std::vector<int64_t> filter, stride;
  long long n_in = 0, batch_size = 0;
  cudaEvent_t done = nullptr;
  int *mailbox = nullptr;
  int *lev = nullptr;  // the chain's device counters, freed when the chain is taken over
};

static cudaStream_t g_side_stream[64] = {nullptr};
static std::mutex g_side_mu;

static int side_stream(cudaStream_t *out) {
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev >= 0 && dev < 64, SCN_ERR_UNSUPPORTED, "device index %d unsupported", dev);
  std::lock_guard<std::mutex> lock(g_side_mu);
  if (!g_side_stream[dev]) SCN_CUDA_CHECK(cudaStreamCreateWithFlags(&g_side_stream[dev], cudaStreamNonBlocking));
  *out = g_side_stream[dev];
  return SCN_OK;
}

static int build_strided_chain_from(scn_metadata *md, std::vector<int64_t> start, const int64_t *filter,
                                    const int64_t *stride, int levels, bool safe, cudaStream_t stream, int *n_built);

// The host looks at a started chain: waits for its event (usually long past), makes its levels the object's, and
// builds again, on `stream` and with the safe bounds, whatever overflowed.  The tables are finished for what follows on
// `stream`, and with `on_host` for whatever is enqueued anywhere after this call.
static int chain_finalize(scn_metadata *md, cudaStream_t stream, int *n_built, bool on_host) {
  PendingChain *p = md->pending;
  if (!p) return SCN_OK;
  md->pending = nullptr;
  int st = SCN_OK;
  if (*(const volatile int *)p->mailbox == kNotPosted || on_host) {
    if (cudaEventQuery(p->done) == cudaErrorNotReady) note_host_wait();
    if (cudaEventSynchronize(p->done) != cudaSuccess || *(const volatile int *)p->mailbox == kNotPosted) {
      set_error("strided chain: CUDA error while waiting for the level counts");
      st = SCN_ERR_CUDA;
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  // the counts are here, the last level's tables perhaps not yet: what follows on `stream` comes behind them
  if (st == SCN_OK && cudaStreamWaitEvent(stream, p->done, 0) != cudaSuccess) {
    set_error("strided chain: could not order the caller's stream behind the side stream");
    st = SCN_ERR_CUDA;
  }
  cudaEventDestroy(p->done);
  const int L = (int)p->plan.size();
  int good = L;
  std::vector<int64_t> rest;
  if (st == SCN_OK) {
    good = chain_collect(md, p->n_in, p->batch_size, p->plan, p->filter.data(), p->stride.data(), p->mailbox, stream,
                         n_built);
    if (good < L) rest = p->plan[good].in_size;
  } else {
    for (auto &lv : p->plan) chain_free_level(lv, false, stream);
  }
  device_free(p->lev, stream);
  mailbox_release(p->mailbox);
  std::vector<int64_t> filter = p->filter, stride = p->stride;
  delete p;
  if (st == SCN_OK && good < L)
    st = build_strided_chain_from(md, rest, filter.data(), stride.data(), L - good, true, stream, n_built);
  if (st == SCN_OK && good < L && on_host) SCN_CUDA_CHECK(cudaStreamSynchronize(stream));
  return st;
}

// Drops a started chain (the object is cleared or destroyed): its arrays go back once its kernels have run.
static void chain_abandon(scn_metadata *md, cudaStream_t stream) {
  PendingChain *p = md->pending;
  if (!p) return;
  md->pending = nullptr;
  cudaEventSynchronize(p->done);
  cudaEventDestroy(p->done);
  for (auto &lv : p->plan) chain_free_level(lv, false, stream);
  device_free(p->lev, stream);
  mailbox_release(p->mailbox);
  delete p;
}

static int build_strided_chain_from(scn_metadata *md, std::vector<int64_t> start, const int64_t *filter,
                                    const int64_t *stride, int levels, bool safe, cudaStream_t stream, int *n_built) {
  while (levels >= 2) {
    Grid *gin = find_grid_now(md, start.data());
    if (!gin || gin->n_active >= (1ll << 31)) return SCN_OK;
    std::vector<ChainLevel> plan;
    chain_plan(md, gin, start, filter, stride, levels, safe, plan);
    const int L = (int)plan.size();
    if (L < 2) return SCN_OK;
    if (!md->mailbox) SCN_TRY(mailbox_acquire(&md->mailbox));
    int *lev = nullptr;
    int st = device_alloc((void **)&lev, sizeof(int) * 3 * L, stream);
    if (st == SCN_OK) st = chain_allocate(plan, stream);
    if (st == SCN_OK) st = chain_enqueue(md, gin, plan, lev, md->mailbox, stream);
    device_free(lev, stream);
    if (st == SCN_OK) {
      st = wait_posted(md->mailbox, stream);
    }
    if (st != SCN_OK) {
      for (auto &lv : plan) chain_free_level(lv, false, stream);
      return st;
    }
    const int good = chain_collect(md, gin->n_active, gin->batch_size, plan, filter, stride, md->mailbox, stream, n_built);
    if (good == L) return SCN_OK;
    // a level shrank less than guessed: that level and the deeper ones again, arrays sized by the input
    start = plan[good].in_size;
    levels = L - good;
    safe = true;
  }
  return SCN_OK;
}

// Builds up to `levels` consecutive rulebooks of (filter_size, filter_stride) starting at the grid of
// `input_size`, each level's output size (in - f) / s + 1.  Does nothing (SCN_OK) where the chain does
// not apply -- fewer than two levels to build, sizes that do not divide, no grid, rulebooks already there --
// because the per-level call that follows builds or reports whatever is left.  A chain that was started
// earlier on the side stream is taken over here.
int build_strided_chain(scn_metadata *md, const int64_t *input_size, const int64_t *filter_size,
                        const int64_t *filter_stride, int levels, cudaStream_t stream, int *n_built) {
  if (n_built) *n_built = 0;
  SCN_TRY(md_touch(md, stream));
  SCN_TRY(chain_finalize(md, stream, n_built));
  if (!chain_applies(md->dim, filter_size, filter_stride)) return SCN_OK;
  return build_strided_chain_from(md, std::vector<int64_t>(input_size, input_size + md->dim), filter_size, filter_stride,
                                  std::min(levels, kMaxChain), false, stream, n_built);
}

// The same chain, started without waiting for it: its kernels go to a side stream of the device behind what
// `stream` holds now (the input grid), so they run beside whatever the caller enqueues on `stream` next -- the
// first level's convolutions of a U-Net -- and the host does not wait here.  Whoever first asks for one of those
// levels (a grid that is not there yet, the rulebook of a level, scn_md_strided_chain) finds the chain finished,
// reads the counts and makes the levels the object's.  Nothing is started when a chain is already under way.
int start_strided_chain(scn_metadata *md, const int64_t *input_size, const int64_t *filter_size,
                        const int64_t *filter_stride, int levels, cudaStream_t stream) {
  SCN_TRY(md_touch(md, stream));
  if (md->pending || !chain_applies(md->dim, filter_size, filter_stride)) return SCN_OK;
  Grid *gin = find_grid_now(md, input_size);
  if (!gin || gin->n_active >= (1ll << 31)) return SCN_OK;
  PendingChain *p = new PendingChain();
  chain_plan(md, gin, std::vector<int64_t>(input_size, input_size + md->dim), filter_size, filter_stride,
             std::min(levels, kMaxChain), false, p->plan);
  if (p->plan.size() < 2) {
    delete p;
    return SCN_OK;
  }
  // The chain's memory comes from `stream` (blocks that earlier work of `stream` gave back can be used again at
  // once; taken on the side stream the pool would have to find blocks nobody can still be using, and grows when it
  // finds none: single steps of 18-22 ms among 13.6 ms ones).  The side stream starts behind that point of
  // `stream`; the scratch goes back when the chain is taken over.
  cudaStream_t side = nullptr;
  cudaEvent_t ready = nullptr;
  int st = side_stream(&side);
  if (st == SCN_OK) st = mailbox_acquire(&p->mailbox);
  if (st == SCN_OK) st = device_alloc((void **)&p->lev, sizeof(int) * 3 * p->plan.size(), stream);
  if (st == SCN_OK) st = chain_allocate(p->plan, stream);
  if (st == SCN_OK && (cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) != cudaSuccess ||
                       cudaEventCreateWithFlags(&p->done, cudaEventDisableTiming) != cudaSuccess ||
                       cudaEventRecord(ready, stream) != cudaSuccess || cudaStreamWaitEvent(side, ready, 0) != cudaSuccess)) {
    set_error("strided chain: could not order the side stream behind the caller's");
    st = SCN_ERR_CUDA;
  }
  bool launched = false;
  if (st == SCN_OK) {
    st = chain_enqueue(md, gin, p->plan, p->lev, p->mailbox, side);
    launched = true;  // (possibly in part)
  }
  if (st == SCN_OK && cudaEventRecord(p->done, side) != cudaSuccess) {
    set_error("strided chain: could not record the end of the chain");
    st = SCN_ERR_CUDA;
  }
  if (ready) cudaEventDestroy(ready);
  if (st != SCN_OK) {
    if (launched) cudaStreamSynchronize(side);  // what was enqueued must not outlive the arrays
    for (auto &lv : p->plan) chain_free_level(lv, false, stream);
    device_free(p->lev, stream);
    if (p->done) cudaEventDestroy(p->done);
    mailbox_release(p->mailbox);
    delete p;
    return st;
  }
  p->filter.assign(filter_size, filter_size + md->dim);
  p->stride.assign(filter_stride, filter_stride + md->dim);
  p->n_in = gin->n_active;
  p->batch_size = gin->batch_size;
  md->pending = p;
  return SCN_OK;
}

// ------------------------------------------------------------------------------------------
// rulebook views
// ------------------------------------------------------------------------------------------

static bool counts_landed(const CountTicket *t) {
  for (int k = 0; k < t->n; ++k)
    if (t->host[k] == kCountPending) return false;
  return true;
}

// Waits until the device has written a ticket's counts: a short look, then for the whole device (the kernel that writes
// them was enqueued before the ticket was handed out, on a stream that may be gone by now).
static int counts_wait(CountTicket *t) {
  if (counts_landed(t)) return SCN_OK;  // an answer that already landed is no wait
  note_host_wait();
  int current = -1;
  SCN_CUDA_CHECK(cudaGetDevice(&current));
  if (current != t->device) SCN_CUDA_CHECK(cudaSetDevice(t->device));
  const cudaError_t e = cudaDeviceSynchronize();
  if (current != t->device) cudaSetDevice(current);
  SCN_CUDA_CHECK(e);
  SCN_REQUIRE(counts_landed(t), SCN_ERR_CUDA, "rule counts were not written");
  return SCN_OK;
}

void count_ticket_release(CountTicket *t) {
  if (!t || t->refs.fetch_sub(1) != 1) return;
  TicketPool &P = ticket_pool();
  std::lock_guard<std::mutex> lock(P.mu);
  P.dropped[t->device].push_back(t);  // its chunk is handed on once the device has written to it
}

int count_ticket_total(CountTicket *t, long long *total) {
  SCN_TRY(counts_wait(t));
  long long s = 0;
  for (int k = 0; k < t->n; ++k) s += (long long)t->host[k];
  *total = s;
  return SCN_OK;
}

static void counts_from_ticket(Rulebook &rb) {
  rb.counts_host.assign(rb.n_offsets, 0);
  for (int k = 0; k < rb.n_offsets; ++k) rb.counts_host[k] = (long long)rb.ticket->host[k];
  long long t = 0;
  for (auto c : rb.counts_host) t += c;
  rb.total_rules = t;
}

// filter volumes beyond a ticket's chunk: plain copy and wait
static int rulebook_counts_blocking(Rulebook &rb, cudaStream_t stream) {
  std::vector<unsigned long long> h(rb.n_offsets);
  SCN_CUDA_CHECK(cudaMemcpyAsync(h.data(), rb.counts_dev, sizeof(unsigned long long) * rb.n_offsets,
                                 cudaMemcpyDeviceToHost, stream));
  note_host_wait();
  SCN_CUDA_CHECK(cudaStreamSynchronize(stream));
  rb.counts_host.assign(h.begin(), h.end());
  long long t = 0;
  for (auto c : rb.counts_host) t += c;
  rb.total_rules = t;
  return SCN_OK;
}

int rulebook_counts_async(Rulebook &rb, cudaStream_t stream) {
  if (rb.total_rules >= 0) return SCN_OK;
  if (!rb.ticket) return rulebook_counts_blocking(rb, stream);
  if (counts_landed(rb.ticket)) counts_from_ticket(rb);
  return SCN_OK;
}

int rulebook_counts(Rulebook &rb, cudaStream_t stream) {
  if (rb.total_rules >= 0) return SCN_OK;
  if (!rb.ticket) return rulebook_counts_blocking(rb, stream);
  SCN_TRY(counts_wait(rb.ticket));
  counts_from_ticket(rb);
  return SCN_OK;
}

__global__ void k_transpose_rules(const int *__restrict__ nbr, long long n_out, long long n_in, int K,
                                  int *__restrict__ tnbr) {
  SCN_GRID_WAIT();
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)K * n_out) return;
  int i = nbr[idx];
  if (i < 0) return;
  long long k = idx / n_out, o = idx % n_out;
  tnbr[k * n_in + i] = (int)o;
}

int rulebook_transposed(Rulebook &rb, cudaStream_t stream) {
  if (rb.tnbr) return SCN_OK;
  size_t bytes = sizeof(int) * (size_t)(rb.n_offsets * std::max<long long>(rb.n_in, 1));
  SCN_TRY(device_alloc((void **)&rb.tnbr, bytes, stream));
  SCN_CUDA_CHECK(cudaMemsetAsync(rb.tnbr, 0xFF, bytes, stream));
  long long total = (long long)rb.n_offsets * rb.n_out;
  if (total > 0) {
    SCN_LAUNCH(k_transpose_rules, (unsigned)ceil_div(total, 256), 256, 0, stream, rb.nbr, rb.n_out, rb.n_in, rb.n_offsets, rb.tnbr);
    SCN_CUDA_CHECK(cudaGetLastError());
  }
  return SCN_OK;
}

__global__ void k_rule_flags(const int *__restrict__ nbr, long long total, int *__restrict__ flag) {
  SCN_GRID_WAIT();
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < total) flag[idx] = nbr[idx] >= 0;
}
__global__ void k_rule_compact(const int *__restrict__ nbr, const int *__restrict__ pos, long long total,
                               long long n_out, int *__restrict__ pairs) {
  SCN_GRID_WAIT();
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  int i = nbr[idx];
  if (i < 0) return;
  long long p = pos[idx];
  pairs[2 * p] = i;
  pairs[2 * p + 1] = (int)(idx % n_out);
}

static int rulebook_export(Rulebook &rb, int64_t *n_offsets, int64_t *counts_host, int32_t *pairs_dev,
                           cudaStream_t stream) {
  SCN_TRY(rulebook_counts(rb, stream));
  if (n_offsets) *n_offsets = rb.n_offsets;
  if (counts_host)
    for (int k = 0; k < rb.n_offsets; ++k) counts_host[k] = rb.counts_host[k];
  if (!pairs_dev) return SCN_OK;
  long long total = (long long)rb.n_offsets * rb.n_out;
  if (total == 0) return SCN_OK;
  SCN_REQUIRE(total < (1ll << 31), SCN_ERR_UNSUPPORTED, "rulebook too large to export");
  int *flag = nullptr;
  SCN_TRY(device_alloc((void **)&flag, sizeof(int) * (size_t)total, stream));
  unsigned blocks = (unsigned)ceil_div(total, 256);
  SCN_LAUNCH(k_rule_flags, blocks, 256, 0, stream, rb.nbr, total, flag);
  SCN_TRY(exclusive_scan_i32(flag, flag, total, nullptr, stream));
  SCN_LAUNCH(k_rule_compact, blocks, 256, 0, stream, rb.nbr, flag, total, rb.n_out, pairs_dev);
  SCN_CUDA_CHECK(cudaGetLastError());
  SCN_TRY(device_free(flag, stream));
  return SCN_OK;
}

}  // namespace scn

// ------------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------------

using namespace scn;

extern "C" {

long long scn_rulebook_build_count(void) { return g_rulebook_builds.load(); }

int scn_md_create(int dimension, scn_metadata **md) {
  SCN_REQUIRE(md, SCN_ERR_BAD_ARG, "null output pointer");
  SCN_REQUIRE(dimension >= 1 && dimension <= SCN_MAX_DIMENSION, SCN_ERR_BAD_ARG,
              "dimension %d not in 1..%d", dimension, SCN_MAX_DIMENSION);
  *md = new scn_metadata();
  (*md)->dim = dimension;
  return SCN_OK;
}

int scn_md_clear(scn_metadata *md, void *stream) {
  SCN_REQUIRE(md, SCN_ERR_BAD_ARG, "null metadata");
  return md_clear(md, (cudaStream_t)stream);
}

static int md_destroy_on(scn_metadata *md, cudaStream_t stream) {
  if (!md) return SCN_OK;
  // free on the device that owns the tables, whatever device is current
  int current = -1;
  const bool switch_device = md->device >= 0 && cudaGetDevice(&current) == cudaSuccess && current != md->device;
  if (switch_device) cudaSetDevice(md->device);
  mailbox_release(md->mailbox);
  md->mailbox = nullptr;
  count_ticket_release(md->last_ticket);
  md->last_ticket = nullptr;
  md_clear(md, stream);
  device_free(md->flags_dev, stream);
  device_free(md->scalars_dev, stream);
  delete md;
  if (switch_device) cudaSetDevice(current);
  return SCN_OK;
}

int scn_md_destroy(scn_metadata *md) {
  // stream-ordered frees behind the last work enqueued on the object: kernels of that stream that
  // still read the tables finish before the memory can be handed out again
  return md_destroy_on(md, md ? md->last_stream : nullptr);
}

int scn_md_destroy_on_stream(scn_metadata *md, void *stream) { return md_destroy_on(md, (cudaStream_t)stream); }

int scn_md_input_layer(scn_metadata *md, const int64_t *spatial_size, const int64_t *coords,
                       int coords_on_device, int64_t n_rows, int n_cols, int64_t batch_size,
                       int mode, void *stream, int64_t *n_active) {
  return md_input_layer(md, spatial_size, coords, coords_on_device, n_rows, n_cols, batch_size, mode, 0,
                        (cudaStream_t)stream, n_active);
}

int scn_md_bl_input_layer(scn_metadata *md, const int64_t *spatial_size, const int64_t *coords,
                          int coords_on_device, int64_t batch_size, int64_t length, int mode, void *stream,
                          int64_t *n_active) {
  SCN_REQUIRE(md, SCN_ERR_BAD_ARG, "null metadata");
  SCN_REQUIRE(batch_size >= 0 && length >= 0, SCN_ERR_BAD_ARG, "negative batch size or length");
  SCN_REQUIRE(mode >= 0 && mode <= 4, SCN_ERR_BAD_ARG, "input layer mode %d not in 0..4", mode);
  // blRules keeps the LAST point of a site in mode 1 and the FIRST in mode 2 (IOLayersRules.h:172-199),
  // inputLayerRules the other way round (IOLayersRules.h:95-106): stored in the latter's terms.
  const int stored_mode = mode == 1 ? 2 : mode == 2 ? 1 : mode;
  // an empty batch x length array still needs a non-zero stride for the sample index
  SCN_TRY(md_input_layer(md, spatial_size, coords, coords_on_device, batch_size * length, md->dim, batch_size,
                         stored_mode, std::max<int64_t>(length, 1), (cudaStream_t)stream, n_active));
  return SCN_OK;
}

int scn_md_poll_errors(scn_metadata *md, void *stream) {
  SCN_REQUIRE(md, SCN_ERR_BAD_ARG, "null metadata");
  if (!md->flags_dev) return SCN_OK;
  SCN_TRY(md_touch(md, (cudaStream_t)stream));
  int flags = 0;
  SCN_TRY(fetch_flags(md, (cudaStream_t)stream, &flags));
  return flags_to_status(flags);
}

int scn_md_n_active(scn_metadata *md, const int64_t *spatial_size, int64_t *n_active) {
  SCN_REQUIRE(md && spatial_size && n_active, SCN_ERR_BAD_ARG, "null argument");
  Grid *g = find_grid(md, spatial_size);
  // the reference's unordered_map lookup default-constructs a zero for an unknown size
  *n_active = g ? g->n_active : 0;
  return SCN_OK;
}

int scn_md_batch_size(scn_metadata *md, const int64_t *spatial_size, int64_t *batch_size) {
  SCN_REQUIRE(md && spatial_size && batch_size, SCN_ERR_BAD_ARG, "null argument");
  Grid *g = find_grid(md, spatial_size);
  *batch_size = g ? g->batch_size : 0;
  return SCN_OK;
}

int scn_md_spatial_locations(scn_metadata *md, const int64_t *spatial_size, int64_t *out_dev,
                             void *stream) {
  SCN_REQUIRE(md && spatial_size, SCN_ERR_BAD_ARG, "null argument");
  Grid *g = find_grid(md, spatial_size);
  SCN_REQUIRE(g, SCN_ERR_NO_GRID, "no grid for that spatial size");
  if (g->n_active == 0) return SCN_OK;
  SCN_REQUIRE(out_dev, SCN_ERR_BAD_ARG, "null output");
  SCN_TRY(md_touch(md, (cudaStream_t)stream));
  SCN_LAUNCH(k_spatial_locations, (unsigned)ceil_div(g->n_active, 256), 256, 0, (cudaStream_t)stream, g->layout, g->row_keys, g->n_active, (long long *)out_dev);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

int scn_md_submanifold_rulebook(scn_metadata *md, const int64_t *spatial_size,
                                const int64_t *filter_size, void *stream, int64_t *n_rules) {
  SCN_REQUIRE(md && spatial_size && filter_size, SCN_ERR_BAD_ARG, "null argument");
  Rulebook *rb = nullptr;
  SCN_TRY(get_submanifold_rulebook(md, spatial_size, filter_size, (cudaStream_t)stream, &rb));
  if (n_rules) {
    SCN_TRY(rulebook_counts(*rb, (cudaStream_t)stream));
    *n_rules = rb->total_rules;
  }
  return SCN_OK;
}

int scn_md_strided_chain(scn_metadata *md, const int64_t *input_size, const int64_t *filter_size,
                         const int64_t *filter_stride, int levels, void *stream, int *n_built) {
  SCN_REQUIRE(md && input_size && filter_size && filter_stride, SCN_ERR_BAD_ARG, "null argument");
  return build_strided_chain(md, input_size, filter_size, filter_stride, levels, (cudaStream_t)stream, n_built);
}

int scn_md_strided_chain_start(scn_metadata *md, const int64_t *input_size, const int64_t *filter_size,
                               const int64_t *filter_stride, int levels, void *stream) {
  SCN_REQUIRE(md && input_size && filter_size && filter_stride, SCN_ERR_BAD_ARG, "null argument");
  return start_strided_chain(md, input_size, filter_size, filter_stride, levels, (cudaStream_t)stream);
}

int scn_md_strided_rulebook(scn_metadata *md, const int64_t *input_size, const int64_t *output_size,
                            const int64_t *filter_size, const int64_t *filter_stride, void *stream,
                            int64_t *n_active_out, int64_t *n_rules) {
  SCN_REQUIRE(md && input_size && output_size && filter_size && filter_stride, SCN_ERR_BAD_ARG,
              "null argument");
  Rulebook *rb = nullptr;
  SCN_TRY(get_strided_rulebook(md, input_size, output_size, filter_size, filter_stride,
                               (cudaStream_t)stream, &rb));
  if (n_active_out) *n_active_out = rb->n_out;
  if (n_rules) {
    SCN_TRY(rulebook_counts(*rb, (cudaStream_t)stream));
    *n_rules = rb->total_rules;
  }
  return SCN_OK;
}

int scn_md_rulebook_export(scn_metadata *md, int kind, const int64_t *sizes_a, const int64_t *sizes_b,
                           const int64_t *sizes_c, int64_t *n_offsets, int64_t *counts_host,
                           int32_t *pairs_dev, void *stream) {
  SCN_REQUIRE(md && sizes_a && sizes_b, SCN_ERR_BAD_ARG, "null argument");
  Rulebook *rb = nullptr;
  if (kind == SCN_RULES_SUBMANIFOLD) {
    auto it = md->sub_rules.find(make_key(md->dim, sizes_a, sizes_b));
    if (it != md->sub_rules.end()) rb = &it->second;
  } else if (kind == SCN_RULES_STRIDED) {
    SCN_REQUIRE(sizes_c, SCN_ERR_BAD_ARG, "null stride");
    auto it = md->strided_rules.find(make_key(md->dim, sizes_a, sizes_b, sizes_c));
    if (it != md->strided_rules.end()) rb = &it->second;
  } else {
    SCN_REQUIRE(false, SCN_ERR_BAD_ARG, "unknown rulebook kind %d", kind);
  }
  SCN_REQUIRE(rb && rb->built, SCN_ERR_NO_GRID, "that rulebook has not been built");
  return rulebook_export(*rb, n_offsets, counts_host, pairs_dev, (cudaStream_t)stream);
}
}
