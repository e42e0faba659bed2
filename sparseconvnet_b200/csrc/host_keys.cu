// Host coordinates -> packed site keys in pinned memory.
//
// A point arrives as dim + 1 64-bit integers in pageable memory.  Copied as they are (32 bytes a point in 3-D, through the
// driver's staging buffers at 12.5 GB/s, with the host held until the stream reaches the copy) 400 k points were 1.0 ms of
// a training step's 9.5.  Here a few host threads check and pack each point into the site table's key (bound by reading the
// coordinates once), and the insert kernel reads those bytes of the keys that are in use across the bus: 4 to 6 instead of 32, no
// staging.
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "metadata.cuh"

namespace scn {
namespace {

// ---- a few helper threads ---------------------------------------------------------------------------
// The caller takes part itself and never waits for a helper that has not taken a piece, so a busy (or, in a forked
// child, missing) helper only costs its share.  One caller at a time; another one does its work alone.
class Helpers {
 public:
  static Helpers &get() {
    static Helpers *h = new Helpers();  // leaked on purpose: threads may be waiting in it at exit
    return *h;
  }
  void run(int pieces, const std::function<void(int)> &fn) {
    std::unique_lock<std::mutex> use(use_, std::try_to_lock);
    if (pieces < 2 || !use.owns_lock()) {
      for (int i = 0; i < pieces; ++i) fn(i);
      return;
    }
    {
      std::lock_guard<std::mutex> lock(mu_);
      while (threads_ < want_) {
        try {
          std::thread(&Helpers::work, this).detach();
          ++threads_;
        } catch (const std::system_error &) {
          want_ = threads_;  // no more threads to be had
        }
      }
      fn_ = &fn;
      pieces_ = pieces;
      next_ = 0;
      busy_ = 0;
      ++turn_;
    }
    wake_.notify_all();
    for (;;) {
      int i;
      {
        std::lock_guard<std::mutex> lock(mu_);
        if (next_ >= pieces_) break;
        i = next_++;
      }
      fn(i);
    }
    std::unique_lock<std::mutex> lock(mu_);
    done_.wait(lock, [&] { return busy_ == 0; });
    fn_ = nullptr;
  }

 private:
  Helpers() {
    const int cores = (int)std::thread::hardware_concurrency();
    want_ = std::max(0, std::min(7, cores / 2 - 1));
  }
  void work() {
    unsigned long long seen = 0;
    std::unique_lock<std::mutex> lock(mu_);
    for (;;) {
      wake_.wait(lock, [&] { return fn_ && turn_ != seen && next_ < pieces_; });
      seen = turn_;
      ++busy_;
      while (next_ < pieces_) {
        const int i = next_++;
        const std::function<void(int)> *fn = fn_;
        lock.unlock();
        (*fn)(i);
        lock.lock();
      }
      if (--busy_ == 0) done_.notify_all();
    }
  }
  std::mutex use_, mu_;
  std::condition_variable wake_, done_;
  const std::function<void(int)> *fn_ = nullptr;
  int pieces_ = 0, next_ = 0, busy_ = 0, threads_ = 0, want_ = 0;
  unsigned long long turn_ = 0;
};

// ---- pinned buffers -------------------------------------------------------------------------------
// Powers of two of bytes; at most kKeepBytes of idle ones are kept (scn_trim_memory gives them back).
constexpr size_t kKeepBytes = 64u << 20;
struct Idle {
  void *p;
  size_t bytes;
};
struct PinnedPool {
  std::mutex mu;
  std::vector<Idle> idle;
  size_t kept = 0;
};
PinnedPool &pinned_pool() {
  static PinnedPool *p = new PinnedPool();
  return *p;
}

// what a packed key is written to
struct WholeKeys {
  unsigned long long *keys;
  void put(long long i, unsigned long long key) { keys[i] = key; }
  unsigned long long any() const { return 0; }
};
struct KeyBytes {
  NarrowKeys keys;
  unsigned long long all = 0;
  void put(long long i, unsigned long long key) {
    keys.low[i] = (unsigned)key;
    keys.high[0][i] = (unsigned char)(key >> 32);
    keys.high[1][i] = (unsigned char)(key >> 40);
    all |= key;
  }
  unsigned long long any() const { return all; }
};

template <int DIM, class Keys>
void pack_rows(const KeyLayout &L, const long long *coords, long long first, long long last, int ncols, long long bl_length,
               Keys &keys, int &samples, bool &bad) {
  const int dim = DIM ? DIM : L.dim;
  long long most = -1;
  bool wrong = false;
  for (long long i = first; i < last; ++i) {
    const long long *c = coords + i * ncols;
    if (bl_length > 0 && c[0] < 0) {  // empty slot of the batch x length array
      keys.put(i, kEmptyKey);
      continue;
    }
    const long long bl = bl_length > 0 ? i / bl_length : (ncols > dim ? c[dim] : 0);
    bool ok = (unsigned long long)bl < (1ull << L.batch_bits);
    unsigned long long key = (unsigned long long)bl << L.batch_shift;
    for (int d = 0; d < dim; ++d) {
      ok &= (unsigned long long)c[d] < (unsigned long long)L.size[d];
      key |= (unsigned long long)c[d] << L.shift[d];
    }
    wrong |= !ok;
    keys.put(i, key);
    most = std::max(most, bl);
  }
  samples = wrong ? 0 : (int)(most + 1);
  bad = wrong;
}

}  // namespace

int pinned_acquire(size_t bytes, void **p, size_t *got) {
  SCN_TRY(test_allocation());
  size_t want = 4096;
  while (want < bytes) want <<= 1;
  *got = want;
  PinnedPool &P = pinned_pool();
  {
    std::lock_guard<std::mutex> lock(P.mu);
    for (size_t i = 0; i < P.idle.size(); ++i)
      if (P.idle[i].bytes == want) {
        *p = P.idle[i].p;
        P.kept -= want;
        P.idle[i] = P.idle.back();
        P.idle.pop_back();
        return SCN_OK;
      }
  }
  SCN_CUDA_CHECK(cudaHostAlloc(p, want, cudaHostAllocMapped | cudaHostAllocPortable));
  return SCN_OK;
}

void pinned_release(void *p, size_t bytes) {
  if (!p) return;
  PinnedPool &P = pinned_pool();
  {
    std::lock_guard<std::mutex> lock(P.mu);
    if (P.kept + bytes <= kKeepBytes) {
      P.idle.push_back({p, bytes});
      P.kept += bytes;
      return;
    }
  }
  cudaFreeHost(p);
}

void pinned_trim() {
  PinnedPool &P = pinned_pool();
  std::vector<Idle> idle;
  {
    std::lock_guard<std::mutex> lock(P.mu);
    idle.swap(P.idle);
    P.kept = 0;
  }
  for (auto &b : idle) cudaFreeHost(b.p);
}

namespace {
template <class Keys>
void pack_all(const KeyLayout &L, const long long *coords, long long n, int ncols, long long bl_length, const Keys &to, int *samples,
              bool *bad, unsigned long long *any) {
  // pieces of 16 k points (~30 us each): below two of them waking a helper costs more than it saves
  constexpr long long kPiece = 16384;
  const int pieces = (int)ceil_div(n, kPiece);
  std::atomic<int> most{0};
  std::atomic<bool> wrong{false};
  std::atomic<unsigned long long> bits{0};
  Helpers::get().run(pieces, [&](int i) {
    const long long first = i * kPiece, last = std::min(n, first + kPiece);
    int s = 0;
    bool b = false;
    Keys keys = to;
    switch (L.dim) {
      case 2: pack_rows<2>(L, coords, first, last, ncols, bl_length, keys, s, b); break;
      case 3: pack_rows<3>(L, coords, first, last, ncols, bl_length, keys, s, b); break;
      case 4: pack_rows<4>(L, coords, first, last, ncols, bl_length, keys, s, b); break;
      default: pack_rows<0>(L, coords, first, last, ncols, bl_length, keys, s, b);
    }
    if (b) wrong.store(true);
    bits.fetch_or(keys.any());
    int was = most.load();
    while (s > was && !most.compare_exchange_weak(was, s)) {
    }
  });
  *samples = most.load();
  *bad = wrong.load();
  if (any) *any = bits.load();
}
}  // namespace

// keys[i] of every row (the empty key for an empty slot); *samples = batch indices in use; *bad: some row lies outside.
void pack_keys(const KeyLayout &L, const long long *coords, long long n, int ncols, long long bl_length,
               unsigned long long *keys, int *samples, bool *bad) {
  pack_all(L, coords, n, ncols, bl_length, WholeKeys{keys}, samples, bad, nullptr);
}
void pack_keys(const KeyLayout &L, const long long *coords, long long n, int ncols, const NarrowKeys &keys, int *samples, bool *bad,
               unsigned long long *any) {
  pack_all(L, coords, n, ncols, 0, KeyBytes{keys}, samples, bad, any);
}

}  // namespace scn
