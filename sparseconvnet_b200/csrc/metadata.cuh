// Host-side description of what a scn_metadata object owns on the device: one Grid per
// spatial scale (site hash + row -> key table) and the dense per-filter-offset rulebooks.
#pragma once

#include <atomic>
#include <map>
#include <vector>

#include "common.cuh"

namespace scn {

// Active sites of one spatial scale.
struct Grid {
  KeyLayout layout{};
  long long n_active = 0;
  long long batch_size = 0;
  bool may_have_blank_rows = false;  // input mode 0: rows whose site a later row took over are in no map
  unsigned long long *row_keys = nullptr;  // [n_active] packed key of every feature row
  HashTable table{};                       // key -> row
};

// Dense rulebook.  The reference stores, per filter offset k, a compacted list of
// (input_row, output_row) pairs (Metadata.h:35).  Because every (offset, output row) has at
// most one rule, the same information is kept here as a table
//     nbr[k * n_out + o] = input row feeding output row o through filter offset k, or -1
// which the output-stationary kernels read with coalesced loads and which the builders write
// without compaction, atomics or a host round trip.  `tnbr` is the transposed view
//     tnbr[k * n_in + i] = output row fed by input row i through offset k, or -1
// used by Deconvolution (the reference swaps the two rule columns, CPU/Deconvolution.cpp:35-37);
// it is valid because every (offset, input row) also has at most one rule.
// A rulebook's per-offset rule counts on their way to the host: the last block of the kernel that builds the rulebook
// writes them into pinned, device-mapped memory.  The multiply-add count the reference's operators return needs these
// totals (CPU/Convolution.cpp:141), and waiting for them where the operator is called would leave the GPU idle once
// per rulebook; a caller that can take the number later is handed the ticket instead.  Reference counted: the ticket
// outlives its rulebook and metadata.
struct CountTicket {
  volatile unsigned long long *host = nullptr;  // [n] pinned; kCountPending until the device has written the value
  unsigned long long *dev = nullptr;            // the same memory as the device sees it
  int n = 0, device = 0;
  std::atomic<int> refs{1};
};
constexpr unsigned long long kCountPending = ~0ull;
void count_ticket_release(CountTicket *t);
int count_ticket_total(CountTicket *t, long long *total);  // waits for the values

// The packing of a table's output rows into tensor-core tiles (row_order.cu): order[p] = output row at position
// p, -1 past the end (padded to whole tiles); tile_bits[t][words] = filter offsets for which any of the 128 rows
// of tile t has a rule; packed[t][j][128] = the table's entries of the tile's rows for the j-th of those offsets,
// -1 where a row has no rule (room for all K offsets per tile, only the tile's own are written).
constexpr int kOrderTile = 128;
constexpr int kOrderMaxOffsets = 128;
inline int mask_words(int K) { return K <= 32 ? 1 : 4; }
struct RowOrder {
  int *order = nullptr;
  unsigned *tile_bits = nullptr;
  int *packed = nullptr;
  int *by_work = nullptr;  // the tiles, those with the most offsets first (null: small levels, tiles in their order)
  int words = 1;  // 32-bit words per tile: 1 up to 32 offsets, else 4
  bool one_offset = false; // every tile has at most one filter offset (rulebook_children_order)
  bool fp32_only = false;  // made by an fp32 convolution of a small level: no reason for its weight gradient to use tiles
  long long n_tiles = 0;
};

struct Rulebook {
  int n_offsets = 0;  // filter volume K
  int dim = 0;
  int64_t filter[kMaxDim] = {0};
  long long n_in = 0, n_out = 0;
  int *nbr = nullptr;
  int *tnbr = nullptr;                       // built on first use
  RowOrder order, torder;                    // of nbr and of tnbr; built on first use
  // offsets with a rule of every output row of nbr, mask_words(K) words each (submanifold rulebooks up to
  // kOrderMaxOffsets offsets; null otherwise)
  unsigned *masks = nullptr;
  // [K] rules per offset, then the builder's count of finished blocks; of a strided rulebook K + 1 more zeros behind
  // them (rulebook_children_order)
  unsigned long long *counts_dev = nullptr;
  std::vector<long long> counts_host;        // filled on first request (waits for the stream)
  long long total_rules = -1;
  CountTicket *ticket = nullptr;             // counts in flight (null above kTicketValues offsets)
  bool built = false;
  bool disjoint = false;   // strided: an input row has at most one rule (windows side by side)
  bool one_parent = false; // strided: every input row has exactly one rule (of the sizes it was built with)
  bool symmetric = false;  // submanifold with odd filter sizes: tnbr[k] is nbr[K - 1 - k]
};

int rulebook_counts(Rulebook &rb, cudaStream_t stream);         // fills counts_host/total_rules (waits)
// Fills counts_host/total_rules without waiting if the counts have landed; total_rules stays -1 while they are in flight.
int rulebook_counts_async(Rulebook &rb, cudaStream_t stream);
int rulebook_transposed(Rulebook &rb, cudaStream_t stream);     // builds tnbr if missing
// builds the packing order of the table [K][n] (nbr or tnbr of `rb`) if missing
int rulebook_row_order(const Rulebook &rb, const int *table, long long n, RowOrder &ord, cudaStream_t stream);
// the same for tnbr of a rulebook with `one_parent` and at most 32 offsets, from nbr in one launch
int rulebook_children_order(const Rulebook &rb, RowOrder &ord, cudaStream_t stream);
constexpr int kChildrenMaxOffsets = 32;
void free_row_order(RowOrder &o, cudaStream_t stream);

struct PendingChain;  // metadata.cu: levels of a strided chain whose kernels run on the side stream

}  // namespace scn

struct scn_metadata {
  int dim = 0;
  // Where the tables live and what last touched them: every entry point that takes the object and
  // a stream notes both (scn::md_touch), so that destroying the object can free on the device that
  // owns the memory and, stream-ordered, behind the last work that reads it.
  int device = -1;
  cudaStream_t last_stream = nullptr;
  std::map<std::vector<int64_t>, scn::Grid> grids;             // key: spatial size
  std::map<std::vector<int64_t>, scn::Rulebook> sub_rules;      // key: size | filter
  std::map<std::vector<int64_t>, scn::Rulebook> strided_rules;  // key: in size | filter | stride

  // input-layer rules of the last scn_md_input_layer call: CSR over output rows of the input
  // rows that land on each site, ascending (the order the reference sums them in).
  int input_mode = -1;
  long long input_n_rows = 0, input_n_active = 0;
  int *input_csr_start = nullptr;  // [n_active + 1]
  int *input_csr_rows = nullptr;   // [n_rows]

  scn::CountTicket *last_ticket = nullptr;  // of the last operator that answered "count pending"
  scn::PendingChain *pending = nullptr;     // a strided chain started with scn_md_strided_chain_start, not yet taken over

  int *flags_dev = nullptr;   // device word the kernels OR DeviceFlag bits into
  int *mailbox = nullptr;     // pinned, device-mapped host slot (8 ints) the waited-for integers are posted to
  int *scalars_dev = nullptr; // small device scratch: [0] batch indices in use, [1] finished blocks
};

namespace scn {
// notes the device (first call) and the stream of an operation on `md`; SCN_ERR_BAD_ARG when the
// object is used from another device than the one that holds its tables
int md_touch(scn_metadata *md, cudaStream_t stream);
std::vector<int64_t> make_key(int dim, const int64_t *a, const int64_t *b = nullptr,
                              const int64_t *c = nullptr);
Grid *find_grid(scn_metadata *md, const int64_t *spatial_size);
// finds or builds
int get_submanifold_rulebook(scn_metadata *md, const int64_t *spatial_size,
                             const int64_t *filter_size, cudaStream_t stream, Rulebook **out);
int get_strided_rulebook(scn_metadata *md, const int64_t *input_size, const int64_t *output_size,
                         const int64_t *filter_size, const int64_t *filter_stride,
                         cudaStream_t stream, Rulebook **out);
// Feature rows in the split form of the tensor-core kernels (k_tile_split), handed from the layer that makes them to the
// one that reads them: what the calling thread's next convolution may read instead of splitting its input, and where it may
// leave its result in that form (scn_set_split_rows).
struct SplitRows {
  const void *in = nullptr;
  void *out = nullptr;
};
SplitRows take_split_rows();  // (once)
void split_rows_written();

// host_keys.cu: host coordinates as packed keys in pinned, device-mapped memory
int pinned_acquire(size_t bytes, void **p, size_t *got);
void pinned_release(void *p, size_t bytes);
void pinned_trim();
void pack_keys(const KeyLayout &L, const long long *coords, long long n, int ncols, long long bl_length,
               unsigned long long *keys, int *samples, bool *bad);
// ... in bytes of their own: bits 0 to 31, 32 to 39, 40 to 47 of every key; *any: the bits that some key has
struct NarrowKeys {
  unsigned *low;
  unsigned char *high[2];
};
void pack_keys(const KeyLayout &L, const long long *coords, long long n, int ncols, const NarrowKeys &keys, int *samples, bool *bad,
               unsigned long long *any);

}  // namespace scn
