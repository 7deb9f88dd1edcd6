// Host-visible interface between the orchestration (spgemm.cu) and the kernel
// translation units.  Plain structs only; no torch types anywhere.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace b200 {

struct DevStatus;

constexpr int kMaxBins = 16;

// Row-bin ladder: row r (key k > 0) goes to the first bin b with k <= limit[b],
// and at least to bin min_bin.  Rows with key 0 have an empty C row and join no
// bin.  The reference's find_bin (binning.cuh:26-35) does the same linear walk
// over its RANGES tables (parameters.cuh:53-64, 85-95, 127-144).
struct Ladder {
    int32_t nb;
    int32_t min_bin;
    int32_t limit[kMaxBins];
};

// Results of a binning pass, mirrored to pinned host memory in one copy.
struct Plan {
    int64_t total_key;        // sum of keys (total NIP, or total nnz)
    int32_t max_key;          // max key over rows
    int32_t overflow;         // a sum left int32 range
    int32_t bin_size[kMaxBins];
    int32_t bin_off[kMaxBins];
    int64_t entries;          // NIP pass: A's entries in these rows (A may be a row range)
};

// Everything a per-bin kernel needs.  Values are passed as void* and cast by
// the typed launcher.
struct ProductArgs {
    const int32_t* a_rpt;
    const int32_t* a_col;
    const void* a_val;
    const int32_t* b_rpt;
    const int32_t* b_col;
    const void* b_val;
    int32_t n_cols;         // B.n
    int32_t* c_rpt;         // NIP / nnz per row (symbolic) or row pointer (fill)
    int32_t* c_col;
    void* c_val;
    DevStatus* status;
    const int32_t* rows;    // this bin's rows
    int32_t nrows;
    // global-bin scratch: nmaps bitmaps of `words` 32-bit words each
    uint32_t* bitmaps;
    int64_t words;
    int32_t nmaps;
    // cluster bins
    int32_t cluster;        // CTAs per cluster
    int32_t* fail_rows;     // rows that spilled out of a cluster table
    int32_t* fail_count;
    // transpose: a 32-bit position in A per entry of T, and the row of A of each
    // entry of A; n_cols and words are then T's rows and entries
    uint32_t* keys;
    const int32_t* tr_row;
    // one-pass fill: c_rpt gives each row a slot of its NIP entries (an upper
    // bound); the kernel writes the row's exact nnz here (nullptr: c_rpt is
    // C's exact row pointer)
    int32_t* row_nnz;
    // one-pass fill: the entries of each row's slot, where the slots are not
    // in row order (nullptr: c_rpt[row + 1] - c_rpt[row]).  It may be row_nnz
    // itself: a row is read and then written by the one kernel that fills it.
    const int32_t* row_slot;
    // column-window bins: the bitmap's words and the sums of a row, and the
    // list of the rows that did not fit (launch_win_spill*)
    int32_t win_words;
    int32_t win_cap;
    int32_t* win_rows;
    int32_t* win_count;
    // SMs of the device (persistent kernels size their grid by it; 0: 148)
    int32_t sm_count;
    // persistent bins: a device counter the CTAs take their next row from
    // (the launcher zeroes it; nullptr: rows dealt out by CTA index)
    int32_t* work;
};

enum class BinKind : int { Team = 0, Cta = 1, Cluster = 2, Global = 3 };

struct BinLauncher {
    BinKind kind;
    int32_t limit;          // largest key the kernel accepts
    int32_t rows_per_cta;   // 1 for CTA/cluster/global kinds
    int32_t threads;
    size_t smem;            // dynamic shared memory per CTA
    const char* name;
    cudaError_t (*launch)(const ProductArgs&, cudaStream_t);
    int32_t win_words;      // column-window bins (ProductArgs' fields)
    int32_t win_cap;
};

// One-pass fill (no count phase) when its temporaries, NIP entries of column
// and value, fit this many bytes and the product has at least kOnePassMinNip
// intermediate products, kOnePassMinNipUnsampled where the compression sample
// did not run (its rows are then hashed, not sorted).  One pass against two,
// whole calls, FP64, us.  Sampled: power-law 13,000 rows at exponent 2.3 (NIP 89 k)
// 141 against 236, 8,000 at 2.0 (211 k) 142 / 240, 30,000 at 2.3 (208 k) 144 / 255;
// uniform 4,500 x 8 (288 k) 80 / 104, 2,000 x 20 (800 k) 105 / 159.  Not sampled,
// forced: power-law 10,000 at 2.3 (73 k) 192 / 228, 5,000 at 2.0 (112 k) 227 / 228;
// uniform 1,000 x 8 (64 k) 86 / 96, 4,096 x 8 (262 k) 89 / 99: one pass, hashing
// too, takes 82-100 % there; the line for it has not been moved.
constexpr uint64_t kOnePassMaxBytes = uint64_t(4) << 30;
constexpr int64_t kOnePassMinNip = int64_t(1) << 16;
constexpr int64_t kOnePassMinNipUnsampled = int64_t(1) << 21;
// Symbolic count ladder (key = NIP of the row).
int sym1_ladder(const BinLauncher** out);
// Fused fill + sort + numeric ladder (key = nnz of the row), per value type.
int s2n_ladder_f64(const BinLauncher** out);
int s2n_ladder_f32(const BinLauncher** out);
// The same for B.n <= kBitmapCols, whose large rows use a shared-memory bitmap.
constexpr int kBitmapCols = 1 << 20;
// The wide ladder's cluster bitmap bin holds up to this many columns (8 CTAs
// of kBitmapCols); past it its rows run in the global bitmap bin.
constexpr int64_t kClusterBitmapCols = int64_t(8) * kBitmapCols;
int s2n_bitmap_ladder_f64(const BinLauncher** out);
int s2n_bitmap_ladder_f32(const BinLauncher** out);
// Expanding, sorting and compressing packs a column, a product's place and, in
// the warp bins, a row into one 32-bit key: B.n up to this.
constexpr int kEscCols = 1 << 22;
// One-pass ladder (key = NIP of the row): its warp, team and 256-thread bins
// expand, sort and compress, for B.n <= kEscCols; its last two are the bitmap
// ladder's bitmap and global bins, for B.n <= kBitmapCols.  Same limits as the
// bitmap ladder and as the wide ladder's first five bins.
int s2n_esc_ladder_f64(const BinLauncher** out);
int s2n_esc_ladder_f32(const BinLauncher** out);
// The one-pass ladder's largest team bin when its split is kEscSplit
// (rows of at most kEscSplit products: a smaller kernel, more CTAs per SM).
const BinLauncher* s2n_esc_split_bin_f64();
const BinLauncher* s2n_esc_split_bin_f32();
// The 256-thread bin's kernels where its rows come in lists by size: rows of
// at most kEscCtaSmall products on 128 threads (which = 0; half the fixed cost
// of each radix pass and scan, twice the CTAs per SM: 1M power-law product, the
// bin 0.233 -> 0.223 ms serialised), of at most kEscCtaMid on 256 with eight
// keys a thread (which = 4; fewer registers: 20-product batch 1.22 -> 1.16 ms,
// 1M power-law 0.992 -> 0.986), the others on 256 with twelve (which = 1).
constexpr int kEscCtaSmall = 1024;
constexpr int kEscCtaMid = 2048;
// which = 2, 3: a wide B's one-pass rows of up to 12,288 products (1,024
// threads), and above (the bitmap bin over ranges of columns).
const BinLauncher* s2n_esc_cta_f64(int which);
const BinLauncher* s2n_esc_cta_f32(int which);

// Column-window bins (k_win.cu): rows whose columns lie inside `words` * 32
// columns of B, with at most `cap` distinct ones, a team of `lanes` lanes each.
constexpr int kWinMaxWords = 2048;
BinLauncher win_fill_bin(int value_bytes, int lanes, int words, int cap);
BinLauncher win_count_bin(int lanes, int words);
// A thread per row of at most kThreadCap columns (others join the same list),
// for at least kThreadRows rows and B.n <= kThreadCols.
constexpr int kThreadCap = 16;
constexpr int kThreadRows = 1 << 16;
constexpr int32_t kThreadCols = int32_t(1) << 26;
BinLauncher thread_fill_bin(int value_bytes);
cudaError_t win_prepare();
// The rows that did not fit (their number is on the device), by hashing: counts
// of rows of up to 3,072 products, fills of rows of up to 3,072 entries.
cudaError_t launch_win_spill_count(const ProductArgs& p, cudaStream_t s);
cudaError_t launch_win_spill_f64(const ProductArgs& p, cudaStream_t s);
cudaError_t launch_win_spill_f32(const ProductArgs& p, cudaStream_t s);

// Sampled compression of the first kEscBins fill bins of a one-pass product:
// the NIP and exact nnz of up to `samples` rows spread evenly over A, summed
// per team bin (rows binned by NIP with `lim`; rows above the last limit are
// only counted in nip_above).  `p` needs A, B and the status word.
constexpr int kEscBins = 4;
constexpr int kEscSamples = 2048;  // (4,096 took the SMs from the NIP pass beside it)
// A team bin expands, sorts and compresses when its sampled NIP / nnz is at
// most this (ESC sorts NIP keys where the hash bin sorts nnz; measured
// crossovers: none up to NIP/nnz 4 for rows of <= 48 products, ~1.45 at
// <= 192, ~1.1 at <= 768).
constexpr double kEscMaxRatio[kEscBins] = {8.0, 8.0, 1.4, 1.1};
// The one-pass ladder's bins that may expand-sort-compress: the team bins and
// the 256-thread bin, which follows the sample of the largest team bin.
constexpr int kEscLadderBins = kEscBins + 1;
// The sample runs for products with more than 2^15 entries in A: a smaller
// product's phases take about as long as the sample, ~20 us.
constexpr int64_t kSampleMinNnz = (int64_t(1) << 15) + 1;
// Products with at least this many entries in A are expected to run one pass:
// they are binned for the fill right after the NIP pass, before the first
// synchronisation (the count binning follows only if they run two).
constexpr int64_t kEarlyOnePassNnz = kSampleMinNnz;
// Auto mode keeps two passes when at least this share of the sampled NIP
// lies in rows above the team bins (one pass bins them by NIP into the CTA
// bins, two passes by nnz into small team tables) and the team bins' sampled
// NIP / nnz is at least kTwoPassMinRatio.
constexpr double kTwoPassMinShare = 0.5;
constexpr double kTwoPassMinRatio = 4.0;
struct EscLimits {
    int32_t limit[kEscBins];
};
struct EscSample {
    int64_t nip[kEscBins];
    int64_t nnz[kEscBins];
    int64_t nip_seen;   // NIP of every sampled row (A-row length for rows
    int64_t nip_above;  // longer than the last limit), and of those above it
    int32_t split;      // written by launch_esc_decide
    int32_t pad;
    // the same sums over more of the rows' products (see k_esc_sample), the
    // sampled rows and their widest column span, with one class more: rows
    // past the last team bin, up to kSampleMaxNip products
    int64_t all_nip[kEscBins + 1];
    int64_t all_nnz[kEscBins + 1];
    int64_t row_nip[kEscBins + 1];
    int64_t rows[kEscBins + 1];
    int32_t span[kEscBins + 1];
    // the most columns of a sampled row whose count ended inside a long B row
    // (an upper bound; 0: no such row): the ratios say little about it
    int32_t cols[kEscBins + 1];
};
constexpr int kSampleMaxNip = 3072;
cudaError_t launch_esc_sample(const ProductArgs& p, int32_t m, int32_t samples,
                              const EscLimits& lim, EscSample* out, cudaStream_t s);
// The fill binning's limits, decided on the device from the sample: when the
// largest team bin expands, sorts and compresses (esc_mode 1, or 0 and its
// sampled NIP/nnz at most kEscMaxRatio), its rows above kEscSplit products
// go to the 256-thread bin (which then expands, sorts and compresses too):
// out = base with limit[kEscBins - 1] = kEscSplit, and sample->split = 1.
constexpr int32_t kEscSplit = 512;
cudaError_t launch_esc_decide(EscSample* sample, const Ladder& base, int esc_mode, Ladder* out,
                              cudaStream_t s);
// One-time per-device attribute setup (dynamic smem opt-in) for all kernels.
cudaError_t sym1_prepare();
cudaError_t s2n_prepare();

// ---- binning / scan kernels (k_bin.cu) ------------------------------------
constexpr int kBinThreads = 256;
constexpr int kBinRowsPerCta = 1024;

inline int bin_ctas(int32_t m) { return (m + kBinRowsPerCta - 1) / kBinRowsPerCta; }

// Pass 1 (key = NIP): writes nip[r] into c_rpt[r] (and nip_copy[r] when not
// nullptr), per-CTA bin histograms and the plan's total / max.  With `fill`
// given, also the per-CTA histograms by that ladder into hist_fill and the
// per-CTA NIP sums into cta_sum (the fill binning's first pass).
cudaError_t launch_nip_hist(const int32_t* a_rpt, const int32_t* a_col, const int32_t* b_rpt,
                            int32_t m, int32_t* c_rpt, int32_t* nip_copy, int32_t* hist,
                            Plan* plan, DevStatus* st, const Ladder& lad, cudaStream_t s,
                            int32_t* hist_fill = nullptr, int64_t* cta_sum = nullptr,
                            const Ladder* fill = nullptr);
// Pass 2 for histograms src_hist counted by a source ladder `src` whose
// limits include every limit of the final ladder (dlad when given, else lad):
// the outputs of launch_bin_offsets for the final ladder, all bins at once,
// except that hist (another array) receives offsets within each bin: the
// scatter that reads them is launched with bin_relative.
cudaError_t launch_bin_offsets_map(const int32_t* src_hist, int32_t* hist, int32_t nctas,
                                   const Ladder& src, int64_t* cta_sum, Plan* plan,
                                   const Ladder& lad, const Ladder* dlad, cudaStream_t s);
// Append binning, one launch a pass (rows into per-bin lists: bin b's rows at
// lists[b * stride ...], stride >= m, their number in plan->bin_size[b]; the
// plan zeroed by the caller receives the keys' total and max).  Used up to
// kAppendMaxRows rows: the lists take kListBins words a row (lists.hpp).
constexpr int32_t kAppendMaxRows = int32_t(1) << 22;
constexpr int kListBins = 12;
static_assert(kListBins <= kMaxBins, "a list per bin");
// key = NIP, written to c_rpt; off (or nullptr) receives each row's slot start
cudaError_t launch_nip_append(const int32_t* a_rpt, const int32_t* a_col, const int32_t* b_rpt,
                              int32_t m, int32_t* c_rpt, int32_t* off, int32_t* lists,
                              int64_t stride, Plan* plan, DevStatus* st, const Ladder& lad,
                              cudaStream_t s);
// keys in memory
cudaError_t launch_key_append(const int32_t* keys, int32_t m, int32_t* off, int32_t* lists,
                              int64_t stride, Plan* plan, const Ladder& lad, cudaStream_t s);
// launch_rpt_scan1 (below) that also appends the rows, keyed by their counts
cudaError_t launch_rpt_scan_append(int32_t* cnt, int32_t m, unsigned long long* state, Plan* plan,
                                   DevStatus* st, int32_t* lists, int64_t stride,
                                   const Ladder& lad, cudaStream_t s);
// Pass 1' (key = nnz already in c_rpt): per-CTA sums and bin histograms.
// dlad: limits chosen on the device (same bin count as lad), or nullptr.
cudaError_t launch_nnz_hist(const int32_t* c_rpt, int32_t m, int32_t* hist, int64_t* cta_sum,
                            Plan* plan, const Ladder& lad, cudaStream_t s,
                            const Ladder* dlad = nullptr);
// Pass 2: exclusive offsets of the per-CTA histograms (and of cta_sum when
// given), bin sizes/offsets into the plan.
cudaError_t launch_bin_offsets(int32_t* hist, int32_t nctas, int64_t* cta_sum, Plan* plan,
                               const Ladder& lad, cudaStream_t s);
// Pass 3: stable scatter of row ids into bins.  When `scan` is set, also
// rewrites c_rpt[0..m] as the exclusive scan of the nnz it holds.
cudaError_t launch_bin_scatter(int32_t* c_rpt, int32_t m, const int32_t* hist_off,
                               const int64_t* cta_off, int32_t* bins, const Plan* plan,
                               const Ladder& lad, bool scan, cudaStream_t s,
                               const Ladder* dlad = nullptr, bool bin_relative = false);
// One-pass row pointer: rewrite cnt[0..m) (each row's nnz) as its exclusive
// scan and cnt[m] as the total, in place, in one launch (tiles chained by
// decoupled look-back); the plan (zeroed by the caller) receives the total,
// the max and the int32 overflow flag.  state holds 1 + rpt_scan_tiles(m)
// zeroed words (a ticket counter, then one per tile); a look-back that waits
// too long reports kStWait in st.  Used for rpt_scan_tiles(m) <=
// kScanMaxTiles (the size of the state in the scratch).
constexpr int kScanTile = 4096;
constexpr int kScanAppendTile = 1024;  // of the scan that also appends
constexpr int kScanMaxTiles = 4096;
static_assert(kAppendMaxRows <= int64_t(kScanAppendTile) * kScanMaxTiles, "scan state");
inline int rpt_scan_tiles(int32_t m) { return (m + kScanTile - 1) / kScanTile; }
cudaError_t launch_rpt_scan1(int32_t* cnt, int32_t m, unsigned long long* state, Plan* plan,
                             DevStatus* st, cudaStream_t s);
// One-pass fill: copy each row's entries from its slot [off[r], ...) of the
// temporary arrays to [rpt[r], rpt[r+1]) of C (values of value_bytes 4 or 8);
// nothing at or past `cap`, C's capacity.
cudaError_t launch_compact_rows(const int32_t* off, const int32_t* rpt, int32_t m,
                                const int32_t* tmp_col, const void* tmp_val, int32_t* col,
                                void* val, int value_bytes, cudaStream_t s, int32_t cap);
// A one-pass C gets the product's NIP as its capacity before its nnz is known
// when the sampled rows' NIP / nnz is at most this; a C with more spare
// capacity than this factor is then copied to arrays of its size.
constexpr double kCapSlack = 1.1;
// `bytes` (a multiple of 4) to page-locked host memory, then *flag = seq there.
cudaError_t launch_publish(const void* src, size_t bytes, void* dst, unsigned long long* flag,
                           unsigned long long seq, cudaStream_t s);
// Operand validation (checked mode).
cudaError_t launch_check_csr(const int32_t* rpt, const int32_t* col, int32_t m, int32_t n,
                             int32_t nnz, DevStatus* st, cudaStream_t s);
// Batched form (k_batch.cu): NIP per product; per-product split of a group's C.
cudaError_t launch_product_nip(const int32_t* a_rpt, const int32_t* a_col, const int32_t* b_rpt,
                               const int32_t* row_off, int32_t count, long long* nip,
                               cudaStream_t s);
cudaError_t launch_unpack(const int32_t* c_rpt, int32_t* c_col, const int32_t* row_off,
                          const int32_t* col_off, const int64_t* out_off, int32_t first,
                          int32_t count, int32_t rows, int32_t nnz, int32_t* rpt_out,
                          int32_t* pos_out, cudaStream_t s);
// CSR transpose (k_transpose.cu): row-sort ladder (key = length of a row of
// A^T), column counts with each entry's rank in its column, and the scatter.
int transpose_ladder_f64(const BinLauncher** out);
int transpose_ladder_f32(const BinLauncher** out);
cudaError_t transpose_prepare();
cudaError_t launch_col_count(const int32_t* col, int32_t nnz, int32_t n, int32_t* cnt,
                             int32_t* rank, cudaStream_t s);
// perm: the entries' positions by T's rows; row_of: the entries' rows of A
cudaError_t launch_tr_scatter(const int32_t* a_rpt, const int32_t* a_col, int32_t m, int32_t nnz,
                              const int32_t* t_rpt, const int32_t* rank, uint32_t* perm,
                              int32_t* row_of, cudaStream_t s);
// NIP of many independent pairs in one launch (spgemm_get_nip_many).
struct NipPair {
    const int32_t* a_col;   // A_i's column indices (nnz entries)
    const int32_t* b_rpt;   // B_i's row pointer
    int32_t nnz;            // nnz(A_i)
    int32_t pad;
};
int32_t pairs_nip_ctas(int32_t nnz);  // CTAs the launch gives one pair
cudaError_t launch_pairs_nip(const NipPair* pairs, const int32_t* cta_off, int32_t count,
                             int32_t ctas, long long* nip, cudaStream_t s);
// Total NIP only (spgemm_get_nip).
cudaError_t launch_total_nip(const int32_t* a_rpt, const int32_t* a_col, const int32_t* b_rpt,
                             int32_t m, long long* out, cudaStream_t s);

}  // namespace b200
