// Column-window kernels: count and fill of rows that repeat their columns inside
// a narrow window of B's columns (a stencil's square, a Galerkin product).
//
// A team of G lanes per row of C.  The row's window [lo, hi] comes from the
// first and last columns of the B rows it reads (sorted rows); a bitmap of the
// window in shared memory, one bit per column, replaces the hash table:
//   1. walk the A entries, one B row after another, G columns at a time, and
//      set the columns' bits: no probing, no compare-and-swap;
//   2. the words' running counts, kept beside the words, give every column its
//      place in the sorted row: no sort;
//   3. (fill) walk again, write each product's column at its place and add the
//      product to the sum there, in shared memory.  A B row's columns are distinct, so the lanes
//      of a team never meet in a place and the sums need no atomics; every
//      entry is summed in the oracle's (Gustavson) order, each product rounded
//      before it is added.
// A row whose window is wider than the bitmap, whose columns outnumber the
// sums, or with a column outside its window (an unsorted B row) goes to the
// fail list, which a hash kernel takes afterwards.
//
// What bounds it: instruction issue.  The hash bins spent it on probing (lanes
// wait for the longest of 27 probe sequences), on a search per product for its
// A entry and, in the fill, on a binary search and a global atomic per product.
// G follows the mean length of the B rows read (a step takes one B row).
// Measured (B200): a 27-point stencil on 60^3 squared, FP32, 149 M products:
// hash bin 1.49 ms -> window fill 0.82 ms (71 % issue-active, 3,100 warp
// instructions a row); R * (A * P) on 100^3: count 0.19 -> 0.08 ms, fill 0.31 ->
// 0.26.  A team per row with a hash table and row-by-row sums in it (no
// window) took 1.05 ms on the stencil: 6.5 probe rounds a step.
#include "cta.cuh"
#include "fill.cuh"
#include "kernels.hpp"

namespace b200 {

namespace {

constexpr int kWinAhead = 4;  // B rows loaded together

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// Bytes of one team's share of shared memory: sums, (bits, place) words,
// columns.  The shares start 2 * lanes banks apart, so that the teams of a warp
// touch different banks when they are at the same place of their shares (with
// 8 teams at equal banks, conflicts took half of the 4-lane kernel's time).
__host__ __device__ constexpr size_t win_bytes(size_t value_bytes, int words, int cap, int lanes) {
    const size_t need = value_bytes * cap + sizeof(uint2) * words + sizeof(int32_t) * cap;
    const size_t step = 2 * lanes % 32 * sizeof(int32_t);
    return (need + 127) / 128 * 128 + (step == 0 ? 0 : step);
}
__host__ __device__ constexpr size_t win_count_bytes(int words, int lanes) {
    return (sizeof(uint32_t) * words + 127) / 128 * 128 + lanes % 32 * sizeof(int32_t);
}

constexpr unsigned kFull = 0xffffffffu;

// Walk each team's A entries [a0, a1) one B row after another and call
// use(column, product, valid) for every G columns of a B row.  The warp's teams
// stay together: the loops run to the longest of their rows, so every shuffle
// and barrier takes the full mask (partial masks cost a warp-sync each).  The
// loads are staged so that none waits for one issued just before it: the A
// entries' columns two chunks of G entries ahead, their B rows' bounds one
// chunk ahead, the B rows kWinAhead at a time one group ahead.
template<int G, bool VALUES, typename V, typename F>
__device__ __forceinline__ void walk_rows(const ProductArgs& p, int a0, int a1, int lane,
                                          F&& use) {
    constexpr int kGroups = G / kWinAhead;  // groups of B rows per chunk of G entries
    static_assert(G % kWinAhead == 0, "a chunk holds whole groups");
    const int most = __reduce_max_sync(kFull, a1 - a0);
    const int groups = (most + kWinAhead - 1) / kWinAhead;
    if (groups == 0) return;  // uniform over the warp
    auto column = [&](int e) { return e < a1 ? __ldg(p.a_col + e) : -1; };
    auto bounds = [&](int k, int e, int& bs, int& len, V& av) {
        len = 0;
        if (k >= 0) {
            bs = __ldg(p.b_rpt + k);
            len = __ldg(p.b_rpt + k + 1) - bs;
            if constexpr (VALUES) av = ldv<V>(p.a_val, e);
        }
    };
    struct Group {
        int32_t col[kWinAhead];
        V prod[kWinAhead];
        int len[kWinAhead];
    };
    int mbs = 0, mlen = 0, nbs = 0, nlen = 0;  // this chunk's bounds, the next one's
    V mav = V(0), nav = V(0);
    int e = a0 + lane;  // this lane's entry of the chunk after next
    const int k0 = column(e);
    const int k1 = column(e + G);
    int k2 = column(e + 2 * G);
    bounds(k0, e, mbs, mlen, mav);
    bounds(k1, e + G, nbs, nlen, nav);
    e += 2 * G;
    auto load = [&](int g, Group& x) {
        if (g > 0 && g % kGroups == 0) {  // into the next chunk
            mbs = nbs;
            mlen = nlen;
            mav = nav;
            bounds(k2, e, nbs, nlen, nav);
            e += G;
            k2 = column(e);
        }
#pragma unroll
        for (int u = 0; u < kWinAhead; u++) {
            const int src = (g % kGroups) * kWinAhead + u;
            const int bs = __shfl_sync(kFull, mbs, src, G);
            x.len[u] = __shfl_sync(kFull, mlen, src, G);
            V av = V(0);
            if constexpr (VALUES) av = __shfl_sync(kFull, mav, src, G);
            if (lane < x.len[u]) {
                x.col[u] = __ldg(p.b_col + bs + lane);
                if constexpr (VALUES) x.prod[u] = mul_rn(av, ldv<V>(p.b_val, bs + lane));
            }
        }
    };
    Group cur;
    load(0, cur);
    for (int g = 0; g < groups; g++) {  // uniform over the warp
        Group next;
        if (g + 1 < groups) load(g + 1, next);
        int longest = 0;
#pragma unroll
        for (int u = 0; u < kWinAhead; u++) longest = max(longest, cur.len[u]);
        if (!__any_sync(kFull, longest > G)) {
#pragma unroll
            for (int u = 0; u < kWinAhead; u++) use(cur.col[u], cur.prod[u], lane < cur.len[u]);
        } else {  // with the rest of long B rows
#pragma unroll
            for (int u = 0; u < kWinAhead; u++) {
                use(cur.col[u], cur.prod[u], lane < cur.len[u]);
                int bs = 0;
                V av = V(0);
                if (cur.len[u] > G) {
                    const int at = a0 + g * kWinAhead + u;
                    bs = __ldg(p.b_rpt + __ldg(p.a_col + at));
                    if constexpr (VALUES) av = ldv<V>(p.a_val, at);
                }
                const int end = __reduce_max_sync(kFull, cur.len[u]);
                for (int i = G + lane; i - lane < end; i += G) {
                    const bool ok = i < cur.len[u];
                    int32_t c = 0;
                    V v = V(0);
                    if (ok) {
                        c = __ldg(p.b_col + bs + i);
                        if constexpr (VALUES) v = mul_rn(av, ldv<V>(p.b_val, bs + i));
                    }
                    use(c, v, ok);
                }
            }
        }
        cur = next;
    }
}

// Steps 1 and 2's counting for the warp's rows, a team's each: sets the
// window's bits and returns the number of columns, or -1 when the row does not
// fit.  lo: the window's first column (a multiple of 32); words: its words;
// run: the words per lane of the counting (odd, against bank conflicts);
// before: the columns in the words of the lanes below.
struct WinRow {
    int lo;
    int words;
    int run;
    int before;
};

// STEP: 32-bit words from one bitmap word to the next.
template<int G, int STEP>
__device__ __forceinline__ int win_columns(const ProductArgs& p, int a0, int a1, int lane,
                                           uint32_t* bm, WinRow& w) {
    int lo = INT32_MAX;
    int hi = -1;
    for (int e = a0 + lane; e < a1; e += G) {
        const int k = __ldg(p.a_col + e);
        const int s0 = __ldg(p.b_rpt + k);
        const int s1 = __ldg(p.b_rpt + k + 1);
        if (s0 < s1) {
            lo = min(lo, __ldg(p.b_col + s0));
            hi = max(hi, __ldg(p.b_col + s1 - 1));
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(kFull, lo, o, G));
        hi = max(hi, __shfl_xor_sync(kFull, hi, o, G));
    }
    // no products, not sorted, or wider than the bitmap
    bool fits = hi >= lo && lo >= 0 && hi < p.n_cols && (hi >> 5) - (lo >> 5) < p.win_words;
    w.lo = lo & ~31;
    w.words = fits ? (hi >> 5) - (lo >> 5) + 1 : 0;
    for (int i = lane; i < w.words; i += G) bm[i * STEP] = 0u;
    __syncwarp();
    bool miss = false;
    const unsigned span = static_cast<unsigned>(w.words) * 32u;
    walk_rows<G, false, float>(p, a0, fits ? a1 : a0, lane, [&](int32_t col, float, bool valid) {
        const unsigned at = static_cast<unsigned>(col) - static_cast<unsigned>(w.lo);
        if (valid && at < span) atomicOr(bm + (at >> 5) * STEP, 1u << (at & 31u));
        miss = miss || (valid && at >= span);
    });
    __syncwarp();
    const unsigned missed = __ballot_sync(kFull, miss);
    fits = fits && (missed & team_mask<G>()) == 0u;
    w.run = ((w.words + G - 1) / G) | 1;
    int cnt = 0;
    for (int i = lane * w.run, e = min(i + w.run, w.words); i < e; i++)
        cnt += __popc(bm[i * STEP]);
    const int inc = team_inclusive_scan<G>(kFull, cnt, lane);
    w.before = inc - cnt;
    const int total = __shfl_sync(kFull, inc, G - 1, G);
    return fits ? total : -1;
}

__device__ __forceinline__ void win_fail(const ProductArgs& p, int row, int lane) {
    if (lane == 0) p.win_rows[atomicAdd(p.win_count, 1)] = row;
}

template<int G>
__global__ __launch_bounds__(256) void k_win_count(ProductArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int team = threadIdx.x / G;
    const int lane = team_lane<G>();
    const int rid = blockIdx.x * (blockDim.x / G) + team;
    const bool mine = rid < p.nrows;  // a team past the list walks no entries
    uint32_t* bm =
        reinterpret_cast<uint32_t*>(smem_raw + team * win_count_bytes(p.win_words, G));
    const int row = mine ? p.rows[rid] : 0;
    const int a0 = mine ? p.a_rpt[row] : 0;
    const int a1 = mine ? p.a_rpt[row + 1] : 0;
    WinRow w;
    const int cnt = win_columns<G, 1>(p, a0, a1, lane, bm, w);
    if (!mine) return;
    if (cnt < 0) win_fail(p, row, lane);
    else if (lane == 0) p.c_rpt[row] = cnt;
}

// Four CTAs an SM: FP64 took 79 registers without the bound, three CTAs (R * AP
// of a 100^3 stencil 0.308 -> 0.264 ms); five spill FP32 (60^3 squared 0.82 ->
// 0.93 ms).
template<typename V, int G>
__global__ __launch_bounds__(256, 4) void k_win_fill(ProductArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int team = threadIdx.x / G;
    const int lane = team_lane<G>();
    const int rid = blockIdx.x * (blockDim.x / G) + team;
    const bool mine = rid < p.nrows;  // a team past the list walks no entries
    unsigned char* share = smem_raw + team * win_bytes(sizeof(V), p.win_words, p.win_cap, G);
    uint2* word = reinterpret_cast<uint2*>(share);  // (bits, place of the first)
    V* vals = reinterpret_cast<V*>(word + p.win_words);
    int32_t* cols = reinterpret_cast<int32_t*>(vals + p.win_cap);
    const int row = mine ? p.rows[rid] : 0;
    const int c0 = mine ? p.c_rpt[row] : 0;
    const int a0 = mine ? p.a_rpt[row] : 0;
    const int a1 = mine ? p.a_rpt[row + 1] : 0;
    WinRow w;
    const int cnt = win_columns<G, 2>(p, a0, a1, lane, &word->x, w);
    const int bound = mine ? slot_entries(p, row, c0) : 0;  // its exact nnz, or its NIP
    const bool fits = cnt >= 0 && cnt <= p.win_cap && cnt <= bound;
    if (fits) {
        for (int i = lane; i < cnt; i += G) vals[i] = V(0);
        unsigned at = w.before;
        for (int i = lane * w.run, e = min(i + w.run, w.words); i < e; i++) {
            word[i].y = at;
            at += __popc(word[i].x);
        }
    }
    __syncwarp();
    walk_rows<G, true, V>(p, a0, fits ? a1 : a0, lane, [&](int32_t col, V prod, bool valid) {
        if (valid) {
            const unsigned x = static_cast<unsigned>(col) - static_cast<unsigned>(w.lo);
            const uint2 at = word[x >> 5];
            const unsigned r = at.y + __popc(at.x & ((1u << (x & 31u)) - 1u));
            cols[r] = col;
            vals[r] += prod;
        }
        __syncwarp();  // the next B row may hold the same columns in other lanes
    });
    if (!mine) return;
    if (!fits) {
        win_fail(p, row, lane);
        return;
    }
    int32_t* out_col = p.c_col + c0;
    V* out_val = static_cast<V*>(p.c_val) + c0;
    for (int i = lane; i < cnt; i += G) {
        out_col[i] = cols[i];
        out_val[i] = vals[i];
    }
    if (lane == 0) {
        if (p.row_nnz != nullptr) p.row_nnz[row] = cnt;
        else if (cnt != bound) report(p.status, kStCapacity, row, cnt);
    }
}

// Rows of few columns that many products fall on (A * P of a multigrid setup: 81
// products, 9 columns): a thread per row, with a list of columns and sums and a
// hash table of list places (one byte each) of its own.  Word i of lane l lies
// at i * 32 + l, so every lane keeps to its own bank whatever it probes, and
// nothing needs an atomic; 64 byte-wide places for at most 16 columns keep the
// lanes of a warp from waiting for one lane's probes.  Neighbouring rows of a
// mesh read neighbouring B rows, so the lanes' reads of B stay close; their A
// entries do not (27 entries apart), so the warp reads its rows' entries and
// their B-row bounds together, kThreadStage entries a row at a time, four rows
// a load, and hands them over through shared memory (a lane's own loads, 32
// lines each, bound the kernel).  1M rows of a 100^3 A * P, FP64: 4-lane hash
// teams 1.1 ms, window teams 1.06, this kernel 0.81 with the lanes' own loads,
// 0.69 with the shared ones; the planned 64^3 A * P 0.242 -> 0.158 ms.
// Sums in Gustavson order, as the window kernels'; the columns are sorted by
// insertion at the end.
constexpr int kThreadPlaces = 64;
constexpr int kThreadLog = 6;
constexpr int kThreadAhead = 4;  // B entries of a row loaded together
constexpr int kThreadStage = 8;
constexpr int kThreadPitch = kThreadStage + 1;  // odd: a lane's entries in banks of its own
constexpr int kThreadBlock = 128;
static_assert(kThreadCap <= 16, "a list place and its sort key's four bits");

template<typename V>
constexpr size_t thread_bytes() {
    return ((sizeof(V) + sizeof(int32_t)) * kThreadCap + kThreadPlaces +
            (sizeof(int2) + sizeof(V)) * kThreadPitch) * kThreadBlock;
}

template<typename V>
__global__ __launch_bounds__(kThreadBlock) void k_thread_fill(ProductArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr size_t kWarpBytes = thread_bytes<V>() / (kThreadBlock / kWarp);
    const int lane = threadIdx.x & 31;
    unsigned char* share = smem_raw + (threadIdx.x >> 5) * kWarpBytes;
    V* vals = reinterpret_cast<V*>(share) + lane;
    share += sizeof(V) * kThreadCap * kWarp;
    int2* stage_b = reinterpret_cast<int2*>(share);  // (start, length) of B rows
    share += sizeof(int2) * kThreadPitch * kWarp;
    V* stage_v = reinterpret_cast<V*>(share);
    share += sizeof(V) * kThreadPitch * kWarp;
    int32_t* keys = reinterpret_cast<int32_t*>(share) + lane;
    uint32_t* table = reinterpret_cast<uint32_t*>(share + sizeof(int32_t) * kThreadCap * kWarp) + lane;
    const int rid = blockIdx.x * kThreadBlock + threadIdx.x;
    const bool mine = rid < p.nrows;
    const int row = mine ? p.rows[rid] : 0;
    const int c0 = mine ? p.c_rpt[row] : 0;
    const int a0 = mine ? p.a_rpt[row] : 0;
    const int a1 = mine ? p.a_rpt[row + 1] : 0;
#pragma unroll
    for (int i = 0; i < kThreadPlaces / 4; i++) table[i * kWarp] = 0u;
    int cnt = 0;  // kThreadCap + 1: too many columns
    auto add = [&](int32_t col, V prod) {
        unsigned h = (static_cast<uint32_t>(col) * 0x9E3779B1u) >> (32 - kThreadLog);
        for (;;) {  // ends: at most kThreadCap of the places are taken
            unsigned char* at = reinterpret_cast<unsigned char*>(table + (h >> 2) * kWarp) + (h & 3u);
            const int i = static_cast<int>(*at) - 1;
            if (i < 0) {  // a new column
                if (cnt < kThreadCap) {
                    keys[cnt * kWarp] = col;
                    vals[cnt * kWarp] = prod;
                    *at = static_cast<unsigned char>(++cnt);
                } else {
                    cnt = kThreadCap + 1;
                }
                return;
            }
            if (keys[i * kWarp] == col) {
                vals[i * kWarp] += prod;
                return;
            }
            h = (h + 1) & (kThreadPlaces - 1);
        }
    };
    // lane (r, j) of load t handles entry j of row 4 t + r of the warp
    constexpr int kLoads = kThreadStage;  // 32 rows * kThreadStage entries / 32 lanes
    const int sr = lane / kThreadStage;
    const int sj = lane % kThreadStage;
    static_assert(kWarp % kThreadStage == 0 && kWarp / kThreadStage * kLoads == kWarp, "loads");
    int32_t k[kLoads];
    auto columns = [&](int base) {
#pragma unroll
        for (int t = 0; t < kLoads; t++) {
            const int r = t * (kWarp / kThreadStage) + sr;
            const int e = __shfl_sync(kFull, a0, r) + base + sj;
            k[t] = e < __shfl_sync(kFull, a1, r) ? __ldg(p.a_col + e) : -1;
        }
    };
    struct Products {
        int32_t col[kThreadAhead];
        V val[kThreadAhead];
    };
    auto products = [&](const int2& b, Products& y) {
#pragma unroll
        for (int u = 0; u < kThreadAhead; u++) {
            if (u < b.y) {
                y.col[u] = __ldg(p.b_col + b.x + u);
                y.val[u] = ldv<V>(p.b_val, b.x + u);
            }
        }
    };
    const int most = __reduce_max_sync(kFull, a1 - a0);
    columns(0);
    for (int base = 0; base < most; base += kThreadStage) {  // uniform over the warp
        __syncwarp();  // the entries staged before are used up
#pragma unroll
        for (int t = 0; t < kLoads; t++) {
            const int r = t * (kWarp / kThreadStage) + sr;
            const int e = __shfl_sync(kFull, a0, r) + base + sj;
            int2 b = make_int2(0, 0);
            if (k[t] >= 0) {
                b.x = __ldg(p.b_rpt + k[t]);
                b.y = __ldg(p.b_rpt + k[t] + 1) - b.x;
                stage_v[r * kThreadPitch + sj] = ldv<V>(p.a_val, e);
            }
            stage_b[r * kThreadPitch + sj] = b;
        }
        __syncwarp();
        columns(base + kThreadStage);
        int2 b0 = stage_b[lane * kThreadPitch];
        Products p0;
        products(b0, p0);
#pragma unroll 1  // (eight copies of the five inserts miss the instruction cache)
        for (int j = 0; j < kThreadStage; j++) {
            int2 b1 = make_int2(0, 0);
            Products p1;
            if (j + 1 < kThreadStage) {
                b1 = stage_b[lane * kThreadPitch + j + 1];
                products(b1, p1);
            }
            const V av = stage_v[lane * kThreadPitch + j];
#pragma unroll
            for (int u = 0; u < kThreadAhead; u++)
                if (u < b0.y) add(p0.col[u], mul_rn(av, p0.val[u]));
            for (int u = kThreadAhead; u < b0.y; u++)
                add(__ldg(p.b_col + b0.x + u), mul_rn(av, ldv<V>(p.b_val, b0.x + u)));
            b0 = b1;
            p0 = p1;
        }
    }
    if (!mine) return;
    const int bound = slot_entries(p, row, c0);  // its exact nnz, or its NIP
    if (cnt > kThreadCap || cnt > bound) {
        p.win_rows[atomicAdd(p.win_count, 1)] = row;
        return;
    }
    // insertion sort of the columns, packed with their places in the list
    // (B.n <= kThreadCols)
    for (int i = 0; i < cnt; i++) {
        const int32_t k = keys[i * kWarp];
        if (static_cast<uint32_t>(k) >= static_cast<uint32_t>(p.n_cols)) {
            report(p.status, kStBadInput, row, k);
            return;
        }
        const int32_t x = (k << 4) | i;
        int at = i;
        for (; at > 0; at--) {
            const int32_t y = keys[(at - 1) * kWarp];
            if (y < x) break;
            keys[at * kWarp] = y;
        }
        keys[at * kWarp] = x;
    }
    int32_t* out_col = p.c_col + c0;
    V* out_val = static_cast<V*>(p.c_val) + c0;
    for (int i = 0; i < cnt; i++) {
        const int32_t x = keys[i * kWarp];
        out_col[i] = x >> 4;
        out_val[i] = vals[(x & 15) * kWarp];
    }
    if (p.row_nnz != nullptr) p.row_nnz[row] = cnt;
    else if (cnt != bound) report(p.status, kStCapacity, row, cnt);
}

template<typename V>
cudaError_t launch_thread(const ProductArgs& p, cudaStream_t s) {
    k_thread_fill<V><<<(p.nrows + kThreadBlock - 1) / kThreadBlock, kThreadBlock,
                       thread_bytes<V>(), s>>>(p);
    return cudaGetLastError();
}

// Threads per CTA: as many teams as leave room for two CTAs on an SM.
constexpr size_t kWinCtaBytes = 112 * 1024;

template<int G>
int win_threads(size_t team_bytes) {
    int t = 256;
    while (t > kWarp && (t / G) * team_bytes > kWinCtaBytes) t /= 2;
    return t;
}

template<int G>
cudaError_t launch_count(const ProductArgs& p, cudaStream_t s) {
    const size_t team = win_count_bytes(p.win_words, G);
    const int t = win_threads<G>(team);
    k_win_count<G><<<(p.nrows + t / G - 1) / (t / G), t, team * (t / G), s>>>(p);
    return cudaGetLastError();
}

template<typename V, int G>
cudaError_t launch_fill(const ProductArgs& p, cudaStream_t s) {
    const size_t team = win_bytes(sizeof(V), p.win_words, p.win_cap, G);
    const int t = win_threads<G>(team);
    k_win_fill<V, G><<<(p.nrows + t / G - 1) / (t / G), t, team * (t / G), s>>>(p);
    return cudaGetLastError();
}

using Launch = cudaError_t (*)(const ProductArgs&, cudaStream_t);

template<typename V>
Launch fill_of(int lanes) {
    return lanes <= 4    ? launch_fill<V, 4>
           : lanes <= 8  ? launch_fill<V, 8>
           : lanes <= 16 ? launch_fill<V, 16>
                         : launch_fill<V, 32>;
}

// Lanes for rows whose team needs team_bytes: more lanes (fewer rows in
// flight) when a warp's rows would not leave room for two CTAs.
int fit_lanes(int lanes, size_t team_bytes) {
    while (lanes < kWarp && (kWarp / lanes) * team_bytes > kWinCtaBytes) lanes *= 2;
    return lanes;
}

const char* const kFillNames[] = {"win_fill4", "win_fill8", "win_fill16", "win_fill32"};
const char* const kCountNames[] = {"win_count4", "win_count8", "win_count16", "win_count32"};
int name_of(int lanes) { return lanes <= 4 ? 0 : lanes <= 8 ? 1 : lanes <= 16 ? 2 : 3; }

template<int G>
cudaError_t prepare() {
    const int most = 232448;
    cudaError_t e = cudaFuncSetAttribute(k_win_count<G>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_win_fill<double, G>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_win_fill<float, G>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e;
}

}  // namespace

BinLauncher win_fill_bin(int value_bytes, int lanes, int words, int cap) {
    lanes = fit_lanes(lanes, win_bytes(value_bytes, words, cap, lanes));
    BinLauncher b = {};
    b.kind = BinKind::Team;
    b.limit = cap;
    b.name = kFillNames[name_of(lanes)];
    b.launch = value_bytes == 8 ? fill_of<double>(lanes) : fill_of<float>(lanes);
    b.win_words = words;
    b.win_cap = cap;
    return b;
}

BinLauncher win_count_bin(int lanes, int words) {
    lanes = fit_lanes(lanes, win_count_bytes(words, lanes));
    BinLauncher b = {};
    b.kind = BinKind::Team;
    b.limit = INT32_MAX;
    b.name = kCountNames[name_of(lanes)];
    b.launch = lanes <= 4    ? launch_count<4>
               : lanes <= 8  ? launch_count<8>
               : lanes <= 16 ? launch_count<16>
                             : launch_count<32>;
    b.win_words = words;
    return b;
}

BinLauncher thread_fill_bin(int value_bytes) {
    BinLauncher b = {};
    b.kind = BinKind::Team;
    b.limit = kThreadCap;
    b.name = "thread_fill";
    b.launch = value_bytes == 8 ? launch_thread<double> : launch_thread<float>;
    return b;
}

cudaError_t win_prepare() {
    cudaError_t e = cudaFuncSetAttribute(k_thread_fill<double>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(thread_bytes<double>()));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_thread_fill<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(thread_bytes<float>()));
    if (e == cudaSuccess) e = prepare<4>();
    if (e == cudaSuccess) e = prepare<8>();
    if (e == cudaSuccess) e = prepare<16>();
    if (e == cudaSuccess) e = prepare<32>();
    return e;
}

}  // namespace b200
