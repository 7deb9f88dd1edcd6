// CSR transpose T = A^T with sorted columns in every row of T.
//
// The reference has no transpose: its Galerkin use (R = P^T for R*A*P) leaves
// the transpose to the caller.  Here it is a library call so that a chained
// product stays on the device:
//   1. column counts of A (warp-aggregated atomics) into T.rpt; the atomic's
//      old value is the entry's rank in its column, kept per entry (in T.col,
//      which nothing else needs yet);
//   2. the product path's binning pass with the scan (k_bin.cu) turns the
//      counts into T.rpt and bins T's rows by length;
//   3. scatter: entry (i, j) of A at position e puts e at place T.rpt[j] + rank
//      and i at row_of[e];
//   4. each row's positions are put in ascending order -- A's entries are in
//      row order, so that is the order of the rows i, and of equal ones by
//      position -- and T.col = row_of[e], T.val = A.val[e] written: rows of up to
//      kTrFlat entries by counting, per entry, the row's smaller positions;
//      longer rows by sorting.
// Bound by random 32-byte sectors: per entry an atomic, a 4-byte write and two
// 4- or 8-byte gathers.  The write is 4 bytes so that its array stays in L2 until
// its sectors are whole: with 16-byte records (key and value, no gathers) the
// scatter of 5.5 M entries took 0.152 ms and 85 MB of DRAM reads to fill partly
// written sectors.  Entries are dealt to lanes flat (a warp per row of A left
// most lanes idle at 5.5 entries a row, and took a second atomic per entry).
// Sorting uses the bitonic network in which every comparator sends the
// smaller key to the lower index; a row of len keys runs the network of the
// next power of two with the missing tail taken as +infinity, and every
// comparator that touches the tail is a no-op, so the tail is never stored.
#include "cta.cuh"
#include "kernels.hpp"

namespace b200 {

namespace {

__device__ __forceinline__ void cas_asc(uint32_t* a, long long lo, long long hi) {
    const uint32_t x = a[lo];
    const uint32_t y = a[hi];
    if (x > y) {
        a[lo] = y;
        a[hi] = x;
    }
}

// Ascending sort of a[0, len) by the CTA (a in shared or global memory).
template<int THREADS>
__device__ void cta_sort_keys(uint32_t* a, long long len) {
    long long N = 1;
    while (N < len) N <<= 1;
    const long long pairs = N >> 1;
    for (long long k = 2; k <= N; k <<= 1) {
        const long long half = k >> 1;
        // flip: i <-> k-1-i inside every block of k
        for (long long p = threadIdx.x; p < pairs; p += THREADS) {
            const long long blk = (p / half) * k;
            const long long i = p & (half - 1);
            const long long hi = blk + k - 1 - i;
            if (hi < len) cas_asc(a, blk + i, hi);
        }
        __syncthreads();
        for (long long j = half >> 1; j > 0; j >>= 1) {
            for (long long p = threadIdx.x; p < pairs; p += THREADS) {
                const long long lo = 2 * p - (p & (j - 1));
                if (lo + j < len) cas_asc(a, lo, lo + j);
            }
            __syncthreads();
        }
    }
}

// One entry of T at `at`: A's entry e.
template<typename V>
__device__ __forceinline__ void store_entry(const ProductArgs& p, int32_t at, uint32_t e) {
    p.c_col[at] = __ldg(p.tr_row + e);
    static_cast<V*>(p.c_val)[at] = __ldg(static_cast<const V*>(p.a_val) + e);
}

// ---- 1. column counts and ranks ---------------------------------------------
// rank[e] = entry e's place among its column's entries, in the order of the
// atomics (any order: step 4 sorts).  A column index outside [0, n) is not
// counted and its rank is -1; the host sees the total fall short of nnz and
// reports the operand as invalid.  kCountUnroll atomics per lane in flight.
// Bound by L2 atomics that return a value: 5.5 M in 0.051 ms, with lanes of one
// column grouped by __match_any_sync (as here, for hot columns) or not.
constexpr int kCountUnroll = 4;

__global__ __launch_bounds__(256) void k_col_count(const int32_t* __restrict__ col, int32_t nnz,
                                                   int32_t n, int32_t* __restrict__ cnt,
                                                   int32_t* __restrict__ rank) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x * kCountUnroll;
    // the loop bound is warp-uniform, so every lane joins each match
    for (long long base = (static_cast<long long>(blockIdx.x) * blockDim.x +
                           (threadIdx.x & ~31)) * kCountUnroll;
         base < nnz; base += stride) {
        int32_t c[kCountUnroll];
        int32_t first[kCountUnroll];
        unsigned peers[kCountUnroll];
#pragma unroll
        for (int u = 0; u < kCountUnroll; u++) {
            const long long e = base + u * kWarp + lane;
            c[u] = e < nnz ? __ldg(col + e) : -1;
            if (c[u] >= n) c[u] = -1;
        }
#pragma unroll
        for (int u = 0; u < kCountUnroll; u++) {
            peers[u] = __match_any_sync(0xffffffffu, c[u]);
            first[u] = 0;
            if (c[u] >= 0 && (peers[u] & below) == 0u)
                first[u] = atomicAdd(cnt + c[u], __popc(peers[u]));
        }
#pragma unroll
        for (int u = 0; u < kCountUnroll; u++) {
            const long long e = base + u * kWarp + lane;
            const int r = __shfl_sync(0xffffffffu, first[u], __ffs(peers[u]) - 1) +
                          __popc(peers[u] & below);
            if (e < nnz) rank[e] = c[u] >= 0 ? r : -1;
        }
    }
}

// ---- 3. scatter of positions --------------------------------------------------
// A warp takes kScatterTile consecutive entries of A, finds the rows of the
// first and the last by a 32-way search of A.rpt, and each lane finds its
// entries' rows by a binary search between them.  Entries whose column is
// outside [0, n) were not ranked and are skipped.
constexpr int kScatterPer = 8;
constexpr int kScatterTile = kWarp * kScatterPer;

// The last r in [0, m) with rpt[r] <= e, by one warp (rpt[0] <= e, m >= 1).
__device__ __forceinline__ int warp_row_of(const int32_t* __restrict__ rpt, int32_t m, int32_t e) {
    const int lane = threadIdx.x & 31;
    int lo = 0;
    int hi = m;
    while (hi - lo > 1) {  // uniform over the warp
        const int step = (hi - lo + kWarp - 1) / kWarp;
        const long long at = lo + static_cast<long long>(lane) * step;
        const unsigned le =
            __ballot_sync(0xffffffffu, lane == 0 || (at < hi && __ldg(rpt + at) <= e));
        // the true lanes are a prefix for a valid row pointer
        const int last = 31 - __clz(le);
        lo += last * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

__global__ __launch_bounds__(256) void k_tr_scatter(const int32_t* __restrict__ a_rpt,
                                                    const int32_t* __restrict__ a_col, int32_t m,
                                                    int32_t nnz,
                                                    const int32_t* __restrict__ t_rpt,
                                                    const int32_t* __restrict__ rank,
                                                    uint32_t* __restrict__ perm,
                                                    int32_t* __restrict__ row_of) {
    const int lane = threadIdx.x & 31;
    const long long tile = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) +
                           (threadIdx.x >> 5);
    const long long e0 = tile * kScatterTile;
    if (e0 >= nnz) return;  // uniform over the warp
    const int e1 = static_cast<int>(min(e0 + kScatterTile, static_cast<long long>(nnz))) - 1;
    const int rlo = warp_row_of(a_rpt, m, static_cast<int>(e0));
    const int rhi = warp_row_of(a_rpt, m, e1);
    int pos[kScatterPer];
#pragma unroll
    for (int k = 0; k < kScatterPer; k++) {
        const long long e = e0 + k * kWarp + lane;
        pos[k] = -1;
        if (e <= e1) {
            const int r = __ldg(rank + e);
            if (r >= 0) pos[k] = __ldg(t_rpt + __ldg(a_col + e)) + r;
        }
    }
#pragma unroll
    for (int k = 0; k < kScatterPer; k++) {
        const int e = static_cast<int>(e0 + k * kWarp + lane);
        if (pos[k] < 0) continue;
        perm[pos[k]] = static_cast<uint32_t>(e);
        int lo = rlo;
        for (int len = rhi - rlo + 1; len > 1;) {
            const int half = len >> 1;
            lo = __ldg(a_rpt + lo + half) <= e ? lo + half : lo;
            len -= half;
        }
        row_of[e] = lo;
    }
}

// ---- 4. the rows' entries in order ---------------------------------------------
// Rows of up to kTrFlat entries: a warp takes rows_per_warp consecutive rows of
// T and walks their entries flat, a lane per entry; the entry's place in its
// row is the number of smaller positions there (one broadcast read per entry of
// the row, most from L1: cheaper than a warp's sorting network for the short
// rows of a graph).  It runs over all rows and leaves the longer ones to their
// bins' kernels.
constexpr int kTrFlat = 128;

template<typename V>
__global__ __launch_bounds__(256) void k_tr_place(ProductArgs p, int32_t rows_per_warp) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t* __restrict__ perm = reinterpret_cast<const uint32_t*>(p.keys);
    const long long r0 = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) +
                          (threadIdx.x >> 5)) * rows_per_warp;
    if (r0 >= p.n_cols) return;  // uniform over the warp
    int t0 = 0;
    int len = 0;
    if (lane < rows_per_warp && r0 + lane < p.n_cols) {
        t0 = __ldg(p.c_rpt + r0 + lane);
        len = __ldg(p.c_rpt + r0 + lane + 1) - t0;
        if (len > kTrFlat) len = 0;
    }
    const int inc = team_inclusive_scan<kWarp>(kFull, len, lane);
    const int total = __shfl_sync(kFull, inc, 31);
    for (int f0 = 0; f0 < total; f0 += kWarp) {  // uniform over the warp
        const int f = f0 + lane;
        // entry f's row: the first lane with inc > f
        int j = -1;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const int v = __shfl_sync(kFull, inc, (j + step) & 31);
            if (v <= f) j += step;
        }
        j = (j + 1) & 31;
        const int start = __shfl_sync(kFull, t0, j);
        const int before = __shfl_sync(kFull, inc - len, j);
        const int count = __shfl_sync(kFull, len, j);
        if (f < total) {
            const uint32_t mine = __ldg(perm + start + (f - before));
            const int32_t row = __ldg(p.tr_row + mine);
            const V val = __ldg(static_cast<const V*>(p.a_val) + mine);
            int place = 0;
#pragma unroll 4
            for (int i = 0; i < count; i++) place += __ldg(perm + start + i) < mine;
            p.c_col[start + place] = row;
            static_cast<V*>(p.c_val)[start + place] = val;
        }
    }
}

// Rows of up to CAP keys: one CTA per row, the keys in shared memory.
template<typename V, int THREADS, int CAP>
__global__ __launch_bounds__(THREADS) void k_tr_sort_cta(ProductArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* s = reinterpret_cast<uint32_t*>(smem_raw);
    const int row = p.rows[blockIdx.x];
    const int t0 = p.c_rpt[row];
    const int len = p.c_rpt[row + 1] - t0;
    if (len > CAP) {  // routed by its length: cannot happen
        if (threadIdx.x == 0) report(p.status, kStCapacity, row, len);
        return;
    }
    for (int i = threadIdx.x; i < len; i += THREADS) s[i] = reinterpret_cast<const uint32_t*>(p.keys)[t0 + i];
    __syncthreads();
    cta_sort_keys<THREADS>(s, len);
    for (int i = threadIdx.x; i < len; i += THREADS) store_entry<V>(p, t0 + i, s[i]);
}

// Longer rows: one CTA per row, sorting the row's positions in place in global
// memory (the network's passes stay in L2 for rows of a few MB).
template<typename V, int THREADS>
__global__ __launch_bounds__(THREADS) void k_tr_sort_global(ProductArgs p) {
    for (int rid = blockIdx.x; rid < p.nrows; rid += gridDim.x) {
        const int row = p.rows[rid];
        const int t0 = p.c_rpt[row];
        const int len = p.c_rpt[row + 1] - t0;
        uint32_t* a = reinterpret_cast<uint32_t*>(p.keys) + t0;
        cta_sort_keys<THREADS>(a, len);
        for (int i = threadIdx.x; i < len; i += THREADS) store_entry<V>(p, t0 + i, a[i]);
        __syncthreads();
    }
}

// Rows per warp of k_tr_place for about kPlaceEntries entries a warp.
constexpr int64_t kPlaceEntries = 256;

// Every row of T, not only this bin's list: the list would cost a gather per
// row, and the rows of other bins only a row-pointer read.
template<typename V>
cudaError_t launch_place(const ProductArgs& p, cudaStream_t s) {
    const int32_t n = p.n_cols;  // rows of T
    const int64_t nnz = p.words; // entries of T
    int rows = 1;
    while (rows < kWarp && (2 * rows) * nnz <= kPlaceEntries * n) rows *= 2;
    const int64_t warps = (static_cast<int64_t>(n) + rows - 1) / rows;
    k_tr_place<V><<<static_cast<unsigned>((warps + 7) / 8), 256, 0, s>>>(p, rows);
    return cudaGetLastError();
}

template<typename V, int THREADS, int CAP>
cudaError_t launch_cta(const ProductArgs& p, cudaStream_t s) {
    k_tr_sort_cta<V, THREADS, CAP><<<p.nrows, THREADS, sizeof(uint32_t) * CAP, s>>>(p);
    return cudaGetLastError();
}

template<typename V, int THREADS>
cudaError_t launch_global(const ProductArgs& p, cudaStream_t s) {
    const int grid = p.nrows < 2 * 148 ? p.nrows : 2 * 148;
    k_tr_sort_global<V, THREADS><<<grid, THREADS, 0, s>>>(p);
    return cudaGetLastError();
}

template<typename V>
struct TransposeLadder {
    static const BinLauncher bins[4];
};

template<typename V>
const BinLauncher TransposeLadder<V>::bins[4] = {
    {BinKind::Team, kTrFlat, 8, 256, 0, "tr_place", launch_place<V>},
    {BinKind::Cta, 2048, 1, 256, sizeof(uint32_t) * 2048, "tr_sort_cta2048",
     launch_cta<V, 256, 2048>},
    {BinKind::Cta, 16384, 1, 1024, sizeof(uint32_t) * 16384, "tr_sort_cta16384",
     launch_cta<V, 1024, 16384>},
    {BinKind::Global, INT32_MAX, 1, 1024, 0, "tr_sort_global", launch_global<V, 1024>},
};

template<typename V>
cudaError_t prepare_ladder() {
    cudaError_t e = cudaFuncSetAttribute(k_tr_sort_cta<V, 1024, 16384>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(uint32_t) * 16384));
    return e;
}

}  // namespace

int transpose_ladder_f64(const BinLauncher** out) {
    *out = TransposeLadder<double>::bins;
    return 4;
}

int transpose_ladder_f32(const BinLauncher** out) {
    *out = TransposeLadder<float>::bins;
    return 4;
}

cudaError_t transpose_prepare() {
    cudaError_t e = prepare_ladder<double>();
    if (e != cudaSuccess) return e;
    return prepare_ladder<float>();
}

cudaError_t launch_col_count(const int32_t* col, int32_t nnz, int32_t n, int32_t* cnt,
                             int32_t* rank, cudaStream_t s) {
    if (nnz <= 0) return cudaSuccess;
    long long g = (static_cast<long long>(nnz) + 256 * kCountUnroll - 1) / (256 * kCountUnroll);
    if (g > 148 * 16) g = 148 * 16;
    k_col_count<<<static_cast<int>(g), 256, 0, s>>>(col, nnz, n, cnt, rank);
    return cudaGetLastError();
}

cudaError_t launch_tr_scatter(const int32_t* a_rpt, const int32_t* a_col, int32_t m, int32_t nnz,
                              const int32_t* t_rpt, const int32_t* rank, uint32_t* perm,
                              int32_t* row_of, cudaStream_t s) {
    if (m <= 0 || nnz <= 0) return cudaSuccess;
    constexpr int kPerCta = 8 * kScatterTile;
    const unsigned g = static_cast<unsigned>((static_cast<long long>(nnz) + kPerCta - 1) / kPerCta);
    k_tr_scatter<<<g, 256, 0, s>>>(a_rpt, a_col, m, nnz, t_rpt, rank, perm, row_of);
    return cudaGetLastError();
}

}  // namespace b200
