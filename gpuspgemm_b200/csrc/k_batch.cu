// Kernels of the batched form: many independent products C_i = A_i * B_i run
// as one product of block-diagonal operands (see spgemm_batch_* in spgemm.cu).
#include "cta.cuh"
#include "kernels.hpp"

namespace b200 {
namespace {

constexpr int kBatchThreads = 256;

// NIP of every product i: sum over its rows r in [row_off[i], row_off[i+1])
// of A of sum_{k in A(r,:)} len(B(k,:)).  gridDim.y CTAs per product, each
// with every gridDim.y-th slice of its entries, adding to nip[i] (zeroed by
// the caller): few large products still fill the chip.
__global__ __launch_bounds__(kBatchThreads) void k_product_nip(
    const int32_t* __restrict__ a_rpt, const int32_t* __restrict__ a_col,
    const int32_t* __restrict__ b_rpt, const int32_t* __restrict__ row_off,
    unsigned long long* __restrict__ nip) {
    __shared__ long long s_part[kBatchThreads / kWarp];
    const int i = blockIdx.x;
    const int r0 = row_off[i];
    const int r1 = row_off[i + 1];
    const int e0 = a_rpt[r0];
    const int e1 = a_rpt[r1];
    const long long stride = static_cast<long long>(gridDim.y) * kBatchThreads;
    long long s = 0;
    for (long long e = e0 + static_cast<long long>(blockIdx.y) * kBatchThreads + threadIdx.x;
         e < e1; e += stride) {
        const int c = __ldg(a_col + e);
        s += __ldg(b_rpt + c + 1) - __ldg(b_rpt + c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long t = 0;
        for (int w = 0; w < kBatchThreads / kWarp; w++) t += s_part[w];
        if (t != 0) atomicAdd(nip + i, static_cast<unsigned long long>(t));
    }
}

// Split a group's C into per-product CSR: product i (rows [r0, r1) of the
// group's C, local row 0 at r0) gets its own row pointer starting at 0 in
// rpt_out + out_off[i], and its columns are shifted back to local indices in
// place.  Bound by memory: C.col is read and written once, so the work is cut
// by entries and rows, not by products (one CTA per product left 20 products
// of 1.4 M entries on 20 SMs: 4.9 ms; by entries 0.04 ms).  The first row_ctas
// CTAs take kUnpackRows rows each, the others kUnpackEntries entries each; a
// CTA finds its first product by a 32-way search.
constexpr int kUnpackRows = 2048;
constexpr int kUnpackEntries = 4096;

// The last i in [lo, hi) with start(i) <= x, by one warp (start(lo) <= x).
template<typename F>
__device__ __forceinline__ int warp_last_le(int lo, int hi, int x, F&& start) {
    const int lane = threadIdx.x & 31;
    while (hi - lo > 1) {  // uniform over the warp
        const int step = (hi - lo + kWarp - 1) / kWarp;
        const long long at = lo + static_cast<long long>(lane) * step;
        const unsigned le = __ballot_sync(0xffffffffu, at < hi && start(static_cast<int>(at)) <= x);
        lo += (31 - __clz(le)) * step;
        hi = min(lo + step, hi);
    }
    return lo;
}

__global__ __launch_bounds__(kBatchThreads) void k_unpack(
    const int32_t* __restrict__ c_rpt, int32_t* __restrict__ c_col,
    const int32_t* __restrict__ row_off, const int32_t* __restrict__ col_off,
    const int64_t* __restrict__ out_off, int32_t first, int32_t count, int32_t row_ctas,
    int32_t nnz, int32_t* __restrict__ rpt_out, int32_t* __restrict__ pos_out) {
    __shared__ int32_t s_first;
    const int tid = threadIdx.x;
    const int last = first + count;
    const int base_row = row_off[first];
    const int rows = row_off[last] - base_row;
    auto entry_start = [&](int i) { return c_rpt[row_off[i] - base_row]; };
    if (static_cast<int>(blockIdx.x) < row_ctas) {
        // per product: its place in C and its row pointer's last word
        for (int i = first + blockIdx.x * kBatchThreads + tid; i < last;
             i += row_ctas * kBatchThreads) {
            const int p0 = entry_start(i);
            const int n = entry_start(i + 1) - p0;
            pos_out[2 * i] = p0;
            pos_out[2 * i + 1] = n;
            rpt_out[out_off[i] + (row_off[i + 1] - row_off[i])] = n;
        }
        const int t0 = blockIdx.x * kUnpackRows;
        const int t1 = rows - t0 < kUnpackRows ? rows : t0 + kUnpackRows;
        if (t0 >= t1) return;  // uniform over the CTA
        if (tid < kWarp) {
            const int i = warp_last_le(first, last, base_row + t0,
                                       [&](int k) { return row_off[k]; });
            if (tid == 0) s_first = i;
        }
        __syncthreads();
        int i = s_first;
        for (int t = t0 + tid; t < t1; t += kBatchThreads) {
            while (row_off[i + 1] - base_row <= t) i++;  // empty products are passed over
            rpt_out[out_off[i] + (t - (row_off[i] - base_row))] = c_rpt[t] - entry_start(i);
        }
        return;
    }
    const int p0 = (blockIdx.x - row_ctas) * kUnpackEntries;
    const int p1 = nnz - p0 < kUnpackEntries ? nnz : p0 + kUnpackEntries;
    if (tid < kWarp) {
        const int i = warp_last_le(first, last, p0, entry_start);
        if (tid == 0) s_first = i;
    }
    __syncthreads();
    int i = s_first;
    int end = entry_start(i + 1);
    int shift = col_off[i];
    if (end >= p1 && p1 - p0 == kUnpackEntries) {  // one product, a whole chunk: 16 bytes a load
        int4* c4 = reinterpret_cast<int4*>(c_col + p0);
#pragma unroll
        for (int k = 0; k < kUnpackEntries / 4 / kBatchThreads; k++) {
            int4 v = c4[k * kBatchThreads + tid];
            v.x -= shift;
            v.y -= shift;
            v.z -= shift;
            v.w -= shift;
            c4[k * kBatchThreads + tid] = v;
        }
        return;
    }
    for (long long p = p0 + tid; p < p1; p += kBatchThreads) {
        if (end <= p) {
            while (entry_start(i + 1) <= p) i++;
            end = entry_start(i + 1);
            shift = col_off[i];
        }
        c_col[p] -= shift;
    }
}

// NIP of many independent pairs (A_i, B_i) in one launch: pair i's A entries
// are cut into chunks of kNipChunk, one CTA per chunk (cta_off[i] is pair i's
// first CTA); each CTA sums len(B_i(k,:)) over its entries and adds the total
// to nip[i] (zeroed by the caller) with one atomic.
constexpr int kNipChunk = 16384;

__global__ __launch_bounds__(kBatchThreads) void k_pairs_nip(const NipPair* __restrict__ pairs,
                                                            const int32_t* __restrict__ cta_off,
                                                            int32_t count,
                                                            long long* __restrict__ nip) {
    __shared__ long long s_part[kBatchThreads / kWarp];
    const int b = blockIdx.x;
    // the pair this CTA belongs to: the last i with cta_off[i] <= b
    int lo = 0;
    int hi = count;  // cta_off[count] > b
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (cta_off[mid] <= b) lo = mid;
        else hi = mid;
    }
    const NipPair pr = pairs[lo];
    const int e0 = (b - cta_off[lo]) * kNipChunk;
    const int e1 = min(e0 + kNipChunk, pr.nnz);
    long long s = 0;
    for (int e = e0 + threadIdx.x; e < e1; e += kBatchThreads) {
        const int c = __ldg(pr.a_col + e);
        s += __ldg(pr.b_rpt + c + 1) - __ldg(pr.b_rpt + c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long t = 0;
        for (int w = 0; w < kBatchThreads / kWarp; w++) t += s_part[w];
        atomicAdd(reinterpret_cast<unsigned long long*>(nip + lo),
                  static_cast<unsigned long long>(t));
    }
}

}  // namespace

int32_t pairs_nip_ctas(int32_t nnz) { return (nnz + kNipChunk - 1) / kNipChunk; }

cudaError_t launch_pairs_nip(const NipPair* pairs, const int32_t* cta_off, int32_t count,
                             int32_t ctas, long long* nip, cudaStream_t s) {
    if (ctas <= 0) return cudaSuccess;
    k_pairs_nip<<<ctas, kBatchThreads, 0, s>>>(pairs, cta_off, count, nip);
    return cudaGetLastError();
}

cudaError_t launch_product_nip(const int32_t* a_rpt, const int32_t* a_col, const int32_t* b_rpt,
                               const int32_t* row_off, int32_t count, long long* nip,
                               cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    if (cudaError_t e = cudaMemsetAsync(nip, 0, sizeof(long long) * static_cast<size_t>(count), s);
        e != cudaSuccess)
        return e;
    // about eight CTAs per SM over all products
    const int per = 148 * 8 / count;
    const dim3 grid(count, per < 1 ? 1 : per > 64 ? 64 : per);
    k_product_nip<<<grid, kBatchThreads, 0, s>>>(a_rpt, a_col, b_rpt, row_off,
                                                 reinterpret_cast<unsigned long long*>(nip));
    return cudaGetLastError();
}

cudaError_t launch_unpack(const int32_t* c_rpt, int32_t* c_col, const int32_t* row_off,
                          const int32_t* col_off, const int64_t* out_off, int32_t first,
                          int32_t count, int32_t rows, int32_t nnz, int32_t* rpt_out,
                          int32_t* pos_out, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    const int row_ctas = rows > 0 ? (rows - 1) / kUnpackRows + 1 : 1;
    const int col_ctas = nnz > 0 ? (nnz - 1) / kUnpackEntries + 1 : 0;
    k_unpack<<<row_ctas + col_ctas, kBatchThreads, 0, s>>>(c_rpt, c_col, row_off, col_off, out_off,
                                                           first, count, row_ctas, nnz, rpt_out,
                                                           pos_out);
    return cudaGetLastError();
}

}  // namespace b200
