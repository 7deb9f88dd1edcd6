// What the fill kernels share.
#pragma once

#include "common.cuh"
#include "kernels.hpp"

namespace b200 {

constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x >> 1); }

template<typename V>
__device__ __forceinline__ V ldv(const void* base, int i) {
    return __ldg(static_cast<const V*>(base) + i);
}

// Entries of a row's slot at c0: its exact nnz, or in one-pass mode its NIP.
__device__ __forceinline__ int slot_entries(const ProductArgs& p, int row, int c0) {
    return p.row_slot != nullptr ? p.row_slot[row] : p.c_rpt[row + 1] - c0;
}

}  // namespace b200
