// Sort of atoms by cell, stable: atoms of a cell in the order of their index. A counting sort: atoms count themselves into
// their cells (k_*_keys of the callers, arrival order), a scan over the cells gives the cell starts, cell_place lists the
// atoms of each cell in arrival order, and whoever reads the list ranks an atom among the few of its cell (cell_slot).
//
// Against a radix sort of (cell, index) pairs: two light passes instead of a histogram and three heavy ones, and the cell
// starts come with it. What bounds it: launches and atomics to L2 (small systems), scattered 4-byte writes (large ones).
// The ranking is quadratic in the atoms of a cell, as the neighbour search behind it is.
#pragma once

#include <cuda_runtime.h>

#include "dsmd_launch.cuh"

namespace dsmd {

// Thread t of `threads`. Atoms [first, end); key, arrival by atom, list by slot. And the counts of `cells` cells, which the scan has
// read, go back to zero for the next sort.
__device__ __forceinline__ void cell_place(int t, int threads, int first, int end, const unsigned* key, const int* arrival,
                                           const int* cell_start, int* __restrict__ list, int cells, int* __restrict__ cell_count) {
    const int i = first + t;
    if (i < end) list[cell_start[key[i]] + arrival[i]] = i;
    for (int k = t; k < cells; k += threads) cell_count[k] = 0;
}

// Final slot of the atom `a` of cell `cell`.
__device__ __forceinline__ int cell_slot(int a, unsigned cell, const int* cell_start, const int* list) {
    const int begin = cell_start[cell], end = cell_start[cell + 1];
    int slot = begin;
    for (int k = begin; k < end; ++k) slot += list[k] < a ? 1 : 0;
    return slot;
}

}  // namespace dsmd
