// Shapes and size classes of the tridiagonal reduction on chip (kernels: trd.cuh, compiled in trd.cu).
#pragma once
#include <cuda_runtime.h>

namespace axg {

constexpr int TRD_THREADS = 256;
constexpr int TRD_SMEM_MAX = 227 * 1024;

// shared memory of one CTA (doubles): v (two buffers), w, reduction slots and barriers; cluster: the
// pairs (row element, y entry) received from all CTAs (two buffers) and the CTA's own pairs; grid: the
// row groups' partial y; then 32 rows of the register columns, and the other columns
__host__ __device__ constexpr int trd_stride(int n) { return (n + 31) & ~31; }
__host__ __device__ constexpr int trd_slots(int n, int G, int TC) { return ((n + G - 1) / G + TC - 1) / TC; }
__host__ __device__ constexpr int trd_smem_cols(int n, int G, int TC, int CR) {
    return trd_slots(n, G, TC) > CR ? (trd_slots(n, G, TC) - CR) * TC : 0;
}
__host__ __device__ constexpr int trd_ylen(int n, int G, int TC) { return trd_slots(n, G, TC) * TC; }
__host__ __device__ constexpr long long trd_smem_doubles(int n, int G, int AW, int CR, bool grid) {
    return (long long)trd_stride(n) * (grid ? 3 : 7) + 48 + (grid ? AW : 2) * trd_ylen(n, G, 8 / AW) +
           32LL * CR * (8 / AW) + (grid ? trd_ylen(n, G, 8 / AW) : 0) + (long long)trd_smem_cols(n, G, 8 / AW, CR) * trd_stride(n);
}

// ---- size classes: row slots per thread and register columns per warp (row group)
struct TrdClass {
    int rt, cr;
    const void* fn;
    const void* teams;  // whole grid: the kernel for several molecules at once (nullptr: sizes that need every CTA)
};
// The class of an n x n matrix on clusters of G CTAs (0: the class that says how many it takes), and on
// the whole grid; nullptr: none.
const TrdClass* trd_class(int n, int G = 0);
const TrdClass* trd_grid_class(int n);
constexpr int TRD_CLUSTER_MAX_NAO = 32 * 24;

}  // namespace axg
