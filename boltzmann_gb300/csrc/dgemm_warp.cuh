// FP64 matrix products of the 1D3V steps: C = A B with a warp per 32 columns x R rows.
//
// GB300's FP64 pipe takes a sub-partition 64 cycles per warp instruction, so a product is bound by
// how evenly its multiply-adds spread over the 4 x 152 sub-partitions, not by its operands: a lane
// keeps one column of R rows in registers, B is read coalesced (one load for R multiply-adds), A
// uniformly from L1, and nothing is staged. R is chosen so that the warps fill whole rounds of the
// GPU (dgw_rows). Each element sums over k in order.
#pragma once
#include <algorithm>
#include <type_traits>
#include "bte_common.cuh"

constexpr int DGW_WARPS = 4;          // warps per CTA: one per sub-partition
constexpr int DGW_RMAX = 12;
constexpr int DGW_SLOTS = 4 * 152;    // sub-partitions

// rows per warp: fewest rounds x rows over the GPU's sub-partitions; the larger R on a tie (it reads B less)
inline int dgw_rows(int M, int N) {
    const long long cg = (N + 31) / 32;
    long long best = -1;
    int r = 1;
    for (int R = 1; R <= DGW_RMAX; ++R) {
        const long long warps = (long long)((M + R - 1) / R) * cg;
        const long long cost = ((warps + DGW_SLOTS - 1) / DGW_SLOTS) * R;
        if (best < 0 || cost <= best) {
            best = cost;
            r = R;
        }
    }
    return r;
}
inline unsigned dgw_grid(int M, int N, int R) {
    const long long warps = (long long)((M + R - 1) / R) * ((N + 31) / 32);
    return (unsigned)((warps + DGW_WARPS - 1) / DGW_WARPS);
}

// acc[i] = sum_k A[i0 + i][k] B[k][col] (TA: A stored transposed, A[k * lda + row]); rows past M repeat
// the last one. With one warp on a sub-partition nothing else hides a load, so they run ahead: A by
// chunks of 32 k (a lane per k, through the warp's shared memory sA: 32 R doubles, read back as
// broadcasts), B by U columns' worth of registers.
template <int R, bool TA>
__device__ inline void dgw_product(int M, int K, const double* __restrict__ A, int lda, const double* __restrict__ B,
                                   long long ldb, int i0, int col, double acc[R], double* sA) {
    constexpr int U = R <= 2 ? 16 : 8;
    const int lane = threadIdx.x & 31;
    const double* b = B + col;
    double an[R], nb[U];
    auto fetch_a = [&](int k0) {
        const int k = min(k0 + lane, K - 1);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = min(i0 + i, M - 1);
            an[i] = TA ? A[(size_t)k * lda + r] : A[(size_t)r * lda + k];
        }
    };
    auto fetch_b = [&](int k0) {
#pragma unroll
        for (int u = 0; u < U; ++u) nb[u] = b[(size_t)min(k0 + u, K - 1) * ldb];
    };
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.0;
    if (K <= 0) return;
    fetch_a(0);
    fetch_b(0);
    for (int k0 = 0; k0 < K; k0 += 32) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < R; ++i) sA[lane * R + i] = an[i];
        __syncwarp();
        if (k0 + 32 < K) fetch_a(k0 + 32);
#pragma unroll
        for (int q = 0; q < 32; q += U) {
            if (k0 + q >= K) break;
            double bv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) bv[u] = nb[u];
            if (k0 + q + U < K) fetch_b(k0 + q + U);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k0 + q + u < K)
#pragma unroll
                    for (int i = 0; i < R; ++i) acc[i] += sA[(q + u) * R + i] * bv[u];
        }
    }
}
// the warp's part of the CTA's buffer
template <int R>
__device__ inline double* dgw_buffer() {
    __shared__ __align__(16) double sA[DGW_WARPS][32 * R];
    return sA[threadIdx.x >> 5];
}

// the row group and column of this lane; false for the warps past the end. Consecutive warps take
// consecutive row groups of one column group, so a CTA reads the same B.
__device__ inline bool dgw_place(int M, int N, int R, int* i0, int* col) {
    const int ng = (M + R - 1) / R, cg = (N + 31) / 32;
    const int w = blockIdx.x * DGW_WARPS + (threadIdx.x >> 5);
    *i0 = (w % ng) * R;
    *col = (w / ng) * 32 + (threadIdx.x & 31);
    return w < ng * cg;
}

// run f(std::integral_constant<int, R>) for the runtime R
template <class F>
inline void dgw_dispatch(int R, F&& f) {
    switch (R) {
        case 1: f(std::integral_constant<int, 1>{}); break;
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 3: f(std::integral_constant<int, 3>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        case 7: f(std::integral_constant<int, 7>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 9: f(std::integral_constant<int, 9>{}); break;
        case 10: f(std::integral_constant<int, 10>{}); break;
        case 11: f(std::integral_constant<int, 11>{}); break;
        default: f(std::integral_constant<int, 12>{}); break;
    }
}
