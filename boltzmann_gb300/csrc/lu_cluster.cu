// Dense FP64 LU with partial pivoting of one matrix per thread-block cluster, the matrix resident
// in the cluster's shared memory.
//
// Same contract as lu.cu (which replaces the batched inverse of bte_0d3v_batched.py:856-880):
// row-major A[r * ld + c] with NC = N or N + 1 columns, rows never exchanged in memory,
// perm[position] = stored row, info = first zero pivot (1-based), 0 if none; the pivot of a
// column is the first position of its largest |a|.
//
// Why a cluster: an SM issues 2 FP64 multiply-adds per clock, so a matrix of N = 385 needs 4.8 ms on
// one SM, and spreading it by launches (panel, triangular solve, tiles) leaves each panel on one SM
// and 3 N / 32 launches in a chain. Here the columns are dealt in blocks of CL_NB to the CTAs of
// a cluster, which keep them in shared memory from the first read to the last write (N = 385:
// 1.2 MB over 8 SMs), and one cluster barrier per block replaces the launches.
// Per block k, owned by CTA k mod C:
//   1. the owner factors it with the rows' values in the registers of a few warps (in FP64 one per
//      sub-partition, whose FP64 pipe takes 64 cycles per warp instruction): per column a search by
//      integer compares (no FP64 instruction), the pivot row through shared memory, one rank-one
//      update. Rows stay with their threads and only their positions change; the block is
//      written to shared memory at the new positions and to A;
//   2. every CTA, after the barrier, copies the block from the owner (distributed shared memory),
//      moves the (at most 2 CL_NB) displaced rows of its own later columns, solves its U rows, writes
//      them to A, and updates its columns: a warp takes 32 rows x CL_NB columns, L in registers,
//      U broadcast. The next block's owner updates that block first and factors it while its
//      other warps, and the other CTAs, are still updating: a CTA only arrives at the barrier
//      when its part of the next block is done, and waits for it after its updates.
// A column's rows above the diagonal and its own block are final when written, so A is read once
// and written once.
#include <cooperative_groups.h>
#include <cstdint>
#include <climits>
#include <algorithm>
#include "bte_common.cuh"

namespace cg = cooperative_groups;

namespace {

// Columns per block. The owner of the next block updates it alone before it factors it: with 8 columns
// that and the panel's rank-one updates took 11.5 multiply-adds per row and column of the chain, with 4 they take
// 5.5, against one more cluster barrier per 8 columns. Measured (us, 8 -> 4): N = 129: 1 matrix 217 -> 191,
// 1000 matrices 2549 -> 2448; N = 385: 1 matrix 1068 -> 923. Finer blocks also let six CTAs hold N = 385
// (16 matrices at once: 2072 -> 1425).
constexpr int CL_NB = 4;
constexpr int CL_NT = 256;     // threads per CTA
constexpr int CL_NW = CL_NT / 32;
constexpr size_t CL_SMEM_MAX = 220 * 1024;

// column pitch: 16-byte aligned columns that do not all start on one bank
__host__ __device__ inline int cl_ldr(int N) {
    const int l = (N + 3) & ~3;
    return (l % 16 == 0) ? l + 4 : l;
}
// local column blocks per CTA, and the CTA's shared memory: its columns, the current block, perm
__host__ __device__ inline int cl_blocks(int NC, int C) { return ((NC + CL_NB - 1) / CL_NB + C - 1) / C; }
__host__ __device__ inline size_t cl_smem(int N, int NC, int C, size_t w) {
    return (size_t)(cl_blocks(NC, C) + 1) * CL_NB * cl_ldr(N) * w + (size_t)N * 4;
}

constexpr int CL_PW = 4;  // warps that factor a block: one per sub-partition

struct ClShared {
    uint4 cand[2][CL_PW];               // a warp's candidate: key (high, low word), position
    double prow[2][CL_NB];              // the pivot row of the block
    double inv[2];
    int2 moved[2 * CL_NB];              // (old, new) position of a displaced row
    int nmoved;
    int info;
    int next;                           // the next update item
};

__device__ inline void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ inline void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }

// |v| as an integer that orders like it; 0 for NaN, so that a NaN is only taken when nothing else is left
__device__ inline unsigned long long cl_key(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull ? 0ull : b + 1;
}
__device__ inline void cl_load8(const double* p, double u[CL_NB]) {
#pragma unroll
    for (int i = 0; i < CL_NB; i += 2) {
        const double2 v = *reinterpret_cast<const double2*>(p + i);
        u[i] = v.x; u[i + 1] = v.y;
    }
}
// Factor block b (columns P, pitch ldr, rows k0 .. N - 1 in position order) by the first NPW warps
template <int RPL>
__device__ inline void cl_panel(ClShared& sh, double* P, int ldr, int N, int NC, int k0, int kb, const int* perm, double* a,
                                int ld) {
    constexpr int PT = 32 * CL_PW;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    auto psync = [&] { asm volatile("bar.sync 1, %0;\n" ::"n"(PT) : "memory"); };
    double v[RPL][CL_NB];
    int pos[RPL];  // the row's position; a row is done when it is before the current column
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
        const int r = k0 + tid + i * PT;
        pos[i] = (r < N) ? r : -1;
#pragma unroll
        for (int c = 0; c < CL_NB; ++c) v[i][c] = (r < N) ? P[(size_t)c * ldr + r] : 0.0;
    }
    if (tid == 0) sh.nmoved = 0;
#pragma unroll
    for (int j = 0; j < CL_NB; ++j) {
        if (j >= kb) break;
        const int q = k0 + j;
        unsigned long long key = 0;
        int at = INT_MAX;
#pragma unroll
        for (int i = 0; i < RPL; ++i)
            if (k0 + i * PT < N) {
                const unsigned long long ki = cl_key(v[i][j]);
                if (pos[i] >= q && (at == INT_MAX || ki > key || (ki == key && pos[i] < at))) { key = ki; at = pos[i]; }
            }
        // of the warp, then of the panel's warps: the largest key, the first position among equals
        auto reduce = [&](unsigned& hi, unsigned& lo, unsigned& ps) {
            const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
            const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
            ps = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? ps : (unsigned)INT_MAX);
            hi = mh;
            lo = ml;
        };
        unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key, ps = (unsigned)at;
        if (at == INT_MAX) hi = lo = 0u;
        reduce(hi, lo, ps);
        if (lane == 0) sh.cand[j & 1][w] = make_uint4(hi, lo, ps, 0u);
        psync();
        const uint4 o = sh.cand[j & 1][lane < CL_PW ? lane : 0];
        hi = o.x; lo = o.y; ps = o.z;
        reduce(hi, lo, ps);
        const int at_p = (int)ps;
        double* prow = sh.prow[j & 1];
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            if (pos[i] == at_p) {
                pos[i] = q;
                const double d = v[i][j];
#pragma unroll
                for (int c = j + 1; c < CL_NB; ++c) prow[c] = v[i][c];
                sh.inv[j & 1] = (d != 0.0) ? 1.0 / d : 0.0;
                if (!(d != 0.0) && sh.info == 0) sh.info = q + 1;
            } else if (pos[i] == q) {
                pos[i] = at_p;
            }
        }
        psync();
        double pr[CL_NB];
#pragma unroll
        for (int c = j + 1; c < CL_NB; ++c) pr[c] = prow[c];
        const double inv = sh.inv[j & 1];
#pragma unroll
        for (int i = 0; i < RPL; ++i)
            if (k0 + i * PT < N) {  // the same for all lanes; done rows keep their values
                const bool on = pos[i] > q;
                const double l = v[i][j] * inv;
                if (on) v[i][j] = l;
#pragma unroll
                for (int c = j + 1; c < CL_NB; ++c) {
                    const double x = v[i][c] - l * pr[c];
                    if (on) v[i][c] = x;
                }
            }
    }
    // the block at the new positions, to A, and the displaced rows
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
        const int r = k0 + tid + i * PT;
        if (r >= N) continue;
        double* row = a + (size_t)perm[r] * ld + k0;
#pragma unroll
        for (int c = 0; c < CL_NB; ++c) {
            P[(size_t)c * ldr + pos[i]] = v[i][c];
            if (k0 + c < NC) row[c] = v[i][c];
        }
        if (pos[i] != r) sh.moved[atomicAdd(&sh.nmoved, 1)] = make_int2(r, pos[i]);
    }
}

template <int RPL, int OCC>
__global__ void __launch_bounds__(CL_NT, OCC)
k_lu_cluster(int N, int NC, double* __restrict__ A, int ld, long long stride, int32_t* __restrict__ perm_out,
             int32_t* __restrict__ info) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ ClShared sh;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int mat = blockIdx.x / C, ldr = cl_ldr(N);
    const int nblk = (NC + CL_NB - 1) / CL_NB, nloc = (nblk - rank + C - 1) / C;  // blocks; mine
    double* S = reinterpret_cast<double*>(smraw);                        // column c of local block lb at (lb CL_NB + c) ldr
    double* Lb = S + (size_t)cl_blocks(NC, C) * CL_NB * ldr;        // the current block
    int* perm = reinterpret_cast<int*>(Lb + (size_t)CL_NB * ldr);
    double* a = A + (size_t)mat * stride;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int r = tid; r < N; r += CL_NT) perm[r] = r;
    if (tid == 0) sh.info = 0;
    for (int lb = 0; lb < nloc; ++lb) {
        const int c = tid % CL_NB, col = (rank + lb * C) * CL_NB + c;
        double* dst = S + (size_t)(lb * CL_NB + c) * ldr;
#pragma unroll 8
        for (int r = tid / CL_NB; r < N; r += CL_NT / CL_NB) dst[r] = (col < NC) ? a[(size_t)r * ld + col] : 0.0;
    }
    __syncthreads();
    if (rank == 0 && w < CL_PW) cl_panel<RPL>(sh, S, ldr, N, NC, 0, min(CL_NB, N), perm, a, ld);
    __syncwarp();
    cl_arrive();
    for (int b = 0; b * CL_NB < N; ++b) {
        const int k0 = b * CL_NB, kb = min(CL_NB, N - k0), owner = b % C;
        cl_wait();
        // the block and the displaced rows
        const ClShared* os = cluster.map_shared_rank(&sh, owner);
        const int nm = os->nmoved;
        const int2 mv = os->moved[lane % (2 * CL_NB)];
        const double* L = S + (size_t)(b / C) * CL_NB * ldr;
        if (rank != owner) {
            const double* src = cluster.map_shared_rank(S, owner) + (size_t)(b / C) * CL_NB * ldr;
            const int nv = (ldr - k0) / 2;
#pragma unroll 4
            for (int e = tid; e < nv * CL_NB; e += CL_NT) {
                const int o = (e / nv) * ldr + k0 + (e % nv) * 2;
                *reinterpret_cast<double2*>(Lb + o) = *reinterpret_cast<const double2*>(src + o);
            }
            L = Lb;
        }
        const int lb0 = (b + 1 - rank + C - 1) / C;  // my first block after b
        if (w == 0) {
            const int p = (lane < nm) ? perm[mv.x] : 0;
            __syncwarp();
            if (lane < nm) perm[mv.y] = p;
        }
        for (int c = lb0 * CL_NB + w; c < nloc * CL_NB; c += CL_NW) {
            double* col = S + (size_t)c * ldr;
            const double x = (lane < nm) ? col[mv.x] : 0.0;
            __syncwarp();
            if (lane < nm) col[mv.y] = x;
        }
        if (tid == 0) sh.next = CL_NW;
        __syncthreads();
        // my U rows
        for (int c = lb0 * CL_NB + tid; c < nloc * CL_NB; c += CL_NT) {
            double* col = S + (size_t)c * ldr + k0;
            const int gc = (rank + (c / CL_NB) * C) * CL_NB + c % CL_NB;
            double u[CL_NB];
#pragma unroll
            for (int p = 0; p < CL_NB; ++p) u[p] = (p < kb) ? col[p] : 0.0;
#pragma unroll
            for (int p = 1; p < CL_NB; ++p)
#pragma unroll
                for (int q = 0; q < p; ++q)
                    if (p < kb) u[p] -= L[(size_t)q * ldr + k0 + p] * u[q];
#pragma unroll
            for (int p = 0; p < CL_NB; ++p)
                if (p < kb) {
                    col[p] = u[p];
                    if (gc < NC) a[(size_t)perm[k0 + p] * ld + gc] = u[p];
                }
        }
        __syncthreads();
        // my columns' rows below the block (there are none unless the block is whole)
        const int r0 = k0 + CL_NB, nrc = (N - r0 + 31) / 32;
        auto item = [&](int rc, int lb) {
            const int r = r0 + rc * 32 + lane;
            if (r < N) {
                double l[CL_NB];
#pragma unroll
                for (int p = 0; p < CL_NB; ++p) l[p] = L[(size_t)p * ldr + r];
                double* col = S + (size_t)lb * CL_NB * ldr;
#pragma unroll
                for (int c = 0; c < CL_NB; ++c) {
                    double acc = col[(size_t)c * ldr + r], u[CL_NB];
                    cl_load8(col + (size_t)c * ldr + k0, u);
#pragma unroll
                    for (int p = 0; p < CL_NB; ++p) acc -= l[p] * u[p];
                    col[(size_t)c * ldr + r] = acc;
                }
            }
            __syncwarp();
        };
        const bool mine = r0 < N && rank == (b + 1) % C;  // I own the next block
        int first = lb0;
        if (mine) {
            for (int rc = w; rc < nrc; rc += CL_NW) item(rc, lb0);
            __syncthreads();
            if (w < CL_PW)
                cl_panel<RPL>(sh, S + (size_t)lb0 * CL_NB * ldr, ldr, N, NC, r0, min(CL_NB, N - r0), perm, a, ld);
            __syncwarp();
            __syncthreads();  // the panel has the FP64 pipe to itself
            first = lb0 + 1;
        }
        if (r0 < N) cl_arrive();
        if (r0 < N) {
            // the items go to the warps as they come free (the panel's warps come last)
            const int n = nrc * (nloc - first);
            int it = w;
            while (it < n) {
                item(it % nrc, first + it / nrc);
                if (lane == 0) it = atomicAdd(&sh.next, 1);
                it = __shfl_sync(0xffffffffu, it, 0);
            }
        }
        __syncthreads();
    }
    cluster.sync();  // every CTA's info is final
    if (rank == 0) {
        for (int r = tid; r < N; r += CL_NT) perm_out[(size_t)mat * N + r] = perm[r];
        if (tid == 0) {
            int inf = 0;
            for (int x = 0; x < C; ++x) {
                const int o = cluster.map_shared_rank(&sh, x)->info;
                if (o != 0 && (inf == 0 || o < inf)) inf = o;
            }
            info[mat] = inf;
        }
    }
    cluster.sync();  // no CTA leaves while its shared memory is read
}

// Sets *ran when the device can hold a cluster of this shape, and launches; a device or a partition of one with
// fewer SMs behind one another than the clusters need leaves the work to the split launches
template <int RPL, int OCC>
cudaError_t launch_cluster(int P, int N, int NC, int C, double* A, int ld, long long stride, int32_t* piv, int32_t* info,
                           cudaStream_t s, bool* ran) {
    const size_t sm = cl_smem(N, NC, C, sizeof(double));
    cudaError_t e = bte_raise_smem_limit((const void*)k_lu_cluster<RPL, OCC>, sm);
    if (e != cudaSuccess) return e;
    if (C > 8) {
        e = cudaFuncSetAttribute((const void*)k_lu_cluster<RPL, OCC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P * C);
    cfg.blockDim = dim3(CL_NT);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int held = 0;
    if (cudaOccupancyMaxActiveClusters(&held, k_lu_cluster<RPL, OCC>, &cfg) != cudaSuccess || held < 1) {
        cudaGetLastError();
        return cudaSuccess;
    }
    *ran = true;
    return cudaLaunchKernelEx(&cfg, k_lu_cluster<RPL, OCC>, N, NC, A, ld, stride, piv, info);
}

}  // namespace

// CTAs per matrix for P matrices of size N, or 0 where the split launches of lu.cu are the faster
// (or no cluster holds a matrix). The choice is free of P's consequences: every element goes
// through the same multiply-adds in the same order in both, so the factors are equal bit by bit.
// Model in microseconds, fitted to measured times (N = 33 to 513, 1 to 1200 matrices): a cluster
// takes 1.4 N for the chain of columns plus its share of the multiply-adds, in waves of as many
// clusters as the GPU holds at once (the occupancy interface's numbers for one CTA per SM; two
// fit below 112 KB and then slow each other by 1.4); the split launches take 6.3 N plus 43 us
// per matrix of N = 385. Measured (us, split / cluster): N = 129: 1 matrix 730 / 191, 1200 matrices
// 5678 / 2920; N = 257: 30 matrices 1855 / 754; N = 385: 1 matrix 2600 / 928, 15 matrices 2954 / 1426,
// 60 matrices 4753 / 4273, 137 matrices 7679 / 8595 (stays split); N = 513: 7 matrices 3988 /
// 1690, 16 matrices 4586 / 5008 (stays split).
int bte_lu_cluster_size(int P, int N, int NC) {
    if (N > 1024) return 0;
    const double n3 = (double)N * N * N;
    const double q = 1.0 + (100.0 / N) * (100.0 / N);
    double best = 6.3 * N + P * q * n3 / 1.43e6;
    int size = 0;
    struct Shape { int C, clusters; };
    constexpr Shape shapes[] = {{1, 152}, {2, 76}, {3, 46}, {4, 36}, {5, 28}, {6, 23}, {7, 15}, {8, 15}, {10, 13}, {16, 7}};
    for (const Shape& h : shapes) {
        const size_t sm = cl_smem(N, NC, h.C, sizeof(double));
        if (sm > CL_SMEM_MAX || (h.C - 1) * CL_NB >= N) continue;
        const bool two = sm <= 112 * 1024 && N <= 512;
        const int hold = two ? 2 * h.clusters : h.clusters;
        double t = (h.C == 1 ? 2.0 : h.C == 16 ? 1.75 : 1.4) * N + n3 / (1.1e4 * h.C);
        if (two && P > h.clusters) t *= 1.4;
        t *= (P + hold - 1) / hold;
        if (t < best) {
            best = t;
            size = h.C;
        }
    }
    return size;
}

// One cluster of C CTAs per matrix. *ran stays false, and nothing is done, where no such cluster fits the device.
cudaError_t bte_lu_factor_cluster(int P, int N, int NC, double* A, int ld, long long stride, int32_t* piv, int32_t* info,
                                  cudaStream_t s, int C, bool* ran) {
    *ran = false;
    constexpr int PT = 32 * CL_PW;
    if (N <= PT) return launch_cluster<1, 2>(P, N, NC, C, A, ld, stride, piv, info, s, ran);
    if (N <= 2 * PT) return launch_cluster<2, 2>(P, N, NC, C, A, ld, stride, piv, info, s, ran);
    if (N <= 4 * PT) return launch_cluster<4, 2>(P, N, NC, C, A, ld, stride, piv, info, s, ran);
    if (N <= 8 * PT) return launch_cluster<8, 1>(P, N, NC, C, A, ld, stride, piv, info, s, ran);
    return cudaErrorInvalidValue;
}
