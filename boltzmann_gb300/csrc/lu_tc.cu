// Batched FP32 LU with partial pivoting whose trailing updates run on the tcgen05 tensor
// cores (kind::tf32, accumulators in tensor memory), with split-TF32 operands so that the
// factors keep FP32 accuracy.
//
// Replaces, like lu.cu, the explicit batched inverse of the Newton Jacobian
// (xp.linalg.inv in bte_0d3v_batched.py:856-880, applied at :933-934). Same storage
// convention as lu.cu: row-major A[r * ld + c] with NC = N or N + 1 columns (the right-hand
// side appended as column N is eliminated with the matrix), rows never exchanged in
// memory, perm[position] = stored row, info = first zero pivot (1-based), 0 if none.
//
// One CTA per matrix, right-looking by 32-column panels:
//   1. panel: the 32 columns of positions k0..N-1 are held in registers; each column costs one
//      barrier: every warp publishes its best candidate row in shared memory, every warp picks
//      the same winner from them (one candidate per lane; largest |a|, lowest position on ties,
//      as LAPACK's i?amax) and applies the rank-one update. A row stays with its thread: only
//      its position changes;
//   2. U12 = L11^-1 A12 for the 32 pivot rows, one thread per column;
//   3. A22 -= L21 U12 in tiles of 128 columns x up to 192 rows (as even as multiples of 32
//      allow): U12^T (M = 128 columns) and L21 (N = rows) are staged in shared memory in the
//      canonical K-major layout (8 x 16 B core matrices, no swizzle), split into a TF32 high
//      part and an FP32 remainder, and one thread issues 4 k-steps x 3 products (hi*hi +
//      hi*lo + lo*hi) of tcgen05.mma.cta_group::1.kind::tf32 into a TMEM accumulator of 128
//      lanes. The warps read their part of A22 (lane = column: 32 consecutive columns of one
//      row, coalesced) before the product is issued and subtract the accumulator
//      (tcgen05.ld) from it after.
// Bound by latency: the panel's chain of columns and the tiles' reads, writes and barriers; two CTAs
// share an SM. Reading A22 only after the product, in groups of 16 rows, with tiles of 128 x 128 and
// rows exchanged between threads under branches, one matrix of N = 385 took 708 us and 4096 took
// 14.4 ms; now 358 us and 7.0 ms.
// Above N = 512 (k_tcs_*) the same steps are separate launches over many CTAs per matrix, with the operands
// split into three BF16 parts.
// The split: hi = tf32(x) (round to nearest), lo = x - hi (exact in FP32); hi*hi is exact
// in the FP32 accumulator, the dropped lo*lo term is below 2^-22 |x y|.
#include <cstdint>
#include <climits>
#include "bte_common.cuh"

namespace {

constexpr int TC_NT = 256;         // threads per CTA of the widest variant (8 warps; also 128)
constexpr int TC_NW = TC_NT / 32;  // shared-memory slots for the warps' pivot candidates
constexpr int TC_NB = 32;          // panel width = K of one block step
constexpr int TC_TM = 128;         // trailing columns per tile: MMA M, TMEM lanes
constexpr int TC_TR = 128;         // trailing rows per tile: MMA N, TMEM columns
constexpr uint32_t TC_TMEM_COLS = 128;
constexpr int TC_TRX = 192;        // tallest tile of k_lu_tc (its tiles are as even as 32 rows allow)
constexpr uint32_t TC_TMEM_COLS_X = 256;
constexpr int TC_PRE = 4;          // groups of 16 rows of a tile read ahead of its product
constexpr int TC_TILE_BYTES = TC_TM * TC_NB * 4;   // one operand part: 16 KB (TM == TR)
constexpr int TC_L11_LD = TC_NB + 4;        // L11 stored transposed, 16-byte rows
constexpr int TC_CAND_LD = TC_NB + 4;              // a candidate row + key + slot, 16-byte rows
constexpr uint32_t TC_WAIT_LIMIT = 1u << 22;       // bounded wait for an MMA commit

// shared memory map (bytes from the 1024-aligned dynamic base)
constexpr int SM_A_HI = 0;
constexpr int SM_A_LO = SM_A_HI + TC_TILE_BYTES;
constexpr int SM_B_HI = SM_A_LO + TC_TILE_BYTES;
constexpr int TC_TILEX_BYTES = TC_TRX * TC_NB * 4;
constexpr int SM_B_LO = SM_B_HI + TC_TILEX_BYTES;
constexpr int SM_L11 = SM_B_LO + TC_TILEX_BYTES;
constexpr int SM_CAND = SM_L11 + ((TC_NB * TC_L11_LD * 4 + 15) & ~15);
constexpr int SM_PERM = SM_CAND + 2 * TC_NW * TC_CAND_LD * 4;
constexpr int TC_OFF_PAD = TC_TRX + 4;  // offsets past the last row, read but not used
__host__ __device__ inline size_t tc_smem_bytes(int N) { return (size_t)SM_PERM + (size_t)(2 * N + 4 + TC_OFF_PAD) * 4 + 1024; }

// byte offset of element (row m, k) in a [rows x 32] TF32 tile, K-major, no swizzle:
// core matrix (m / 8, k / 4) at (m / 8) * 1024 + (k / 4) * 128, rows of a core matrix 16 B apart
__device__ inline int op_off(int m, int k) { return (m >> 3) * 1024 + (k >> 2) * 128 + (m & 7) * 16 + (k & 3) * 4; }

__device__ inline uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor (tcgen05): start address >> 4 (bits 0-13), leading byte
// offset >> 4 (bits 16-29: next core matrix along K), stride byte offset >> 4 (bits 32-45:
// next 8-row group), descriptor version 1 (bits 46-47), base offset 0, no swizzle (61-63)
__device__ inline uint64_t op_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46);
}

// instruction descriptor of kind::tf32: D F32 (bits 4-5 = 1), A and B TF32 (bits 7-9, 10-12
// = 2), both K-major (bits 15, 16 = 0), N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ inline void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ inline void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar)
                 : "memory");
}
__device__ inline void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ inline void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ inline void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ inline void mbar_init(uint32_t a, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(a), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ inline bool mbar_try_wait(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}

// tensor-memory allocation, one full warp
__device__ inline void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(dst_smem), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ inline void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}

// 16 consecutive TMEM columns of the warp's 32 lanes (lane i of the warp reads TMEM lane
// base + i): v[c] = D[lane][col + c]
__device__ inline void tmem_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ inline float tf32_rn(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// four values of one operand row (m, k..k+3) as high and low parts
__device__ inline void put_split4(unsigned char* sm, int m, int k, float a, float b, float c, float d,
                                  int lo_off = TC_TILE_BYTES) {
    float4 hi = make_float4(tf32_rn(a), tf32_rn(b), tf32_rn(c), tf32_rn(d));
    float4 lo = make_float4(a - hi.x, b - hi.y, c - hi.z, d - hi.w);
    const int o = op_off(m, k);
    *reinterpret_cast<float4*>(sm + o) = hi;
    *reinterpret_cast<float4*>(sm + lo_off + o) = lo;
}

// Predicated stores, for the panels' chain of columns: a branch that may diverge costs about 50 cycles
// there, whether taken or not.
__device__ inline void put_if(bool on, uint32_t addr, float x, float y, float z, float w) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t@p st.shared.v4.f32 [%1], {%2, %3, %4, %5};\n\t}\n" ::"r"(
                     (uint32_t)on),
                 "r"(addr), "f"(x), "f"(y), "f"(z), "f"(w)
                 : "memory");
}
__device__ inline void put_if(bool on, uint32_t addr, uint32_t x, uint32_t y) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t@p st.shared.v2.b32 [%1], {%2, %3};\n\t}\n" ::"r"((uint32_t)on),
                 "r"(addr), "r"(x), "r"(y)
                 : "memory");
}
// x -= l u under a predicate
__device__ inline void sub_if(bool on, float& x, float l, float u) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p fma.rn.f32 %0, %1, %2, %0;\n\t}\n"
        : "+f"(x)
        : "f"(-l), "f"(u), "r"((uint32_t)on));
}

template <int ROWS, int OCC, int NT>
__global__ void __launch_bounds__(NT, OCC)
k_lu_tc(int N, int NC, float* __restrict__ A, int ld, long long stride, int32_t* __restrict__ perm_out,
        int32_t* __restrict__ info, int vec4) {
    extern __shared__ unsigned char smraw[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fault;
    // 1024-aligned base for the operand tiles
    unsigned char* sm = smraw + ((1024 - (smem_u32(smraw) & 1023)) & 1023);
    float* L11 = reinterpret_cast<float*>(sm + SM_L11);
    float* cand = reinterpret_cast<float*>(sm + SM_CAND);
    int* perm = reinterpret_cast<int*>(sm + SM_PERM);  // stored row of a position
    int* roff = perm + ((N + 3) & ~3);                 // its offset in elements, 0 past the last

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    float* a = A + (size_t)blockIdx.x * stride;
    for (int r = tid; r < N; r += NT) perm[r] = r;
    for (int r = tid; r < N + TC_OFF_PAD; r += NT) roff[r] = (r < N) ? r * ld : 0;
    const uint32_t mb = smem_u32(&mbar);
    if (tid == 0) {
        mbar_init(mb, 1);
        s_fault = 0;
    }
    if (wid == 0) tmem_alloc(smem_u32(&tmem_slot), TC_TMEM_COLS_X);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    uint32_t phase = 0;
    int inf = 0;

    for (int k0 = 0; k0 < N; k0 += TC_NB) {
        const int mrows = N - k0;
        const int kb = min(TC_NB, mrows);
        const int ncol = min(TC_NB, NC - k0);
        // ---- 1. panel: positions k0.., columns k0..k0+31 in registers. A row stays with its thread
        // and only its position changes; the warps' candidates are compared by one lane each.
        float pr[ROWS][TC_NB];
        int pos[ROWS], row[ROWS];  // position relative to k0 (-1: no row), stored row
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const int s = tid + i * NT;
            pos[i] = (s < mrows) ? s : -1;
            row[i] = perm[k0 + min(s, mrows - 1)];
            const float* src = a + (size_t)row[i] * ld + k0;
            if (vec4 && ncol == TC_NB) {
#pragma unroll
                for (int c = 0; c < TC_NB; c += 4) {
                    float4 v = (s < mrows) ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                    pr[i][c] = v.x; pr[i][c + 1] = v.y; pr[i][c + 2] = v.z; pr[i][c + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int c = 0; c < TC_NB; ++c) pr[i][c] = (s < mrows && c < ncol) ? src[c] : 0.f;
            }
        }
#pragma unroll
        for (int j = 0; j < TC_NB; ++j) {
            if (j >= kb) break;
            float* cb = cand + (j & 1) * TC_NW * TC_CAND_LD;
            // the thread's and the warp's candidate among positions >= j: largest |a| (NaN counts
            // as 0), first position
            uint32_t key = 0, at = 0xffffffffu;
            int bi = 0;
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
                {
                    const float v = fabsf(pr[i][j]);
                    const uint32_t k = (v == v) ? __float_as_uint(v) : 0u;
                    const bool better = pos[i] >= j && (at == 0xffffffffu || k > key || (k == key && (uint32_t)pos[i] < at));
                    key = better ? k : key;
                    at = better ? (uint32_t)pos[i] : at;
                    bi = better ? i : bi;
                }
            const uint32_t wk = __reduce_max_sync(0xffffffffu, key);
            const uint32_t wa = __reduce_min_sync(0xffffffffu, key == wk ? at : 0xffffffffu);
            const bool mine = wa == 0xffffffffu ? lane == 0 : at == wa;
            const uint32_t my = smem_u32(cb + wid * TC_CAND_LD);
            put_if(mine, my + TC_NB * 4, wk, wa);
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
#pragma unroll
                for (int c = (j & ~3); c < TC_NB; c += 4)
                    put_if(mine && i == bi, my + c * 4, pr[i][c], pr[i][c + 1], pr[i][c + 2], pr[i][c + 3]);
            __syncthreads();
            // the same winner in every thread
            const uint2 o = (lane < NT / 32) ? *reinterpret_cast<const uint2*>(cb + lane * TC_CAND_LD + TC_NB)
                                             : make_uint2(0u, 0xffffffffu);
            const uint32_t bk = __reduce_max_sync(0xffffffffu, o.y == 0xffffffffu ? 0u : o.x);
            const uint32_t S = __reduce_min_sync(0xffffffffu, o.x == bk ? o.y : 0xffffffffu);
            const int W = __ffs(__ballot_sync(0xffffffffu, o.x == bk && o.y == S)) - 1;
            const float* prow = cb + W * TC_CAND_LD;
            // the pivot row's columns j.. in registers (16-byte loads from the 4-aligned start)
            float pv[TC_NB];
#pragma unroll
            for (int c = (j & ~3); c < TC_NB; c += 4) {
                const float4 v = *reinterpret_cast<const float4*>(prow + c);
                pv[c] = v.x; pv[c + 1] = v.y; pv[c + 2] = v.z; pv[c + 3] = v.w;
            }
            const float d = pv[j];
            inf = (!(d != 0.f) && inf == 0) ? k0 + j + 1 : inf;
            const float inv = (d != 0.f) ? __frcp_rn(d) : 0.f;
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                pos[i] = pos[i] == (int)S ? j : (pos[i] == j ? (int)S : pos[i]);
                // rows that are done keep their values, also where the pivot row holds an infinity
                const bool on = pos[i] > j;
                const float l = pr[i][j] * inv;
                pr[i][j] = on ? l : pr[i][j];
#pragma unroll
                for (int c = j + 1; c < TC_NB; ++c) sub_if(on, pr[i][c], l, pv[c]);
            }
        }
        // write the panel back (each position's data returns to its own stored row), the positions
        // and L11
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            if (pos[i] < 0) continue;
            float* dst = a + (size_t)row[i] * ld + k0;
            if (vec4 && ncol == TC_NB) {
#pragma unroll
                for (int c = 0; c < TC_NB; c += 4)
                    *reinterpret_cast<float4*>(dst + c) = make_float4(pr[i][c], pr[i][c + 1], pr[i][c + 2], pr[i][c + 3]);
            } else {
#pragma unroll
                for (int c = 0; c < TC_NB; ++c)
                    if (c < ncol) dst[c] = pr[i][c];
            }
            perm[k0 + pos[i]] = row[i];
            roff[k0 + pos[i]] = row[i] * ld;
            if (pos[i] < TC_NB) {
#pragma unroll
                for (int c = 0; c < TC_NB; ++c) L11[c * TC_L11_LD + pos[i]] = pr[i][c];
            }
        }
        const int ncols = NC - k0 - TC_NB;   // columns right of the panel (> 0 implies kb == 32)
        const int nrows = N - k0 - TC_NB;    // trailing rows
        __syncthreads();  // the panel's positions and L11
        if (ncols <= 0) break;
        // ---- 2. U12 = L11^-1 A12, one thread per column
        for (int c = tid; c < ncols; c += NT) {
            float x[TC_NB];
#pragma unroll
            for (int j = 0; j < TC_NB; ++j) x[j] = a[roff[k0 + j] + k0 + TC_NB + c];
#pragma unroll
            for (int i = 0; i < TC_NB; ++i) {
                // keeps the compiler from hoisting all 496 multipliers into registers
                asm volatile("" ::: "memory");
                float lc[TC_NB];
#pragma unroll
                for (int j = ((i + 1) & ~3); j < TC_NB; j += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(L11 + i * TC_L11_LD + j);
                    lc[j] = v.x; lc[j + 1] = v.y; lc[j + 2] = v.z; lc[j + 3] = v.w;
                }
#pragma unroll
                for (int j = i + 1; j < TC_NB; ++j) x[j] -= lc[j] * x[i];
            }
#pragma unroll
            for (int j = 0; j < TC_NB; ++j) a[roff[k0 + j] + k0 + TC_NB + c] = x[j];
        }
        if (nrows <= 0) break;  // last panel
        __syncthreads();
        // ---- 3. A22 -= L21 U12 on the tensor cores
        const int nrt = (nrows + TC_TRX - 1) / TC_TRX;              // row tiles
        const int th = ((nrows + nrt - 1) / nrt + 31) & ~31;        // rows of each, a multiple of 32
        const uint32_t idesc = idesc_tf32(TC_TM, th);
        for (int g0 = 0; g0 < nrows; g0 += th) {
            // B operand: L21 rows g0.., K = the panel's 32 columns
            // Groups of rows are loaded together, 8 lanes on consecutive rows: their 16-byte stores
            // fill one core matrix.
            const int br = (tid & 7) + (tid >> 6) * 8, bk = ((tid >> 3) & 7) * 4;
#pragma unroll 1
            for (int rb = br; rb < th; rb += 3 * (NT / 8)) {
                float4 bv[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int r = rb + i * (NT / 8);
                    bv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (r < th && g0 + r < nrows) {
                        const float* src = a + roff[k0 + TC_NB + g0 + r] + k0 + bk;
                        if (vec4) bv[i] = *reinterpret_cast<const float4*>(src);
                        else bv[i] = make_float4(src[0], src[1], src[2], src[3]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int r = rb + i * (NT / 8);
                    if (r < th) put_split4(sm + SM_B_HI, r, bk, bv[i].x, bv[i].y, bv[i].z, bv[i].w, TC_TILEX_BYTES);
                }
            }
            for (int c0 = 0; c0 < ncols; c0 += TC_TM) {
                // A operand: U12^T, row m = column c0 + m of U12, k = pivot row; and the warp's first
                // 16 TC_PRE rows of A22, read ahead of the product. Warp w updates the columns of
                // TMEM lanes 32 (w % 4).. in its share of the rows: all of the tile's with 4
                // warps, half with 8.
                constexpr int AI = TC_TM * (TC_NB / 4) / NT;
                const int am = tid & (TC_TM - 1);
                const float* ap = a + k0 + TC_NB + min(c0 + am, ncols - 1);
                float av[AI][4];
#pragma unroll
                for (int i = 0; i < AI; ++i) {
                    const int4 ro = *reinterpret_cast<const int4*>(roff + k0 + ((tid >> 7) + i * (NT / TC_TM)) * 4);
                    av[i][0] = ap[ro.x]; av[i][1] = ap[ro.y]; av[i][2] = ap[ro.z]; av[i][3] = ap[ro.w];
                }
                const int wq = wid & 3, rh = th / (NT / 128), rw = g0 + rh * (wid >> 2);
                const bool colok = (c0 + 32 * wq + lane) < ncols;
                float* colp = a + k0 + TC_NB + min(c0 + 32 * wq + lane, ncols - 1);
                const int* ro = roff + k0 + TC_NB + rw;
                const int nr = min(rh, nrows - rw);  // rows of this warp (none if <= 0)
                float old[TC_PRE][16] = {};
                auto ahead = [&](int u, float (&x)[16]) {  // 16 rows of A22 (row 0 past the last one)
#pragma unroll
                    for (int t = 0; t < 16; t += 4) {
                        const int4 r4 = *reinterpret_cast<const int4*>(ro + u * 16 + t);
                        x[t] = colp[r4.x]; x[t + 1] = colp[r4.y]; x[t + 2] = colp[r4.z]; x[t + 3] = colp[r4.w];
                    }
                };
#pragma unroll
                for (int u = 0; u < TC_PRE; ++u)
                    if (u * 16 < nr) ahead(u, old[u]);
#pragma unroll
                for (int i = 0; i < AI; ++i) {
                    const int k = ((tid >> 7) + i * (NT / TC_TM)) * 4;
                    if (c0 + am < ncols) put_split4(sm + SM_A_HI, am, k, av[i][0], av[i][1], av[i][2], av[i][3]);
                    else put_split4(sm + SM_A_HI, am, k, 0.f, 0.f, 0.f, 0.f);
                }
                fence_async_smem();
                tc_fence_before();
                __syncthreads();
                if (tid == 0) {
                    tc_fence_after();
                    const uint32_t ahi = smem_u32(sm + SM_A_HI), alo = smem_u32(sm + SM_A_LO);
                    const uint32_t bhi = smem_u32(sm + SM_B_HI), blo = smem_u32(sm + SM_B_LO);
#pragma unroll
                    for (int ks = 0; ks < TC_NB / 8; ++ks) {
                        const uint32_t o = ks * 256;
                        mma_tf32(tbase, op_desc(alo + o), op_desc(bhi + o), idesc, ks > 0 ? 1u : 0u);
                        mma_tf32(tbase, op_desc(ahi + o), op_desc(blo + o), idesc, 1u);
                        mma_tf32(tbase, op_desc(ahi + o), op_desc(bhi + o), idesc, 1u);
                    }
                    mma_commit(mb);
                    uint32_t it = 0;
                    while (!mbar_try_wait(mb, phase))
                        if (++it > TC_WAIT_LIMIT) { s_fault = 1; break; }
                }
                phase ^= 1u;
                __syncthreads();
                tc_fence_after();
                if (s_fault) break;
                const uint32_t trow = tbase + ((uint32_t)(32 * wq) << 16) + (uint32_t)(rw - g0);
#pragma unroll 1
                for (int u0 = 0; u0 * 16 < nr; u0 += TC_PRE) {
#pragma unroll
                    for (int v = 0; v < TC_PRE; ++v) {
                        const int u = u0 + v;
                        if (u * 16 >= nr) break;  // warp-uniform
                        float dv[16];
                        tmem_ld16(trow + u * 16, dv);
#pragma unroll
                        for (int t = 0; t < 16; t += 4) {
                            const int4 r4 = *reinterpret_cast<const int4*>(ro + u * 16 + t);
                            const int n4 = colok ? nr - u * 16 - t : 0;
                            if (n4 > 0) colp[r4.x] = old[v][t] - dv[t];
                            if (n4 > 1) colp[r4.y] = old[v][t + 1] - dv[t + 1];
                            if (n4 > 2) colp[r4.z] = old[v][t + 2] - dv[t + 2];
                            if (n4 > 3) colp[r4.w] = old[v][t + 3] - dv[t + 3];
                        }
                        if ((u + TC_PRE) * 16 < nr) ahead(u + TC_PRE, old[v]);
                    }
                }
                tc_fence_before();
                __syncthreads();  // TMEM and the operand tiles are free again
            }
            if (s_fault) break;
        }
        if (s_fault) break;
        __syncthreads();
    }
    if (s_fault) {
        // an MMA commit never arrived: wait once more (bounded) for its phase, the one before `phase`, before
        // giving TMEM back
        if (tid == 0) {
            uint32_t it = 0;
            while (!mbar_try_wait(mb, phase ^ 1u) && ++it < TC_WAIT_LIMIT) {}
        }
        __syncthreads();
    }
    for (int r = tid; r < N; r += NT) perm_out[(size_t)blockIdx.x * N + r] = perm[r];
    if (tid == 0) info[blockIdx.x] = s_fault ? -1 : inf;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (wid == 0) tmem_dealloc(tbase, TC_TMEM_COLS_X);
}

// ---------------------------------------------------------------------------------
// N > 512: one factorization split over many CTAs, two launches per panel of NB columns:
//   k_tcs_panel   one CTA per matrix: pivoting of the panel with the rows in registers (rows stay
//                 with their threads, only their positions change; one barrier per column), then
//                 U12 = L11^-1 A12, one thread per column;
//   k_tcs_update  one CTA per 128 x 128 tile of the trailing matrix: A22 -= L21 U12 with the tile's layout
//                 of k_lu_tc. These sizes had FP32 multiply-adds before, so the product must not be less
//                 exact than they: each operand is split into three BF16 parts, whose sum is the FP32
//                 value, and the six products of parts down to 2^-16 of the largest are taken, the
//                 smallest first, so that the accumulator (which truncates) is rounded at the size of the
//                 sum in the last two only. Backward error of the factors (Frobenius, in FP32 units of
//                 |L| |U|), FP32 multiply-adds / two TF32 parts and three products / this: N = 513 0.050 /
//                 0.102 / 0.027; N = 769 0.042 / 0.087 / 0.021; three TF32 parts give 0.030 but their 96 KB
//                 of operands leave two CTAs per SM (75 matrices of N = 769 2024 us against 1631).
// A matrix of N = 769 keeps one CTA busy for 5.5 ms (k_lu_right), with half the SMs idle for 75 of them;
// split, the trailing updates spread over the GPU and the chain is the panels' columns.
// Bound by that chain for few matrices and by the trailing matrices' reads and writes for many.
// The result does not depend on the number of matrices. Measured (us, k_lu_right -> these):
// N = 513: 2090 -> 540 (1 matrix), 2380 -> 986 (150); N = 769: 5521 -> 889 (1), 6118 -> 1631 (75),
// 19415 -> 6438 (400); N = 1281: 41980 -> 4699 (48); N = 2048: 247724 -> 3558 (2).
// ---------------------------------------------------------------------------------
constexpr int TS_NT = 512;             // threads of the panel kernel
constexpr int TS_NW = TS_NT / 32;
constexpr int TS_LD = TC_NB + 4;       // a published row, 16-byte aligned

template <int NB, int ROWS>
__global__ void __launch_bounds__(TS_NT, 1)
k_tcs_panel(int N, int NC, int k0, float* __restrict__ A, int ld, long long stride, int32_t* __restrict__ perm_g,
            int32_t* __restrict__ info, int vec4) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(16) float cand[2][TS_NW][TS_LD];  // a warp's best row of the column
    __shared__ uint2 ckey[2][TS_NW];                       // its |a| as bits, its position
    __shared__ __align__(16) float L11[NB][NB + 4];        // transposed: L11[column][row]
    int* pos2row = reinterpret_cast<int*>(smraw);          // stored row at position k0 + i
    const int mrows = N - k0, kb = min(NB, mrows), ncol = min(NB, NC - k0);
    const int mat = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    float* a = A + (size_t)mat * stride;
    int32_t* pg = perm_g + (size_t)mat * N;
    float pr[ROWS][NB];
    int pos[ROWS], row[ROWS];  // position relative to k0 (-1: no row), stored row
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int s = tid + i * TS_NT;
        pos[i] = (s < mrows) ? s : -1;
        row[i] = (s < mrows) ? (k0 == 0 ? s : pg[k0 + s]) : 0;
        const float* src = a + (size_t)row[i] * ld + k0;
        if (vec4 && ncol == NB) {
#pragma unroll
            for (int c = 0; c < NB; c += 4) {
                const float4 v = (s < mrows) ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                pr[i][c] = v.x; pr[i][c + 1] = v.y; pr[i][c + 2] = v.z; pr[i][c + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int c = 0; c < NB; ++c) pr[i][c] = (s < mrows && c < ncol) ? src[c] : 0.f;
        }
    }
    int inf = 0;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        if (j >= kb) break;
        // the thread's, the warp's and the CTA's candidate: largest |a| (NaN counts as 0), first position
        uint32_t key = 0, at = 0xffffffffu;
        int bi = 0;
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
            if (pos[i] >= j) {
                const float v = fabsf(pr[i][j]);
                const uint32_t k = (v == v) ? __float_as_uint(v) : 0u;
                if (at == 0xffffffffu || k > key || (k == key && (uint32_t)pos[i] < at)) { key = k; at = pos[i]; bi = i; }
            }
        const uint32_t wk = __reduce_max_sync(0xffffffffu, key);
        const uint32_t wa = __reduce_min_sync(0xffffffffu, key == wk ? at : 0xffffffffu);
        if (wa == 0xffffffffu ? lane == 0 : at == wa) {
            float* my = cand[j & 1][wid];
            ckey[j & 1][wid] = make_uint2(wk, wa);
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
                if (i == bi) {
#pragma unroll
                    for (int c = (j & ~3); c < NB; c += 4)
                        *reinterpret_cast<float4*>(my + c) = make_float4(pr[i][c], pr[i][c + 1], pr[i][c + 2], pr[i][c + 3]);
                }
        }
        __syncthreads();
        const uint2 o = (lane < TS_NW) ? ckey[j & 1][lane] : make_uint2(0u, 0xffffffffu);
        const uint32_t bk = __reduce_max_sync(0xffffffffu, o.y == 0xffffffffu ? 0u : o.x);
        const uint32_t S = __reduce_min_sync(0xffffffffu, o.x == bk ? o.y : 0xffffffffu);
        const int W = __ffs(__ballot_sync(0xffffffffu, o.x == bk && o.y == S)) - 1;
        const float* prow = cand[j & 1][W];
        float pv[NB];
#pragma unroll
        for (int c = (j & ~3); c < NB; c += 4) {
            const float4 v = *reinterpret_cast<const float4*>(prow + c);
            pv[c] = v.x; pv[c + 1] = v.y; pv[c + 2] = v.z; pv[c + 3] = v.w;
        }
        const float d = pv[j];
        if (!(d != 0.f) && inf == 0) inf = k0 + j + 1;
        const float inv = (d != 0.f) ? __frcp_rn(d) : 0.f;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            if (pos[i] == (int)S) pos[i] = j;
            else if (pos[i] == j) pos[i] = (int)S;
            if (pos[i] > j) {
                const float l = pr[i][j] * inv;
                pr[i][j] = l;
#pragma unroll
                for (int c = j + 1; c < NB; ++c) pr[i][c] -= l * pv[c];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
        if (pos[i] >= 0) {
            float* dst = a + (size_t)row[i] * ld + k0;
            if (vec4 && ncol == NB) {
#pragma unroll
                for (int c = 0; c < NB; c += 4)
                    *reinterpret_cast<float4*>(dst + c) = make_float4(pr[i][c], pr[i][c + 1], pr[i][c + 2], pr[i][c + 3]);
            } else {
#pragma unroll
                for (int c = 0; c < NB; ++c)
                    if (c < ncol) dst[c] = pr[i][c];
            }
            pos2row[pos[i]] = row[i];
            if (pos[i] < NB)
#pragma unroll
                for (int c = 0; c < NB; ++c) L11[c][pos[i]] = pr[i][c];
        }
    __syncthreads();
    for (int r = tid; r < mrows; r += TS_NT) pg[k0 + r] = pos2row[r];
    if (tid == 0) {
        const int cur = (k0 == 0) ? 0 : info[mat];
        info[mat] = cur != 0 ? cur : inf;
    }
    if (kb < NB) return;  // the last panel: nothing to its right but columns it holds
    // U12 = L11^-1 A12, one thread per column
    for (int c = k0 + NB + tid; c < NC; c += TS_NT) {
        float x[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) x[j] = a[(size_t)pos2row[j] * ld + c];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            asm volatile("" ::: "memory");  // keeps the compiler from hoisting all multipliers into registers
            float lc[NB];
#pragma unroll
            for (int j = ((i + 1) & ~3); j < NB; j += 4) {
                const float4 v = *reinterpret_cast<const float4*>(&L11[i][j]);
                lc[j] = v.x; lc[j + 1] = v.y; lc[j + 2] = v.z; lc[j + 3] = v.w;
            }
#pragma unroll
            for (int j = i + 1; j < NB; ++j) x[j] -= lc[j] * x[i];
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) a[(size_t)pos2row[j] * ld + c] = x[j];
    }
}

constexpr int TS_PART = TC_TM * TC_NB * 2;   // one part of an operand: 8 KB
// byte offset of element (row m, k) in a [rows x 32] BF16 tile, K-major, no swizzle: core matrix (m / 8, k / 8)
// at (m / 8) * 512 + (k / 8) * 128, rows of a core matrix 16 B apart
__device__ inline int ts_off(int m, int k) { return (m >> 3) * 512 + (k >> 3) * 128 + (m & 7) * 16 + (k & 7) * 2; }
// shared-memory matrix descriptor as op_desc, 8-row groups 512 B apart
__device__ inline uint64_t ts_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) |
           ((uint64_t)1 << 46);
}
// instruction descriptor of kind::f16 with A and B BF16 (bits 7-9, 10-12 = 1), else as idesc_tf32
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ inline void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
// two values rounded to BF16 (x in the low half)
__device__ inline uint32_t bf16x2(float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(y), "f"(x));
    return r;
}
// four values of one operand row (m, k..k+3) as three BF16 parts whose sum is the value
__device__ inline void put_split3(unsigned char* sm, int m, int k, float a, float b, float c, float d) {
    const int o = ts_off(m, k);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const uint32_t u = bf16x2(a, b), v = bf16x2(c, d);
        *reinterpret_cast<uint2*>(sm + p * TS_PART + o) = make_uint2(u, v);
        a -= __uint_as_float(u << 16);
        b -= __uint_as_float(u & 0xffff0000u);
        c -= __uint_as_float(v << 16);
        d -= __uint_as_float(v & 0xffff0000u);
    }
}

// one 128 x 128 tile of A22 -= L21 U12 (kb = 16 or 32 panel columns at k0)
__global__ void __launch_bounds__(256, 3)
k_tcs_update(int N, int NC, int k0, int kb, int nct, int nrt, float* __restrict__ A, int ld, long long stride,
             const int32_t* __restrict__ perm_g, int32_t* __restrict__ info, int vec4) {
    extern __shared__ unsigned char smraw[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fault;
    __shared__ int rows[TC_TR], piv[TC_NB];
    unsigned char* sm = smraw + ((1024 - (smem_u32(smraw) & 1023)) & 1023);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per = nct * nrt, mat = blockIdx.x / per, t = blockIdx.x % per;
    const int c0 = k0 + kb + (t % nct) * TC_TM, r0 = k0 + kb + (t / nct) * TC_TR;
    const int ncols = min(TC_TM, NC - c0), nrows = min(TC_TR, N - r0);
    float* a = A + (size_t)mat * stride;
    const int32_t* pg = perm_g + (size_t)mat * N;
    const uint32_t mb = smem_u32(&mbar);
    if (tid < TC_TR) rows[tid] = (tid < nrows) ? pg[r0 + tid] * ld : -1;  // N ld < 2^31
    if (tid >= 128 && tid < 128 + kb) piv[tid - 128] = pg[k0 + tid - 128] * ld;
    if (tid == 0) {
        mbar_init(mb, 1);
        s_fault = 0;
    }
    if (wid == 0) tmem_alloc(smem_u32(&tmem_slot), TC_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    const int k4 = kb / 4;
    // B operand: rows of L21; A operand: U12^T (row m = column c0 + m)
    for (int e = tid; e < TC_TR * k4; e += 256) {
        const int r = e / k4, k = (e % k4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (rows[r] >= 0) {
            const float* src = a + rows[r] + k0 + k;
            if (vec4) v = *reinterpret_cast<const float4*>(src);
            else v = make_float4(src[0], src[1], src[2], src[3]);
        }
        put_split3(sm + 3 * TS_PART, r, k, v.x, v.y, v.z, v.w);
    }
    for (int e = tid; e < TC_TM * k4; e += 256) {
        const int m = e & (TC_TM - 1), k = (e >> 7) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (m < ncols)
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = a[piv[k + q] + c0 + m];
        put_split3(sm, m, k, v[0], v[1], v[2], v[3]);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
        tc_fence_after();
        constexpr int pa[6] = {1, 0, 2, 0, 1, 0}, pb[6] = {1, 2, 0, 1, 0, 0};  // parts, the smallest products first
        const uint32_t as = smem_u32(sm), bs = as + 3 * TS_PART;
        constexpr uint32_t idesc = idesc_bf16(TC_TM, TC_TR);
#pragma unroll
        for (int p = 0; p < 6; ++p)
            for (int ks = 0; ks < kb / 16; ++ks)
                mma_bf16(tbase, ts_desc(as + pa[p] * TS_PART + ks * 256), ts_desc(bs + pb[p] * TS_PART + ks * 256), idesc,
                         p + ks > 0 ? 1u : 0u);
        mma_commit(mb);
    }
    // the tile's first values while the products run: warp w reads TMEM lanes 32 (w % 4) .. (columns)
    // and 64 (w / 4) .. of the TMEM columns (rows)
    const int q = wid & 3, h = wid >> 2, m = 32 * q + lane;
    const bool colok = m < ncols;
    float* colp = a + c0 + m;
    float old[16];
    auto fetch = [&](int rr) {
#pragma unroll
        for (int i = 0; i < 16; ++i) old[i] = (colok && rows[rr + i] >= 0) ? colp[rows[rr + i]] : 0.f;
    };
    fetch(64 * h);
    if (tid == 0) {
        uint32_t it = 0;
        while (!mbar_try_wait(mb, 0))
            if (++it > TC_WAIT_LIMIT) { s_fault = 1; break; }
    }
    __syncthreads();
    tc_fence_after();
    if (!s_fault) {
#pragma unroll 1
        for (int rr = 64 * h; rr < 64 * h + 64; rr += 16) {
            if (rr >= nrows) break;  // warp-uniform
            float dv[16];
            tmem_ld16(tbase + ((uint32_t)(32 * q) << 16) + (uint32_t)rr, dv);
            float out[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) out[i] = old[i] - dv[i];
            if (rr + 16 < 64 * h + 64) fetch(rr + 16);
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (colok && rows[rr + i] >= 0) colp[rows[rr + i]] = out[i];
        }
    } else {
        // an MMA commit never arrived: wait once more (bounded) before giving TMEM back
        if (tid == 0) {
            uint32_t it = 0;
            while (!mbar_try_wait(mb, 0) && ++it < TC_WAIT_LIMIT) {}
            info[mat] = -1;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (wid == 0) tmem_dealloc(tbase, TC_TMEM_COLS);
}

template <int NB, int ROWS>
cudaError_t launch_tcs_panel(int P, int N, int NC, int k0, float* A, int ld, long long stride, int32_t* piv, int32_t* info,
                             cudaStream_t s, int vec4) {
    k_tcs_panel<NB, ROWS><<<P, TS_NT, (size_t)(N - k0) * 4, s>>>(N, NC, k0, A, ld, stride, piv, info, vec4);
    return cudaGetLastError();
}

template <int ROWS, int OCC, int NT>
cudaError_t launch_tc(int P, int N, int NC, float* A, int ld, long long stride, int32_t* piv, int32_t* info,
                      cudaStream_t s) {
    const size_t sm = tc_smem_bytes(N);
    cudaError_t e = bte_raise_smem_limit((const void*)k_lu_tc<ROWS, OCC, NT>, sm);
    if (e != cudaSuccess) return e;
    const int vec4 = (ld % 4 == 0 && stride % 4 == 0 && ((uintptr_t)A & 15) == 0) ? 1 : 0;
    k_lu_tc<ROWS, OCC, NT><<<P, NT, sm, s>>>(N, NC, A, ld, stride, piv, info, vec4);
    return cudaGetLastError();
}

}  // namespace

// FP32 factorization of P matrices with N > 512 (any N up to 2048) by panels: 32 columns while two
// rows per thread hold them (up to 1024 rows), 16 above
cudaError_t bte_lu_factor_tcs(int P, int N, int NC, float* A, int ld, long long stride, int32_t* piv, int32_t* info,
                              cudaStream_t s) {
    if (P <= 0) return cudaSuccess;
    if (N < 1 || N > 4 * TS_NT || NC < N || NC > N + 1 || ld < NC) return cudaErrorInvalidValue;
    if ((long long)N * ld >= (1ll << 31)) return cudaErrorInvalidValue;  // row offsets are 32-bit
    const int vec4 = (ld % 4 == 0 && stride % 4 == 0 && ((uintptr_t)A & 15) == 0) ? 1 : 0;
    const size_t usm = (size_t)6 * TS_PART + 1024;
    cudaError_t e = bte_raise_smem_limit((const void*)k_tcs_update, usm);
    if (e != cudaSuccess) return e;
    for (int k0 = 0; k0 < N;) {
        const int mrows = N - k0, nb = mrows > 2 * TS_NT ? 16 : 32;
        if (mrows > 2 * TS_NT) e = launch_tcs_panel<16, 4>(P, N, NC, k0, A, ld, stride, piv, info, s, vec4);
        else if (mrows > TS_NT) e = launch_tcs_panel<32, 2>(P, N, NC, k0, A, ld, stride, piv, info, s, vec4);
        else e = launch_tcs_panel<32, 1>(P, N, NC, k0, A, ld, stride, piv, info, s, vec4);
        if (e != cudaSuccess) return e;
        const int nr = mrows - nb, ncol = NC - k0 - nb;
        if (nr > 0 && ncol > 0) {
            const int nct = (ncol + TC_TM - 1) / TC_TM, nrt = (nr + TC_TR - 1) / TC_TR;
            k_tcs_update<<<(unsigned)P * nct * nrt, 256, usm, s>>>(N, NC, k0, nb, nct, nrt, A, ld, stride, piv, info, vec4);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        k0 += nb;
    }
    return cudaSuccess;
}

// largest N the tensor-core kernel takes (its panel is two 32-column rows per thread)
int bte_lu_tc_max_n() { return 2 * TC_NT; }

// variant 0: 256 threads, two CTAs per SM (the registers of two, 2 x 256 tensor-memory
// columns); 1: 256 threads, one CTA per SM (half the matrices in flight, so that their
// trailing updates stay in L2); 2: 128 threads (4 warps: half the per-column pivot-search work
// per matrix, up to four panel rows per thread), two CTAs per SM
cudaError_t bte_lu_factor_tc(int P, int N, int NC, float* A, int ld, long long stride, int32_t* piv, int32_t* info,
                             cudaStream_t s, int variant) {
    if (P <= 0) return cudaSuccess;
    if (N < 1 || N > 2 * TC_NT || NC < N || NC > N + 1 || ld < NC) return cudaErrorInvalidValue;
    if ((long long)N * ld >= (1ll << 31)) return cudaErrorInvalidValue;  // row offsets are 32-bit
    if (variant == 2) {
        if (N <= 128) return launch_tc<1, 2, 128>(P, N, NC, A, ld, stride, piv, info, s);
        if (N <= 256) return launch_tc<2, 2, 128>(P, N, NC, A, ld, stride, piv, info, s);
        if (N <= 384) return launch_tc<3, 2, 128>(P, N, NC, A, ld, stride, piv, info, s);
        return launch_tc<4, 2, 128>(P, N, NC, A, ld, stride, piv, info, s);
    }
    if (variant == 1) {
        if (N <= TC_NT) return launch_tc<1, 1, 256>(P, N, NC, A, ld, stride, piv, info, s);
        return launch_tc<2, 1, 256>(P, N, NC, A, ld, stride, piv, info, s);
    }
    if (N <= TC_NT) return launch_tc<1, 2, 256>(P, N, NC, A, ld, stride, piv, info, s);
    return launch_tc<2, 2, 256>(P, N, NC, A, ld, stride, piv, info, s);
}
