// Finite-volume 1D3V fully implicit step on the GPU (sm_103a): the reference's
// solver_type "fully_implicit" (bte_1d3v_solver.py:1890-2009), preconditioned by its op-split
// step (:1745-1870, type XVTVRC).
//
// Operator: one fused kernel (k_fvm_mvec, fvm_core.h's fvm_mvec_tab_at on the step's tabulated
// coefficients) reads each value's upwind stencils along x, v_r and v_theta and writes one
// output, after the ordinate moments m = w^T v (k_fvm_moment) and the gain product G m over
// the few non-zeros of G's rows (k_fvm_gain). The reference
// multiplies dense (Nr Nvt)^2 collision and advection matrices instead; here the work per
// value is O(p + Nr), so the operator is one read and one write of v (HBM-bound).
// Preconditioner: the collision inverse in closed form, (D^-1 (x) I + H (x) 1 w^T) v (k_fvm_hmul), then the
// v_r, v_theta and x sweeps in the natural layout: the v_r and v_theta recurrences run one
// thread per line with the warp's lanes on consecutive x (coalesced), the x recurrence on rows
// staged in shared memory; the reference (and the drop-in sweeps of sweeps.cu) swap layouts
// between the sweeps instead.
// Solver: restarted right-preconditioned GMRES (fvm_core.h), device vectors, FP64.
// Semi-Lagrangian step (solver_type "sl_implicit", :2024-2027): one kernel interpolates every
// value at its departure point (k_fvm_sl), then the closed-form collision inverse.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "bte_common.cuh"
#include "fvm_core.h"
#include "../../include/bte_fvm_gb300.h"
#include "../../include/bte_sweeps_gb300.h"

struct bte_fvm {
    int device = 0;
    int Nr = 0, Nvt = 0, Nx = 0, ndr = 0, ndt = 0, ndx = 0;
    size_t N = 0;
    double *vr = nullptr, *vt = nullptr, *cos_t = nullptr, *w = nullptr, *loss = nullptr, *gain = nullptr;
    int8_t* north = nullptr;
    double *vrL = nullptr, *vrR = nullptr, *vtL = nullptr, *vtR = nullptr, *xL = nullptr, *xR = nullptr;
    double *dinv = nullptr, *H = nullptr;   // collision inverse factors (set per step size)
    bool have_inverse = false;
    double *M = nullptr, *T = nullptr, *aE = nullptr, *axvr = nullptr;   // (Nr, Nx), (Nr, Nx), Nx, Nr
    double *A = nullptr, *Bf = nullptr;                                  // N each
    // operator coefficients of a step (k_fvm_mvec_coef) and their set-up parts
    double *bx = nullptr, *arc = nullptr, *lr = nullptr, *vinv = nullptr;  // Nx, Nr Nvt, Nr, Nr
    int8_t *eflag = nullptr, *cpos = nullptr;                             // Nx: bit 0 E >= 0, bit 1 E < 0; Nvt: cos > 0
    int32_t *gptr = nullptr, *gcol = nullptr;                             // the gain matrix by rows (exact non-zeros)
    double* gval = nullptr;
    uint32_t* hmask = nullptr;   // per 8-row tile of H: which chunks of HC columns hold a non-zero
    int32_t* bad = nullptr;      // per x: a non-finite ordinate moment (it reaches every row of G m and H m)
    double* swc = nullptr;       // sweep coefficients (k_fvm_sweep_coef), allocated with the collision inverse if there is room
    double *B = nullptr, *X = nullptr, *R = nullptr, *W = nullptr, *Z = nullptr, *Tv = nullptr;
    double* Kr = nullptr;
    int kcap = 0;
    double *part = nullptr, *hd = nullptr;
    double* hp = nullptr;  // pinned: what the reductions gave
    double *xg = nullptr, *vrp = nullptr, *vta = nullptr;   // semi-Lagrangian grids (set once)
    double sl_vmin = 0.0;
    bool have_sl = false;
    std::vector<void*> allocs;
    long long launches = 0;
};

namespace {

constexpr int FT = 256;          // threads of the element kernels
constexpr int FVM_RED = 120;     // partial-sum blocks of the reductions (fixed: deterministic order)

thread_local std::string g_fvm_err;

int fvm_fail(int code, const std::string& msg) {
    g_fvm_err = msg;
    return code;
}

inline unsigned fblocks(size_t n) { return (unsigned)((n + FT - 1) / FT); }

FvmView view_of(const bte_fvm* h) {
    FvmView v;
    v.Nr = h->Nr; v.Nvt = h->Nvt; v.Nx = h->Nx;
    v.ndr = h->ndr; v.ndt = h->ndt; v.ndx = h->ndx;
    v.vr = h->vr; v.cos_t = h->cos_t; v.north = h->north; v.w = h->w; v.loss = h->loss;
    v.vrL = h->vrL; v.vrR = h->vrR; v.vtL = h->vtL; v.vtR = h->vtR; v.xL = h->xL; v.xR = h->xR;
    return v;
}

// GB300 runs FP64 at 2 fused multiply-adds per clock and SM: a warp instruction (compares and
// conversions included) occupies its sub-partition's FP64 pipe for 64 cycles, and 16 bytes from
// L2 cost less than one. The kernels of this file are bound by that pipe, so what does not depend
// on the vector is tabulated once per step, divisions above all.

// m[r][x] = sum_j w_j X[r][j][x], one thread per (r, x); bad[x] is set where a moment is not finite
__global__ void k_fvm_moment(FvmView v, const double* __restrict__ X, double* __restrict__ m, int32_t* bad) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)v.Nr * v.Nx) return;
    const int x = (int)(i % v.Nx), r = (int)(i / v.Nx);
    const double s = fvm_moment_at(v, X, r, x);
    m[i] = s;
    if ((__double2hiint(s) & 0x7ff00000) == 0x7ff00000) bad[x] = 1;  // Inf or NaN, without an FP64 instruction
}

// The operator's coefficients for a step: bx = dt tau cA E, arc = dtx ax v_r cos(theta), lr =
// dt tau kappa loss, and the sign of E as bits
__global__ void k_fvm_mvec_coef(FvmView v, FvmCoef c, const double* __restrict__ E, double* __restrict__ bx,
                                double* __restrict__ arc, double* __restrict__ lr, int8_t* __restrict__ eflag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < v.Nx) {
        bx[i] = fvm_coef_field(c, E[i]);
        eflag[i] = (int8_t)fvm_field_sign(E[i]);
    }
    if (i < v.Nr) lr[i] = fvm_coef_loss(v, c, i);
    if (i < v.Nr * v.Nvt) arc[i] = fvm_coef_drift(v, c, i / v.Nvt, i % v.Nvt);
}

// T = kt (G m) over the non-zeros of G's rows: at most two per process and row
__global__ void k_fvm_gain(int Nr, int Nx, double kt, const int32_t* __restrict__ ptr, const int32_t* __restrict__ col,
                           const double* __restrict__ val, const double* __restrict__ m, const int32_t* __restrict__ bad,
                           double* __restrict__ T) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Nr * Nx) return;
    const int x = i % Nx, r = i / Nx;
    double s = 0.0;
    for (int e = ptr[r]; e < ptr[r + 1]; ++e) s += val[e] * m[(size_t)col[e] * Nx + x];
    T[i] = bad[x] ? __longlong_as_double(0x7ff8000000000000ll) : kt * s;
}

// Y = rhs_mvec(X) (fvm_mvec_tab_at) with the tabulated coefficients, one thread per value, x fastest:
// three stencils and seven more FP64 instructions per value; the form that computes them all per
// value took 33 with a division (976,000 values, 200 x 305 x 16: 61 us -> 29 us; 16 FP64
// instructions take 26 us). T = dt tau kappa G m.
__global__ void k_fvm_mvec(FvmView v, const double* __restrict__ bx, const double* __restrict__ arc,
                           const double* __restrict__ lr, const double* __restrict__ vinv,
                           const int8_t* __restrict__ eflag, const int8_t* __restrict__ cpos,
                           const double* __restrict__ T, const double* __restrict__ X, double* __restrict__ Y,
                           int32_t* bad) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)v.Nr * v.Nvt * v.Nx;
    if (i >= n) return;
    const int x = (int)(i % v.Nx);
    const int rj = (int)(i / v.Nx);
    const int j = rj % v.Nvt, r = rj / v.Nvt;
    if (rj == 0) bad[x] = 0;  // the moments of the next product start clean
    Y[i] = fvm_mvec_tab_at(v, bx[x], arc[rj], lr[r], vinv[r], eflag[x], cpos[j] != 0, T[(size_t)r * v.Nx + x], X, r, j, x);
}

// T = H M (Nr x Nr by Nr x Nx) for the collision inverse. One warp per 8 rows x 32 columns and a
// quarter of the columns of H, the four partial sums added in a fixed order. Chunks of HC columns
// that hold no non-zero in the 8 rows are passed over: collisions only move electrons down in
// energy, so most of H below its diagonal is zero. 305 x 305 by 200: 101 us as a general product
// of 32 x 32 tiles (70 CTAs) -> 38 us; all its FP64 multiply-adds take 31 us.
constexpr int HR = 8;    // rows per tile
constexpr int HC = 16;   // columns of H per chunk
__global__ void __launch_bounds__(128)
k_fvm_hmul(int Nr, int Nx, int words, const uint32_t* __restrict__ mask, const double* __restrict__ H,
           const double* __restrict__ M, const int32_t* __restrict__ bad, double* __restrict__ T) {
    __shared__ double part[3][HR][32];
    __shared__ __align__(16) double sh[4][HC][HR];  // a warp's chunk of H, transposed
    const int r0 = blockIdx.y * HR, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int x = blockIdx.x * 32 + lane, xc = min(x, Nx - 1);
    const uint32_t* mk = mask + (size_t)blockIdx.y * words;
    double acc[HR];
#pragma unroll
    for (int i = 0; i < HR; ++i) acc[i] = 0.0;
    double mv[HC], hv[HR * HC / 32];
    // chunk c: HC rows of M, and H's HR x HC block (rows r0 .., lane -> column lane % HC)
    auto fetch = [&](int c) {
        const int k0 = c * HC;
#pragma unroll
        for (int k = 0; k < HC; ++k) mv[k] = M[(size_t)min(k0 + k, Nr - 1) * Nx + xc];
        const int k = min(k0 + lane % HC, Nr - 1);
#pragma unroll
        for (int q = 0; q < HR * HC / 32; ++q) {
            const int r = min(r0 + lane / HC + q * (32 / HC), Nr - 1);
            hv[q] = (k0 + lane % HC < Nr) ? H[(size_t)r * Nr + k] : 0.0;
        }
    };
    int seen = 0;  // the tile's chunks go to the four warps in turn
    for (int cw = 0; cw < words; ++cw) {
        uint32_t bits = mk[cw];
        while (bits) {
            const int c = 32 * cw + __ffs(bits) - 1;
            bits &= bits - 1;
            if ((seen++ & 3) != w) continue;
            fetch(c);
            __syncwarp();
#pragma unroll
            for (int q = 0; q < HR * HC / 32; ++q) sh[w][lane % HC][lane / HC + q * (32 / HC)] = hv[q];
            __syncwarp();
#pragma unroll
            for (int k = 0; k < HC; ++k)
#pragma unroll
                for (int i = 0; i < HR; i += 2) {
                    const double2 h2 = *reinterpret_cast<const double2*>(&sh[w][k][i]);
                    acc[i] += h2.x * mv[k];
                    acc[i + 1] += h2.y * mv[k];
                }
        }
    }
    if (w > 0)
#pragma unroll
        for (int i = 0; i < HR; ++i) part[w - 1][i][lane] = acc[i];
    __syncthreads();
    if (w > 0 || x >= Nx) return;
    const bool nan = bad[x] != 0;
#pragma unroll
    for (int i = 0; i < HR; ++i)
        if (r0 + i < Nr)
            T[(size_t)(r0 + i) * Nx + x] = nan ? __longlong_as_double(0x7ff8000000000000ll)
                                               : ((acc[i] + part[0][i][lane]) + part[1][i][lane]) + part[2][i][lane];
}

// out (Nx, Nvt, Nr) = the collision inverse applied to B (Nr, Nvt, Nx), one thread per output
__global__ void k_fvm_coll_permute(FvmView v, const double* __restrict__ dinv, const double* __restrict__ T,
                                   const double* __restrict__ B, double* __restrict__ out, int32_t* bad) {
    const size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)v.Nr * v.Nvt * v.Nx;
    if (o >= n) return;
    const int r = (int)(o % v.Nr);
    const size_t xj = o / v.Nr;
    const int j = (int)(xj % v.Nvt), x = (int)(xj / v.Nvt);
    if (j == 0 && r == 0) bad[x] = 0;
    out[o] = fvm_coll_apply_at(v, dinv, T, B, r, j, x);
}

// Y (Nr, Nvt, Nx) = the collision inverse applied to B, same layout, times sc where given (the
// diagonal reciprocals of the sweep that follows)
__global__ void k_fvm_coll_apply(FvmView v, const double* __restrict__ dinv, const double* __restrict__ T,
                                 const double* __restrict__ B, const double* __restrict__ sc, double* __restrict__ Y,
                                 int32_t* bad) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)v.Nr * v.Nvt * v.Nx;
    if (i >= n) return;
    const int x = (int)(i % v.Nx);
    const size_t rj = i / v.Nx;
    if (rj == 0) bad[x] = 0;  // the moments of the next product start clean
    const double y = fvm_coll_apply_at(v, dinv, T, B, (int)(rj / v.Nvt), (int)(rj % v.Nvt), x);
    Y[i] = sc ? y * sc[i] : y;
}

// ---- preconditioner sweeps in the natural (Nr, Nvt, Nx) layout --------------------------------
// An upwind backward-Euler solve (I + a h D) o = b along a line is the recurrence
//   o_i = (b_i - a h sum_k D[i][i -/+ k] o_{i -/+ k}) / (1 + a h D[i][i])
// (bands column-stored: lower D[i][i-k] = L[k][i-k], upper D[i][i+k] = R[k][i+k],
// rawkernel.py:168-375). The lines are few and long (one warp on an SM sub-partition, 64 cycles
// per FP64 instruction), so the chain is cut to its nd - 1 multiply-adds: k_fvm_sweep_coef
// tabulates rho_i = 1 / (1 + a h D[i][i]) and c_k,i = a h D[i][i -/+ k] rho_i once per step, the
// kernel before each sweep (or its load) multiplies b by rho, and the sweep is
//   o_i = b_i - sum_k c_k,i o_{i -/+ k}.
// Along v_r (stride Nvt Nx) and v_theta (stride Nx) the threads of a warp take consecutive x, so
// every step is one coalesced access; x rows are staged in shared memory, their c_k in
// line-fastest order. Against recurrences of five FP64 instructions (200 x 305 x 16): v_r 94 ->
// 30 us, v_theta 35 -> 12 us, x 66 -> 39 us, and no reciprocals per application (37 us).
constexpr int SW_NDMAX = 4;
constexpr int SW_U = 16;  // steps of a long line whose loads are in flight ahead of the chain
constexpr int SW_US = 8;  // of the short v_theta lines, where more resident warps pay instead

// a of the three sweeps' lines and the direction: 0 v_r (a = -aE cos, rawkernel.py:168-230),
// 1 v_theta (a = aE / v_r, sweeping left to right when -a >= 0, :232-296), 2 x (a = ax v_r cos, :298-375)
struct FvmSweep {
    const double *L, *R;
    int nd, N;
};
__device__ inline void sweep_coef(const FvmSweep& d, double ad, bool ltr, int i, double* rho, double c[SW_NDMAX - 1]) {
    const double* B = ltr ? d.L : d.R;
    const double q = 1.0 / (1.0 + ad * B[i]);
    *rho = q;
#pragma unroll
    for (int k = 1; k < SW_NDMAX; ++k) {
        const int o = ltr ? i - k : i + k;
        c[k - 1] = (k < d.nd && o >= 0 && o < d.N) ? ad * B[(size_t)k * d.N + o] * q : 0.0;
    }
}

// Layout of the table (arrays of N values): v_r rho, c_1 .., v_theta rho, c_1 .., x rho, all in the
// natural layout, then the x sweep's c_1 .. at [x][line], line = r Nvt + j. One CTA per (line
// block of 32, x block of 32).
__global__ void __launch_bounds__(256)
k_fvm_sweep_coef(FvmView v, const double* __restrict__ aE, const double* __restrict__ axvr, double h,
                 double* __restrict__ tab) {
    __shared__ double tile[SW_NDMAX - 1][32][33];
    const int nlines = v.Nr * v.Nvt;
    const size_t n = (size_t)nlines * v.Nx;
    const int l0 = blockIdx.x * 32, x0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double* tr = tab;
    double* tt = tr + (size_t)v.ndr * n;
    double* xr = tt + (size_t)v.ndt * n;
    double* xc = xr + n;
    double rho, c[SW_NDMAX - 1];
    for (int l = ty; l < 32; l += 8) {
        const int line = l0 + l, x = x0 + tx;
#pragma unroll
        for (int k = 0; k < SW_NDMAX - 1; ++k) c[k] = 0.0;
        if (line < nlines && x < v.Nx) {
            const int j = line % v.Nvt, r = line / v.Nvt;
            const size_t o = (size_t)line * v.Nx + x;
            double a = -aE[x] * v.cos_t[j];
            sweep_coef(FvmSweep{v.vrL, v.vrR, v.ndr, v.Nr}, a * h, a >= 0.0, r, &rho, c);
            tr[o] = rho;
            for (int k = 1; k < v.ndr; ++k) tr[k * n + o] = c[k - 1];
            a = aE[x] / v.vr[r];
            sweep_coef(FvmSweep{v.vtL, v.vtR, v.ndt, v.Nvt}, a * h, -a >= 0.0, j, &rho, c);
            tt[o] = rho;
            for (int k = 1; k < v.ndt; ++k) tt[k * n + o] = c[k - 1];
            a = axvr[r] * v.cos_t[j];
            sweep_coef(FvmSweep{v.xL, v.xR, v.ndx, v.Nx}, a * h, a >= 0.0, x, &rho, c);
            xr[o] = rho;
        }
#pragma unroll
        for (int k = 0; k < SW_NDMAX - 1; ++k) tile[k][l][tx] = c[k];
    }
    __syncthreads();
    for (int x = ty; x < 32; x += 8)
        if (x0 + x < v.Nx && l0 + tx < nlines)
            for (int k = 1; k < v.ndx; ++k)
                xc[(k - 1) * n + (size_t)(x0 + x) * nlines + l0 + tx] = tile[k - 1][tx][x];
}

// The recurrence along one line of N values spaced `stride`: v in and out (v already times rho
// unless rho is given), c_k at c + k cstep with spacing cstride
template <int ND, int U, bool RHO>
__device__ inline void sweep_line(int N, bool ltr, double* v, long long stride, const double* __restrict__ c,
                                  size_t cstep, long long cstride, const double* __restrict__ rho) {
    double prev[ND > 1 ? ND - 1 : 1];
#pragma unroll
    for (int k = 0; k < ND - 1; ++k) prev[k] = 0.0;
    double nb[U], nc[ND > 1 ? ND - 1 : 1][U], nr[U];
    auto fetch = [&](int s0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int st = min(s0 + u, N - 1);
            const int i = ltr ? st : N - 1 - st;
            nb[u] = v[i * stride];
            if (RHO) nr[u] = rho[i * stride];
#pragma unroll
            for (int k = 0; k < ND - 1; ++k) nc[k][u] = c[k * cstep + i * cstride];
        }
    };
    fetch(0);
    for (int s0 = 0; s0 < N; s0 += U) {
        double b[U], cc[ND > 1 ? ND - 1 : 1][U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            b[u] = RHO ? nb[u] * nr[u] : nb[u];
#pragma unroll
            for (int k = 0; k < ND - 1; ++k) cc[k][u] = nc[k][u];
        }
        if (s0 + U < N) fetch(s0 + U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (s0 + u >= N) break;
            const int i = ltr ? s0 + u : N - 1 - s0 - u;
            double o = b[u];
            // the oldest value first: only the last multiply-add waits for the step before
#pragma unroll
            for (int k = ND - 2; k >= 0; --k) o -= cc[k][u] * prev[k];
#pragma unroll
            for (int k = ND - 2; k > 0; --k) prev[k] = prev[k - 1];
            if (ND > 1) prev[0] = o;
            v[i * stride] = o;
        }
    }
}
template <int U, bool RHO>
__device__ inline void sweep_line_nd(int nd, int N, bool ltr, double* v, long long stride, const double* c, size_t cstep,
                                     long long cstride, const double* rho) {
    if (nd == 1) sweep_line<1, U, RHO>(N, ltr, v, stride, c, cstep, cstride, rho);
    else if (nd == 2) sweep_line<2, U, RHO>(N, ltr, v, stride, c, cstep, cstride, rho);
    else if (nd == 3) sweep_line<3, U, RHO>(N, ltr, v, stride, c, cstep, cstride, rho);
    else sweep_line<4, U, RHO>(N, ltr, v, stride, c, cstep, cstride, rho);
}

// v_r sweep of V (times rho already): line (j, x), one thread each
__global__ void k_fvm_sweep_vr(FvmView v, const double* __restrict__ aE, double* __restrict__ V,
                               const double* __restrict__ c) {
    const int line = blockIdx.x * blockDim.x + threadIdx.x;
    if (line >= v.Nvt * v.Nx) return;
    const int j = line / v.Nx, x = line % v.Nx;
    const long long st = (long long)v.Nvt * v.Nx;
    const double a = -aE[x] * v.cos_t[j];
    sweep_line_nd<SW_U, false>(v.ndr, v.Nr, a >= 0.0, V + line, st, c + line, (size_t)v.Nr * st, st, nullptr);
}

// v_theta sweep: line (r, x), one thread each
__global__ void k_fvm_sweep_vt(FvmView v, const double* __restrict__ aE, double* __restrict__ V,
                               const double* __restrict__ rho, const double* __restrict__ c) {
    const int line = blockIdx.x * blockDim.x + threadIdx.x;
    if (line >= v.Nr * v.Nx) return;
    const int r = line / v.Nx, x = line % v.Nx;
    const size_t o = (size_t)r * v.Nvt * v.Nx + x;
    // the direction -aE / v_r >= 0 without the division (v_r > 0; a quotient that underflows to 0
    // leaves the line as it is in either direction)
    sweep_line_nd<SW_US, true>(v.ndt, v.Nvt, aE[x] <= 0.0, V + o, (long long)v.Nx, c + o, (size_t)v.Nr * v.Nvt * v.Nx,
                        (long long)v.Nx, rho + o);
}

// x sweep with the inflow values zeroed first: line (r, j) is a contiguous row of Nx values; a CTA
// stages `rows` consecutive rows times rho in shared memory with coalesced loads, one thread
// sweeps each row there (row pitch Nx + 1 against bank conflicts), and the block is written back
// coalesced
constexpr int XT_L = 32;       // most rows per CTA
constexpr int XT_T = 128;      // threads per CTA: all load and store, the first `rows` sweep (registers of two CTAs per SM)
__global__ void __launch_bounds__(XT_T, 2) k_fvm_sweep_x(FvmView v, int rows, const double* __restrict__ axvr,
                                                      const double* __restrict__ B, double* __restrict__ Y,
                                                      const double* __restrict__ rho, const double* __restrict__ c) {
    extern __shared__ double buf[];  // [rows][Nx + 1]
    const int Nx = v.Nx, pitch = Nx + 1;
    const int nlines = v.Nr * v.Nvt;
    const int l0 = blockIdx.x * rows;
    const int nl = min(rows, nlines - l0);
    const double* src = B + (size_t)l0 * Nx;
    const double* rs = rho + (size_t)l0 * Nx;
#pragma unroll 4
    for (int e = threadIdx.x; e < nl * Nx; e += blockDim.x) {
        const int l = e / Nx, x = e % Nx;
        const int j = (l0 + l) % v.Nvt;
        const bool inflow = v.north[j] ? (x == 0) : (x == Nx - 1);
        const double y = src[e] * rs[e];
        buf[l * pitch + x] = inflow ? 0.0 : y;
    }
    __syncthreads();
    if (threadIdx.x < nl) {
        const int line = l0 + threadIdx.x;
        const double a = axvr[line / v.Nvt] * v.cos_t[line % v.Nvt];
        sweep_line_nd<SW_U, false>(v.ndx, Nx, a >= 0.0, buf + threadIdx.x * pitch, 1, c + line, (size_t)nlines * Nx,
                             (long long)nlines, nullptr);
    }
    __syncthreads();
    double* dst = Y + (size_t)l0 * Nx;
    for (int e = threadIdx.x; e < nl * Nx; e += blockDim.x) dst[e] = buf[(e / Nx) * pitch + e % Nx];
}

// Y = the semi-Lagrangian advection of V, one thread per value
__global__ void k_fvm_sl(FvmSl sl, const double* __restrict__ E, const double* __restrict__ V, double* __restrict__ Y) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)sl.Nr * sl.Nvt * sl.Nx;
    if (i >= n) return;
    const int x = (int)(i % sl.Nx);
    const size_t rj = i / sl.Nx;
    Y[i] = fvm_sl_at(sl, E, V, (int)(rj / sl.Nvt), (int)(rj % sl.Nvt), x);
}

// y = a x (x may alias y)
__global__ void k_fvm_scale(size_t n, double a, const double* x, double* y) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = a * x[i];
}
__global__ void k_fvm_axpy(size_t n, double a, const double* __restrict__ x, double* __restrict__ y) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += a * x[i];
}
__global__ void k_fvm_sub(size_t n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ c) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) c[i] = a[i] - b[i];
}
// w -= sum_j h_j V_j
__global__ void k_fvm_sub_combo(size_t n, int k, const double* __restrict__ V, const double* __restrict__ h,
                                double* __restrict__ w) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = w[i];
    for (int j = 0; j < k; ++j) s -= h[j] * V[(size_t)j * n + i];
    w[i] = s;
}
// y = sum_j c_j V_j
__global__ void k_fvm_combo(size_t n, int k, const double* __restrict__ V, const double* __restrict__ c,
                            double* __restrict__ y) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    for (int j = 0; j < k; ++j) s += c[j] * V[(size_t)j * n + i];
    y[i] = s;
}
// part[j][block] = partial sums of V_j . w over a fixed grid-stride split
__global__ void k_fvm_dots_partial(size_t n, const double* __restrict__ V, const double* __restrict__ w,
                                   double* __restrict__ part) {
    __shared__ double red[32];
    const int j = blockIdx.y;
    const double* v = V + (size_t)j * n;
    double s = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        s += v[i] * w[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) part[(size_t)j * gridDim.x + blockIdx.x] = s;
}
__global__ void k_fvm_dots_final(int nb, const double* __restrict__ part, double* __restrict__ out) {
    __shared__ double red[32];
    const int j = blockIdx.x;
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) s += part[(size_t)j * nb + i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) out[j] = s;
}

int launched(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return BTE_OK;
    return fvm_fail(BTE_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

int fvm_alloc(bte_fvm* h, void** p, size_t bytes) {
    if (cudaMalloc(p, std::max<size_t>(bytes, 8)) != cudaSuccess) return fvm_fail(BTE_ERR_ALLOC, "device allocation failed");
    h->allocs.push_back(*p);
    return BTE_OK;
}

void fvm_free(bte_fvm* h) {
    for (void* p : h->allocs) cudaFree(p);
    h->allocs.clear();
}

int sweep_rc(int rc, const char* what) {
    if (rc == 0) return BTE_OK;
    return fvm_fail(BTE_ERR_CUDA, std::string(what) + ": " + bte_sweep_last_error());
}

// the coefficients of rhs_mvec for a step at field E
int fvm_mvec_coef(bte_fvm* h, const FvmCoef& c, const double* E, cudaStream_t s) {
    const size_t m = std::max((size_t)h->Nr * h->Nvt, (size_t)h->Nx);
    k_fvm_mvec_coef<<<fblocks(m), FT, 0, s>>>(view_of(h), c, E, h->bx, h->arc, h->lr, h->eflag);
    ++h->launches;
    return launched("k_fvm_mvec_coef");
}

// Y = rhs_mvec(X) on stream s (fvm_mvec_coef done)
int fvm_mvec(bte_fvm* h, const FvmCoef& c, const double* X, double* Y, cudaStream_t s) {
    const FvmView v = view_of(h);
    const size_t nrx = (size_t)h->Nr * h->Nx;
    k_fvm_moment<<<fblocks(nrx), FT, 0, s>>>(v, X, h->M, h->bad);
    if (int rc = launched("k_fvm_moment")) return rc;
    k_fvm_gain<<<fblocks(nrx), FT, 0, s>>>(h->Nr, h->Nx, c.dt * c.tau * c.kappa, h->gptr, h->gcol, h->gval, h->M, h->bad,
                                           h->T);
    if (int rc = launched("k_fvm_gain")) return rc;
    k_fvm_mvec<<<fblocks(h->N), FT, 0, s>>>(v, h->bx, h->arc, h->lr, h->vinv, h->eflag, h->cpos, h->T, X, Y, h->bad);
    h->launches += 3;
    return launched("k_fvm_mvec");
}

// T = H (moments of X)
int fvm_hmul(bte_fvm* h, const double* X, cudaStream_t s) {
    const int Nr = h->Nr, Nx = h->Nx;
    k_fvm_moment<<<fblocks((size_t)Nr * Nx), FT, 0, s>>>(view_of(h), X, h->M, h->bad);
    if (int rc = launched("k_fvm_moment")) return rc;
    const int words = ((Nr + HC - 1) / HC + 31) / 32;
    k_fvm_hmul<<<dim3((unsigned)((Nx + 31) / 32), (unsigned)((Nr + HR - 1) / HR)), 128, 0, s>>>(Nr, Nx, words, h->hmask,
                                                                                            h->H, h->M, h->bad, h->T);
    h->launches += 2;
    return launched("k_fvm_hmul");
}

// rows per CTA of the x sweep: two CTAs per SM where the lines allow it, as many rows as fit in
// 200 KB; 0 when not even four do
int sweep_x_rows(const bte_fvm* h) {
    const int lines = h->Nr * h->Nvt;
    const int fit = (int)(200 * 1024 / ((size_t)(h->Nx + 1) * sizeof(double)));
    const int want = std::max(4, (lines + 2 * 152 - 1) / (2 * 152));
    const int rows = std::min(std::min(XT_L, fit), want);
    return rows >= 4 ? rows : 0;
}

// the sweeps that run on the natural layout: stencils up to SW_NDMAX points, x rows that fit
bool natural_sweeps(const bte_fvm* h) {
    return h->ndr <= SW_NDMAX && h->ndt <= SW_NDMAX && h->ndx <= SW_NDMAX && sweep_x_rows(h) > 0;
}

// The sweep coefficients (5 N to 12 N values) only make the sweeps faster, so they never take the room of
// something that has to be there: they are allocated when the longest Krylov basis (501 N) would still fit
// beside them, and without them the sweeps run on permuted copies.
void fvm_alloc_sweep_coef(bte_fvm* h) {
    if (h->swc || !natural_sweeps(h)) return;
    const size_t bytes = (size_t)(h->ndr + h->ndt + h->ndx) * h->N * sizeof(double);
    size_t room = 0, all = 0;
    if (cudaMemGetInfo(&room, &all) != cudaSuccess || room < bytes + (size_t)501 * h->N * sizeof(double) ||
        fvm_alloc(h, (void**)&h->swc, bytes) != BTE_OK) {
        h->swc = nullptr;
        cudaGetLastError();
    }
}

// the sweep coefficients for step h at the coefficients in h->aE, h->axvr
int fvm_sweep_coef(bte_fvm* h, double hstep, cudaStream_t s) {
    if (!h->swc) return BTE_OK;
    // x rows that fit in shared memory are short; the lines can be more than a grid's 65535 x 32 rows
    const dim3 grid((unsigned)((h->Nr * h->Nvt + 31) / 32), (unsigned)((h->Nx + 31) / 32));
    k_fvm_sweep_coef<<<grid, 256, 0, s>>>(view_of(h), h->aE, h->axvr, hstep, h->swc);
    ++h->launches;
    return launched("k_fvm_sweep_coef");
}

// Y = the op-split step applied to X (aE = cE E must already be in h->aE, ax v_r in h->axvr, and
// the sweep coefficients of hstep tabulated)
int fvm_precond(bte_fvm* h, double hstep, const double* X, double* Y, cudaStream_t s) {
    const FvmView v = view_of(h);
    const int Nr = h->Nr, Nvt = h->Nvt, Nx = h->Nx;
    if (int rc = fvm_hmul(h, X, s)) return rc;
    if (!h->swc) {
        // stencils wider than the register recurrence, x lines longer than the staged rows or no room for
        // the coefficients: the drop-in sweeps on permuted copies
        k_fvm_coll_permute<<<fblocks(h->N), FT, 0, s>>>(v, h->dinv, h->T, X, h->A, h->bad);   // (Nx, Nvt, Nr)
        if (int rc = launched("k_fvm_coll_permute")) return rc;
        int rc = sweep_rc(bte_adv_be_sweep(0, h->vrL, h->vrR, h->aE, h->cos_t, hstep, h->A, h->Bf, h->ndr, Nr, Nvt, Nx, s),
                          "v_r sweep");
        if (!rc) rc = sweep_rc(bte_permute3(Nx, Nvt, Nr, 0, 2, 1, h->Bf, h->A, s), "layout");   // (Nx, Nr, Nvt)
        if (!rc)
            rc = sweep_rc(bte_adv_be_sweep(1, h->vtL, h->vtR, h->aE, h->vr, hstep, h->A, h->Bf, h->ndt, Nr, Nvt, Nx, s),
                          "v_theta sweep");
        if (!rc) rc = sweep_rc(bte_permute3(Nx, Nr, Nvt, 1, 2, 0, h->Bf, h->A, s), "layout");   // (Nr, Nvt, Nx)
        if (!rc) rc = sweep_rc(bte_fvm_inflow_zero(Nr, Nvt, Nx, h->vt, h->A, s), "inflow");
        if (!rc)
            rc = sweep_rc(bte_adv_be_sweep(2, h->xL, h->xR, h->axvr, h->cos_t, hstep, h->A, Y, h->ndx, Nr, Nvt, Nx, s),
                          "x sweep");
        h->launches += 8;
        return rc;
    }
    const size_t n = h->N;
    const double* tr = h->swc;
    const double* tt = tr + (size_t)h->ndr * n;
    const double* xr = tt + (size_t)h->ndt * n;
    k_fvm_coll_apply<<<fblocks(n), FT, 0, s>>>(v, h->dinv, h->T, X, tr, h->A, h->bad);
    if (int rc = launched("k_fvm_coll_apply")) return rc;
    // the v_r lines are few (Nvt Nx) and long: CTAs of one warp spread them over the SMs
    k_fvm_sweep_vr<<<(unsigned)(((size_t)Nvt * Nx + 31) / 32), 32, 0, s>>>(v, h->aE, h->A, tr + n);
    if (int rc = launched("k_fvm_sweep_vr")) return rc;
    k_fvm_sweep_vt<<<(unsigned)(((size_t)Nr * Nx + 127) / 128), 128, 0, s>>>(v, h->aE, h->A, tt, tt + n);
    if (int rc = launched("k_fvm_sweep_vt")) return rc;
    const int rows = sweep_x_rows(h);
    const size_t xsm = (size_t)rows * (Nx + 1) * sizeof(double);
    if (bte_raise_smem_limit((const void*)k_fvm_sweep_x, xsm) != cudaSuccess)
        return fvm_fail(BTE_ERR_CUDA, "x sweep: shared-memory limit");
    k_fvm_sweep_x<<<(unsigned)((Nr * Nvt + rows - 1) / rows), XT_T, xsm, s>>>(v, rows, h->axvr, h->A, Y, xr, xr + n);
    h->launches += 4;
    return launched("k_fvm_sweep_x");
}

// aE = cE E on the device, axvr = ax v_r
int fvm_coefficients(bte_fvm* h, double cE, double ax, const double* E, cudaStream_t s) {
    k_fvm_scale<<<fblocks(h->Nx), FT, 0, s>>>((size_t)h->Nx, cE, E, h->aE);
    k_fvm_scale<<<fblocks(h->Nr), FT, 0, s>>>((size_t)h->Nr, ax, h->vr, h->axvr);
    h->launches += 2;
    return launched("coefficients");
}

FvmSl sl_of(const bte_fvm* h, const FvmCoef& c) {
    FvmSl sl;
    sl.Nr = h->Nr; sl.Nvt = h->Nvt; sl.Nx = h->Nx;
    sl.vr = h->vr; sl.vt = h->vt; sl.cos_t = h->cos_t; sl.vrp = h->vrp; sl.vta = h->vta; sl.x = h->xg;
    sl.vmin = h->sl_vmin;
    sl.cX = c.dt * c.ax;
    sl.cE = c.dt * c.tau * c.cA;
    return sl;
}

// Y = step_adv_vx_sl(V) (Y must not alias V)
int fvm_sl(bte_fvm* h, const FvmCoef& c, const double* E, const double* V, double* Y, cudaStream_t s) {
    k_fvm_sl<<<fblocks(h->N), FT, 0, s>>>(sl_of(h, c), E, V, Y);
    ++h->launches;
    return launched("k_fvm_sl");
}

// Y = (I - c C)^-1 B in the natural layout (Y must not alias B)
int fvm_coll_solve(bte_fvm* h, const double* B, double* Y, cudaStream_t s) {
    if (int rc = fvm_hmul(h, B, s)) return rc;
    k_fvm_coll_apply<<<fblocks(h->N), FT, 0, s>>>(view_of(h), h->dinv, h->T, B, nullptr, Y, h->bad);
    ++h->launches;
    return launched("k_fvm_coll_apply");
}

struct DeviceOps {
    bte_fvm* h;
    cudaStream_t s;
    FvmCoef c;
    double hstep;
    size_t N;
    double *B, *X, *R, *W, *Z, *T, *Kr;
    bool identity;   // pc_type "none": no preconditioner

    int matvec(const double* x, double* y) { return fvm_mvec(h, c, x, y, s); }
    int precond(const double* x, double* y) {
        if (!identity) return fvm_precond(h, hstep, x, y, s);
        if (cudaMemcpyAsync(y, x, N * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
            return fvm_fail(BTE_ERR_CUDA, "copy failed");
        return BTE_OK;
    }
    // k products into hd, and from there to pinned memory
    int queue_dots(int k, const double* V, const double* w, double* pinned) {
        k_fvm_dots_partial<<<dim3(FVM_RED, k), FT, 0, s>>>(N, V, w, h->part);
        k_fvm_dots_final<<<k, FT, 0, s>>>(FVM_RED, h->part, h->hd);
        h->launches += 2;
        if (int rc = launched("dots")) return rc;
        if (cudaMemcpyAsync(pinned, h->hd, (size_t)k * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess)
            return fvm_fail(BTE_ERR_CUDA, "dots: copy to the host failed");
        return BTE_OK;
    }
    int wait() {
        return cudaStreamSynchronize(s) == cudaSuccess ? BTE_OK : fvm_fail(BTE_ERR_CUDA, "dots: copy to the host failed");
    }
    int dots(int k, const double* V, const double* w, double* out) {
        if (int rc = queue_dots(k, V, w, h->hp)) return rc;
        if (int rc = wait()) return rc;
        std::copy(h->hp, h->hp + k, out);
        return BTE_OK;
    }
    // Both passes of Gram-Schmidt and the norm queued at once: the combinations take their
    // coefficients from hd, where the products left them, and the host waits once (it waited for
    // each of the three reductions and sent the coefficients back).
    int orthogonalize(int k, double* w, double* h0, double* h1, double* ww) {
        double* hp1 = h->hp + h->kcap + 1;
        double* hp2 = hp1 + h->kcap + 1;
        for (int pass = 0; pass < 2; ++pass) {
            if (int rc = queue_dots(k, Kr, w, pass == 0 ? h->hp : hp1)) return rc;
            k_fvm_sub_combo<<<fblocks(N), FT, 0, s>>>(N, k, Kr, h->hd, w);
            ++h->launches;
            if (int rc = launched("sub_combo")) return rc;
        }
        if (int rc = queue_dots(1, w, w, hp2)) return rc;
        if (int rc = wait()) return rc;
        std::copy(h->hp, h->hp + k, h0);
        std::copy(hp1, hp1 + k, h1);
        *ww = *hp2;
        return BTE_OK;
    }
    int to_device(int k, const double* host) {
        if (cudaMemcpyAsync(h->hd, host, (size_t)k * 8, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return fvm_fail(BTE_ERR_CUDA, "coefficient copy failed");
        return BTE_OK;
    }
    int combo(int k, const double* V, const double* cc, double* y) {
        if (int rc = to_device(k, cc)) return rc;
        k_fvm_combo<<<fblocks(N), FT, 0, s>>>(N, k, V, h->hd, y);
        ++h->launches;
        return launched("combo");
    }
    int scale(double a, const double* x, double* y) {
        k_fvm_scale<<<fblocks(N), FT, 0, s>>>(N, a, x, y);
        ++h->launches;
        return launched("scale");
    }
    int axpy(double a, const double* x, double* y) {
        k_fvm_axpy<<<fblocks(N), FT, 0, s>>>(N, a, x, y);
        ++h->launches;
        return launched("axpy");
    }
    int sub(const double* a, const double* b, double* cc) {
        k_fvm_sub<<<fblocks(N), FT, 0, s>>>(N, a, b, cc);
        ++h->launches;
        return launched("sub");
    }
};

bool coef_ok(const bte_fvm_coef* c) {
    return c && std::isfinite(c->dt) && std::isfinite(c->dtx) && std::isfinite(c->tau) && std::isfinite(c->kappa) &&
           std::isfinite(c->cA) && std::isfinite(c->ax);
}

FvmCoef coef_of(const bte_fvm_coef* c) {
    FvmCoef f;
    f.dt = c->dt; f.dtx = c->dtx; f.tau = c->tau; f.kappa = c->kappa; f.cA = c->cA; f.ax = c->ax;
    return f;
}

}  // namespace

extern "C" {

const char* bte_fvm_last_error(void) { return g_fvm_err.c_str(); }

int bte_fvm_create(int device, int Nr, int Nvt, int Nx, int ndr, int ndt, int ndx, const double* vr, const double* vt,
                   const double* w, const double* loss, const double* gain, const double* vr_l2r,
                   const double* vr_r2l, const double* vt_l2r, const double* vt_r2l, const double* x_l2r,
                   const double* x_r2l, bte_fvm** out) {
    if (!out) return fvm_fail(BTE_ERR_ARG, "bte_fvm_create: null handle pointer");
    *out = nullptr;
    if (!vr || !vt || !w || !loss || !gain || !vr_l2r || !vr_r2l || !vt_l2r || !vt_r2l || !x_l2r || !x_r2l)
        return fvm_fail(BTE_ERR_ARG, "bte_fvm_create: null argument");
    if (Nr < 2 || Nvt < 2 || (Nvt & 1) || Nx < 2 || ndr < 1 || ndt < 1 || ndx < 1 || ndr > Nr || ndt > Nvt || ndx > Nx)
        return fvm_fail(BTE_ERR_ARG, "bte_fvm_create: sizes out of range (Nr, Nx >= 2, Nvt even >= 2, 1 <= nd <= N)");
    const size_t N = (size_t)Nr * Nvt * Nx;
    if (N > ((size_t)1 << 31)) return fvm_fail(BTE_ERR_ARG, "bte_fvm_create: Nr * Nvt * Nx above 2^31");
    for (int r = 0; r < Nr; ++r)
        if (!(vr[r] > 0.0)) return fvm_fail(BTE_ERR_ARG, "bte_fvm_create: cell centres must be positive");
    if (cudaSetDevice(device) != cudaSuccess) return fvm_fail(BTE_ERR_CUDA, "cudaSetDevice failed");
    bte_fvm* h = new bte_fvm();
    h->device = device; h->Nr = Nr; h->Nvt = Nvt; h->Nx = Nx; h->ndr = ndr; h->ndt = ndt; h->ndx = ndx; h->N = N;
    int rc = BTE_OK;
    auto A = [&](double** p, size_t count) { if (rc == BTE_OK) rc = fvm_alloc(h, (void**)p, count * 8); };
    A(&h->vr, Nr); A(&h->vt, Nvt); A(&h->cos_t, Nvt); A(&h->w, Nvt); A(&h->loss, Nr); A(&h->gain, (size_t)Nr * Nr);
    A(&h->vrL, (size_t)ndr * Nr); A(&h->vrR, (size_t)ndr * Nr); A(&h->vtL, (size_t)ndt * Nvt);
    A(&h->vtR, (size_t)ndt * Nvt); A(&h->xL, (size_t)ndx * Nx); A(&h->xR, (size_t)ndx * Nx);
    A(&h->dinv, Nr); A(&h->H, (size_t)Nr * Nr);
    A(&h->M, (size_t)Nr * Nx); A(&h->T, (size_t)Nr * Nx); A(&h->aE, Nx); A(&h->axvr, Nr);
    A(&h->bx, Nx); A(&h->arc, (size_t)Nr * Nvt); A(&h->lr, Nr); A(&h->vinv, Nr);
    // the gain matrix by rows; the scattered entries of at most two per process and row
    std::vector<int32_t> gptr(1, 0), gcol;
    std::vector<double> gval;
    for (int r = 0; r < Nr; ++r) {
        for (int k = 0; k < Nr; ++k)
            if (gain[(size_t)r * Nr + k] != 0.0) {
                gcol.push_back(k);
                gval.push_back(gain[(size_t)r * Nr + k]);
            }
        gptr.push_back((int32_t)gcol.size());
    }
    const size_t hwords = (size_t)((Nr + HR - 1) / HR) * (((Nr + HC - 1) / HC + 31) / 32);
    auto Ab = [&](void** p, size_t bytes) { if (rc == BTE_OK) rc = fvm_alloc(h, p, bytes); };
    Ab((void**)&h->eflag, Nx); Ab((void**)&h->cpos, Nvt); Ab((void**)&h->gptr, gptr.size() * 4);
    Ab((void**)&h->gcol, gcol.size() * 4); Ab((void**)&h->gval, gval.size() * 8);
    Ab((void**)&h->hmask, hwords * 4); Ab((void**)&h->bad, (size_t)Nx * 4);
    A(&h->A, N); A(&h->Bf, N); A(&h->B, N); A(&h->X, N); A(&h->R, N); A(&h->W, N); A(&h->Z, N); A(&h->Tv, N);
    if (rc == BTE_OK) rc = fvm_alloc(h, (void**)&h->north, Nvt);
    if (rc != BTE_OK) {
        fvm_free(h);
        delete h;
        return rc;
    }
    std::vector<double> cth(Nvt);
    std::vector<int8_t> north(Nvt), cpos(Nvt);
    std::vector<double> vinv(Nr);
    std::vector<int32_t> zero((size_t)Nx, 0);
    for (int r = 0; r < Nr; ++r) vinv[r] = 1.0 / vr[r];
    const double half_pi = 0.5 * 3.14159265358979323846;
    for (int j = 0; j < Nvt; ++j) {
        cth[j] = std::cos(vt[j]);
        north[j] = vt[j] <= half_pi ? 1 : 0;
        cpos[j] = cth[j] > 0.0 ? 1 : 0;
    }
    struct Cp { void* d; const void* s; size_t b; };
    const Cp cps[] = {{h->vr, vr, (size_t)Nr * 8}, {h->vt, vt, (size_t)Nvt * 8}, {h->cos_t, cth.data(), (size_t)Nvt * 8},
                      {h->w, w, (size_t)Nvt * 8}, {h->loss, loss, (size_t)Nr * 8}, {h->gain, gain, (size_t)Nr * Nr * 8},
                      {h->vrL, vr_l2r, (size_t)ndr * Nr * 8}, {h->vrR, vr_r2l, (size_t)ndr * Nr * 8},
                      {h->vtL, vt_l2r, (size_t)ndt * Nvt * 8}, {h->vtR, vt_r2l, (size_t)ndt * Nvt * 8},
                      {h->xL, x_l2r, (size_t)ndx * Nx * 8}, {h->xR, x_r2l, (size_t)ndx * Nx * 8},
                      {h->north, north.data(), (size_t)Nvt}, {h->cpos, cpos.data(), (size_t)Nvt},
                      {h->vinv, vinv.data(), (size_t)Nr * 8}, {h->gptr, gptr.data(), gptr.size() * 4},
                      {h->gcol, gcol.data(), gcol.size() * 4}, {h->gval, gval.data(), gval.size() * 8},
                      {h->bad, zero.data(), (size_t)Nx * 4}};
    for (const Cp& c : cps)
        if (c.b && cudaMemcpy(c.d, c.s, c.b, cudaMemcpyHostToDevice) != cudaSuccess) {
            fvm_free(h);
            delete h;
            return fvm_fail(BTE_ERR_CUDA, "bte_fvm_create: copy of the set-up failed");
        }
    *out = h;
    return BTE_OK;
}

int bte_fvm_destroy(bte_fvm* h) {
    if (!h) return BTE_OK;
    cudaSetDevice(h->device);
    cudaFree(h->Kr);   // the GMRES buffers, sized by the largest restart so far
    cudaFree(h->part);
    cudaFree(h->hd);
    cudaFreeHost(h->hp);
    fvm_free(h);
    delete h;
    return BTE_OK;
}

long long bte_fvm_launches(const bte_fvm* h) { return h ? h->launches : 0; }

int bte_fvm_set_collision_inverse(bte_fvm* h, const double* dinv, const double* H) {
    if (!h || !dinv || !H) return fvm_fail(BTE_ERR_ARG, "bte_fvm_set_collision_inverse: null argument");
    cudaSetDevice(h->device);
    fvm_alloc_sweep_coef(h);
    const int Nr = h->Nr, words = ((Nr + HC - 1) / HC + 31) / 32;
    std::vector<uint32_t> mask((size_t)((Nr + HR - 1) / HR) * words, 0u);
    for (int r = 0; r < Nr; ++r)
        for (int k = 0; k < Nr; ++k)
            if (H[(size_t)r * Nr + k] != 0.0) mask[(size_t)(r / HR) * words + k / HC / 32] |= 1u << (k / HC % 32);
    if (cudaMemcpy(h->dinv, dinv, (size_t)h->Nr * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->H, H, (size_t)h->Nr * h->Nr * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->hmask, mask.data(), mask.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess)
        return fvm_fail(BTE_ERR_CUDA, "bte_fvm_set_collision_inverse: copy failed");
    h->have_inverse = true;
    return BTE_OK;
}

int bte_fvm_mvec(bte_fvm* h, const bte_fvm_coef* c, const double* E, const double* X, double* Y, void* stream) {
    if (!h || !E || !X || !Y) return fvm_fail(BTE_ERR_ARG, "bte_fvm_mvec: null argument");
    if (!coef_ok(c)) return fvm_fail(BTE_ERR_ARG, "bte_fvm_mvec: coefficients missing or not finite");
    if (X == Y) return fvm_fail(BTE_ERR_ARG, "bte_fvm_mvec: Y must not alias X");
    cudaSetDevice(h->device);
    if (int rc = fvm_mvec_coef(h, coef_of(c), E, (cudaStream_t)stream)) return rc;
    return fvm_mvec(h, coef_of(c), X, Y, (cudaStream_t)stream);
}

int bte_fvm_precond(bte_fvm* h, double cE, double ax, double hstep, const double* E, const double* X, double* Y,
                    void* stream) {
    if (!h || !E || !X || !Y) return fvm_fail(BTE_ERR_ARG, "bte_fvm_precond: null argument");
    if (!h->have_inverse) return fvm_fail(BTE_ERR_STATE, "bte_fvm_precond: no collision inverse set");
    if (X == Y || X == h->A || X == h->Bf) return fvm_fail(BTE_ERR_ARG, "bte_fvm_precond: Y must not alias X");
    cudaSetDevice(h->device);
    cudaStream_t s = (cudaStream_t)stream;
    if (int rc = fvm_coefficients(h, cE, ax, E, s)) return rc;
    if (int rc = fvm_sweep_coef(h, hstep, s)) return rc;
    return fvm_precond(h, hstep, X, Y, s);
}

int bte_fvm_set_sl_grid(bte_fvm* h, const double* x, double vmin, double vmax) {
    if (!h || !x) return fvm_fail(BTE_ERR_ARG, "bte_fvm_set_sl_grid: null argument");
    const int Nr = h->Nr, Nvt = h->Nvt, Nx = h->Nx;
    std::vector<double> hv(Nvt);
    if (cudaSetDevice(h->device) != cudaSuccess ||
        cudaMemcpy(hv.data(), h->vt, (size_t)Nvt * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
        return fvm_fail(BTE_ERR_CUDA, "bte_fvm_set_sl_grid: copy failed");
    std::vector<double> hr(Nr);
    if (cudaMemcpy(hr.data(), h->vr, (size_t)Nr * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
        return fvm_fail(BTE_ERR_CUDA, "bte_fvm_set_sl_grid: copy failed");
    const double pi = 3.14159265358979323846;
    std::vector<double> vrp(Nr + 2), vta(Nvt + 2);
    vrp[0] = vmin;
    vrp[Nr + 1] = vmax;
    for (int r = 0; r < Nr; ++r) vrp[r + 1] = hr[r];
    vta[0] = 0.0;
    vta[Nvt + 1] = pi;
    for (int j = 0; j < Nvt; ++j) vta[j + 1] = hv[Nvt - 1 - j];
    bool ascending = true;
    for (int i = 0; i + 1 < Nr + 2; ++i) ascending = ascending && vrp[i] < vrp[i + 1];
    for (int i = 0; i + 1 < Nvt + 2; ++i) ascending = ascending && vta[i] < vta[i + 1];
    for (int i = 0; i + 1 < Nx; ++i) ascending = ascending && x[i] < x[i + 1];
    if (!ascending)
        return fvm_fail(BTE_ERR_ARG, "bte_fvm_set_sl_grid: need vmin < vr < vmax, ordinates in (0, pi) descending, x ascending");
    int rc = BTE_OK;
    if (!h->have_sl) {
        if (rc == BTE_OK) rc = fvm_alloc(h, (void**)&h->xg, (size_t)Nx * 8);
        if (rc == BTE_OK) rc = fvm_alloc(h, (void**)&h->vrp, (size_t)(Nr + 2) * 8);
        if (rc == BTE_OK) rc = fvm_alloc(h, (void**)&h->vta, (size_t)(Nvt + 2) * 8);
        if (rc != BTE_OK) return rc;
    }
    if (cudaMemcpy(h->xg, x, (size_t)Nx * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->vrp, vrp.data(), (size_t)(Nr + 2) * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->vta, vta.data(), (size_t)(Nvt + 2) * 8, cudaMemcpyHostToDevice) != cudaSuccess)
        return fvm_fail(BTE_ERR_CUDA, "bte_fvm_set_sl_grid: copy failed");
    h->sl_vmin = vmin;
    h->have_sl = true;
    return BTE_OK;
}

int bte_fvm_sl_advect(bte_fvm* h, const bte_fvm_coef* c, const double* E, const double* V, double* Y, void* stream) {
    if (!h || !E || !V || !Y) return fvm_fail(BTE_ERR_ARG, "bte_fvm_sl_advect: null argument");
    if (!coef_ok(c)) return fvm_fail(BTE_ERR_ARG, "bte_fvm_sl_advect: coefficients missing or not finite");
    if (!h->have_sl) return fvm_fail(BTE_ERR_STATE, "bte_fvm_sl_advect: no semi-Lagrangian grid set");
    if (V == Y) return fvm_fail(BTE_ERR_ARG, "bte_fvm_sl_advect: Y must not alias V");
    cudaSetDevice(h->device);
    return fvm_sl(h, coef_of(c), E, V, Y, (cudaStream_t)stream);
}

int bte_fvm_sl_step(bte_fvm* h, const bte_fvm_coef* c, const double* E, const double* V, double* Y, void* stream) {
    if (!h || !E || !V || !Y) return fvm_fail(BTE_ERR_ARG, "bte_fvm_sl_step: null argument");
    if (!coef_ok(c)) return fvm_fail(BTE_ERR_ARG, "bte_fvm_sl_step: coefficients missing or not finite");
    if (!h->have_sl) return fvm_fail(BTE_ERR_STATE, "bte_fvm_sl_step: no semi-Lagrangian grid set");
    if (!h->have_inverse) return fvm_fail(BTE_ERR_STATE, "bte_fvm_sl_step: no collision inverse set");
    if (V == Y || V == h->A || Y == h->A) return fvm_fail(BTE_ERR_ARG, "bte_fvm_sl_step: Y must not alias V");
    cudaSetDevice(h->device);
    cudaStream_t s = (cudaStream_t)stream;
    if (int rc = fvm_sl(h, coef_of(c), E, V, h->A, s)) return rc;
    return fvm_coll_solve(h, h->A, Y, s);
}

int bte_fvm_step(bte_fvm* h, const bte_fvm_coef* c, double alpha, int pc_mode, const double* E, double* V, double rtol,
                 double atol, int restart, int max_iter, double* info4, void* stream) {
    if (!h || !E || !V || !info4) return fvm_fail(BTE_ERR_ARG, "bte_fvm_step: null argument");
    if (!coef_ok(c) || !std::isfinite(alpha)) return fvm_fail(BTE_ERR_ARG, "bte_fvm_step: coefficients not finite");
    if (restart < 1 || restart > 500 || max_iter < 0) return fvm_fail(BTE_ERR_ARG, "bte_fvm_step: 1 <= restart <= 500");
    if (pc_mode < 0 || pc_mode > 2) return fvm_fail(BTE_ERR_ARG, "bte_fvm_step: pc_mode must be 0, 1 or 2");
    if (pc_mode != 2 && !h->have_inverse) return fvm_fail(BTE_ERR_STATE, "bte_fvm_step: no collision inverse set");
    cudaSetDevice(h->device);
    cudaStream_t s = (cudaStream_t)stream;
    const size_t N = h->N;
    if (restart > h->kcap) {
        double *Kr = nullptr, *part = nullptr, *hd = nullptr, *hp = nullptr;
        if (cudaMalloc((void**)&Kr, (size_t)(restart + 1) * N * 8) != cudaSuccess)
            return fvm_fail(BTE_ERR_ALLOC, "bte_fvm_step: Krylov basis allocation failed");
        if (cudaMalloc((void**)&part, (size_t)(restart + 1) * FVM_RED * 8) != cudaSuccess ||
            cudaMalloc((void**)&hd, (size_t)(restart + 1) * 8) != cudaSuccess ||
            cudaMallocHost((void**)&hp, (size_t)(2 * (restart + 1) + 1) * 8) != cudaSuccess) {
            cudaFree(Kr);
            cudaFree(part);
            cudaFree(hd);
            return fvm_fail(BTE_ERR_ALLOC, "bte_fvm_step: reduction buffers allocation failed");
        }
        if (h->Kr) {
            cudaFree(h->Kr);
            cudaFree(h->part);
            cudaFree(h->hd);
            cudaFreeHost(h->hp);
        }
        h->Kr = Kr;
        h->part = part;
        h->hd = hd;
        h->hp = hp;
        h->kcap = restart;
    }
    const FvmCoef fc = coef_of(c);
    if (int rc = fvm_coefficients(h, fc.tau * fc.cA, fc.ax, E, s)) return rc;
    if (int rc = fvm_mvec_coef(h, fc, E, s)) return rc;
    if (pc_mode != 2)
        if (int rc = fvm_sweep_coef(h, alpha * fc.dt, s)) return rc;
    // right-hand side: V with its inflow values zeroed (bte_1d3v_solver.py:1907-1911)
    if (cudaMemcpyAsync(h->B, V, N * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
        return fvm_fail(BTE_ERR_CUDA, "bte_fvm_step: copy of the state failed");
    if (int rc = sweep_rc(bte_fvm_inflow_zero(h->Nr, h->Nvt, h->Nx, h->vt, h->B, s), "inflow")) return rc;
    DeviceOps op{h, s, fc, alpha * fc.dt, N, h->B, h->X, h->R, h->W, h->Z, h->Tv, h->Kr, pc_mode == 2};
    FvmGmresInfo info{};
    if (int rc = pc_mode == 1 ? fvm_gmres_left(op, restart, rtol, atol, max_iter, &info)
                              : fvm_gmres(op, restart, rtol, atol, max_iter, &info))
        return rc;
    if (cudaMemcpyAsync(V, h->X, N * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return fvm_fail(BTE_ERR_CUDA, "bte_fvm_step: copy of the solution failed");
    info4[0] = info.iterations;
    info4[1] = info.rnorm;
    info4[2] = info.bnorm > 0.0 ? info.rnorm / info.bnorm : 0.0;
    info4[3] = info.converged ? 0.0 : 1.0;
    return BTE_OK;
}

}  // extern "C"
