// Forms of the substitution kernel k_lu_solve (lu.cu) and the order of its diagonal blocks: which
// form a size takes, which warp owns a block, and which named barrier publishes it. Plain C++, so that
// the CPU tests walk the same sequence of barriers.
#pragma once

// bytes per load (a block is 8 loads wide), most threads and least CTAs per SM (launch bounds), groups of
// 32 rows per warp
struct SolveForm {
    int bytes, nt_max, occ, rows;
};
constexpr SolveForm SOLVE_FORMS[] = {{16, 256, 2, 1}, {16, 512, 1, 1}, {16, 256, 3, 2},
                                     {16, 512, 1, 2}, {16, 512, 1, 3}, {8, 512, 1, 4}};
constexpr int SOLVE_MAX_N = 2048;

// The form for P matrices of size N (up to SOLVE_MAX_N). Few matrices (at most two per SM) are bound by the chain of
// diagonal blocks: one group per warp, the next block's loads in registers (N = 385, 137
// matrices: 43 us in FP32 against 55 with two groups per warp and loads when used). More
// matrices than that hide one another's loads, and more resident CTAs pay: two groups per warp
// without the prefetch registers (N = 385, 4096 matrices: 705 us against 984 in FP32, 2822
// against 4161 in FP64). The third CTA per SM is worth the registers that it makes spill (with two 828 us in
// FP32, 3131 in FP64). Up to N = 256 the prefetching form has one group per warp and two
// CTAs per SM and is the faster one for any P (N = 129, 4096 matrices: 146 us against 163). Above
// N = 1400 the diagonal blocks of 16-byte loads no longer fit in shared memory.
constexpr int solve_form(int P, int N) {
    return N <= 256 ? 0 : N <= 512 ? (P <= 304 ? 1 : 2) : N <= 1024 ? 3 : N <= 1400 ? 4 : 5;
}
constexpr int solve_block_width(const SolveForm& f, int elem) { return 8 * f.bytes / elem; }
// as many warps as hold all groups of 32 rows; group w + i NW belongs to warp w
constexpr int solve_warps(const SolveForm& f, int N) { return ((N + 31) / 32 + f.rows - 1) / f.rows; }
constexpr int solve_owner(int block, int width, int warps) { return block * width / 32 % warps; }

// The owner of a block arrives at its barrier and goes on, every other warp waits there. A group's owner
// arrives for 32 / width blocks in a row (1, 2 or 4) before it waits itself, so it meets the next barrier while
// another warp may not have come to the first of them: the barriers must not repeat within
// 32 / width + 1 blocks, or the owner would be counted twice in one of them and open it early.
constexpr int SOLVE_BARRIERS = 8;
constexpr int solve_barrier(int step) { return 1 + step % SOLVE_BARRIERS; }
