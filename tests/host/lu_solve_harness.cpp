// Host build of the substitution's form rule and barrier order (boltzmann_gb300/csrc/lu_solve_form.h):
// out = {width of a diagonal block, warps, barriers}; steps of a sweep with their owner and barrier.
#include "../../boltzmann_gb300/csrc/lu_solve_form.h"

extern "C" void solve_shape(int elem, int P, int N, int* out) {
    const SolveForm f = SOLVE_FORMS[solve_form(P, N)];
    out[0] = solve_block_width(f, elem);
    out[1] = solve_warps(f, N);
    out[2] = f.nt_max / 32;
    out[3] = f.rows;
}
extern "C" int solve_step_owner(int block, int width, int warps) { return solve_owner(block, width, warps); }
extern "C" int solve_step_barrier(int step) { return solve_barrier(step); }
