// chol_core.cuh -- the batched Cholesky solve in shared memory, shared by
// chol.cu (magma_?potrs_batched) and ir.cu (the corrections of the
// mixed-precision SPD refinement).
#pragma once
#include "common.cuh"
#include "solve_core.cuh"

namespace mlu {

// Solves L L^T X = B for the nr right-hand sides in shared memory (column c at
// sB + c * ldx, ldx = solve_ldx(n)): forward L y = b, y_t = y_t * (1/l_tt) (sfmin
// rule), then y_i = fma(-l_it, y_t, y_i) for i > t; backward x_t = x_t * (1/l_tt),
// then x_i = fma(-l_ti, x_t, x_i) for i < t.  The sweeps of the LU solves
// (solve_core.cuh); D: room for one diagonal block.
template <typename T, int CG>
__device__ __forceinline__ void chol_solve_smem(int n, const T *A, int lda, T *sB, int ldx, int nr, Diag<T> &D)
{
    tri_sweep<T, CG, false, true, false, 32>(n, A, lda, sB, ldx, nr, D);
    tri_sweep<T, CG, true, false, false, 32>(n, A, lda, sB, ldx, nr, D);
}

}  // namespace mlu
