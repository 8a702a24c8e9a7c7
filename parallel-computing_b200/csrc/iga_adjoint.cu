// Variable coefficient kappa and the adjoint gradient dJ/dkappa
// (no counterpart in the reference, whose operator has kappa = 1).
//
// For -div(kappa grad u) = f discretised with kappa at the quadrature points,
// K(kappa) = sum_q kappa_q K_q, and for J(u(kappa)) with K lambda = dJ/du
// (lambda = 0 on the boundary):
//     dJ/dkappa_q = -lambda^T K_q u = -(grad lambda . grad u)(x_q) * JxW_q.
// K is symmetric, so the adjoint solve is the forward solver with another
// right-hand side.
#include <cuda_runtime.h>

#include <string>

#include "../../include/iga_solve.h"
#include "iga_column.cuh"
#include "iga_plan.hpp"

using namespace iga;

extern "C" {

int iga_adjoint_grad(iga_plan *pl, const double *u, const double *lam, double *g, void *stream)
{
    if (!pl || !u || !lam || !g) return IGA_ERR_ARG;
    const StripGrid &sg = pl->grid;
    const int rows = column_rows(sg.NSX, sg.ney, pl->nsm);
    const unsigned grid = (unsigned)((long long)sg.NSX * column_chunks(sg.ney, rows));
    const cudaStream_t s = (cudaStream_t)stream;
    switch (pl->p) {
    case 1: adjoint_kernel<1><<<grid, kSW * 2, 0, s>>>(u, lam, g, pl->tabX64, pl->tabY64, pl->CP, pl->qw, sg, rows); break;
    case 2: adjoint_kernel<2><<<grid, kSW * 3, 0, s>>>(u, lam, g, pl->tabX64, pl->tabY64, pl->CP, pl->qw, sg, rows); break;
    case 3: adjoint_kernel<3><<<grid, kSW * 4, 0, s>>>(u, lam, g, pl->tabX64, pl->tabY64, pl->CP, pl->qw, sg, rows); break;
    case 4: adjoint_kernel<4><<<grid, kSW * 5, 0, s>>>(u, lam, g, pl->tabX64, pl->tabY64, pl->CP, pl->qw, sg, rows); break;
    default: adjoint_kernel<5><<<grid, kSW * 6, 0, s>>>(u, lam, g, pl->tabX64, pl->tabY64, pl->CP, pl->qw, sg, rows); break;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("iga_adjoint_grad: ") + cudaGetErrorString(e));
        return IGA_ERR_CUDA;
    }
    return IGA_OK;
}

}  // extern "C"
