// cg_small.cuh -- CG solves of small grids in one cooperative launch (cg_small.cu).
#pragma once
#include "fft_green.cuh"
#include "krylov.cuh"

constexpr int CG_SMALL_PART = 2048;  // partial sums the caller's part buffer must hold

// grids whose FP64 solves run in one launch
bool cg_small_fp64(int N);

// The plain FP64 CG on G(K4 : x) = b from x = 0 with the reference's stop test (||r|| <=
// tol ||b|| or <= tol, max_iter iterations).  r, p, p2, Ap: scratch fields.  Results in sc:
// SC_CNT iterations, SC_STOP (STOP_*), SC_RRNEW <r, r>, SC_RN ||b||.
cudaError_t cg_small_solve(const double* b, double* x, double* r, double* p, double* p2, double* Ap,
                           const double* K4, double2* S, const double2* tw, const GridDesc& g,
                           double tol, int max_iter, double* part, double* sc, unsigned* bar,
                           cudaStream_t st);
