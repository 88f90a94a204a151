// reduce.cuh -- the end of a device-wide sum: the last block to finish adds all blocks'
// partials in a fixed order (so runs repeat bit for bit) and applies the CG's scalar
// follow-up, which saves the launch of a one-block kernel.  FP32 CG iteration on a GB300 with
// separate final kernels / this: 24^3 46 / 40 us, 27^3 51 / 44, 40^3 56 / 50, 48^3 66 / 62.
#pragma once
#include "krylov.cuh"

namespace {

// End-of-iteration test of a preconditioned FP32 CG segment (described in krylov.cuh)
__device__ __forceinline__ void cg_cond(double* sc, cudaGraphConditionalHandle h, int use_handle) {
  const double rr = sc[SC_RRNEW];
  const double cnt = sc[SC_CNT] + 1.0;
  sc[SC_CNT] = cnt;
  int stop = STOP_NONE;
  if (!isfinite(rr)) {
    stop = STOP_NONFINITE;
  } else if (!(sc[SC_RR0] > 0.0)) {
    stop = STOP_TEST;  // nothing to reduce: let the caller's true residual decide
  } else {
    const double red = sqrt(fmax(rr, 0.0) / sc[SC_RR0]), est = sc[SC_RN] * red;
    if (red < sc[SC_DELTA] || est <= sc[SC_TOLB] || est <= sc[SC_TOL]) stop = STOP_TEST;
    else if (cnt >= sc[SC_MAXIT]) stop = STOP_MAXIT;
  }
  sc[SC_STOP] = (double)stop;
  if (use_handle) cudaGraphSetConditional(h, stop == STOP_NONE ? 1u : 0u);
}

// what follows a finished sum v (one thread)
struct FinalOp {
  double* sc;
  int slot, op;                       // OP_*
  cudaGraphConditionalHandle handle;  // OP_BETA_COND in a captured iteration
  int use_handle;
};
__device__ __forceinline__ void apply_final(const FinalOp& f, double v) {
  double* sc = f.sc;
  sc[f.slot] = v;
  if (f.op == OP_ALPHA) sc[SC_ALPHA] = sc[SC_RR] / v;                            // alpha = rr / pAp
  else if (f.op == OP_BETA || f.op == OP_BETA_COND) sc[SC_BETA] = v / sc[SC_RR];  // beta = rr_new / rr
  if (f.op == OP_BETA_COND) cg_cond(sc, f.handle, f.use_handle);
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// sum over the block (fixed order), valid in thread 0; ws: 32 doubles of shared memory
__device__ __forceinline__ double block_sum(double v, double* ws) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) ws[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0.0;
    v = warp_sum(v);
  }
  return v;
}

// true in every thread of the block that arrives last; the partials all blocks wrote before
// are then visible to it.  The counter sits behind the context's scalars and returns to zero.
__device__ __forceinline__ bool last_block(double* sc) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned* ticket = reinterpret_cast<unsigned*>(sc + SC_COUNT);
    s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  return s_last != 0;
}

// v: this block's threads' values; part: gridDim.x partials
__device__ __forceinline__ void grid_sum(double v, double* part, const FinalOp& f) {
  __shared__ double ws[32];
  v = block_sum(v, ws);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
  if (!last_block(f.sc)) return;
  double t = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) t += __ldcg(part + i);
  t = block_sum(t, ws);
  if (threadIdx.x == 0) apply_final(f, t);
}

// the same for the nine sums v[0 .. 8] into slots slot .. slot + 8 (part: 9 x gridDim.x)
__device__ __forceinline__ void grid_sum9(const double* v, double* part, double* sc, int slot) {
  __shared__ double ws[32];
  for (int c = 0; c < 9; c++) {
    const double b = block_sum(v[c], ws);
    if (threadIdx.x == 0) part[c * gridDim.x + blockIdx.x] = b;
  }
  if (!last_block(sc)) return;
  for (int c = 0; c < 9; c++) {
    double t = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) t += __ldcg(part + c * gridDim.x + i);
    t = block_sum(t, ws);
    if (threadIdx.x == 0) sc[slot + c] = t;
  }
}

}  // namespace
