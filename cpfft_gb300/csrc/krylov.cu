// krylov.cu -- vector kernels of the device-resident Newton-Krylov loop: CG updates,
// deterministic reductions (warp shuffles inside a block, one partial per block, added in a
// fixed order by the last block, reduce.cuh), field fills and precision casts.
#include <algorithm>

#include "krylov.cuh"
#include "reduce.cuh"

namespace {

constexpr int RB = 256;  // threads per reduction block

template <typename TA, typename TB>
__global__ void __launch_bounds__(RB) k_dot(const TA* __restrict__ a, const TB* __restrict__ b,
                                            long long n, double* __restrict__ part, FinalOp f) {
  TA s = 0;
  for (long long i = (long long)blockIdx.x * RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB)
    s += a[i] * (TA)b[i];
  grid_sum((double)s, part, f);
}

// sum of partials a transform pass left (grids whose passes do not finish them themselves)
__global__ void __launch_bounds__(1024) k_final(const double* __restrict__ part, int np, FinalOp f) {
  __shared__ double ws[32];
  double v = 0.0;
  for (int i = threadIdx.x; i < np; i += 1024) v += part[i];
  v = block_sum(v, ws);
  if (threadIdx.x == 0) apply_final(f, v);
}

// x += alpha p ; r -= alpha Ap ; partial r.r
template <typename T>
__global__ void __launch_bounds__(RB) k_cg_xr(T* __restrict__ x, T* __restrict__ r,
                                              const T* __restrict__ p, const T* __restrict__ Ap,
                                              long long n, const double* __restrict__ sc,
                                              double* __restrict__ part, FinalOp f) {
  // arithmetic in T: on GB300 an FP64 instruction costs ~64 FP32 ones, so the FP32
  // vectors stay in FP32; per-thread partial sums are promoted only for the block sum
  const T alpha = (T)sc[SC_ALPHA];
  T s = 0;
  for (long long i = (long long)blockIdx.x * RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB) {
    x[i] = x[i] + alpha * p[i];
    T ri = r[i] - alpha * Ap[i];
    r[i] = ri;
    s += ri * ri;
  }
  grid_sum((double)s, part, f);
}

// FP32 form with 16-byte vector accesses (n % 4 elements handled by a scalar tail)
__global__ void __launch_bounds__(RB) k_cg_xr4(float* __restrict__ x, float* __restrict__ r,
                                               const float* __restrict__ p,
                                               const float* __restrict__ Ap, long long n,
                                               const double* __restrict__ sc,
                                               double* __restrict__ part, FinalOp f) {
  const float alpha = (float)sc[SC_ALPHA];
  const long long n4 = n >> 2, stride = (long long)gridDim.x * RB;
  float4* x4 = reinterpret_cast<float4*>(x);
  float4* r4 = reinterpret_cast<float4*>(r);
  const float4* p4 = reinterpret_cast<const float4*>(p);
  const float4* a4 = reinterpret_cast<const float4*>(Ap);
  float s = 0.f;
  const long long t0 = (long long)blockIdx.x * RB + threadIdx.x;
  for (long long i = t0; i < n4; i += stride) {
    float4 xv = x4[i], pv = p4[i], rv = r4[i], av = a4[i];
    xv.x += alpha * pv.x; xv.y += alpha * pv.y; xv.z += alpha * pv.z; xv.w += alpha * pv.w;
    rv.x -= alpha * av.x; rv.y -= alpha * av.y; rv.z -= alpha * av.z; rv.w -= alpha * av.w;
    x4[i] = xv;
    r4[i] = rv;
    s += rv.x * rv.x + rv.y * rv.y + rv.z * rv.z + rv.w * rv.w;
  }
  for (long long i = 4 * n4 + t0; i < n; i += stride) {
    x[i] = x[i] + alpha * p[i];
    float ri = r[i] - alpha * Ap[i];
    r[i] = ri;
    s += ri * ri;
  }
  grid_sum((double)s, part, f);
}

__global__ void k_cg_p4(float* __restrict__ p, const float* __restrict__ r, long long n,
                        double* __restrict__ sc) {
  const float beta = (float)sc[SC_BETA];
  const long long n4 = n >> 2, stride = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  float4* p4 = reinterpret_cast<float4*>(p);
  const float4* r4 = reinterpret_cast<const float4*>(r);
  for (long long i = t0; i < n4; i += stride) {
    float4 pv = p4[i], rv = r4[i];
    pv.x = rv.x + beta * pv.x; pv.y = rv.y + beta * pv.y;
    pv.z = rv.z + beta * pv.z; pv.w = rv.w + beta * pv.w;
    p4[i] = pv;
  }
  for (long long i = 4 * n4 + t0; i < n; i += stride) p[i] = r[i] + beta * p[i];
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0) sc[SC_RR] = sc[SC_RRNEW];
}

// p = r + beta p ; rr <- rr_new
template <typename T>
__global__ void k_cg_p(T* __restrict__ p, const T* __restrict__ r, long long n,
                       double* __restrict__ sc) {
  const T beta = (T)sc[SC_BETA];
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    p[i] = r[i] + beta * p[i];
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0) sc[SC_RR] = sc[SC_RRNEW];
}

__global__ void k_axpy(double* __restrict__ y, const double* __restrict__ x, double a, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}
__global__ void k_scale(double* __restrict__ y, double a, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] *= a;
}
__global__ void k_scale_f(float* __restrict__ y, float a, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] *= a;
}
__global__ void k_sub(double* __restrict__ y, const double* __restrict__ a,
                      const double* __restrict__ b, long long n) {  // y = a - b
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = a[i] - b[i];
}
// fill component c of a (9, N3) field with v[c]
__global__ void k_fill9(double* __restrict__ y, long long N3, double v0, double v1, double v2,
                        double v3, double v4, double v5, double v6, double v7, double v8) {
  const double v[9] = {v0, v1, v2, v3, v4, v5, v6, v7, v8};
  long long n = 9 * N3;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = v[i / N3];
}
__global__ void k_add_const(double* __restrict__ y, double v, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] += v;
}
// y = s * (double)x_f, or zero after a segment that ended on a non-finite value; x_f = 0
__global__ void k_take_f32(double* __restrict__ y, float* __restrict__ x, double s, long long n,
                           const double* __restrict__ sc) {
  const bool drop = sc[SC_STOP] == (double)STOP_NONFINITE;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    y[i] = drop ? 0.0 : s * (double)x[i];
    x[i] = 0.0f;
  }
}
// y_f = (float)(x * s), p_f *= k
__global__ void k_restart_f32(float* __restrict__ y, const double* __restrict__ x, double s,
                              float* __restrict__ p, float k, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    y[i] = (float)(x[i] * s);
    p[i] *= k;
  }
}
// y = a - b and the sum of y^2
__global__ void __launch_bounds__(RB) k_sub_norm(double* __restrict__ y, const double* __restrict__ a,
                                                 const double* __restrict__ b, long long n,
                                                 double* __restrict__ part, FinalOp f) {
  double s = 0.0;
  for (long long i = (long long)blockIdx.x * RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB) {
    const double d = a[i] - b[i];
    y[i] = d;
    s += d * d;
  }
  grid_sum(s, part, f);
}
// the scalars of a CG segment that starts from the <r, r>_K0 in SC_RRNEW
__global__ void k_cg_start(double* __restrict__ sc, double rn, double tolb, double tol, double delta,
                           double it, double maxit, double rrk2) {
  const double rr = sc[SC_RRNEW];
  sc[SC_BETA] = rrk2 > 0.0 ? rr / rrk2 : 0.0;
  sc[SC_RR0] = rr;
  sc[SC_RN] = rn;
  sc[SC_TOLB] = tolb;
  sc[SC_TOL] = tol;
  sc[SC_DELTA] = delta;
  sc[SC_CNT] = it;
  sc[SC_MAXIT] = maxit;
  sc[SC_STOP] = 0.0;
}
// y_f = (float)(x * s)
__global__ void k_to_f32(float* __restrict__ y, const double* __restrict__ x, double s, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = (float)(x[i] * s);
}
// y += s * (double)x_f
__global__ void k_add_f32(double* __restrict__ y, const float* __restrict__ x, double s, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] += s * (double)x[i];
}
// sums of each of the 9 components of a (9, N3) field
__global__ void __launch_bounds__(RB) k_sum9(const double* __restrict__ x, long long N3,
                                             double* __restrict__ part, double* __restrict__ sc,
                                             int slot) {
  double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long long i = (long long)blockIdx.x * RB + threadIdx.x; i < N3; i += (long long)gridDim.x * RB)
#pragma unroll
    for (int c = 0; c < 9; c++) s[c] += x[c * N3 + i];
  grid_sum9(s, part, sc, slot);
}

// the nine components of K4 : x summed over the grid (x read once for all nine)
__global__ void __launch_bounds__(RB) k_homo9(const double* __restrict__ K4, const double* __restrict__ x,
                                              long long N3, double* __restrict__ part,
                                              double* __restrict__ sc, int slot) {
  double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long long v = (long long)blockIdx.x * RB + threadIdx.x; v < N3; v += (long long)gridDim.x * RB) {
    double xv[9];
#pragma unroll
    for (int k = 0; k < 9; k++) xv[k] = x[k * N3 + v];
#pragma unroll
    for (int j = 0; j < 9; j++)
#pragma unroll
      for (int k = 0; k < 9; k++) s[j] += K4[(9 * j + k) * N3 + v] * xv[k];
  }
  grid_sum9(s, part, sc, slot);
}

// ---- K0-weighted forms of the reference-medium preconditioned FP32 CG ----------------
// The CG of the preconditioned operator G0(K : .) runs in the inner product
// <a, b>_K0 = sum_v a_v . (K0 b_v), K0 the (normalised, symmetrised) 9x9 reference stiffness
// of the calling context (device memory, staged in shared memory per block).
__device__ __forceinline__ void load_k0(const float* __restrict__ k0, float* s_k0) {
  for (int i = threadIdx.x; i < 81; i += blockDim.x) s_k0[i] = k0[i];
  __syncthreads();
}
__device__ __forceinline__ float k0_form(const float* s_k0, const float* a, const float* b) {
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 9; i++) {
    float t = 0.f;
#pragma unroll
    for (int j = 0; j < 9; j++) t += s_k0[9 * i + j] * b[j];
    s += a[i] * t;
  }
  return s;
}

// x += alpha p ; r -= alpha Ap ; <r, r>_K0 -- one voxel's 9 components per thread
// (component-major fields), four voxels at a time with 16-byte accesses when N3 % 4 == 0
__global__ void __launch_bounds__(RB) k_cg_xr_k0(float* __restrict__ x, float* __restrict__ r,
                                                 const float* __restrict__ p,
                                                 const float* __restrict__ Ap, long long N3,
                                                 const float* __restrict__ k0,
                                                 const double* __restrict__ sc,
                                                 double* __restrict__ part, FinalOp f) {
  __shared__ float s_k0[81];
  load_k0(k0, s_k0);
  const float alpha = (float)sc[SC_ALPHA];
  const long long stride = (long long)gridDim.x * RB, t0 = (long long)blockIdx.x * RB + threadIdx.x;
  float s = 0.f;
  if ((N3 & 3) == 0) {
    const long long n4 = N3 >> 2;
    for (long long v = t0; v < n4; v += stride) {
      float rv[4][9];
#pragma unroll
      for (int i = 0; i < 9; i++) {
        const long long k = i * n4 + v;
        float4 xv = reinterpret_cast<float4*>(x)[k];
        const float4 pv = reinterpret_cast<const float4*>(p)[k];
        float4 qv = reinterpret_cast<float4*>(r)[k];
        const float4 av = reinterpret_cast<const float4*>(Ap)[k];
        xv.x += alpha * pv.x; xv.y += alpha * pv.y; xv.z += alpha * pv.z; xv.w += alpha * pv.w;
        qv.x -= alpha * av.x; qv.y -= alpha * av.y; qv.z -= alpha * av.z; qv.w -= alpha * av.w;
        reinterpret_cast<float4*>(x)[k] = xv;
        reinterpret_cast<float4*>(r)[k] = qv;
        rv[0][i] = qv.x; rv[1][i] = qv.y; rv[2][i] = qv.z; rv[3][i] = qv.w;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) s += k0_form(s_k0, rv[u], rv[u]);
    }
  } else {
    for (long long v = t0; v < N3; v += stride) {
      float rv[9];
#pragma unroll
      for (int i = 0; i < 9; i++) {
        const long long k = i * N3 + v;
        x[k] += alpha * p[k];
        rv[i] = r[k] - alpha * Ap[k];
        r[k] = rv[i];
      }
      s += k0_form(s_k0, rv, rv);
    }
  }
  grid_sum((double)s, part, f);
}

// partial <a, b>_K0
__global__ void __launch_bounds__(RB) k_dot_k0(const float* __restrict__ a, const float* __restrict__ b,
                                               long long N3, const float* __restrict__ k0,
                                               double* __restrict__ part, FinalOp f) {
  __shared__ float s_k0[81];
  load_k0(k0, s_k0);
  float s = 0.f;
  for (long long v = (long long)blockIdx.x * RB + threadIdx.x; v < N3; v += (long long)gridDim.x * RB) {
    float av[9], bv[9];
#pragma unroll
    for (int i = 0; i < 9; i++) { av[i] = a[i * N3 + v]; bv[i] = b[i * N3 + v]; }
    s += k0_form(s_k0, av, bv);
  }
  grid_sum((double)s, part, f);
}

// component sums of an (81, N3) FP32 field: part[m * gridDim.x + blockIdx.x]
__global__ void __launch_bounds__(RB) k_sum81(const float* __restrict__ K, long long N3,
                                              double* __restrict__ part) {
  const int m = blockIdx.y;
  double s = 0.0;
  for (long long v = (long long)blockIdx.x * RB + threadIdx.x; v < N3; v += (long long)gridDim.x * RB)
    s += (double)K[m * N3 + v];
  __shared__ double ws[32];
  s = block_sum(s, ws);
  if (threadIdx.x == 0) part[m * gridDim.x + blockIdx.x] = s;
}

// out[m] = sum of the np partials of row m (one block of 64 threads per row, np <= 64)
__global__ void __launch_bounds__(64) k_final_rows(const double* __restrict__ part, int np,
                                                   double* __restrict__ out) {
  __shared__ double ws[2];
  double v = threadIdx.x < np ? part[blockIdx.x * np + threadIdx.x] : 0.0;
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) out[blockIdx.x] = ws[0] + ws[1];
}

// Ellipticity of the reference medium K0 = sym(sums / N3) / its largest entry: the acoustic
// tensor A(n)_ik = K0_ijkl n_j n_l on MEDIUM_ROWS x 128 directions of the sphere, one a thread;
// out[b] = the least det A / tr(A)^3 of block b's directions (it bounds the smallest
// eigenvalue's share from below), -1 where A is not positive definite (Sylvester).  On the host
// the 8,320 directions held up every stress pass of the fast form with the GPU idle; here they
// run between the sums and their read-back (a 12^3 pass 1.17 to 0.95 ms, a 62^3 one 8.16 to
// 7.98).
__global__ void __launch_bounds__(128) k_medium(const double* __restrict__ sc81, long long N3,
                                                double* __restrict__ out) {
  __shared__ double K0[81], wmin[4], s_mx;
  const int t = threadIdx.x;
  if (t < 81) K0[t] = 0.5 * (sc81[t] + sc81[9 * (t % 9) + t / 9]) / (double)N3;
  __syncthreads();
  if (t < 32) {
    double m = fmax(fabs(K0[t]), fabs(K0[t + 32]));
    if (t + 64 < 81) m = fmax(m, fabs(K0[t + 64]));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (t == 0) s_mx = m;
  }
  __syncthreads();
  if (t < 81) K0[t] /= s_mx;
  __syncthreads();
  double n[3], sth, cth, sph, cph;
  sincospi(blockIdx.x / (double)(MEDIUM_ROWS - 1), &sth, &cth);
  sincospi(t / 64.0, &sph, &cph);
  n[0] = sth * cph; n[1] = sth * sph; n[2] = cth;
  double a[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int k = 0; k < 3; k++) {
      a[i][k] = 0.0;
#pragma unroll
      for (int j = 0; j < 3; j++) {
        double v = 0.0;
#pragma unroll
        for (int l = 0; l < 3; l++) v += K0[9 * (3 * i + j) + 3 * k + l] * n[l];
        a[i][k] += v * n[j];
      }
    }
  const double m2 = a[0][0] * a[1][1] - a[0][1] * a[0][1];
  const double det = a[0][0] * (a[1][1] * a[2][2] - a[1][2] * a[1][2]) -
                     a[0][1] * (a[0][1] * a[2][2] - a[1][2] * a[0][2]) +
                     a[0][2] * (a[0][1] * a[1][2] - a[1][1] * a[0][2]);
  const double tr = a[0][0] + a[1][1] + a[2][2];
  double q = a[0][0] > 0.0 && m2 > 0.0 && det > 0.0 && tr > 0.0 ? det / (tr * tr * tr) : -1.0;
  for (int o = 16; o > 0; o >>= 1) q = fmin(q, __shfl_xor_sync(0xffffffffu, q, o));
  if ((t & 31) == 0) wmin[t >> 5] = q;
  __syncthreads();
  if (t == 0) out[blockIdx.x] = fmin(fmin(wmin[0], wmin[1]), fmin(wmin[2], wmin[3]));
}

// The iteration graph's first node: its WHILE loop runs only if the iterations are not
// already stopped (an eager first iteration may have met the stop test), so the host
// launches the graph without reading the stop flag first.
__global__ void k_cg_gate(const double* __restrict__ sc, cudaGraphConditionalHandle h) {
  cudaGraphSetConditional(h, sc[SC_STOP] == (double)STOP_NONE ? 1u : 0u);
}

int grid_for(long long n, int bs) {
  long long b = (n + bs - 1) / bs;
  return (int)(b < 1 ? 1 : (b > 2048 ? 2048 : b));
}

}  // namespace

static cudaError_t counted(int k) {
  g_kernel_launches += k;
  return cudaGetLastError();
}

// blocks of a reduction over n values: enough for every SM, at most NPART
static int blocks_for(long long n) { return (int)std::max<long long>(1, std::min<long long>(NPART, (n + RB - 1) / RB)); }

cudaError_t dev_dot(const double* a, const double* b, long long n, double* part, double* sc,
                    int slot, int op, cudaStream_t st) {
  k_dot<double, double><<<blocks_for(n), RB, 0, st>>>(a, b, n, part, FinalOp{sc, slot, op, 0, 0});
  return counted(1);
}
cudaError_t dev_dot_f(const float* a, const float* b, long long n, double* part, double* sc,
                      int slot, int op, cudaStream_t st) {
  k_dot<float, float><<<blocks_for(n), RB, 0, st>>>(a, b, n, part, FinalOp{sc, slot, op, 0, 0});
  return counted(1);
}
template <typename T>
cudaError_t dev_cg_xr(T* x, T* r, const T* p, const T* Ap, long long n, double* part, double* sc,
                      cudaStream_t st) {
  const FinalOp f{sc, SC_RRNEW, OP_BETA, 0, 0};
  if (sizeof(T) == 4)
    k_cg_xr4<<<blocks_for(n / 4), RB, 0, st>>>((float*)x, (float*)r, (const float*)p, (const float*)Ap,
                                               n, sc, part, f);
  else
    k_cg_xr<T><<<blocks_for(n), RB, 0, st>>>(x, r, p, Ap, n, sc, part, f);
  return counted(1);
}
template <typename T>
cudaError_t dev_cg_p(T* p, const T* r, long long n, double* sc, cudaStream_t st) {
  if (sizeof(T) == 4)
    k_cg_p4<<<grid_for(n / 4 + 1, 256), 256, 0, st>>>((float*)p, (const float*)r, n, sc);
  else
    k_cg_p<T><<<grid_for(n, 256), 256, 0, st>>>(p, r, n, sc);
  return counted(1);
}
cudaError_t dev_final(double* part, int np, double* sc, int slot, int op, cudaStream_t st,
                      cudaGraphConditionalHandle h, bool use_handle) {
  k_final<<<1, 1024, 0, st>>>(part, np, FinalOp{sc, slot, op, h, use_handle ? 1 : 0});
  return counted(1);
}
template cudaError_t dev_cg_xr<double>(double*, double*, const double*, const double*, long long,
                                       double*, double*, cudaStream_t);
template cudaError_t dev_cg_xr<float>(float*, float*, const float*, const float*, long long,
                                      double*, double*, cudaStream_t);
template cudaError_t dev_cg_p<double>(double*, const double*, long long, double*, cudaStream_t);
template cudaError_t dev_cg_p<float>(float*, const float*, long long, double*, cudaStream_t);

cudaError_t dev_axpy(double* y, const double* x, double a, long long n, cudaStream_t st) {
  k_axpy<<<grid_for(n, 256), 256, 0, st>>>(y, x, a, n);
  return counted(1);
}
cudaError_t dev_scale(double* y, double a, long long n, cudaStream_t st) {
  k_scale<<<grid_for(n, 256), 256, 0, st>>>(y, a, n);
  return counted(1);
}
cudaError_t dev_scale_f(float* y, float a, long long n, cudaStream_t st) {
  k_scale_f<<<grid_for(n, 256), 256, 0, st>>>(y, a, n);
  return counted(1);
}
cudaError_t dev_sub(double* y, const double* a, const double* b, long long n, cudaStream_t st) {
  k_sub<<<grid_for(n, 256), 256, 0, st>>>(y, a, b, n);
  return counted(1);
}
cudaError_t dev_fill9(double* y, long long N3, const double* v, cudaStream_t st) {
  k_fill9<<<grid_for(9 * N3, 256), 256, 0, st>>>(y, N3, v[0], v[1], v[2], v[3], v[4], v[5], v[6],
                                                  v[7], v[8]);
  return counted(1);
}
cudaError_t dev_add_const(double* y, double v, long long n, cudaStream_t st) {
  k_add_const<<<grid_for(n, 256), 256, 0, st>>>(y, v, n);
  return counted(1);
}
cudaError_t dev_to_f32(float* y, const double* x, double s, long long n, cudaStream_t st) {
  k_to_f32<<<grid_for(n, 256), 256, 0, st>>>(y, x, s, n);
  return counted(1);
}
cudaError_t dev_add_f32(double* y, const float* x, double s, long long n, cudaStream_t st) {
  k_add_f32<<<grid_for(n, 256), 256, 0, st>>>(y, x, s, n);
  return counted(1);
}
cudaError_t dev_take_f32(double* y, float* x, double s, long long n, const double* sc,
                         cudaStream_t st) {
  k_take_f32<<<grid_for(n, 256), 256, 0, st>>>(y, x, s, n, sc);
  return counted(1);
}
cudaError_t dev_restart_f32(float* y, const double* x, double s, float* p, float k, long long n,
                            cudaStream_t st) {
  k_restart_f32<<<grid_for(n, 256), 256, 0, st>>>(y, x, s, p, k, n);
  return counted(1);
}
cudaError_t dev_sub_norm(double* y, const double* a, const double* b, long long n, double* part,
                         double* sc, int slot, cudaStream_t st) {
  k_sub_norm<<<blocks_for(n), RB, 0, st>>>(y, a, b, n, part, FinalOp{sc, slot, OP_STORE, 0, 0});
  return counted(1);
}
cudaError_t dev_cg_start(double* sc, double rn, double tolb, double tol, double delta, int it,
                         int maxit, double rrk2, cudaStream_t st) {
  k_cg_start<<<1, 1, 0, st>>>(sc, rn, tolb, tol, delta, (double)it, (double)maxit, rrk2);
  return counted(1);
}
cudaError_t dev_sum9(const double* x, long long N3, double* part, double* sc, int slot0,
                     cudaStream_t st) {
  k_sum9<<<blocks_for(N3), RB, 0, st>>>(x, N3, part, sc, slot0);
  return counted(1);
}
cudaError_t dev_homo9(const double* K4, const double* x, long long N3, double* part, double* sc,
                      int slot, cudaStream_t st) {
  k_homo9<<<blocks_for(N3), RB, 0, st>>>(K4, x, N3, part, sc, slot);
  return counted(1);
}

cudaError_t dev_cg_xr_k0(float* x, float* r, const float* p, const float* Ap, long long N3,
                         const float* k0, double* part, double* sc, cudaGraphConditionalHandle h,
                         bool use_handle, cudaStream_t st) {
  k_cg_xr_k0<<<blocks_for(N3), RB, 0, st>>>(x, r, p, Ap, N3, k0, sc, part,
                                            FinalOp{sc, SC_RRNEW, OP_BETA_COND, h, use_handle ? 1 : 0});
  return counted(1);
}
cudaError_t dev_dot_k0(const float* a, const float* b, long long N3, const float* k0,
                       double* part, double* sc, int slot, int op, cudaStream_t st) {
  k_dot_k0<<<blocks_for(N3), RB, 0, st>>>(a, b, N3, k0, part, FinalOp{sc, slot, op, 0, 0});
  return counted(1);
}
cudaError_t dev_mean81(const float* K, long long N3, double* part, double* sc81, cudaStream_t st) {
  constexpr int NB = 64;
  k_sum81<<<dim3(NB, 81), RB, 0, st>>>(K, N3, part);
  k_final_rows<<<81, 64, 0, st>>>(part, NB, sc81);
  return counted(2);
}
cudaError_t dev_medium(const double* sc81, long long N3, double* out, cudaStream_t st) {
  k_medium<<<MEDIUM_ROWS, 128, 0, st>>>(sc81, N3, out);
  return counted(1);
}
cudaError_t dev_cg_gate(const double* sc, cudaGraphConditionalHandle h, cudaStream_t st) {
  k_cg_gate<<<1, 1, 0, st>>>(sc, h);
  return counted(1);
}
