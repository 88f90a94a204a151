// disp.cu -- nodal displacements from the deformation gradient field: replaces f2disp
// (src/f2disp.f:16-135) with form_BTB (:136-400) and its PARDISO solve.
//
// The reference fits nodal positions x on the (N+1)^3 node mesh of the voxel grid (the
// hexahedral elements of oumodel's blkgen, src/oumodel.f:178-330) to F in the least-squares
// sense: (sum_e int B^T B) x = sum_e B^T F_e, B the gradient of the trilinear shape
// functions, the left side integrated with 2x2x2 Gauss points, the right side with one,
// node 1 held at the origin; u = x - X.  On the regular grid the left-side operator is the
// tensor product K(x)M(x)M + M(x)K(x)M + M(x)M(x)K of the 1-D linear-element stiffness K
// and consistent mass M (2-point Gauss integrates them exactly), which the DCT-I
// diagonalises: K v_k = lambda_K(k) W v_k, M v_k = lambda_M(k) W v_k with v_k(i) =
// cos(pi k i / N), W = diag(1/2, 1, .., 1, 1/2), lambda_K = (2/h)(1 - cos(pi k/N)),
// lambda_M = (h/3)(2 + cos(pi k/N)).  The pinned problem is the pure-Neumann one with node
// 1's equation replaced by the reaction that makes it compatible, shifted so that node 1
// stays at the origin.  So the solve is exact and direct: three separable DCT-I passes,
// a diagonal scaling, three more passes -- no sparse factorisation.
//
// The passes are small dense products C z with the cosine table: the FP64 pipe bounds them.
// cos(pi k (N - i) / N) = (-1)^k cos(pi k i / N), so even k take the sums z_i + z_(N-i) and odd
// k the differences: half the products.  Every pass stages its lines in shared memory and
// reads and writes whole 32-point segments; the forward and inverse passes along the third
// axis and the scaling between them are one kernel.  At 63^3 on a GB300 the call takes 0.60 ms;
// with full products, a thread a point reading across the lines, the table's (N + 1)^2 cosines
// formed on the host and three allocations in each call it took 4.1 ms.
//
// Layouts: voxel v = a + N b + N^2 c with c along X (direction 1), b along Y, a along Z
// (the reference's element order, z fastest, src/oumodel.f:612-700); node n = i + (N+1) j
// + (N+1)^2 k with i along X (src/oumodel.f:855-900).  The work fields are (3, N1, N1, N1) with
// k (Z) fastest, as the voxels are; k_disp_out turns them into the reference's order.
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int NT = 256, TL = 32;  // threads, lines per block of a transform

// b: sum over the elements around each node of vol grad N_a(centre) . F_e (one-point
// rule).  Node 0's entry is the reaction that makes the pinned system compatible, minus the
// sum of all others: the gradients of an element's shape functions sum to zero, so that is
// the entry the rule itself gives, without the cancellation of the sum.
__global__ void __launch_bounds__(NT) k_disp_rhs(const double* __restrict__ F, int N, double hx,
                                                 double hy, double hz, double* __restrict__ b) {
  const long long N1 = N + 1, nodes = N1 * N1 * N1, N3 = (long long)N * N * N;
  const double cx = 0.25 * hy * hz, cy = 0.25 * hx * hz, cz = 0.25 * hx * hy;
  for (long long t = (long long)blockIdx.x * NT + threadIdx.x; t < nodes; t += (long long)gridDim.x * NT) {
    const int k = (int)(t % N1), j = (int)((t / N1) % N1), i = (int)(t / (N1 * N1));
    double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int di = -1; di <= 0; di++)
#pragma unroll
      for (int dj = -1; dj <= 0; dj++)
#pragma unroll
        for (int dk = -1; dk <= 0; dk++) {
          const int ei = i + di, ej = j + dj, ek = k + dk;  // element's lowest corner
          if (ei < 0 || ej < 0 || ek < 0 || ei >= N || ej >= N || ek >= N) continue;
          // this node's local coordinates in that element: -1 at its lower face, +1 upper
          const double xi = di == 0 ? -cx : cx, eta = dj == 0 ? -cy : cy, zeta = dk == 0 ? -cz : cz;
          const long long v = ek + (long long)N * ej + (long long)N * N * ei;  // a=z, b=y, c=x
#pragma unroll
          for (int r = 0; r < 3; r++)  // component r of x: F_r1, F_r2, F_r3 at (3r..3r+2)
            s[r] += xi * F[(3 * r + 0) * N3 + v] + eta * F[(3 * r + 1) * N3 + v] +
                    zeta * F[(3 * r + 2) * N3 + v];
        }
    for (int r = 0; r < 3; r++) b[r * nodes + t] = s[r];
  }
}

// Fold a line's points i and N - i in place, TL lines in shared memory (line l at
// z[i * TL + l]): the sums at i <= N / 2, the differences at the mirrored places
__device__ __forceinline__ void fold(double* z, int N) {
  for (int t = threadIdx.x; t < (N + 1) / 2 * TL; t += NT) {  // i < N - i
    const int i = t / TL, l = t % TL;
    const double p = z[i * TL + l], q = z[(N - i) * TL + l];
    z[i * TL + l] = p + q;
    z[(N - i) * TL + l] = p - q;
  }
}
// sum_i cos(pi k i / N) z_i of a folded line (even k: sums, odd k: differences); row: the
// table's row k
__device__ __forceinline__ double dct_point(const double* z, const double* __restrict__ row, int N,
                                            int k, int l) {
  const int h = (N + 1) / 2;  // folded pairs; even N has a middle point of its own
  double s = 0.0;
  if (k & 1) {
    for (int i = 0; i < h; i++) s += __ldg(row + i) * z[(N - i) * TL + l];
  } else {
    for (int i = 0; i < h; i++) s += __ldg(row + i) * z[i * TL + l];
  }
  // the middle point i = N / 2 of even N: cos(pi k / 2), zero for odd k
  if (!(N & 1) && !(k & 1)) s += __ldg(row + N / 2) * z[N / 2 * TL + l];
  return s;
}

// DCT-I along a strided axis: TL neighbouring lines (fastest axis) of one slab a block
__global__ void __launch_bounds__(NT) k_dct_strided(double* __restrict__ z, int N, long long stride,
                                                    const double* __restrict__ ctab) {
  extern __shared__ double sz[];
  const int N1 = N + 1;
  const long long lines = stride;  // contiguous lines per slab
  const long long slab = blockIdx.y * stride * N1;
  const long long l0 = (long long)blockIdx.x * TL;
  for (int t = threadIdx.x; t < N1 * TL; t += NT) {
    const int i = t / TL, l = t % TL;
    sz[t] = l0 + l < lines ? z[slab + i * stride + l0 + l] : 0.0;
  }
  __syncthreads();
  fold(sz, N);
  __syncthreads();
  for (int t = threadIdx.x; t < N1 * TL; t += NT) {
    const int k = t / TL, l = t % TL;
    const double s = dct_point(sz, ctab + (long long)k * N1, N, k, l);
    if (l0 + l < lines) z[slab + k * stride + l0 + l] = s;
  }
}

// Along the fastest axis: forward, the diagonal scaling (2/N)^3 W3 / Lambda (mode (0, 0, 0)
// zero), and back; TL rows (j or i, j) of one component a block.  Lanes of a warp share k and
// hold one row each, so the table reads are broadcasts.
__global__ void __launch_bounds__(NT) k_dct_solve(double* __restrict__ z, int N, double hx, double hy,
                                                  double hz, const double* __restrict__ ctab) {
  extern __shared__ double sz[];
  const int N1 = N + 1;
  const long long rows = 3LL * N1 * N1, r0 = (long long)blockIdx.x * TL;
  double* sy = sz + (size_t)N1 * TL;
  for (int t = threadIdx.x; t < N1 * TL; t += NT) {
    const int l = t / N1, k = t - l * N1;  // coalesced along the row
    sz[k * TL + l] = r0 + l < rows ? z[(r0 + l) * N1 + k] : 0.0;
  }
  __syncthreads();
  fold(sz, N);
  __syncthreads();
  const double f = 2.0 / N, f3 = f * f * f;
  const double* c = ctab + N1;  // row 1: cos(pi k / N)
  {
    const int l = threadIdx.x % TL;
    const long long row = r0 + l;
    const int j = (int)(row % N1), i = (int)((row / N1) % N1);
    const double c1 = __ldg(c + i), c2 = __ldg(c + j);
    const double K1 = 2.0 / hx * (1.0 - c1), K2 = 2.0 / hy * (1.0 - c2);
    const double M1 = hx / 3.0 * (2.0 + c1), M2 = hy / 3.0 * (2.0 + c2);
    const double w12 = f3 * (i == 0 || i == N ? 0.5 : 1.0) * (j == 0 || j == N ? 0.5 : 1.0);
    const double a = K1 * M2 + M1 * K2, m12 = M1 * M2;
    for (int k = threadIdx.x / TL; k < N1; k += NT / TL) {
      const double c3 = __ldg(c + k);
      const double lam = a * (hz / 3.0 * (2.0 + c3)) + m12 * (2.0 / hz * (1.0 - c3));
      const double w = k == 0 || k == N ? 0.5 * w12 : w12;
      const double s = dct_point(sz, ctab + (long long)k * N1, N, k, l);
      sy[k * TL + l] = i == 0 && j == 0 && k == 0 ? 0.0 : s * (w / lam);
    }
  }
  __syncthreads();
  fold(sy, N);
  __syncthreads();
  {
    const int l = threadIdx.x % TL;
    for (int k = threadIdx.x / TL; k < N1; k += NT / TL)
      sz[k * TL + l] = dct_point(sy, ctab + (long long)k * N1, N, k, l);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < N1 * TL; t += NT) {
    const int l = t / N1, k = t - l * N1;
    if (r0 + l < rows) z[(r0 + l) * N1 + k] = sz[k * TL + l];
  }
}

// u[3 n + r] = z[r][n] - z[r][0] - X_r(n): positions relative to node 1, minus the
// reference coordinates (the reference's u array, node-major, i fastest): 32 x 32 tiles of
// (i, k) at one j, transposed through shared memory
__global__ void __launch_bounds__(NT) k_disp_out(const double* __restrict__ z, int N, double hx,
                                                 double hy, double hz, double* __restrict__ u) {
  __shared__ double s[3][32][33];
  const long long N1 = N + 1, nodes = N1 * N1 * N1;
  const int j = blockIdx.z, i0 = 32 * blockIdx.x, k0 = 32 * blockIdx.y;
  for (int t = threadIdx.x; t < 32 * 32; t += NT) {
    const int k = t % 32, i = t / 32;
    if (i0 + i < N1 && k0 + k < N1)
      for (int r = 0; r < 3; r++)
        s[r][i][k] = z[r * nodes + ((i0 + i) * N1 + j) * N1 + k0 + k] - z[r * nodes];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 32 * 96; t += NT) {
    const int k = t / 96, q = t - k * 96, i = q / 3, r = q - 3 * i;
    if (i0 + i >= N1 || k0 + k >= N1) continue;
    const long long n = i0 + i + N1 * j + N1 * N1 * (k0 + k);
    const double X = r == 0 ? (i0 + i) * hx : r == 1 ? j * hy : (k0 + k) * hz;
    u[3 * n + r] = n == 0 ? 0.0 : s[r][i][k] - X;
  }
}

}  // namespace

// u (device, 3 x nodes doubles, node-major) from the device field F (9, N^3); work: one nodal
// field (3 x nodes doubles); ctab: the (N+1)^2 table cos(pi k i / N)
cudaError_t f2disp_device(const double* F, int N, double lx, double ly, double lz,
                          const double* ctab, double* work, double* u, cudaStream_t st) {
  const long long N1 = N + 1, nodes = N1 * N1 * N1;
  const double hx = lx / N, hy = ly / N, hz = lz / N;
  const size_t line = sizeof(double) * (size_t)N1 * TL;
  cudaError_t e;
  if ((e = raise_max_dynamic_smem((const void*)k_dct_strided, line))) return e;
  if ((e = raise_max_dynamic_smem((const void*)k_dct_solve, 2 * line))) return e;
  const int nb = (int)std::min<long long>((nodes + NT - 1) / NT, 65535);
  k_disp_rhs<<<nb, NT, 0, st>>>(F, N, hx, hy, hz, work);
  const dim3 gx((unsigned)((N1 * N1 + TL - 1) / TL), 3), gy((unsigned)((N1 + TL - 1) / TL), (unsigned)(3 * N1));
  const unsigned gz = (unsigned)((3 * N1 * N1 + TL - 1) / TL);
  k_dct_strided<<<gx, NT, line, st>>>(work, N, N1 * N1, ctab);
  k_dct_strided<<<gy, NT, line, st>>>(work, N, N1, ctab);
  k_dct_solve<<<gz, NT, 2 * line, st>>>(work, N, hx, hy, hz, ctab);
  k_dct_strided<<<gy, NT, line, st>>>(work, N, N1, ctab);
  k_dct_strided<<<gx, NT, line, st>>>(work, N, N1 * N1, ctab);
  const unsigned nt = (unsigned)((N1 + 31) / 32);
  k_disp_out<<<dim3(nt, nt, (unsigned)N1), NT, 0, st>>>(work, N, hx, hy, hz, u);
  g_kernel_launches += 7;
  return cudaGetLastError();
}
