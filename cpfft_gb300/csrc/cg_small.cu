// cg_small.cu -- a whole FP64 CG solve in one cooperative launch, for grids whose iterations
// are too short for separate kernels.
//
// What bounds a small grid is latency, not work: the five transform passes of G(K : p) at
// 15^3 need about 4 us of FP64 instructions on 152 SMs, but nine launches, their gaps and
// the host's stop test took 92 us an iteration.  Here the passes are three phases of one
// persistent kernel (the tiles of green_small.cuh, dealt to the blocks in turn) separated by
// grid barriers (1.4 to 1.9 us each, measured), the dot products are block partials that
// every block sums in the same fixed order after a barrier (so all blocks take the same
// decision and runs repeat bit for bit), and the loop ends on the device.  Measured figures
// and the range of grids: cg_small_fp64 below.
#include <algorithm>

#include "cg_small.cuh"
#include "green_small.cuh"

namespace {

// ---- grid barrier ---------------------------------------------------------------------
// Arrivals count up in *cnt (zero at launch); the wait has a limit after which the kernel
// gives up with an error code (every block then runs out of its own wait as well).
constexpr unsigned BARRIER_POLLS = 1u << 25;

struct GridBarrier {
  unsigned* cnt;
  unsigned target;
  bool broken;
};

__device__ __forceinline__ void grid_sync(GridBarrier& b) {
  __syncthreads();
  __shared__ int s_broken;
  if (threadIdx.x == 0) {
    b.target += gridDim.x;
    __threadfence();
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(b.cnt) : "memory");
    unsigned seen, polls = 0;
    int broken = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(b.cnt) : "memory");
      if (seen >= b.target) break;
      if (++polls >= BARRIER_POLLS) { broken = 1; break; }
    }
    __threadfence();
    s_broken = broken;
  }
  __syncthreads();
  if (s_broken) b.broken = true;
}

// fixed-order sum of the blocks' partials, the same in every block; valid in all threads
template <int NT>
__device__ __forceinline__ double sum_partials(const double* part, double* s_red) {
  double v = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += NT) v += __ldcg(part + i);
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int k = 0; k < NT / 32; k++) t += s_red[k];
  __syncthreads();
  return t;
}
template <int NT>
__device__ __forceinline__ void put_partial(double v, double* part, double* s_red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < NT / 32; k++) t += s_red[k];
    part[blockIdx.x] = t;
  }
  __syncthreads();
}

constexpr int NT = 128;  // one warp a quarter of the SM: the FP64 pipe takes no more

struct SmallCg {
  double *x, *r, *p[2], *Ap;  // r, p, Ap: scratch of the solve
  const double* b;
  const double* K4;
  double2* S;
  const double2* tw;
  GridDesc g;
  double* part;               // 2 x blocks partials
  double* sc;                 // results: SC_CNT, SC_STOP, SC_RRNEW, SC_RN
  unsigned* bar;              // barrier counter, zeroed before the launch
  double tol;
  int max_iter;
};

template <bool SPLIT>
__global__ void __launch_bounds__(NT) k_cg_small(SmallCg a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_red[NT / 32];
  const GridDesc& g = a.g;
  const int N = g.N, H = g.H;
  const long long N3 = g.N3, n9 = 9 * N3, plane = (long long)N * N;
  double2* tw = reinterpret_cast<double2*>(smem_raw);
  double2* b0 = tw + N;
  double2* b1 = b0 + max(plane_cols(N), 3 * SMALL_TKC) * padlen(N);
  load_tw(tw, a.tw, N);
  const int hc = (H + SMALL_TKC - 1) / SMALL_TKC, tiles_c = 3 * N * hc;
  const float iN = 1.0f / (float)N, ihc = 1.0f / (float)hc;
  double* part0 = a.part;
  double* part1 = a.part + gridDim.x;
  GridBarrier bar{a.bar, 0u, false};
  double s0 = 0.0;
  for (long long i = (long long)blockIdx.x * NT + threadIdx.x; i < n9; i += (long long)gridDim.x * NT) {
    const double v = a.b[i];
    a.r[i] = v;
    a.x[i] = 0.0;
    s0 += v * v;
  }
  put_partial<NT>(s0, part1, s_red);
  grid_sync(bar);
  double rr = sum_partials<NT>(part1, s_red), beta = 0.0;
  const double n2b = sqrt(rr), tolb = a.tol * n2b;
  int cnt = 0, cur = 0;
  int stop = !isfinite(n2b) ? STOP_NONFINITE : n2b <= 2.220446049250313e-16 ? STOP_TEST : STOP_NONE;
  while (stop == STOP_NONE && !bar.broken) {
    const double* pold = a.p[cur];
    double* pnew = a.p[1 - cur];
    // planes forward: p = r + beta p (the first iteration's p is r), y_i = (K : p)_i
    for (int tile = blockIdx.x; tile < 9 * N; tile += gridDim.x) {
      const int i = fdiv(tile, iN), c0 = tile - i * N;
      const long long v0 = plane * c0;
      plane_forward<double2, double, SPLIT>(
          [&](int u) {
            double s = 0.0;
            const long long v = v0 + u;
#pragma unroll
            for (int j = 0; j < 9; j++) {
              double pv = a.r[j * N3 + v];
              if (cnt) pv += beta * pold[j * N3 + v];
              if (i == j) pnew[j * N3 + v] = pv;
              s += __ldg(a.K4 + (9 * i + j) * N3 + v) * pv;
            }
            return s;
          },
          a.S, i, c0, g, tw, b0, b1);
    }
    grid_sync(bar);
    for (int tile = blockIdx.x; tile < tiles_c; tile += gridDim.x) {
      const int rem = fdiv(tile, ihc), row = fdiv(rem, iN);
      column_tile<double2, double, SPLIT>(a.S, row, rem - row * N, (tile - rem * hc) * SMALL_TKC, g,
                                          tw, b0, b1);
    }
    grid_sync(bar);
    double dsum = 0.0;  // p . Ap
    for (int tile = blockIdx.x; tile < 9 * N; tile += gridDim.x) {
      const int i = fdiv(tile, iN), c0 = tile - i * N;
      const long long v0 = i * N3 + plane * c0;
      plane_inverse<double2, double, SPLIT>(
          [&](int u, double ap) {
            a.Ap[v0 + u] = ap;
            dsum += pnew[v0 + u] * ap;
          },
          a.S, i, c0, g, tw, b0, b1);
    }
    __syncthreads();
    put_partial<NT>(dsum, part0, s_red);
    grid_sync(bar);
    const double alpha = rr / sum_partials<NT>(part0, s_red);
    double s = 0.0;
    for (long long i = (long long)blockIdx.x * NT + threadIdx.x; i < n9; i += (long long)gridDim.x * NT) {
      a.x[i] += alpha * pnew[i];
      const double ri = a.r[i] - alpha * a.Ap[i];
      a.r[i] = ri;
      s += ri * ri;
    }
    put_partial<NT>(s, part1, s_red);
    grid_sync(bar);
    const double rnew = sum_partials<NT>(part1, s_red), rn = sqrt(rnew);
    beta = rnew / rr;
    rr = rnew;
    cnt++;
    cur = 1 - cur;
    if (!isfinite(rn)) stop = STOP_NONFINITE;
    else if (rn <= tolb || rn <= a.tol) stop = STOP_TEST;
    else if (cnt >= a.max_iter) stop = STOP_MAXIT;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.sc[SC_RRNEW] = rr;
    a.sc[SC_RN] = n2b;
    a.sc[SC_CNT] = (double)cnt;
    a.sc[SC_STOP] = (double)(bar.broken ? STOP_BARRIER : stop);
  }
}

template <bool SPLIT>
cudaError_t launch_small(SmallCg& a, cudaStream_t st) {
  const int N = a.g.N;
  const size_t sm = smem_small<double>(N);
  const void* f = (const void*)k_cg_small<SPLIT>;
  cudaError_t e = raise_max_dynamic_smem(f, sm);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, occ = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_cg_small<SPLIT>, NT, sm)) != cudaSuccess) return e;
  if (occ < 1) return cudaErrorCooperativeLaunchTooLarge;
  // two blocks an SM where they fit (one hides the other's loads: 24^3 74 against 118 us an
  // iteration with one, 84 with three), no more than the busiest phase has tiles
  const int hc = (a.g.H + SMALL_TKC - 1) / SMALL_TKC, most = std::max(9 * N, 3 * N * hc);
  const int blocks = std::min(std::min(sms * std::min(occ, 2), most), CG_SMALL_PART / 2);
  if ((e = cudaMemsetAsync(a.bar, 0, sizeof(unsigned), st)) != cudaSuccess) return e;
  void* args[] = {&a};
  e = cudaLaunchCooperativeKernel(f, dim3(blocks), dim3(NT), args, sm, st);
  g_kernel_launches += 1;
  return e;
}

}  // namespace

// One launch against separate kernels, us per iteration (one GB300): 5^3 25 / 82, 9^3 28 / 99,
// 15^3 41 / 91, 16^3 42 / 93, 20^3 59 / 95, 24^3 74 / 111, 27^3 94 / 127, 31^3 166 / 177,
// 33^3 145 / 152, 36^3 220 / 187, 48^3 383 / 264: above, the separate kernels' 256-thread
// blocks fill the SMs better than the two 128-thread blocks that all phases share.
bool cg_small_fp64(int N) { return N <= 33; }

cudaError_t cg_small_solve(const double* b, double* x, double* r, double* p, double* p2, double* Ap,
                           const double* K4, double2* S, const double2* tw, const GridDesc& g,
                           double tol, int max_iter, double* part, double* sc, unsigned* bar,
                           cudaStream_t st) {
  SmallCg a{x, r, {p, p2}, Ap, b, K4, S, tw, g, part, sc, bar, tol, max_iter};
  // split stages while the butterflies' depth is what a phase waits for: 11^3 42 against
  // 53 us an iteration, 13^3 58 / 67, but 12^3 37 / 36, 16^3 43 / 42 and 20^3 81 / 59
  if (g.N <= 11 || g.N == 13) {
    a.g.plan = split_plan(g.N);
    return launch_small<true>(a, st);
  }
  return launch_small<false>(a, st);
}
