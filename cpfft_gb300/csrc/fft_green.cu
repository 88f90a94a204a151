// fft_green.cu -- y = G(K : x) or y = G(x) on the GPU: a hand-written real-to-complex
// 3-D FFT of the 9 tensor components fused with the spectral Green operator.
//
// Replaces G_K_dF / fftfem3d / ifftfem3d / ddot42n (src/G_K_dF.f:11-268), which run 18
// complex 3-D MKL transforms per call on real data and read an 81-wide stored Green
// table (src/FFT_init.f:272-340).  Here:
//   pass A  K:x fused into a real-to-complex transform along the fastest axis (two real
//           lines packed into one complex transform);
//   pass B  complex transform along the middle axis, tiles of columns in shared memory;
//   pass C  transform along the slowest axis, Green contraction evaluated from q on the
//           fly for all 9 components while they sit in shared memory, inverse transform
//           along the same axis -- the spectrum never round-trips HBM between the
//           transform and the contraction;
//   pass D  inverse along the middle axis;
//   pass E  complex-to-real inverse along the fastest axis, unpacking the line pairs.
// The reference's result is Re(IDFT(Ghat(q(f)) X(f))); for real input that equals
// IDFT(Hs(f) X(f)) with Hs(f) = (Ghat(q(f)) + Ghat(q(-f)))/2, which keeps the half
// spectrum Hermitian and is what pass C applies, for both frequency mappings.
#include <algorithm>

#include "green_passes.cuh"
#include "green_small.cuh"


FftPlan make_plan(int N) {
  FftPlan p;
  p.n = N;
  p.nst = 0;
  int m = N, Ns = 1;
  auto push = [&](int r) {
    p.R[p.nst] = r;
    p.Ns[p.nst] = Ns;
    Ns *= r;
    p.nst++;
    m /= r;
  };
  // a prime without a register butterfly comes first (Ns = 1, no twiddles; N <= 256 has at
  // most one), then as few stages as the radices allow (63 = 7 x 9, 48 = 6 x 8)
  for (int f = 17; f <= m; f += 2)
    while (m % f == 0) {
      bool prime = true;
      for (int d = 3; d * d <= f; d += 2) prime &= f % d != 0;
      if (!prime) break;
      push(f);
    }
  for (int r : {13, 11, 7}) while (m % r == 0) push(r);
  while (m % 9 == 0) push(9);
  while (m % 5 == 0) push(5);
  // powers of two, with a left-over 3 folded into a radix 6 where one stage is saved
  int two = 0;
  for (int k = m; k % 2 == 0; k /= 2) two++;
  if (m % 3 == 0 && two % 3 == 1) push(6);
  while (m % 3 == 0) push(3);
  while (m % 8 == 0) push(8);
  while (m % 4 == 0) push(4);
  while (m % 2 == 0) push(2);
  return p;
}

// Threads per block of the five-pass form's shared-memory passes (grids above small_max) and of
// pass C, which the FP32 three-pass form runs too.  A stage has (columns x N / radix) butterflies
// -- 81 to 162 for the radices 7 to 9 at N = 63 -- so 256 threads leave half of the block idle
// while its registers (about 112 a thread in FP64) hold back other blocks; only pass C of small
// FP32 grids does not fill the SMs, and there the wider block shortens the copy loops.  Launches
// of G(K : x) with 256 / 128 threads, us (ncu, one GB300): FP64 63^3 passes A and E 130 + 93 /
// 117 + 88, pass B 78 / 75; FP32 pass C 48^3 23 / 19, 40^3 13.7 / 17.9
constexpr int PASS_THREADS = 128;
template <typename T>
int column_threads(int N) { return sizeof(T) == 4 && N < 44 ? 256 : PASS_THREADS; }

// ---- small grids: planes forward, columns, planes inverse (green_small.cuh) -------------
template <typename T, bool SPLIT>
__global__ void __launch_bounds__(256) small_forward(const T* __restrict__ x, const T* __restrict__ K4,
                                                     int flgK, typename Vec2<T>::t* __restrict__ S,
                                                     GridDesc g, const typename Vec2<T>::t* __restrict__ twg,
                                                     double* __restrict__ part, double* scf) {
  using T2 = typename Vec2<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = g.N;
  const long long N3 = g.N3;
  T2* tw = reinterpret_cast<T2*>(smem_raw);
  T2* b0 = tw + N;
  load_tw(tw, twg, N);
  const int i = blockIdx.x / N, c0 = blockIdx.x - i * N;
  const long long v0 = (long long)N * N * c0;
  T dsum = 0;
  plane_forward<T2, T, SPLIT>(
      [&](int u) {
        const long long v = v0 + u;
        if (!flgK) return x[i * N3 + v];
        T xv[9], s = 0;
#pragma unroll
        for (int j = 0; j < 9; j++) xv[j] = x[j * N3 + v];
#pragma unroll
        for (int j = 0; j < 9; j++) s += K4[(9 * i + j) * N3 + v] * xv[j];
        if (part) dsum += s * x[i * N3 + v];
        return s;
      },
      S, i, c0, g, tw, b0, b0 + std::max(plane_cols(N), 3 * SMALL_TKC) * padlen(N));
  if (part && scf) grid_sum((double)dsum, part, FinalOp{scf, SC_PAP, OP_ALPHA, 0, 0});
  else if (part) block_partial<256>((double)dsum, part + blockIdx.x);
}

template <bool SPLIT>
__global__ void __launch_bounds__(128) small_columns(double2* __restrict__ S, GridDesc g,
                                                     const double2* __restrict__ twg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* tw = reinterpret_cast<double2*>(smem_raw);
  double2* b0 = tw + g.N;
  load_tw(tw, twg, g.N);
  column_tile<double2, double, SPLIT>(S, blockIdx.z, blockIdx.y, blockIdx.x * SMALL_TKC, g, tw, b0,
                                      b0 + 3 * SMALL_TKC * padlen(g.N));
}

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(256) small_inverse(const typename Vec2<T>::t* __restrict__ S,
                                                     T* __restrict__ y, GridDesc g,
                                                     const typename Vec2<T>::t* __restrict__ twg) {
  using T2 = typename Vec2<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = g.N;
  T2* tw = reinterpret_cast<T2*>(smem_raw);
  T2* b0 = tw + N;
  load_tw(tw, twg, N);
  const int i = blockIdx.x / N, c0 = blockIdx.x - i * N;
  T* out = y + i * g.N3 + (long long)N * N * c0;
  plane_inverse<T2, T, SPLIT>([&](int u, T v) { out[u] = v; }, S, i, c0, g, tw, b0,
                              b0 + std::max(plane_cols(N), 3 * SMALL_TKC) * padlen(N));
}

// The largest grid of the three-pass form.  It saves two launches and one round trip of the
// half spectrum and balances better, but a plane tile reads all nine components of x for
// each one it writes and its FP64 stages fill the lanes less well than the wider line and
// column tiles.  Three against five passes, us per G(K : x) (ncu, one GB300): FP64 9^3 25 / 61,
// 16^3 29 / 46, 24^3 51 / 58, 32^3 69 / 95 (register passes), 48^3 204 / 212, 56^3 367 / 331;
// FP32 15^3 21 / 31, 27^3 30 / 37, 48^3 47 / 59, 63^3 75 / 90, 80^3 174 / 193, 96^3 306 / 309.
template <typename T>
constexpr int small_max() { return sizeof(T) == 8 ? 48 : 80; }

template <typename T, bool SPLIT>
void small_apply(const T* x, const T* K4, int flgK, T* y, typename Vec2<T>::t* S,
                 const typename Vec2<T>::t* tw, const GridDesc& g, cudaStream_t st, double* part,
                 double* scf) {
  const int N = g.N;
  const size_t sm = smem_small<T>(N);
  constexpr int BT = 256;
  small_forward<T, SPLIT><<<9 * N, BT, sm, st>>>(x, K4, flgK, S, g, tw, part, scf);
  if constexpr (sizeof(T) == 8) {
    small_columns<SPLIT><<<dim3((g.H + SMALL_TKC - 1) / SMALL_TKC, N, 3), 128, sm, st>>>(S, g, tw);
  } else {
    GridDesc gc = g;
    gc.tkc = tile_c<T>();
    pass_c<T><<<dim3((g.H + gc.tkc - 1) / gc.tkc, N), column_threads<T>(N), smem_c<T>(N, gc.tkc), st>>>(S, gc, tw);
  }
  small_inverse<T, SPLIT><<<9 * N, BT, sm, st>>>(S, y, g, tw);
}

template <typename T>
cudaError_t green_setup(int N) {
  cudaError_t e;
  // power-of-two grids take the register-FFT passes (FP64 too: 3.72 against 3.98 ms for
  // the shared-memory Stockham passes at 128^3, measured on a GB300)
  {
    switch (N) {
      case 32:
        if constexpr (sizeof(T) == 4) return wgreen_setup<1, T>();
        break;
      case 64: return wgreen_setup<2, T>();
      case 128: return wgreen_setup<4, T>();
      case 256: return wgreen_setup<8, T>();
      default: break;
    }
  }
  size_t a = smem_a<T>(N), b = smem_b<T>(N, 16), c = smem_c<T>(N, tile_c<T>());
  // the shared-memory passes serve every N: the attribute only ever grows, so contexts of
  // different grids (concurrent ones included) never lower it under each other
  if ((e = raise_max_dynamic_smem((const void*)pass_a<T, T>, a))) return e;
  if ((e = raise_max_dynamic_smem((const void*)pass_b<T>, b))) return e;
  if ((e = raise_max_dynamic_smem((const void*)pass_c<T>, c))) return e;
  if ((e = raise_max_dynamic_smem((const void*)pass_e<T>, a))) return e;
  // the three-pass kernels run up to small_max only; a plane of a larger grid outgrows a block
  // (FP64: from 112^3 on)
  if (N <= small_max<T>()) {
    const size_t sm = smem_small<T>(N);
    if ((e = raise_max_dynamic_smem((const void*)small_forward<T, false>, sm))) return e;
    if ((e = raise_max_dynamic_smem((const void*)small_inverse<T, false>, sm))) return e;
    if constexpr (sizeof(T) == 8) {
      if ((e = raise_max_dynamic_smem((const void*)small_columns<false>, sm))) return e;
    }
  }
  return cudaSuccess;
}

template <typename T>
cudaError_t green_apply_dot(const T* x, const T* K4, int flgK, T* y, typename Vec2<T>::t* S,
                            const typename Vec2<T>::t* tw, GridDesc g, cudaStream_t st,
                            double* part, int* nparts, const T* rfuse, double* scf) {
  const int N = g.N, H = g.H;
  bool warp_path = false;
  if (nparts) *nparts = 0;
  if (rfuse && !flgK) return cudaErrorInvalidValue;  // the fused update serves G(K : p) only
  {
    warp_path = true;
    switch (N) {
      case 32:
        if constexpr (sizeof(T) == 4)
          wgreen_apply<1, T>(x, K4, nullptr, flgK, y, S, tw, g, st, part, rfuse, scf);
        else
          warp_path = false;
        break;
      case 64: wgreen_apply<2, T>(x, K4, nullptr, flgK, y, S, tw, g, st, part, rfuse, scf); break;
      case 128: wgreen_apply<4, T>(x, K4, nullptr, flgK, y, S, tw, g, st, part, rfuse, scf); break;
      case 256: wgreen_apply<8, T>(x, K4, nullptr, flgK, y, S, tw, g, st, part, rfuse, scf); break;
      default: warp_path = false;
    }
  }
  if (rfuse && !warp_path) return cudaErrorNotSupported;  // the fused update needs the warp passes
  if (N <= small_max<T>() && !warp_path) {
    double* part_a = (g.pre && part && flgK) ? part : nullptr;
    if (part_a && nparts) *nparts = scf ? -1 : 9 * N;
    if constexpr (sizeof(T) == 8) {
      if (N <= 16) {  // split stages: 15^3 35 against 38 us; a call at 17^3 86 against 43, 20^3 62 / 43
        g.plan = split_plan(N);
        small_apply<T, true>(x, K4, flgK, y, S, tw, g, st, part_a, scf);
      } else {
        small_apply<T, false>(x, K4, flgK, y, S, tw, g, st, part_a, scf);
      }
    } else {
      small_apply<T, false>(x, K4, flgK, y, S, tw, g, st, part_a, scf);
    }
    g_kernel_launches += 3;
    return cudaGetLastError();
  }
  if (warp_path) {
    if (part && nparts) *nparts = (N / 2) * N;
    g_kernel_launches += 5;
    return cudaGetLastError();
  }
  g.tkb = 16;
  g.tkc = tile_c<T>();
  const int npair = (N + 1) / 2;
  // the reference-medium operator's product <K : x, x> is summed in pass A; the plain
  // operator's <x, y> is left to the caller on this path
  double* part_a = (g.pre && part && flgK) ? part : nullptr;
  if (part_a && nparts) *nparts = npair * N;
  pass_a<T, T><<<npair * N, PASS_THREADS, smem_a<T>(N), st>>>(x, K4, flgK, S, g, tw, part_a);
  dim3 gb((H + g.tkb - 1) / g.tkb, N, 9);
  pass_b<T><<<gb, PASS_THREADS, smem_b<T>(N, g.tkb), st>>>(S, g, tw, 0);
  dim3 gc((H + g.tkc - 1) / g.tkc, N);
  pass_c<T><<<gc, column_threads<T>(N), smem_c<T>(N, g.tkc), st>>>(S, g, tw);
  pass_b<T><<<gb, PASS_THREADS, smem_b<T>(N, g.tkb), st>>>(S, g, tw, 1);
  pass_e<T><<<npair * N, PASS_THREADS, smem_a<T>(N), st>>>(S, y, g, tw);
  g_kernel_launches += 5;
  return cudaGetLastError();
}

template <typename T>
cudaError_t green_apply(const T* x, const T* K4, int flgK, T* y, typename Vec2<T>::t* S,
                        const typename Vec2<T>::t* tw, GridDesc g, cudaStream_t st) {
  return green_apply_dot<T>(x, K4, flgK, y, S, tw, g, st, nullptr, nullptr, nullptr, nullptr);
}

cudaError_t green_cg_iteration(float* x, float* r, float* p, const float* K4, float2* S,
                               const float2* tw, const GridDesc& g, cudaStream_t st,
                               double* part_a, double* part_e, const float* k0, double* sc,
                               cudaGraphConditionalHandle h, bool uh) {
  switch (g.N) {
    case 32: wcg_iteration<1>(x, r, p, K4, S, tw, g, st, part_a, part_e, k0, sc, h, uh); break;
    case 64: wcg_iteration<2>(x, r, p, K4, S, tw, g, st, part_a, part_e, k0, sc, h, uh); break;
    case 128: wcg_iteration<4>(x, r, p, K4, S, tw, g, st, part_a, part_e, k0, sc, h, uh); break;
    case 256: wcg_iteration<8>(x, r, p, K4, S, tw, g, st, part_a, part_e, k0, sc, h, uh); break;
    default: return cudaErrorNotSupported;
  }
  g_kernel_launches += 5;  // the transform passes (dev_final counts its own launch)
  return cudaGetLastError();
}

cudaError_t green_autotune_f32(const float* x, const float* K4, float* y, float2* S,
                               const float2* tw, GridDesc* g, cudaStream_t st, float* best_ms) {
  if (!green_df_supported(g->N)) return cudaSuccess;
  GridDesc t = *g;
  cudaError_t e = tune_tiles(t, [&](const GridDesc& gg) {
    green_apply_dot<float>(x, K4, 1, y, S, tw, gg, st, nullptr, nullptr, nullptr, nullptr);
  }, st, best_ms, true);
  if (e == cudaSuccess) { g->wtb = t.wtb; g->wtc = t.wtc; g->wc2 = t.wc2; }
  return e;
}


template cudaError_t green_setup<double>(int);
template cudaError_t green_setup<float>(int);
template cudaError_t green_apply<double>(const double*, const double*, int, double*, double2*,
                                         const double2*, GridDesc, cudaStream_t);
template cudaError_t green_apply<float>(const float*, const float*, int, float*, float2*,
                                        const float2*, GridDesc, cudaStream_t);
template cudaError_t green_apply_dot<float>(const float*, const float*, int, float*, float2*,
                                            const float2*, GridDesc, cudaStream_t, double*, int*,
                                            const float*, double*);
