// green_small.cuh -- tiles of G(K : x) on small grids: the transforms along the two fastest
// axes of one component's plane in one tile, so the operator is three passes (planes, columns
// with the Green contraction, planes) instead of five.  Used by the kernels of fft_green.cu
// and by the one-launch CG of cg_small.cu.
//
// A small grid is bound by latency.  An FP64 warp instruction holds its SM quarter for 64
// clocks whatever the number of active lanes and whatever else is in flight (measured: one
// warp, 1 to 32 lanes, 1 to 8 independent chains), so a tile takes as long as its longest
// chain of FP64 instructions, and each pass adds a launch or grid barrier and a round trip
// to L2.  SPLIT stages give each real part of each output to a thread of its own (2 R
// instructions deep, the twiddle folded into the DFT matrix) where a register butterfly is
// about 60 deep for radix 5: twice the instructions, but in lanes that a small tile leaves
// idle.
#pragma once
#include <algorithm>

#include "green_passes.cuh"

namespace {

// One forward Stockham stage of radix R on ncols columns: the sums over r of
// src[j + r N/R] exp(-2 pi i r (jm N/(Ns R) + s N/R) / N), a thread per real part.  Even R: a
// thread forms outputs s and s + R/2, the sum and difference of its even and odd r.  Two partial
// sums in either case keep the rounding at a butterfly's (one chain of 2 R - 2 products: G(x)
// at 13^3 4.4e-16 from long double, this 3.6e-16, the five-pass form 3.7e-16).
template <typename T2, typename T>
__device__ __forceinline__ void stage_split(const T2* src, T2* dst, int ncols, int cs, int N,
                                            int R, int Ns, const T2* tw) {
  const bool paired = (R & 1) == 0;
  const int NR = N / R, tstride = NR / Ns, per = paired ? N / 2 : N, items = ncols * per;
  const float iper = 1.0f / (float)per, iNR = 1.0f / (float)NR, iNs = 1.0f / (float)Ns;
  for (int t = threadIdx.x; t < 2 * items; t += blockDim.x) {
    const bool im = t >= items;
    const int u = im ? t - items : t;
    const int col = fdiv(u, iper), rem = u - col * per;
    const int s = fdiv(rem, iNR), j = rem - s * NR;
    const int jq = fdiv(j, iNs), jm = j - jq * Ns;
    int step = jm * tstride + s * NR;
    if (step >= N) step -= N;
    const T2* c = src + col * cs;
    T2* d = dst + col * cs;
    const int o = jq * Ns * R + jm + s * Ns;
    T a = im ? c[pidx(j)].y : c[pidx(j)].x, b = 0;
    int e = 0;
    auto next = [&](int r, T2& v, T2& w) {
      e += step;
      if (e >= N) e -= N;
      v = c[pidx(j + r * NR)];
      w = tw[e];
    };
    T2 v, w;
    if (paired) {
      for (int r = 1; r < R; r++) {
        next(r, v, w);
        b += v.x * (im ? w.y : w.x);
        b += im ? v.y * w.x : -v.y * w.y;
        if (++r == R) break;
        next(r, v, w);
        a += v.x * (im ? w.y : w.x);
        a += im ? v.y * w.x : -v.y * w.y;
      }
      if (im) {
        d[pidx(o)].y = a + b;
        d[pidx(o + R / 2 * Ns)].y = a - b;
      } else {
        d[pidx(o)].x = a + b;
        d[pidx(o + R / 2 * Ns)].x = a - b;
      }
    } else {
      for (int r = 1; r < R; r++) {
        next(r, v, w);
        a += v.x * (im ? w.y : w.x);
        b += im ? v.y * w.x : -v.y * w.y;
      }
      if (im) d[pidx(o)].y = a + b;
      else d[pidx(o)].x = a + b;
    }
  }
}

template <typename T2, typename T, bool SPLIT>
__device__ __forceinline__ T2* small_cols(T2* a, T2* b, int ncols, int cs, const FftPlan& P,
                                          const T2* tw) {
  if constexpr (SPLIT) {
    for (int s = 0; s < P.nst; s++) {
      stage_split<T2, T>(a, b, ncols, cs, P.n, P.R[s], P.Ns[s], tw);
      __syncthreads();
      T2* t = a; a = b; b = t;
    }
    return a;
  } else {
    return fft_cols<T2, T>(a, b, ncols, cs, P, tw);
  }
}

// columns of a plane tile's buffers: line pairs of the fastest axis, then half-spectrum columns
__host__ __device__ __forceinline__ int plane_cols(int N) { return N / 2 + 1; }

// Forward transforms of one component's plane (component i, plane c0) into S; y(u) gives the
// field at voxel u of the plane.  b0, b1: plane_cols(N) columns each.
template <typename T2, typename T, bool SPLIT, typename F>
__device__ __forceinline__ void plane_forward(F&& y, T2* S, int i, int c0, const GridDesc& g,
                                              const T2* tw, T2* b0, T2* b1) {
  const int N = g.N, H = g.H, Lp = padlen(N), np = (N + 1) / 2;
  const float iN = 1.0f / (float)N, iH = 1.0f / (float)H;
  __syncthreads();  // the buffers' last readers are done
  for (int t = threadIdx.x; t < 2 * np * N; t += blockDim.x) {
    const int b = fdiv(t, iN), a = t - b * N;
    const T v = b < N ? y(t) : (T)0;
    T2* d = b0 + (b >> 1) * Lp + pidx(a);
    if (b & 1) d->y = v;
    else d->x = v;
  }
  __syncthreads();
  T2* r = small_cols<T2, T, SPLIT>(b0, b1, np, Lp, g.plan, tw);
  T2* o = r == b0 ? b1 : b0;
  for (int t = threadIdx.x; t < np * H; t += blockDim.x) {
    const int lp = fdiv(t, iH), k = t - lp * H;
    const T2 z = r[lp * Lp + pidx(k)], w = conjg(r[lp * Lp + pidx(k ? N - k : 0)]);
    T2 X0, X1;
    X0.x = (T)0.5 * (z.x + w.x); X0.y = (T)0.5 * (z.y + w.y);
    X1.x = (T)0.5 * (z.y - w.y); X1.y = (T)-0.5 * (z.x - w.x);
    T2* col = o + k * Lp;
    col[pidx(2 * lp)] = X0;
    if (2 * lp + 1 < N) col[pidx(2 * lp + 1)] = X1;
  }
  __syncthreads();
  r = small_cols<T2, T, SPLIT>(o, r, H, Lp, g.plan, tw);
  T2* plane = S + ((long long)i * N + c0) * N * H;
  for (int t = threadIdx.x; t < N * H; t += blockDim.x) {
    const int kb = fdiv(t, iH), ka = t - kb * H;
    plane[t] = r[ka * Lp + pidx(kb)];
  }
}

// Inverse transforms of one component's plane; out(u, v) takes the value at voxel u
template <typename T2, typename T, bool SPLIT, typename F>
__device__ __forceinline__ void plane_inverse(F&& out, const T2* S, int i, int c0,
                                              const GridDesc& g, const T2* tw, T2* b0, T2* b1) {
  const int N = g.N, H = g.H, Lp = padlen(N), np = (N + 1) / 2;
  const float iN = 1.0f / (float)N, iH = 1.0f / (float)H;
  const bool even = (N & 1) == 0;
  const T2* plane = S + ((long long)i * N + c0) * N * H;
  __syncthreads();
  for (int t = threadIdx.x; t < N * H; t += blockDim.x) {
    const int kb = fdiv(t, iH), ka = t - kb * H;
    b0[ka * Lp + pidx(kb)] = conjg(plane[t]);
  }
  __syncthreads();
  T2* r = small_cols<T2, T, SPLIT>(b0, b1, H, Lp, g.plan, tw);
  T2* o = r == b0 ? b1 : b0;
  // r holds the conjugates; conj(Z), Z = X0 + i X1, of each line pair for the next inverse
  for (int t = threadIdx.x; t < np * N; t += blockDim.x) {
    const int lp = fdiv(t, iN), k = t - lp * N;
    const int kk = k < H ? k : N - k;
    T2 X0 = conjg(r[kk * Lp + pidx(2 * lp)]), X1;
    X1.x = 0; X1.y = 0;
    if (2 * lp + 1 < N) X1 = conjg(r[kk * Lp + pidx(2 * lp + 1)]);
    if (kk == 0 || (even && kk == N / 2)) { X0.y = 0; X1.y = 0; }
    if (k >= H) { X0.y = -X0.y; X1.y = -X1.y; }
    T2 z;
    z.x = X0.x - X1.y;
    z.y = -(X0.y + X1.x);
    o[lp * Lp + pidx(k)] = z;
  }
  __syncthreads();
  r = small_cols<T2, T, SPLIT>(o, r, np, Lp, g.plan, tw);
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
    const int b = fdiv(t, iN), a = t - b * N;
    const T2 z = r[(b >> 1) * Lp + pidx(a)];  // conj of the unscaled inverse
    out(t, b & 1 ? -z.y : z.x);
  }
}

constexpr int SMALL_TKC = 2;  // ka columns of a column tile (three components each)

// Columns (kb, ka0 ..) along the slowest axis of the three components of one row, with the
// plain Green contraction (which acts row by row).  b0, b1: 3 SMALL_TKC columns each.
template <typename T2, typename T, bool SPLIT>
__device__ __forceinline__ void column_tile(T2* S, int row, int kb, int ka0, const GridDesc& g,
                                            const T2* tw, T2* b0, T2* b1) {
  constexpr int TK = SMALL_TKC;
  const int N = g.N, H = g.H, Lp = padlen(N), i0 = 3 * row;
  const float iN = 1.0f / (float)N;
  const long long cstr = (long long)N * H;
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * TK * N; t += blockDim.x) {
    const int rem = t / TK, kk = t % TK;
    const int i = fdiv(rem, iN), c = rem - i * N;
    T2 v;
    v.x = 0; v.y = 0;
    if (ka0 + kk < H) v = S[((long long)(i0 + i) * N + c) * cstr + (long long)kb * H + ka0 + kk];
    b0[(i * TK + kk) * Lp + pidx(c)] = v;
  }
  __syncthreads();
  T2* r = small_cols<T2, T, SPLIT>(b0, b1, 3 * TK, Lp, g.plan, tw);
  T2* o = r == b0 ? b1 : b0;
  const int Nh = g.Nhalf, gm = g.gmap;
  const bool even = (N & 1) == 0;
  for (int t = threadIdx.x; t < N * TK; t += blockDim.x) {
    const int kc = t / TK, kk = t % TK, ka = ka0 + kk;
    const bool nyq = gm == CPFFT_G_CENTERED && even && (2 * kc == N || 2 * kb == N || 2 * ka == N);
    T2 A[3], out[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      A[i] = r[(i * TK + kk) * Lp + pidx(kc)];
      out[i].x = 0; out[i].y = 0;
    }
    if (ka < H && !nyq) {
      const int p0 = qmap(kc, N, Nh, gm), p1 = qmap(kb, N, Nh, gm), p2 = qmap(ka, N, Nh, gm);
      const int m0 = qmap(kc ? N - kc : 0, N, Nh, gm), m1 = qmap(kb ? N - kb : 0, N, Nh, gm),
                m2 = qmap(ka ? N - ka : 0, N, Nh, gm);
      const bool sym = m0 == -p0 && m1 == -p1 && m2 == -p2;
      const T w = sym ? (T)g.inv_n3 : (T)0.5 * (T)g.inv_n3;
      green_row_plain<T2, T>(A, p0, p1, p2, w, out);
      if (!sym) green_row_plain<T2, T>(A, m0, m1, m2, w, out);
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      out[i].y = -out[i].y;
      o[(i * TK + kk) * Lp + pidx(kc)] = out[i];
    }
  }
  __syncthreads();
  r = small_cols<T2, T, SPLIT>(o, r, 3 * TK, Lp, g.plan, tw);
  for (int t = threadIdx.x; t < 3 * TK * N; t += blockDim.x) {
    const int rem = t / TK, kk = t % TK;
    const int i = fdiv(rem, iN), c = rem - i * N;
    if (ka0 + kk < H)
      S[((long long)(i0 + i) * N + c) * cstr + (long long)kb * H + ka0 + kk] =
          conjg(r[(i * TK + kk) * Lp + pidx(c)]);
  }
}

// stages of the split transform: fours, then the primes (2 R instructions each)
inline FftPlan split_plan(int N) {
  FftPlan p;
  p.n = N;
  p.nst = 0;
  int m = N, Ns = 1;
  auto push = [&](int r) {
    p.R[p.nst] = r;
    p.Ns[p.nst++] = Ns;
    Ns *= r;
    m /= r;
  };
  while (m % 4 == 0) push(4);
  for (int f = 2; m > 1; f++)
    while (m % f == 0) push(f);
  return p;
}

template <typename T>
size_t smem_small(int N) {
  const int cols = std::max(plane_cols(N), 3 * SMALL_TKC);
  return sizeof(typename Vec2<T>::t) * (size_t)(N + 2 * cols * padlen(N));
}

}  // namespace
