// Kernels of libcfft_b200 for channel grids of any 2-3-5 shape (sm_100a): unequal axes,
// plane groups, and cubic edges without a compile-time sized kernel.
//
// As on the compile-time sized path the inverse gather works by fibers (k_inv_fiber) and the
// orbit expansion feeds the inverse z lines.  Each field has its own workspace slot and
// complex transform: two fields as a + i b would halve the line transforms (GPU us of a round
// trip, paired / alone: P6/mmm 60 x 60 x 80 FP64 x4 43 / 63, Im-3m 160^3 FP64 x8 91 / 119, p4mm
// 160^2 FP64 x64 34 / 35), but the rounding error of one would then scale with the other, and a
// NaN or the imaginary part of an inverse would cross over.  A line of n = A x B points is two
// in-place register passes through one shared-memory buffer, the radices 2 to 16 chosen at
// run time; lengths that do not split that way keep the Stockham kernels of exec.cu (out of
// place, a pass per factor up to 8), which these replace: P6/mmm 60 x 60 x 80 FP64, 4 fields, plane kernels 45 / 47 us,
// z 25 / 25, inverse gather 33 before.
#pragma once

#include "device_common.cuh"
#include "fast_api.h"
#include "launch.cuh"

namespace cfft {
namespace {

// At most.  FP32 keeps two such blocks on an SM with 64 registers, which spills 36 to 284 bytes a
// thread around the larger radices; 384 threads with 80 registers and no spills were slower
// (Pm-3m 90^3, 20 contour steps, 192 us against 176).
constexpr int kGenThreads = 512;

// n / d for n d < 2^32 by one multiplication (mul = ceil(2^32 / d), 0 for d = 1).
__device__ __forceinline__ int div_by(int n, uint32_t mul) {
  return mul ? static_cast<int>(__umulhi(static_cast<uint32_t>(n), mul)) : n;
}

// e^{-2 pi i j / N} of the composite radices as compile-time constants (Taylor series on the
// first octant, folded by symmetry).
struct Unit { double c, s; };
constexpr double series(double x, double first, int k0) {
  double term = first, sum = first;
  for (int k = k0; k < k0 + 30; k += 2) { term *= -x * x / (k * (k + 1)); sum += term; }
  return sum;
}
constexpr Unit unit_root(int j, int N) {
  const int j8 = 8 * (j % N);  // angle in units of 2 pi / (8 N)
  const int oct = j8 / N;      // octant
  const int r = oct % 2 == 0 ? j8 - oct * N : (oct + 1) * N - j8;
  const double x = 6.283185307179586476925286766559 * r / (8.0 * N);
  const double c = series(x, 1.0, 1), s = series(x, x, 2);
  const double cs[8] = {c, s, -s, -c, -c, -s, s, c}, sn[8] = {s, c, c, s, -s, -c, -c, -s};
  return Unit{cs[oct], -sn[oct]};
}
constexpr int small_radix(int n) {
  return n % 8 == 0 && n != 16 ? 8 : n % 4 == 0 ? 4 : n % 5 == 0 ? 5 : n % 3 == 0 ? 3 : 2;
}
template <typename C, bool INV, int N, int Ns, int Rem>
struct RadixFFT {
  static __device__ __forceinline__ void run(C* v) {
    constexpr int R = small_radix(Rem), NB = N / R, STEP = N / (Ns * R);
    C w[N];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int k = j % Ns;
      C x[R];
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = v[j + r * NB];
      if (k != 0) {
#pragma unroll
        for (int r = 1; r < R; ++r) {
          using T = decltype(C::x);
          const C t = mk<C>(static_cast<T>(root(r * k * STEP).c), static_cast<T>(root(r * k * STEP).s));
          x[r] = INV ? cmulc(x[r], t) : cmul(x[r], t);
        }
      }
      dftR<C, INV, R>(x);
      const int o = (j / Ns) * Ns * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) w[o + r * Ns] = x[r];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = w[i];
    RadixFFT<C, INV, N, Ns * R, Rem / R>::run(v);
  }
  // Constant after unrolling: a switch over compile-time roots.
  static __device__ __forceinline__ Unit root(int i) {
    constexpr Unit u[16] = {unit_root(0, N),  unit_root(1, N),  unit_root(2, N),  unit_root(3, N),
                            unit_root(4, N),  unit_root(5, N),  unit_root(6, N),  unit_root(7, N),
                            unit_root(8, N),  unit_root(9, N),  unit_root(10, N), unit_root(11, N),
                            unit_root(12, N), unit_root(13, N), unit_root(14, N), unit_root(15, N)};
    return u[i];
  }
};
template <typename C, bool INV, int N, int Ns>
struct RadixFFT<C, INV, N, Ns, 1> {
  static __device__ __forceinline__ void run(C*) {}
};

#define CFFT_RADIX(R, ...)                                   \
  switch (R) {                                               \
    case 2: { constexpr int RR = 2; __VA_ARGS__; } break;    \
    case 3: { constexpr int RR = 3; __VA_ARGS__; } break;    \
    case 4: { constexpr int RR = 4; __VA_ARGS__; } break;    \
    case 5: { constexpr int RR = 5; __VA_ARGS__; } break;    \
    case 6: { constexpr int RR = 6; __VA_ARGS__; } break;    \
    case 8: { constexpr int RR = 8; __VA_ARGS__; } break;    \
    case 9: { constexpr int RR = 9; __VA_ARGS__; } break;    \
    case 10: { constexpr int RR = 10; __VA_ARGS__; } break;  \
    case 12: { constexpr int RR = 12; __VA_ARGS__; } break;  \
    case 15: { constexpr int RR = 15; __VA_ARGS__; } break;  \
    case 16: { constexpr int RR = 16; __VA_ARGS__; } break;  \
    default: { constexpr int RR = 1; __VA_ARGS__; } break;   \
  }

// One pass over `lines` lines: the butterfly of `radix` values j (< count) of line l is read
// by ld(l, j, r), transformed, multiplied by tw[j k] when TW (the first pass), and written by
// stv(l, j, k, value).  Consecutive threads take consecutive lines.
template <typename C, bool INV, bool TW, int R, typename Load, typename Store>
__device__ __forceinline__ void line_pass_r(int count, int lines, uint32_t dlines, const C* tw, Load ld, Store stv) {
  for (int i = threadIdx.x; i < lines * count; i += blockDim.x) {
    const int j = div_by(i, dlines), l = i - j * lines;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(l, j, r);
    RadixFFT<C, INV, R, 1, R>::run(v);
    if (TW && j) {
#pragma unroll
      for (int k = 1; k < R; ++k) v[k] = INV ? cmulc(v[k], tw[j * k]) : cmul(v[k], tw[j * k]);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) stv(l, j, k, v[k]);
  }
}
template <typename C, bool INV, bool TW, typename Load, typename Store>
__device__ __forceinline__ void line_pass(int radix, int count, int lines, uint32_t dlines, const C* tw, Load ld, Store stv) {
  CFFT_RADIX(radix, (line_pass_r<C, INV, TW, RR>(count, lines, dlines, tw, ld, stv)))
}

template <typename C> __device__ __forceinline__ void copy_twiddles(C* dst, const C* __restrict__ src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
}

// Forward plane kernel: fold (or plain load) of a field, x and y lines, -> W[field][c][z][y][x].
// The fold puts x at position x / B + A (x mod B) (y likewise), so the first pass works on
// contiguous blocks of A and both passes leave frequencies in natural order: the last one
// stores straight to the workspace along x.
template <typename T>
__global__ void __launch_bounds__(kGenThreads, sizeof(T) == 4 ? 2 : 1)
k_gplane_fwd(const GenShape s, const typename Cx<T>::type* __restrict__ tables, const T* __restrict__ f0,
             const T* __restrict__ E, typename Cx<T>::type* __restrict__ W) {
  using C = typename Cx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int H0 = s.H[0], H1 = s.H[1], H2 = s.H[2], nch = s.nch, S = s.S, PL = H1 * S;
  C* tw0 = buf + nch * PL;
  C* tw1 = tw0 + H0;
  copy_twiddles(tw0, tables + s.tw[0], H0);
  copy_twiddles(tw1, tables + s.tw[1], H1);
  pdl_enter();
  const int iz = blockIdx.x, f = blockIdx.y;
  const T zero = static_cast<T>(0);
  const T* src = f0 + static_cast<size_t>(f) * s.mvol;
  const T* Ef = E ? E + static_cast<size_t>(f) * s.mvol : nullptr;
  const int A0 = s.A[0], B0 = s.B[0], A1 = s.A[1], B1 = s.B[1];
  const int plane = H0 * H1;
  auto place = [&](int iy, int ix) {
    const int qx = div_by(ix, s.dB[0]), qy = div_by(iy, s.dB[1]);
    return buf + (qy + A1 * (iy - qy * B1)) * S + qx + A0 * (ix - qx * B0);
  };
  if (!s.centered) {
    constexpr int U = 8;  // values in flight per thread
    for (int e0 = threadIdx.x; e0 < plane; e0 += U * blockDim.x) {
      T v[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int e = e0 + k * blockDim.x;
        v[k] = e < plane ? __ldcs(src + iz * plane + e) : zero;
      }
      if (Ef) {
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int e = e0 + k * blockDim.x;
          if (e < plane) v[k] *= __ldg(Ef + iz * plane + e);
        }
      }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int e = e0 + k * blockDim.x, iy = div_by(e, s.dH[0]);
        if (e < plane) *place(iy, e - iy * H0) = mk<C>(v[k], zero);
      }
    }
  } else {
    const int M0 = 2 * H0, M1 = 2 * H1;
    for (int e = threadIdx.x; e < plane; e += blockDim.x) {
      const int iy = div_by(e, s.dH[0]), ix = e - iy * H0;
      C* d = place(iy, ix);
      T p[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        p[k] = __ldcs(src + ((iz + ((k >> 2) & 1) * H2) * M1 + iy + ((k >> 1) & 1) * H1) * M0 + ix + (k & 1) * H0);
      if (Ef) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          p[k] *= __ldg(Ef + ((iz + ((k >> 2) & 1) * H2) * M1 + iy + ((k >> 1) & 1) * H1) * M0 + ix + (k & 1) * H0);
      }
      wht8(p);
      const C tx = tables[s.ftw[0] + ix], ty = tables[s.ftw[1] + iy], tz = tables[s.ftw[2] + iz];
      const C txy = cmul(tx, ty);
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        const int c = s.chan[o];
        if (c < 0) continue;
        C w = mk<C>(p[o], zero);
        if ((o & 3) == 3) w = cscale(txy, p[o]);
        else if (o & 1) w = cscale(tx, p[o]);
        else if (o & 2) w = cscale(ty, p[o]);
        if (o == 4) w = cscale(tz, p[o]);
        else if (o & 4) w = cmul(w, tz);
        d[c * PL] = w;
      }
    }
  }
  __syncthreads();
  const int Lx = nch * H1, Ly = nch * H0;
  auto at0 = [&](int l, int j, int r) { return buf + l * S + j * A0 + r; };
  line_pass<C, false, true>(A0, B0, Lx, s.dLx, tw0, [&](int l, int j, int r) { return *at0(l, j, r); },
                            [&](int l, int j, int k, C v) { *at0(l, j, k) = v; });
  __syncthreads();
  if (B0 > 1) {
    auto at = [&](int l, int k1, int r) { return buf + l * S + k1 + A0 * r; };
    line_pass<C, false, false>(B0, A0, Lx, s.dLx, tw0, [&](int l, int j, int r) { return *at(l, j, r); },
                               [&](int l, int j, int k, C v) { *at(l, j, k) = v; });
    __syncthreads();
  }
  // y lines: line l = (c, x)
  auto col = [&](int l) { const int c = div_by(l, s.dH[0]); return c * PL + l - c * H0; };
  C* dst = W + static_cast<size_t>(f) * nch * s.hvol + static_cast<size_t>(iz) * plane;
  auto out = [&](int l, int ky) { const int c = div_by(l, s.dH[0]); return dst + static_cast<size_t>(c) * s.hvol + ky * H0 + l - c * H0; };
  if (B1 > 1) {
    line_pass<C, false, true>(A1, B1, Ly, s.dLy, tw1, [&](int l, int j, int r) { return buf[col(l) + (j * A1 + r) * S]; },
                              [&](int l, int j, int k, C v) { buf[col(l) + (j * A1 + k) * S] = v; });
    __syncthreads();
    line_pass<C, false, false>(B1, A1, Ly, s.dLy, tw1, [&](int l, int j, int r) { return buf[col(l) + (j + A1 * r) * S]; },
                               [&](int l, int j, int k, C v) { *out(l, j + A1 * k) = v; });
  } else {
    line_pass<C, false, false>(A1, 1, Ly, s.dLy, tw1, [&](int l, int, int r) { return buf[col(l) + r * S]; },
                               [&](int l, int, int k, C v) { *out(l, k) = v; });
  }
}

// X at a channel point from the packed expansion entry (orbit | phase << 21) and the
// representatives' rows G0P[field / 2][orbit][field & 1].
template <typename C>
__device__ __forceinline__ C expand_point(const uint32_t* __restrict__ et, const C* __restrict__ rp, const C* __restrict__ ph) {
  const uint32_t t = __ldg(et);
  return cmulc(__ldg(rp + 2 * static_cast<size_t>(t & 0x1FFFFFu)), __ldg(ph + (t >> 21)));
}

// Backward plane kernel: inverse y and x lines of W[field][c][iz] (or, for a single z plane,
// of the orbit expansion itself) and the unfold's real part.  Natural order in, so x comes out at
// (x mod A) B + x / A, where the unfold reads it.
template <typename T, bool EXPAND>
__global__ void __launch_bounds__(kGenThreads, sizeof(T) == 4 ? 2 : 1)
k_gplane_bwd(const GenShape s, const typename Cx<T>::type* __restrict__ tables, const typename Cx<T>::type* __restrict__ W,
             const uint32_t* __restrict__ ETP, const typename Cx<T>::type* __restrict__ G0P, const T* __restrict__ E,
             T* __restrict__ f0) {
  using C = typename Cx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int H0 = s.H[0], H1 = s.H[1], H2 = s.H[2], nch = s.nch, S = s.S, PL = H1 * S;
  C* tw0 = buf + nch * PL;
  C* tw1 = tw0 + H0;
  copy_twiddles(tw0, tables + s.tw[0], H0);
  copy_twiddles(tw1, tables + s.tw[1], H1);
  pdl_enter();
  const int iz = blockIdx.x, f = blockIdx.y;
  const int A0 = s.A[0], B0 = s.B[0], A1 = s.A[1], B1 = s.B[1];
  const int plane = H0 * H1, Lx = nch * H1, Ly = nch * H0;
  __syncthreads();
  const C* src = EXPAND ? nullptr : W + static_cast<size_t>(f) * nch * s.hvol + static_cast<size_t>(iz) * plane;
  const C* rp = EXPAND ? G0P + static_cast<size_t>(f >> 1) * s.n_orbits * 2 + (f & 1) : nullptr;
  auto in = [&](int l, int ky) {
    const int c = div_by(l, s.dH[0]);
    const size_t at = static_cast<size_t>(c) * s.hvol + ky * H0 + l - c * H0;
    if constexpr (EXPAND) return expand_point(ETP + at, rp, tables + s.ph);
    else return src[at];
  };
  auto col = [&](int l) { const int c = div_by(l, s.dH[0]); return c * PL + l - c * H0; };
  line_pass<C, true, true>(A1, B1, Ly, s.dLy, tw1, [&](int l, int j, int r) { return in(l, j + B1 * r); },
                           [&](int l, int j, int k, C v) { buf[col(l) + (j + B1 * k) * S] = v; });
  __syncthreads();
  if (B1 > 1) {
    line_pass<C, true, false>(B1, A1, Ly, s.dLy, tw1, [&](int l, int j, int r) { return buf[col(l) + (j * B1 + r) * S]; },
                              [&](int l, int j, int k, C v) { buf[col(l) + (j * B1 + k) * S] = v; });
    __syncthreads();
  }
  line_pass<C, true, true>(A0, B0, Lx, s.dLx, tw0, [&](int l, int j, int r) { return buf[l * S + j + B0 * r]; },
                           [&](int l, int j, int k, C v) { buf[l * S + j + B0 * k] = v; });
  __syncthreads();
  if (B0 > 1) {
    line_pass<C, true, false>(B0, A0, Lx, s.dLx, tw0, [&](int l, int j, int r) { return buf[l * S + j * B0 + r]; },
                              [&](int l, int j, int k, C v) { buf[l * S + j * B0 + k] = v; });
    __syncthreads();
  }
  T* dst = f0 + static_cast<size_t>(f) * s.mvol;
  const T* Ef = E ? E + static_cast<size_t>(f) * s.mvol : nullptr;
  // v / V as two terms, the first rounded down: see div_const.
  const T hi = sizeof(T) == 4 ? static_cast<T>(__double2float_rd(s.inv_v)) : static_cast<T>(s.inv_v);
  const T lo = static_cast<T>(s.inv_v - static_cast<double>(hi));
  auto put = [&](int idx, T v) {
    T a = lo == static_cast<T>(0) ? v * hi : fma(v, hi, v * lo);
    if (Ef) a *= __ldg(Ef + idx);
    __stcs(dst + idx, a);
  };
  for (int e = threadIdx.x; e < plane; e += blockDim.x) {
    const int iy = div_by(e, s.dH[0]), ix = e - iy * H0;
    const int qx = div_by(ix, s.dA[0]), qy = div_by(iy, s.dA[1]);
    const C* d = buf + ((iy - qy * A1) * B1 + qy) * S + (ix - qx * A0) * B0 + qx;
    if (!s.centered) {
      put(iz * plane + e, d->x);
    } else {
      const int M0 = 2 * H0, M1 = 2 * H1;
      const C tx = tables[s.ftw[0] + ix], ty = tables[s.ftw[1] + iy], tz = tables[s.ftw[2] + iz];
      const C txy = cmul(tx, ty);
      T p[8];
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        const int c = s.chan[o];
        C w = mk<C>(static_cast<T>(0), static_cast<T>(0));
        if (c >= 0) {
          w = d[c * PL];
          if ((o & 3) == 3) w = cmulc(w, txy);
          else if (o & 1) w = cmulc(w, tx);
          else if (o & 2) w = cmulc(w, ty);
          if (o & 4) w = cmulc(w, tz);
        }
        p[o] = w.x;
      }
      wht8(p);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        put(((iz + ((k >> 2) & 1) * H2) * M1 + iy + ((k >> 1) & 1) * H1) * M0 + ix + (k & 1) * H0, p[k]);
    }
  }
}

// z lines of one (y, c, field): forward in place on W, or inverse from the orbit expansion
// into W.  Both ends in natural order: the first pass loads, the second stores, along x.
template <typename T, bool INV>
__global__ void __launch_bounds__(kGenThreads, sizeof(T) == 4 ? 2 : 1)
k_gline_z(const GenShape s, const typename Cx<T>::type* __restrict__ tables, const uint32_t* __restrict__ ETP,
          const typename Cx<T>::type* __restrict__ G0P, typename Cx<T>::type* __restrict__ W) {
  using C = typename Cx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);  // [z position][x]
  const int H0 = s.H[0], A = s.A[2], B = s.B[2];
  C* tw = buf + H0 * s.H[2];
  copy_twiddles(tw, tables + s.tw[2], s.H[2]);
  pdl_enter();
  const int y = blockIdx.x, c = blockIdx.y, f = blockIdx.z;
  const size_t plane = static_cast<size_t>(H0) * s.H[1];
  const size_t at = static_cast<size_t>(c) * s.hvol + static_cast<size_t>(y) * H0;
  C* w = W + static_cast<size_t>(f) * s.nch * s.hvol + at;
  const C* rp = INV ? G0P + static_cast<size_t>(f >> 1) * s.n_orbits * 2 + (f & 1) : nullptr;
  auto in = [&](int x, int z) {
    if constexpr (INV) return expand_point(ETP + at + z * plane + x, rp, tables + s.ph);
    else return w[z * plane + x];
  };
  if (B == 1) {
    line_pass<C, INV, false>(A, 1, H0, s.dH[0], tw, [&](int x, int, int r) { return in(x, r); },
                             [&](int x, int, int k, C v) { w[k * plane + x] = v; });
    return;
  }
  __syncthreads();
  line_pass<C, INV, true>(A, B, H0, s.dH[0], tw, [&](int x, int j, int r) { return in(x, j + B * r); },
                          [&](int x, int j, int k, C v) { buf[(j + B * k) * H0 + x] = v; });
  __syncthreads();
  line_pass<C, INV, false>(B, A, H0, s.dH[0], tw, [&](int x, int j, int r) { return buf[(j * B + r) * H0 + x]; },
                           [&](int x, int j, int k, C v) { w[(j + A * k) * plane + x] = v; });
}

// Spectral-ASU gather from W: F(h) = sum_r e^{-2 pi i h.t_r / N} G0(R_r^T h mod M).  Indices
// are computed on the fly (h and R are small, the moduli multiplications).
template <typename T>
__global__ void __launch_bounds__(128)
k_grecon(const GenShape s, const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
         const uint32_t* __restrict__ spec_h, const T* __restrict__ K, const typename Cx<T>::type* __restrict__ W,
         typename Cx<T>::type* __restrict__ F) {
  using C = typename Cx<T>::type;
  __shared__ int sR[8][9], sT[8][3];
  const int D = s.d;
  for (int i = threadIdx.x; i < D * 9; i += blockDim.x) sR[i / 9][i % 9] = g->rep_R[i / 9][i % 9];
  for (int i = threadIdx.x; i < D * 3; i += blockDim.x) {
    const int t = g->rep_t[i / 3][i % 3] % s.N[i % 3];
    sT[i / 3][i % 3] = t < 0 ? t + s.N[i % 3] : t;
  }
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;
  const uint32_t hp = __ldg(spec_h + min(i, s.n_spec - 1));
  pdl_enter();
  if (i >= s.n_spec) return;
  const int h[3] = {static_cast<int>(hp & 1023u), static_cast<int>((hp >> 10) & 1023u), static_cast<int>((hp >> 20) & 1023u)};
  const C* Wb = W + static_cast<size_t>(f) * s.nch * s.hvol;
  const int sh = s.centered ? 1 : 0;
  C acc = mk<C>(static_cast<T>(0), static_cast<T>(0));
#pragma unroll 4
  for (int r = 0; r < D; ++r) {
    int q[3], j = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      // |v| <= 3 x 1023; a multiple of M above that makes it positive
      const int v = sR[r][d] * h[0] + sR[r][3 + d] * h[1] + sR[r][6 + d] * h[2] + s.lift[d];
      q[d] = v - div_by(v, s.dM[d]) * s.M[d];
      const int a = h[d] * sT[r][d];
      j += (a - div_by(a, s.dN[d]) * s.N[d]) * s.PN[d];
    }
    if (j >= s.P) j -= s.P;
    if (j >= s.P) j -= s.P;
    int c = 0;
    if (s.centered) {
      c = s.chan[(q[0] & 1) + 2 * (q[1] & 1) + 4 * (q[2] & 1)];
      if (c < 0) continue;
    }
    const C* Wc = Wb + static_cast<size_t>(c) * s.hvol;
    const C X = __ldg(Wc + (static_cast<size_t>(q[2] >> sh) * s.H[1] + (q[1] >> sh)) * s.H[0] + (q[0] >> sh));
    acc = cadd(acc, cmul(X, __ldg(tables + s.ph + j)));
  }
  if (K) acc = cscale(acc, K[i]);
  F[static_cast<size_t>(f) * s.n_spec + i] = acc;
}

inline int gen_threads(long items) {  // one butterfly or value per thread, in warps
  const long t = (items + 31) / 32 * 32;
  return static_cast<int>(t < 64 ? 64 : t > kGenThreads ? kGenThreads : t);
}

template <typename T>
Status gen_unit_init(std::string* err) {
  cudaError_t e = cudaSuccess;
  for (const void* k : {reinterpret_cast<const void*>(k_gplane_fwd<T>), reinterpret_cast<const void*>(k_gplane_bwd<T, false>),
                        reinterpret_cast<const void*>(k_gplane_bwd<T, true>), reinterpret_cast<const void*>(k_gline_z<T, false>),
                        reinterpret_cast<const void*>(k_gline_z<T, true>)})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  return fast_cuda(e, "general kernels' shared-memory attribute", err);
}

template <typename T>
Status gen_unit_launch(const FastArgs& a, const GenShape& s, std::string* err) {
  using C = typename Cx<T>::type;
  const C* tab = static_cast<const C*>(a.tables);
  C* W = static_cast<C*>(a.W);
  const uint32_t* et = static_cast<const uint32_t*>(a.expand);
  const C* rep = static_cast<const C*>(a.G0R);
  cudaStream_t st = static_cast<cudaStream_t>(a.stream);
  const size_t cs = sizeof(C);
  const size_t smem_p = (static_cast<size_t>(s.nch) * s.H[1] * s.S + s.H[0] + s.H[1]) * cs;
  const size_t smem_z = (static_cast<size_t>(s.H[0]) * s.H[2] + s.H[2]) * cs;
  const int thr_p = gen_threads(static_cast<long>(s.nch) * s.H[1] * s.B[0]);
  const int thr_z = gen_threads(static_cast<long>(s.H[0]) * s.B[2]);
  const dim3 gp(s.H[2], a.nb), gz(s.H[1], s.nch, a.nb);
  switch (a.stage) {
    case 0:
      launch_k(k_gplane_fwd<T>, gp, thr_p, smem_p, st, s, tab, static_cast<const T*>(a.f0), static_cast<const T*>(a.E), W);
      break;
    case 1:
      launch_k(k_gline_z<T, false>, gz, thr_z, smem_z, st, s, tab, nullptr, nullptr, W);
      break;
    case 2:
      launch_k(k_grecon<T>, dim3((s.n_spec + 127) / 128, a.nb), 128, 0, st, s, static_cast<const DevGeom*>(a.geom), tab,
               static_cast<const uint32_t*>(a.spec_h), a.use_K ? static_cast<const T*>(a.K) : nullptr, W, static_cast<C*>(a.F));
      break;
    case 4:
      launch_k(k_gline_z<T, true>, gz, thr_z, smem_z, st, s, tab, et, rep, W);
      break;
    default:
      if (s.H[2] == 1)
        launch_k(k_gplane_bwd<T, true>, gp, thr_p, smem_p, st, s, tab, W, et, rep, static_cast<const T*>(a.E), static_cast<T*>(a.f0_out));
      else
        launch_k(k_gplane_bwd<T, false>, gp, thr_p, smem_p, st, s, tab, W, nullptr, nullptr, static_cast<const T*>(a.E),
                 static_cast<T*>(a.f0_out));
      break;
  }
  const cudaError_t le = launch_error();
  launch_error() = cudaSuccess;
  const cudaError_t ge = cudaGetLastError();
  return fast_cuda(le != cudaSuccess ? le : ge, "general launch", err);
}

}  // namespace
}  // namespace cfft
