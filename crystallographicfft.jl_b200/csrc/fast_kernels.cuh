// Compile-time sized fast-path kernels of libcfft_b200 (sm_100a).  Included by the four
// fast_*.cu translation units; each defines CFFT_FAST_T (float/double) and
// CFFT_FAST_GROUP (0: plane stages 0 and 5, 1: stages 1-4) before including it, so
// every unit instantiates only its own kernels.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include <cooperative_groups.h>

#include "device_common.cuh"
#include "fast_api.h"
#include "launch.cuh"

namespace cfft {
namespace {

// ---------------------------------------------------------------- compile-time sized path
// For cubic channel grids with H in {4, 6, 8, 12, 16, 24, 32, 48} every line FFT is a
// fully unrolled mixed-radix Stockham in registers (one thread per line), with its
// twiddles in constant memory, so no runtime division or shared-memory pass remains
// inside an FFT.  Shared-memory rows are padded to an odd stride (H + 1 complex) so
// row and column accesses of a warp are bank-conflict free.

// Drop one 128-byte L2 line without writing it back (its contents become undefined).
// Used on channel-workspace lines that have been read for the last time, so the dirty
// intermediate never travels to HBM.
__device__ __forceinline__ void discard_l2_line(const void* p) {
  asm volatile("discard.global.L2 [%0], 128;\n" ::"l"(p) : "memory");
}

constexpr int kTwOff4 = 0, kTwOff6 = 4, kTwOff8 = 10, kTwOff12 = 18, kTwOff16 = 30, kTwOff24 = 46,
              kTwOff32 = 70, kTwOff48 = 102, kTwTotal = 150;
__constant__ float2 c_tw_f[kTwTotal];
__constant__ double2 c_tw_d[kTwTotal];

template <int N> constexpr int tw_offset() {
  return N == 4 ? kTwOff4 : N == 6 ? kTwOff6 : N == 8 ? kTwOff8 : N == 12 ? kTwOff12 : N == 16 ? kTwOff16
       : N == 24 ? kTwOff24 : N == 32 ? kTwOff32 : kTwOff48;
}
constexpr int pick_radix(int rem) { return rem % 8 == 0 ? 8 : rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : rem % 3 == 0 ? 3 : 5; }

template <typename C> __device__ __forceinline__ C ctw(int i);
template <> __device__ __forceinline__ float2 ctw<float2>(int i) { return c_tw_f[i]; }
template <> __device__ __forceinline__ double2 ctw<double2>(int i) { return c_tw_d[i]; }

template <typename C, bool INV, int N, int Ns, int Rem>
struct RegFFT {
  static __device__ __forceinline__ void run(C* v) {
    constexpr int R = pick_radix(Rem);
    constexpr int NB = N / R;
    constexpr int STEP = N / (Ns * R);
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
          const C t = ctw<C>(tw_offset<N>() + r * k * STEP);
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
    RegFFT<C, INV, N, Ns * R, Rem / R>::run(v);
  }
};
template <typename C, bool INV, int N, int Ns>
struct RegFFT<C, INV, N, Ns, 1> {
  static __device__ __forceinline__ void run(C*) {}
};
template <typename C, bool INV, int N> __device__ __forceinline__ void reg_fft(C* v) { RegFFT<C, INV, N, 1, N>::run(v); }

// Alive parity channels per centring (WHT index o = o0 + 2 o1 + 4 o2 of each channel),
// as compile-time data so channel loops unroll with constant register indices.
// CT: 0 plain (no fold), 1 I, 2 F, 3 C, 4 A (same order as the plan's offsets).
template <int CT> struct Cent {
  static constexpr int n = CT == 0 ? 1 : CT == 2 ? 2 : 4;
  static __host__ __device__ constexpr int off(int c) {
    return CT == 1 ? (c == 0 ? 0 : c == 1 ? 3 : c == 2 ? 5 : 6)
         : CT == 2 ? (c == 0 ? 0 : 7)
         : CT == 3 ? (c == 0 ? 0 : c == 1 ? 3 : c == 2 ? 4 : 7)
         : CT == 4 ? (c == 0 ? 0 : c == 1 ? 6 : c == 2 ? 1 : 7) : 0;
  }
};

// Two real fields share one complex transform on the fast path: slot s of the
// channel workspace holds g_a + i g_b for fields a = 2s and b = 2s + 1 (b may be
// absent at the end of a batch).  The forward gather separates them with
// G_a(p) = (X(p) + conj X(-p)) / 2 and G_b(p) = (X(p) - conj X(-p)) / 2i, the backward
// builds X = G_a + i G_b and the unfold reads field a from the real part and field b
// from the imaginary part.  This halves the FFT work and the workspace traffic.

// Place of column x in a row that is written or read VW consecutive values per thread:
// value l of thread m sits at l * (H / VW) + m, so the lanes of a warp access
// neighbouring words (natural order makes them VW-way bank conflicts).  The x-line pass,
// one row per thread, takes either order at no cost.
template <int H, int VW> constexpr __host__ __device__ int fold_pos(int x) { return (x % VW) * (H / VW) + x / VW; }

// Item e of the vector fold and unfold: columns ix0 .. ix0 + VW - 1 of row iy.  The rows a
// warp touches lie H / (rows per warp) apart: with the odd row stride their words then
// fall into different banks (adjacent rows overlap in all but one).
template <int H, int VW> __device__ __forceinline__ void fold_item(int e, int* ix0, int* iy) {
  constexpr int PR = H / VW;                                  // items per row
  constexpr int RW = PR < 32 && 32 % PR == 0 && H % (32 / PR) == 0 ? 32 / PR : 1;  // rows per warp
  const int r = e / PR;
  *ix0 = (e % PR) * VW;
  *iy = (r % RW) * (H / RW) + r / RW;
}

// Row / column FFTs of nch padded planes for a group of threads (gtid of gnth); rows are
// read in fold_pos<H, PI> order and left in fold_pos<H, PO> order.
template <typename C, bool INV, int H, int PI = 1, int PO = 1>
__device__ __forceinline__ void group_rows(C* buf, int nlines, int tid, int nth) {
  constexpr int S = H + 1;
  for (int l = tid; l < nlines; l += nth) {
    C* p = buf + l * S;
    C v[H];
#pragma unroll
    for (int i = 0; i < H; ++i) v[i] = p[fold_pos<H, PI>(i)];
    reg_fft<C, INV, H>(v);
#pragma unroll
    for (int i = 0; i < H; ++i) p[fold_pos<H, PO>(i)] = v[i];
  }
}
template <typename C, bool INV, int H>
__device__ __forceinline__ void group_cols(C* buf, int nlines, int tid, int nth) {
  constexpr int S = H + 1;
  for (int l = tid; l < nlines; l += nth) {
    C* p = buf + (l / H) * (H * S) + (l % H);
    C v[H];
#pragma unroll
    for (int i = 0; i < H; ++i) v[i] = p[i * S];
    reg_fft<C, INV, H>(v);
#pragma unroll
    for (int i = 0; i < H; ++i) p[i * S] = v[i];
  }
}

// Fold of VW consecutive x values (ix0 .. ix0 + VW - 1) of channel row iy: the eight
// octant values of fields a and b (va[k], vb[k], octant k = kx + 2 ky + 4 kz) go through
// the WHT8, each alive channel takes its fold twiddle, and the results land in the
// padded planes at buf (PV > 1: columns at fold_pos<H, PV>).
template <typename T, int H, int CT, int VW, int PV = 1>
__device__ __forceinline__ void fold_emit(const T (&va)[8][VW], const T (&vb)[8][VW], int ix0, int iy,
                                          const typename Cx<T>::type* __restrict__ ftx,
                                          typename Cx<T>::type ftz, typename Cx<T>::type* buf) {
  using C = typename Cx<T>::type;
  constexpr int S = H + 1;
  constexpr int PL = H * S;
  constexpr int nch = Cent<CT>::n;
  const T zero = static_cast<T>(0);
  const C ty = ftx[iy];
#pragma unroll
  for (int l = 0; l < VW; ++l) {
    C p8[8];  // field a in the real lane, field b in the imaginary lane
#pragma unroll
    for (int k = 0; k < 8; ++k) p8[k] = mk<C>(va[k][l], vb[k][l]);
    wht8c(p8);
    const int ix = ix0 + l;
    const C tx = ftx[ix];
#pragma unroll
    for (int c = 0; c < nch; ++c) {
      const int o = Cent<CT>::off(c);
      C w = mk<C>(static_cast<T>(1), zero);
      if (o & 1) w = tx;
      if (o & 2) w = cmul(w, ty);
      if (o & 4) w = cmul(w, ftz);
      buf[c * PL + iy * S + fold_pos<H, PV>(ix)] = o ? cmul(p8[o], w) : p8[o];
    }
  }
}

// Fold (or plain load, CT = 0) of the two fields of one slot at channel z-plane iz into
// the nch padded planes at buf (channel c at buf + c * H * (H + 1)), with the fold
// twiddles e^{-2 pi i off.n / M} and the interaction factors E when given.  Work is
// spread over threads tid of nth.
template <typename T, int H, int CT, int PV = 1>
__device__ __forceinline__ void fold_plane(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                                           const T* __restrict__ srca, const T* __restrict__ srcb,
                                           const T* __restrict__ Ea, const T* __restrict__ Eb, bool has_b, bool USE_E,
                                           int iz, typename Cx<T>::type* buf, int tid, int nth) {
  using C = typename Cx<T>::type;
  constexpr int S = H + 1;
  constexpr int PL = H * S;
  constexpr int nch = Cent<CT>::n;
  const T zero = static_cast<T>(0);
  if constexpr (CT == 0) {
    const size_t zoff = static_cast<size_t>(iz) * H * H;
    for (int e = tid; e < H * H; e += nth) {
      T va = srca[zoff + e];
      T vb = has_b ? srcb[zoff + e] : zero;
      if (USE_E) { va *= Ea[zoff + e]; if (has_b) vb *= Eb[zoff + e]; }
      buf[(e / H) * S + fold_pos<H, PV>(e % H)] = mk<C>(va, vb);
    }
  } else {
    constexpr int M = 2 * H;
    constexpr int VW = 16 / static_cast<int>(sizeof(T));  // elements per 16-byte vector
    using V = typename Vec16<T>::type;
    const C* ftx = tables + g->ftw_off[0];
    const C ftz = tables[g->ftw_off[2] + iz];
    const bool vec = (H % VW == 0) && (reinterpret_cast<uintptr_t>(srca) % 16 == 0) &&
                     (!USE_E || reinterpret_cast<uintptr_t>(Ea) % 16 == 0);
    if (vec) {
      for (int e = tid; e < H * H / VW; e += nth) {
        int ix0, iy;
        fold_item<H, VW>(e, &ix0, &iy);
        // All sixteen field loads first (field a stands in for a missing b), then the factors:
        // interleaved, every octant's product waits for its own loads before the next
        // octant's are issued.
        T va[8][VW], vb[8][VW];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix0 + (k & 1) * H;
          vload_stream<T>(va[k], srca + idx);
          vload_stream<T>(vb[k], (has_b ? srcb : srca) + idx);
        }
        if (!has_b) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int l = 0; l < VW; ++l) vb[k][l] = zero;
        }
        if (USE_E) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix0 + (k & 1) * H;
            T ea[VW], eb[VW];
            vload_nc<T>(ea, Ea + idx);
            vload_nc<T>(eb, (has_b ? Eb : Ea) + idx);
#pragma unroll
            for (int l = 0; l < VW; ++l) { va[k][l] *= ea[l]; vb[k][l] *= eb[l]; }
          }
        }
        fold_emit<T, H, CT, VW, PV>(va, vb, ix0, iy, ftx, ftz, buf);
      }
    } else {
      for (int e = tid; e < H * H; e += nth) {
        const int ix = e % H, iy = e / H;
        T va[8], vb[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix + (k & 1) * H;
          va[k] = srca[idx];
          vb[k] = has_b ? srcb[idx] : zero;
          if (USE_E) { va[k] *= Ea[idx]; if (has_b) vb[k] *= Eb[idx]; }
        }
        wht8(va);
        wht8(vb);
        const C tx = ftx[ix], ty = ftx[iy];  // cubic: the y fold twiddle table equals x's
#pragma unroll
        for (int c = 0; c < nch; ++c) {
          const int o = Cent<CT>::off(c);
          C w = mk<C>(static_cast<T>(1), zero);
          if (o & 1) w = tx;
          if (o & 2) w = cmul(w, ty);
          if (o & 4) w = cmul(w, ftz);
          buf[c * PL + iy * S + fold_pos<H, PV>(ix)] = cmul(mk<C>(va[o], vb[o]), w);
        }
      }
    }
  }
}

// v / V for the inverse transform's normalisation.  1/V rounded to FP32 is off by 7.5e-9
// for edges with a factor 3, the same way in every step of a contour loop (7.5e-7 after a
// hundred); its remainder as a second term makes the product correct to a rounding, which
// does not accumulate.  Powers of two have no remainder.  The first term is rounded down, so
// that the remainder is positive and an overflowed sum stays infinite (inf - inf would be NaN).
template <typename T> constexpr T round_down(double x) {  // x in the normal range
  const T r = static_cast<T>(x);
  return static_cast<double>(r) > x ? static_cast<T>(x * (1.0 - 0x1p-24)) : r;
}
template <typename T, int V> __device__ __forceinline__ T div_const(T v) {
  constexpr T hi = round_down<T>(1.0 / V);
  constexpr T lo = sizeof(T) == 4 ? static_cast<T>(1.0 / V - static_cast<double>(hi)) : static_cast<T>(0);
  if constexpr (lo == static_cast<T>(0)) return v * hi;
  else return fma(v, hi, v * lo);
}

// Unfold of the nch inverse-transformed planes at buf (channel z-plane iz) into the two
// fields of the slot: conjugate fold twiddle, inverse WHT8 / 8, real part -> field a,
// imaginary part -> field b, times E when given.
template <typename T, int H, int CT, bool VEC = false, int PV = 1>
__device__ __forceinline__ void unfold_plane(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                                             const typename Cx<T>::type* buf, T* __restrict__ dsta, T* __restrict__ dstb,
                                             const T* __restrict__ Ea, const T* __restrict__ Eb, bool has_b, bool USE_E,
                                             int iz, int tid, int nth) {
  using C = typename Cx<T>::type;
  constexpr int S = H + 1;
  constexpr int PL = H * S;
  constexpr int nch = Cent<CT>::n;
  if constexpr (CT == 0) {
    constexpr int V = H * H * H;
    const size_t zoff = static_cast<size_t>(iz) * H * H;
    for (int e = tid; e < H * H; e += nth) {
      const C x = buf[(e / H) * S + fold_pos<H, PV>(e % H)];
      T va = div_const<T, V>(x.x), vb = div_const<T, V>(x.y);
      if (USE_E) { va *= Ea[zoff + e]; if (has_b) vb *= Eb[zoff + e]; }
      dsta[zoff + e] = va;
      if (has_b) dstb[zoff + e] = vb;
    }
  } else {
    constexpr int M = 2 * H;
    constexpr int V = 8 * H * H * H;
    const C* ftx = tables + g->ftw_off[0];
    const C ftz = tables[g->ftw_off[2] + iz];
    constexpr int VW = 16 / static_cast<int>(sizeof(T));  // elements per 16-byte vector
    const bool vec = VEC && (H % VW == 0) && (reinterpret_cast<uintptr_t>(dsta) % 16 == 0) &&
                     (!has_b || reinterpret_cast<uintptr_t>(dstb) % 16 == 0) &&
                     (!USE_E || (reinterpret_cast<uintptr_t>(Ea) % 16 == 0 && (!has_b || reinterpret_cast<uintptr_t>(Eb) % 16 == 0)));
    if (vec) {
      // VW consecutive x values per thread; each octant row piece leaves as one 16-byte store.
      for (int e = tid; e < H * H / VW; e += nth) {
        int ix0, iy;
        fold_item<H, VW>(e, &ix0, &iy);
        const C ty = ftx[iy];
        T oa[8][VW], ob[8][VW];
#pragma unroll
        for (int l = 0; l < VW; ++l) {
          const int ix = ix0 + l;
          const C tx = ftx[ix];
          T va[8], vb[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) { va[k] = static_cast<T>(0); vb[k] = static_cast<T>(0); }
#pragma unroll
          for (int c = 0; c < nch; ++c) {
            const int o = Cent<CT>::off(c);
            C w = mk<C>(static_cast<T>(1), static_cast<T>(0));
            if (o & 1) w = tx;
            if (o & 2) w = cmul(w, ty);
            if (o & 4) w = cmul(w, ftz);
            const C y = cmulc(buf[c * PL + iy * S + fold_pos<H, PV>(ix)], w);
            va[o] = y.x;
            vb[o] = y.y;
          }
          wht8(va);
          wht8(vb);
#pragma unroll
          for (int k = 0; k < 8; ++k) { oa[k][l] = div_const<T, V>(va[k]); ob[k][l] = div_const<T, V>(vb[k]); }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix0 + (k & 1) * H;
          if (USE_E) {
            T ea[VW], eb[VW];
            vload_nc<T>(ea, Ea + idx);
            vload_nc<T>(eb, (has_b ? Eb : Ea) + idx);
#pragma unroll
            for (int l = 0; l < VW; ++l) { oa[k][l] *= ea[l]; ob[k][l] *= eb[l]; }
          }
          vstore_stream<T>(dsta + idx, oa[k]);
          if (has_b) vstore_stream<T>(dstb + idx, ob[k]);
        }
      }
    } else {
      for (int e = tid; e < H * H; e += nth) {
        const int ix = e % H, iy = e / H;
        T va[8], vb[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) { va[k] = static_cast<T>(0); vb[k] = static_cast<T>(0); }
        const C tx = ftx[ix], ty = ftx[iy];
#pragma unroll
        for (int c = 0; c < nch; ++c) {
          const int o = Cent<CT>::off(c);
          C w = mk<C>(static_cast<T>(1), static_cast<T>(0));
          if (o & 1) w = tx;
          if (o & 2) w = cmul(w, ty);
          if (o & 4) w = cmul(w, ftz);
          const C y = cmulc(buf[c * PL + iy * S + fold_pos<H, PV>(ix)], w);  // x * conj(w)
          va[o] = y.x;
          vb[o] = y.y;
        }
        wht8(va);
        wht8(vb);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix + (k & 1) * H;
          T a = div_const<T, V>(va[k]), bq = div_const<T, V>(vb[k]);
          if (USE_E) { a *= Ea[idx]; if (has_b) bq *= Eb[idx]; }
          dsta[idx] = a;
          if (has_b) dstb[idx] = bq;
        }
      }
    }
  }
}

// y lines of the nch padded planes at buf: each thread owns the column (c, x),
// transforms it and stores it straight to the workspace plane dst0 (channel stride
// H^3, consecutive threads write consecutive x).
template <typename C, int H, int nch>
__device__ __forceinline__ void y_lines_to_workspace(const C* buf, C* __restrict__ dst0, int tid, int nth) {
  constexpr int S = H + 1;
  constexpr int PL = H * S;
  constexpr int HV = H * H * H;
  for (int l = tid; l < nch * H; l += nth) {
    const int c = l / H, x = l % H;
    const C* p = buf + c * PL + x;
    C v[H];
#pragma unroll
    for (int i = 0; i < H; ++i) v[i] = p[i * S];
    reg_fft<C, false, H>(v);
    C* d = dst0 + static_cast<size_t>(c) * HV + x;
#pragma unroll
    for (int i = 0; i < H; ++i) d[i * H] = v[i];
  }
}

// y lines of the nch planes at src0 (channel stride H^3) straight into registers (coalesced
// across x), inverse FFT, into the padded planes at buf.
template <typename C, int H, int nch>
__device__ __forceinline__ void inverse_y_lines(const C* __restrict__ src0, C* buf, int tid, int nth) {
  constexpr int S = H + 1, PL = H * S, HV = H * H * H;
  for (int l = tid; l < nch * H; l += nth) {
    const int c = l / H, x = l % H;
    const C* q = src0 + static_cast<size_t>(c) * HV + x;
    C v[H];
#pragma unroll
    for (int i = 0; i < H; ++i) v[i] = q[i * H];
    reg_fft<C, true, H>(v);
    C* p = buf + c * PL + x;
#pragma unroll
    for (int i = 0; i < H; ++i) p[i * S] = v[i];
  }
}
// After the last read of those planes: drop their lines from L2 without a write-back.
template <typename C, int H, int nch>
__device__ __forceinline__ void discard_planes(const C* src0, int tid, int nth) {
  if constexpr ((H * H * sizeof(C)) % 128 == 0) {
    constexpr int HV = H * H * H, LPP = static_cast<int>(H * H * sizeof(C) / 128);
    for (int i = tid; i < nch * LPP; i += nth)
      discard_l2_line(reinterpret_cast<const char*>(src0 + static_cast<size_t>(i / LPP) * HV) + (i % LPP) * 128);
  }
}

// Values per thread of the centred fold and unfold's vector path (the fold_pos order of
// their rows); 1 where that path does not apply.
template <typename T, int H, int CT> constexpr int row_vec() {
  constexpr int v = 16 / static_cast<int>(sizeof(T));
  return CT != 0 && H % v == 0 ? v : 1;
}

// Threads of the line-per-thread plane kernels: one per line, in warps, at least two warps;
// two warps more where that saves the fold a round (H = 24: 144 items on 160 threads instead
// of 96 or 128).  Measured, Ia-3d 96^3 FP32 contour steps of 256 fields, us for three: 637 /
// 680 / 620 / 693 with 96 / 128 / 160 / 192 threads; Im-3m 64^3 FP32 round trips of 256
// fields: 40.7 / 43.9 with 64 / 128; Pmmm 64^3 FP64, 256 fields: 217 / 229 with 64 / 128.  FP64,
// forward + backward with / without the two warps: Im-3m 64^3 x64 27.7 / 31.9, 64^3 x256 69.2 /
// 69.8, 48^3 x64 19.2 / 20.3, 96^3 x32 (384 blocks) 42.1 / 46.5, but 96^3 x135 (816 per lane)
// 126.3 / 122.8 and three contour steps there 599 / 551: at H = 24 only up to four blocks per SM.
// F centring (two channels), FP32: Fm-3m 96^3 x32 (384 blocks) 29.1 / 30.0, x135 (1632) 55.0 / 53.1, x256
// (1536 per lane) 83.7 / 79.7, so the same there; 128^3 x57 58.9 / 61.4; FP64 48^3 x256 31.0 / 33.0, 64^3
// x64 20.7 / 22.2.
template <typename T> inline int plane_line_threads(int H, int nch, bool folded, int ntasks) {
  constexpr int v = 16 / static_cast<int>(sizeof(T));
  const int base = std::max(64, ((nch * H + 31) / 32) * 32);
  const int items = H * H / (H % v == 0 ? v : 1);
  const auto rounds = [&](int t) { return (items + t - 1) / t; };
  const bool fits = H != 24 || (sizeof(T) == 4 && nch == 4) || ntasks <= 4 * kSMs;
  return folded && fits && rounds(base + 64) < rounds(base) && rounds(base + 64) <= 2 ? base + 64 : base;
}

// Registers of the forward plane kernel: with its sixteen loads in flight it takes 138 (FP32,
// H = 32) without factors and 168 with them, three blocks of 128 threads on an SM; the factors are
// a template parameter so that a plain transform does not carry them (as a run-time choice: 162
// for both; FP64, H = 16, 166 instead of 114; forward us of Im-3m 128^3 FP32 x64 36.4 / 35.2,
// 96^3 FP64 x135 66 / 60).  FP32 at H = 24 is capped at 112, one more block (forward us of Im-3m
// 96^3 x135: 30.0 / 32.5 without, Ia-3d 96^3 x256: 50.1 / 54.4).  Not elsewhere: H = 8 then spills
// (Im-3m 32^3 x256 8.3 / 7.3 without), H = 12 and 16 are even, and 128 at H = 32 is slower (Im-3m
// 128^3 x128, three contour steps 674 / 659).
template <typename T, int H> constexpr int fold_registers() { return sizeof(T) == 4 && H == 24 ? 112 : 255; }

// Forward plane kernel, cubic H: fold (or plain load) of two fields + x FFT + y FFT
// -> W[slot][c][z][y][x].
template <typename T, int H, int CT, bool UE>
__global__ void __maxnreg__((fold_registers<T, H>())) k_plane_fwd_h(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                              const T* __restrict__ f0, const T* __restrict__ E, typename Cx<T>::type* __restrict__ W,
                              int nfields) {
  pdl_enter();
  using C = typename Cx<T>::type;
  constexpr int nch = Cent<CT>::n, PV = row_vec<T, H, CT>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int iz = blockIdx.x, slot = blockIdx.y;
  const int fa = 2 * slot;
  const bool has_b = fa + 1 < nfields;
  constexpr bool USE_E = UE;
  const int tid = threadIdx.x, nth = blockDim.x;
  const size_t mvol = static_cast<size_t>(g->M[0]) * g->M[1] * g->M[2];
  const T* srca = f0 + static_cast<size_t>(fa) * mvol;
  const T* Ea = USE_E ? E + static_cast<size_t>(fa) * mvol : nullptr;
  fold_plane<T, H, CT, PV>(g, tables, srca, srca + mvol, Ea, USE_E ? Ea + mvol : nullptr, has_b, USE_E, iz, buf, tid, nth);
  __syncthreads();
  group_rows<C, false, H, PV, 1>(buf, nch * H, tid, nth);   // x lines
  __syncthreads();
  constexpr int HV = H * H * H;
  y_lines_to_workspace<C, H, nch>(buf, W + static_cast<size_t>(slot) * nch * HV + iz * H * H, tid, nth);
}

// Backward plane kernel, cubic H: inverse x/y FFT of W[slot][c][iz] + unfold of the two
// fields (real part -> field a, imaginary part -> field b).
template <typename T, int H, int CT>
__global__ void k_plane_bwd_h(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                              const typename Cx<T>::type* __restrict__ W, const T* __restrict__ E, T* __restrict__ f0,
                              int nfields) {
  pdl_enter();
  using C = typename Cx<T>::type;
  constexpr int nch = Cent<CT>::n, PV = row_vec<T, H, CT>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int iz = blockIdx.x, slot = blockIdx.y;
  const int fa = 2 * slot;
  const bool has_b = fa + 1 < nfields;
  const bool USE_E = E != nullptr;  // warp-uniform
  const int tid = threadIdx.x, nth = blockDim.x;
  constexpr int HV = H * H * H;
  const C* src0 = W + static_cast<size_t>(slot) * nch * HV + iz * H * H;
  inverse_y_lines<C, H, nch>(src0, buf, tid, nth);
  __syncthreads();
  discard_planes<C, H, nch>(src0, tid, nth);
  group_rows<C, true, H, 1, PV>(buf, nch * H, tid, nth);
  __syncthreads();
  const size_t mvol = static_cast<size_t>(g->M[0]) * g->M[1] * g->M[2];
  T* dsta = f0 + static_cast<size_t>(fa) * mvol;
  const T* Ea = USE_E ? E + static_cast<size_t>(fa) * mvol : nullptr;
  unfold_plane<T, H, CT, true, PV>(g, tables, buf, dsta, dsta + mvol, Ea, USE_E ? Ea + mvol : nullptr, has_b, USE_E, iz, tid, nth);
}

// ---------------------------------------------------------------- split lines
// A line of H = A x B points is transformed by two register passes through shared
// memory, in place: pass 1 takes the B butterflies of A points {j + B r}, multiplies
// output k1 by e^{-2 pi i j k1 / H} and writes it back to position j + B k1; pass 2 takes
// the A butterflies of B points {B k1 + j} and leaves frequency k1 + A k2 at position
// B k1 + k2 (line_pos).  A butterfly holds at most 8 values, so a plane is worked by
// four to eight times the threads of a line-per-thread kernel, at about half the
// registers: the plane and z kernels wait on memory, not on arithmetic, and need warps.
template <int H> constexpr int split_a() { return H == 12 || H == 16 ? 4 : H == 24 ? 6 : H >= 32 ? 8 : H; }
template <int H> constexpr int split_b() { return H / split_a<H>(); }
template <int H> __device__ __forceinline__ int line_pos(int k) {
  constexpr int A = split_a<H>(), B = split_b<H>();
  return B == 1 ? k : (k % A) * B + k / A;
}

// Twiddles e^{-2 pi i k / H} of the plan's tables into shared memory (lanes of a warp mostly
// share an index, but not for every H: constant memory would replay those reads).
template <typename C, int H>
__device__ __forceinline__ void load_line_twiddles(const DevGeom* __restrict__ g, const C* __restrict__ tables, C* tw) {
  if constexpr (split_b<H>() > 1)
    for (int i = threadIdx.x; i < H; i += blockDim.x) tw[i] = __ldg(tables + g->tw_off[0] + i);
}

// Butterfly j of pass 1 on the values v (already loaded): DFT_A and the twiddles.
template <typename C, bool INV, int H>
__device__ __forceinline__ void split_pass1(C (&v)[split_a<H>()], int j, const C* tw) {
  constexpr int A = split_a<H>();
  reg_fft<C, INV, A>(v);
  if constexpr (split_b<H>() > 1) {
#pragma unroll
    for (int k = 1; k < A; ++k) {
      const C t = tw[j * k];
      v[k] = INV ? cmulc(v[k], t) : cmul(v[k], t);
    }
  }
}

// In-place passes over `nlines` lines (line l at base(l), element stride ES) by all
// threads; consecutive threads take consecutive lines.
template <typename C, bool INV, int H, int ES, typename Base>
__device__ __forceinline__ void split_pass1_smem(C* buf, int nlines, Base base, const C* tw) {
  constexpr int A = split_a<H>(), B = split_b<H>();
  for (int i = threadIdx.x; i < nlines * B; i += blockDim.x) {
    const int j = i / nlines;
    C* p = buf + base(i - j * nlines) + j * ES;
    C v[A];
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = p[r * B * ES];
    split_pass1<C, INV, H>(v, j, tw);
#pragma unroll
    for (int r = 0; r < A; ++r) p[r * B * ES] = v[r];
  }
}
template <typename C, bool INV, int H, int ES, typename Base>
__device__ __forceinline__ void split_pass2_smem(C* buf, int nlines, Base base) {
  constexpr int A = split_a<H>(), B = split_b<H>();
  if constexpr (B > 1) {
    for (int i = threadIdx.x; i < nlines * A; i += blockDim.x) {
      const int k1 = i / nlines;
      C* p = buf + base(i - k1 * nlines) + k1 * B * ES;
      C v[B];
#pragma unroll
      for (int r = 0; r < B; ++r) v[r] = p[r * ES];
      reg_fft<C, INV, B>(v);
#pragma unroll
      for (int r = 0; r < B; ++r) p[r * ES] = v[r];
    }
  }
}

// Values per thread and octant row of the fold and the unfold: 8-byte accesses (two
// floats, one double).  Wider ones need twice the registers for the eight octants of two
// fields, which costs the resident warps more than the wider accesses give.
template <typename T> constexpr int fold_width() { return 8 / static_cast<int>(sizeof(T)); }
template <typename T, int VW> __device__ __forceinline__ void vw_load_stream(T (&o)[VW], const T* p) {
  if constexpr (VW == 2 && sizeof(T) == 4) {
    const float2 v = __ldcs(reinterpret_cast<const float2*>(p));
    o[0] = v.x; o[1] = v.y;
  } else {
#pragma unroll
    for (int l = 0; l < VW; ++l) o[l] = __ldcs(p + l);
  }
}
template <typename T, int VW> __device__ __forceinline__ void vw_load(T (&o)[VW], const T* p) {
  if constexpr (VW == 2 && sizeof(T) == 4) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    o[0] = v.x; o[1] = v.y;
  } else {
#pragma unroll
    for (int l = 0; l < VW; ++l) o[l] = __ldg(p + l);
  }
}
template <typename T, int VW> __device__ __forceinline__ void vw_store_stream(T* p, const T (&o)[VW]) {
  if constexpr (VW == 2 && sizeof(T) == 4) __stcs(reinterpret_cast<float2*>(p), make_float2(o[0], o[1]));
  else {
#pragma unroll
    for (int l = 0; l < VW; ++l) __stcs(p + l, o[l]);
  }
}

// Fold (or plain load) of the two fields of a slot at channel z-plane iz, VW consecutive
// x values per thread and step, into the nch planes at buf (row stride H + 1).
template <typename T, int H, int CT, int VW>
__device__ __forceinline__ void fold_rows(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                                          const T* __restrict__ srca, const T* __restrict__ srcb,
                                          const T* __restrict__ Ea, const T* __restrict__ Eb, bool has_b, bool USE_E,
                                          int iz, typename Cx<T>::type* buf) {
  using C = typename Cx<T>::type;
  constexpr int S = H + 1;
  const T zero = static_cast<T>(0);
  if constexpr (CT == 0) {
    const int zoff = iz * H * H;
    for (int e = threadIdx.x; e < H * H / VW; e += blockDim.x) {
      const int ix0 = (e % (H / VW)) * VW, iy = e / (H / VW);
      const int idx = zoff + iy * H + ix0;
      T va[VW], vb[VW], ea[VW];
      vw_load_stream<T, VW>(va, srca + idx);
#pragma unroll
      for (int l = 0; l < VW; ++l) vb[l] = zero;
      if (has_b) vw_load_stream<T, VW>(vb, srcb + idx);
      if (USE_E) {
        vw_load<T, VW>(ea, Ea + idx);
#pragma unroll
        for (int l = 0; l < VW; ++l) va[l] *= ea[l];
        if (has_b) {
          vw_load<T, VW>(ea, Eb + idx);
#pragma unroll
          for (int l = 0; l < VW; ++l) vb[l] *= ea[l];
        }
      }
#pragma unroll
      for (int l = 0; l < VW; ++l) buf[iy * S + ix0 + l] = mk<C>(va[l], vb[l]);
    }
  } else {
    constexpr int M = 2 * H;
    const C* ftx = tables + g->ftw_off[0];
    const C ftz = tables[g->ftw_off[2] + iz];
    for (int e = threadIdx.x; e < H * H / VW; e += blockDim.x) {
      const int ix0 = (e % (H / VW)) * VW, iy = e / (H / VW);
      T va[8][VW], vb[8][VW];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix0 + (k & 1) * H;
        vw_load_stream<T, VW>(va[k], srca + idx);
        vw_load_stream<T, VW>(vb[k], (has_b ? srcb : srca) + idx);
      }
      if (!has_b) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int l = 0; l < VW; ++l) vb[k][l] = zero;
      }
      if (USE_E) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix0 + (k & 1) * H;
          T ea[VW], eb[VW];
          vw_load<T, VW>(ea, Ea + idx);
          vw_load<T, VW>(eb, (has_b ? Eb : Ea) + idx);
#pragma unroll
          for (int l = 0; l < VW; ++l) { va[k][l] *= ea[l]; vb[k][l] *= eb[l]; }
        }
      }
      fold_emit<T, H, CT, VW>(va, vb, ix0, iy, ftx, ftz, buf);
    }
  }
}

// Unfold of the nch inverse-transformed planes at buf (x and y in line_pos order) into
// the two fields of the slot: conjugate fold twiddle, inverse WHT8 / 8, real part ->
// field a, imaginary part -> field b, times E when given.
template <typename T, int H, int CT, int VW>
__device__ __forceinline__ void unfold_rows(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                                            const typename Cx<T>::type* buf, T* __restrict__ dsta, T* __restrict__ dstb,
                                            const T* __restrict__ Ea, const T* __restrict__ Eb, bool has_b, bool USE_E,
                                            int iz) {
  using C = typename Cx<T>::type;
  constexpr int S = H + 1;
  constexpr int PL = H * S;
  constexpr int nch = Cent<CT>::n;
  if constexpr (CT == 0) {
    constexpr int V = H * H * H;
    for (int e = threadIdx.x; e < H * H / VW; e += blockDim.x) {
      const int ix0 = (e % (H / VW)) * VW, iy = e / (H / VW);
      const int idx = iz * H * H + iy * H + ix0;
      T va[VW], vb[VW], ea[VW];
#pragma unroll
      for (int l = 0; l < VW; ++l) {
        const C x = buf[line_pos<H>(iy) * S + line_pos<H>(ix0 + l)];
        va[l] = div_const<T, V>(x.x);
        vb[l] = div_const<T, V>(x.y);
      }
      if (USE_E) {
        vw_load<T, VW>(ea, Ea + idx);
#pragma unroll
        for (int l = 0; l < VW; ++l) va[l] *= ea[l];
        if (has_b) {
          vw_load<T, VW>(ea, Eb + idx);
#pragma unroll
          for (int l = 0; l < VW; ++l) vb[l] *= ea[l];
        }
      }
      vw_store_stream<T, VW>(dsta + idx, va);
      if (has_b) vw_store_stream<T, VW>(dstb + idx, vb);
    }
  } else {
    constexpr int M = 2 * H;
    constexpr int V = 8 * H * H * H;
    const C* ftx = tables + g->ftw_off[0];
    const C ftz = tables[g->ftw_off[2] + iz];
    for (int e = threadIdx.x; e < H * H / VW; e += blockDim.x) {
      const int ix0 = (e % (H / VW)) * VW, iy = e / (H / VW);
      const C ty = ftx[iy];
      const C* row = buf + line_pos<H>(iy) * S;
      T oa[8][VW], ob[8][VW];
#pragma unroll
      for (int l = 0; l < VW; ++l) {
        const C tx = ftx[ix0 + l];
        const int px = line_pos<H>(ix0 + l);
        C p8[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) p8[k] = mk<C>(static_cast<T>(0), static_cast<T>(0));
#pragma unroll
        for (int c = 0; c < nch; ++c) {
          const int o = Cent<CT>::off(c);
          C w = mk<C>(static_cast<T>(1), static_cast<T>(0));
          if (o & 1) w = tx;
          if (o & 2) w = cmul(w, ty);
          if (o & 4) w = cmul(w, ftz);
          p8[o] = o ? cmulc(row[c * PL + px], w) : row[c * PL + px];
        }
        wht8c(p8);
#pragma unroll
        for (int k = 0; k < 8; ++k) { oa[k][l] = div_const<T, V>(p8[k].x); ob[k][l] = div_const<T, V>(p8[k].y); }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int idx = ((iz + ((k >> 2) & 1) * H) * M + iy + ((k >> 1) & 1) * H) * M + ix0 + (k & 1) * H;
        if (USE_E) {
          T ea[VW], eb[VW];
          vw_load<T, VW>(ea, Ea + idx);
          vw_load<T, VW>(eb, (has_b ? Eb : Ea) + idx);
#pragma unroll
          for (int l = 0; l < VW; ++l) { oa[k][l] *= ea[l]; ob[k][l] *= eb[l]; }
        }
        vw_store_stream<T, VW>(dsta + idx, oa[k]);
        if (has_b) vw_store_stream<T, VW>(dstb + idx, ob[k]);
      }
    }
  }
}

// Threads of the split plane kernels: enough for the pass-1 butterflies in one to three
// rounds, on the plain path also for the plane's values in two, at most 512.
template <int H, int CT> constexpr int split_threads() {
  constexpr int n = CT == 0 && H * H / 2 > H * split_b<H>() ? H * H / 2 : Cent<CT>::n * H * split_b<H>();
  constexpr int t = n <= 512 ? n : (n + 1) / 2 <= 512 ? (n + 1) / 2 : (n + 2) / 3;
  return t < 64 ? 64 : ((t + 31) / 32) * 32;
}
template <typename T, int H, int CT> constexpr int split_blocks() {
  constexpr int by_threads = (sizeof(T) == 4 ? 1024 : 768) / split_threads<H, CT>();
  constexpr int by_smem = static_cast<int>((220 * 1024) / (Cent<CT>::n * H * (H + 1) * 2 * sizeof(T) + 1024));
  constexpr int b = by_threads < by_smem ? by_threads : by_smem;
  return b < 1 ? 1 : b > 8 ? 8 : b;
}

// Forward plane kernel, cubic H: fold (or plain load) of two fields + x FFT + y FFT
// -> W[slot][c][z][y][x].
template <typename T, int H, int CT>
__global__ void __launch_bounds__(split_threads<H, CT>(), split_blocks<T, H, CT>())
k_plane_fwd_s(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
              const T* __restrict__ f0, const T* __restrict__ E, typename Cx<T>::type* __restrict__ W, int nfields) {
  using C = typename Cx<T>::type;
  constexpr int nch = Cent<CT>::n, S = H + 1, PL = H * S, A = split_a<H>(), B = split_b<H>(), HV = H * H * H;
  constexpr int VW = H % fold_width<T>() == 0 ? fold_width<T>() : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  C* tw = buf + nch * PL;
  load_line_twiddles<C, H>(g, tables, tw);
  pdl_enter();
  const int iz = blockIdx.x, slot = blockIdx.y;
  const int fa = 2 * slot;
  const bool has_b = fa + 1 < nfields;
  const bool USE_E = E != nullptr;  // warp-uniform
  constexpr size_t mvol = static_cast<size_t>(CT ? 8 : 1) * HV;
  const T* srca = f0 + static_cast<size_t>(fa) * mvol;
  const T* Ea = USE_E ? E + static_cast<size_t>(fa) * mvol : nullptr;
  const T* Eb = USE_E ? Ea + mvol : nullptr;
  // Rows hold an even number of values, so the caller's base decides the alignment.
  if (VW == 1 || ((reinterpret_cast<uintptr_t>(f0) | reinterpret_cast<uintptr_t>(E)) & 7u) == 0)
    fold_rows<T, H, CT, VW>(g, tables, srca, srca + mvol, Ea, Eb, has_b, USE_E, iz, buf);
  else
    fold_rows<T, H, CT, 1>(g, tables, srca, srca + mvol, Ea, Eb, has_b, USE_E, iz, buf);
  __syncthreads();
  auto row = [](int l) { return l * S; };                          // line (c, y)
  auto col = [](int l) { return (l / H) * PL + (l % H); };         // line (c, x position)
  split_pass1_smem<C, false, H, 1>(buf, nch * H, row, tw);
  __syncthreads();
  if constexpr (B > 1) {
    split_pass2_smem<C, false, H, 1>(buf, nch * H, row);
    __syncthreads();
    split_pass1_smem<C, false, H, S>(buf, nch * H, col, tw);
    __syncthreads();
  }
  // Last pass straight to the workspace: butterfly k1 of column (c, x position) holds the
  // rows k1 + A r.
  C* dst0 = W + static_cast<size_t>(slot) * nch * HV + iz * H * H;
  constexpr int R = B > 1 ? B : A, NB = H / R;
  for (int i = threadIdx.x; i < nch * H * NB; i += blockDim.x) {
    const int k1 = i / (nch * H), l = i - k1 * (nch * H);
    const int c = l / H, px = l % H;
    const C* p = buf + c * PL + px + k1 * R * S;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[r * S];
    reg_fft<C, false, R>(v);
    const int kx = B > 1 ? px / B + A * (px % B) : px;
    C* d = dst0 + static_cast<size_t>(c) * HV + k1 * H + kx;
#pragma unroll
    for (int r = 0; r < R; ++r) d[r * NB * H] = v[r];
  }
}

// Backward plane kernel, cubic H: inverse x/y FFT of W[slot][c][iz] + unfold of the two
// fields (real part -> field a, imaginary part -> field b).
template <typename T, int H, int CT>
__global__ void __launch_bounds__(split_threads<H, CT>(), split_blocks<T, H, CT>())
k_plane_bwd_s(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
              const typename Cx<T>::type* __restrict__ W, const T* __restrict__ E, T* __restrict__ f0, int nfields) {
  using C = typename Cx<T>::type;
  constexpr int nch = Cent<CT>::n, S = H + 1, PL = H * S, A = split_a<H>(), B = split_b<H>(), HV = H * H * H;
  constexpr int VW = H % fold_width<T>() == 0 ? fold_width<T>() : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  C* tw = buf + nch * PL;
  load_line_twiddles<C, H>(g, tables, tw);
  pdl_enter();
  const int iz = blockIdx.x, slot = blockIdx.y;
  const int fa = 2 * slot;
  const bool has_b = fa + 1 < nfields;
  const bool USE_E = E != nullptr;  // warp-uniform
  __syncthreads();
  // First pass of the y lines straight from the workspace (coalesced across x).
  const C* src0 = W + static_cast<size_t>(slot) * nch * HV + iz * H * H;
  for (int i = threadIdx.x; i < nch * H * B; i += blockDim.x) {
    const int j = i / (nch * H), l = i - j * (nch * H);
    const int c = l / H, x = l % H;
    const C* q = src0 + static_cast<size_t>(c) * HV + j * H + x;
    C v[A];
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = q[r * B * H];
    split_pass1<C, true, H>(v, j, tw);
    C* p = buf + c * PL + j * S + x;
#pragma unroll
    for (int r = 0; r < A; ++r) p[r * B * S] = v[r];
  }
  __syncthreads();
  // Last read of these workspace planes: drop their lines from L2 without a write-back.
  if constexpr ((H * H * sizeof(C)) % 128 == 0) {
    constexpr int LPP = static_cast<int>(H * H * sizeof(C) / 128);
    for (int i = threadIdx.x; i < nch * LPP; i += blockDim.x)
      discard_l2_line(reinterpret_cast<const char*>(src0 + static_cast<size_t>(i / LPP) * HV) + (i % LPP) * 128);
  }
  auto row = [](int l) { return l * S; };
  auto col = [](int l) { return (l / H) * PL + (l % H); };
  if constexpr (B > 1) {
    split_pass2_smem<C, true, H, S>(buf, nch * H, col);
    __syncthreads();
  }
  split_pass1_smem<C, true, H, 1>(buf, nch * H, row, tw);
  __syncthreads();
  if constexpr (B > 1) {
    split_pass2_smem<C, true, H, 1>(buf, nch * H, row);
    __syncthreads();
  }
  constexpr size_t mvol = static_cast<size_t>(CT ? 8 : 1) * HV;
  T* dsta = f0 + static_cast<size_t>(fa) * mvol;
  const T* Ea = USE_E ? E + static_cast<size_t>(fa) * mvol : nullptr;
  const T* Eb = USE_E ? Ea + mvol : nullptr;
  if (VW == 1 || ((reinterpret_cast<uintptr_t>(f0) | reinterpret_cast<uintptr_t>(E)) & 7u) == 0)
    unfold_rows<T, H, CT, VW>(g, tables, buf, dsta, dsta + mvol, Ea, Eb, has_b, USE_E, iz);
  else
    unfold_rows<T, H, CT, 1>(g, tables, buf, dsta, dsta + mvol, Ea, Eb, has_b, USE_E, iz);
}

#include "tma_planes.cuh"

// ---------------------------------------------------------------- cluster kernels
// One thread-block cluster of KC CTAs holds the whole channel volume of one workspace
// slot (two fields) in distributed shared memory: CTA r owns the channel z-planes
// [ZPC r, ZPC r + ZPC), ZPC = H / KC, as padded nch x H x (H+1)
// planes.  The z transforms then read (forward) or write (backward) the peers' planes
// directly, so the channel workspace never makes the plane <-> z round trip through L2.
template <int H, int CT, int KC> struct ClusterShape {
  static constexpr int nch = Cent<CT>::n;
  static constexpr int zpc = H / KC;                    // channel z-planes per CTA
  static constexpr int threads = nch * zpc * H;         // one z line (c, y, x) per thread
  static constexpr int group = nch * H;                 // threads per plane in the x/y phase
};
// KC = 8 (portable) for H = 16, 24, 32; KC = 16 (non-portable, two CTAs per SM) for H = 32.
template <typename T, int H, int CT, int KC>
constexpr bool cluster_fits() {
  return H % KC == 0 && H >= 16 && H <= 32 && (KC == 8 || (KC == 16 && H == 32)) &&
         ClusterShape<H, CT, KC>::threads >= 32 && ClusterShape<H, CT, KC>::threads <= 1024 &&
         static_cast<long>(ClusterShape<H, CT, KC>::zpc) * Cent<CT>::n * H * (H + 1) * 2 * sizeof(T) <= 227 * 1024;
}
template <typename T, int H, int CT, int KC>
constexpr size_t cluster_smem() {
  return static_cast<size_t>(ClusterShape<H, CT, KC>::zpc) * Cent<CT>::n * H * (H + 1) * 2 * sizeof(T);
}

// Forward: fold + x/y FFT of the CTA's ZPC planes, cluster barrier, z FFT of the lines
// (c, y in the CTA's rows, x) gathered from the peers' planes, cluster barrier (every
// peer has finished reading), then the lines are transposed through the CTA's own
// shared memory and stored z-fastest: WT[slot][c][x][y][z].
template <typename T, int H, int CT, int KC>
__global__ void __launch_bounds__(ClusterShape<H, CT, KC>::threads)
k_fwd_cluster_h(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                const T* __restrict__ f0, const T* __restrict__ E, typename Cx<T>::type* __restrict__ WT, int nfields) {
  using C = typename Cx<T>::type;
  using CS = ClusterShape<H, CT, KC>;
  constexpr int S = H + 1, PL = H * S, NCH = CS::nch, ZPC = CS::zpc, HV = H * H * H;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int r = static_cast<int>(cluster.block_rank());
  const int slot = blockIdx.y;
  const int fa = 2 * slot;
  const bool has_b = fa + 1 < nfields;
  const bool USE_E = E != nullptr;
  const int tid = threadIdx.x;
  const size_t mvol = static_cast<size_t>(g->M[0]) * g->M[1] * g->M[2];
  {
    const int grp = tid / CS::group, gtid = tid % CS::group;
    C* pbuf = buf + grp * NCH * PL;
    const T* srca = f0 + static_cast<size_t>(fa) * mvol;
    const T* Ea = USE_E ? E + static_cast<size_t>(fa) * mvol : nullptr;
    fold_plane<T, H, CT>(g, tables, srca, srca + mvol, Ea, USE_E ? Ea + mvol : nullptr, has_b, USE_E, ZPC * r + grp,
                         pbuf, gtid, CS::group);
    __syncthreads();
    group_rows<C, false, H>(pbuf, NCH * H, gtid, CS::group);
    __syncthreads();
    group_cols<C, false, H>(pbuf, NCH * H, gtid, CS::group);
  }
  cluster.sync();
  const int c = tid / (ZPC * H), yy = (tid / H) % ZPC, x = tid % H;
  const int y = ZPC * r + yy;
  C v[H];
#pragma unroll
  for (int z = 0; z < H; ++z) {
    const C* rb = cluster.map_shared_rank(buf, z / ZPC);
    v[z] = rb[((z % ZPC) * NCH + c) * PL + y * S + x];
  }
  reg_fft<C, false, H>(v);
  cluster.sync();
  constexpr int RUN = ZPC * H, PCX = RUN + 1;  // staging [c][x][yy][z], padded per (c, x)
#pragma unroll
  for (int z = 0; z < H; ++z) buf[(c * H + x) * PCX + yy * H + z] = v[z];
  __syncthreads();
  C* dst = WT + static_cast<size_t>(slot) * NCH * HV;
  for (int e = tid; e < NCH * H * RUN; e += CS::threads) {
    const int cx = e / RUN, rr = e % RUN;
    dst[static_cast<size_t>(cx / H) * HV + ((cx % H) * H + ZPC * r) * H + rr] = buf[cx * PCX + rr];
  }
}

// Backward: cluster barrier (every peer is running), orbit expansion + inverse z FFT of
// the CTA's lines (c, y, x) from the combined representatives G0P[slot / 2][o][slot & 1]
// and the packed expansion entries (orbit | phase << 21), written into the owning
// peers' planes; cluster barrier; inverse x/y FFT + unfold of the CTA's own planes.
template <typename T, int H, int CT, int KC>
__global__ void __launch_bounds__(ClusterShape<H, CT, KC>::threads)
k_bwd_cluster_h(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                const uint32_t* __restrict__ ETP, const typename Cx<T>::type* __restrict__ G0P,
                const T* __restrict__ E, T* __restrict__ f0, int nfields) {
  using C = typename Cx<T>::type;
  using CS = ClusterShape<H, CT, KC>;
  constexpr int S = H + 1, PL = H * S, NCH = CS::nch, ZPC = CS::zpc, HV = H * H * H;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int r = static_cast<int>(cluster.block_rank());
  const int slot = blockIdx.y;
  const int tid = threadIdx.x;
  cluster.sync();
  {
    const int c = tid / (ZPC * H), yy = (tid / H) % ZPC, x = tid % H;
    const int y = ZPC * r + yy;
    const uint32_t* et = ETP + static_cast<size_t>(c) * HV + y * H + x;
    const C* rp = G0P + static_cast<size_t>(slot >> 1) * g->n_orbits * 2 + (slot & 1);
    const C* ph = tables + g->ph_off;
    C v[H];
#pragma unroll
    for (int z = 0; z < H; ++z) {
      const uint32_t t = __ldg(et + z * H * H);
      v[z] = cmulc(__ldg(rp + 2 * static_cast<size_t>(t & 0x1FFFFFu)), ph[t >> 21]);
    }
    reg_fft<C, true, H>(v);
#pragma unroll
    for (int z = 0; z < H; ++z) {
      C* rb = cluster.map_shared_rank(buf, z / ZPC);
      rb[((z % ZPC) * NCH + c) * PL + y * S + x] = v[z];
    }
  }
  cluster.sync();
  const int grp = tid / CS::group, gtid = tid % CS::group;
  C* pbuf = buf + grp * NCH * PL;
  group_rows<C, true, H>(pbuf, NCH * H, gtid, CS::group);
  __syncthreads();
  group_cols<C, true, H>(pbuf, NCH * H, gtid, CS::group);
  __syncthreads();
  const int fa = 2 * slot;
  const bool has_b = fa + 1 < nfields;
  const bool USE_E = E != nullptr;
  const size_t mvol = static_cast<size_t>(g->M[0]) * g->M[1] * g->M[2];
  T* dsta = f0 + static_cast<size_t>(fa) * mvol;
  const T* Ea = USE_E ? E + static_cast<size_t>(fa) * mvol : nullptr;
  unfold_plane<T, H, CT>(g, tables, pbuf, dsta, dsta + mvol, Ea, USE_E ? Ea + mvol : nullptr, has_b, USE_E,
                         ZPC * r + grp, gtid, CS::group);
}

constexpr int kZB = kFastZB;
// Threads of the z kernels that take one (y, x) line each: kZB y values x H lines, in
// whole warps, at least 64.
template <int H> constexpr int z_threads() { return ((kZB * H + 31) / 32) * 32 < 64 ? 64 : ((kZB * H + 31) / 32) * 32; }

// Forward z FFT, cubic H: W[slot][c][z][y][x] (in) -> WT[slot][c][x][y][z] (z fastest,
// out, same storage: each CTA reads and writes exactly the same addresses).  Thread
// (yy, x) loads its z line straight into registers (coalesced across x); the
// transposed store goes through shared memory.  Launched with z_threads<H>() threads;
// when kZB divides H every CTA holds kZB y values and the store loop's bounds and
// divisors are compile-time constants.
template <typename T, int H>
__global__ void k_fft_z_fwd_h(const DevGeom* __restrict__ g, const typename Cx<T>::type* W,
                              typename Cx<T>::type* WT) {
  pdl_enter();
  using C = typename Cx<T>::type;
  constexpr int S = H + 1;
  constexpr int HV = H * H * H;
  constexpr int kThr = z_threads<H>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);  // [yy][x][z] padded
  const int y0 = blockIdx.x * kZB, c = blockIdx.y, slot = blockIdx.z;
  const int ny = H % kZB == 0 ? kZB : min(kZB, H - y0);
  const int tid = threadIdx.x;
  const size_t base = (static_cast<size_t>(slot) * g->n_ch + c) * HV;
  const int yy = tid / H, x = tid % H;
  if (yy < ny) {
    const C* src = W + base + (y0 + yy) * H + x;
    C v[H];
#pragma unroll
    for (int z = 0; z < H; ++z) v[z] = src[z * H * H];
    reg_fft<C, false, H>(v);
    C* row = buf + (yy * H + x) * S;
#pragma unroll
    for (int z = 0; z < H; ++z) row[z] = v[z];
  }
  __syncthreads();
  C* dst = WT + base;
  if constexpr (H % kZB == 0) {
    constexpr int run = kZB * H;  // contiguous (yy, z) run per x
#pragma unroll 4
    for (int e = tid; e < H * run; e += kThr) {
      const int xx = e / run, r = e % run;
      const int y2 = r / H, z = r % H;
      dst[(xx * H + y0) * H + r] = buf[(y2 * H + xx) * S + z];
    }
  } else {
    const int run = ny * H;
    for (int e = tid; e < H * run; e += kThr) {
      const int xx = e / run, r = e % run;
      const int y2 = r / H, z = r % H;
      dst[(xx * H + y0) * H + r] = buf[(y2 * H + xx) * S + z];
    }
  }
}

// Spectral-ASU gather from the z-fastest packed workspace, cubic M (= 2H centred,
// = H plain), D representative operations; separates the two fields of the slot on
// the fly.  The geometry is staged in shared memory once per CTA.
template <typename T, int M, int D, bool USE_K, bool PERM>
__global__ void k_recon_h(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                          const uint32_t* __restrict__ spec_h, const T* __restrict__ K,
                          const typename Cx<T>::type* __restrict__ WT, typename Cx<T>::type* __restrict__ F,
                          int nfields) {
  pdl_enter();
  using C = typename Cx<T>::type;
  __shared__ int sR[D][9];
  __shared__ int sPS[D][3];
  __shared__ int sTP[D][3];
  __shared__ int sCh[8];
  const int tid = threadIdx.x;
  if (tid < D * 9) sR[tid / 9][tid % 9] = g->rep_R[tid / 9][tid % 9];
  if (tid < D * 3) { sPS[tid / 3][tid % 3] = g->rep_ps[tid / 3][tid % 3]; sTP[tid / 3][tid % 3] = g->rep_tp[tid / 3][tid % 3]; }
  if (tid < 8) sCh[tid] = g->chan_of_parity[tid];
  __syncthreads();
  const int s = blockIdx.x * blockDim.x + tid;
  const int slot = blockIdx.y;
  if (s >= g->n_spec) return;
  const int fa = 2 * slot;
  const bool has_b = fa + 1 < nfields;
  const uint32_t hp = spec_h[s];
  const int h[3] = {static_cast<int>(hp & 1023u), static_cast<int>((hp >> 10) & 1023u), static_cast<int>((hp >> 20) & 1023u)};
  const bool cen = g->centered;
  constexpr int Hc2 = M / 2;
  const int Hc = cen ? Hc2 : M;
  const int ls = cen ? 1 : 0;  // channel coordinate = q >> ls
  const size_t hvol = static_cast<size_t>(Hc) * Hc * Hc;
  const C* Wb = WT + static_cast<size_t>(slot) * g->n_ch * hvol;
  const C* ph = tables + g->ph_off;
  const int P = g->P, pmask = g->pmask;
  const T half = static_cast<T>(0.5);
  C acca = mk<C>(static_cast<T>(0), static_cast<T>(0));
  C accb = acca;
#pragma unroll
  for (int r = 0; r < D; ++r) {
    int q[3], qn[3];
#pragma unroll
    for (int dd = 0; dd < 3; ++dd) {
      int v;
      if (PERM) {
        const int ps = sPS[r][dd];
        v = h[ps & 3];
        if (ps & 4) v = -v;
      } else {
        v = sR[r][dd] * h[0] + sR[r][3 + dd] * h[1] + sR[r][6 + dd] * h[2];
      }
      q[dd] = mod_m<M>(v);
      qn[dd] = mod_m<M>(M - q[dd]);
    }
    int c = 0;
    if (cen) {
      c = sCh[(q[0] & 1) + 2 * (q[1] & 1) + 4 * (q[2] & 1)];
      if (c < 0) continue;
    }
    const size_t base = static_cast<size_t>(c) * hvol;
    const size_t idx = base + (static_cast<size_t>(q[0] >> ls) * Hc + (q[1] >> ls)) * Hc + (q[2] >> ls);
    const size_t idn = base + (static_cast<size_t>(qn[0] >> ls) * Hc + (qn[1] >> ls)) * Hc + (qn[2] >> ls);
    const C X = Wb[idx], Xn = Wb[idn];
    const C Ga = mk<C>(half * (X.x + Xn.x), half * (X.y - Xn.y));   // (X + conj Xn) / 2
    const C Gb = mk<C>(half * (X.y + Xn.y), half * (Xn.x - X.x));   // (X - conj Xn) / 2i
    int j = h[0] * sTP[r][0] + h[1] * sTP[r][1] + h[2] * sTP[r][2];
    j = pmask >= 0 ? (j & pmask) : ((j % P) + P) % P;
    const C w = ph[j];
    acca = cadd(acca, cmul(Ga, w));
    accb = cadd(accb, cmul(Gb, w));
  }
  if (USE_K) { const T k = K[s]; acca = cscale(acca, k); accb = cscale(accb, k); }
  F[static_cast<size_t>(fa) * g->n_spec + s] = acca;
  if (has_b) F[static_cast<size_t>(fa + 1) * g->n_spec + s] = accb;
}

// Spectral-ASU gather when the 8 representative operations are the diagonal sign
// matrices diag(+-1, +-1, +-1) (any translations): the 8 taps read G0 at the sign
// images s.h of h, which all lie in one parity channel, and the Hermitian partner
// X(-q) of tap s is tap ~s.  Eight workspace loads per point and slot.
constexpr int kDiagSlots = 2;
template <typename T, int M, bool USE_K>
__global__ void k_recon_diag8(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                              const uint32_t* __restrict__ spec_h, const T* __restrict__ K,
                              const typename Cx<T>::type* __restrict__ WT, typename Cx<T>::type* __restrict__ F,
                              int nfields) {
  pdl_enter();
  using C = typename Cx<T>::type;
  __shared__ int sTP[8][3];  // indexed by sign pattern
  __shared__ int sCh[8];
  const int tid = threadIdx.x;
  if (tid < 24) sTP[tid / 3][tid % 3] = g->rep_tp[g->sign_op[tid / 3]][tid % 3];
  if (tid < 8) sCh[tid] = g->chan_of_parity[tid];
  __syncthreads();
  const int s = blockIdx.x * blockDim.x + tid;
  if (s >= g->n_spec) return;
  const int ns = g->n_spec;
  const uint32_t hp = spec_h[s];
  const int h0 = static_cast<int>(hp & 1023u), h1 = static_cast<int>((hp >> 10) & 1023u), h2 = static_cast<int>((hp >> 20) & 1023u);
  const bool cen = g->centered;
  const int Hc = cen ? M / 2 : M;
  const int ls = cen ? 1 : 0;
  const int hvol = Hc * Hc * Hc;
  // per-axis (+h, -h) positions mod M, in channel coordinates
  const int p0 = mod_m<M>(h0), p1 = mod_m<M>(h1), p2 = mod_m<M>(h2);
  const int m0 = mod_m<M>(M - p0), m1 = mod_m<M>(M - p1), m2 = mod_m<M>(M - p2);
  int c = 0;
  if (cen) c = sCh[(p0 & 1) + 2 * (p1 & 1) + 4 * (p2 & 1)];
  // This thread serves kDiagSlots consecutive slots (fields 2 slot, 2 slot + 1): the
  // indices and phases are shared, the gathers of all its slots are in flight together.
  const int slot0 = blockIdx.y * kDiagSlots;
  if (c < 0) {  // extinct parity class: every tap reads zero
    const C z = mk<C>(static_cast<T>(0), static_cast<T>(0));
    for (int f = 2 * slot0; f < min(nfields, 2 * (slot0 + kDiagSlots)); ++f) F[static_cast<size_t>(f) * ns + s] = z;
    return;
  }
  const int X0[2] = {(p0 >> ls) * Hc * Hc, (m0 >> ls) * Hc * Hc};
  const int X1[2] = {(p1 >> ls) * Hc, (m1 >> ls) * Hc};
  const int X2[2] = {p2 >> ls, m2 >> ls};
  C X[kDiagSlots][8];
#pragma unroll
  for (int k = 0; k < kDiagSlots; ++k) {
    const int slot = min(slot0 + k, (nfields - 1) / 2);  // clamped: beyond the batch the result is dropped
    const C* Wb = WT + (static_cast<size_t>(slot) * g->n_ch + c) * hvol;
#pragma unroll
    for (int sg = 0; sg < 8; ++sg) X[k][sg] = Wb[X0[sg & 1] + X1[(sg >> 1) & 1] + X2[(sg >> 2) & 1]];
  }
  const C* ph = tables + g->ph_off;
  const int P = g->P, pmask = g->pmask;
  C w[8];
#pragma unroll
  for (int sg = 0; sg < 8; ++sg) {
    int j = h0 * sTP[sg][0] + h1 * sTP[sg][1] + h2 * sTP[sg][2];
    j = pmask >= 0 ? (j & pmask) : ((j % P) + P) % P;
    w[sg] = ph[j];
  }
  // Taps sg and 7 - sg are Hermitian partners: with u = w[sg], v = w[7 - sg] and
  // 2 G = (a, b), G u + conj(G) v = (a Pw.x + b Qw.x, a Pw.y + b Qw.y) for
  // Pw = (u + v) / 2, Qw = ((v.y - u.y) / 2, (u.x - v.x) / 2), shared by every slot
  // and both fields.
  const T half = static_cast<T>(0.5);
  C Pw[4], Qw[4];
#pragma unroll
  for (int sg = 0; sg < 4; ++sg) {
    const C u = w[sg], v = w[7 - sg];
    Pw[sg] = mk<C>(half * (u.x + v.x), half * (u.y + v.y));
    Qw[sg] = mk<C>(half * (v.y - u.y), half * (u.x - v.x));
  }
  const T kk = USE_K ? K[s] : static_cast<T>(1);
#pragma unroll
  for (int k = 0; k < kDiagSlots; ++k) {
    const int fa = 2 * (slot0 + k);
    if (fa >= nfields) break;
    C acca = mk<C>(static_cast<T>(0), static_cast<T>(0));
    C accb = acca;
#pragma unroll
    for (int sg = 0; sg < 4; ++sg) {
      const C Xs = X[k][sg], Xn = X[k][7 - sg];
      const T a = Xs.x + Xn.x, b = Xs.y - Xn.y;    // 2 G_a
      const T a2 = Xs.y + Xn.y, b2 = Xn.x - Xs.x;  // 2 G_b
      acca.x = fma(a, Pw[sg].x, fma(b, Qw[sg].x, acca.x));
      acca.y = fma(a, Pw[sg].y, fma(b, Qw[sg].y, acca.y));
      accb.x = fma(a2, Pw[sg].x, fma(b2, Qw[sg].x, accb.x));
      accb.y = fma(a2, Pw[sg].y, fma(b2, Qw[sg].y, accb.y));
    }
    if (USE_K) { acca = cscale(acca, kk); accb = cscale(accb, kk); }
    F[static_cast<size_t>(fa) * ns + s] = acca;
    if (fa + 1 < nfields) F[static_cast<size_t>(fa + 1) * ns + s] = accb;
  }
}

// Weights of the Hermitian tap pairs (sg, 7 - sg) of the fused gather's points, once per plan:
// with u = w[sg], v = w[7 - sg] the phases e^{-2 pi i h.t / N} of the two sign images,
// Pw = (u + v) / 2 and Qw = ((v.y - u.y) / 2, (u.x - v.x) / 2).
template <typename T>
__global__ void __launch_bounds__(256) k_zr_weights(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                                                    const uint2* __restrict__ pts, int npts, typename Cx<T>::type* __restrict__ pq) {
  using C = typename Cx<T>::type;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npts) return;
  const uint32_t hp = pts[i].y;
  const int h[3] = {static_cast<int>(hp & 1023u), static_cast<int>((hp >> 10) & 1023u), static_cast<int>((hp >> 20) & 1023u)};
  const int P = g->P;
  C w[8];
  for (int sg = 0; sg < 8; ++sg) {
    const int* tp = g->rep_tp[g->sign_op[sg]];
    const int j = (h[0] * tp[0] + h[1] * tp[1] + h[2] * tp[2]) % P;
    w[sg] = tables[g->ph_off + (j < 0 ? j + P : j)];
  }
  const T half = static_cast<T>(0.5);
  for (int sg = 0; sg < 4; ++sg) {
    const C u = w[sg], v = w[7 - sg];
    pq[static_cast<size_t>(2 * sg) * npts + i] = mk<C>(half * (u.x + v.x), half * (u.y + v.y));
    pq[static_cast<size_t>(2 * sg + 1) * npts + i] = mk<C>(half * (v.y - u.y), half * (u.x - v.x));
  }
}

// Forward z FFT fused with the spectral-ASU gather, for diagonal-sign representative
// operations (the taps of a spectral point h read G0 at the sign images of h, which lie
// in one channel c on the rows y = p1 >> ls and its mirror y' = m1 >> ls).  A CTA
// takes one unit (channel c and a mirrored pair of channel rows y_a, y_b; y_b < 0 when
// the unit has one row) and SL workspace slots:
//   1. the z lines W[slot][c][z][y_row][x] (coalesced across x) are transformed and kept
//      in shared memory [slot][row][x][z];
//   2. the unit's spectral points (a list built at plan time) are gathered from shared
//      memory as in k_recon_diag8 and written to F.
// The transposed workspace of the separate z kernel is never written or read back.
// Unit entry: x = c | y_a << 8 | (y_b + 1) << 16, y = first point, z = point count.
// Points: pts[i] = (spectral index, packed h); weights pq[2 sg][i] = Pw, pq[2 sg + 1][i] = Qw
// of the four Hermitian tap pairs (sg, 7 - sg): looking the eight phases up per point instead costs
// eight divergent table reads for values that every slot and both fields share.
// SPLIT: lines of two passes (see split_pass1) instead of one line per thread, for H = 48, where
// a line per thread leaves 8 to 11 warps on an SM, and for small launches.
template <int H> constexpr bool zr_split() { return H > 32; }
template <int H, int SL, bool SPLIT> constexpr int zr_threads() {
  constexpr int n = SL * 2 * H * (SPLIT ? split_b<H>() : 1);
  return n <= 64 ? 64 : SPLIT && n > 256 ? 256 : ((n + 31) / 32) * 32;
}
template <typename T, int H, int SL, bool SPLIT>
__global__ void __launch_bounds__(zr_threads<H, SL, SPLIT>())
k_fft_z_recon_diag8(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                    const T* __restrict__ K, const uint4* __restrict__ units, const uint2* __restrict__ pts,
                    const typename Cx<T>::type* __restrict__ pq, int npts,
                    const typename Cx<T>::type* __restrict__ W, typename Cx<T>::type* __restrict__ F, int nfields) {
  using C = typename Cx<T>::type;
  constexpr int S = H + 1, HV = H * H * H, NTH = zr_threads<H, SL, SPLIT>(), NL = SL * 2 * H;
  constexpr int RS = H * S;  // one row of (x, z) lines
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);  // [slot][row][x][z] padded
  const int tid = threadIdx.x;
  const uint4 un = units[blockIdx.x];
  const int c = static_cast<int>(un.x & 0xFFu), ya = static_cast<int>((un.x >> 8) & 0xFFu);
  const int yb = static_cast<int>((un.x >> 16) & 0xFFu) - 1;
  const int slot0 = blockIdx.y * SL;
  const int nslots = (nfields + 1) / 2;
  const int nch = g->n_ch;
  C* tw = buf + SL * 2 * RS;
  if constexpr (SPLIT) load_line_twiddles<C, H>(g, tables, tw);
  // The first round of points and weights does not depend on the previous kernel either.
  auto load_point = [&](int i, uint2* pt, C (&Pw)[4], C (&Qw)[4]) {
    *pt = __ldg(pts + un.y + i);
#pragma unroll
    for (int sg = 0; sg < 4; ++sg) {
      const C* p = pq + static_cast<size_t>(2 * sg) * npts + un.y + i;
      Pw[sg] = __ldg(p);
      Qw[sg] = __ldg(p + npts);
    }
  };
  constexpr bool EARLY = SL == 1;
  uint2 pt0 = make_uint2(0u, 0u);
  C P0[4], Q0[4];
  if (EARLY && tid < static_cast<int>(un.z)) load_point(tid, &pt0, P0, Q0);
  pdl_enter();
  if constexpr (!SPLIT) {
    if (tid < NL) {
      const int k = tid / (2 * H), r = (tid / H) & 1, x = tid % H;
      const int slot = slot0 + k;
      const int y = r ? yb : ya;
      if (slot < nslots && y >= 0) {
        const C* src = W + (static_cast<size_t>(slot) * nch + c) * HV + y * H + x;
        C v[H];
#pragma unroll
        for (int z = 0; z < H; ++z) v[z] = src[static_cast<size_t>(z) * H * H];
        reg_fft<C, false, H>(v);
        C* row = buf + (k * 2 + r) * RS + x * S;
#pragma unroll
        for (int z = 0; z < H; ++z) row[z] = v[z];
      }
    }
  } else {
    constexpr int A = split_a<H>(), B = split_b<H>();
    if constexpr (B > 1) __syncthreads();
    for (int i = tid; i < NL * B; i += NTH) {
      const int l = i % NL, j = i / NL;
      const int k = l / (2 * H), r = (l / H) & 1, x = l % H;
      const int slot = slot0 + k, y = r ? yb : ya;
      if (slot < nslots && y >= 0) {
        const C* src = W + (static_cast<size_t>(slot) * nch + c) * HV + y * H + x + j * H * H;
        C v[A];
#pragma unroll
        for (int q = 0; q < A; ++q) v[q] = src[static_cast<size_t>(q) * B * H * H];
        split_pass1<C, false, H>(v, j, tw);
        C* row = buf + l * S + j;
#pragma unroll
        for (int q = 0; q < A; ++q) row[q * B] = v[q];
      }
    }
    if constexpr (B > 1) {
      // Pass 2 through registers, so the lines come out in natural order for the gather.
      constexpr int R2 = (NL * A + NTH - 1) / NTH;
      C v[R2][B];
      __syncthreads();
#pragma unroll
      for (int t = 0; t < R2; ++t) {
        const int i = tid + t * NTH, l = i % NL, k1 = i / NL;
        if (k1 < A) {
          const C* row = buf + l * S + k1 * B;
#pragma unroll
          for (int q = 0; q < B; ++q) v[t][q] = row[q];
          reg_fft<C, false, B>(v[t]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int t = 0; t < R2; ++t) {
        const int i = tid + t * NTH, l = i % NL, k1 = i / NL;
        if (k1 < A) {
          C* row = buf + l * S + k1;
#pragma unroll
          for (int q = 0; q < B; ++q) row[q * A] = v[t][q];
        }
      }
    }
  }
  __syncthreads();
  // Every workspace row (slot, c, z, y) of this unit is read by this CTA alone and never
  // again: drop its lines from L2 (rows that fill whole 128-byte lines only).
  if constexpr ((H * sizeof(C)) % 128 == 0) {
    constexpr int LPR = static_cast<int>(H * sizeof(C) / 128);
    for (int i = tid; i < SL * 2 * H * LPR; i += NTH) {
      const int li = i % LPR, z = (i / LPR) % H, r = (i / (LPR * H)) & 1, k = i / (LPR * H * 2);
      const int slot = slot0 + k, y = r ? yb : ya;
      if (slot < nslots && y >= 0)
        discard_l2_line(reinterpret_cast<const char*>(W + (static_cast<size_t>(slot) * nch + c) * HV +
                                                      static_cast<size_t>(z) * H * H + y * H) + li * 128);
    }
  }
  const bool cen = g->centered;
  const int M = cen ? 2 * H : H;
  const int ls = cen ? 1 : 0;
  const int ns = g->n_spec;
  const int nvalid = min(SL, nslots - slot0);
  for (int i = tid; i < static_cast<int>(un.z); i += NTH) {
    uint2 pt;
    C Pw[4], Qw[4];
    if (EARLY && i == tid) {
      pt = pt0;
#pragma unroll
      for (int sg = 0; sg < 4; ++sg) { Pw[sg] = P0[sg]; Qw[sg] = Q0[sg]; }
    } else {
      load_point(i, &pt, Pw, Qw);
    }
    const uint32_t sidx = pt.x, hp = pt.y;
    const int h0 = static_cast<int>(hp & 1023u), h1 = static_cast<int>((hp >> 10) & 1023u), h2 = static_cast<int>((hp >> 20) & 1023u);
    const int p0 = cen ? mod_m<2 * H>(h0) : mod_m<H>(h0);
    const int p1 = cen ? mod_m<2 * H>(h1) : mod_m<H>(h1);
    const int p2 = cen ? mod_m<2 * H>(h2) : mod_m<H>(h2);
    const int m0 = p0 ? M - p0 : 0, m1 = p1 ? M - p1 : 0, m2 = p2 ? M - p2 : 0;
    const int X0[2] = {(p0 >> ls) * S, (m0 >> ls) * S};
    const int X1[2] = {((p1 >> ls) != ya) * RS, ((m1 >> ls) != ya) * RS};
    const int X2[2] = {p2 >> ls, m2 >> ls};
    const T kk = K ? K[sidx] : static_cast<T>(1);
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      if (k >= nvalid) break;
      const C* b = buf + k * 2 * RS;
      C X[8];
#pragma unroll
      for (int sg = 0; sg < 8; ++sg) X[sg] = b[X0[sg & 1] + X1[(sg >> 1) & 1] + X2[(sg >> 2) & 1]];
      C acca = mk<C>(static_cast<T>(0), static_cast<T>(0)), accb = acca;
#pragma unroll
      for (int sg = 0; sg < 4; ++sg) {
        const C Xs = X[sg], Xn = X[7 - sg];
        const T a = Xs.x + Xn.x, bq = Xs.y - Xn.y;
        const T a2 = Xs.y + Xn.y, b2 = Xn.x - Xs.x;
        acca.x = fma(a, Pw[sg].x, fma(bq, Qw[sg].x, acca.x));
        acca.y = fma(a, Pw[sg].y, fma(bq, Qw[sg].y, acca.y));
        accb.x = fma(a2, Pw[sg].x, fma(b2, Qw[sg].x, accb.x));
        accb.y = fma(a2, Pw[sg].y, fma(b2, Qw[sg].y, accb.y));
      }
      if (K) { acca = cscale(acca, kk); accb = cscale(accb, kk); }
      const int fa = 2 * (slot0 + k);
      F[static_cast<size_t>(fa) * ns + sidx] = acca;
      if (fa + 1 < nfields) F[static_cast<size_t>(fa + 1) * ns + sidx] = accb;
    }
  }
}

// Walsh-Hadamard transform of D = 1, 2, 4 or 8 complex values.
template <typename C, int D> __device__ __forceinline__ void wht_d(C (&v)[D]) {
#pragma unroll
  for (int s = 1; s < D; s <<= 1)
#pragma unroll
    for (int i = 0; i < D; ++i)
      if (!(i & s)) { const C a = v[i], b = v[i + s]; v[i] = cadd(a, b); v[i + s] = csub(a, b); }
}

// ---------------------------------------------------------------- inverse gather by fibers
// The d aliases q + M m of a subgrid frequency q (its fiber) determine G0 at all d
// images R_b^T q of the representative operations at once:
//   e^{-2 pi i q.t_b / N} G0(R_b^T q) = (1/d) sum_m (-1)^{m . t_b} F(q + M m),
// a Walsh-Hadamard transform of the d values, because the translations t_b run through
// the parity classes once each.  One fiber therefore serves up to d orbits: its d spectrum
// values are loaded once instead of once per orbit, and the d x d phases become d + d.
// Taps (fiber-fastest, [m][fiber]): x = spectral index + 1 | conjugate << 31 (0: extinct),
// y = phase numerator j, F(q + M m) = e^{2 pi i j / P} F[x] (conjugated first where
// flagged).  Outputs ([b][fiber]): x = orbit + 1 (0: none), y = phase numerator.
//
// Each spectrum value is read once or twice (plain and conjugated taps make different fibers,
// which neighbour one another), so the gather reads F field by field as the caller stores
// it: a warp takes 32 fibers of one workspace slot, whose taps are near neighbours in the
// spectral order.  The slot inputs X = G_a + i G_b of the L slots of a
// group are exchanged through shared memory and leave as whole rows G0P[group][orbit][L]
// for the expansion.  Im-3m 128^3 FP32, 64 fields: 7.5 + 15.0 us (regroup of the spectra
// and one gather per orbit, 8 x the loads) before.
// NF: fields per slot, 2 or, for the general kernels, 1.
constexpr int kFibers = 32;
template <typename T, int D, int L, int NF>
__global__ void __launch_bounds__(kFibers * L)
k_inv_fiber(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
            const uint2* __restrict__ taps, const uint2* __restrict__ outs, int nf,
            const typename Cx<T>::type* __restrict__ F, typename Cx<T>::type* __restrict__ G0P, int nb) {
  using C = typename Cx<T>::type;
  constexpr int RS = L + 1;
  __shared__ C tile[D * kFibers * RS];
  const int lane = threadIdx.x % kFibers, j = threadIdx.x / kFibers;
  const int f0 = blockIdx.x * kFibers, f = f0 + lane;
  // Rows of two slots are small launches that wait on the previous kernel: their table loads
  // go before the wait.  Full rows would pay for the registers (Ia-3d 96^3 contour steps of 256
  // fields: 3339 us with it, 3235 without).
  constexpr bool EARLY = L == 2;
  uint2 t[D], o[D];
  if constexpr (!EARLY) pdl_enter();
#pragma unroll
  for (int m = 0; m < D; ++m) {
    t[m] = f < nf ? __ldg(taps + static_cast<size_t>(m) * nf + f) : make_uint2(0u, 0u);
    if (EARLY) o[m] = f < nf ? __ldg(outs + static_cast<size_t>(m) * nf + f) : make_uint2(0u, 0u);
  }
  if constexpr (EARLY) pdl_enter();
  const int gq = blockIdx.y;
  const int fa = NF * (gq * L + j);
  const C* ph = tables + g->ph_off;
  const int ns = g->n_spec;
  const C zero = mk<C>(static_cast<T>(0), static_cast<T>(0));
  C x[D];
  if (f < nf && fa < nb) {
    const C* Fa = F + static_cast<size_t>(fa) * ns;
    const bool has_b = NF == 2 && fa + 1 < nb;
    C va[D], vb[D];
#pragma unroll
    for (int m = 0; m < D; ++m) {
      const uint32_t sp = t[m].x & 0x7FFFFFFFu;
      va[m] = sp ? __ldg(Fa + sp - 1) : zero;
      vb[m] = sp && has_b ? __ldg(Fa + ns + sp - 1) : zero;
    }
#pragma unroll
    for (int m = 0; m < D; ++m) {
      const T sg = (t[m].x >> 31) ? static_cast<T>(-1) : static_cast<T>(1);
      const C v = mk<C>(va[m].x - sg * vb[m].y, sg * va[m].y + vb[m].x);
      x[m] = cmulc(v, ph[t[m].y]);
    }
    wht_d<C, D>(x);
  } else {
#pragma unroll
    for (int m = 0; m < D; ++m) x[m] = zero;
  }
  if (f < nf) {
    const T inv_d = static_cast<T>(1.0 / static_cast<double>(D));
#pragma unroll
    for (int b = 0; b < D; ++b) {
      if (!EARLY) o[b] = __ldg(outs + static_cast<size_t>(b) * nf + f);
      if (o[b].x) tile[(b * kFibers + lane) * RS + j] = cscale(cmulc(x[b], ph[o[b].y]), inv_d);
    }
  }
  __syncthreads();
  const int no = g->n_orbits;
  const int cnt = min(kFibers, nf - f0);
  C* dst = G0P + static_cast<size_t>(gq) * no * L;
#pragma unroll
  for (int e = threadIdx.x; e < D * kFibers * L; e += kFibers * L) {
    const int k = e % L, fb = (e / L) % kFibers, b = e / (L * kFibers);
    if (fb < cnt) {
      const uint32_t at = __ldg(outs + static_cast<size_t>(b) * nf + f0 + fb).x;
      if (at) dst[static_cast<size_t>(at - 1) * L + k] = tile[(b * kFibers + fb) * RS + k];
    }
  }
}

// ---------------------------------------------------------------- orbit expansion + inverse z FFT
// X(R^T q) = X(q_o) e^{2 pi i j / P} at every channel point from the packed entries (orbit
// in bits 0-20, phase numerator in bits 21-31) and the rows G0P[group][orbit][L], then the
// inverse z FFT -> W[slot][c][z][y][x].  A CTA takes one (y, c) and LS of the group's L
// slots.  The lanes of a row fetch it in 16-byte pieces; the values meet their z lines in
// shared memory, so the workspace stores run along x (storing straight from the fetching
// lanes splits every store over eight slots).  SPLIT: lines of two passes (see
// split_pass1), for FP64 and small launches, where one thread per line leaves too few
// warps.
template <typename C> constexpr int wide_slots() { return static_cast<int>(64 / sizeof(C)); }  // 8 FP32, 4 FP64
template <typename C, int H, int L> constexpr int expand_slots() {
  int ls = L;
  while (ls > 2 && ls * H * H * static_cast<int>(sizeof(C)) > 72 * 1024) ls /= 2;
  return ls;
}
template <int H> constexpr int expand_plane() { return ((H * H + 7) / 8) * 8 + 2; }
template <typename C, int H, int LS> constexpr int expand_threads() {
  constexpr int items = H * H * LS * static_cast<int>(sizeof(C)) / 16;
  constexpr int t = items / 4 > LS * H ? items / 4 : LS * H;
  return t <= 64 ? 64 : t >= 256 ? 256 : ((t + 31) / 32) * 32;
}
// Inverse z FFT of LS planes [slot][z][x] (expand_plane apart) in shared memory, stored for
// the first `live` slots to dst + slot * sstride + z * H * H + x.
template <typename C, int H, int LS, bool SPLIT>
__device__ __forceinline__ void inverse_z_planes(C* buf, const C* tw, C* __restrict__ dst, size_t sstride, int live) {
  constexpr int PS = expand_plane<H>();
  const int tid = threadIdx.x, nth = blockDim.x;
  if constexpr (!SPLIT) {
    for (int i = tid; i < LS * H; i += nth) {
      const int x = i % H, j = i / H;
      const C* p = buf + j * PS + x;
      C v[H];
#pragma unroll
      for (int z = 0; z < H; ++z) v[z] = p[z * H];
      reg_fft<C, true, H>(v);
      if (j < live) {
        C* d = dst + j * sstride + x;
#pragma unroll
        for (int z = 0; z < H; ++z) d[z * H * H] = v[z];
      }
    }
  } else {
    constexpr int A = split_a<H>(), B = split_b<H>(), R = B > 1 ? B : A, NB = H / R;
    if constexpr (B > 1) {
      for (int i = tid; i < LS * H * B; i += nth) {
        const int x = i % H, j = (i / H) % LS, jj = i / (H * LS);
        C* p = buf + j * PS + jj * H + x;
        C v[A];
#pragma unroll
        for (int r = 0; r < A; ++r) v[r] = p[r * B * H];
        split_pass1<C, true, H>(v, jj, tw);
#pragma unroll
        for (int r = 0; r < A; ++r) p[r * B * H] = v[r];
      }
      __syncthreads();
    }
    for (int i = tid; i < LS * H * NB; i += nth) {
      const int x = i % H, j = (i / H) % LS, k1 = i / (H * LS);
      if (j >= live) continue;
      const C* p = buf + j * PS + k1 * R * H + x;
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * H];
      reg_fft<C, true, R>(v);
      C* d = dst + j * sstride + static_cast<size_t>(k1) * H * H + x;
#pragma unroll
      for (int r = 0; r < R; ++r) d[static_cast<size_t>(r) * NB * H * H] = v[r];
    }
  }
}

template <typename T, int H, int L, int LS, bool SPLIT>
__global__ void __launch_bounds__(expand_threads<typename Cx<T>::type, H, LS>())
k_expand_ifft_z(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                const uint32_t* __restrict__ ETP, const typename Cx<T>::type* __restrict__ G0P,
                typename Cx<T>::type* __restrict__ W, int nfields) {
  using C = typename Cx<T>::type;
  constexpr int HV = H * H * H, PS = expand_plane<H>(), NTH = expand_threads<C, H, LS>();
  constexpr int SPV = 16 / static_cast<int>(sizeof(C)), NP = LS / SPV;  // slots per 16 bytes, pieces per row
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);  // [slot][z][x]
  C* tw = buf + LS * PS;
  const int y = blockIdx.x, c = blockIdx.y, gq = blockIdx.z / (L / LS), part = blockIdx.z % (L / LS);
  const int slot0 = gq * L + part * LS;
  if (2 * slot0 >= nfields) {
    pdl_enter();
    return;
  }
  const uint32_t* et = ETP + static_cast<size_t>(c) * HV + y * H;
  const C* rp = G0P + static_cast<size_t>(gq) * g->n_orbits * L + part * LS;
  const C* ph = tables + g->ph_off;
  // Entries and phases of a short loop are fetched before the previous kernel has finished.
  constexpr int ITEMS = H * H * NP, ROUNDS = (ITEMS + NTH - 1) / NTH, AHEAD = ROUNDS <= 6 ? ROUNDS : 0;
  if constexpr (SPLIT) load_line_twiddles<C, H>(g, tables, tw);
  uint32_t te[AHEAD > 0 ? AHEAD : 1];
  C we[AHEAD > 0 ? AHEAD : 1];
#pragma unroll
  for (int k = 0; k < AHEAD; ++k) {
    const int i = min(static_cast<int>(threadIdx.x) + k * NTH, ITEMS - 1);
    te[k] = __ldg(et + i / (NP * H) * H * H + (i / NP) % H);
    we[k] = __ldg(ph + (te[k] >> 21));
  }
  pdl_enter();
  auto put = [&](int i, uint32_t t, C w) {
    const int p = i % NP, x = (i / NP) % H, z = i / (NP * H);
    const C* src = rp + static_cast<size_t>(L) * (t & 0x1FFFFFu) + p * SPV;
    C* d = buf + (p * SPV) * PS + z * H + x;
    if constexpr (SPV == 2) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(src));
      d[0] = cmulc(mk<C>(u.x, u.y), w);
      d[PS] = cmulc(mk<C>(u.z, u.w), w);
    } else {
      d[0] = cmulc(__ldg(src), w);
    }
  };
  if constexpr (AHEAD > 0) {
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      const int i = threadIdx.x + k * NTH;
      if (ITEMS % NTH == 0 || i < ITEMS) put(i, te[k], we[k]);
    }
  } else {
#pragma unroll 4
    for (int i = threadIdx.x; i < ITEMS; i += NTH) {
      const uint32_t t = __ldg(et + i / (NP * H) * H * H + (i / NP) % H);
      put(i, t, ph[t >> 21]);
    }
  }
  __syncthreads();
  const int live = min(LS, (nfields + 1) / 2 - slot0);
  inverse_z_planes<C, H, LS, SPLIT>(buf, tw, W + (static_cast<size_t>(slot0) * g->n_ch + c) * HV + y * H,
                                    static_cast<size_t>(g->n_ch) * HV, live);
}

// The same for rows of two slots (small batches), one z line per thread straight from the
// gather to the workspace, no shared memory: half of a CTA takes each slot, YB rows y.
template <typename T, int H, int YB>
__global__ void k_expand2_ifft_z(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                                 const uint32_t* __restrict__ ETP, const typename Cx<T>::type* __restrict__ G0P,
                                 typename Cx<T>::type* __restrict__ W, int nfields) {
  pdl_enter();
  using C = typename Cx<T>::type;
  constexpr int HV = H * H * H;
  constexpr int kHalf = ((YB * H + 31) / 32) * 32;
  const int c = blockIdx.y, q = blockIdx.z;
  const int half = threadIdx.x / kHalf, r = threadIdx.x % kHalf;
  const int slot = 2 * q + half, y = blockIdx.x * YB + r / H, x = r % H;
  if (2 * slot >= nfields || r >= YB * H || y >= H) return;
  const uint32_t* et = ETP + static_cast<size_t>(c) * HV + y * H + x;
  const C* rp = G0P + static_cast<size_t>(q) * g->n_orbits * 2 + half;
  const C* ph = tables + g->ph_off;
  C v[H];
#pragma unroll
  for (int z = 0; z < H; ++z) {
    const uint32_t t = __ldg(et + z * H * H);
    v[z] = cmulc(__ldg(rp + 2 * static_cast<size_t>(t & 0x1FFFFFu)), ph[t >> 21]);
  }
  reg_fft<C, true, H>(v);
  C* dst = W + (static_cast<size_t>(slot) * g->n_ch + c) * HV + y * H + x;
#pragma unroll
  for (int z = 0; z < H; ++z) dst[z * H * H] = v[z];
}

// Q-matrix diffusion step (execute_m2_q! / execute_m7_scft!, src/q_fused_krfft.jl:553-667,
// 870-895): for every channel point (c, x, y, z) of a slot, q its subgrid position,
//   Y'(q) = sum_b Q_b(q) G0(R_b^T q mod M)
// with G0 gathered from the forward workspace WT (z-fastest; index -1 marks a parity
// class without a channel, where G0 = 0), then the inverse z FFT, stored
// W2[slot][c][z][y][x] for the inverse plane kernel.  Both fields of the slot
// (G0_a + i G0_b) go through the same complex-linear map.  A CTA takes one (y, c, slot), a
// thread one point at a time: the d gathers of a point are independent, but a thread that
// gathers a whole line makes H of them wait for one another.
template <typename T, int H>
__global__ void __launch_bounds__(expand_threads<typename Cx<T>::type, H, 2>())
k_qmul_ifft_z_h(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
                const typename Cx<T>::type* __restrict__ QT, const int32_t* __restrict__ GT,
                const typename Cx<T>::type* __restrict__ WT, typename Cx<T>::type* __restrict__ W2) {
  using C = typename Cx<T>::type;
  constexpr int HV = H * H * H;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);  // [z][x]
  C* tw = buf + expand_plane<H>();
  load_line_twiddles<C, H>(g, tables, tw);
  pdl_enter();
  const int y = blockIdx.x, c = blockIdx.y, slot = blockIdx.z;
  const int d = g->d;
  const size_t np = static_cast<size_t>(g->n_ch) * HV;
  const C* wt = WT + static_cast<size_t>(slot) * g->n_ch * HV;
  for (int i = threadIdx.x; i < H * H; i += blockDim.x) {
    const int x = i % H, z = i / H;
    const size_t pos = static_cast<size_t>(c) * HV + (z * H + y) * H + x;
    C acc = mk<C>(static_cast<T>(0), static_cast<T>(0));
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if (b < d) {
        const int32_t gi = __ldg(GT + b * np + pos);
        if (gi >= 0) acc = cadd(acc, cmul(__ldg(QT + b * np + pos), __ldg(wt + gi)));
      }
    }
    buf[z * H + x] = acc;
  }
  __syncthreads();
  inverse_z_planes<C, H, 1, true>(buf, tw, W2 + (static_cast<size_t>(slot) * g->n_ch + c) * HV + y * H, 0, 1);
}

// Separable Q-multiply of the M2Q step for Pmmm-like plans (_q_multiply_separable!,
// src/q_fused_krfft.jl:606-667; detection _is_pmmm_like, :431-454): d = 8, L = (2, 2, 2),
// the representatives diag(s) with translations 0 or -1, and an orthogonal cell.  Then
// B = WHT8 diag(tw^alpha) and the first row of Q = B^-1 diag(K) B gives
//   Y'(q) = (1/8) sum_m K(q + M alpha_m) [WHT8 (tw^alpha_a(q) Y(s_a q mod M))]_m,
// tw_d(q) = e^{2 pi i q_d / N_d}, K(h) = prod_d exp(-ds (2 pi h_c,d / a_d)^2).  The eight
// images s_a q form a closed set on which the spectrum only changes by the twiddle, so
//   Y'(s_a q) = conj(tw^alpha_a(q)) / 8 [WHT8 (K WHT8 (tw^alpha Y))]_a
// maps the eight values in place: one pair of transforms per eight points instead of
// one gather of eight per point.  The images lie on the channel rows y and -y and the
// lines x and -x, so a CTA that holds those lines does the whole middle of the step: forward
// z FFT, the map, inverse z FFT, in place on the workspace W[slot][z][y][x] (plain path, one
// channel, H = M).  Blocks: rows y <= H / 2, PP pairs of lines (x, -x), slots; fewer pairs
// per block while the launch would not fill the SMs.  The lines stay in line_pos order
// between the transforms, whose passes run in reverse on the way back.  Pm-3m 48^3 FP64,
// 4 fields: 5 us z FFT + 20 us gather (and its second workspace) before.
// QS holds the 1-D twiddles (3 x H complex) and the 1-D kernel factors (3 x 2H, real parts).
constexpr int kSepThreads = 128;
template <typename T, int H>
__global__ void __launch_bounds__(kSepThreads)
k_qsep_z(const DevGeom* __restrict__ g, const typename Cx<T>::type* __restrict__ tables,
         const typename Cx<T>::type* __restrict__ QS, typename Cx<T>::type* __restrict__ W, int PP) {
  using C = typename Cx<T>::type;
  constexpr int HV = H * H * H, S = H + 1, A = split_a<H>(), B = split_b<H>(), HP = H / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);  // [row][side][pair][z]
  C* tw = buf + 4 * PP * S;
  load_line_twiddles<C, H>(g, tables, tw);
  pdl_enter();
  const int y = blockIdx.x, ym = y ? H - y : 0, rows = ym == y ? 1 : 2;
  const int p0 = blockIdx.y * PP, np = min(PP, HP - p0), slot = blockIdx.z;
  const int lines = rows * 2 * np;
  C* Ws = W + static_cast<size_t>(slot) * HV;
  // line l: row r, side (x or -x), pair p; -1 where the line is its own mirror image
  auto line = [&](int l, int* off) {
    const int r = l / (2 * np), m = l - r * 2 * np, side = m / np, k = m - side * np, p = p0 + k;
    if (side && (p == 0 || 2 * p == H)) return -1;
    *off = (r ? ym : y) * H + (side ? H - p : p);
    return ((r * 2 + side) * PP + k) * S;
  };
  if constexpr (B > 1) __syncthreads();
  for (int i = threadIdx.x; i < lines * B; i += kSepThreads) {
    const int j = i / lines;
    int off = 0;
    const int at = line(i - j * lines, &off);
    if (at < 0) continue;
    const C* src = Ws + off + j * H * H;
    C v[A];
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = src[r * B * H * H];
    split_pass1<C, false, H>(v, j, tw);
    C* row = buf + at + j;
#pragma unroll
    for (int r = 0; r < A; ++r) row[r * B] = v[r];
  }
  __syncthreads();
  if constexpr (B > 1) {
    for (int i = threadIdx.x; i < lines * A; i += kSepThreads) {
      const int k1 = i / lines;
      int off = 0;
      const int at = line(i - k1 * lines, &off);
      if (at < 0) continue;
      C* row = buf + at + k1 * B;
      C v[B];
#pragma unroll
      for (int r = 0; r < B; ++r) v[r] = row[r];
      reg_fft<C, false, B>(v);
#pragma unroll
      for (int r = 0; r < B; ++r) row[r] = v[r];
    }
    __syncthreads();
  }
  {
    const C* tq = QS;          // tq[d * H + q]
    const C* kf = QS + 3 * H;  // kf[d * 2H + h].x
    int img[8];                // representative a negates the axes of bit set img[a]
#pragma unroll
    for (int a = 0; a < 8; ++a)
      img[a] = (g->rep_R[a][0] < 0 ? 1 : 0) | (g->rep_R[a][4] < 0 ? 2 : 0) | (g->rep_R[a][8] < 0 ? 4 : 0);
    const C twy = tq[H + y];
    const T ky0 = kf[2 * H + y].x, ky1 = kf[2 * H + y + H].x;
    for (int i = threadIdx.x; i < np * HP; i += kSepThreads) {
      const int k = i / HP, z = i - k * HP, p = p0 + k;
      const int zm = z ? H - z : 0;
      const bool sx = p == 0 || 2 * p == H, sy = rows == 1, sz = zm == z;
      const int xo[2] = {k * S, sx ? k * S : (PP + k) * S}, yo[2] = {0, sy ? 0 : 2 * PP * S};
      const int zo[2] = {line_pos<H>(z), line_pos<H>(zm)};
      const C twx = tq[p], twz = tq[2 * H + z];
      const C txy = cmul(twx, twy), txz = cmul(twx, twz), tyz = cmul(twy, twz), txyz = cmul(txy, twz);
      const C t8[8] = {mk<C>(static_cast<T>(1), static_cast<T>(0)), twx, twy, txy, twz, txz, tyz, txyz};
      const T kx0 = kf[p].x, kx1 = kf[p + H].x, kz0 = kf[4 * H + z].x, kz1 = kf[4 * H + z + H].x;
      const T e = static_cast<T>(0.125);
      const T k00 = e * kx0 * ky0, k10 = e * kx1 * ky0, k01 = e * kx0 * ky1, k11 = e * kx1 * ky1;
      const T km[8] = {k00 * kz0, k10 * kz0, k01 * kz0, k11 * kz0, k00 * kz1, k10 * kz1, k01 * kz1, k11 * kz1};
      C v[8];
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        v[a] = buf[xo[img[a] & 1] + yo[(img[a] >> 1) & 1] + zo[(img[a] >> 2) & 1]];
        if (a) v[a] = cmul(v[a], t8[a]);
      }
      wht8c(v);
#pragma unroll
      for (int a = 0; a < 8; ++a) v[a] = cscale(v[a], km[a]);
      wht8c(v);
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const int m = img[a];
        if (((m & 1) && sx) || ((m & 2) && sy) || ((m & 4) && sz)) continue;  // the same point again
        buf[xo[m & 1] + yo[(m >> 1) & 1] + zo[(m >> 2) & 1]] = a ? cmulc(v[a], t8[a]) : v[a];
      }
    }
  }
  __syncthreads();
  if constexpr (B > 1) {
    for (int i = threadIdx.x; i < lines * A; i += kSepThreads) {
      const int k1 = i / lines;
      int off = 0;
      const int at = line(i - k1 * lines, &off);
      if (at < 0) continue;
      C* row = buf + at + k1 * B;
      C v[B];
#pragma unroll
      for (int r = 0; r < B; ++r) v[r] = row[r];
      reg_fft<C, true, B>(v);
#pragma unroll
      for (int r = 0; r < B; ++r) row[r] = r ? cmulc(v[r], tw[r * k1]) : v[r];
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < lines * B; i += kSepThreads) {
    const int j = i / lines;
    int off = 0;
    const int at = line(i - j * lines, &off);
    if (at < 0) continue;
    const C* row = buf + at + j;
    C v[A];
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = row[r * B];
    reg_fft<C, true, A>(v);
    C* dst = Ws + off + j * H * H;
#pragma unroll
    for (int r = 0; r < A; ++r) dst[r * B * H * H] = v[r];
  }
}

constexpr int kMaxDynSmemFast = 227 * 1024;

// Persistent bulk-copy plane kernels (tma_planes.cuh).  They serve centred plans with
// H >= 16 whose per-group stage and buffer fit at least two groups into one CTA's
// shared memory.  CFFT_TMA selects them: "fwd" (the forward plane stage), "all" (both
// stages), unset or "0" (neither).  Measured on Im-3m 128^3 FP32 (B200): the forward
// one is 2-5% slower than the per-plane kernel and the backward one 30% slower -- with
// one 195 KB CTA per SM they run 8 and 12 warps per SM against the per-plane kernels'
// 20, and the FFT phases, not the loads, bound the stage -- so both are opt-in.
inline int tma_mode() {  // bit 0: forward, bit 1: backward
  static const int m = [] {
    const char* e = std::getenv("CFFT_TMA");
    if (!e) return 0;
    if (e[0] == '0') return 0;
    if (e[0] == 'a' || e[0] == '1') return 3;
    if (e[0] == 'b') return 2;
    return 1;
  }();
  return m;
}
inline bool tma_enabled() { return tma_mode() != 0; }
template <typename T, int H, int CT, bool USE_E>
constexpr bool fwd_tma_fits() {
  if constexpr (CT == 0 || H < 16 || H % (16 / static_cast<int>(sizeof(T))) != 0) return false;
  else return tma_groups<FwdTmaShape<T, H, CT, USE_E>>() >= 2;
}
template <typename T, int H, int CT>
constexpr bool bwd_tma_fits() {
  if constexpr (CT == 0 || H < 16 || H % (16 / static_cast<int>(sizeof(T))) != 0) return false;
  else return tma_groups<BwdTmaShape<T, H, CT>>() >= 2;
}
// Persistent grid of a bulk-copy plane kernel: every SM's resident CTAs, or fewer when
// the tasks run out.  The resident count is looked up once per kernel and device (the
// kernels of different H share a function type, so the cache is keyed by address) under
// a lock, since plans may be executed from several host threads.
template <typename K>
int tma_grid(K kernel, int threads, size_t smem, int ntasks, int ng) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> resident;
  int dev = 0;
  cudaGetDevice(&dev);
  int cap = 1;
  {
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
    auto it = resident.find(key);
    if (it == resident.end()) {
      int occ = 0, sms = 0;
      if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 1;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess) occ = 1;
      it = resident.emplace(key, std::max(1, occ) * std::max(1, sms)).first;
    }
    cap = it->second;
  }
  const int need = (ntasks + ng - 1) / ng;
  return std::max(1, std::min(need, cap));
}

// Workspace slots per CTA of the fused z FFT + gather: 4, or 2 with CFFT_ZR_SLOTS=2
// (measured on Im-3m 128^3 FP32: 4 slots slightly ahead).
inline int zr_slots() {
  static const int n = [] {
    const char* e = std::getenv("CFFT_ZR_SLOTS");
    return (e && e[0] == '2') ? 2 : 4;
  }();
  return n;
}


#define CFFT_FOR_H(H, ...)                                                        \
  switch (H) {                                                                    \
    case 4: { constexpr int HH = 4; __VA_ARGS__; } break;                         \
    case 6: { constexpr int HH = 6; __VA_ARGS__; } break;                         \
    case 8: { constexpr int HH = 8; __VA_ARGS__; } break;                         \
    case 12: { constexpr int HH = 12; __VA_ARGS__; } break;                       \
    case 16: { constexpr int HH = 16; __VA_ARGS__; } break;                       \
    case 24: { constexpr int HH = 24; __VA_ARGS__; } break;                       \
    case 32: { constexpr int HH = 32; __VA_ARGS__; } break;                       \
    default: { constexpr int HH = sizeof(T) == 4 ? 48 : 32; __VA_ARGS__; } break; \
  }

#define CFFT_FOR_M(M, ...)                                        \
  switch (M) {                                                     \
    case 4: { constexpr int MM = 4; __VA_ARGS__; } break;         \
    case 6: { constexpr int MM = 6; __VA_ARGS__; } break;         \
    case 8: { constexpr int MM = 8; __VA_ARGS__; } break;         \
    case 12: { constexpr int MM = 12; __VA_ARGS__; } break;       \
    case 16: { constexpr int MM = 16; __VA_ARGS__; } break;       \
    case 24: { constexpr int MM = 24; __VA_ARGS__; } break;       \
    case 32: { constexpr int MM = 32; __VA_ARGS__; } break;       \
    case 48: { constexpr int MM = 48; __VA_ARGS__; } break;       \
    case 64: { constexpr int MM = 64; __VA_ARGS__; } break;       \
    default: { constexpr int MM = 96; __VA_ARGS__; } break;       \
  }

#define CFFT_FOR_CT(CTV, ...)                                      \
  switch (CTV) {                                                   \
    case 1: { constexpr int CTT = 1; __VA_ARGS__; } break;         \
    case 2: { constexpr int CTT = 2; __VA_ARGS__; } break;         \
    case 3: { constexpr int CTT = 3; __VA_ARGS__; } break;         \
    case 4: { constexpr int CTT = 4; __VA_ARGS__; } break;         \
    default: { constexpr int CTT = 0; __VA_ARGS__; } break;        \
  }

// Cluster kernels: attributes, launch (cluster size at run time, through
// cudaLaunchKernelEx) and occupancy, for the instantiations that fit.
template <typename T, int H, int CT, int KC>
void cluster_attrs() {
  if constexpr (cluster_fits<T, H, CT, KC>()) {
    const int smem = static_cast<int>(cluster_smem<T, H, CT, KC>());
    cudaFuncSetAttribute(k_fwd_cluster_h<T, H, CT, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_bwd_cluster_h<T, H, CT, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (KC > 8) {
      cudaFuncSetAttribute(k_fwd_cluster_h<T, H, CT, KC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      cudaFuncSetAttribute(k_bwd_cluster_h<T, H, CT, KC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
  }
}

template <typename T, int H, int CT, int KC>
cudaLaunchConfig_t cluster_config(int nslots, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(KC, static_cast<unsigned>(nslots), 1);
  cfg.blockDim = dim3(ClusterShape<H, CT, KC>::threads, 1, 1);
  cfg.dynamicSmemBytes = cluster_smem<T, H, CT, KC>();
  cfg.stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = KC;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <typename T, int H, int CT, int KC>
bool cluster_launch(int stage, int nslots, cudaStream_t st, const DevGeom* g, const typename Cx<T>::type* tab,
                    const T* f0, const T* E, typename Cx<T>::type* W, const uint32_t* ETP,
                    const typename Cx<T>::type* G0P, T* f0_out, int nb, cudaError_t* ce) {
  if constexpr (cluster_fits<T, H, CT, KC>()) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cluster_config<T, H, CT, KC>(nslots, st, &attr);
    if (stage == 0) *ce = cudaLaunchKernelEx(&cfg, k_fwd_cluster_h<T, H, CT, KC>, g, tab, f0, E, W, nb);
    else *ce = cudaLaunchKernelEx(&cfg, k_bwd_cluster_h<T, H, CT, KC>, g, tab, ETP, G0P, E, f0_out, nb);
    return true;
  }
  return false;
}

template <typename T, int H, int CT, int KC>
cudaError_t cluster_occupancy(int* max_clusters) {
  if constexpr (cluster_fits<T, H, CT, KC>()) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cluster_config<T, H, CT, KC>(1, nullptr, &attr);
    int nf = 0, nbk = 0;
    cudaError_t e = cudaOccupancyMaxActiveClusters(&nf, k_fwd_cluster_h<T, H, CT, KC>, &cfg);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&nbk, k_bwd_cluster_h<T, H, CT, KC>, &cfg);
    if (e == cudaSuccess) *max_clusters = std::min(nf, nbk);
    return e;
  }
  *max_clusters = 0;
  return cudaSuccess;
}

// Per-device set-up of this unit: its own copy of the constant-memory twiddles
// e^{-2 pi i j / N} (FP64 values rounded) and the shared-memory limits of its kernels.
template <typename T, int GROUP>
Status fast_unit_init(std::string* err) {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  Status s = fast_cuda(cudaGetDevice(&dev), "cudaGetDevice", err);
  if (s != Status::kOk) return s;
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return Status::kOk;
  std::vector<float2> tf(kTwTotal);
  std::vector<double2> td(kTwTotal);
  const int sizes[8] = {4, 6, 8, 12, 16, 24, 32, 48};
  const int offs[8] = {kTwOff4, kTwOff6, kTwOff8, kTwOff12, kTwOff16, kTwOff24, kTwOff32, kTwOff48};
  for (int k = 0; k < 8; ++k)
    for (int j = 0; j < sizes[k]; ++j) {
      const double c = std::cos(2.0 * M_PI * j / sizes[k]), sn = -std::sin(2.0 * M_PI * j / sizes[k]);
      td[offs[k] + j] = make_double2(c, sn);
      tf[offs[k] + j] = make_float2(static_cast<float>(c), static_cast<float>(sn));
    }
  if ((s = fast_cuda(cudaMemcpyToSymbol(c_tw_f, tf.data(), sizeof(float2) * kTwTotal), "upload twiddles", err)) != Status::kOk) return s;
  if ((s = fast_cuda(cudaMemcpyToSymbol(c_tw_d, td.data(), sizeof(double2) * kTwTotal), "upload twiddles", err)) != Status::kOk) return s;
  for (int H : {4, 6, 8, 12, 16, 24, 32, 48}) {
    if (!fast_size_ok(H, sizeof(T))) continue;
    CFFT_FOR_H(H, {
      if constexpr (GROUP == 0) {
        for (int ct = 0; ct < 5; ++ct) {
          CFFT_FOR_CT(ct, {
            cudaFuncSetAttribute(k_plane_fwd_h<T, HH, CTT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
            cudaFuncSetAttribute(k_plane_fwd_h<T, HH, CTT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
            cudaFuncSetAttribute(k_plane_bwd_h<T, HH, CTT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
            if constexpr (HH <= 32) {
              cudaFuncSetAttribute(k_plane_fwd_s<T, HH, CTT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
              cudaFuncSetAttribute(k_plane_bwd_s<T, HH, CTT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
            }
            // The bulk-copy kernels also hold a little static shared memory, so their
            // dynamic limit is their exact need; a refusal is reported.
            cudaError_t te = cudaSuccess;
            if constexpr (fwd_tma_fits<T, HH, CTT, false>()) {
              using SH = FwdTmaShape<T, HH, CTT, false>;
              constexpr int NG = tma_groups<SH>();
              te = cudaFuncSetAttribute(k_plane_fwd_tma<T, HH, CTT, NG, false>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(NG * SH::group));
            }
            if constexpr (fwd_tma_fits<T, HH, CTT, true>()) {
              using SH = FwdTmaShape<T, HH, CTT, true>;
              constexpr int NG = tma_groups<SH>();
              if (te == cudaSuccess)
                te = cudaFuncSetAttribute(k_plane_fwd_tma<T, HH, CTT, NG, true>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(NG * SH::group));
            }
            if constexpr (bwd_tma_fits<T, HH, CTT>()) {
              using SH = BwdTmaShape<T, HH, CTT>;
              constexpr int NG = tma_groups<SH>();
              if (te == cudaSuccess)
                te = cudaFuncSetAttribute(k_plane_bwd_tma<T, HH, CTT, NG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(NG * SH::group));
            }
            if (te != cudaSuccess) return fast_cuda(te, "bulk-copy plane kernel shared-memory attribute", err);
            cluster_attrs<T, HH, CTT, 8>();
            cluster_attrs<T, HH, CTT, 16>();
          });
        }
      } else {
        cudaFuncSetAttribute(k_fft_z_fwd_h<T, HH>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
        // The fused kernel also holds 96 bytes of static shared memory; its dynamic
        // share above 48 KB (FP64, 4 slots) needs the attribute, so failures are reported.
        {
          constexpr int kZr = kMaxDynSmemFast - 1024;
          constexpr bool SP = zr_split<HH>();
          cudaError_t ze = cudaFuncSetAttribute(k_fft_z_recon_diag8<T, HH, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kZr);
          if (ze == cudaSuccess) ze = cudaFuncSetAttribute(k_fft_z_recon_diag8<T, HH, 2, SP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kZr);
          if (ze == cudaSuccess) ze = cudaFuncSetAttribute(k_fft_z_recon_diag8<T, HH, 4, SP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kZr);
          if (ze != cudaSuccess) return fast_cuda(ze, "fused z FFT + gather shared-memory attribute", err);
        }
        using CC = typename Cx<T>::type;
        cudaFuncSetAttribute(k_expand_ifft_z<T, HH, wide_slots<CC>(), expand_slots<CC, HH, wide_slots<CC>()>(), sizeof(T) == 8>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
        if constexpr (HH <= 32)
          cudaFuncSetAttribute(k_expand_ifft_z<T, HH, 2, 2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
        cudaFuncSetAttribute(k_qsep_z<T, HH>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmemFast);
      }
    });
  }
  if ((s = fast_cuda(cudaGetLastError(), "set shared-memory attributes", err)) != Status::kOk) return s;
  if (dev >= 0 && dev < 64) done[dev] = true;
  return Status::kOk;
}

// Occupancy of the fused cluster kernels with KC CTAs per cluster: resident clusters
// (the smaller of the forward and backward kernels), 0 when they do not fit.
template <typename T>
Status fast_unit_cluster_probe(int H, int ct, int kc, int* max_clusters, std::string* err) {
  *max_clusters = 0;
  Status s = fast_unit_init<T, 0>(err);
  if (s != Status::kOk) return s;
  cudaError_t e = cudaSuccess;
  CFFT_FOR_H(H, {
    CFFT_FOR_CT(ct, {
      if (kc == 16) e = cluster_occupancy<T, HH, CTT, 16>(max_clusters);
      else e = cluster_occupancy<T, HH, CTT, 8>(max_clusters);
    });
  });
  if (e != cudaSuccess) {  // e.g. a cluster size this device does not allow: not used
    cudaGetLastError();
    *max_clusters = 0;
  }
  return Status::kOk;
}

template <typename T>
void fast_unit_tma_planes(int H, int ct, int tma, bool* fwd, bool* fwd_e, bool* bwd) {
  *fwd = *fwd_e = *bwd = false;
  const int mode = tma >= 0 ? tma : tma_mode();
  if (!mode || !fast_size_ok(H, sizeof(T))) return;
  CFFT_FOR_H(H, {
    CFFT_FOR_CT(ct, {
      *fwd = (mode & 1) && fwd_tma_fits<T, HH, CTT, false>();
      *fwd_e = (mode & 1) && fwd_tma_fits<T, HH, CTT, true>();
      *bwd = (mode & 2) && bwd_tma_fits<T, HH, CTT>();
    });
  });
}

// One fast-path stage for `a.nb` fields (two per workspace slot).
template <typename T, int GROUP>
Status fast_unit_launch(const FastArgs& a, std::string* err) {
  using C = typename Cx<T>::type;
  const DevGeom* g = static_cast<const DevGeom*>(a.geom);
  const C* tab = static_cast<const C*>(a.tables);
  C* W = static_cast<C*>(a.W);
  C* G0R = static_cast<C*>(a.G0R);
  const T* f0 = static_cast<const T*>(a.f0);
  const T* E = static_cast<const T*>(a.E);
  C* F = static_cast<C*>(a.F);
  const C* Fin = static_cast<const C*>(a.Fin);
  T* f0_out = static_cast<T*>(a.f0_out);
  cudaStream_t st = static_cast<cudaStream_t>(a.stream);
  const int H = a.H, nb = a.nb, nch = a.n_ch;
  const int nslots = (nb + 1) / 2;
  const size_t cs = sizeof(C);
  if constexpr (GROUP == 0) {
    if (a.cluster) {
      bool launched = false;
      cudaError_t ce = cudaSuccess;
      CFFT_FOR_H(H, {
        CFFT_FOR_CT(a.cent_type, {
          if (a.cluster_ctas == 16) {
            launched = cluster_launch<T, HH, CTT, 16>(a.stage, nslots, st, g, tab, f0, E, W,
                                                      static_cast<const uint32_t*>(a.expand), G0R, f0_out, nb, &ce);
          } else {
            launched = cluster_launch<T, HH, CTT, 8>(a.stage, nslots, st, g, tab, f0, E, W,
                                                     static_cast<const uint32_t*>(a.expand), G0R, f0_out, nb, &ce);
          }
        });
      });
      if (!launched) {
        *err = "no fused cluster kernel for this channel grid";
        return Status::kUnsupported;
      }
      if (ce != cudaSuccess) return fast_cuda(ce, "fused cluster launch", err);
      return fast_cuda(cudaGetLastError(), "fused cluster launch", err);
    }
    const int ntasks = nslots * H;
    const int thr_plane = plane_line_threads<T>(H, nch, a.cent_type != 0, ntasks);
    const size_t smem_plane = static_cast<size_t>(nch) * H * (H + 1) * cs;
    // Split lines while the launch has at most one CTA per SM, or as few lines as half the
    // SMs' blocks of 128: then the length of a thread's chain counts, beyond that the extra
    // shared-memory passes do.  GPU us of three contour steps, split / a line per thread: Ia-3d
    // 96^3 FP32 x2 / x32, 69 / 84 and 140 / 140; Pm-3m 48^3 FP32 x16 (192 CTAs, 4608 lines) 47 / 55, Fm-3m
    // 96^3 FP64 x16 (192, 9216) 89 / 100, but 96^3 FP32 x32 (384, 18432) 109 / 106, Im-3m 96^3 FP64 x16 (192,
    // 18432) 114 / 105.  FP64 folds at H = 32, whose lines take 150 registers, gain from it for twice the
    // lines of one CTA per SM, in all lanes: Im-3m 128^3 x16 (256, 32768) 188 / 226, Fm-3m 128^3 x32 (512,
    // 32768) 271 / 359, Im-3m 128^3 x32 (two lanes) forward + backward 90 / 76.  Above H = 32 the plane
    // takes a whole SM either way and the split loses at every size.
    const int lines = ntasks * nch * H;
    const bool split = H <= 32 && (ntasks <= kSMs || lines <= kSMs * 64 ||
                                   (sizeof(T) == 8 && H == 32 && a.cent_type != 0 && a.lanes * lines <= kSMs * 256));
    auto al16 = [](const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const int tmode = a.tma >= 0 ? a.tma : tma_mode();
    const bool tma = al16(f0) && al16(E) && al16(f0_out) && al16(W) && (tmode & (a.stage == 0 ? 1 : 2));
    if (a.stage == 0) {
      CFFT_FOR_H(H, {
        CFFT_FOR_CT(a.cent_type, {
          bool done = false;
          if (tma && E == nullptr) {
            if constexpr (fwd_tma_fits<T, HH, CTT, false>()) {
              using SH = FwdTmaShape<T, HH, CTT, false>;
              constexpr int NG = tma_groups<SH>();
              auto* k = k_plane_fwd_tma<T, HH, CTT, NG, false>;
              const int grid = tma_grid(k, NG * SH::threads, NG * SH::group, ntasks, NG);
              launch_k(k, dim3(grid), NG * SH::threads, NG * SH::group, st, g, tab, f0, E, W, nb, ntasks,
                       static_cast<uint64_t>(a.timeout_ns), a.status);
              done = true;
            }
          } else if (tma) {
            if constexpr (fwd_tma_fits<T, HH, CTT, true>()) {
              using SH = FwdTmaShape<T, HH, CTT, true>;
              constexpr int NG = tma_groups<SH>();
              auto* k = k_plane_fwd_tma<T, HH, CTT, NG, true>;
              const int grid = tma_grid(k, NG * SH::threads, NG * SH::group, ntasks, NG);
              launch_k(k, dim3(grid), NG * SH::threads, NG * SH::group, st, g, tab, f0, E, W, nb, ntasks,
                       static_cast<uint64_t>(a.timeout_ns), a.status);
              done = true;
            }
          }
          if constexpr (HH <= 32)
            if (!done && split) {
              launch_k(k_plane_fwd_s<T, HH, CTT>, dim3(H, nslots), split_threads<HH, CTT>(), smem_plane + HH * cs, st, g, tab, f0, E, W, nb);
              done = true;
            }
          if (!done)
            launch_k(E ? k_plane_fwd_h<T, HH, CTT, true> : k_plane_fwd_h<T, HH, CTT, false>, dim3(H, nslots), thr_plane, smem_plane, st, g, tab, f0, E, W, nb);
        });
      });
    } else {
      CFFT_FOR_H(H, {
        CFFT_FOR_CT(a.cent_type, {
          bool done = false;
          if (tma) {
            if constexpr (bwd_tma_fits<T, HH, CTT>()) {
              using SH = BwdTmaShape<T, HH, CTT>;
              constexpr int NG = tma_groups<SH>();
              auto* k = k_plane_bwd_tma<T, HH, CTT, NG>;
              const int grid = tma_grid(k, NG * SH::threads, NG * SH::group, ntasks, NG);
              launch_k(k, dim3(grid), NG * SH::threads, NG * SH::group, st, g, tab, static_cast<const C*>(W), E, f0_out,
                       nb, ntasks, static_cast<uint64_t>(a.timeout_ns), a.status);
              done = true;
            }
          }
          if constexpr (HH <= 32)
            if (!done && split) {
              launch_k(k_plane_bwd_s<T, HH, CTT>, dim3(H, nslots), split_threads<HH, CTT>(), smem_plane + HH * cs, st, g, tab, W, E, f0_out, nb);
              done = true;
            }
          if (!done)
            launch_k(k_plane_bwd_h<T, HH, CTT>, dim3(H, nslots), thr_plane, smem_plane, st, g, tab, W, E, f0_out, nb);
        });
      });
    }
  } else {
    const size_t smem_z = static_cast<size_t>(kZB) * H * (H + 1) * cs;
    const dim3 gz((H + kZB - 1) / kZB, nch, nslots);
    switch (a.stage) {
      case 1:
        CFFT_FOR_H(H, { launch_k(k_fft_z_fwd_h<T, HH>, gz, z_threads<HH>(), smem_z, st, g, W, W); });
        break;
      case 2: {
        const dim3 gr((a.n_spec + 255) / 256, nslots);
        const int M = a.centered ? 2 * H : H;
        const T* K = static_cast<const T*>(a.K);
        const uint32_t* sh = static_cast<const uint32_t*>(a.spec_h);
        const bool use_K = a.use_K, perm = a.rep_perm;
        if (a.rep_diag8) {
          const dim3 gd((a.n_spec + 255) / 256, (nslots + kDiagSlots - 1) / kDiagSlots);
          CFFT_FOR_M(M, {
            if (use_K) launch_k(k_recon_diag8<T, MM, true>, gd, 256, 0, st, g, tab, sh, K, W, F, nb);
            else launch_k(k_recon_diag8<T, MM, false>, gd, 256, 0, st, g, tab, sh, nullptr, W, F, nb);
          });
          break;
        }
#define CFFT_RECON_D(DD)                                                                                  \
  CFFT_FOR_M(M, {                                                                                         \
    if (use_K) {                                                                                          \
      if (perm) launch_k(k_recon_h<T, MM, DD, true, true>, gr, 256, 0, st, g, tab, sh, K, W, F, nb);            \
      else launch_k(k_recon_h<T, MM, DD, true, false>, gr, 256, 0, st, g, tab, sh, K, W, F, nb);                \
    } else {                                                                                              \
      if (perm) launch_k(k_recon_h<T, MM, DD, false, true>, gr, 256, 0, st, g, tab, sh, nullptr, W, F, nb);     \
      else launch_k(k_recon_h<T, MM, DD, false, false>, gr, 256, 0, st, g, tab, sh, nullptr, W, F, nb);         \
    }                                                                                                     \
  })
        switch (a.d) {
          case 1: CFFT_RECON_D(1); break;
          case 2: CFFT_RECON_D(2); break;
          case 4: CFFT_RECON_D(4); break;
          default: CFFT_RECON_D(8); break;
        }
#undef CFFT_RECON_D
        break;
      }
      case 6: {
        // Fused z FFT + diagonal-sign gather.  One slot per CTA (split lines) while that
        // gives at most two CTAs per SM, else four (two on request), one line per thread.  FP64 below
        // H = 24, whose blocks of four slots are 64 to 128 threads, changes over at 2048 CTAs of one
        // slot (forward us with 1 / 4 slots: Im-3m 48^3 x64, 896 CTAs, 7.8 / 10.6; 64^3 x64, 1152, 10.6 /
        // 13.3; Fm-3m 64^3 x256, 2304, 22.8 / 21.8; Im-3m 48^3 x256, 3584, 18.6 / 16.4; from H = 24 on
        // 4 slots are ahead at every size: Im-3m 96^3 x135 61.6 / 45.3, Pm-3m 48^3 x256 29.3 / 24.3).
        // H = 48: 2 split slots where the units hold many points, whose weights the slots share,
        // else 1.
        const T* K = a.use_K ? static_cast<const T*>(a.K) : nullptr;
        const uint4* un = static_cast<const uint4*>(a.zr_units);
        const uint2* pt = static_cast<const uint2*>(a.zr_pts);
        const C* pq = static_cast<const C*>(a.zr_pq);
        const C* Wc = W;
        CFFT_FOR_H(H, {
          constexpr bool SP = zr_split<HH>();
          const int one = a.zr_n_units * nslots;  // CTAs of one slot
          const int sl = a.zr_slots == 2 || a.zr_slots == 4 ? a.zr_slots
                         : one <= 2 * kSMs || (sizeof(T) == 8 && HH < 24 && one < 2048) ? 1
                         : SP ? (a.n_spec_pts > 512 * a.zr_n_units ? 2 : 1) : zr_slots();
          const size_t sm = (static_cast<size_t>(sl) * 2 * HH * (HH + 1) + HH) * cs;
          const dim3 gzr(a.zr_n_units, (nslots + sl - 1) / sl);
          if (sl == 1)
            launch_k(k_fft_z_recon_diag8<T, HH, 1, true>, gzr, zr_threads<HH, 1, true>(), sm, st, g, tab, K, un, pt, pq, a.n_spec_pts, Wc, F, nb);
          else if (sl == 4)
            launch_k(k_fft_z_recon_diag8<T, HH, 4, SP>, gzr, zr_threads<HH, 4, SP>(), sm, st, g, tab, K, un, pt, pq, a.n_spec_pts, Wc, F, nb);
          else
            launch_k(k_fft_z_recon_diag8<T, HH, 2, SP>, gzr, zr_threads<HH, 2, SP>(), sm, st, g, tab, K, un, pt, pq, a.n_spec_pts, Wc, F, nb);
        });
        break;
      }
      case 8:  // plan set-up: weights of the fused gather
        k_zr_weights<T><<<(a.n_spec_pts + 255) / 256, 256, 0, st>>>(g, tab, static_cast<const uint2*>(a.zr_pts), a.n_spec_pts,
                                                                   static_cast<C*>(const_cast<void*>(a.zr_pq)));
        break;
      case 7:  // forward z FFT + separable Q-multiply + inverse z FFT, in place on W
        CFFT_FOR_H(H, {
          constexpr int HP = HH / 2 + 1;
          const int want = (2 * kSMs + HP * nslots - 1) / (HP * nslots);  // blocks per row that give two CTAs per SM
          const int pp = std::max(2, (HP + want - 1) / want);
          launch_k(k_qsep_z<T, HH>, dim3(HP, (HP + pp - 1) / pp, nslots), kSepThreads,
                   (static_cast<size_t>(4) * pp * (HH + 1) + HH) * sizeof(C), st, g, tab, static_cast<const C*>(a.QS), W, pp);
        });
        break;
      case 3: {
        const uint2* tp = static_cast<const uint2*>(a.fib_taps);
        const uint2* fo = static_cast<const uint2*>(a.fib_outs);
        const int fb = (a.n_fib + kFibers - 1) / kFibers;
#define CFFT_INV_FIBER(LL, NF)                                                                                          \
  {                                                                                                                     \
    const int ns = (nb + (NF) - 1) / (NF);                                                                              \
    const dim3 gf(fb, (ns + (LL) - 1) / (LL));                                                                          \
    switch (a.d) {                                                                                                      \
      case 1: launch_k(k_inv_fiber<T, 1, LL, NF>, gf, kFibers * (LL), 0, st, g, tab, tp, fo, a.n_fib, Fin, G0R, nb); break; \
      case 2: launch_k(k_inv_fiber<T, 2, LL, NF>, gf, kFibers * (LL), 0, st, g, tab, tp, fo, a.n_fib, Fin, G0R, nb); break; \
      case 4: launch_k(k_inv_fiber<T, 4, LL, NF>, gf, kFibers * (LL), 0, st, g, tab, tp, fo, a.n_fib, Fin, G0R, nb); break; \
      default: launch_k(k_inv_fiber<T, 8, LL, NF>, gf, kFibers * (LL), 0, st, g, tab, tp, fo, a.n_fib, Fin, G0R, nb); break; \
    }                                                                                                                   \
  }
        if (a.slot_fields == 1) CFFT_INV_FIBER(2, 1)
        else if (a.reps_wide) CFFT_INV_FIBER(wide_slots<C>(), 2)
        else CFFT_INV_FIBER(2, 2)
#undef CFFT_INV_FIBER
        break;
      }
      default:
        if (a.q_step) {
          CFFT_FOR_H(H, {
            launch_k(k_qmul_ifft_z_h<T, HH>, dim3(HH, nch, nslots), expand_threads<C, HH, 2>(),
                     (expand_plane<HH>() + HH) * sizeof(C), st, g, tab, static_cast<const C*>(a.QT),
                     static_cast<const int32_t*>(a.GT), W, static_cast<C*>(a.W2));
          });
          break;
        }
        CFFT_FOR_H(H, {
          const uint32_t* et = static_cast<const uint32_t*>(a.expand);
          // Rows of two slots: split lines through shared memory for launches of at most one CTA
          // per SM (Im-3m 128^3 FP32, one field, round trip 19.6 against 21.6 us; 8 fields 32.1
          // against 29.8), never above H = 32 (192^3, one field: 44.0 against 30.8).
          if (a.reps_wide) {
            constexpr int L = wide_slots<C>(), LS = expand_slots<C, HH, L>();
            launch_k(k_expand_ifft_z<T, HH, L, LS, sizeof(T) == 8>, dim3(HH, nch, (nslots + L - 1) / L * (L / LS)),
                     expand_threads<C, HH, LS>(), (expand_plane<HH>() * LS + HH) * sizeof(C), st, g, tab, et, G0R, W, nb);
          } else if (HH > 32 || HH * nch * ((nslots + 1) / 2) > kSMs) {
            constexpr int half = ((2 * HH + 31) / 32) * 32;
            launch_k(k_expand2_ifft_z<T, HH, 2>, dim3((HH + 1) / 2, nch, (nslots + 1) / 2), 2 * half, 0, st, g, tab, et, G0R, W, nb);
          } else if constexpr (HH <= 32) {
            launch_k(k_expand_ifft_z<T, HH, 2, 2, true>, dim3(HH, nch, (nslots + 1) / 2), expand_threads<C, HH, 2>(),
                     (expand_plane<HH>() * 2 + HH) * sizeof(C), st, g, tab, et, G0R, W, nb);
          }
        });
        break;
    }
  }
  const cudaError_t le = launch_error();
  launch_error() = cudaSuccess;
  const cudaError_t ge = cudaGetLastError();
  return fast_cuda(le != cudaSuccess ? le : ge, "fast-path launch", err);
}

}  // namespace
}  // namespace cfft
