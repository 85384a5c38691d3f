// Interface between the host execution layer (exec.cu) and the compile-time sized
// fast-path kernels, which are compiled in four translation units (plane stages /
// other stages x float / double) so the build runs in parallel.
#pragma once

#include <string>

#include "cfft_internal.h"

namespace cfft {

struct FastArgs {
  // plan state (device pointers)
  const void* geom = nullptr;
  const void* tables = nullptr;
  const void* spec_h = nullptr;
  const void* K = nullptr;
  const void* fib_taps = nullptr;  // inverse gather by fibers: taps and outputs (uint2)
  const void* fib_outs = nullptr;
  int n_fib = 0;
  const void* expand = nullptr;
  void* W = nullptr;      // channel workspace of this lane
  void* G0R = nullptr;    // representative workspace of this lane
  // call operands
  const void* f0 = nullptr;
  void* F = nullptr;
  const void* Fin = nullptr;
  void* f0_out = nullptr;
  const void* E = nullptr;
  // geometry / dispatch
  int slot_fields = 2;    // fields per workspace slot (1: general kernels)
  int lanes = 1;          // chunks that run concurrently with this one, itself included
  int stage = 0, nb = 0, H = 0, n_ch = 1, centered = 0, cent_type = 0, d = 1;
  int n_spec = 0;
  bool use_K = false, rep_diag8 = false, rep_perm = false;
  bool reps_wide = false;  // representatives in rows of 64 bytes (8 FP32 / 4 FP64 slots), else 2 slots
  // Stage 6 (fused z FFT + diagonal-sign gather): unit table and spectral points.
  const void* zr_units = nullptr;
  const void* zr_pts = nullptr;   // (spectral index, packed h) per point, in unit order
  const void* zr_pq = nullptr;    // weights of the four tap pairs per point
  int n_spec_pts = 0;             // points in the unit lists
  int zr_n_units = 0;
  bool cluster = false;   // fused cluster kernels for stages 0 (with 1) and 5 (with 4)
  int cluster_ctas = 8;   // CTAs per cluster (8, or 16 where the device allows it)
  // Q-matrix step: stage 4 reads W (forward G0, z-fastest) and writes W2; a separable plan
  // runs stage 7 in place on W instead of stages 1 and 4
  bool q_step = false;
  const void* QT = nullptr;   // d x n_ch x H^3 coefficients
  const void* GT = nullptr;   // d x n_ch x H^3 int32 workspace indices (-1: extinct)
  void* W2 = nullptr;
  const void* QS = nullptr;   // 1-D twiddles and kernel factors of the separable Q-multiply
  void* stream = nullptr;
  // bounded device waits of the persistent bulk-copy kernels: limit, and the plan's
  // status word that a wait which runs out sets to CFFT_ERR_TIMEOUT
  unsigned long long timeout_ns = 1000000000ull;
  int* status = nullptr;
  // per-plan choices (0 / -1: the process default)
  int zr_slots = 0;
  int tma = -1;
};

// Geometry of the general kernels (any 2-3-5 channel grid), passed by value.  Each axis length
// is A x B with both factors in general_radix; a "d" member is the multiplier of div_by.
struct GenShape {
  int H[3], A[3], B[3], M[3], N[3];
  int nch, centered, d, P, n_spec, n_orbits;
  int S;             // shared-memory row stride (odd)
  int chan[8];       // channel of a parity class, or -1
  int tw[3], ftw[3], ph;  // table offsets: line twiddles, fold twiddles, phases
  int lift[3];       // multiple of M above any |R^T h|
  int PN[3];         // P / N
  uint32_t dH[3], dA[3], dB[3], dM[3], dN[3], dLx, dLy;
  size_t hvol, mvol;
  double inv_v;      // normalisation of the inverse
};
Status general_f32(const FastArgs& a, const GenShape& s, std::string* err);
Status general_f64(const FastArgs& a, const GenShape& s, std::string* err);
Status general_init_f32(std::string* err);
Status general_init_f64(std::string* err);

// Stages 0 and 5 (plane kernels) and stages 1-4 (z FFTs, gathers).
Status fast_planes_f32(const FastArgs& a, std::string* err);
Status fast_planes_f64(const FastArgs& a, std::string* err);
Status fast_other_f32(const FastArgs& a, std::string* err);
Status fast_other_f64(const FastArgs& a, std::string* err);
// Largest number of concurrently resident kc-CTA clusters of the fused forward and
// backward kernels for channel edge H and centring type ct (0 if they cannot run).
Status fast_cluster_probe_f32(int H, int ct, int kc, int* max_clusters, std::string* err);
Status fast_cluster_probe_f64(int H, int ct, int kc, int* max_clusters, std::string* err);
// Whether the persistent bulk-copy plane kernels serve channel edge H and centring
// type ct (forward without / with interaction factors, backward).
void fast_tma_planes_f32(int H, int ct, int tma, bool* fwd, bool* fwd_e, bool* bwd);
void fast_tma_planes_f64(int H, int ct, int tma, bool* fwd, bool* fwd_e, bool* bwd);
// Launches the bounded-wait self-test kernel (k_wait_selftest) on `stream`.
Status fast_wait_selftest(unsigned long long timeout_ns, int* status, void* stream, std::string* err);
// Per-device set-up of each unit: constant-memory twiddles and shared-memory limits.
Status fast_init_planes_f32(std::string* err);
Status fast_init_planes_f64(std::string* err);
Status fast_init_other_f32(std::string* err);
Status fast_init_other_f64(std::string* err);

// Cubic channel edges with compile-time sized kernels for element size `real_bytes`.
inline bool fast_size_ok(int H, int real_bytes) {
  return H == 4 || H == 6 || H == 8 || H == 12 || H == 16 || H == 24 || H == 32 || (H == 48 && real_bytes == 4);
}
constexpr int kFastZB = 4;  // xz-planes (y values) per CTA in the z kernels

// The fused cluster kernels hold one slot's channel volume in the shared memory of 8
// CTAs (H / 8 z-planes of nch padded H x (H + 1) planes each, one z line per thread).
inline bool fast_cluster_fits(int H, int nch, int real_bytes) {
  if (H % 8 != 0 || H < 16 || H > 32) return false;
  const long threads = static_cast<long>(nch) * (H / 8) * H;
  const long smem = static_cast<long>(H / 8) * nch * H * (H + 1) * 2 * real_bytes;
  return threads >= 32 && threads <= 1024 && smem <= 227 * 1024;
}

}  // namespace cfft
