// IMRPhenomXHM at the frequencies for sm_100a: the modes h_{l,-m} of
// (2,2), (2,1), (3,3), (3,2), (4,4) and (h+, hx) from the tables of
// wfx_xhm_setup (models/xhm/core.py:409-556), and the C-ABI entry.
//
// One block per (binary, run of frequencies), the binary's row staged in
// shared memory; one thread per frequency. The (2,2) is IMRPhenomXAS's
// point (point.cuh); each higher mode's amplitude and phase follow
// mode_rest (core.py:429-518): the phase of the region, with the (2,2)
// leading term rescaled, T0_lm f^-5/3, in the inspiral; the (3,2) ringdown
// rotates the recycled (2,2) mode with its own spheroidal ringdown.
//  * FP64: the reference's float64 evaluation;
//  * FP32: float, with each region's constant (the (2,2) anchor folded in,
//    reduced modulo 2 pi at set-up), coefficient of f and leading term in
//    double-float, as IMRPhenomXAS's FP32 phase.
// t_c multiplies every mode by exp(-2 pi i f t_c) (an extension; zero
// reproduces the reference).
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/waveformx_b200.h"
#include "dual_point.cuh"
#include "internal.h"
#include "matrix_sums.cuh"
#include "point.cuh"
#include "setup_xhm.cuh"
#include "tables.cuh"

namespace wfx {

namespace {

constexpr int kXhmBlock = 128;
constexpr int kXhmBinariesPerBlock = 8;
constexpr int kModesOut = 5;

template <class S>
struct C2 {
  S re, im;
};

template <class S>
struct XhmRow;
// (kMinBlocks: the launch bound, blocks of 128 per SM; measured on the
// 4096 x 4017 batch: FP32 4 blocks 1.05 ms, 5 0.93, 6 0.89, 8 0.80 (64
// registers, a little spilled); FP64 4 blocks 2.45 ms, 6 2.24)
template <>
struct XhmRow<float> {
  static constexpr int kStride = kXhmStride32, kMode = kXhmModeStride32, kMinBlocks = 8;
};
template <>
struct XhmRow<double> {
  static constexpr int kStride = kXhmStride64, kMode = kXhmModeStride64, kMinBlocks = 6;
};

// FP32: atan(y / x) by the minimax atan of point.cuh (2.6e-7 absolute), moved
// to the quadrant of (x, y) (x < 0: plus or minus pi by the sign of y, signed
// zeros included); the modulus of O(1) values from the sum of squares; the
// sine and cosine of an angle reduced modulo 2 pi (2 pi in two floats) by
// the fast intrinsic. FP64: the library's functions.
__device__ __forceinline__ float m_atan2(float y, float x) {
  const float a = m_atan(__fdividef(y, x));
  return x < 0.0f ? a + copysignf(3.14159265358979323846f, y) : a;
}
__device__ __forceinline__ double m_atan2(double y, double x) { return atan2(y, x); }
__device__ __forceinline__ float m_hypot(float a, float b) { return sqrtf(__fmaf_rn(a, a, b * b)); }
__device__ __forceinline__ double m_hypot(double a, double b) { return hypot(a, b); }
__device__ __forceinline__ void full_sincos(float x, float* s, float* c) {
  const float k = rintf(x * kInvTwoPi);
  const float r = __fmaf_rn(-k, kTwoPiLo, __fmaf_rn(-k, kTwoPiHi, x));
  __sincosf(r, s, c);
}
__device__ __forceinline__ void full_sincos(double x, double* s, double* c) { sincos(x, s, c); }

// The amplitude (amp0 included, >= 0 but FALSE_ZERO) and the phase of the
// higher mode of table M (emm its m; mixing: the (3,2)) at one frequency;
// (c22, s22): the (2,2) mode without its anchor, A22 (cos, sin) of its
// phase (core.py:429-518, 524-547).
template <class S>
__device__ __forceinline__ void mode_point(const S* __restrict__ M, const S* __restrict__ H, const Freq<S>& q,
                                           int emm, bool mixing, S c22, S s22, const S* __restrict__ T22, S t0_lm,
                                           S& amp, S& phi) {
  using namespace xhm;
  constexpr bool kF32 = sizeof(S) == 4;
  const S f = q.f, t = q.t, m1 = q.m1, lf = q.lf;
  const S t2 = t * t, mt1 = t2 * m1, m2 = m1 * m1;
  const S s = H[H_S], amp0 = H[H_AMP0];
  const bool past_ins = f >= M[M_F_PHASE_IN];
  const bool rd_phase = f >= M[M_F_PHASE_IM];
  const int region = rd_phase ? 2 : (past_ins ? 1 : 0);
  const S* R = M + M_PHASE + region * kBasis;
  // the region's sum (core.py:453-460), but (FP32) its constant and its
  // coefficient of f, which go in double-float below
  S sum = kF32 ? S(0) : R[B_1] + R[B_F] * f;
  if (region == 0) {
    sum = sum + R[B_M4_3] * (m1 * mt1);
    sum = sum + R[B_M1] * m1;
    sum = sum + R[B_M2_3] * (mt1 * mt1);
    sum = sum + R[B_M1_3] * mt1;
    sum = sum + R[B_1_3] * t;
    sum = sum + R[B_2_3] * t2;
    sum = sum + R[B_4_3] * (f * t);
    sum = sum + R[B_5_3] * (f * t2);
    sum = sum + R[B_F2] * (f * f);
    sum = sum + R[B_7_3] * (f * f * t);
    sum = sum + R[B_LOG] * lf;
    sum = sum + R[B_1_3_LOG] * (t * lf);
    sum = sum + R[B_F_LOG] * (f * lf);
    sum = sum + R[B_4_3_LOG] * (f * t * lf);
  } else if (region == 1) {
    sum = sum + R[B_LOG] * lf;
    sum = sum + R[B_M1] * m1;
    sum = sum + R[B_M2] * m2;
    sum = sum + R[B_M3] * (m2 * m1);
  } else if (!mixing) {
    sum = sum + R[B_M1] * m1;
  }
  const S y = f - M[M_SHIFT];
  const bool amp_rd_region = f >= M[M_F_AMP_IM];
  // the ringdown amplitude: the Lorentzian, the fall-off, the cubic of the
  // (3,2) below f_aux; then the (3,2)'s rotation (core.py:462-497)
  S amp_rd = S(0), rest_rd = S(0);
  if (rd_phase || amp_rd_region) {
    const S u = s * y;
    S arg = M[M_RD + 1] * u;
    arg = arg < S(-30) ? S(-30) : (arg > S(30) ? S(30) : arg);
    const S lor = m_div(M[M_RD + 0], m_exp(arg) * (u * u + M[M_RD + 2]));
    const S fo2 = M[M_FALLOFF + 2];
    const S over = f - fo2;
    const S fall = M[M_FALLOFF + 0] * m_exp(-M[M_FALLOFF + 1] * (over > S(0) ? over : S(0)));
    amp_rd = f >= fo2 ? fall : lor;
    const S at_rd = M[M_ATAN_A + 2] * m_atan(M[M_ATAN_W + 2] * y);
    if (mixing) {
      const S* a = M + M_AUX;
      const S aux = ((a[3] * f + a[2]) * f + a[1]) * f + a[0];
      amp_rd = f < M[M_F_AUX] ? aux : amp_rd;
      const S phi_s = M[M_SPH + 0] * f + M[M_SPH + 1] + M[M_SPH + 2] * m1 + M[M_SPH + 3] * (m2 * m1) + at_rd;
      S sn, cn;
      full_sincos(phi_s, &sn, &cn);
      const S cs = amp_rd * cn, ss = amp_rd * sn;
      const S m2r = M[M_MIX + 0], m2i = M[M_MIX + 1], m3r = M[M_MIX + 2], m3i = M[M_MIX + 3];
      const S re = c22 * m2r + s22 * m2i + cs * m3r + ss * m3i;
      const S im = s22 * m2r - c22 * m2i + ss * m3r - cs * m3i;
      const bool nonzero = (m_abs(re) > m_abs(im) ? m_abs(re) : m_abs(im)) > 1e-37;
      amp_rd = nonzero ? m_hypot(re, im) : S(0);
      rest_rd = nonzero ? m_atan2(im, re) : S(0);
    } else {
      rest_rd = at_rd;
    }
  }
  S rest;
  if (region == 2) {
    rest = sum + rest_rd;
  } else if (region == 1) {
    rest = sum + M[M_ATAN_A + 1] * m_atan(M[M_ATAN_W + 1] * y);
  } else {
    rest = sum;
  }
  // the amplitude (core.py:500-517)
  S a;
  if (f < M[M_F_AMP_IN]) {
    S pr = M[M_PN_RE + 6], pi = M[M_PN_IM + 6];
#pragma unroll
    for (int k = 5; k >= 0; --k) {
      pr = pr * t + M[M_PN_RE + k];
      pi = pi * t + M[M_PN_IM + k];
    }
    const S t3 = t * t * t;
    const S t7 = t3 * t3 * t;
    const S pseudo = t7 * (M[M_PSEUDO + 0] + t * (M[M_PSEUDO + 1] + t * M[M_PSEUDO + 2]));
    a = q.m76 * (m_hypot(pr, pi) + pseudo);
  } else if (amp_rd_region) {
    a = amp_rd;
  } else {
    const S v = (f - M[M_INTER_C]) * M[M_INTER_H];
    S inter = M[M_INTER + 7];
#pragma unroll
    for (int j = 6; j >= 0; --j) inter = inter * v + M[M_INTER + j];
    a = q.m76 * inter;
  }
  amp = a < S(0) ? S(kFalseZero) * amp0 : a;
  // the phase: [inspiral] T0_lm f^-5/3 - (m/2) A + rest, reduced
  const S m_over_2 = S(emm) * S(0.5);
  if constexpr (kF32) {
    const int cs = M_PHASE + region * kBasis + B_1, ls = M_PHASE + region * kBasis + B_F;
    const df p = two_prod(M[ls], f);
    S ph = M[cs] + reduce_df(p.hi, __fmaf_rn(M[HM32_LIN_LO + region], f, p.lo));
    if (!past_ins) {
      const df big = df_mul(df{M[HM32_T0_HI], M[HM32_T0_LO]}, q.y);
      ph = ph + reduce_df(big.hi, big.lo);
    }
    ph = ph + rest;
    const S k = round_nearest(ph * kInvTwoPi);
    ph = __fmaf_rn(-k, kTwoPiHi, ph);
    phi = __fmaf_rn(-k, kTwoPiLo, ph);
  } else {
    S ph = !past_ins ? t0_lm * q.y : S(0);
    ph = ph - m_over_2 * T22[X_ANCHOR];
    ph = ph + rest;
    phi = ph - m_round(ph / kTwoPi) * kTwoPi;
  }
}

// e^(-2 pi i f t_c) as (cos, sin).
__device__ __forceinline__ void tc_factor(float f, float t_c, float& c, float& s) {
  const TcF tc = make_tc(t_c);
  const df p = two_prod(tc.hi, f);
  const float ph = reduce_df(p.hi, __fmaf_rn(tc.lo, f, p.lo));
  __sincosf(-ph, &s, &c);
}
__device__ __forceinline__ void tc_factor(double f, double t_c, double& c, double& s) {
  double ph = kTwoPi * f * t_c;
  ph = ph - rint(ph / kTwoPi) * kTwoPi;
  sincos(-ph, &s, &c);
}

template <class S>
__global__ void __launch_bounds__(kXhmBlock, XhmRow<S>::kMinBlocks)
    k_xhm(const S* __restrict__ table, const S* __restrict__ freqs, const int64_t* __restrict__ offsets, int64_t B,
          int64_t n, const S* __restrict__ t_c, C2<S>* __restrict__ hp, C2<S>* __restrict__ hc,
          C2<S>* __restrict__ modes) {
  constexpr bool kF32 = sizeof(S) == 4;
  constexpr int kStride = XhmRow<S>::kStride, kMode = XhmRow<S>::kMode;
  __shared__ __align__(16) S T[kStride];
  __shared__ S t0_lm[4];  // (FP64) the rescaled leading term (m/2)^(8/3) T0 of each mode
  // (a shared grid with at most one frequency a thread: each thread's
  // frequency powers, computed for the block's first binary and read back
  // for the others)
  __shared__ Freq<S> powers[kXhmBlock];
  const bool reuse = offsets == nullptr && n <= static_cast<int64_t>(gridDim.x) * blockDim.x;
  bool have_powers = false;
  for (int64_t b = blockIdx.y; b < B; b += gridDim.y) {
    __syncthreads();  // (T is rewritten)
    for (int k = threadIdx.x; k < kStride; k += blockDim.x) T[k] = table[b * kStride + k];
    if (!kF32 && threadIdx.x < 4) {
      const int m = threadIdx.x;
      const double emm = m == 0 ? 1.0 : (m == 1 ? 3.0 : (m == 2 ? 2.0 : 4.0));
      t0_lm[m] = S(pow(emm * 0.5, 8.0 / 3.0) * double(table[b * kStride + X_T0]));
    }
    __syncthreads();
    if constexpr (kF32) {
      if (threadIdx.x == 0) {
        const int cs[3] = {xas_const_slot(0), xas_const_slot(1), xas_const_slot(2)};
        const int ls[3] = {xas_lin_slot(0), xas_lin_slot(1), xas_lin_slot(2)};
        prepare_f32<3>(T, cs, X32_CONST_LO, ls, X32_LIN_LO, 0.0f);
      }
      __syncthreads();
    }
    const S tcb = t_c != nullptr ? t_c[b] : S(0);

    const S* Hd = T;
    // (a shared grid: frequencies [0, n), outputs at b n + j; ragged: the
    // binary's own [offsets[b], offsets[b + 1]) of the flat arrays, clamped
    // to [0, n]: inconsistent offsets read and write nothing out of bounds)
    const int64_t lo = offsets != nullptr ? min(max(offsets[b], int64_t(0)), n) : 0;
    const int64_t hi = offsets != nullptr ? min(max(offsets[b + 1], lo), n) : n;
    const int64_t row = offsets != nullptr ? 0 : b * n;
    for (int64_t j = lo + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < hi;
         j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
      const S f = freqs[j];
      Freq<S> q;
      if (reuse && have_powers) {
        q = powers[threadIdx.x];
      } else {
        q = freq_powers(f);
        if (reuse) {
          powers[threadIdx.x] = q;
          have_powers = true;
        }
      }
      typename TcOf<S>::type zero{};
      const Point<S> p22 = xas_point<S>(T, q, zero);
      S tcc = S(1), tcs = S(0);
      if (t_c != nullptr) tc_factor(f, tcb, tcc, tcs);
      C2<S> sp{S(0), S(0)}, sc{S(0), S(0)};
      // adds mode k (t_c applied) to the polarizations, and writes it
      auto add = [&](int k, S re, S im) {
        const S* F = Hd + H_FACTORS + 4 * k;
        const C2<S> x{re * tcc - im * tcs, im * tcc + re * tcs};
        sp.re = sp.re + (F[0] * x.re - F[1] * x.im);
        sp.im = sp.im + (F[0] * x.im + F[1] * x.re);
        sc.re = sc.re + (F[2] * x.re - F[3] * x.im);
        sc.im = sc.im + (F[2] * x.im + F[3] * x.re);
        if (modes != nullptr) modes[(b * kModesOut + k) * n + j] = x;
      };
      const S h22r = p22.amp * p22.c, h22i = p22.amp * p22.s;
      add(0, h22r, h22i);
      // the (2,2) without its anchor: the angle turned by A
      const S ca = Hd[H_COS_A], sa = Hd[H_SIN_A];
      const S c22 = h22r * ca - h22i * sa, s22 = h22i * ca + h22r * sa;
#pragma unroll 1
      for (int m = 0; m < 4; ++m) {
        const S* M = T + H_MODES + m * kMode;
        const int emm = m == 0 ? 1 : (m == 1 ? 3 : (m == 2 ? 2 : 4));
        S amp, phi;
        mode_point<S>(M, Hd, q, emm, m == 2, c22, s22, T, t0_lm[m], amp, phi);
        const S sign = (m == 0 || m == 3) ? S(1) : S(-1);  // (-1)^l
        const S a = sign * M[xhm::M_ON] * amp;
        S sn, cn;
        m_sincos(phi, &sn, &cn);
        add(m + 1, a * cn, a * sn);
      }
      hp[row + j] = sp;
      hc[row + j] = sc;
    }
  }
}

// (h+, hx) of IMRPhenomXHM on dual numbers at the powers q of one frequency,
// the modes summed as k_xhm sums them; (tcc, tcs) = e^(-2 pi i f t_c) as
// (cos, sin), double where it carries no derivative, Dual where it does.
template <class TC>
__device__ __forceinline__ void xhm_dual_sum(const Dual* T, const Dual* t0_lm, const Freq<Dual>& q, TC tcc, TC tcs,
                                             C2<Dual>& sp, C2<Dual>& sc) {
  constexpr int kMode = kXhmModeStride64;
  const Point<Dual> p22 = xas_point<Dual>(T, q, 0.0);
  sp = C2<Dual>{Dual(0.0), Dual(0.0)};
  sc = C2<Dual>{Dual(0.0), Dual(0.0)};
  auto add = [&](int k, Dual re, Dual im) {
    const Dual* F = T + H_FACTORS + 4 * k;
    const C2<Dual> x{re * tcc - im * tcs, im * tcc + re * tcs};
    sp.re = sp.re + (F[0] * x.re - F[1] * x.im);
    sp.im = sp.im + (F[0] * x.im + F[1] * x.re);
    sc.re = sc.re + (F[2] * x.re - F[3] * x.im);
    sc.im = sc.im + (F[2] * x.im + F[3] * x.re);
  };
  const Dual h22r = p22.amp * p22.c, h22i = p22.amp * p22.s;
  add(0, h22r, h22i);
  const Dual ca = T[H_COS_A], sa = T[H_SIN_A];
  const Dual c22 = h22r * ca - h22i * sa, s22 = h22i * ca + h22r * sa;
#pragma unroll 1
  for (int m = 0; m < 4; ++m) {
    const Dual* M = T + H_MODES + m * kMode;
    const int emm = m == 0 ? 1 : (m == 1 ? 3 : (m == 2 ? 2 : 4));
    Dual amp, phi;
    mode_point<Dual>(M, T, q, emm, m == 2, c22, s22, T, t0_lm[m], amp, phi);
    const double sign = (m == 0 || m == 3) ? 1.0 : -1.0;  // (-1)^l
    const Dual a = sign * M[xhm::M_ON] * amp;
    Dual sn, cn;
    m_sincos(phi, &sn, &cn);
    add(m + 1, a * cn, a * sn);
  }
}

// IMRPhenomXHM's gradient in reverse mode: the cotangents of (h+, hx) at each
// frequency become sums of dL/d(row) over the binary's row (table64), which
// the block contracts with dtable. (The reference's GPU port contracts forward
// derivatives along the eight parameters, models/xhm/mlx/_api.py:30-46; the
// reverse pass evaluates each mode once instead of eight times on dual
// numbers.)
//
// Block: one binary, kAdjSpan frequencies at a time:
//  1. thread i takes the span's frequency i: its powers, the (2,2)
//     (xas_point) and the cotangents turned by e^(2 pi i f t_c); the basis of
//     the phases (HM_BASIS), f^-5/3 and the cotangents become the rows of a
//     matrix over the span's frequencies in shared memory;
//  2. warp w takes the higher mode w over the whole span, 32 frequencies at a
//     time: its value, and the cotangents of its phase and amplitude, which
//     become eight columns over the 32 frequencies (the phase's in the column
//     of its region, zero in the others');
//  3. each warp takes the (2,2) at its own frequencies, with what the (3,2)'s
//     rotation of the recycled (2,2) sent back.
// The sums over the frequencies are products of the rows with the columns, on
// the FP64 matrix instruction (m8n8k4: 24 rows x 8 columns take 24 of them for
// 32 frequencies, in 12 registers a lane). With a register per sum and lane
// instead, the kernel held 255 registers, two blocks a SM: 856 us for 250 x
// 4017 against 439 (705 held to 128 registers), and 2156 for the eight
// directions on dual numbers. Bound by latency: 15 warps a SM issue in 35 % of
// the cycles (instruction fetch, the elementary functions' chains, the
// barriers between the stages).
constexpr int kAdjSpan = kSpan;
constexpr int kAdjWarps = kXhmBlock / 32;
static_assert(kAdjSpan == kXhmBlock && kAdjWarps == xhm::kModes, "a thread a frequency, a warp a higher mode");
// Blocks of a launch before a block takes more than one span of a binary (each
// block pays one contraction with dtable): four waves of four blocks a SM.
constexpr int64_t kAdjBlocks = 4 * 4 * 148;

// The rows of the span's matrix: HM_BASIS (t^0 .. t^7 at kRowT + k), f^-5/3,
// the cotangents.
constexpr int kRowT = xhm::B_1, kRowF = xhm::B_F, kRowF2 = xhm::B_F2;
constexpr int kRowY = xhm::kBasis, kRowG = kRowY + 1, kRows = kRowG + 4;
static_assert(kRowT + 7 == xhm::B_7_3 && kRows <= 24, "three tiles of eight rows");
// Sums of a warp outside its mode's table: the (2,2)'s slots, then t_c and the
// head's.
enum WarpSum : int { W_TC = 58, W_S = 60, W_AMP0 = 61, W_COS = 62, W_SIN = 63, W_FACTOR = 64, W_FACTOR22 = 68 };

struct AdjShared {
  double T[kXhmStride64];
  double rows[kRows * kRowStride];
  double m76[kAdjSpan];
  double h22r[kAdjSpan], h22i[kAdjSpan];  // the (2,2); from the (3,2)'s warp on, its cotangent from the rotation
  double stage[kAdjWarps][kStage];
  double modes[xhm::kModes * kXhmModeStride64];  // dL/d(mode tables); warp m its own
  double sums[kAdjWarps][kTableStride];
};
static_assert(sizeof(AdjShared) <= 48 * 1024, "static shared memory");

// The derivatives of a mode's factors from the products of its value (columns
// 6, 7 of stage) with the cotangents: factor i of Re F+, Im F+, Re Fx, Im Fx.
__device__ __forceinline__ double factor_sum(const double* stage, int i) {
  const double* g = stage + 8 * (kRowG + (i & 2));
  return (i & 1) ? g[8 + 6] - g[7] : g[6] + g[8 + 7];
}

// The cotangent of a mode's value from those of the polarizations, its factors
// F.
__device__ __forceinline__ C2<double> mode_cotangent(const double* F, double gpr, double gpi, double gcr, double gci) {
  return C2<double>{F[0] * gpr + F[1] * gpi + F[2] * gcr + F[3] * gci,
                    F[0] * gpi - F[1] * gpr + F[2] * gci - F[3] * gcr};
}

// Stage 2: the higher mode m over the span's first `count` frequencies. (One
// instance for the four modes, the (3,2)'s rotation a branch: the block's
// warps then fetch the same instructions, 439 us against 508 for 250 x 4017
// with the (3,2) compiled apart.)
__device__ __forceinline__ void mode_reverse(AdjShared& sh, int m, int count, int lane) {
  using namespace xhm;
  const bool mix = m == 2;
  const double* T = sh.T;
  const double* M = T + H_MODES + m * kXhmModeStride64;
  const double* F = T + H_FACTORS + 4 * (m + 1);
  double* stage = sh.stage[m];
  const double m_over_2 = m == 0 ? 0.5 : (m == 1 ? 1.5 : (m == 2 ? 1.0 : 2.0));
  const double t0_scale = pow(m_over_2, 8.0 / 3.0), t0_lm = t0_scale * T[X_T0];
  const double on = ((m == 0 || m == 3) ? 1.0 : -1.0) * M[M_ON];  // (-1)^l
  double d1[3][2] = {}, di[2] = {}, dr[2] = {}, dm[3][2] = {};
  // the arc tangents' sums, dL/d(shift), amp0's and (mix) sin A's
  double at1_sum = 0.0, w1_sum = 0.0, at2_sum = 0.0, w2_sum = 0.0, shift = 0.0, amp0 = 0.0, sin_a = 0.0;
  bool any_inter = false, any_ring = false;
  for (int base = 0; base < count; base += 32) {
    const int i = base + lane;  // (frequencies past the span's count have zero cotangents)
    const double* q = sh.rows + i;
    const double f = q[kRowF * kRowStride], t = q[B_1_3 * kRowStride], m1 = q[B_M1 * kRowStride];
    const double t2 = q[B_2_3 * kRowStride], m3 = q[B_M3 * kRowStride], m76 = sh.m76[i];
    const int region = f >= M[M_F_PHASE_IM] ? 2 : (f >= M[M_F_PHASE_IN] ? 1 : 0);
    const int amp_region = f < M[M_F_AMP_IN] ? 0 : (f >= M[M_F_AMP_IM] ? 2 : 1);
    const bool ring = mix ? (region == 2 || amp_region == 2) : amp_region == 2;
    const double y = f - M[M_SHIFT];
    // --- the value (mode_point's)
    const double* R = M + M_PHASE + region * kBasis;
    double rest = R[B_1] + R[B_F] * f;
    if (region == 0) {
      rest += R[B_M4_3] * q[B_M4_3 * kRowStride];
      rest += R[B_M1] * m1;
      rest += R[B_M2_3] * q[B_M2_3 * kRowStride];
      rest += R[B_M1_3] * q[B_M1_3 * kRowStride];
      rest += R[B_1_3] * t;
      rest += R[B_2_3] * t2;
      rest += R[B_4_3] * q[B_4_3 * kRowStride];
      rest += R[B_5_3] * q[B_5_3 * kRowStride];
      rest += R[B_F2] * q[B_F2 * kRowStride];
      rest += R[B_7_3] * q[B_7_3 * kRowStride];
      rest += R[B_LOG] * q[B_LOG * kRowStride];
      rest += R[B_1_3_LOG] * q[B_1_3_LOG * kRowStride];
      rest += R[B_F_LOG] * q[B_F_LOG * kRowStride];
      rest += R[B_4_3_LOG] * q[B_4_3_LOG * kRowStride];
      rest += t0_lm * q[kRowY * kRowStride];
    } else if (region == 1) {
      rest += R[B_LOG] * q[B_LOG * kRowStride];
      rest += R[B_M1] * m1;
      rest += R[B_M2] * q[B_M2 * kRowStride];
      rest += R[B_M3] * m3;
    } else if (!mix) {
      rest += R[B_M1] * m1;
    }
    // the arc tangents of the intermediate and of the ringdown (the (3,2): of
    // its spheroidal phase), each with 1 / (1 + z^2)
    double at1 = 0.0, zz1 = 0.0, at2 = 0.0, zz2 = 0.0;
    if (region == 1) {
      const double z = M[M_ATAN_W + 1] * y;
      at1 = atan(z);
      zz1 = 1.0 / (1.0 + z * z);
      rest += M[M_ATAN_A + 1] * at1;
    }
    if (mix ? ring : region == 2) {
      const double z = M[M_ATAN_W + 2] * y;
      at2 = atan(z);
      zz2 = 1.0 / (1.0 + z * z);
      if (!mix) rest += M[M_ATAN_A + 2] * at2;
    }
    // the ringdown's amplitude before the (3,2)'s rotation
    double lor = 0.0, inv_lor = 0.0, u = 0.0, fall = 0.0, over = 0.0, mag = 0.0;
    bool clipped = false, is_fall = false, is_aux = false;
    if (ring) {
      is_aux = mix && f < M[M_F_AUX];
      is_fall = !is_aux && f >= M[M_FALLOFF + 2];
      if (is_aux) {
        const double* a = M + M_AUX;
        mag = ((a[3] * f + a[2]) * f + a[1]) * f + a[0];
      } else if (is_fall) {
        over = f - M[M_FALLOFF + 2];
        fall = exp(-M[M_FALLOFF + 1] * over);
        mag = M[M_FALLOFF + 0] * fall;
      } else {
        u = T[H_S] * y;
        double arg = M[M_RD + 1] * u;
        clipped = arg < -30.0 || arg > 30.0;
        arg = arg < -30.0 ? -30.0 : (arg > 30.0 ? 30.0 : arg);
        inv_lor = 1.0 / (u * u + M[M_RD + 2]);
        lor = inv_lor * exp(-arg);
        mag = M[M_RD + 0] * lor;
      }
    }
    double re = 0.0, im = 0.0, cn = 0.0, sn = 0.0, hr = 0.0, hi = 0.0, rot = 0.0;
    bool nonzero = false;
    if (mix && ring) {
      hr = sh.h22r[i];
      hi = sh.h22i[i];
      const double ca = T[H_COS_A], sa = T[H_SIN_A];
      const double c22 = hr * ca - hi * sa, s22 = hi * ca + hr * sa;
      const double phi_s = M[M_SPH + 0] * f + M[M_SPH + 1] + M[M_SPH + 2] * m1 + M[M_SPH + 3] * m3 +
                           M[M_ATAN_A + 2] * at2;
      sincos(phi_s, &sn, &cn);
      const double cs = mag * cn, ss = mag * sn;
      const double m2r = M[M_MIX + 0], m2i = M[M_MIX + 1], m3r = M[M_MIX + 2], m3i = M[M_MIX + 3];
      re = c22 * m2r + s22 * m2i + cs * m3r + ss * m3i;
      im = s22 * m2r - c22 * m2i + ss * m3r - cs * m3i;
      nonzero = fmax(fabs(re), fabs(im)) > 1e-37;
      rot = nonzero ? sqrt(re * re + im * im) : 0.0;
      if (region == 2 && nonzero) rest += atan2(im, re);
    }
    double a, pr = 0.0, pi = 0.0, t7 = 0.0, root = 0.0, v = 0.0;
    if (amp_region == 0) {
      pr = M[M_PN_RE + 6];
      pi = M[M_PN_IM + 6];
#pragma unroll
      for (int k = 5; k >= 0; --k) {
        pr = pr * t + M[M_PN_RE + k];
        pi = pi * t + M[M_PN_IM + k];
      }
      t7 = q[B_7_3 * kRowStride];
      root = sqrt(pr * pr + pi * pi);
      a = m76 * (root + t7 * (M[M_PSEUDO + 0] + t * (M[M_PSEUDO + 1] + t * M[M_PSEUDO + 2])));
    } else if (amp_region == 2) {
      a = mix ? rot : mag;
    } else {
      v = (f - M[M_INTER_C]) * M[M_INTER_H];
      double inter = M[M_INTER + 7];
#pragma unroll
      for (int j = 6; j >= 0; --j) inter = inter * v + M[M_INTER + j];
      a = m76 * inter;
    }
    const bool below = a < 0.0;
    const double amp = on * (below ? kFalseZero * T[H_AMP0] : a);
    double phi = rest - m_over_2 * T[X_ANCHOR];
    phi = phi - rint(phi / kTwoPi) * kTwoPi;
    double sphi, cphi;
    sincos(phi, &sphi, &cphi);
    // --- the cotangents of the amplitude and the phase
    const double* g = q + kRowG * kRowStride;
    const C2<double> xb = mode_cotangent(F, g[0], g[kRowStride], g[2 * kRowStride], g[3 * kRowStride]);
    double ab = on * (xb.re * cphi + xb.im * sphi);
    const double pb = amp * (xb.im * cphi - xb.re * sphi);
    if (below) {
      amp0 += kFalseZero * ab;
      ab = 0.0;
    }
    {
      const double h = amp_region == 0 ? ab * m76 : 0.0, inv = root > 0.0 ? h / root : 0.0;
      put_columns(stage, {region == 0 ? pb : 0.0, region == 1 ? pb : 0.0, region == 2 ? pb : 0.0, pr * inv, pi * inv,
                          h * t7, amp * cphi, amp * sphi}, lane);
      mma_rows<kRows>(d1, sh.rows + base, stage, lane);
    }
    if (region == 1) {
      const double gz = pb * M[M_ATAN_A + 1] * zz1;
      at1_sum += pb * at1;
      w1_sum += gz * y;
      shift -= gz * M[M_ATAN_W + 1];
    } else if (!mix && region == 2) {
      const double gz = pb * M[M_ATAN_A + 2] * zz2;
      at2_sum += pb * at2;
      w2_sum += gz * y;
      shift -= gz * M[M_ATAN_W + 2];
    }
    if (__any_sync(0xffffffffu, amp_region == 1)) {
      // the sums of w v^j, j = 0..7: the powers of v as rows, w as column 0
      any_inter = true;
      const double v2 = v * v, v4 = v2 * v2;
      put_columns(stage, {1.0, v, v2, v2 * v, v4, v4 * v, v4 * v2, v4 * v2 * v}, lane);
      const double w = amp_region == 1 ? ab * m76 : 0.0;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const double b = __shfl_sync(0xffffffffu, w, 4 * s + (lane & 3));
        mma_f64(di, stage[(lane >> 2) * kStageStride + 4 * s + (lane & 3)], lane < 4 ? b : 0.0);
      }
    }
    if (__any_sync(0xffffffffu, ring)) {
      any_ring = true;
      double mb = ring ? ab : 0.0;  // the cotangent of the magnitude before the rotation
      double b_re = 0.0, b_im = 0.0;
      if (mix) {
        mb = 0.0;
        double psb = 0.0, m2rb = 0.0, m2ib = 0.0, m3rb = 0.0, m3ib = 0.0, cos_a = 0.0;
        if (nonzero) {
          const double arb = amp_region == 2 ? ab : 0.0, prb = region == 2 ? pb : 0.0;
          const double inv = 1.0 / rot, er = re * inv, ei = im * inv;
          const double reb = arb * er - prb * ei * inv, imb = arb * ei + prb * er * inv;
          const double m2r = M[M_MIX + 0], m2i = M[M_MIX + 1], m3r = M[M_MIX + 2], m3i = M[M_MIX + 3];
          const double ca = T[H_COS_A], sa = T[H_SIN_A];
          const double c22 = hr * ca - hi * sa, s22 = hi * ca + hr * sa, cs = mag * cn, ss = mag * sn;
          m2rb = reb * c22 + imb * s22;
          m2ib = reb * s22 - imb * c22;
          m3rb = reb * cs + imb * ss;
          m3ib = reb * ss - imb * cs;
          const double c22b = reb * m2r - imb * m2i, s22b = reb * m2i + imb * m2r;
          const double csb = reb * m3r - imb * m3i, ssb = reb * m3i + imb * m3r;
          mb = csb * cn + ssb * sn;
          psb = mag * (ssb * cn - csb * sn);
          const double gz = psb * M[M_ATAN_A + 2] * zz2;
          at2_sum += psb * at2;
          w2_sum += gz * y;
          shift -= gz * M[M_ATAN_W + 2];
          b_re = c22b * ca + s22b * sa;
          b_im = s22b * ca - c22b * sa;
          cos_a = c22b * hr + s22b * hi;
          sin_a += s22b * hr - c22b * hi;
        }
        const double w = is_aux ? mb : 0.0;
        put_columns(stage, {psb, w, w * f, m2rb, m2ib, m3rb, m3ib, cos_a}, lane);
        mma_rows<kRows>(dm, sh.rows + base, stage, lane);
      }
      const double d = mb * mag;  // (d lor / d arg = -lor)
      const double dl = is_aux || is_fall ? 0.0 : d, df = is_fall ? d : 0.0;
      double ub = -2.0 * dl * u * inv_lor;  // from u^2 + g
      if (!clipped) ub -= dl * M[M_RD + 1];
      shift -= ub * T[H_S];
      put_columns(stage, {is_aux || is_fall ? 0.0 : mb * lor, clipped ? 0.0 : -dl * u, -dl * inv_lor,
                          is_fall ? mb * fall : 0.0, -df * over, over > 0.0 ? df * M[M_FALLOFF + 1] : 0.0, ub * y, sin_a},
                  lane);
      sin_a = 0.0;
      mma_ones(dr, stage, lane);
      if (mix) {
        sh.h22r[i] = b_re;
        sh.h22i[i] = b_im;
      }
    } else if (mix) {
      sh.h22r[i] = 0.0;
      sh.h22i[i] = 0.0;
    }
  }
  // --- the sums
  double* sums = sh.modes + m * kXhmModeStride64;
  double* head = sh.sums[m];
  put_products(stage, d1, lane);
  for (int e = lane; e < 24 * 8; e += 32) {
    const int row = e >> 3, col = e & 7;
    const double x = stage[e];
    if (col < 3) {
      if (row < kBasis) sums[M_PHASE + col * kBasis + row] += x;
    } else if (row >= kRowT && row < kRowT + 7) {
      if (col == 3) sums[M_PN_RE + row - kRowT] += x;
      if (col == 4) sums[M_PN_IM + row - kRowT] += x;
      if (col == 5 && row < kRowT + 3) sums[M_PSEUDO + row - kRowT] += x;
    }
  }
  if (lane < 4) {
    head[W_FACTOR + lane] += factor_sum(stage, lane);
  } else if (lane == 4) {
    head[X_T0] += t0_scale * stage[8 * kRowY];
  } else if (lane == 5) {
    head[X_ANCHOR] -= m_over_2 * (stage[8 * kRowT] + stage[8 * kRowT + 1] + stage[8 * kRowT + 2]);
  } else if (lane == 6) {
    head[W_TC] -= kTwoPi * (stage[8 * kRowF] + stage[8 * kRowF + 1] + stage[8 * kRowF + 2]);
  }
  double total[1][2] = {};
  put_columns(stage, {at1_sum, w1_sum, at2_sum, w2_sum, shift, amp0, 0.0, 0.0}, lane);
  mma_ones(total[0], stage, lane);
  put_products(stage, total, lane);
  if (lane < 2) sums[M_ATAN_A + 1 + lane] += stage[2 * lane];
  if (lane == 2 || lane == 3) sums[M_ATAN_W + lane - 1] += stage[2 * (lane - 2) + 1];
  if (lane == 4) sums[M_SHIFT] += stage[4];
  if (lane == 5) head[W_AMP0] += stage[5];
  if (any_inter) {
    // S_j = sum w v^j in lane 4 j; from them d/dC = -H sum_j j c_j S_(j-1)
    // and d/dH = (1 / H) sum_j j c_j S_j
    const double below = __shfl_up_sync(0xffffffffu, di[0], 4);
    const int j = lane >> 2;
    const bool mine = (lane & 3) == 0;
    if (mine) sums[M_INTER + j] += di[0];
    double dc = mine && j > 0 ? j * M[M_INTER + j] * below : 0.0, dh = mine ? j * M[M_INTER + j] * di[0] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dc += __shfl_xor_sync(0xffffffffu, dc, o);
      dh += __shfl_xor_sync(0xffffffffu, dh, o);
    }
    if (lane == 0) {
      sums[M_INTER_C] -= dc * M[M_INTER_H];
      sums[M_INTER_H] += dh / M[M_INTER_H];
    }
  }
  if (any_ring) {
    if (mix) {
      put_products(stage, dm, lane);
      if (lane < 4) {
        const int row = lane == 0 ? kRowF : (lane == 1 ? kRowT : (lane == 2 ? B_M1 : B_M3));
        sums[M_SPH + lane] += stage[8 * row];
      } else if (lane < 8) {
        const int k = lane - 4;
        sums[M_AUX + k] += k == 3 ? stage[8 * kRowF2 + 2] : stage[8 * (kRowT + 3 * k) + 1];
      } else if (lane < 12) {
        sums[M_MIX + lane - 8] += stage[8 * kRowT + lane - 5];
      } else if (lane == 12) {
        head[W_COS] += stage[8 * kRowT + 7];
      }
    }
    total[0][0] = dr[0];
    total[0][1] = dr[1];
    put_products(stage, total, lane);
    if (lane < 3) sums[M_RD + lane] += stage[lane];
    if (lane >= 3 && lane < 6) sums[M_FALLOFF + lane - 3] += stage[lane];
    if (lane == 6) head[W_S] += stage[6];
    if (lane == 7) head[W_SIN] += stage[7];
  }
}

// Stage 3: the (2,2) at the lane's frequency (q, pt; h its value), xb the
// cotangent of its value, direct that without the (3,2)'s part; rows: the
// warp's 32 frequencies of the span's matrix.
__device__ __forceinline__ void reverse_22(AdjShared& sh, const double* rows, int warp, int lane,
                                           const Freq<double>& q, const Point<double>& pt, C2<double> h,
                                           C2<double> xb, C2<double> direct) {
  const double* T = sh.T;
  double* stage = sh.stage[warp];
  double* sums = sh.sums[warp];
  const bool zero = pt.amp == 0.0;  // (above the cutoff nothing depends on the row)
  const double ab = zero ? 0.0 : xb.re * pt.c + xb.im * pt.s;
  const double pb = zero ? 0.0 : xb.im * h.re - xb.re * h.im;
  const double f = q.f, y = f - T[X_SHIFT];
  double d[3][2] = {};
  {
    const bool inspiral = !zero && pt.ra == 0;
    const double w = inspiral ? ab * q.m76 : 0.0, t2 = q.t * q.t, t8 = inspiral ? t2 * t2 * t2 * t2 : 0.0;
    put_columns(stage, {pt.rp == 0 ? pb : 0.0, pt.rp == 1 ? pb : 0.0, pt.rp == 2 ? pb : 0.0, w, w * t8,
                        direct.im * h.re - direct.re * h.im, h.re, h.im}, lane);
    mma_rows<kRows>(d, rows, stage, lane);
  }
  put_products(stage, d, lane);
  // (the order of X_PH_INS, X_PH_INT and X_PH_RD in rows of HM_BASIS)
  using namespace xhm;
  if (lane < 13) {
    constexpr int kIns[13] = {B_M1, B_M2_3, B_M1_3, B_LOG, B_1, B_1_3, B_1_3_LOG, B_2_3, B_F, B_F_LOG, B_4_3, B_5_3,
                              B_F2};
    int row = B_1;
#pragma unroll
    for (int k = 0; k < 13; ++k) row = lane == k ? kIns[k] : row;
    sums[X_PH_INS + lane] += stage[8 * row];
  } else if (lane < 19) {
    const int k = lane - 13;
    const int row = k == 0 ? B_1 : (k == 1 ? B_F : (k == 2 ? B_LOG : (k == 3 ? B_M1 : (k == 4 ? B_M2 : B_M3))));
    sums[X_PH_INT + k] += stage[8 * row + 1];
  } else if (lane < 24) {
    const int k = lane - 19;
    const int row = k == 0 ? B_1 : (k == 1 ? B_F : (k == 2 ? B_2_3 : (k == 3 ? B_M1 : B_M3)));
    sums[X_PH_RD + k] += stage[8 * row + 2];
  } else if (lane == 24) {
    sums[X_T0] += stage[8 * kRowY];
  } else if (lane == 25) {
    sums[X_ANCHOR] -= stage[8 * kRowT] + stage[8 * kRowT + 1] + stage[8 * kRowT + 2];
  } else if (lane == 26) {
    sums[W_TC] -= kTwoPi * stage[8 * kRowF + 5];
  } else if (lane < 31) {
    sums[W_FACTOR22 + lane - 27] += factor_sum(stage, lane - 27);
  }
  if (lane < 10) sums[X_AMP_INS + lane] += lane < 8 ? stage[8 * (kRowT + lane) + 3] : stage[8 * (kRowT + lane - 8) + 4];
  // past the inspiral: the arc tangents, the intermediate and ringdown
  // amplitudes
  const bool past = !zero && (pt.rp > 0 || pt.ra > 0);
  if (!__any_sync(0xffffffffu, past)) return;
  double n = 0.0, w = 0.0, rd_n = 0.0, rd_gr = 0.0, rd_g = 0.0, ub = 0.0, gz = 0.0, shift = 0.0, at = 0.0;
  if (past && pt.rp > 0) {
    gz = pb * T[X_ATAN_A + pt.rp - 1] * pt.zz;
    at = pb * pt.at;
    shift = -gz * T[X_ATAN_W + pt.rp - 1];
  }
  if (past && pt.ra == 1) {
    const double inv = 1.0 / pt.a0;
    n = ab * inv;
    w = -n * pt.amp;
  } else if (past && pt.ra == 2) {
    const double u = pt.a0, g = ab * pt.amp, inv = 1.0 / (u * u + T[X_AMP_RD_G]);
    rd_n = ab * q.m76 * pt.a1;
    rd_gr = -g * u;
    rd_g = -g * inv;
    ub = g * (-T[X_AMP_RD_GR] - 2.0 * u * inv);
    shift -= ub * T[X_AMP_RD_S];
  }
  double d2[2][2] = {};
  put_columns(stage, {w, past && pt.ra == 1 ? w * (f * f) : 0.0, n, rd_n, rd_gr, past ? ub * y : 0.0, rd_g, shift}, lane);
  mma_rows<kRows>(d2, rows, stage, lane);
  double d3[1][2] = {};
  put_columns(stage, {pt.rp == 1 ? at : 0.0, pt.rp == 2 ? at : 0.0, past && pt.rp == 1 ? gz * y : 0.0,
                      past && pt.rp == 2 ? gz * y : 0.0, 0.0, 0.0, 0.0, 0.0}, lane);
  mma_ones(d3[0], stage, lane);
  put_products(stage, d2, lane);
  if (lane < 5) {
    // d_j: w f^j, j = 0..2 from column 0, j = 3, 4 from column 1 (w f^2)
    const int row = lane == 0 ? kRowT : ((lane & 1) ? kRowF : kRowF2);
    sums[X_AMP_INT_D + lane] += stage[8 * row + (lane > 2 ? 1 : 0)];
  } else if (lane < 11) {
    constexpr int kSlot[6] = {X_AMP_INT_N, X_AMP_RD_N, X_AMP_RD_GR, X_AMP_RD_S, X_AMP_RD_G, X_SHIFT};
    int slot = X_AMP_INT_N;
#pragma unroll
    for (int k = 0; k < 6; ++k) slot = lane - 5 == k ? kSlot[k] : slot;
    sums[slot] += stage[8 * kRowT + lane - 3];
  }
  put_products(stage, d3, lane);
  if (lane < 4) sums[X_ATAN_A + lane] += stage[lane];
}
static_assert(X_ATAN_W == X_ATAN_A + 2, "the arc tangents' four slots are contiguous");

__global__ void __launch_bounds__(kXhmBlock, 4)
    k_xhm_adj(const double* __restrict__ table, const double* __restrict__ dtable, const double* __restrict__ freqs,
              const int64_t* __restrict__ offsets, int64_t B, int64_t n, const double* __restrict__ t_c,
              const C2<double>* __restrict__ g_p, const C2<double>* __restrict__ g_c, double* __restrict__ grad) {
  using namespace xhm;
  constexpr int kStride = kXhmStride64;
  __shared__ AdjShared sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t b = blockIdx.y; b < B; b += gridDim.y) {
    __syncthreads();  // (the row and the sums are rewritten)
    for (int k = threadIdx.x; k < kStride; k += kXhmBlock) sh.T[k] = table[b * kStride + k];
    for (int k = threadIdx.x; k < kModes * kXhmModeStride64; k += kXhmBlock) sh.modes[k] = 0.0;
    for (int k = threadIdx.x; k < kAdjWarps * kTableStride; k += kXhmBlock) (&sh.sums[0][0])[k] = 0.0;
    __syncthreads();
    const int64_t lo = offsets != nullptr ? min(max(offsets[b], int64_t(0)), n) : 0;
    const int64_t hi = offsets != nullptr ? min(max(offsets[b + 1], lo), n) : n;
    const int64_t row = offsets != nullptr ? 0 : b * n;
    for (int64_t j0 = lo + static_cast<int64_t>(blockIdx.x) * kAdjSpan; j0 < hi;
         j0 += static_cast<int64_t>(gridDim.x) * kAdjSpan) {
      const int count = static_cast<int>(min(static_cast<int64_t>(kAdjSpan), hi - j0));
      const int i = threadIdx.x;
      const bool in = i < count;
      const int64_t j = j0 + (in ? i : 0);
      const Freq<double> p = freq_powers(freqs[j]);
      const Point<double> p22 = xas_point<double>(sh.T, p, 0.0);
      const C2<double> h22{p22.amp * p22.c, p22.amp * p22.s};
      C2<double> gp{0.0, 0.0}, gc{0.0, 0.0};
      if (in) {
        gp = g_p[row + j];
        gc = g_c[row + j];
      }
      if (t_c != nullptr) {
        double c, s;
        tc_factor(p.f, t_c[b], c, s);
        gp = C2<double>{gp.re * c + gp.im * s, gp.im * c - gp.re * s};
        gc = C2<double>{gc.re * c + gc.im * s, gc.im * c - gc.re * s};
      }
      double* q = sh.rows + i;
      const double t2 = p.t * p.t, mt1 = t2 * p.m1, m2 = p.m1 * p.m1, ff = p.f * p.f, ft = p.f * p.t;
      q[B_M3 * kRowStride] = row_entry(m2 * p.m1);
      q[B_M2 * kRowStride] = row_entry(m2);
      q[B_M4_3 * kRowStride] = row_entry(p.m1 * mt1);
      q[B_M1 * kRowStride] = row_entry(p.m1);
      q[B_M2_3 * kRowStride] = row_entry(mt1 * mt1);
      q[B_M1_3 * kRowStride] = row_entry(mt1);
      q[B_1 * kRowStride] = 1.0;
      q[B_1_3 * kRowStride] = row_entry(p.t);
      q[B_2_3 * kRowStride] = row_entry(t2);
      q[B_F * kRowStride] = row_entry(p.f);
      q[B_4_3 * kRowStride] = row_entry(ft);
      q[B_5_3 * kRowStride] = row_entry(p.f * t2);
      q[B_F2 * kRowStride] = row_entry(ff);
      q[B_7_3 * kRowStride] = row_entry(ff * p.t);
      q[B_LOG * kRowStride] = row_entry(p.lf);
      q[B_1_3_LOG * kRowStride] = row_entry(p.t * p.lf);
      q[B_F_LOG * kRowStride] = row_entry(p.f * p.lf);
      q[B_4_3_LOG * kRowStride] = row_entry(ft * p.lf);
      q[kRowY * kRowStride] = row_entry(p.y);
      q[kRowG * kRowStride] = gp.re;
      q[(kRowG + 1) * kRowStride] = gp.im;
      q[(kRowG + 2) * kRowStride] = gc.re;
      q[(kRowG + 3) * kRowStride] = gc.im;
      sh.m76[i] = row_m76(p.f, p.y, p.m76);
      sh.h22r[i] = h22.re;
      sh.h22i[i] = h22.im;
      __syncthreads();
      mode_reverse(sh, warp, count, lane);
      __syncthreads();
      if (32 * warp < count) {
        const C2<double> direct = mode_cotangent(sh.T + H_FACTORS, gp.re, gp.im, gc.re, gc.im);
        const C2<double> xb{direct.re + sh.h22r[i], direct.im + sh.h22i[i]};
        reverse_22(sh, sh.rows + 32 * warp, warp, lane, p, p22, h22, xb, direct);
      }
      __syncthreads();  // (the rows are rewritten)
    }
    // the whole row's sums in place of the row, then their product with
    // dtable: thread (r, d) takes the slots r + 16 i of direction d (a slot
    // that nothing touched adds nothing, whatever its tangent)
    double tc = 0.0;
    for (int k = threadIdx.x; k < kStride; k += kXhmBlock) {
      double s = 0.0;
      if (k >= H_MODES) {
        s = sh.modes[k - H_MODES];
      } else if (k >= H_FACTORS + 4 && k < H_FACTORS + kHeadFactors) {
        s = sh.sums[(k - H_FACTORS) / 4 - 1][W_FACTOR + (k & 3)];
      } else {
        const int w = k < X_USED ? k
                                 : (k >= H_FACTORS && k < H_FACTORS + 4
                                        ? W_FACTOR22 + k - H_FACTORS
                                        : (k == H_AMP0 ? W_AMP0
                                                       : (k == H_S ? W_S
                                                                   : (k == H_COS_A ? W_COS
                                                                                   : (k == H_SIN_A ? W_SIN : -1)))));
        if (w >= 0) {
          for (int v = 0; v < kAdjWarps; ++v) s += sh.sums[v][w];
        }
      }
      sh.T[k] = s;
    }
    if (threadIdx.x == 0) {
      for (int v = 0; v < kAdjWarps; ++v) tc += sh.sums[v][W_TC];
    }
    __syncthreads();
    const int d = threadIdx.x & 7;
    double g = 0.0;
    for (int k = threadIdx.x >> 3; k < kStride; k += kXhmBlock / 8) {
      const double s = sh.T[k];
      if (s != 0.0) g += s * dtable[(b * kStride + k) * 8 + d];
    }
    g += __shfl_xor_sync(0xffffffffu, g, 8);
    g += __shfl_xor_sync(0xffffffffu, g, 16);
    if (lane < 8) sh.m76[8 * warp + lane] = g;
    __syncthreads();
    if (threadIdx.x < 8) {
      double total = 0.0;
      for (int w = 0; w < kAdjWarps; ++w) total += sh.m76[8 * w + threadIdx.x];
      atomicAdd(&grad[b * 9 + threadIdx.x], total);
    }
    if (threadIdx.x == 0) atomicAdd(&grad[b * 9 + 8], tc);
  }
}
static_assert((H_FACTORS & 3) == 0, "factor i of mode k at H_FACTORS + 4 k + i");

// IMRPhenomXHM's derivative with respect to the grid (the reference's
// drop-in differentiates its model with respect to the frequencies,
// src/waveformx/torch.py:87-91; models/xhm/model.py:40 takes the set-up's
// first frequency without a derivative): the FP64 evaluation of k_xhm
// with the table's tangents zero and the frequency's powers carrying d/df
// (freq_powers_dual), e^(-2 pi i f t_c) differentiated in f too, contracted
// with the cotangents: d[b][j] = Re(conj(g+) dh+/df + conj(gx) dhx/df).
// Blocks (run of kXhmBlock frequencies, group): on a shared grid a group is
// kXhmBinariesPerBlock consecutive binaries, whose terms each thread sums
// before one atomic per element and group into grad_f (n, zeroed
// beforehand); on a ragged grid a group is one binary, whose elements are
// its own (stored). The offsets are clamped to [0, n].
__global__ void __launch_bounds__(kXhmBlock, 4)
    k_xhm_grid_vjp(const double* __restrict__ table, const double* __restrict__ freqs,
                   const int64_t* __restrict__ offsets, int64_t B, int64_t n, const double* __restrict__ t_c,
                   const C2<double>* __restrict__ g_p, const C2<double>* __restrict__ g_c,
                   double* __restrict__ grad_f) {
  constexpr int kStride = kXhmStride64;
  // (Dual has a constructor: raw storage, every entry written before read)
  __shared__ __align__(16) double t_raw[2 * kStride];
  __shared__ __align__(16) double t0_raw[2 * 4];
  Dual* T = reinterpret_cast<Dual*>(t_raw);
  Dual* t0_lm = reinterpret_cast<Dual*>(t0_raw);
  const bool ragged = offsets != nullptr;
  const int64_t group = ragged ? 1 : kXhmBinariesPerBlock;
  const int64_t groups = (B + group - 1) / group;
  for (int64_t g = blockIdx.y; g < groups; g += gridDim.y) {
    const int64_t b0 = g * group, b1 = min(b0 + group, B);
    const int64_t lo = ragged ? min(max(offsets[b0], int64_t(0)), n) : 0;
    const int64_t hi = ragged ? min(max(offsets[b0 + 1], lo), n) : n;
    for (int64_t j0 = static_cast<int64_t>(blockIdx.x) * blockDim.x; j0 < hi - lo;
         j0 += static_cast<int64_t>(gridDim.x) * blockDim.x) {
      const int64_t j = lo + j0 + threadIdx.x;
      const bool in = j < hi;
      const double f = in ? freqs[j] : 0.0;
      double acc = 0.0;
      for (int64_t b = b0; b < b1; ++b) {
        __syncthreads();  // (T is rewritten)
        for (int k = threadIdx.x; k < kStride; k += blockDim.x) T[k] = Dual(table[b * kStride + k], 0.0);
        if (threadIdx.x < 4) {
          const int m = threadIdx.x;
          const double emm = m == 0 ? 1.0 : (m == 1 ? 3.0 : (m == 2 ? 2.0 : 4.0));
          t0_lm[m] = Dual(pow(emm * 0.5, 8.0 / 3.0) * table[b * kStride + X_T0], 0.0);
        }
        __syncthreads();
        if (!in) continue;
        const Freq<Dual> q = freq_powers_dual(f);
        // e^(-2 pi i f t_c) = (c, s) and its derivative 2 pi t_c (s, -c)
        double c = 1.0, sn = 0.0;
        const double tcb = t_c != nullptr ? t_c[b] : 0.0;
        if (t_c != nullptr) tc_factor(f, tcb, c, sn);
        const double w = kTwoPi * tcb;
        C2<Dual> sp, sc;
        xhm_dual_sum(T, t0_lm, q, Dual(c, w * sn), Dual(sn, -w * c), sp, sc);
        const int64_t e = ragged ? j : b * n + j;
        const C2<double> gp = g_p[e], gc = g_c[e];
        acc += gp.re * sp.re.d + gp.im * sp.im.d + gc.re * sc.re.d + gc.im * sc.im.d;
      }
      if (!in) continue;
      if (ragged) {
        grad_f[j] = acc;
      } else {
        atomicAdd(&grad_f[j], acc);
      }
    }
  }
}

int launched() {
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? 0 : static_cast<int>(err);
}

}  // namespace

int xhm_grid_vjp(const double* table, const double* freqs, const int64_t* offsets, int64_t B, int64_t n,
                 const double* t_c, const void* cot_hp, const void* cot_hc, double* grad_f, cudaStream_t s) {
  // (a run of frequencies per block; on a ragged grid enough runs for the
  // rows' mean length, longer rows looping in their blocks)
  const int64_t span = offsets != nullptr ? (n + B - 1) / B : n;
  const int64_t runs = (span + kXhmBlock - 1) / kXhmBlock;
  const int64_t groups = offsets != nullptr ? B : (B + kXhmBinariesPerBlock - 1) / kXhmBinariesPerBlock;
  const dim3 grid(static_cast<unsigned>(runs < 1024 ? runs : 1024),
                  static_cast<unsigned>(groups < 65535 ? groups : 65535));
  k_xhm_grid_vjp<<<grid, kXhmBlock, 0, s>>>(table, freqs, offsets, B, n, t_c,
                                            static_cast<const C2<double>*>(cot_hp),
                                            static_cast<const C2<double>*>(cot_hc), grad_f);
  return launched();
}

}  // namespace wfx

using namespace wfx;

extern "C" {

int wfx_xhm_polarizations(int precision, const void* table, const void* freqs, const int64_t* offsets, int64_t B,
                          int64_t n, int64_t max_len, const void* t_c, void* hp, void* hc, void* modes,
                          wfx_stream_t stream) {
  if (table == nullptr || freqs == nullptr || hp == nullptr || hc == nullptr || B <= 0 || n <= 0) return WFX_EINVAL;
  if ((reinterpret_cast<uintptr_t>(table) & 15u) != 0) return WFX_EINVAL;
  if (offsets != nullptr && (modes != nullptr || max_len <= 0)) return WFX_EINVAL;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int64_t span = offsets != nullptr ? max_len : n;
  const int64_t runs = (span + kXhmBlock - 1) / kXhmBlock;
  // (a shared grid: kXhmBinariesPerBlock binaries a block, which share the
  // frequencies' powers; a ragged one: one binary a block)
  const int64_t rows = offsets != nullptr ? B : (B + kXhmBinariesPerBlock - 1) / kXhmBinariesPerBlock;
  const dim3 grid(static_cast<unsigned>(runs < 4096 ? runs : 4096), static_cast<unsigned>(rows < 65535 ? rows : 65535));
  if (precision == WFX_FP32) {
    k_xhm<float><<<grid, kXhmBlock, 0, s>>>(static_cast<const float*>(table), static_cast<const float*>(freqs), offsets,
                                             B, n,
                                             static_cast<const float*>(t_c), static_cast<C2<float>*>(hp),
                                             static_cast<C2<float>*>(hc), static_cast<C2<float>*>(modes));
  } else if (precision == WFX_FP64) {
    k_xhm<double><<<grid, kXhmBlock, 0, s>>>(static_cast<const double*>(table), static_cast<const double*>(freqs),
                                              offsets, B, n, static_cast<const double*>(t_c), static_cast<C2<double>*>(hp),
                                              static_cast<C2<double>*>(hc), static_cast<C2<double>*>(modes));
  } else {
    return WFX_EINVAL;
  }
  return launched();
}

int wfx_xhm_vjp(const double* table, const double* dtable, const double* freqs, const int64_t* offsets, int64_t B,
                int64_t n, int64_t max_len, const double* t_c, const void* cot_hp, const void* cot_hc, double* grad,
                wfx_stream_t stream) {
  if (table == nullptr || dtable == nullptr || freqs == nullptr || cot_hp == nullptr || cot_hc == nullptr ||
      grad == nullptr || B <= 0 || n <= 0 || (offsets != nullptr && max_len <= 0))
    return WFX_EINVAL;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const cudaError_t rc = cudaMemsetAsync(grad, 0, sizeof(double) * 9 * static_cast<size_t>(B), s);
  if (rc != cudaSuccess) return static_cast<int>(rc);
  // (blocks a binary: one span each while the batch is short of kAdjBlocks
  // blocks, then several spans a block, which cost it one contraction)
  const int64_t spans = ((offsets != nullptr ? max_len : n) + kAdjSpan - 1) / kAdjSpan;
  const int64_t each = B * spans > kAdjBlocks ? B * spans / kAdjBlocks : 1;
  const int64_t runs = (spans + each - 1) / each;
  const dim3 grid(static_cast<unsigned>(runs < 65535 ? runs : 65535), static_cast<unsigned>(B < 65535 ? B : 65535));
  k_xhm_adj<<<grid, kXhmBlock, 0, s>>>(table, dtable, freqs, offsets, B, n, t_c, static_cast<const C2<double>*>(cot_hp),
                                       static_cast<const C2<double>*>(cot_hc), grad);
  return launched();
}

}  // extern "C"
