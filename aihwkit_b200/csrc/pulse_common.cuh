// Pieces of the pulsed update that its kernels share: update management, pulse trains and the
// device rules (one pulse with the clip behind it).
#pragma once

#include "mvm_common.cuh"
#include "tile.h"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

namespace ab200 {

__device__ __forceinline__ float blockMax(float v, float *sh) {
  for (int o = 16; o > 0; o >>= 1) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    sh[w] = v;
  }
  __syncthreads();
  float r = 0.0f;
  for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
    r = fmaxf(r, sh[i]);
  }
  __syncthreads();
  return r;
}

// calculateBlAB + performUpdateManagement, fp32 with the reference's association
// (rpu_pulsed_meta_parameter.cpp:153-236). BL == 0 means "no update for this sample".
__device__ __forceinline__ void
blAB(const UpEff &up, float lr, float dw_min, float xm, float dm, int &BL, float &A, float &B) {
  if (lr == 0.0f) {
    BL = 0;
    A = B = 0.0f;
    return;
  }
  if (up.fixed_bl || up.update_bl_management) {
    BL = up.desired_bl;
    A = __fsqrt_rn(__fdiv_rn(lr, __fmul_rn(dw_min, (float)BL)));
    B = A;
  } else {
    if (__fmul_rn(dw_min, (float)up.desired_bl) < lr) {
      A = B = 1.0f;
      BL = max((int)ceilf(__fdiv_rn(lr, dw_min)), 1);
    } else {
      BL = up.desired_bl;
      A = __fsqrt_rn(__fdiv_rn(lr, __fmul_rn(dw_min, (float)BL)));
      B = A;
    }
  }
  if (up.update_bl_management || up.update_management) {
    if (xm == 0.0f || dm == 0.0f) {
      BL = 0;
      A = B = 1.0f;
      return;
    }
    float x_val = xm;
    float d_val = __fmul_rn(up.um_grad_scale, dm);
    float k_val = __fdiv_rn(__fmul_rn(__fmul_rn(lr, x_val), d_val), dw_min);
    if (up.update_bl_management) {
      BL = (int)ceilf(k_val);
      if (BL > up.desired_bl) {
        BL = up.desired_bl;
      }
      A = __fsqrt_rn(__fdiv_rn(lr, __fmul_rn(dw_min, (float)BL)));
      B = A;
    }
    if (up.update_management) {
      if (k_val > (float)up.desired_bl) {
        d_val = __fmul_rn(d_val, __fdiv_rn((float)up.desired_bl, k_val));
      }
      A = __fmul_rn(A, __fsqrt_rn(__fdiv_rn(x_val, d_val)));
      B = __fmul_rn(B, __fsqrt_rn(__fdiv_rn(d_val, x_val)));
    }
  }
}

// The longest train that blAB returns for any sample of an update with these settings: without a fixed length
// and without update BL management a train has ceil(lr / dw_min) slots where that is more than desired_bl.
static inline int longestTrain(const UpEff &up, float lr, float dw_min) {
  if (up.fixed_bl || up.update_bl_management || !(dw_min * (float)up.desired_bl < lr)) {
    return up.desired_bl;
  }
  const float bl = std::ceil(lr / dw_min);
  return bl < 2147483648.0f ? std::max((int)bl, 1) : INT_MAX;
}

// Pulses of an implicit pair of lines with c = d * BL * x: |c| to the nearest integer, ties to even; none for
// NaN. Up to kShortTrain slots (|c| <= BL) by adding 2^23, whose neighbours are 1 apart, which keeps the
// count off the conversion pipe.
constexpr int kShortTrain = 1 << 20;
__host__ __device__ inline int implicitPulses(float c, bool short_train) {
  const float a = fmaxf(fabsf(c), 0.0f);
#ifdef __CUDA_ARCH__
  return short_train ? __float_as_int(__fadd_rn(a, 8388608.0f)) - 0x4B000000 : __float2int_rn(a);
#else
  if (short_train) {
    const float v = a + 8388608.0f;
    int bits;
    std::memcpy(&bits, &v, sizeof(bits));
    return bits - 0x4B000000;
  }
  return a < 2147483648.0f ? (int)std::nearbyint(a) : INT_MAX;
#endif
}

// Stream of the device noise of a launch of the staged kernel. A batch in which transfers fall is applied in ranges of
// its rows, a launch each, under one call counter: the first row keeps their draws apart (a whole batch starts at
// row 0).
__device__ __forceinline__ uint32_t deviceNoiseTag(const UpdateProblem &p) {
  return TAG_DEVICE + (uint32_t)p.s_begin;
}

// Place in a warp's pool of `kNoisePool` Gaussians from which lane `lane` takes, or would take, its next one:
// `pos` are gone, `takers` take one each and fit. All lanes look, those past the last taker just behind it: one
// place behind the end when the pool is used up, which a row of the pool has.
constexpr int kNoisePool = 256, kNoisePoolRow = kNoisePool + 1;
__host__ __device__ inline int noisePoolSlot(int pos, uint32_t takers, int lane) {
  const uint32_t before = takers & ((1u << lane) - 1u);
#ifdef __CUDA_ARCH__
  return pos + __popc(before);
#else
  return pos + __builtin_popcount(before);
#endif
}

// A draw u of 16 bits gives a pulse when u + 0.5 < 65536 pp; as a comparison u < threshold of integers,
// which keeps the draws off the conversion pipe.
__device__ __forceinline__ int pulseThreshold(float pp) {
  return __float2int_ru(__fadd_rn(__fmul_rn(pp, 65536.0f), -0.5f));
}

// One stochastic pulse train (generateCounts, sparse_bit_line_maker.cpp:200-238): BL Bernoulli
// draws with probability pp; each draw compares pp against a 16-bit uniform, 8 draws per
// Philox call. (A bit-serial comparison of all slots at once - one random word per bit of pp until
// every slot is decided - needs fewer calls per lane but as many per warp, and measured slower.)
__device__ __forceinline__ uint32_t
pulseTrain(float pp, int BL, int seg, PhiloxKey key, uint32_t line, uint32_t sample, uint32_t call,
           uint32_t tag) {
  // slots [seg * 31, min(BL, seg * 31 + 31)) of the train, as bits 1.. of one word
  const int k0 = seg * kPulseSegSlots;
  const int nk = min(BL - k0, kPulseSegSlots);
  const int thr = pulseThreshold(pp);
  uint32_t bits = 0;
  int k = 0;
  for (int q = 0; q * 8 < nk; q++) {
    uint32_t r[4];
    philox4x32<7>(line, sample, call, tag + (uint32_t)(seg * 4 + q), key, r);
#pragma unroll
    for (int h = 0; h < 8; h++) {
      const int u16 = (int)((r[h >> 1] >> ((h & 1) * 16)) & 0xFFFFu);
      if (k < nk && u16 < thr) {
        bits |= 1u << (k + 1);
      }
      k++;
    }
  }
  return bits;
}

// getDiscretizedValue of a pulse probability (src/rpucuda/utility_functions.h:186-193): to the
// nearest multiple of `res`, or - with sto_round - up or down at random in proportion to the
// remainder; the uniform of a line is a function of (line, sample, call).
__device__ __forceinline__ float
pulseProb(const UpdateProblem &p, float v, float res, uint32_t line, uint32_t sample, uint32_t tag) {
  if (!p.up.sto_round || !(res > 0.0f)) {
    return discretize(v, res);
  }
  uint32_t r[4];
  philox4x32<7>(line, sample, p.call, tag ^ 0x08000000u, p.key, r);
  return __fmul_rn(rintf(__fadd_rn(__fdiv_rn(v, res), __fadd_rn(u01(r[0]), -0.5f))), res);
}

// ---------------------------------------------------------------------------------------------
// device rules: one pulse, clipped immediately. `down` = weight decreases.
// par4 = {scale_up, scale_down, max_bound, min_bound}
// ---------------------------------------------------------------------------------------------
template <int KIND>
__device__ __forceinline__ float pulseOnce(float w, bool down, const float4 &q, const float2 &e,
                                           float xi, int mult_noise, const float4 &es0,
                                           const float4 &es1, const float *pw = nullptr,
                                           int pw_n = 0) {
  if (KIND == AB200_DEVICE_PIECEWISE_STEP) {
    // PiecewiseStepRPUDevice update_once (rpu_piecewisestep_device.cpp:30-80): the step factor is
    // interpolated linearly between pw_n nodes spread evenly over [min_bound, max_bound];
    // pw[0..pw_n) are the up factors, pw[pw_n..2 pw_n) the down factors
    const float *tab = down ? pw + pw_n : pw;
    const int n_sec = pw_n - 1;
    float f;
    if (n_sec <= 0 || q.z <= q.w) {
      f = __ldg(tab);
    } else {
      const float ws = fmaxf(
          __fmul_rn(__fdiv_rn(__fsub_rn(w, q.w), __fsub_rn(q.z, q.w)), (float)n_sec), 0.0f);
      const int idx = min((int)floorf(ws), n_sec - 1);
      const float t = fminf(__fsub_rn(ws, (float)idx), 1.0f);
      const float t1 = __fsub_rn(1.0f, t);
      f = __fadd_rn(__fmul_rn(t1, __ldg(tab + idx)), __fmul_rn(t, __ldg(tab + idx + 1)));
    }
    const float step = __fmul_rn(__fmul_rn(down ? q.y : q.x, f), __fadd_rn(1.0f, xi));
    w = down ? __fsub_rn(w, step) : __fadd_rn(w, step);
    w = fmaxf(w, q.w);
    w = fminf(w, q.z);
    return w;
  } else if (KIND == AB200_DEVICE_EXP_STEP) {
    // ExpStepRPUDevice update_once / update_once_complex_noise (rpu_expstep_device.cpp:18-100):
    // z = 2 w / (max - min) * a + b;  step = scale * max(1 - A exp(+-gamma z), 0)
    // es0 = {a, b, A_up, A_down}, es1 = {gamma_up, gamma_down, std_add, std_slope}; xi = std * N
    const float b_diff = __fsub_rn(q.z, q.w);
    if (!(b_diff > 0.0f)) {
      return w;
    }
    const float z = __fadd_rn(__fmul_rn(__fdiv_rn(__fmul_rn(2.0f, w), b_diff), es0.x), es0.y);
    const float y = down ? fmaxf(__fsub_rn(1.0f, __fmul_rn(es0.w, expf(__fmul_rn(es1.y, -z)))), 0.0f)
                         : fmaxf(__fsub_rn(1.0f, __fmul_rn(es0.z, expf(__fmul_rn(es1.x, z)))), 0.0f);
    if (es1.z != 0.0f || es1.w != 0.0f) {
      const float dw = down ? -__fmul_rn(y, q.y) : __fmul_rn(y, q.x);
      const float spread =
          __fadd_rn(__fadd_rn(fabsf(dw), es1.z), __fmul_rn(es1.w, fabsf(w)));
      w = __fadd_rn(w, __fadd_rn(dw, __fmul_rn(spread, xi)));
    } else {
      const float step = __fmul_rn(__fmul_rn(y, __fadd_rn(1.0f, xi)), down ? q.y : q.x);
      w = down ? __fsub_rn(w, step) : __fadd_rn(w, step);
    }
    w = fminf(w, q.z);
    w = fmaxf(w, q.w);
    return w;
  } else if (KIND == AB200_DEVICE_POW_STEP) {
    // PowStepRPUDevice update_once (rpu_powstep_device.cpp:91-121): the step shrinks with a power
    // of the distance to the bound, e = {gamma_up, gamma_down}
    const float range = __fsub_rn(q.z, q.w);
    if (range == 0.0f) {
      return w;
    }
    if (down) {
      const float f = powf(__fdiv_rn(__fsub_rn(w, q.w), range), e.y);
      w = __fsub_rn(w, __fmul_rn(__fmul_rn(q.y, f), __fadd_rn(1.0f, xi)));
    } else {
      const float f = powf(__fdiv_rn(__fsub_rn(q.z, w), range), e.x);
      w = __fadd_rn(w, __fmul_rn(__fmul_rn(q.x, f), __fadd_rn(1.0f, xi)));
    }
    w = fmaxf(w, q.w);
    w = fminf(w, q.z);
    return w;
  } else if (KIND == AB200_DEVICE_CONSTANT_STEP) {
    float dw = __fmul_rn(__fadd_rn(1.0f, xi), down ? q.y : q.x);
    w = down ? __fsub_rn(w, dw) : __fadd_rn(w, dw);
    w = fminf(w, q.z);
    w = fmaxf(w, q.w);
    return w;
  } else if (KIND == AB200_DEVICE_LINEAR_STEP) {
    float slope = down ? e.y : e.x;
    float sc = down ? q.y : q.x;
    float dw;
    if (mult_noise) {
      dw = __fmul_rn(__fadd_rn(__fmul_rn(slope, w), sc), __fadd_rn(1.0f, xi));
    } else {
      dw = __fadd_rn(__fmul_rn(slope, w), __fmul_rn(sc, __fadd_rn(1.0f, xi)));
    }
    w = down ? __fsub_rn(w, dw) : __fadd_rn(w, dw);
    w = fmaxf(w, q.w);
    w = fminf(w, q.z);
    return w;
  } else { // SOFT_BOUNDS_REFERENCE
    float ref = e.x;
    w = __fadd_rn(w, ref);
    float bound = down ? q.w : q.z;
    bool ok = down ? (bound < 0.0f) : (bound > 0.0f);
    float a = ok ? __fdiv_rn(w, bound) : 0.0f;
    float sc = down ? q.y : q.x;
    float dw;
    if (mult_noise) {
      dw = __fmul_rn(__fmul_rn(sc, __fsub_rn(1.0f, a)), __fadd_rn(1.0f, xi));
    } else {
      dw = __fmul_rn(sc, __fadd_rn(__fsub_rn(1.0f, a), xi));
    }
    w = down ? __fsub_rn(w, dw) : __fadd_rn(w, dw);
    w = fmaxf(w, q.w);
    w = fminf(w, q.z);
    return __fsub_rn(w, ref);
  }
}

// What a pulse needs of its element, by direction, with the sign of the direction in it: w += signed
// step instead of w -= step (round-to-nearest is symmetric, so the bits are those of pulseOnce).
//
// SoftBoundsReference divides the weight by its bound in every pulse. Where the bounds are ordinary numbers the
// quotient comes from their reciprocals, taken once, and two residual corrections q += (w - b q) y, which
// give the correctly rounded quotient (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990: y the rounded reciprocal; the first correction leaves q within an ulp, the second
// rounds it correctly). Residuals below the normal range only occur for quotients that 1 - q does not see.
template <int KIND> struct PulseStep {
  float4 q;
  float2 e;
  float scale_dn, slope_dn;
  bool by_reciprocal = false; // the same for a whole warp
  __device__ __forceinline__ void set(const float4 &q_, const float2 &e_) {
    q = q_;
    e = e_;
    scale_dn = -q.y;
    slope_dn = -e.y;
  }
  // for all lanes of a warp together; `used` = the lane owns a weight
  __device__ __forceinline__ void prepare(float w, bool used) {
    if (KIND == AB200_DEVICE_SOFT_BOUNDS_REFERENCE) {
      const float lo = 8.7e-19f, hi = 1.15e18f; // 2^-60, 2^60
      by_reciprocal = __all_sync(0xffffffffu, !used || (q.z > lo && q.z < hi && q.w < -lo && q.w > -hi &&
                                                        fabsf(w) < hi && fabsf(e.x) < hi));
      e.y = __fdiv_rn(1.0f, q.z); // (the rule uses e.x alone)
      slope_dn = __fdiv_rn(1.0f, q.w);
    }
  }
  // the noise of a pulse enters the rule as 1 + xi; kept in that form from the draw on
  static constexpr bool kOnePlus =
      KIND == AB200_DEVICE_CONSTANT_STEP || KIND == AB200_DEVICE_LINEAR_STEP;
  __device__ __forceinline__ float apply(const UpdateProblem &p, float w, bool down, float xi) const {
    return apply(p, w, down, xi, p.mult_noise != 0);
  }
  __device__ __forceinline__ float apply(const UpdateProblem &p, float w, bool down, float xi, bool mult) const {
    if (KIND == AB200_DEVICE_CONSTANT_STEP) {
      w = __fadd_rn(w, __fmul_rn(xi, down ? scale_dn : q.x));
      return fmaxf(fminf(w, q.z), q.w);
    } else if (KIND == AB200_DEVICE_LINEAR_STEP) {
      const float sc = down ? scale_dn : q.x, sl = __fmul_rn(down ? slope_dn : e.x, w);
      const float dw = mult ? __fmul_rn(__fadd_rn(sl, sc), xi) : __fadd_rn(sl, __fmul_rn(sc, xi));
      return fminf(fmaxf(__fadd_rn(w, dw), q.w), q.z);
    } else if (KIND == AB200_DEVICE_SOFT_BOUNDS_REFERENCE && by_reciprocal) {
      const float bound = down ? q.w : q.z, y = down ? slope_dn : e.y, sc = down ? scale_dn : q.x;
      w = __fadd_rn(w, e.x);
      float a = __fmul_rn(w, y);
      a = __fmaf_rn(__fmaf_rn(-bound, a, w), y, a);
      a = __fmaf_rn(__fmaf_rn(-bound, a, w), y, a);
      const float rest = __fsub_rn(1.0f, a);
      const float dw = mult ? __fmul_rn(__fmul_rn(sc, rest), __fadd_rn(1.0f, xi)) : __fmul_rn(sc, __fadd_rn(rest, xi));
      w = fminf(fmaxf(__fadd_rn(w, dw), q.w), q.z);
      return __fsub_rn(w, e.x);
    } else {
      return pulseOnce<KIND>(w, down, q, e, xi, p.mult_noise, p.es0, p.es1, p.pw, p.pw_n);
    }
  }
};

// the same problem in rows of pulse words: a sample has nseg of them
static inline UpdateProblem inRows(const UpdateProblem &p0) {
  UpdateProblem p = p0;
  const int nseg = p0.nseg > 0 ? p0.nseg : 1;
  p.m = p0.m * nseg;
  p.s_begin = p0.s_begin * nseg;
  p.s_end = p0.s_end * nseg;
  p.nseg = 1;
  return p;
}

} // namespace ab200
