// Pulsed weight update.
//
//   pulsePrepareKernel   per sample: |x|max, |d|max -> BL, A, B (update management), then the pulse
//                        train of every x- and d-line packed into one 32-bit word (bit 0 = sign,
//                        bits 1..BL = pulses), or the implicit pulse values for the deterministic
//                        pulse type.
//   pulsedUpdateKernel   per weight element: coincidences by AND + popc over the batch, device
//                        rule applied pulse by pulse in place; weights and per-element parameters
//                        are read with coalesced 128-bit loads, once per call.
//
// Reference semantics restated here:
//   update management      src/rpucuda/rpu_pulsed_meta_parameter.cpp:153-236
//   stochastic trains      src/rpucuda/sparse_bit_line_maker.cpp:200-238, 288-353
//   implicit pulses        src/rpucuda/dense_bit_line_maker.cpp:210-264
//   coincidence loop       src/rpucuda/rpu_weight_updater.cpp:236-291
//   ConstantStep           src/rpucuda/rpu_constantstep_device.cpp:28-78
//   LinearStep/SoftBounds  src/rpucuda/rpu_linearstep_device.cpp:113-164
//   SoftBoundsReference    src/rpucuda/rpu_softbounds_reference_device.cpp:107-175
#include "pulse_common.cuh"

namespace ab200 {

__global__ void __launch_bounds__(256) pulsePrepareKernel(UpdateProblem p) {
  pdlEnter();
  __shared__ float sh[8];
  __shared__ float s_A, s_B;
  __shared__ int s_BL;
  const int s = blockIdx.x;
  const float *xr = p.x + (long long)s * p.x_ss;
  const float *dr = p.d + (long long)s * p.d_ss;
  const bool need_max = p.up.update_management || p.up.update_bl_management;
  // samples gathered from whole images (indexed convolution interface) or plain rows
  const bool gathered = p.gather.idx != nullptr;
  auto xValue = [&](int j) -> float {
    if (gathered) {
      return gatherRowElement(p.gather, p.x, s, j);
    }
    return j < p.x_real ? xr[(long long)j * p.x_fs] : 1.0f;
  };
  float xm = 0.0f, dm = 0.0f;
  if (need_max) {
    for (int j = threadIdx.x; j < p.x_size; j += blockDim.x) {
      xm = fmaxf(xm, fabsf(xValue(j)));
    }
    for (int i = threadIdx.x; i < p.d_size; i += blockDim.x) {
      dm = fmaxf(dm, fabsf(dr[(long long)i * p.d_fs]));
    }
    xm = blockMax(xm, sh);
    dm = blockMax(dm, sh);
  }
  if (threadIdx.x == 0) {
    int BL;
    float A, B;
    blAB(p.up, p.lr, p.dw_min, xm, dm, BL, A, B);
    s_BL = BL;
    s_A = A;
    s_B = B;
  }
  __syncthreads();
  const int BL = s_BL;
  const float A = s_A, B = s_B;
  const int nseg = p.nseg > 0 ? p.nseg : 1;
  uint32_t *xw = p.xw + (long long)s * nseg * p.x_size;
  uint32_t *dw = p.dw + (long long)s * nseg * p.d_size;
  const bool implicit = p.up.pulse_type == AB200_PULSE_DETERMINISTIC_IMPLICIT;
  const bool mean_count = p.up.pulse_type == AB200_PULSE_MEAN_COUNT;

  for (int l = threadIdx.x; l < p.x_size + p.d_size; l += blockDim.x) {
    const bool is_x = l < p.x_size;
    const int idx = is_x ? l : l - p.x_size;
    float v = is_x ? xValue(idx) : dr[(long long)idx * p.d_fs];
    const float P = is_x ? B : A;
    uint32_t word;
    if (implicit) {
      // generateDetImplicit (dense_bit_line_maker.cpp:210-238); d-values carry the factor BL
      // (generateCoincidencesDetI :240-264)
      float vv = p.lr_neg ? -v : v;
      float pp = pulseProb(p, __fmul_rn(fabsf(vv), P), is_x ? p.up.x_res_implicit : p.up.d_res_implicit,
                           (uint32_t)idx, (uint32_t)s, is_x ? TAG_PULSE_X : TAG_PULSE_D);
      pp = fmaxf(fminf(pp, 1.0f), 0.0f);
      float sv = vv >= 0.0f ? pp : -pp;
      if (BL == 0) {
        sv = 0.0f;
      }
      if (!is_x) {
        sv = __fmul_rn(sv, (float)BL);
      }
      word = __float_as_uint(sv);
    } else if (mean_count) {
      // generateCountsMean / generateCoincidences (dense_bit_line_maker.cpp:142-204): the mean
      // number of pulses per line, no fluctuation; the d count carries the factor 1 / BL, so the
      // coincidences are rint(d * x) like those of the implicit type
      const float vv = p.lr_neg ? -v : v;
      const float pp = pulseProb(p, __fmul_rn(fabsf(vv), P), p.up.res, (uint32_t)idx, (uint32_t)s,
                                 is_x ? TAG_PULSE_X : TAG_PULSE_D);
      float sv = 0.0f;
      if (pp != 0.0f && BL > 0) {
        const int ntimes = max(min((int)rintf(__fmul_rn((float)BL, pp)), BL), 0);
        sv = (vv >= 0.0f || ntimes == 0) ? (float)ntimes : -(float)ntimes;
        if (!is_x) {
          sv = __fdiv_rn(sv, (float)BL);
        }
      }
      word = __float_as_uint(sv);
    } else {
      float pp = 0.0f;
      uint32_t neg = 0u;
      if (BL > 0) {
        pp = pulseProb(p, __fmul_rn(fabsf(v), P), p.up.res, (uint32_t)idx, (uint32_t)s,
                       is_x ? TAG_PULSE_X : TAG_PULSE_D);
        neg = v > 0.0f ? 0u : 1u;
        if (!is_x && p.lr_neg) {
          neg ^= 1u;
        }

      }
      const int n_lines = is_x ? p.x_size : p.d_size;
      for (int g = 0; g < nseg; g++) {
        word = 0;
        if (pp != 0.0f && g * kPulseSegSlots < BL) {
          word = pulseTrain(pp, BL, g, p.key, (uint32_t)idx, (uint32_t)s, p.call,
                            is_x ? TAG_PULSE_X : TAG_PULSE_D);
          word = word ? (word | neg) : 0u;
        }
        (is_x ? xw : dw)[(long long)g * n_lines + idx] = word;
      }
      continue;
    }
    (is_x ? xw : dw)[idx] = word;
  }
}

constexpr int UT_I = 64; // d-lines per CTA (contiguous in memory)
constexpr int UT_J = 16; // x-lines per CTA
constexpr int UBLK = 32; // samples per block = bits of one non-zero bitmap word
constexpr int UT_JP = UT_J + 1; // padded row length of the staged x words (bank spread)

// Bitmaps of the non-empty pulse words: bit s of the word of a line is set when the pulse word of
// sample blk * 32 + s on that line carries at least one pulse (or a non-zero implicit value). The
// update kernel builds them in shared memory while it stages the words, intersects the bitmaps of
// a d-line and an x-line and only looks at the samples that survive - the GPU form of the index
// lists the reference CPU builds per pulse slot (src/rpucuda/sparse_bit_line_maker.cpp:200-238).

// Every thread owns EJ weights (one d-line, EJ x-lines; EJ = 4 with 256 threads per CTA for large
// problems, EJ = 1 with 1024 threads when the grid would otherwise not fill the GPU). The loop
// over a thread's weights is NOT unrolled: its body always works on slot 0 of the register arrays,
// which are rotated by one after every weight, so the (large) body exists once and stays in the
// instruction cache. Per super-block of 128 samples the thread
// walks, for each of its weights, the samples where both lines pulsed; the walk is decoupled from
// the (expensive, rare) pulse application: each lane first advances to ITS next coincidence, then
// the whole warp applies one event per lane together, so lanes whose events fall on different
// samples do not serialise each other. The super-block is long so that the number of events per
// lane has a small relative spread (the warp runs as many rounds as its busiest lane). Weights
// are independent, so the per-weight sample order - the only order the reference defines
// (rpu_weight_updater.cpp:243-291) - is preserved.
constexpr int USUP = 4;              // bitmap words per super-block
constexpr int USAMP = USUP * UBLK;   // samples per super-block
constexpr int URES = 8;              // Gaussians per thread in the reservoir

template <int NT, int UTJ> struct UpdateSmem {
  uint32_t sd[USAMP][UT_I];
  uint32_t sx[USAMP][(UTJ + 1)];
  uint32_t sdnz[USUP][UT_I];
  uint32_t sxnz[USUP][UTJ];
  float sz[URES][NT];
};

// Eight fresh Gaussians for one thread's column of the reservoir. Kept out of line: the refill is
// rare, and inlining it into each of the four per-weight loop bodies makes the kernel spill out of
// the instruction cache.
__device__ __noinline__ void refillReservoir(PhiloxKey key, uint32_t gid, uint32_t refills,
                                             uint32_t call, uint32_t tag, float *column, int stride) {
  float z[8];
  gauss8(key, (uint64_t)gid | ((uint64_t)refills << 32), call, tag, z);
#pragma unroll
  for (int r = 0; r < URES; r++) {
    column[r * stride] = z[r];
  }
}

template <int KIND, bool IMPLICIT, bool NOISY, int EJ, int UTJ>
__global__ void __launch_bounds__(UT_I *UTJ / EJ, (UT_I * UTJ / EJ) >= 1024 ? 1 : 4)
    pulsedUpdateKernel(UpdateProblem p) {
  pdlEnter();
  constexpr int UE_J = EJ;
  constexpr int UNT = UT_I * UTJ / EJ; // threads per CTA
  extern __shared__ __align__(16) unsigned char smem_raw[];
  UpdateSmem<UNT, UTJ> &sm = *reinterpret_cast<UpdateSmem<UNT, UTJ> *>(smem_raw);
  const int ti = threadIdx.x & (UT_I - 1);
  const int tj = threadIdx.x / UT_I;
  const int i = blockIdx.x * UT_I + ti;
  const int j0 = blockIdx.y * UTJ + tj * UE_J;
  const bool i_ok = i < p.d_size;

  float w[UE_J];
  float4 q[UE_J];
  float2 e[UE_J];
  bool loaded[UE_J], dirty[UE_J];
#pragma unroll
  for (int t = 0; t < UE_J; t++) {
    loaded[t] = false;
    dirty[t] = false;
    w[t] = 0.0f;
    q[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    e[t] = make_float2(0.f, 0.f);
  }
  const float std = p.dw_min_std;
  const uint32_t gid = (blockIdx.y * gridDim.x + blockIdx.x) * (uint32_t)UNT + threadIdx.x;
  uint32_t refills = 0;
  int rc = 0;

  const int b_first = p.s_begin / USAMP, b_last = (p.s_end - 1) / USAMP;
  for (int blk = b_first; blk <= b_last; blk++) {
    const int s0 = blk * USAMP;
    // bitmaps of the non-empty words of this super-block, built while the words are staged
    for (int t = threadIdx.x; t < USUP * (UT_I + UTJ); t += blockDim.x) {
      if (t < USUP * UT_I) {
        (&sm.sdnz[0][0])[t] = 0u;
      } else {
        (&sm.sxnz[0][0])[t - USUP * UT_I] = 0u;
      }
    }
    __syncthreads();
    {
      // every thread stages one fixed column of the x words and one of the d words, so the
      // loop only advances a pointer by a row; it collects the column's bitmap bits of its
      // samples in registers (the word a sample falls into is known at compile time, or one of
      // a few) and adds them to the shared bitmap at the end
      constexpr int STEP = UNT / UTJ;               // samples between two rows of a thread
      constexpr int WPS = STEP >= 32 ? STEP / 32 : 1; // bitmap words its first row can fall into
      const int jj = threadIdx.x % UTJ, sj = threadIdx.x / UTJ;
      const int gj = blockIdx.y * UTJ + jj;
      const uint32_t *src = p.xw + (long long)(s0 + sj) * p.x_size + gj;
      const long long step = (long long)STEP * p.x_size;
      uint32_t nzb[USUP];
#pragma unroll
      for (int wq = 0; wq < USUP; wq++) {
        nzb[wq] = 0u;
      }
#pragma unroll
      for (int k = 0; k < USAMP / STEP; k++, src += step) {
        const int ss = sj + STEP * k;
        const uint32_t wv = (gj < p.x_size && s0 + ss < p.m) ? *src : 0u;
        sm.sx[ss][jj] = wv;
        const bool nz = (IMPLICIT ? (wv & 0x7fffffffu) : wv) != 0u;
        const uint32_t bit = nz ? 1u << (ss & 31) : 0u;
        if (STEP < 32) {
          nzb[(STEP * k) >> 5] |= bit;
        } else {
#pragma unroll
          for (int c = 0; c < WPS; c++) {
            nzb[WPS * k + c] |= (sj >> 5) == c ? bit : 0u;
          }
        }
      }
#pragma unroll
      for (int wq = 0; wq < USUP; wq++) {
        if (nzb[wq] != 0u) {
          atomicOr(&sm.sxnz[wq][jj], nzb[wq]);
        }
      }
    }
    {
      constexpr int STEP = UNT / UT_I; // 4 or 16: a thread's rows never leave the word of STEP * k
      const int ii = threadIdx.x % UT_I, si = threadIdx.x / UT_I;
      const int gi = blockIdx.x * UT_I + ii;
      const uint32_t *src = p.dw + (long long)(s0 + si) * p.d_size + gi;
      const long long step = (long long)STEP * p.d_size;
      uint32_t nzb[USUP];
#pragma unroll
      for (int wq = 0; wq < USUP; wq++) {
        nzb[wq] = 0u;
      }
#pragma unroll
      for (int k = 0; k < USAMP / STEP; k++, src += step) {
        const int ss = si + STEP * k;
        const int sg = s0 + ss;
        const uint32_t wv = (gi < p.d_size && sg < p.m) ? *src : 0u;
        sm.sd[ss][ii] = wv;
        // samples of this super-block that belong to [s_begin, s_end): only the d bitmap needs
        // the range, a candidate needs both lines
        const bool nz = (IMPLICIT ? (wv & 0x7fffffffu) : wv) != 0u && sg >= p.s_begin && sg < p.s_end;
        nzb[(STEP * k) >> 5] |= nz ? 1u << (ss & 31) : 0u;
      }
#pragma unroll
      for (int wq = 0; wq < USUP; wq++) {
        if (nzb[wq] != 0u) {
          atomicOr(&sm.sdnz[wq][ii], nzb[wq]);
        }
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < UE_J; t++) {
      const int jl = tj * UE_J + t;
      const long long idx = (long long)(j0 + t) * p.d_size + i;
      // chopped transfer compound: the pulses of this weight enter with the opposite sign when
      // exactly one of its two lines is chopped (ChoppedTransferRPUDevice::doSparseUpdate /
      // doDenseUpdate, rpu_chopped_transfer_device.cpp:472-515); read per launch, so a flip by
      // a transfer between two launches of a batch takes effect for the samples after it
      bool chop_flip = false;
      if (p.chop_x != nullptr) {
        chop_flip = ((j0 + t < p.x_size ? p.chop_x[j0 + t] : 0) != 0) != ((i_ok ? p.chop_d[i] : 0) != 0);
      }
      int wi = 0;
      uint32_t cand = sm.sdnz[0][ti] & sm.sxnz[0][jl];
      while (true) {
        // advance to this lane's next coincidence
        int n = 0;
        bool down = false;
        while (true) {
          if (cand == 0u) {
            if (++wi >= USUP) {
              break;
            }
            cand = sm.sdnz[wi][ti] & sm.sxnz[wi][jl];
            continue;
          }
          const int ss = wi * UBLK + __ffs(cand) - 1;
          cand &= cand - 1u;
          const uint32_t dwv = sm.sd[ss][ti], xwv = sm.sx[ss][jl];
          if (IMPLICIT) {
            // n = rint(d * BL * x), positive = decrease (dense_bit_line_maker.cpp:240-264)
            float c = rintf(__fmul_rn(__uint_as_float(dwv), __uint_as_float(xwv)));
            n = (int)fabsf(c);
            down = (c > 0.0f) != chop_flip;
          } else {
            // coincidences of the two trains; equal line signs = decrease
            // (rpu_weight_updater.cpp:246-268)
            n = __popc((xwv & dwv) >> 1);
            down = (((xwv ^ dwv) & 1u) == 0u) != chop_flip;
          }
          if (n != 0) {
            break;
          }
        }
        if (!__any_sync(0xffffffffu, n != 0)) {
          break;
        }
        if (n != 0) {
          if (!loaded[0]) {
            w[0] = p.w[idx];
            q[0] = p.par4[idx];
            if (KIND != AB200_DEVICE_CONSTANT_STEP && KIND != AB200_DEVICE_EXP_STEP &&
                KIND != AB200_DEVICE_PIECEWISE_STEP) {
              e[0] = p.par2[idx];
            }
            loaded[0] = true;
          }
          dirty[0] = true;
        }
        if (!NOISY) {
          for (int k = 0; k < n; k++) {
            w[0] = pulseOnce<KIND>(w[0], down, q[0], e[0], 0.0f, p.mult_noise, p.es0, p.es1, p.pw, p.pw_n);
          }
        } else {
          // One Gaussian per pulse, taken from a per-thread reservoir in shared memory: the
          // generator - by far the most expensive part of a pulse - runs once per several
          // events instead of per event. The whole warp refills together as soon as one lane
          // cannot serve its event (leftovers are discarded), so the refill is never divergent;
          // only an event with more pulses than the reservoir holds refills on its own.
          if (__any_sync(0xffffffffu, n > rc)) {
            refillReservoir(p.key, gid, refills, p.call, deviceNoiseTag(p), &sm.sz[0][threadIdx.x], UNT);
            rc = URES;
            refills++;
          }
          for (int k = 0; k < n; k++) {
            if (rc == 0) {
              refillReservoir(p.key, gid, refills, p.call, deviceNoiseTag(p), &sm.sz[0][threadIdx.x], UNT);
              rc = URES;
              refills++;
            }
            rc--;
            w[0] = pulseOnce<KIND>(w[0], down, q[0], e[0], std * sm.sz[rc][threadIdx.x], p.mult_noise, p.es0,
                                    p.es1, p.pw, p.pw_n);
          }
        }
      }
      if (UE_J > 1) {
        // rotate the register arrays by one: the next weight moves into slot 0
        const float w0 = w[0];
        const float4 q0 = q[0];
        const float2 e0 = e[0];
        const bool l0 = loaded[0], d0 = dirty[0];
#pragma unroll
        for (int k = 0; k + 1 < UE_J; k++) {
          w[k] = w[k + 1];
          q[k] = q[k + 1];
          e[k] = e[k + 1];
          loaded[k] = loaded[k + 1];
          dirty[k] = dirty[k + 1];
        }
        w[UE_J - 1] = w0;
        q[UE_J - 1] = q0;
        e[UE_J - 1] = e0;
        loaded[UE_J - 1] = l0;
        dirty[UE_J - 1] = d0;
      }
    }
    __syncthreads();
  }
  if (i_ok) {
#pragma unroll
    for (int t = 0; t < UE_J; t++) {
      if (dirty[t]) {
        p.w[(long long)(j0 + t) * p.d_size + i] = w[t];
      }
    }
  }
}

template <int KIND, bool IMPLICIT, bool NOISY, int EJ, int UTJ>
static void launchUpdateVariant(const UpdateProblem &p, cudaStream_t stream) {
  constexpr int NT = UT_I * UTJ / EJ;
  static bool configured[64] = {};
  int dev = 0;
  AB200_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && !configured[dev]) {
    AB200_CUDA(cudaFuncSetAttribute(pulsedUpdateKernel<KIND, IMPLICIT, NOISY, EJ, UTJ>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(UpdateSmem<NT, UTJ>)));
    configured[dev] = true;
  }
  dim3 grid((p.d_size + UT_I - 1) / UT_I, (p.x_size + UTJ - 1) / UTJ);
  AB200_CUDA(launchChained(pulsedUpdateKernel<KIND, IMPLICIT, NOISY, EJ, UTJ>, grid, dim3(NT),
                           sizeof(UpdateSmem<NT, UTJ>), stream, p));
}

template <int KIND, bool IMPLICIT, bool NOISY>
static void launchUpdateInstance(const UpdateProblem &p, dim3 grid, cudaStream_t stream) {
  // `grid` = CTAs of 64 d-lines x 16 x-lines. Four weights per thread (256 threads, four CTAs
  // per SM) once that grid fills the GPU several times over; one weight per thread (1024
  // threads) for small tiles; and CTAs of 64 x 4 weights (256 threads) when even that would
  // leave SMs without a CTA (a 256 x 256 tile is 64 CTAs of 64 x 16, but 256 of 64 x 4)
  static int n_sm = 0;
  if (n_sm == 0) {
    int dev = 0;
    AB200_CUDA(cudaGetDevice(&dev));
    AB200_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  }
  const long long n = (long long)grid.x * grid.y;
  if (n >= 3LL * n_sm) {
    launchUpdateVariant<KIND, IMPLICIT, NOISY, 4, UT_J>(p, stream);
  } else if (n >= n_sm) {
    launchUpdateVariant<KIND, IMPLICIT, NOISY, 1, UT_J>(p, stream);
  } else {
    launchUpdateVariant<KIND, IMPLICIT, NOISY, 1, 4>(p, stream);
  }
}

// ---------------------------------------------------------------------------------------------
// Implicit pulses without device noise: every pair of lines of a sample has a value, so there is nothing to
// skip and nothing to look up but n = rint(d * BL * x) (dense_bit_line_maker.cpp:240-264). A thread
// owns EJ weights of one d-line and takes the samples in order; the warp applies pulse k of a sample to the
// weights with more than k of them, all EJ chains at once, until none is left. Bound by the instructions of
// that (26 per pair of lines and warp, 0.6 of the issue slots used). The staged kernel searched bitmaps
// that are all ones and took one event per lane and round: 512 x 512, 128 samples, 245 -> 39 us.
// ---------------------------------------------------------------------------------------------
constexpr int UD_I = 64;    // d-lines per CTA
constexpr int UD_S = 64;    // samples staged at a time
constexpr int UD_T = 4;     // groups of 64 threads, EJ x-lines each

template <int KIND, int EJ>
__global__ void __launch_bounds__(UD_I *UD_T) pulsedUpdateDenseKernel(UpdateProblem p, bool short_train) {
  pdlEnter();
  constexpr int UJ = UD_T * EJ;
  __shared__ float sd[UD_S][UD_I];
  __shared__ __align__(16) float sx[UD_S][UJ];
  const int ti = threadIdx.x % UD_I, tj = threadIdx.x / UD_I;
  const int i = blockIdx.x * UD_I + ti, j0 = blockIdx.y * UJ;
  const bool i_ok = i < p.d_size;
  float w[EJ], w_in[EJ];
  PulseStep<KIND> step[EJ];
  bool flip[EJ];
#pragma unroll
  for (int t = 0; t < EJ; t++) {
    const int j = j0 + tj * EJ + t;
    const bool ok = i_ok && j < p.x_size;
    const long long idx = ok ? (long long)j * p.d_size + i : 0;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    float2 e = make_float2(0.f, 0.f);
    w[t] = 0.0f;
    flip[t] = false;
    if (ok) {
      w[t] = p.w[idx];
      q = p.par4[idx];
      if (KIND != AB200_DEVICE_CONSTANT_STEP && KIND != AB200_DEVICE_EXP_STEP &&
          KIND != AB200_DEVICE_PIECEWISE_STEP) {
        e = p.par2[idx];
      }
      if (p.chop_x != nullptr) {
        flip[t] = (p.chop_x[j] != 0) != (p.chop_d[i] != 0);
      }
    }
    step[t].set(q, e);
    w_in[t] = w[t];
  }
  for (int s0 = p.s_begin; s0 < p.s_end; s0 += UD_S) {
    const int n_s = min(UD_S, p.s_end - s0);
#pragma unroll 8
    for (int r = tj; r < UD_S; r += UD_T) {
      sd[r][ti] = (r < n_s && i_ok) ? __uint_as_float(p.dw[(long long)(s0 + r) * p.d_size + i]) : 0.0f;
    }
#pragma unroll
    for (int e = threadIdx.x; e < UD_S * UJ; e += UD_I * UD_T) {
      const int r = e / UJ, j = j0 + e % UJ;
      sx[r][e % UJ] =
          (r < n_s && j < p.x_size) ? __uint_as_float(p.xw[(long long)(s0 + r) * p.x_size + j]) : 0.0f;
    }
    __syncthreads();
    for (int r = 0; r < n_s; r++) {
      const float dv = sd[r][ti];
      float c[EJ];
      int n[EJ], most = 0;
#pragma unroll
      for (int t = 0; t < EJ; t++) {
        c[t] = __fmul_rn(dv, sx[r][tj * EJ + t]);
        n[t] = implicitPulses(c[t], short_train);
        most = max(most, n[t]);
      }
      // (counted in whole numbers: the end is reached whatever the length of the train)
      for (int k = 0; __any_sync(0xffffffffu, most > k); k++) {
#pragma unroll
        for (int t = 0; t < EJ; t++) {
          // positive = decrease
          const float w_new = step[t].apply(p, w[t], (c[t] > 0.0f) != flip[t], PulseStep<KIND>::kOnePlus ? 1.0f : 0.0f);
          w[t] = n[t] > k ? w_new : w[t];
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < EJ; t++) {
    const int j = j0 + tj * EJ + t;
    if (i_ok && j < p.x_size && w[t] != w_in[t]) {
      p.w[(long long)j * p.d_size + i] = w[t];
    }
  }
}

template <int KIND> static void launchUpdateDense(const UpdateProblem &p, cudaStream_t stream) {
  static int n_sm = 0; // SMs of the GPUs of this process (one kind per process)
  if (n_sm == 0) {
    int dev = 0;
    AB200_CUDA(cudaGetDevice(&dev));
    AB200_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  }
  // four weights per thread where that still gives every SM a CTA, else one
  const int gx = (p.d_size + UD_I - 1) / UD_I, gy4 = (p.x_size + 15) / 16, gy1 = (p.x_size + 3) / 4;
  const bool st = longestTrain(p.up, p.lr, p.dw_min) <= kShortTrain;
  if ((long long)gx * gy4 >= n_sm) {
    AB200_CUDA(launchChained(pulsedUpdateDenseKernel<KIND, 4>, dim3(gx, gy4), dim3(UD_I * UD_T), 0, stream, p, st));
  } else {
    AB200_CUDA(launchChained(pulsedUpdateDenseKernel<KIND, 1>, dim3(gx, gy1), dim3(UD_I * UD_T), 0, stream, p, st));
  }
}

static int g_update_path = 0;
void setUpdatePath(int mode) { g_update_path = mode; }

bool planeUpdateEligible(const UpdateProblem &p) {
  if (g_update_path == 1 || p.up.pulse_type != AB200_PULSE_STOCHASTIC_COMPRESSED) {
    return false;
  }
  return g_update_path == 2 || p.m * (p.nseg > 0 ? p.nseg : 1) >= kPlaneUpdateMinRows;
}

void launchPulsePrepare(const UpdateProblem &p, cudaStream_t stream) {
  if (p.m <= 0) {
    return;
  }
  AB200_CUDA(launchChained(pulsePrepareKernel, dim3(p.m), dim3(256), 0, stream, p));
  AB200_LAUNCH_CHECK();
}

void launchPulsedUpdate(const UpdateProblem &p0, cudaStream_t stream) {
  const UpdateProblem p = inRows(p0);
  if (p.s_end <= p.s_begin) {
    return;
  }
  dim3 grid((p.d_size + UT_I - 1) / UT_I, (p.x_size + UT_J - 1) / UT_J);
  const bool implicit = p.up.pulse_type == AB200_PULSE_DETERMINISTIC_IMPLICIT ||
                        p.up.pulse_type == AB200_PULSE_MEAN_COUNT;
  const bool noisy = p.dw_min_std > 0.0f;
#define AB200_UPD2(KIND, IMPL)                                                                     \
  if (noisy) {                                                                                     \
    launchUpdateInstance<KIND, IMPL, true>(p, grid, stream);                                       \
  } else {                                                                                         \
    launchUpdateInstance<KIND, IMPL, false>(p, grid, stream);                                      \
  }
#define AB200_UPD(KIND)                                                                            \
  if (implicit && !noisy) {                                                                        \
    launchUpdateDense<KIND>(p, stream);                                                            \
  } else if (implicit) {                                                                           \
    launchUpdateInstance<KIND, true, true>(p, grid, stream);                                       \
  } else {                                                                                         \
    AB200_UPD2(KIND, false)                                                                        \
  }
  switch (p.kind) {
  case AB200_DEVICE_CONSTANT_STEP:
    AB200_UPD(AB200_DEVICE_CONSTANT_STEP);
    break;
  case AB200_DEVICE_LINEAR_STEP:
  case AB200_DEVICE_SOFT_BOUNDS:
    AB200_UPD(AB200_DEVICE_LINEAR_STEP);
    break;
  case AB200_DEVICE_SOFT_BOUNDS_REFERENCE:
    AB200_UPD(AB200_DEVICE_SOFT_BOUNDS_REFERENCE);
    break;
  case AB200_DEVICE_POW_STEP:
    AB200_UPD(AB200_DEVICE_POW_STEP);
    break;
  case AB200_DEVICE_EXP_STEP:
    AB200_UPD(AB200_DEVICE_EXP_STEP);
    break;
  case AB200_DEVICE_PIECEWISE_STEP:
    AB200_UPD(AB200_DEVICE_PIECEWISE_STEP);
    break;
  default:
    AB200_FATAL("pulsed update: device kind not implemented");
  }
#undef AB200_UPD
#undef AB200_UPD2
  AB200_LAUNCH_CHECK();
}

// Signed coincidence counts of sample 0 as int32 [d][x] (DenseBitLineMaker::makeCoincidences).
__global__ void coincidenceKernel(UpdateProblem p, int32_t *counts) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)p.x_size * p.d_size) {
    return;
  }
  int i = (int)(t / p.x_size), j = (int)(t % p.x_size);
  uint32_t xwv = p.xw[j], dwv = p.dw[i];
  int n;
  if (p.up.pulse_type == AB200_PULSE_DETERMINISTIC_IMPLICIT ||
      p.up.pulse_type == AB200_PULSE_MEAN_COUNT) {
    n = dwv == 0u ? 0 : (int)rintf(__fmul_rn(__uint_as_float(dwv), __uint_as_float(xwv)));
  } else {
    n = 0;
    const int nseg = p.nseg > 0 ? p.nseg : 1;
    for (int g = 0; g < nseg; g++) {
      xwv = p.xw[(long long)g * p.x_size + j];
      dwv = p.dw[(long long)g * p.d_size + i];
      const int c = __popc((xwv & dwv) >> 1);
      n += ((xwv ^ dwv) & 1u) != 0u ? -c : c;
    }
  }
  counts[t] = n;
}

// Pulse counters (kernelPulseCounter, src/rpucuda/cuda/pwu_kernel.h:1523-1620): a pass of its
// own over the prepared pulse words, one thread per weight, before the update applies them.
__global__ void __launch_bounds__(256)
    pulseCounterKernel(UpdateProblem p, unsigned long long *up, unsigned long long *down) {
  pdlEnter();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)p.x_size * p.d_size) {
    return;
  }
  const int j = (int)(t / p.d_size), i = (int)(t % p.d_size); // the weights' own order [x][d]
  const bool implicit = p.up.pulse_type == AB200_PULSE_DETERMINISTIC_IMPLICIT ||
                        p.up.pulse_type == AB200_PULSE_MEAN_COUNT;
  const int nseg = p.nseg > 0 ? p.nseg : 1;
  unsigned long long n_up = 0, n_down = 0;
  for (int s = p.s_begin; s < p.s_end; s++) {
    const uint32_t *xw = p.xw + (long long)s * nseg * p.x_size;
    const uint32_t *dw = p.dw + (long long)s * nseg * p.d_size;
    if (implicit) {
      const uint32_t dwv = dw[i];
      const int n = dwv == 0u ? 0 : (int)rintf(__fmul_rn(__uint_as_float(dwv), __uint_as_float(xw[j])));
      // a positive product lowers the weight (w -= lr d x)
      if (n > 0) {
        n_down += (unsigned)n;
      } else {
        n_up += (unsigned)(-n);
      }
    } else {
      for (int g = 0; g < nseg; g++) {
        const uint32_t xwv = xw[(long long)g * p.x_size + j], dwv = dw[(long long)g * p.d_size + i];
        const unsigned c = (unsigned)__popc((xwv & dwv) >> 1);
        if (((xwv ^ dwv) & 1u) == 0u) {
          n_down += c;
        } else {
          n_up += c;
        }
      }
    }
  }
  up[t] += n_up;
  down[t] += n_down;
}

void launchPulseCounter(const UpdateProblem &p, unsigned long long *up, unsigned long long *down,
                        cudaStream_t stream) {
  if (p.s_end <= p.s_begin) {
    return;
  }
  const long long n = (long long)p.x_size * p.d_size;
  AB200_CUDA(launchChained(pulseCounterKernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, p, up,
                           down));
  AB200_LAUNCH_CHECK();
}

void launchCoincidences(const UpdateProblem &p, int32_t *counts_dx, cudaStream_t stream) {
  long long n = (long long)p.x_size * p.d_size;
  coincidenceKernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(p, counts_dx);
  AB200_LAUNCH_CHECK();
}

// Floating-point update W[x][d] -= lr * sum_s x[s][x] d[s][d] (RPUSimple::updateMatrix,
// src/rpucuda/rpu.cpp:700-745), used by ideal devices / PulseType::None.
// `overwrite`: the target receives -lr * sum alone (delta-weight mode: beta = 0, rpu.cpp:1509-1511)
//
// T x T sums per thread, 16 x 16 threads; the samples come in steps through registers into one of two
// buffers, so that the loads of a step are in flight while the one before is multiplied. Bound by issue slots (0.65
// used) and shared memory, the fp32 units are 45 % active; 64 x 16 sums per CTA with a barrier on each side of an
// unpipelined load took 194 us for 1024 x 1024 and 512 samples, this takes 41.
//
// With 64 x 64 sums per CTA two groups of 256 threads share them, each with every other step, and add up at the
// end: one group's eight warps do not hide the latency of shared memory.
//
// FEW: one step of samples (T = 4). The weights are most of the traffic then: one group, which reads them before
// the samples. 2048 x 2048, 4 / 16 samples: 22.8 / 23.0 -> 9.0 / 9.3 us.
__host__ __device__ constexpr int fpUpdateGroups(int T) { return T == 4 ? 2 : 1; }

template <int T, bool FEW = false>
__global__ void __launch_bounds__(256 * (FEW ? 1 : fpUpdateGroups(T)))
    fpUpdateKernel(UpdateProblem p, float lr_signed, int overwrite) {
  pdlEnter();
  constexpr int BN = 16 * T, BK = 64 / T; // lines and samples per step: four values per thread and operand
  constexpr int G = FEW ? 1 : fpUpdateGroups(T);
  __shared__ __align__(16) float xs_all[G][2][BK][BN + 4], ds_all[G][2][BK][BN + 4];
  const int grp = G == 1 ? 0 : threadIdx.x >> 8;
  float(*const xs)[BK][BN + 4] = xs_all[grp];
  float(*const ds)[BK][BN + 4] = ds_all[grp];
  const int tid = threadIdx.x & 255, tx = tid & 15, ty = tid >> 4;
  const int i0 = blockIdx.x * BN, j0 = blockIdx.y * BN;
  float rx[4], rd[4], acc[T][T];
#pragma unroll
  for (int a = 0; a < T; a++) {
#pragma unroll
    for (int b = 0; b < T; b++) {
      acc[a][b] = 0.0f;
    }
  }
  // four neighbouring lines of a sample per thread (or four samples of a line where those are contiguous),
  // in one load where alignment and sizes allow
  const bool x_line = p.x_fs == 1 || p.x_ss != 1, d_line = p.d_fs == 1 || p.d_ss != 1;
  const int LV = BN / 4, SV = BK / 4;
  const int x_s = x_line ? tid / LV : (tid % SV) * 4, x_j = x_line ? (tid % LV) * 4 : tid / SV;
  const int d_s = d_line ? tid / LV : (tid % SV) * 4, d_i = d_line ? (tid % LV) * 4 : tid / SV;
  auto vec = [&](const float *v, long long fs, long long ss, bool line, int lines, int real) {
    return (line ? fs == 1 && (ss & 3) == 0 && (lines & 3) == 0 : ss == 1 && (fs & 3) == 0 && (p.m & 3) == 0) &&
           real == lines && (reinterpret_cast<uintptr_t>(v) & 15) == 0;
  };
  const bool x_vec = vec(p.x, p.x_fs, p.x_ss, x_line, p.x_size, p.x_real);
  const bool d_vec = vec(p.d, p.d_fs, p.d_ss, d_line, p.d_size, p.d_size);
  const float *x_src = p.x + (long long)x_s * p.x_ss + (long long)(j0 + x_j) * p.x_fs;
  const float *d_src = p.d + (long long)d_s * p.d_ss + (long long)(i0 + d_i) * p.d_fs;
  auto load4 = [&](float *r, bool v4, const float *src, long long ss, long long fs, bool line, int s, int l, int lines,
                   int real) {
    if (v4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s < p.m && l < lines) {
        v = __ldg(reinterpret_cast<const float4 *>(src));
      }
      r[0] = v.x;
      r[1] = v.y;
      r[2] = v.z;
      r[3] = v.w;
    } else {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int gs = s + (line ? 0 : u), gl = l + (line ? u : 0);
        r[u] = 0.0f;
        if (gs < p.m && gl < lines) {
          r[u] = 1.0f; // the bias line
          if (gl < real) {
            r[u] = src[line ? u * fs : u * ss];
          }
        }
      }
    }
  };
  auto load = [&](int s0) {
    load4(rx, x_vec, x_src + s0 * p.x_ss, p.x_ss, p.x_fs, x_line, s0 + x_s, j0 + x_j, p.x_size, p.x_real);
    load4(rd, d_vec, d_src + s0 * p.d_ss, p.d_ss, p.d_fs, d_line, s0 + d_s, i0 + d_i, p.d_size, p.d_size);
  };
  auto stage4 = [&](float (*dst)[BN + 4], const float *r, bool line, int s, int l) {
    if (line) {
      *reinterpret_cast<float4 *>(&dst[s][l]) = make_float4(r[0], r[1], r[2], r[3]);
    } else {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        dst[s + u][l] = r[u];
      }
    }
  };
  auto stage = [&](int buf) {
    stage4(xs[buf], rx, x_line, x_s, x_j);
    stage4(ds[buf], rd, d_line, d_s, d_i);
  };
  const bool w_vec = T == 4 && (p.d_size & 3) == 0 && (reinterpret_cast<uintptr_t>(p.w) & 15) == 0;
  auto loadWeights = [&](int u, float *old) {
    const int j = j0 + ty * T + u, i = i0 + tx * T;
    if (overwrite || j >= p.x_size || i >= p.d_size) {
      return;
    }
    const float *w = p.w + (long long)j * p.d_size + i;
    if (w_vec) {
      loadRow<T>(w, old);
    } else {
#pragma unroll
      for (int v = 0; v < T; v++) {
        old[v] = i + v < p.d_size ? w[v] : 0.0f;
      }
    }
  };
  float before[FEW ? T : 1][T];
  if (FEW) {
#pragma unroll
    for (int u = 0; u < T; u++) {
      loadWeights(u, before[FEW ? u : 0]);
    }
  }
  // (both groups take the same number of steps; past the end the operands are zeros)
  load(grp * BK);
  stage(0);
  __syncthreads();
  for (int sb = 0, buf = 0; sb < p.m; sb += G * BK, buf ^= 1) {
    const bool more = sb + G * BK < p.m;
    if (more) {
      load(sb + (G + grp) * BK);
    }
    float an[T], bn[T]; // operands of the next sample, on their way from shared memory
    loadRow<T>(&xs[buf][0][ty * T], an);
    loadRow<T>(&ds[buf][0][tx * T], bn);
#pragma unroll
    for (int s = 0; s < BK; s++) {
      float a[T], b[T];
#pragma unroll
      for (int u = 0; u < T; u++) {
        a[u] = an[u];
        b[u] = bn[u];
      }
      if (s + 1 < BK) {
        loadRow<T>(&xs[buf][s + 1][ty * T], an);
        loadRow<T>(&ds[buf][s + 1][tx * T], bn);
      }
#pragma unroll
      for (int u = 0; u < T; u++) {
#pragma unroll
        for (int v = 0; v < T; v++) {
          acc[u][v] = fmaf(a[u], b[v], acc[u][v]);
        }
      }
    }
    if (more) {
      stage(buf ^ 1);
    }
    __syncthreads();
  }
  if (G > 1) {
    static_assert(G == 1 || sizeof(xs_all) >= sizeof(float) * BN * BN, "room for the sums");
    float *const sums = &xs_all[0][0][0][0];
    if (grp == 1) {
#pragma unroll
      for (int u = 0; u < T; u++) {
#pragma unroll
        for (int v = 0; v < T; v++) {
          sums[(u * T + v) * 256 + tid] = acc[u][v];
        }
      }
    }
    __syncthreads();
    if (grp == 1) {
      return;
    }
#pragma unroll
    for (int u = 0; u < T; u++) {
#pragma unroll
      for (int v = 0; v < T; v++) {
        acc[u][v] += sums[(u * T + v) * 256 + tid];
      }
    }
  }
  // Weights in fours where alignment and size allow: with few samples they are most of the traffic (2048 x 2048, 16
  // samples: 23.0 -> 16.6 us, without FEW)
#pragma unroll
  for (int u = 0; u < T; u++) {
    const int j = j0 + ty * T + u, i = i0 + tx * T;
    if (j >= p.x_size || i >= p.d_size) {
      continue;
    }
    float *const w = p.w + (long long)j * p.d_size + i;
    float old[T];
    if (!FEW) {
      loadWeights(u, old);
    }
#pragma unroll
    for (int v = 0; v < T; v++) {
      acc[u][v] = overwrite ? -lr_signed * acc[u][v] : (FEW ? before[FEW ? u : 0][v] : old[v]) - lr_signed * acc[u][v];
    }
    if (w_vec) {
      *reinterpret_cast<float4 *>(w) = make_float4(acc[u][0], acc[u][T > 1 ? 1 : 0], acc[u][T > 2 ? 2 : 0],
                                                   acc[u][T > 3 ? 3 : 0]);
    } else {
#pragma unroll
      for (int v = 0; v < T; v++) {
        if (i + v < p.d_size) {
          w[v] = acc[u][v];
        }
      }
    }
  }
}

// PulseType::NoneWithDevice: the rank-one update of every sample is followed by the clip to the
// element's bounds (rpu_weight_updater.cpp:216-223), so the samples are applied to the weight one after the
// other instead of being summed first.
__global__ void __launch_bounds__(256) fpUpdateClipKernel(UpdateProblem p, float lr_signed) {
  pdlEnter();
  __shared__ float xs[16][16 + 1];
  __shared__ float ds[16][64 + 1];
  const int ti = threadIdx.x & 63, tj = threadIdx.x >> 6; // 64 d-lines x 4 groups of 4 x-lines
  const int i = blockIdx.x * 64 + ti;
  const int jb = blockIdx.y * 16;
  float wv[4] = {0.f, 0.f, 0.f, 0.f}, hi[4], lo[4];
#pragma unroll
  for (int t = 0; t < 4; t++) {
    const int j = jb + tj * 4 + t;
    hi[t] = lo[t] = 0.0f;
    if (i < p.d_size && j < p.x_size) {
      const long long idx = (long long)j * p.d_size + i;
      wv[t] = p.w[idx];
      if (p.par4 != nullptr) {
        const float4 q = p.par4[idx];
        hi[t] = q.z;
        lo[t] = q.w;
      } else {
        // no bounds: the digital accumulator of a mixed-precision compound
        hi[t] = 3.4e38f;
        lo[t] = -3.4e38f;
      }
    }
  }
  for (int s0 = 0; s0 < p.m; s0 += 16) {
    {
      int ss = threadIdx.x >> 4, jj = threadIdx.x & 15;
      int gs = s0 + ss, gj = jb + jj;
      float v = 0.0f;
      if (gs < p.m && gj < p.x_size) {
        v = gj < p.x_real ? p.x[(long long)gs * p.x_ss + (long long)gj * p.x_fs] : 1.0f;
      }
      xs[ss][jj] = v;
    }
    for (int t = threadIdx.x; t < 16 * 64; t += 256) {
      int ss = t >> 6, ii = t & 63;
      int gs = s0 + ss, gi = blockIdx.x * 64 + ii;
      ds[ss][ii] = (gs < p.m && gi < p.d_size) ? p.d[(long long)gs * p.d_ss + (long long)gi * p.d_fs] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int ss = 0; ss < 16; ss++) {
      float dv = ds[ss][ti];
#pragma unroll
      for (int t = 0; t < 4; t++) {
        wv[t] = __fsub_rn(wv[t], __fmul_rn(__fmul_rn(lr_signed, dv), xs[ss][tj * 4 + t]));
        wv[t] = fmaxf(fminf(wv[t], hi[t]), lo[t]);
      }
    }
    __syncthreads();
  }
  if (i < p.d_size) {
#pragma unroll
    for (int t = 0; t < 4; t++) {
      int j = jb + tj * 4 + t;
      if (j < p.x_size) {
        p.w[(long long)j * p.d_size + i] = wv[t];
      }
    }
  }
}

void launchFPUpdate(const UpdateProblem &p, float lr_signed, cudaStream_t stream, bool overwrite,
                    bool clip_each) {
  if (clip_each) {
    dim3 grid((p.d_size + 63) / 64, (p.x_size + 15) / 16);
    AB200_CUDA(launchChained(fpUpdateClipKernel, grid, dim3(256), 0, stream, p, lr_signed));
    AB200_LAUNCH_CHECK();
    return;
  }
  static int n_sm = 0; // SMs of the GPUs of this process (one kind per process)
  if (n_sm == 0) {
    int dev = 0;
    AB200_CUDA(cudaGetDevice(&dev));
    AB200_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  }
  // the largest tile that still gives every SM a CTA (or, with many x-lines, fits the grid)
  auto grid = [&](int t) { return dim3((p.d_size + 16 * t - 1) / (16 * t), (p.x_size + 16 * t - 1) / (16 * t)); };
  auto fits = [&](int t) { return (long long)grid(t).x * grid(t).y >= n_sm; };
  const int ow = overwrite ? 1 : 0;
  if (p.m <= 16 && (fits(4) || p.x_size > 65535 * 16)) {
    AB200_CUDA(launchChained(fpUpdateKernel<4, true>, grid(4), dim3(256), 0, stream, p, lr_signed, ow));
  } else if (fits(4) || p.x_size > 65535 * 16) {
    AB200_CUDA(launchChained(fpUpdateKernel<4>, grid(4), dim3(256 * fpUpdateGroups(4)), 0, stream, p, lr_signed, ow));
  } else if (fits(2)) {
    AB200_CUDA(launchChained(fpUpdateKernel<2>, grid(2), dim3(256), 0, stream, p, lr_signed, ow));
  } else {
    AB200_CUDA(launchChained(fpUpdateKernel<1>, grid(1), dim3(256), 0, stream, p, lr_signed, ow));
  }
  AB200_LAUNCH_CHECK();
}

// Mixed-precision compound (MixedPrecRPUDevice::doDirectVectorUpdate,
// rpu_mixedprec_device.cpp:196-345): x and d of every sample quantised to n bins of their abs-max,
// q = clip(rint(v / width + u - 0.5), +-half) * width with width = amax / half, half = n / 2.
__global__ void __launch_bounds__(256)
    mixedQuantizeKernel(const float *x, long long x_ss, long long x_fs, int x_real, const float *d,
                        long long d_ss, long long d_fs, int x_size, int d_size, int n_x_bins, int n_d_bins,
                        int sr_x, int sr_d, PhiloxKey key, uint32_t call, float *qx, float *qd) {
  pdlEnter();
  __shared__ float sh[8];
  const int s = blockIdx.x;
  const float *xr = x + (long long)s * x_ss, *dr = d + (long long)s * d_ss;
  float xm = 0.0f, dm = 0.0f;
  for (int j = threadIdx.x; j < x_size; j += blockDim.x) {
    xm = fmaxf(xm, fabsf(j < x_real ? xr[(long long)j * x_fs] : 1.0f));
  }
  for (int i = threadIdx.x; i < d_size; i += blockDim.x) {
    dm = fmaxf(dm, fabsf(dr[(long long)i * d_fs]));
  }
  xm = blockMax(xm, sh);
  dm = blockMax(dm, sh);
  const float half_x = (float)(n_x_bins / 2), half_d = (float)(n_d_bins / 2);
  float x_width = __fdiv_rn(xm, half_x), d_width = __fdiv_rn(dm, half_d);
  x_width = x_width == 0.0f ? 1.0f : x_width;
  d_width = d_width == 0.0f ? 1.0f : d_width;
  for (int l = threadIdx.x; l < x_size + d_size; l += blockDim.x) {
    const bool is_x = l < x_size;
    const int idx = is_x ? l : l - x_size;
    const float v = is_x ? (idx < x_real ? xr[(long long)idx * x_fs] : 1.0f) : dr[(long long)idx * d_fs];
    const float width = is_x ? x_width : d_width, half = is_x ? half_x : half_d;
    float st = 0.0f;
    if (is_x ? sr_x : sr_d) {
      uint32_t r[4];
      philox4x32<7>((uint32_t)idx, (uint32_t)s, call, is_x ? TAG_PULSE_X : TAG_PULSE_D, key, r);
      st = __fadd_rn(u01(r[0]), -0.5f);
    }
    float q = rintf(__fadd_rn(__fdiv_rn(v, width), st));
    // (a zero stays a zero also where a single bin makes the width infinite: the reference skips it)
    q = q == 0.0f ? 0.0f : __fmul_rn(fminf(fmaxf(q, -half), half), width);
    if (is_x) {
      qx[(long long)s * x_size + idx] = q;
    } else {
      qd[(long long)s * d_size + idx] = q;
    }
  }
}

// The whole multiples of the granularity in rows [row0, row0 + n_rows) (mod d_size) of chi leave
// it as pulse counts (forwardUpdate, rpu_mixedprec_device.cpp:148-190); also writes the one-hot
// d vectors of the rows. chi is [x][d] like the weights.
__global__ void __launch_bounds__(256)
    mixedTruncateKernel(float *chi, int x_size, int d_size, int row0, int n_rows, float gran, float *counts,
                        float *onehot) {
  pdlEnter();
  const int j = blockIdx.y;
  const int row = (row0 + j) % d_size;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < x_size) {
    const long long idx = (long long)t * d_size + row;
    const float value = chi[idx];
    const float dw = truncf(__fdiv_rn(value, gran));
    counts[(long long)j * x_size + t] = dw;
    chi[idx] = __fsub_rn(value, __fmul_rn(dw, gran));
  }
  if (t < d_size) {
    onehot[(long long)j * d_size + t] = t == row ? 1.0f : 0.0f;
  }
}

void launchMixedQuantize(const UpdateProblem &p, int n_x_bins, int n_d_bins, int sr_x, int sr_d, float *qx,
                         float *qd, cudaStream_t stream) {
  AB200_CUDA(launchChained(mixedQuantizeKernel, dim3(p.m), dim3(256), 0, stream, p.x, p.x_ss, p.x_fs, p.x_real,
                           p.d, p.d_ss, p.d_fs, p.x_size, p.d_size, n_x_bins, n_d_bins, sr_x, sr_d, p.key,
                           p.call, qx, qd));
  AB200_LAUNCH_CHECK();
}

void launchMixedTruncate(float *chi, int x_size, int d_size, int row0, int n_rows, float gran, float *counts,
                         float *onehot, cudaStream_t stream) {
  const int width = x_size > d_size ? x_size : d_size;
  AB200_CUDA(launchChained(mixedTruncateKernel, dim3((width + 255) / 256, n_rows), dim3(256), 0, stream, chi,
                           x_size, d_size, row0, n_rows, gran, counts, onehot));
  AB200_LAUNCH_CHECK();
}

// Tiki-Taka read of one column of the fast tile: forward of a one-hot vector through the transfer
// IO (noise and bound management off) with alpha = -1
// (TransferRPUDevice::readVector / readAndUpdate, rpu_transfer_device.cpp:410-470). Also writes
// the one-hot vector that the following pulsed write uses as its x input.
__global__ void transferReadKernel(const float *w_fast, int col, int d_size, IOEff io,
                                   PhiloxKey key, uint32_t call, float *x_onehot, int x_size,
                                   float *r_out, float alpha) {
  pdlEnter();
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < x_size) {
    x_onehot[t] = t == col ? 1.0f : 0.0f;
  }
  if (t >= d_size) {
    return;
  }
  float y;
  if (io.is_perfect) {
    y = w_fast[(long long)col * d_size + t] * (alpha * io.out_scale);
  } else {
    float v = prepareInput(io, 1.0f, 1.0f);
    float acc = __fmul_rn(w_fast[(long long)col * d_size + t], v);
    float sigma = outputSigma(io, fabsf(v));
    float z[4] = {0.f, 0.f, 0.f, 0.f};
    if (sigma > 0.0f) {
      gauss4(key, (uint64_t)(t >> 2), call, TAG_TRANSFER_READ, z);
    }
    bool ex = false;
    y = finalizeOutput(io, acc, sigma, z[t & 3], ex);
    y = __fmul_rn(y, __fmul_rn(io.out_scale, alpha));
  }
  r_out[t] = y;
}

// Buffered transfer (Tiki-Taka v2), BufferedTransferRPUDevice::readAndUpdate
// (src/rpucuda/rpu_buffered_transfer_device.cpp:178-208): omega = H + read * |lr|;
// n = trunc(omega / granularity) limited to +-max_steps; H keeps omega * momentum (forget) or
// omega minus the transferred part; the slow tile is then pulsed with d = -n.
__global__ void transferBufferKernel(float *buffer_col, float *read_inout, int d_size, float lr_abs,
                                     float bg, float max_steps, float momentum, int forget_buffer) {
  pdlEnter();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d_size) {
    return;
  }
  const float omega = __fadd_rn(buffer_col[t], __fmul_rn(read_inout[t], lr_abs));
  const float n = fmaxf(fminf(truncf(__fdiv_rn(omega, bg)), max_steps), -max_steps);
  float h = omega;
  if (n != 0.0f) {
    const float sub_momentum = 1.0f - fmaxf(fminf(momentum, 1.0f), 0.0f);
    h = forget_buffer ? __fmul_rn(omega, momentum)
                      : __fsub_rn(omega, __fmul_rn(__fmul_rn(sub_momentum, n), bg));
  }
  buffer_col[t] = h;
  read_inout[t] = -n;
}

__global__ void __launch_bounds__(256)
    transferChopBufferKernel(float *buffer_col, float *read_inout, int d_size, float lr_scale,
                             float max_steps, float momentum, int forget_buffer, int no_buffer,
                             unsigned char *chop_in, int col, const unsigned char *chop_out,
                             int flip_in) {
  pdlEnter();
  // one CTA: the in chopper of the column is read by all threads before thread 0 flips it
  const bool in_chop = chop_in[col] != 0;
  const float sub_momentum = 1.0f - fmaxf(fminf(momentum, 1.0f), 0.0f);
  for (int t = threadIdx.x; t < d_size; t += blockDim.x) {
    float omega = no_buffer ? 0.0f : buffer_col[t];
    const float val = __fmul_rn(read_inout[t], lr_scale);
    omega = __fadd_rn(omega, (in_chop != (chop_out[t] != 0)) ? -val : val);
    float n = 0.0f;
    if (fabsf(omega) >= 1.0f) {
      n = fmaxf(fminf(truncf(omega), max_steps), -max_steps);
      omega = forget_buffer ? __fmul_rn(omega, momentum) : __fsub_rn(omega, __fmul_rn(sub_momentum, n));
    }
    buffer_col[t] = omega;
    read_inout[t] = -n;
  }
  __syncthreads();
  if (threadIdx.x == 0 && flip_in) {
    chop_in[col] = in_chop ? 0 : 1;
  }
}

__global__ void __launch_bounds__(256)
    transferDynamicBufferKernel(float *buffer_col, float *mean_col, float *past_col, float *read_inout,
                                int d_size, float lr_scale, float max_steps, float momentum,
                                int forget_buffer, float buffer_cap, float sample_momentum,
                                int previously_switched, unsigned char *chop_in, int col,
                                const unsigned char *chop_out, int flip_in) {
  pdlEnter();
  // one CTA: the in chopper of the column is read by all threads before thread 0 flips it
  const bool in_chop = chop_in[col] != 0;
  const float keep = 1.0f - sample_momentum, forget = 1.0f - momentum;
  for (int t = threadIdx.x; t < d_size; t += blockDim.x) {
    const float val = read_inout[t];
    float omega = buffer_col[t];
    float mu_past = past_col[t];
    const float mean = mean_col[t];
    if (previously_switched) {
      // a new chopper phase: the mean of the phase that ended becomes the reference
      mu_past = mean;
      past_col[t] = mean;
    }
    float dw = __fsub_rn(val, mu_past);
    dw = (in_chop != (chop_out[t] != 0)) ? -dw : dw;
    omega = __fadd_rn(omega, __fmul_rn(dw, lr_scale));
    float n = 0.0f;
    if (fabsf(omega) >= 1.0f) {
      n = fmaxf(fminf(truncf(omega), max_steps), -max_steps);
      if (forget_buffer) {
        omega = __fmul_rn(omega, momentum);
      } else {
        omega = __fsub_rn(omega, __fmul_rn(forget, n));
        if (buffer_cap > 0.0f) {
          omega = fminf(fmaxf(omega, -buffer_cap), buffer_cap);
        }
      }
    }
    buffer_col[t] = omega;
    read_inout[t] = -n;
    mean_col[t] = __fadd_rn(__fmul_rn(mean, keep), __fmul_rn(val, sample_momentum));
  }
  __syncthreads();
  if (threadIdx.x == 0 && flip_in) {
    chop_in[col] = in_chop ? 0 : 1;
  }
}

__global__ void __launch_bounds__(256)
    flipChoppersKernel(unsigned char *chop, int n, float prob, PhiloxKey key, uint32_t call) {
  pdlEnter();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) {
    return;
  }
  uint32_t r[4];
  philox4x32<7>((uint32_t)t, 0u, call, TAG_TRANSFER_READ ^ 0x01000000u, key, r);
  if (u01(r[0]) < prob) {
    chop[t] = chop[t] ? 0 : 1;
  }
}

void launchTransferChopBuffer(float *buffer_col, float *read_inout, int d_size, float lr_scale,
                              float max_steps, float momentum, int forget_buffer, int no_buffer,
                              unsigned char *chop_in, int col, const unsigned char *chop_out,
                              int flip_in, cudaStream_t stream) {
  AB200_CUDA(launchChained(transferChopBufferKernel, dim3(1), dim3(256), 0, stream, buffer_col, read_inout,
                           d_size, lr_scale, max_steps, momentum, forget_buffer, no_buffer, chop_in, col,
                           chop_out, flip_in));
  AB200_LAUNCH_CHECK();
}

void launchTransferDynamicBuffer(float *buffer_col, float *mean_col, float *past_col,
                                 float *read_inout, int d_size, float lr_scale, float max_steps,
                                 float momentum, int forget_buffer, float buffer_cap,
                                 float sample_momentum, int previously_switched,
                                 unsigned char *chop_in, int col, const unsigned char *chop_out,
                                 int flip_in, cudaStream_t stream) {
  AB200_CUDA(launchChained(transferDynamicBufferKernel, dim3(1), dim3(256), 0, stream, buffer_col, mean_col,
                           past_col, read_inout, d_size, lr_scale, max_steps, momentum, forget_buffer,
                           buffer_cap, sample_momentum, previously_switched, chop_in, col, chop_out,
                           flip_in));
  AB200_LAUNCH_CHECK();
}

void launchFlipChoppers(unsigned char *chop, int n, float prob, PhiloxKey key, uint32_t call,
                        cudaStream_t stream) {
  AB200_CUDA(launchChained(flipChoppersKernel, dim3((n + 255) / 256), dim3(256), 0, stream, chop, n, prob, key,
                           call));
  AB200_LAUNCH_CHECK();
}

void launchTransferBuffer(float *buffer_col, float *read_inout, int d_size, float lr_abs,
                          float buffer_granularity, float max_steps, float momentum,
                          int forget_buffer, cudaStream_t stream) {
  AB200_CUDA(launchChained(transferBufferKernel, dim3((d_size + 255) / 256), dim3(256), 0, stream,
                           buffer_col, read_inout, d_size, lr_abs, buffer_granularity, max_steps,
                           momentum, forget_buffer));
  AB200_LAUNCH_CHECK();
}

void launchTransferRead(const float *w_fast, int col, int d_size, const IOEff &io, PhiloxKey key,
                        uint32_t call, float *x_onehot, int x_size, float *r_out, float alpha,
                        cudaStream_t stream) {
  int n = d_size > x_size ? d_size : x_size;
  AB200_CUDA(launchChained(transferReadKernel, dim3((n + 255) / 256), dim3(256), 0, stream, w_fast, col,
                           d_size, io, key, call, x_onehot, x_size, r_out, alpha));
  AB200_LAUNCH_CHECK();
}

// dst[c][r] = src[r][c]  (host [d][x] <-> device [x][d] conversions)
__global__ void transposeKernel(const float *src, float *dst, int rows, int cols) {
  __shared__ float tile[32][33];
  int c = blockIdx.x * 32 + threadIdx.x, r = blockIdx.y * 32 + threadIdx.y;
  for (int k = 0; k < 32; k += 8) {
    if (c < cols && r + k < rows) {
      tile[threadIdx.y + k][threadIdx.x] = src[(long long)(r + k) * cols + c];
    }
  }
  __syncthreads();
  int oc = blockIdx.y * 32 + threadIdx.x, orow = blockIdx.x * 32 + threadIdx.y;
  for (int k = 0; k < 32; k += 8) {
    if (oc < rows && orow + k < cols) {
      dst[(long long)(orow + k) * rows + oc] = tile[threadIdx.x][threadIdx.y + k];
    }
  }
}

void launchTransposeDX(const float *src, float *dst, int rows, int cols, cudaStream_t stream) {
  dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
  transposeKernel<<<grid, block, 0, stream>>>(src, dst, rows, cols);
  AB200_LAUNCH_CHECK();
}

// PulsedRPUDevice::onSetWeights: clip to the per-element bounds (rpu_pulsed_device.cpp:545-571).
__global__ void clipKernel(float *w, const float4 *par4, long long n) {
  pdlEnter();
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t < n) {
    float4 q = par4[t];
    w[t] = fmaxf(fminf(w[t], q.z), q.w);
  }
}

void launchClipToBounds(float *w, const float4 *par4, long long n, cudaStream_t stream) {
  AB200_CUDA(launchChained(clipKernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, w, par4, n));
  AB200_LAUNCH_CHECK();
}

// Throughput of the arithmetic a coincidence costs at the least - one AND, one population count,
// one add per pair of pulse words - with everything in registers and four independent chains per
// thread: the integer ceiling the update kernel's pair rate is reported against.
__global__ void __launch_bounds__(256) popcPeakKernel(uint32_t *sink, int iters) {
  uint32_t a0 = threadIdx.x * 2654435761u + 1u, a1 = a0 ^ 0x9E3779B9u, a2 = a0 + 0x7F4A7C15u,
           a3 = a1 * 3u;
  const uint32_t b = blockIdx.x * 40503u + 0x5bd1e995u;
  uint32_t c0 = 0, c1 = 0, c2 = 0, c3 = 0;
  for (int k = 0; k < iters; k++) {
#pragma unroll
    for (int u = 0; u < 8; u++) {
      c0 += __popc(a0 & (b + c3));
      c1 += __popc(a1 & (b + c0));
      c2 += __popc(a2 & (b + c1));
      c3 += __popc(a3 & (b + c2));
    }
  }
  if (c0 + c1 + c2 + c3 == 0xFFFFFFFFu) {
    sink[0] = c0; // never true in practice: keeps the loop alive
  }
}

double measurePopcPeak(cudaStream_t stream) {
  int dev = 0, n_sm = 0;
  AB200_CUDA(cudaGetDevice(&dev));
  AB200_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  uint32_t *sink = nullptr;
  AB200_CUDA(cudaMalloc(&sink, sizeof(uint32_t)));
  cudaEvent_t e0, e1;
  AB200_CUDA(cudaEventCreate(&e0));
  AB200_CUDA(cudaEventCreate(&e1));
  const int iters = 4096, blocks = n_sm * 8;
  popcPeakKernel<<<blocks, 256, 0, stream>>>(sink, 64); // warm-up
  AB200_CUDA(cudaEventRecord(e0, stream));
  popcPeakKernel<<<blocks, 256, 0, stream>>>(sink, iters);
  AB200_CUDA(cudaEventRecord(e1, stream));
  AB200_CUDA(cudaEventSynchronize(e1));
  float ms = 0.0f;
  AB200_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(sink);
  AB200_LAUNCH_CHECK();
  const double pairs = (double)blocks * 256.0 * (double)iters * 32.0;
  return pairs / ((double)ms * 1e-3);
}

__global__ void __launch_bounds__(256)
    addBlockKernel(const float *src, long long src_ld, float *dst, long long dst_ld, int cols,
                   long long n) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t < n) {
    const long long r = t / cols, c = t - r * cols;
    dst[r * dst_ld + c] += src[r * src_ld + c];
  }
}

void launchAddBlock(const float *src, long long src_ld, float *dst, long long dst_ld, int rows,
                    int cols, cudaStream_t stream) {
  const long long n = (long long)rows * cols;
  if (n <= 0) {
    return;
  }
  addBlockKernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(src, src_ld, dst, dst_ld, cols, n);
  AB200_LAUNCH_CHECK();
}

} // namespace ab200
