// IO-managed matrix-vector batch for small batches, CUDA cores, one launch per layer.
//
// A handful of rows through a matrix is bound by latency: noise management, DAC and product were two
// kernels per tile whose K loop waits for memory once per step, and a mapped layer ran its tiles one
// after the other. Here a CTA owns 4, 8 or 16 rows and 32 output columns, its sixteen warps share the K
// dimension of up to 512 features at a time, so that all weights a CTA needs are in flight at once,
// before the first input has arrived; the warp of a row reduces its statistics, quantises it into shared
// memory and later finishes its outputs. The tiles of a mapped layer are column blocks of one grid; the
// CTA walks the in-splits and adds their outputs after each tile's ADC (array.py:155-182), then the
// digital bias.
//
// Measured, 16 rows: 768 -> 3072 on 2 x 6 tiles 267 -> 15.4 us (24 launches -> 1), 1024 x 1024 42 -> 17.5 us, one row
// through 512 x 512 20 -> 5.4 us on the GPU. Bound by latency: a chain of load, reduce, quantise, product and output
// stage on sixteen warps per SM, 0.4 of the issue slots used; waits for shared memory, for the instruction before
// and at the barriers about alike.
//
// Weights, products and sums stay fp32. Element-wise semantics are the helpers of mvm_common.cuh, with the
// noise counters of the other kernels.
#include "mvm_common.cuh"
#include "tile.h"

#include <type_traits>

namespace ab200 {

constexpr int SM_WARPS = 16;
constexpr int SM_K = 512;            // features per step: 32 per warp at most
constexpr int SM_K_SHORT = 128;      // the same where a single tile has no more

// STRIDED (single tiles): the features of a row are not neighbours in memory (transposed inputs, [features][rows]).
// Neighbouring threads then load neighbouring rows, and the step goes through shared memory to the warps of the
// rows.
// STEP: features per step, SM_K or - for rows that end there - SM_K_SHORT, whose work in front of the product is a
// quarter (same sums; 64 x 64, 1000 rows: 6.8 -> 4.3 us).
template <int ROWS, bool K_FAST, bool STRIDED, int STEP, typename Splits>
__global__ void __launch_bounds__(32 * SM_WARPS) mvmSmallKernel(const __grid_constant__ MvmProblem p,
                                                                const __grid_constant__ Splits sp) {
  // prepared inputs of a step, later the partial sums of the warps
  constexpr int SE = ROWS * STEP / (32 * SM_WARPS); // elements of a strided step per thread
  constexpr int LD = STRIDED ? STEP + 4 : STEP; // (the rows of a feature in other banks)
  __shared__ __align__(16) float buf[ROWS * LD > SM_WARPS * ROWS * 32 ? ROWS * LD : SM_WARPS * ROWS * 32];
  const IOEff &io = p.io;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int o = 0;
  while ((int)blockIdx.x >= sp.col_blk[o + 1]) {
    o++;
  }
  const int N = sp.out_size[o];
  const int c = ((int)blockIdx.x - sp.col_blk[o]) * 32 + lane;
  const bool c_ok = c < N;
  const int row = blockIdx.y * ROWS + warp; // the row this warp prepares and finishes
  const bool mine = warp < ROWS && row < p.m;
  const uint64_t n4 = (uint64_t)(((N + 7) >> 3) << 1);
  const bool norm = !io.is_perfect && io.w_noise_type == AB200_WNOISE_ADDITIVE_CONSTANT && io.w_noise > 0.0f;
  const bool plain_dac = !io.is_perfect && !inputIsRandom(io) && io.inp_asym == 1.0f;
  const float inv_res = __fdiv_rn(1.0f, io.res_in); // (read with res_in > 0 only)
  pdlEnter();
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && !p.backward && p.bm_stats) {
    p.bm_stats[0] = 0; // counters of the bound-management re-run of this pass
    p.bm_stats[1] = 0;
  }

  // One step: up to 512 features of one tile. The loads of the next step are issued before the outputs of
  // a finished tile are worked out.
  float xr[STEP / 32], w[STEP / SM_WARPS];
  int ii = 0, k0 = 0;
  int K = sp.in_size[0], kn, kw, kb;
  const float *x_row = p.in + (long long)row * p.in_ss; // (read for rows of the batch only)
  auto load = [&]() {
    const SmallTile &t = sp.tile[ii * sp.n_out + o];
    kn = min(K - k0, STEP);
    kw = ((kn + SM_WARPS - 1) / SM_WARPS + 3) & ~3; // features per warp, in fours
    kb = warp * kw;                                 // this warp's first, within the step
    if (STRIDED) { // element q: row threadIdx.x % ROWS, feature threadIdx.x / ROWS + q * (threads / ROWS)
      const int r = blockIdx.y * ROWS + threadIdx.x % ROWS, f = threadIdx.x / ROWS;
      const float *x = p.in + (long long)r * p.in_ss + (long long)(k0 + f) * p.in_fs;
#pragma unroll
      for (int q = 0; q < SE; q++) {
        const int k = f + q * (32 * SM_WARPS / ROWS);
        xr[q] = 0.0f;
        if (r < p.m && k < kn) {
          xr[q] = 1.0f; // the bias line
          if (k0 + k < p.in_real) {
            xr[q] = *x;
          }
        }
        x += (32 * SM_WARPS / ROWS) * p.in_fs;
      }
    } else if (warp < ROWS) { // the inputs first: all that follows waits for them
      const int real = sp.n_in == 1 ? p.in_real - k0 : kn;
      const float *x = x_row + sp.in_off[ii] + k0 + lane;
#pragma unroll
      for (int q = 0; q < STEP / 32; q++) {
        xr[q] = 0.0f;
        if (mine && q * 32 + lane < kn) {
          xr[q] = 1.0f; // the bias line
          if (q * 32 + lane < real) {
            xr[q] = x[q * 32];
          }
        }
      }
    }
    const int n_mine = min(kw, kn - kb);
    if (K_FAST) {
      const float *wp = t.w + (c_ok ? c : 0) * t.ld + k0 + kb;
      if (sp.vec) { // n_mine is a multiple of four
#pragma unroll
        for (int q = 0; q < STEP / SM_WARPS; q += 4) {
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (q < n_mine) {
            v = *reinterpret_cast<const float4 *>(wp + q);
          }
          w[q] = v.x;
          w[q + 1] = v.y;
          w[q + 2] = v.z;
          w[q + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < STEP / SM_WARPS; q++) {
          w[q] = 0.0f;
          if (q < n_mine) {
            w[q] = wp[q];
          }
        }
      }
    } else {
      const float *wp = t.w + (k0 + kb) * t.ld + (c_ok ? c : 0);
#pragma unroll
      for (int q = 0; q < STEP / SM_WARPS; q++) {
        w[q] = 0.0f;
        if (q < n_mine) {
          w[q] = *wp;
        }
        wp += t.ld;
      }
    }
  };
  load();

  float acc[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    acc[r] = 0.0f;
  }
  float total = 0.0f, scale = 0.0f, sval = 0.0f, vn = 0.0f;
  const long long fs = STRIDED ? p.in_fs : 1;
  while (true) {
    if (STRIDED) {
#pragma unroll
      for (int q = 0; q < SE; q++) {
        buf[threadIdx.x % ROWS * LD + threadIdx.x / ROWS + q * (32 * SM_WARPS / ROWS)] = xr[q];
      }
      __syncthreads();
      if (warp < ROWS) {
#pragma unroll
        for (int q = 0; q < STEP / 32; q++) {
          xr[q] = buf[warp * LD + q * 32 + lane];
        }
      }
    }
    if (warp < ROWS) {
      const SmallTile &t = sp.tile[ii * sp.n_out + o];
      float *const v_row = buf + warp * LD;
      if (k0 == 0) {
        NmStats st;
        if (nmNeedsStats(io)) {
          if (io.nm == AB200_NM_ABS_MAX) {
#pragma unroll
            for (int q = 0; q < STEP / 32; q++) {
              st.amax = fmaxf(st.amax, fabsf(xr[q])); // (zeros past the end change no maximum of |x|)
            }
          } else {
#pragma unroll
            for (int q = 0; q < STEP / 32; q++) {
              if (q * 32 + lane < kn) {
                st.add(xr[q]);
              }
            }
          }
          if (mine) {
            const int real = sp.n_in == 1 ? p.in_real : K;
#pragma unroll 4
            for (int k = STEP + lane; k < K; k += 32) {
              st.add(k < real ? x_row[sp.in_off[ii] + k * fs] : 1.0f);
            }
          }
          if (io.nm == AB200_NM_ABS_MAX) {
            for (int s = 16; s > 0; s >>= 1) {
              st.amax = fmaxf(st.amax, __shfl_xor_sync(0xffffffffu, st.amax, s));
            }
          } else {
            st.warpReduce();
          }
        }
        sval = nmValue(io, st);
        scale = mine ? inputScale(io, sval, /*reduction=*/1.0f, !p.backward) : 0.0f;
        vn = 0.0f;
      }
      if (plain_dac) {
        // dacPlain without its branch: the few features next to a rounding tie are divided afterwards
        uint32_t ties = 0;
#pragma unroll
        for (int q = 0; q < STEP / 32; q++) {
          float v = __fmul_rn(xr[q], scale);
          const float f = __fmul_rn(v, inv_res), code = rintf(f);
          ties |= (fabsf(__fsub_rn(f, code)) > 0.4999f || !(fabsf(f) < 512.0f)) ? 1u << q : 0u;
          v = io.res_in > 0.0f ? __fmul_rn(code, io.res_in) : v;
          v = v > io.inp_bound ? io.inp_bound : v;
          v = v < -io.inp_bound ? -io.inp_bound : v;
          // (features past the end: zero whatever the scale, which is infinite for a row of very small numbers)
          v = scale != 0.0f && q * 32 + lane < kn ? v : 0.0f;
          xr[q] = v;
          v_row[q * 32 + lane] = v;
        }
        if (io.res_in > 0.0f && scale != 0.0f && ties != 0u) {
          const int real = sp.n_in == 1 ? p.in_real : K;
          const float *x = x_row + sp.in_off[ii];
#pragma unroll
          for (int q = 0; q < STEP / 32; q++) {
            const int k = k0 + q * 32 + lane;
            if (((ties >> q) & 1u) != 0u && q * 32 + lane < kn) {
              xr[q] = dacPlain(io, inv_res, k < real ? x[k * fs] : 1.0f, scale);
              v_row[q * 32 + lane] = xr[q];
            }
          }
        }
#pragma unroll
        for (int q = 0; q < STEP / 32; q++) {
          vn = fmaf(xr[q], xr[q], vn);
        }
      } else if (io.is_perfect) {
#pragma unroll
        for (int q = 0; q < STEP / 32; q++) {
          v_row[q * 32 + lane] = xr[q];
        }
      } else {
        const ElemRng g{t.key, t.call, (p.backward ? TAG_BWD_IN : TAG_FWD_IN) + t.noise_id};
#pragma unroll
        for (int q = 0; q < STEP / 32; q++) {
          v_row[q * 32 + lane] = xr[q];
        }
#pragma unroll 1
        for (int k = lane; k < STEP; k += 32) {
          float v = 0.0f;
          if (scale != 0.0f && k < kn) {
            v = prepareInput(io, v_row[k], scale, g, (uint32_t)row, (uint32_t)(k0 + k));
          }
          vn = fmaf(v, v, vn);
          v_row[k] = v;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < STEP / SM_WARPS; q += 4) {
      if (q < kw) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
          const float4 a = *reinterpret_cast<const float4 *>(buf + r * LD + kb + q);
          acc[r] = fmaf(a.x, w[q], acc[r]);
          acc[r] = fmaf(a.y, w[q + 1], acc[r]);
          acc[r] = fmaf(a.z, w[q + 2], acc[r]);
          acc[r] = fmaf(a.w, w[q + 3], acc[r]);
        }
      }
    }
    __syncthreads();
    const bool tile_done = k0 + STEP >= K;
    const int it = ii;
    if (tile_done) {
      ii++;
      k0 = 0;
      K = ii < sp.n_in ? sp.in_size[ii] : 0;
    } else {
      k0 += STEP;
    }
    const bool more = ii < sp.n_in;
    if (more) {
      load();
    }
    if (tile_done) {
      const SmallTile &t = sp.tile[it * sp.n_out + o];
#pragma unroll
      for (int r = 0; r < ROWS; r++) {
        buf[(warp * ROWS + r) * 32 + lane] = acc[r];
        acc[r] = 0.0f;
      }
      __syncthreads();
      if (mine) {
        float y = 0.0f;
#pragma unroll
        for (int wv = 0; wv < SM_WARPS; wv++) {
          y += buf[(wv * ROWS + warp) * 32 + lane];
        }
        if (norm) {
          for (int s = 16; s > 0; s >>= 1) {
            vn += __shfl_xor_sync(0xffffffffu, vn, s);
          }
          vn = sqrtf(vn);
        } else {
          vn = 0.0f;
        }
        const float fac = outputFactor(io, t.alpha, sval, scale, p.backward);
        bool exceeded = false;
        if (scale == 0.0f) {
          y = 0.0f;
        } else if (io.is_perfect) {
          y *= fac;
        } else {
          // (out_noise_std > 0: a standard deviation for every line)
          const float sigma = p.out_noise_vals != nullptr
                                  ? outputSigmaLine(io, vn, p.out_noise_vals, c_ok ? c : 0, 0.0f)
                                  : outputSigma(io, vn);
          const uint64_t blk = (uint64_t)row * n4 + (uint64_t)(c >> 2);
          const int q = lane & 3; // column blocks start at multiples of 32
          float z = 0.0f, uq = 0.5f;
          if (sigma > 0.0f) {
            z = gaussOf4(t.key, blk, t.call, (p.backward ? TAG_BWD_OUT : TAG_FWD_OUT) + t.noise_id, q);
          }
          if (io.out_sto_round) {
            float u[4];
            uniform4(t.key, blk, t.call, (p.backward ? TAG_BWD_OUT_U : TAG_FWD_OUT_U) + t.noise_id, u);
            uq = q == 0 ? u[0] : (q == 1 ? u[1] : (q == 2 ? u[2] : u[3]));
          }
          y = finalizeOutput(io, y, sigma, z, exceeded, uq) * fac;
        }
        total = it == 0 ? y : total + y;
        if (sp.n_in == 1) {
          if (exceeded && c_ok && io.bm != AB200_BM_NONE) {
            atomicOr(&p.flags[row], 1);
          }
          if (blockIdx.x == 0 && lane == 0 && p.scale) {
            // what the re-run reads; the flags are zero between passes (it clears those it has served)
            p.scale[row] = scale;
            p.sval[row] = sval;
            p.factor[row] = fac;
            p.vnorm[row] = vn;
          }
        }
      }
      if (!more) {
        break;
      }
      __syncthreads(); // the partial sums are read before the next tile's inputs replace them
    }
  }
  if (mine && c_ok) {
    const int col = sp.out_off[o] + c;
    if (sp.bias) {
      total += sp.bias[col];
    }
    if (col < p.out_store) {
      float *dst = mvmOutPtr(p, row, col);
      *dst = p.accumulate ? *dst + total : total;
    }
  }
}

static bool smallMvmTileIo(const IOEff &io) {
  const bool running = !io.is_perfect && (io.nm == AB200_NM_AVERAGE_ABS_MAX ||
                                          io.nm == AB200_NM_AVERAGE_ABS_MAX_SINGLE_VALUE);
  return !running && !ioNeedsLineChain(io);
}
bool smallMvmIo(const IOEff &io) { return smallMvmTileIo(io) && !ioLineSigma(io); }

static int smCount() {
  static int n_sm = 0; // SMs of the GPUs of this process (one kind per process)
  if (n_sm == 0) {
    int dev = 0;
    AB200_CUDA(cudaGetDevice(&dev));
    AB200_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  }
  return n_sm;
}

int smallMvmMaxCtas(int in_size) {
  // Four rounds of one CTA per SM; with more, the 64 x 64 tiles of the general kernel fill the GPU as well and
  // load less per product. 2048 x 2048, forward, this kernel against the general one: 16 rows (64 CTAs) 28
  // against 91 us, 64 rows (256) 56 against 179; 4096 x 4096, 32 rows (256) 109 against 367.
  // Short rows give a CTA little to hide its barriers behind: 64 x 64, 4000 rows (500 CTAs) 13.9 against 15.5 us, but
  // transposed 16.4 against 12.0, and 32 x 300, 900 rows (570) 13.8 against 11.2.
  return (in_size > 128 ? 4 : 2) * smCount();
}

template <int ROWS, bool STRIDED, int STEP, typename Splits>
static void launchKernel(const MvmProblem &p, const Splits &sp, bool k_fast, cudaStream_t stream) {
  dim3 grid(sp.col_blk[sp.n_out], (p.m + ROWS - 1) / ROWS);
  auto kernel = k_fast ? mvmSmallKernel<ROWS, true, STRIDED, STEP, Splits>
                       : mvmSmallKernel<ROWS, false, STRIDED, STEP, Splits>;
  AB200_CUDA(launchChained(kernel, grid, dim3(32 * SM_WARPS), 0, stream, p, sp));
  AB200_LAUNCH_CHECK();
}

template <int ROWS, typename Splits>
static void launchRows(const MvmProblem &p, const Splits &sp, bool k_fast, cudaStream_t stream) {
  if constexpr (std::is_same<Splits, SmallSplitsT<1, 1>>::value) {
    const bool strided = p.in_fs != 1;
    if (p.in_size <= SM_K_SHORT) {
      if (strided) {
        launchKernel<ROWS, true, SM_K_SHORT>(p, sp, k_fast, stream);
      } else {
        launchKernel<ROWS, false, SM_K_SHORT>(p, sp, k_fast, stream);
      }
      return;
    }
    if (strided) {
      launchKernel<ROWS, true, SM_K>(p, sp, k_fast, stream);
      return;
    }
  }
  launchKernel<ROWS, false, SM_K>(p, sp, k_fast, stream);
}

template <typename Splits> static void launchSplits(const MvmProblem &p, Splits &sp, cudaStream_t stream) {
  const bool k_fast = p.wn != 1;
  sp.vec = 1;
  for (int i = 0; i < sp.n_in; i++) {
    sp.vec &= (sp.in_size[i] & 3) == 0;
  }
  for (int i = 0; i < sp.n_in * sp.n_out; i++) {
    sp.vec &= (reinterpret_cast<uintptr_t>(sp.tile[i].w) & 15) == 0 && (sp.tile[i].ld & 3) == 0;
  }
  sp.col_blk[0] = 0;
  for (int i = 0; i < sp.n_out; i++) {
    sp.col_blk[i + 1] = sp.col_blk[i] + (sp.out_size[i] + 31) / 32;
  }
  if (p.m <= 4) {
    launchRows<4>(p, sp, k_fast, stream);
  } else if (p.m <= 8) {
    launchRows<8>(p, sp, k_fast, stream);
  } else {
    launchRows<16>(p, sp, k_fast, stream);
  }
}

void launchMvmSmall(const MvmProblem &p, SmallSplits &sp, cudaStream_t stream) { launchSplits(p, sp, stream); }

bool smallMvmEligible(const MvmProblem &p) {
  if ((p.wk != 1 && p.wn != 1) || p.gather.idx != nullptr || !smallMvmTileIo(p.io)) {
    return false;
  }
  return (long long)((p.out_size + 31) / 32) * ((p.m + 15) / 16) <= smallMvmMaxCtas(p.in_size);
}

bool smallMvmOneRound(const MvmProblem &p) {
  return smallMvmEligible(p) && p.out_noise_vals == nullptr && p.in_size <= SM_K &&
         (long long)((p.out_size + 31) / 32) * ((p.m + 15) / 16) <= smCount();
}

void launchMvmSmallTile(const MvmProblem &p, cudaStream_t stream) {
  SmallSplitsT<1, 1> sp{};
  sp.n_in = sp.n_out = 1;
  sp.in_size[0] = p.in_size;
  sp.out_size[0] = p.out_size;
  sp.tile[0] = SmallTile{p.w, p.wn != 1 ? p.wn : p.wk, p.alpha, p.call, p.noise_id, p.key};
  launchSplits(p, sp, stream);
}

} // namespace ab200
