// Pulsed update with stochastic trains, on bit planes.
//
//   pulseStatsKernel / pulseStatsGatherKernel
//                      per sample |x|max, |d|max -> train length BL and the probabilities' factors
//                      A, B (update management).
//   pulsePlanesKernel  the trains of 32 rows of every line as bit planes: plane 0 holds the signs of the 32
//                      rows, plane k their pulses in slot k. A row is a sample, or a segment of at most
//                      31 slots of it. Four planes of a line lie side by side, [block][plane / 4][line][4], so
//                      that one 16-byte load brings trains of up to three slots.
//   pulsedUpdatePlanesKernel
//                      a warp owns 32 d-lines of ONE x-line; AND of the two lines' planes gives the
//                      coincidences of 32 rows at a time.
//
// Update management shortens the trains to what a sample needs (BL = ceil(lr |x|max |d|max / dw_min)), one
// or two slots in ordinary training, so 32 rows take one or two ANDs where words per row took 32 ANDs,
// 32 population counts and 32 loads. Only planes up to the longest train of a block are written and read.
// Before, the words of a line were transposed and compacted to lists of (sample, word), two launches more.
// Measured, update of a 256 x 2304 SoftBounds tile with 131072 rows, gathered from images: 27.4 -> 18.3 ms; 1024 x
// 1024 Tiki-Taka step with 256 rows 407 -> 220 us.
#include "pulse_common.cuh"

#include <algorithm>

namespace ab200 {

// The problems of one launch: a tile, or tiles of a mapped layer along the last grid dimension. Grids are those
// of the largest tile.
template <int N> struct UpdateBatch {
  UpdateProblem tile[N];
};
#define AB200_BATCH_TILE(z) batch.tile[N == 1 ? 0 : (z)]

// ---------------------------------------------------------------------------------------------
// update management per sample
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void storeSampleParams(const UpdateProblem &p, int s, float xm, float dm) {
  if (s == 0) {
    *p.plane_max = 0; // the planes' kernel raises it
  }
  int BL;
  float A, B;
  blAB(p.up, p.lr, p.dw_min, xm, dm, BL, A, B);
  p.plane_bl[s] = BL;
  p.plane_ab[s] = make_float2(A, B);
}

// plain rows (any strides) and rows gathered through a row-major index array: one CTA per sample
template <int N>
__global__ void __launch_bounds__(128) pulseStatsKernel(const __grid_constant__ UpdateBatch<N> batch) {
  const UpdateProblem &p = AB200_BATCH_TILE(blockIdx.y);
  pdlEnter();
  __shared__ float sh[4];
  const int s = blockIdx.x;
  float xm = 0.0f, dm = 0.0f;
  if (p.up.update_management || p.up.update_bl_management) {
    if (p.gather.idx != nullptr) {
      for (int j = threadIdx.x; j < p.x_size; j += 128) {
        xm = fmaxf(xm, fabsf(gatherRowElement(p.gather, p.x, s, j)));
      }
    } else {
      const float *xr = p.x + (long long)s * p.x_ss;
#pragma unroll 8
      for (int j = threadIdx.x; j < p.x_real; j += 128) {
        xm = fmaxf(xm, fabsf(xr[(long long)j * p.x_fs]));
      }
      if (p.x_real < p.x_size) {
        xm = fmaxf(xm, 1.0f); // the bias line
      }
    }
    const float *dr = p.d + (long long)s * p.d_ss;
#pragma unroll 8
    for (int i = threadIdx.x; i < p.d_size; i += 128) {
      dm = fmaxf(dm, fabsf(dr[(long long)i * p.d_fs]));
    }
    // (rounding keeps the order, so the largest quotient is that of the largest value)
    dm = N > 1 && p.d_div != 0.0f ? fabsf(__fdiv_rn(dm, p.d_div)) : dm;
    xm = blockMax(xm, sh);
    dm = blockMax(dm, sh);
  }
  if (threadIdx.x == 0) {
    storeSampleParams(p, s, xm, dm);
  }
}

// Images gathered through an index array [x_size][m_batch]: lanes are 32 neighbouring positions, whose
// indices are contiguous and whose pixels nearly are, and the warps of the CTA share the x-lines.
__global__ void __launch_bounds__(1024) pulseStatsGatherKernel(UpdateProblem p) {
  pdlEnter();
  __shared__ float shx[32][33], shd[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s = blockIdx.x * 32 + lane;
  float xm = 0.0f;
  if (s < p.m) {
    const int n = s / p.gather.m_batch, l = s - n * p.gather.m_batch;
    const float *img = p.x + (long long)n * p.gather.image_size - 2;
    const int32_t *col = p.gather.idx_t + l;
#pragma unroll 6
    for (int k = warp; k < p.x_size; k += 32) {
      const int e = __ldg(col + (long long)k * p.gather.m_batch);
      xm = fmaxf(xm, e <= 1 ? (float)e : fabsf(__ldg(img + e)));
    }
  }
  shx[warp][lane] = xm;
  const int sd = blockIdx.x * 32 + warp;
  float dm = 0.0f;
  if (sd < p.m) {
    const float *dr = p.d + (long long)sd * p.d_ss;
#pragma unroll 8
    for (int i = lane; i < p.d_size; i += 32) {
      dm = fmaxf(dm, fabsf(dr[(long long)i * p.d_fs]));
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    dm = fmaxf(dm, __shfl_xor_sync(0xffffffffu, dm, o));
  }
  if (lane == 0) {
    shd[warp] = dm;
  }
  __syncthreads();
  if (warp == 0 && s < p.m) {
    xm = 0.0f;
#pragma unroll 8
    for (int w = 0; w < 32; w++) {
      xm = fmaxf(xm, shx[w][lane]);
    }
    storeSampleParams(p, s, xm, shd[lane]);
  }
}

// ---------------------------------------------------------------------------------------------
// trains of 32 rows as planes
// ---------------------------------------------------------------------------------------------
constexpr int PP_LINES = 64; // lines per CTA, eight per warp

// Lane = row: a ballot then yields one plane word of one line. The values are staged through shared
// memory where the rows are contiguous along the lines, and read directly where they are contiguous
// along the rows (transposed inputs, index arrays [x_size][m_batch]).
template <int N>
__global__ void __launch_bounds__(256) pulsePlanesKernel(const __grid_constant__ UpdateBatch<N> batch) {
  const UpdateProblem &p = AB200_BATCH_TILE(blockIdx.y);
  pdlEnter();
  __shared__ float tile[PP_LINES][33];
  __shared__ uint32_t planes[32][PP_LINES + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nseg = p.nseg > 0 ? p.nseg : 1;
  const int n_xchunk = (p.x_size + PP_LINES - 1) / PP_LINES;
  const int n_chunk = n_xchunk + (p.d_size + PP_LINES - 1) / PP_LINES;
  const int blk = (int)(blockIdx.x / (unsigned)n_chunk), chunk = (int)(blockIdx.x - (unsigned)blk * n_chunk);
  if (N > 1 && blk * 32 >= p.m * nseg) {
    return;
  }
  const bool is_x = chunk < n_xchunk;
  const int line0 = (is_x ? chunk : chunk - n_xchunk) * PP_LINES;
  const int n_lines = is_x ? p.x_size : p.d_size;
  const int real = is_x ? p.x_real : p.d_size;
  const float *src = is_x ? p.x : p.d;
  const long long ss = is_x ? p.x_ss : p.d_ss, fs = is_x ? p.x_fs : p.d_fs;
  const bool gathered = is_x && p.gather.idx != nullptr;
  const bool divide = N > 1 && !is_x && p.d_div != 0.0f; // (only tiles of a layer have scales)
  const bool gather_t = gathered && p.gather.idx_t != nullptr;
  const bool direct = gather_t || (!gathered && ss == 1 && fs != 1);

  const int row = blk * 32 + lane;
  const int s = nseg == 1 ? row : row / nseg;
  const int seg = nseg == 1 ? 0 : row - s * nseg;
  const bool row_ok = s < p.m;
  const int BL = row_ok ? p.plane_bl[s] : 0;
  float P = 0.0f;
  if (row_ok) {
    const float2 ab = p.plane_ab[s];
    P = is_x ? ab.y : ab.x;
  }
  const int nk = max(min(BL - seg * kPulseSegSlots, kPulseSegSlots), 0);
  const int nk_max = __reduce_max_sync(0xffffffffu, nk);
  if (chunk == 0 && threadIdx.x == 0) {
    p.plane_nk[blk] = nk_max;
    if (nk_max > 3) {
      atomicMax(p.plane_max, nk_max);
    }
  }

  if (!direct) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int rr = warp * 4 + q;
      const int rs = (blk * 32 + rr) / nseg;
#pragma unroll
      for (int h = 0; h < PP_LINES; h += 32) {
        const int line = line0 + h + lane;
        float v = 0.0f;
        if (rs < p.m && line < n_lines) {
          if (gathered) {
            v = gatherRowElement(p.gather, p.x, rs, line);
          } else {
            v = line < real ? src[(long long)rs * ss + (long long)line * fs] : 1.0f;
            v = divide ? __fdiv_rn(v, p.d_div) : v;
          }
        }
        tile[h + lane][rr] = v;
      }
    }
    __syncthreads();
  }
  int img_n = 0, img_l = 0;
  if (gather_t && row_ok) {
    img_n = s / p.gather.m_batch;
    img_l = s - img_n * p.gather.m_batch;
  }
  float v[PP_LINES / 8];
#pragma unroll
  for (int q = 0; q < PP_LINES / 8; q++) {
    const int ll = warp * (PP_LINES / 8) + q, line = line0 + ll;
    v[q] = 0.0f;
    if (!direct) {
      v[q] = tile[ll][lane];
    } else if (row_ok && line < n_lines) {
      if (gather_t) {
        const int e = __ldg(p.gather.idx_t + (long long)line * p.gather.m_batch + img_l);
        v[q] = e <= 1 ? (float)e : __ldg(p.x + (long long)img_n * p.gather.image_size + (e - 2));
      } else {
        v[q] = line < real ? src[s + (long long)line * fs] : 1.0f;
        v[q] = divide ? __fdiv_rn(v[q], p.d_div) : v[q];
      }
    }
  }
  const uint32_t tag = is_x ? TAG_PULSE_X : TAG_PULSE_D;
  const uint32_t flip = (!is_x && p.lr_neg) ? 1u : 0u;
  const bool plain = !(p.up.res > 0.0f);
#pragma unroll
  for (int q = 0; q < PP_LINES / 8; q++) {
    const int ll = warp * (PP_LINES / 8) + q;
    const uint32_t line = (uint32_t)(line0 + ll);
    // the train of pulseTrain (pulse_common.cuh), slot by slot across the 32 rows
    float pp = __fmul_rn(fabsf(v[q]), P);
    if (!plain) {
      pp = pulseProb(p, pp, p.up.res, line, (uint32_t)s, tag);
    }
    const int thr = pulseThreshold(pp);
    const uint32_t signs = __ballot_sync(0xffffffffu, ((v[q] > 0.0f ? 0u : 1u) ^ flip) != 0u);
    uint32_t mine = lane == 0 ? signs : 0u;
    for (int k0 = 0; k0 < nk_max; k0 += 8) {
      uint32_t r[4];
      philox4x32<7>(line, (uint32_t)s, p.call, tag + (uint32_t)(seg * 4 + (k0 >> 3)), p.key, r);
#pragma unroll
      for (int h = 0; h < 4; h++) {
        if (k0 + 2 * h < nk_max) {
          const uint32_t lo =
              __ballot_sync(0xffffffffu, k0 + 2 * h < nk && (int)(r[h] & 0xffffu) < thr);
          const uint32_t hi =
              __ballot_sync(0xffffffffu, k0 + 2 * h + 1 < nk && (int)(r[h] >> 16) < thr);
          mine = lane == k0 + 2 * h + 1 ? lo : mine;
          mine = lane == k0 + 2 * h + 2 ? hi : mine;
        }
      }
    }
    planes[lane][ll] = mine;
  }
  __syncthreads();
  uint4 *dst = reinterpret_cast<uint4 *>(is_x ? p.xw : p.dw) + (long long)blk * 8 * n_lines + line0;
  for (int t = threadIdx.x; t < (nk_max / 4 + 1) * PP_LINES; t += 256) {
    const int g = t / PP_LINES, l = t % PP_LINES;
    if (line0 + l < n_lines) {
      dst[(long long)g * n_lines + l] =
          make_uint4(planes[4 * g][l], planes[4 * g + 1][l], planes[4 * g + 2][l], planes[4 * g + 3][l]);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// the update
// ---------------------------------------------------------------------------------------------
constexpr int UP_WARPS = 4;   // x-lines per CTA (neighbours share the sectors of the x planes)
constexpr int UP_POOL = kNoisePool; // Gaussians per warp pool (eight per lane and refill)
// most refills per row: 31 pulses of 32 weights, and up to 31 values of a pool are left when it is refilled
constexpr uint32_t UP_ROW_REFILLS = 5;
static_assert(kPulseSegSlots * 32 <= (int)UP_ROW_REFILLS * (UP_POOL - 31), "room for the refills of a row");
constexpr int UP_DRAIN = 20;  // a lane with more events than this has the warp apply all events
constexpr int UP_EVENTS = 24; // most events of a lane between two drains

struct UpdatePlanesSmem {
  float pool[UP_WARPS][kNoisePoolRow];
  uint8_t counts[UP_WARPS][UP_EVENTS][32]; // pulses of the events that have more than one
};

// Eight fresh Gaussians per lane for a warp's pool, as offset + std * z. Out of line: rare against the pulses
// that take from the pool at two places, and the largest piece of code among them.
__device__ __noinline__ void refillPool(PhiloxKey key, uint64_t pair, uint32_t call, float std, float offset,
                                        float *column) {
  float z[8];
  gauss8(key, pair, call, TAG_DEVICE, z);
#pragma unroll
  for (int rr = 0; rr < 8; rr++) {
    column[rr * 32] = __fadd_rn(offset, __fmul_rn(std, z[rr]));
  }
}

// Per block of 32 rows a lane gets one word of coincidences and appends their directions to a queue of
// bits in a register. The pulses are applied in rounds, one event per
// lane and round, oldest first, one pulse at a time with the clip after each as in
// rpu_weight_updater.cpp:243-291; Gaussians of the device noise come from a pool per warp that all lanes
// refill together and take from without gaps (ballot + prefix count). Rounds start when, after a group of
// four rows in which the x-line pulsed, a lane holds more than UP_DRAIN events: that point fixes
// which Gaussian an event gets, so it is found exactly, also inside a word.
//
// Bound by instructions (0.75 of the issue slots used): about 60 per block of 32 rows, 45 per round, and 150 per
// refill; the busiest lane sets the number of rounds, 0.66 of the lanes have an event in one. A list of
// {coincidences, directions} words in shared memory instead of the queue of bits took 7 % fewer instructions
// and the same time (24 instead of 32 warps per SM).
//
// SHORT: a range of one row, of a batch that transfers cut up; x-lines without a pulse in it are left out before
// their weights are read.
template <int KIND, bool NOISY, bool MULT, int N, bool SHORT>
__global__ void __launch_bounds__(32 * UP_WARPS, 8)
    pulsedUpdatePlanesKernel(const __grid_constant__ UpdateBatch<N> batch) {
  const UpdateProblem &p = AB200_BATCH_TILE(blockIdx.y);
  pdlEnter();
  __shared__ UpdatePlanesSmem sm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_dblk = (p.d_size + 31) >> 5;
  const int jg = (int)(blockIdx.x / (unsigned)n_dblk), dblk = (int)(blockIdx.x - (unsigned)jg * n_dblk);
  const int j = jg * UP_WARPS + warp;
  if (j >= p.x_size) {
    return;
  }
  const long long task = (long long)j * n_dblk + dblk;
  const int i = dblk * 32 + lane;
  const bool i_ok = i < p.d_size;
  const long long idx = (long long)j * p.d_size + (i_ok ? i : 0);
  if (SHORT && *p.plane_max <= 3) {
    // an x-line without a pulse in the range leaves the weights and their parameters where they are
    const uint4 xv = reinterpret_cast<const uint4 *>(p.xw)[(long long)(p.s_begin >> 5) * 8 * p.x_size + j];
    const uint32_t rows = (0xffffffffu << (p.s_begin & 31)) & (0xffffffffu >> (31 - ((p.s_end - 1) & 31)));
    if (((xv.y | xv.z | xv.w) & rows) == 0u) {
      return;
    }
  }
  float w = 0.0f;
  PulseStep<KIND> step;
  {
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    float2 e = make_float2(0.f, 0.f);
    if (i_ok) {
      w = p.w[idx];
      q = p.par4[idx];
      if (KIND != AB200_DEVICE_CONSTANT_STEP && KIND != AB200_DEVICE_EXP_STEP &&
          KIND != AB200_DEVICE_PIECEWISE_STEP) {
        e = p.par2[idx];
      }
    }
    step.set(q, e);
    step.prepare(w, i_ok);
  }
  const float w_in = w;
  const float std = p.dw_min_std;
  // chopped transfer compound: direction flipped when exactly one of the two lines is chopped
  uint32_t flip = 0xffffffffu; // equal line signs = decrease (rpu_weight_updater.cpp:246-268)
  if (p.chop_x != nullptr && (p.chop_x[j] != 0) != (i_ok && p.chop_d[i] != 0)) {
    flip = 0u;
  }
  float *const pool = sm.pool[warp];
  uint8_t *const counts = &sm.counts[warp][0][lane];
  int cnt = 0;        // events in the queue
  uint32_t queue = 0; // their directions, the newest in bit 0
  uint32_t multi = 0; // events (by ordinal) of more than one pulse,
  uint32_t triple = 0; // and of three (where trains are longer, the counts are in shared memory)
  const bool deep = *p.plane_max > 3; // some train has more slots than the first four planes hold
  int pool_pos = UP_POOL; // empty
  // Refills are numbered over the whole batch: a batch in which transfers fall is applied in ranges of its rows, a
  // launch each, and a row takes no more than UP_ROW_REFILLS.
  uint32_t refills = UP_ROW_REFILLS * (uint32_t)p.s_begin;
  const uint32_t lt_mask = (1u << lane) - 1u;

  // one pulse for the lanes in `act`
  auto pulse = [&](bool act, bool down) {
    float xi = PulseStep<KIND>::kOnePlus ? 1.0f : 0.0f;
    if (NOISY) {
      const uint32_t takers = __ballot_sync(0xffffffffu, act);
      const int n_take = __popc(takers);
      if (pool_pos + n_take > UP_POOL) {
        // all lanes refill together; what is left of the old pool is dropped
        __syncwarp();
        refillPool(p.key, (uint64_t)(task * 32 + lane) | ((uint64_t)refills << 40), p.call, std,
                   PulseStep<KIND>::kOnePlus ? 1.0f : 0.0f, pool + lane);
        __syncwarp();
        refills++;
        pool_pos = 0;
      }
      xi = pool[noisePoolSlot(pool_pos, takers, lane)];
      pool_pos += n_take;
    }
    const float w_new = step.apply(p, w, down, xi, MULT);
    w = act ? w_new : w;
  };

  auto drain = [&]() {
    const int rounds = __reduce_max_sync(0xffffffffu, cnt);
    uint32_t multi_any = __reduce_or_sync(0xffffffffu, multi);
    queue = __funnelshift_lc(0u, queue, 32 - cnt); // the oldest first
    for (int r = 0; r < rounds; r++) {
      const bool down = (int)queue < 0;
      queue <<= 1;
      pulse(r < cnt, down);
      if ((multi_any & 1u) != 0u) {
        int n = 0;
        if (((multi >> r) & 1u) != 0u) {
          n = deep ? counts[r * 32] : 2 + (int)((triple >> r) & 1u);
        }
        for (int k = 1; __any_sync(0xffffffffu, k < n); k++) {
          pulse(k < n, down);
        }
      }
      multi_any >>= 1;
    }
    cnt = 0;
    queue = 0u;
    multi = triple = 0u;
  };

  const int b_first = p.s_begin >> 5, b_last = (p.s_end - 1) >> 5;
  const uint4 *xb = reinterpret_cast<const uint4 *>(p.xw) + (long long)b_first * 8 * p.x_size + j;
  const uint4 *db = reinterpret_cast<const uint4 *>(p.dw) + (long long)b_first * 8 * p.d_size + (i_ok ? i : 0);
  const long long x_step = 8LL * p.x_size, d_step = 8LL * p.d_size;
  // rows of the first / last block outside of [s_begin, s_end)
  const uint32_t rows_first = 0xffffffffu << (p.s_begin & 31);
  const uint32_t rows_last = 0xffffffffu >> (31 - ((p.s_end - 1) & 31));
  const uint32_t lane_on = i_ok ? 0xffffffffu : 0u;
  uint32_t rank0 = 0; // pulsing rows of the x-line before this block, from s_begin on
  uint32_t group = 0; // group in which a lane has passed the mark

  auto push = [&](uint32_t ev, uint32_t dir) {
    // (most words hold no more than a few events: the first three without a branch)
#pragma unroll
    for (int u = 0; u < 3; u++) {
      const uint32_t rest = ev & (ev - 1u);
      const uint32_t next = queue * 2u + ((dir & (ev ^ rest)) != 0u ? 1u : 0u);
      queue = ev != 0u ? next : queue;
      ev = rest;
    }
    while (ev != 0u) {
      const uint32_t rest = ev & (ev - 1u);
      queue = queue * 2u + ((dir & (ev ^ rest)) != 0u ? 1u : 0u);
      ev = rest;
    }
  };
  // the events of more than one pulse among `ev`, which start at ordinal `before`; c0..c4 the bits of the counts
  auto pushCounts = [&](uint32_t more, uint32_t ev, int before, uint32_t c0) {
    while (more != 0u) {
      const uint32_t bit = more & (0u - more);
      more ^= bit;
      const uint32_t at = 1u << (before + __popc(ev & (bit - 1u)));
      multi |= at;
      triple |= (c0 & bit) != 0u ? at : 0u;
    }
  };
  auto pushDeepCounts = [&](uint32_t more, uint32_t ev, int before, uint32_t c0, uint32_t c1, uint32_t c2,
                            uint32_t c3, uint32_t c4) {
    while (more != 0u) {
      const uint32_t bit = more & (0u - more);
      more ^= bit;
      const int at = before + __popc(ev & (bit - 1u));
      counts[at * 32] = (uint8_t)(((c0 & bit) ? 1 : 0) + ((c1 & bit) ? 2 : 0) + ((c2 & bit) ? 4 : 0) +
                                  ((c3 & bit) ? 8 : 0) + ((c4 & bit) ? 16 : 0));
      multi |= 1u << at;
    }
  };

  int b = b_first;
  while (true) {
    // Two inner blocks at a time as long as no lane fills up in them and no train of theirs is longer than
    // three slots.
    while (b > b_first && b + 1 < b_last && (!deep || (p.plane_nk[b] <= 3 && p.plane_nk[b + 1] <= 3))) {
      const uint4 x0 = xb[0], x1 = xb[x_step], d0 = db[0], d1 = db[d_step];
      const uint32_t p0 = x0.y & d0.y, p1 = x0.z & d0.z, p2 = x0.w & d0.w;
      const uint32_t q0 = x1.y & d1.y, q1 = x1.z & d1.z, q2 = x1.w & d1.w;
      const uint32_t any0 = (p0 | p1 | p2) & lane_on, any1 = (q0 | q1 | q2) & lane_on;
      const int n0 = __popc(any0), n1 = __popc(any1);
      if (__any_sync(0xffffffffu, cnt + n0 + n1 > UP_DRAIN)) {
        break;
      }
      push(any0, x0.x ^ d0.x ^ flip);
      push(any1, x1.x ^ d1.x ^ flip);
      const uint32_t m0 = (p0 & p1) | (p0 & p2) | (p1 & p2), m1 = (q0 & q1) | (q0 & q2) | (q1 & q2);
      if (((m0 | m1) & lane_on) != 0u) {
        if (deep) {
          pushDeepCounts(m0 & lane_on, any0, cnt, p0 ^ p1 ^ p2, m0, 0u, 0u, 0u);
          pushDeepCounts(m1 & lane_on, any1, cnt + n0, q0 ^ q1 ^ q2, m1, 0u, 0u, 0u);
        } else {
          pushCounts(m0 & lane_on, any0, cnt, p0 ^ p1 ^ p2);
          pushCounts(m1 & lane_on, any1, cnt + n0, q0 ^ q1 ^ q2);
        }
      }
      cnt += n0 + n1;
      rank0 += (uint32_t)(__popc(x0.y | x0.z | x0.w) + __popc(x1.y | x1.z | x1.w));
      b += 2;
      xb += 2 * x_step;
      db += 2 * d_step;
    }
    // One block; after the last one a turn that applies what is left.
    const bool end = b > b_last;
    uint32_t any = 0, dir = 0, xnz = 0, c0 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0;
    if (!end) {
      const uint4 xv = *xb, dv = *db;
      // coincidences and, in c0..c4, the bits of their pulse counts
      dir = xv.x ^ dv.x ^ flip;
      xnz = xv.y | xv.z | xv.w;
      const uint32_t a1 = xv.y & dv.y, a2 = xv.z & dv.z, a3 = xv.w & dv.w;
      any = a1 | a2 | a3;
      c0 = a1 ^ a2 ^ a3;
      c1 = (a1 & a2) | (a1 & a3) | (a2 & a3);
      if (deep) {
        const int nk = p.plane_nk[b];
        const uint4 *xg = xb, *dg = db;
        for (int k = 4; k <= nk; k += 4) {
          xg += p.x_size;
          dg += p.d_size;
          const uint4 xk = *xg, dk = *dg;
          const uint32_t a[4] = {xk.x & dk.x, xk.y & dk.y, xk.z & dk.z, xk.w & dk.w};
          xnz |= xk.x | xk.y | xk.z | xk.w;
#pragma unroll
          for (int u = 0; u < 4; u++) {
            any |= a[u];
            const uint32_t t0 = c0 & a[u];
            c0 ^= a[u];
            const uint32_t t1 = c1 & t0;
            c1 ^= t0;
            const uint32_t t2 = c2 & t1;
            c2 ^= t1;
            const uint32_t t3 = c3 & t2;
            c3 ^= t2;
            c4 ^= t3;
          }
        }
      }
      xnz &= b == b_first ? rows_first : 0xffffffffu;
      xnz &= b == b_last ? rows_last : 0xffffffffu;
      any &= xnz & lane_on;
    }
    const uint32_t rank_end = rank0 + (uint32_t)__popc(xnz);
    while (true) {
      // events of this word that belong to the list being filled
      uint32_t ev = any;
      const int total = cnt + __popc(any);
      bool full = __any_sync(0xffffffffu, total > UP_DRAIN);
      if (full && !end) {
        // the group of four pulsing rows in which the first lane passes the mark
        uint32_t g = 0xffffffffu;
        if (total > UP_DRAIN) {
          if (cnt > UP_DRAIN) {
            g = group; // passed it in an earlier word, in a group that goes on in this one
          } else {
            uint32_t t = any;
            for (int k = cnt; k < UP_DRAIN; k++) {
              t &= t - 1u;
            }
            const uint32_t at = t & (0u - t);
            g = (rank0 + (uint32_t)__popc(xnz & (at - 1u))) >> 2;
          }
        }
        group = __reduce_min_sync(0xffffffffu, g);
        full = rank_end >= 4u * group + 4u; // else the group ends in a later word
        if (full) {
          // rows of this word up to the end of the group
          ev &= __ballot_sync(0xffffffffu, rank0 + (uint32_t)__popc(xnz & lt_mask) < 4u * group + 4u);
        }
      }
      if (ev != 0u) {
        push(ev, dir);
        if (deep) {
          pushDeepCounts(ev & (c1 | c2 | c3 | c4), ev, cnt, c0, c1, c2, c3, c4);
        } else {
          pushCounts(ev & c1, ev, cnt, c0);
        }
        cnt += __popc(ev);
      }
      if (!full && !end) {
        break;
      }
      drain();
      any ^= ev;
      if (end) {
        break;
      }
    }
    if (end) {
      break;
    }
    rank0 = rank_end;
    b++;
    xb += x_step;
    db += d_step;
  }
  if (i_ok && w != w_in) {
    p.w[idx] = w;
  }
}

template <int KIND, bool NOISY, bool MULT, int N>
static void launchPlanesInstance(const UpdateBatch<N> &batch, int n, cudaStream_t stream) {
  long long blocks = 0;
  for (int k = 0; k < n; k++) {
    const UpdateProblem &p = batch.tile[k];
    blocks = std::max(blocks, (long long)((p.d_size + 31) / 32) * ((p.x_size + UP_WARPS - 1) / UP_WARPS));
  }
  auto kernel = pulsedUpdatePlanesKernel<KIND, NOISY, MULT, N, false>;
  const UpdateProblem &p = batch.tile[0];
  // Weights and parameters of a large tile are most of what a launch over one row takes: a transfer after every row,
  // us per 64 rows, 1024 x 1024 2764 -> 2481, 512 x 512 1096 -> 1077. In small tiles and with more rows the look at the
  // line first costs more than it spares (64 x 64 566 -> 599; 1024 x 1024, a transfer after five rows, 627 -> 643).
  if (N == 1 && p.m > 1 && p.s_end - p.s_begin == 1 && (long long)p.x_size * p.d_size >= 1 << 18) {
    kernel = pulsedUpdatePlanesKernel<KIND, NOISY, MULT, N, N == 1>;
  }
  AB200_CUDA(launchChained(kernel, dim3((unsigned)blocks, n), dim3(32 * UP_WARPS), 0, stream, batch));
}

template <int KIND, int N> static void launchPlanesKind(const UpdateBatch<N> &batch, int n, cudaStream_t stream) {
  const UpdateProblem &p = batch.tile[0];
  // (the two rules that have it multiply the noise with the step or add it)
  constexpr bool can_mult = KIND == AB200_DEVICE_LINEAR_STEP || KIND == AB200_DEVICE_SOFT_BOUNDS_REFERENCE;
  const bool mult = can_mult && p.mult_noise != 0;
  if (p.dw_min_std > 0.0f) {
    if (mult) {
      launchPlanesInstance<KIND, true, can_mult>(batch, n, stream);
    } else {
      launchPlanesInstance<KIND, true, false>(batch, n, stream);
    }
  } else if (mult) {
    launchPlanesInstance<KIND, false, can_mult>(batch, n, stream);
  } else {
    launchPlanesInstance<KIND, false, false>(batch, n, stream);
  }
}

template <int N> static void launchPlanesOf(const UpdateBatch<N> &batch, int n, cudaStream_t stream) {
  const UpdateProblem &p0 = batch.tile[0];
  if (p0.gather.idx != nullptr && p0.gather.idx_t != nullptr) {
    AB200_CUDA(launchChained(pulseStatsGatherKernel, dim3((p0.m + 31) / 32), dim3(1024), 0, stream, p0));
  } else {
    AB200_CUDA(launchChained(pulseStatsKernel<N>, dim3(p0.m, n), dim3(128), 0, stream, batch));
  }
  AB200_LAUNCH_CHECK();
  long long blocks = 0;
  for (int k = 0; k < n; k++) {
    const UpdateProblem &p = batch.tile[k];
    const long long n_blk = (p.m * (p.nseg > 0 ? p.nseg : 1) + 31) / 32;
    blocks = std::max(blocks, n_blk * ((p.x_size + PP_LINES - 1) / PP_LINES + (p.d_size + PP_LINES - 1) / PP_LINES));
  }
  AB200_CUDA(launchChained(pulsePlanesKernel<N>, dim3((unsigned)blocks, n), dim3(256), 0, stream, batch));
  AB200_LAUNCH_CHECK();
}

template <int N> static void launchUpdateOf(const UpdateBatch<N> &batch0, int n, cudaStream_t stream) {
  UpdateBatch<N> batch = batch0;
  for (int k = 0; k < n; k++) {
    batch.tile[k] = inRows(batch0.tile[k]);
  }
  switch (batch.tile[0].kind) {
  case AB200_DEVICE_CONSTANT_STEP:
    launchPlanesKind<AB200_DEVICE_CONSTANT_STEP>(batch, n, stream);
    break;
  case AB200_DEVICE_LINEAR_STEP:
  case AB200_DEVICE_SOFT_BOUNDS:
    launchPlanesKind<AB200_DEVICE_LINEAR_STEP>(batch, n, stream);
    break;
  case AB200_DEVICE_SOFT_BOUNDS_REFERENCE:
    launchPlanesKind<AB200_DEVICE_SOFT_BOUNDS_REFERENCE>(batch, n, stream);
    break;
  case AB200_DEVICE_POW_STEP:
    launchPlanesKind<AB200_DEVICE_POW_STEP>(batch, n, stream);
    break;
  case AB200_DEVICE_EXP_STEP:
    launchPlanesKind<AB200_DEVICE_EXP_STEP>(batch, n, stream);
    break;
  case AB200_DEVICE_PIECEWISE_STEP:
    launchPlanesKind<AB200_DEVICE_PIECEWISE_STEP>(batch, n, stream);
    break;
  default:
    AB200_FATAL("pulsed update: device kind not implemented");
  }
  AB200_LAUNCH_CHECK();
}

void launchPulsePlanes(const UpdateProblem &p, cudaStream_t stream) {
  launchPlanesOf(UpdateBatch<1>{{p}}, 1, stream);
}

void launchPulsedUpdatePlanes(const UpdateProblem &p, cudaStream_t stream) {
  if (p.s_end > p.s_begin) {
    launchUpdateOf(UpdateBatch<1>{{p}}, 1, stream);
  }
}

void launchPulsedUpdateTiles(const UpdateProblem *p, int n, cudaStream_t stream) {
  if (n == 1 && p[0].d_div == 0.0f) { // (the kernels of single tiles divide nothing)
    launchPulsePlanes(p[0], stream);
    launchPulsedUpdatePlanes(p[0], stream);
    return;
  }
  if (n < 1 || n > kUpdateBatch) {
    AB200_FATAL("pulsed update: invalid number of tiles in a launch");
  }
  UpdateBatch<kUpdateBatch> batch{};
  std::copy(p, p + n, batch.tile);
  launchPlanesOf(batch, n, stream);
  launchUpdateOf(batch, n, stream);
}

} // namespace ab200
