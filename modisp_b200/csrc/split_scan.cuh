// split_scan.cuh -- the single-precision scan as rounds of separate kernels.
//
// The fused scan (scan<float, WAVE>) runs one trace per warp from start to end:
// each 32-sample step computes positions, evaluates them, re-evaluates the
// sign-uncertain ones in FP64 and does the bookkeeping, all latency-bound
// work of one warp.  Here the same steps run as rounds over an active set of
// traces, each stage with the parallel shape that suits it:
//   split_feed_count/fill  the active set refilled from the trace list (new
//                          traces start from scan_start)
//   split_positions        one warp per trace: the next SPLIT_STEPS steps'
//                          positions, merged exactly as the fused scan merges
//                          them (scan_positions, scan_position32)
//   split_eval32_pair      one thread per two samples of a trace, evaluated
//                          together in paired FP32 instructions (sm_100 .f32x2);
//                          the near-cutoff band takes the trace's FP64 tail
//                          values; sign-uncertain samples are listed for FP64
//   split_redo             one thread per listed sample: its FP64 value
//   split_book             one thread per trace: the samples in order through
//                          the fused scan's bookkeeping (sign changes, regular
//                          samples, trough tests), brackets appended; a trough
//                          that needs a window pauses the trace at that sample,
//                          the last cell of a finished trace is requested too
//   split_zoom             one warp per request: the FP32 screen and the FP64
//                          zoom of a trough window (screen_trough32,
//                          zoom_trough), or the last cell (last_cell)
// Every sample goes through the same arithmetic and every decision through the
// same rule as in the fused scan, in the same order, so the brackets -- and the
// roots -- are the fused scan's bit for bit.  The state between rounds is the
// fused scan's ScanState; a paused trace resumes from its cursors (the samples
// after the pause are positioned and evaluated again).  Traces still unfinished
// after the last round, and any the rounds never reached, are finished by the
// fused kernel (resume mode).
#pragma once
#include "kernels.cuh"

namespace md200 {

// Compile-time tuning: 32-sample steps per trace per round (two measured best:
// fewer samples evaluated past a trace's last bracket than four, half the rounds of
// one; the paired evaluation takes one sample of each); the evaluation kernel's
// minimum resident CTAs per SM (Rayleigh 4: 128 registers; 3 CTAs ran 10 % slower,
// 5 CTAs 2 %.  Love 6: 8 ran 3 % slower, 5 the same) and its grid in CTAs per SM
// (64: 2.4 % faster than 16, 128 no faster; a warp then takes a few traces).
#ifndef MD200_SPLIT_PAIR_BLOCKS
#define MD200_SPLIT_PAIR_BLOCKS 4
#endif
#ifndef MD200_SPLIT_PAIR_BLOCKS_LOVE
#define MD200_SPLIT_PAIR_BLOCKS_LOVE 6
#endif
#ifndef MD200_SPLIT_PAIR_GRID
#define MD200_SPLIT_PAIR_GRID 64
#endif
constexpr int SPLIT_STEPS = 2;                    // 32-sample steps per trace per round
constexpr int SPLIT_SAMPLES = 32 * SPLIT_STEPS;  // sample slots per active trace
constexpr int SPLIT_ACTIVE_MAX = 1 << 20;         // active-set capacity (traces)
// Runs with fewer traces use the fused kernel.  Scan stage, fused against split, five
// modes: Rayleigh 9,000 traces 0.58 / 0.75 ms, 17,400 1.01 / 1.01, 24,000 1.37 / 1.24,
// 150,000 8.2 / 5.0, 1.2 million 61 / 36; Love, whose step is a tenth of the work, 60,000
// 0.96 / 1.11, 132,000 2.07 / 2.13, 198,000 3.08 / 3.03, 258,000 4.01 / 3.86, 1.2 million
// 19.1 / 16.8.  With a hundred modes the lines lie somewhat higher for Love (132,000
// 3.38 / 3.65, 198,000 5.05 / 5.23, 300,000 7.7 / 7.7) and are the same for Rayleigh.
constexpr int SPLIT_MIN_TRACES[2] = {16384, 196608};
constexpr unsigned SK_SEED = 1, SK_NEAR = 2, SK_EXACT = 4, SK_REDO = 8;
constexpr int ZOOM_TROUGH = 0, ZOOM_LAST = 1;

}  // namespace md200

// One trace's samples of a round: positions, FP32 secular values, shape features
// and log-magnitudes, bits (seed, near cutoff, FP64 value), and the FP64 values of
// the samples that have one.  By field, so that a warp's stores and loads of 32
// slots are whole sectors and the bookkeeping thread fetches four samples' fields
// 16 bytes at a time.  (As 32-byte records every field of every slot was a sector
// of its own: scan stage of 20,000 models, Love 17.2 -> 16.8 ms, Rayleigh 36.9 ->
// 36.4.)  The trough tests and windows take the shape feature and
// log-magnitude in single precision only, and of an FP32 value the bookkeeping
// takes the sign, so float keeps every decision of the fused scan.
struct md200::SplitRound {
  double c[md200::SPLIT_SAMPLES];
  float F[md200::SPLIT_SAMPLES], g[md200::SPLIT_SAMPLES], M[md200::SPLIT_SAMPLES];
  unsigned k[md200::SPLIT_SAMPLES];
  double F64[md200::SPLIT_SAMPLES];
};

// An active trace's constants for the evaluation threads, written by its
// positions warp: one load instead of the chain trace -> model -> table.
struct md200::SplitTrace {
  double w;
  int t, b, L, water, pad0, pad1;
};

namespace md200 {
static_assert(sizeof(SplitRound) % 16 == 0 && SPLIT_SAMPLES % 4 == 0, "16-byte copies of four samples");

// Warp-aggregated append: every lane of the warp calls it (n = 0 where there is
// nothing to add); returns this lane's base index in the list behind `counter`.
__device__ __forceinline__ int warp_append(int *counter, int n, int lane) {
  int incl = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  int base = 0;
  if (lane == 31 && total) base = atomicAdd(counter, total);
  base = __shfl_sync(FULL, base, 31);
  return base + incl - n;
}

__device__ __forceinline__ void split_count(const Dev &d, unsigned long long evals, unsigned long long evals32,
                                            unsigned long long steps, unsigned long long steps32, int lane) {
  if (!d.stats) return;
  for (int o = 16; o; o >>= 1) {
    evals += __shfl_xor_sync(FULL, evals, o);
    evals32 += __shfl_xor_sync(FULL, evals32, o);
    steps += __shfl_xor_sync(FULL, steps, o);
    steps32 += __shfl_xor_sync(FULL, steps32, o);
  }
  if (lane == 0) {
    if (evals) atomicAdd(&d.stats[0], evals);
    if (evals32) atomicAdd(&d.stats[1], evals32);
    if (steps) atomicAdd(&d.stats[2], steps);
    if (steps32) atomicAdd(&d.stats[3], steps32);
  }
}

// ---------------------------------------------------------------------------
// The active set of round r lives in sp_act[p], p = r & 1; traces that go on to
// the next round are appended to sp_act[1 - p].
// ---------------------------------------------------------------------------
__global__ void split_feed_count(Dev d, int p) {
  int *c = d.ctr;
  const int n_act = c[C_SP_ACT0 + p], n_list = c[C_NTRACE], feed = c[C_SP_FEED];
  const int room = d.sp_cap - n_act, left = n_list - feed;
  const int take = room < left ? room : left;
  c[C_SP_BASE] = n_act;
  c[C_SP_TAKE] = take;
  c[C_SP_ACT0 + p] = n_act + take;
  c[C_SP_FEED] = feed + take;
  c[C_SP_ACT0 + 1 - p] = 0;
  c[C_SP_REDO] = 0;
  c[C_SP_ZOOM] = 0;
}

__global__ void split_feed_fill(Dev d, int p) {
  const int base = d.ctr[C_SP_BASE], take = d.ctr[C_SP_TAKE];
  const int first = d.ctr[C_SP_FEED] - take;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < take; i += gridDim.x * blockDim.x) {
    const int t = d.trace_list[first + i];
    d.sp_act[p][base + i] = t;
    const ScanState st = scan_start(d, trace_ctx(d, t));
    d.sp_state[t] = st;
    d.sp_kf[t] = max(0, static_cast<int>(st.gi) - 2);  // (as in the fused scan)
  }
}

// One warp per active trace: positions of its next SPLIT_STEPS steps from the
// state's cursors.  Slots past the window hold INFINITY.
__global__ void __launch_bounds__(128) split_positions(Dev d, int p) {
  __shared__ double mbuf_all[4][32];
  __shared__ unsigned char kbuf_all[4][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  double *mbuf = mbuf_all[wib];
  unsigned char *kbuf = kbuf_all[wib];
  const int n = d.ctr[C_SP_ACT0 + p];
  const double step = 1. / d.density;
  for (int i = blockIdx.x * 4 + wib; i < n; i += gridDim.x * 4) {
    const int t = d.sp_act[p][i];
    const TraceCtx x = trace_ctx(d, t);
    ScanState st = d.sp_state[t];
    // the knot interval of the round's first grid point: no later target of this
    // trace lies below it (consumed samples only move the cursors up)
    int kfrom = d.sp_kf[t];
    if (lane == 0) {
      SplitTrace tr;
      tr.w = x.w;
      tr.t = t;
      tr.b = x.b;
      tr.L = d.mL[x.b];
      tr.water = d.mwater[x.b];
      tr.pad0 = tr.pad1 = 0;
      d.sp_tr[i] = tr;
    }
    SplitRound &ss = d.sp_s[i];
    bool done = false;
    for (int s = 0; s < SPLIT_STEPS; ++s) {
      double c = INFINITY;
      unsigned seeds = 0;
      if (!done) {
        int kfirst;
        const unsigned vm = scan_positions<true>(x, st, step, lane, mbuf, kfrom, c, kbuf, &seeds, &kfirst);
        done = vm == 0;
        if (s == 0 && lane == 0) d.sp_kf[t] = kfirst;
      }
      unsigned k = 0;
      if (c < INFINITY) {
        bool near_cut;
        scan_position32(c, x.hi, near_cut);
        k = ((seeds >> lane) & 1u ? SK_SEED : 0u) | (near_cut ? SK_NEAR : 0u);
      }
      ss.c[s * 32 + lane] = c;
      ss.k[s * 32 + lane] = k;
    }
  }
}

// A near-cutoff sample: the trace's FP64 tail value when it is at this position
// (returns false), else true (the sample goes to the FP64 list).
__device__ __forceinline__ bool split_near(const Dev &d, int t, SplitRound &smp, int j, double c, unsigned &k) {
  const double4 *tail = d.tail + 2 * static_cast<size_t>(t);
  const double4 t0 = tail[0], t1 = tail[1];
  const double4 tv = c == t0.x ? t0 : t1;
  if (c == tv.x && isfinite(tv.y)) {
    smp.F64[j] = tv.y;
    smp.g[j] = static_cast<float>(tv.z);
    smp.M[j] = static_cast<float>(tv.w);
    k |= SK_EXACT;
    return false;
  }
  return true;
}

// One thread per pair of sample slots of an active trace -- slot j of its first
// 32-sample step and slot j of its second -- whose FP32 values come from one paired
// evaluation (rayleigh_eval32<R2>, love_eval32<R2>: each half bit for bit the
// single evaluation the fused scan makes).  A slot past the
// window or in the near-cutoff band leaves its half to a copy of the other
// sample, whose result is not stored.
//
// A warp takes one trace's 32 pairs after another.  The layer records of the next
// trace's model come into shared memory (cp.async) while the current trace is
// evaluated: read from global memory layer by layer, each layer's loads missed L1
// (neighbouring traces are of different models) and waited 1.6 warps an issue.
// The layer step without per-half sign flips (step32) and the staged records,
// evaluation of 20,000 low-velocity-layer models x 60 periods: 26.8 -> 22.9 ms (18 %
// fewer instructions, FMA pipe 67 % busy; the FMA pipe's own time is 15 ms).
// Dynamic shared memory: `buffers` (2, or 1 where two would cost resident CTAs)
// x Ls records for each of the 4 warps.
static_assert(SPLIT_SAMPLES == 64, "the paired evaluation takes the two 32-sample steps of a round");
inline size_t split_pair_smem(int wave, int Ls, int buffers) {
  return static_cast<size_t>(4) * buffers * Ls * pair_row(wave) * 2 * sizeof(float);
}
inline int split_pair_buffers(int wave, int Ls) { return Ls <= (wave ? 168 : 56) ? 2 : 1; }

template <int WAVE>
__global__ void __launch_bounds__(128, WAVE ? MD200_SPLIT_PAIR_BLOCKS_LOVE : MD200_SPLIT_PAIR_BLOCKS)
    split_eval32_pair(Dev d, int p, int buffers) {
  extern __shared__ __align__(16) float4 pair_rec[];
  const int lane = threadIdx.x & 31;
  const int n16 = d.Ls * (pair_row(WAVE) / 2);  // 16-byte pieces of a model's records
  float4 *mine = pair_rec + (threadIdx.x >> 5) * buffers * n16;
  const long long n = static_cast<long long>(d.ctr[C_SP_ACT0 + p]) * 32;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  auto stage = [&](long long q, int buf) {  // the records of the trace that slot q belongs to
    if (q < n) {
      const float4 *src = reinterpret_cast<const float4 *>(d.pair32) + static_cast<size_t>(d.sp_tr[q >> 5].b) * n16;
      for (int j = lane; j < n16; j += 32) cp_async16(mine + buf * n16 + j, src + j);
    }
    cp_async_commit();
  };
  unsigned long long steps = 0;
  int buf = 0;
  const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (buffers == 2) stage(first, 0);
  // whole warps run the loop (n and stride are multiples of 32): appends are warp-wide
  for (long long q = first; q < n; q += stride, buf ^= buffers - 1) {
    if (buffers == 2) {
      stage(q + stride, buf ^ 1);
      cp_async_wait<1>();
    } else {
      stage(q, 0);
      cp_async_wait<0>();
    }
    __syncwarp();
    const int i = static_cast<int>(q >> 5);
    const int j0 = static_cast<int>(q & 31), j1 = j0 + 32;
    SplitRound &smp = d.sp_s[i];
    const double c0 = smp.c[j0], c1 = smp.c[j1];
    unsigned k0 = smp.k[j0], k1 = smp.k[j1];
    bool redo0 = false, redo1 = false;
    if (c0 < INFINITY || c1 < INFINITY) {
      const SplitTrace tr = d.sp_tr[i];
      const bool e0 = c0 < INFINITY && !(k0 & SK_NEAR), e1 = c1 < INFINITY && !(k1 & SK_NEAR);
      if (c0 < INFINITY && !e0) redo0 = split_near(d, tr.t, smp, j0, c0, k0);
      if (c1 < INFINITY && !e1) redo1 = split_near(d, tr.t, smp, j1, c1, k1);
      if (e0 || e1) {
        const LayerView<float> view = make_view<float>(layer_table<float>(d, tr.b), d.Ls, tr.L, tr.water);
        const float w = static_cast<float>(tr.w);
        const float x0 = static_cast<float>(e0 ? c0 : c1), x1 = static_cast<float>(e1 ? c1 : c0);
        const float2 kk = make_float2(w / x0, w / x1);
        float2 F, g, M;
        if constexpr (WAVE) love_eval32<R2>(Love2{view, mine + buf * n16}, kk, w, &F, &g, &M);
        else rayleigh_eval32<R2>(Layers2{view, mine + buf * n16}, kk, make_float2(w / kk.x, w / kk.y), w, &F, &g, &M);
        const unsigned long long ls = layer_steps(tr.L, tr.water);
        if (e0) {
          smp.F[j0] = F.x;
          smp.g[j0] = g.x;
          smp.M[j0] = M.x;
          redo0 = !(fabs(static_cast<double>(g.x)) > MD200_REDO_G);
          steps += ls;
        }
        if (e1) {
          smp.F[j1] = F.y;
          smp.g[j1] = g.y;
          smp.M[j1] = M.y;
          redo1 = !(fabs(static_cast<double>(g.y)) > MD200_REDO_G);
          steps += ls;
        }
      }
      if (c0 < INFINITY && !redo0) smp.k[j0] = k0;
      if (c1 < INFINITY && !redo1) smp.k[j1] = k1;
    }
    __syncwarp();  // the records are read: their buffer may be filled again
    int at = warp_append(&d.ctr[C_SP_REDO], (redo0 ? 1 : 0) + (redo1 ? 1 : 0), lane);
    if (redo0) d.sp_redo[at++] = i * SPLIT_SAMPLES + j0;
    if (redo1) d.sp_redo[at] = i * SPLIT_SAMPLES + j1;
  }
  if (d.stats) {
    for (int o = 16; o; o >>= 1) steps += __shfl_xor_sync(FULL, steps, o);
    if (lane == 0 && steps) atomicAdd(&d.stats[19], steps);
  }
}

// One thread per listed sample: its FP64 value (eval64_outline, as in the fused
// scan).
template <int WAVE>
__global__ void __launch_bounds__(128) split_redo(Dev d, int p) {
  const int n = d.ctr[C_SP_REDO];
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int q = d.sp_redo[r];
    const SplitTrace tr = d.sp_tr[q / SPLIT_SAMPLES];
    SplitRound &smp = d.sp_s[q / SPLIT_SAMPLES];
    const int j = q % SPLIT_SAMPLES;
    double g, M;
    smp.F64[j] = eval64_outline(make_view<double>(layer_table<double>(d, tr.b), d.Ls, tr.L, tr.water), WAVE, tr.w,
                                smp.c[j], &g, &M);
    smp.g[j] = static_cast<float>(g);
    smp.M[j] = static_cast<float>(M);
    smp.k[j] |= SK_EXACT | SK_REDO;
  }
}

// A finished trace's brackets published for refinement (scan_finish without
// the last cell), one thread per trace; every lane of the warp calls it.
__device__ __forceinline__ void split_publish(const Dev &d, int t, const ScanState &st, bool publish, int lane) {
  int n = 0;
  if (publish) {
    d.nbr[t] = st.nbr;
    if (st.tfl) atomicOr(&d.tflags[t], st.tfl);
    if (!d.model_lists && !(st.tfl & TRACE_SEARCH_UNCONVERGED)) n = st.nbr;
  }
  const int base = warp_append(&d.ctr[C_NREFINE], n, lane);
  for (int k = 0; k < n; ++k) d.refine_list[base + k] = t * d.KB + k;
}

// Does a finished trace need its last cell examined (scan_finish's condition)?
// -- and does the shape feature fall into the window end steeply enough that
// last_cell would screen the cell (its first test, evaluated here so that only
// those traces take a warp)?
__device__ __forceinline__ bool needs_last_cell(const ScanState &st, int K) {
  if (!((st.bits & SS_FINISHED) && st.nbr < K && !(st.tfl & TRACE_SEARCH_UNCONVERGED) && (st.bits & SS_HR1) &&
        (st.bits & SS_HR2) && st.R2.c < st.R1.c && st.zoom_right <= st.R2.c &&
        sample_segment(st.R1) == sample_segment(st.R2)))
    return false;
  const double sgn = sample_sign(st.R1);
  const float u = static_cast<float>(sgn) * st.R2.g, v = static_cast<float>(sgn) * st.R1.g;
  const float h0 = static_cast<float>(st.R1.c - st.R2.c);
  const float noise = pair_noise(true, st.R2, st.R1);
  return u > v + noise && v / ((u - v) / h0) < 1.25f * h0;
}

// The bookkeeping loop is a chain of dependent decisions, its loads need not be: each
// thread has the next four samples' fields on their way to shared memory while it
// works on four (one sample ahead, in registers, it waited 8 warps an issue for
// memory).
constexpr int BOOK_FIELDS = 6;  // 16-byte pieces of four samples: c (2), F, g, M, k

// One thread per active trace: its samples of this round in order, through the
// bookkeeping of scan_bookkeep (one lane's share of it, carried sample by
// sample).  Ends at the trace's K-th bracket, at the end of its window, at a
// non-finite value, at a trough that needs a window (paused there), or at the
// end of the round's samples (continued next round).
template <int WAVE>
__global__ void __launch_bounds__(128) split_book(Dev d, int p) {
  constexpr bool single = true;
  __shared__ float4 ring[2][BOOK_FIELDS][128];
  const int lane = threadIdx.x & 31;
  const int n = d.ctr[C_SP_ACT0 + p];
  const int stride = gridDim.x * blockDim.x;
  const int n_pad = (n + 31) & ~31;
  // samples 4 grp .. 4 grp + 3 of a trace into this thread's places
  auto fetch = [&](const SplitRound &r, int grp) {
    if (grp < SPLIT_SAMPLES / 4) {
      float4(&to)[BOOK_FIELDS][128] = ring[grp & 1];
      cp_async16(&to[0][threadIdx.x], &r.c[4 * grp]);
      cp_async16(&to[1][threadIdx.x], &r.c[4 * grp + 2]);
      cp_async16(&to[2][threadIdx.x], &r.F[4 * grp]);
      cp_async16(&to[3][threadIdx.x], &r.g[4 * grp]);
      cp_async16(&to[4][threadIdx.x], &r.M[4 * grp]);
      cp_async16(&to[5][threadIdx.x], &r.k[4 * grp]);
    }
    cp_async_commit();
  };
  // counters of the samples the bookkeeping consumes, as the fused scan counts
  // its steps' samples: each an FP32 evaluation, the re-evaluated ones also FP64
  unsigned long long ev = 0, ev32 = 0, sts = 0, sts32 = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pad; i += stride) {
    const bool active = i < n;
    int t = 0;
    ScanState st;
    int K = 0;
    bool go_on = false, publish = false, zoom = false;
    int ztype = ZOOM_TROUGH;
    if (active) {
      t = d.sp_act[p][i];
      st = d.sp_state[t];
      K = d.tr_modes[t] + 2;
      double *slot = d.slot + static_cast<size_t>(t) * d.KB * SLOT;
      const SplitRound &round = d.sp_s[i];
      const SplitTrace tr = d.sp_tr[i];
      const unsigned long long nsteps = layer_steps(tr.L, tr.water);
      bool stop = false;  // the K-th bracket, the window end or a non-finite value
      fetch(round, 0);
      for (int j = 0; j < SPLIT_SAMPLES; ++j) {
        if ((j & 3) == 0) {
          fetch(round, j / 4 + 1);
          cp_async_wait<1>();
        }
        const float4(&at)[BOOK_FIELDS][128] = ring[(j >> 2) & 1];
        auto field = [&](int q) { return reinterpret_cast<const float *>(&at[q][threadIdx.x])[j & 3]; };
        const double c = reinterpret_cast<const double *>(&at[(j & 3) >> 1][threadIdx.x])[j & 1];
        if (!(c < INFINITY)) {  // the window is exhausted
          st.bits |= SS_FINISHED;
          stop = true;
          break;
        }
        const unsigned k = __float_as_uint(field(5));
        const bool exact = (k & SK_EXACT) != 0;
        const double F = exact ? round.F64[j] : static_cast<double>(field(2));
        const float gf = field(3), Mf = field(4);
        const double g = gf;
        ++ev32;
        sts32 += nsteps;
        ev += (k & SK_REDO) ? 2 : 1;
        sts += (k & SK_REDO) ? 2 * nsteps : nsteps;
        if (!(isfinite(F) && isfinite(g))) {
          st.tfl |= TRACE_NONFINITE | TRACE_SEARCH_UNCONVERGED;
          st.bits |= SS_FINISHED;
          stop = true;
          break;
        }
        // sign change against the previous sample
        const bool vl = (st.bits & SS_HAVE1) != 0;
        const double cl = st.c1, Fl = st.F1;
        const bool exl = (st.bits & SS_EX1) != 0;
        const bool sc = vl && (signbit(Fl) != signbit(F));
        const int myseg = st.nseg + (sc ? 1 : 0);
        const Sample me{c, gf, Mf, myseg | (exact ? (1 << 29) : 0) | (signbit(F) ? (1 << 30) : 0)};
        const bool reg = !(vl && c - cl < 1e-6 * c);
        const Sample P1 = st.R1, P2 = st.R2;
        const bool hp1 = (st.bits & SS_HR1) != 0, hp2 = (st.bits & SS_HR2) != 0;
        bool tr = false, trm = false;
        if (reg && hp1 && hp2 && sample_segment(P2) == myseg && sample_segment(P1) == myseg) {
          const double sgn = sample_sign(P1);
          tr = trough_may_hide_roots(P2.c, P1.c, c, sgn * P2.g, sgn * P1.g, sgn * gf, pair_noise(single, P2, P1),
                                     pair_noise(single, P1, me));
          if (!tr) trm = magnitude_dip(P2.c, P1.c, c, P2.M, P1.M, Mf) > MDIP;
          tr = tr || trm;
        }
        bool pause = false;
        if (sc) {
          if (st.nbr < K) {
            put_bracket(slot, st.nbr, cl, c, exl ? Fl : NAN, exact ? F : NAN);
            ++st.nbr;
          }
        } else if (tr && st.nbr < K) {
          double x0 = P2.c, sa, ma;
          const double x1 = P1.c, x2 = c;
          const double sgn = sample_sign(P1);
          sa = sgn * P2.g;
          ma = P2.M;
          if (x0 < st.zoom_right) {  // overlaps the previous window: start at its middle sample
            x0 = x1;
            sa = sgn * P1.g;
            ma = P1.M;
          }
          st.zoom_right = x2;
          double *za = d.sp_zarg + static_cast<size_t>(i) * 8;
          za[0] = x0;
          za[1] = x2;
          za[2] = sa;
          za[3] = sgn * g;
          za[4] = ma;
          za[5] = Mf;
          za[6] = sgn;
          za[7] = trm ? 1. : 0.;
          pause = true;
        }
        // carries
        st.nseg = myseg;
        st.c1 = c;
        st.F1 = F;
        st.bits = (st.bits & ~SS_EX1) | SS_HAVE1 | (exact ? SS_EX1 : 0);
        if (reg) {
          st.R2 = st.R1;
          st.bits = (st.bits & ~SS_HR2) | ((st.bits & SS_HR1) ? SS_HR2 : 0);
          st.R1 = me;
          st.bits |= SS_HR1;
        }
        if (k & SK_SEED) ++st.si;
        else ++st.gi;
        if (pause) {
          zoom = true;
          ztype = ZOOM_TROUGH;
          break;
        }
        if (st.nbr >= K) {
          stop = true;
          break;
        }
      }
      if (stop) {
        if (needs_last_cell(st, K)) {
          zoom = true;
          ztype = ZOOM_LAST;
        } else {
          publish = true;
        }
      } else if (!zoom) {
        go_on = true;  // the round's samples are used up: more next round
      }
      d.sp_state[t] = st;
      cp_async_wait<0>();  // (the next trace's records take the same places)
    }
    split_publish(d, t, st, publish, lane);
    const int za = warp_append(&d.ctr[C_SP_ZOOM], zoom ? 1 : 0, lane);
    if (zoom) d.sp_zoom[za] = ztype == ZOOM_LAST ? -(i + 1) : i;
    const int ga = warp_append(&d.ctr[C_SP_ACT0 + 1 - p], go_on ? 1 : 0, lane);
    if (go_on) d.sp_act[1 - p][ga] = t;
  }
  split_count(d, ev, ev32, sts, sts32, lane);
}

// (Four resident CTAs: unbounded, 167 registers left room for three and a seventh of
// the warps; the scan stage of 20,000 models 37.9 -> 37.1 ms.)
// One warp per window request: a trough window (screened in FP32, zoomed in
// FP64 unless dismissed) after which the trace goes on, or the last cell of a
// finished trace, after which it is published.
template <int WAVE>
__global__ void __launch_bounds__(128, 4) split_zoom(Dev d, int p) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int n = d.ctr[C_SP_ZOOM];
  for (int r = blockIdx.x * (blockDim.x >> 5) + wib; r < n; r += gridDim.x * (blockDim.x >> 5)) {
    const int code = d.sp_zoom[r];
    const bool last = code < 0;
    const int i = last ? -code - 1 : code;
    const int t = d.sp_act[p][i];
    const TraceCtx x = trace_ctx(d, t);
    ScanState st = d.sp_state[t];
    const LayerView<float> view = make_view<float>(layer_table<float>(d, x.b), d.Ls, d.mL[x.b], d.mwater[x.b]);
    const LayerView<double> view64 = global_view(d, x.b);
    unsigned long long ev = 0, ev32 = 0, s = 0, s32 = 0, zooms = 0;
    if (last) {
      st.nbr = last_cell<float, WAVE>(view, view64, x.w, st.R2, st.R1, d.tol, x.slot, st.nbr, x.K, lane, x.nsteps,
                                      ev, ev32, s, s32, zooms);
    } else {
      const double *za = d.sp_zarg + static_cast<size_t>(i) * 8;
      const double x0 = za[0], x2 = za[1], sa = za[2], sb = za[3], ma = za[4], mb = za[5], sgn = za[6];
      const int mode = za[7] != 0. ? 1 : 0;
      unsigned long long se = 0;
      const bool dismissed = screen_trough32<WAVE>(view, static_cast<float>(x.w), x0, x2, sa, sb, ma, mb, sgn, mode,
                                                   lane, se);
      ev += se;
      ev32 += se;
      s += se * x.nsteps;
      s32 += se * x.nsteps;
      if (!dismissed) {
        unsigned long long ze = 0;
        st.nbr = zoom_trough<WAVE>(view64, x.w, x0, x2, sa, sb, ma, mb, sgn, mode, d.tol, x.slot, st.nbr, x.K, lane,
                                   ze);
        ev += ze;
        s += ze * x.nsteps;
        ++zooms;
      }
    }
    __syncwarp();
    if (lane == 0) {
      if (d.stats) {
        if (ev) atomicAdd(&d.stats[0], ev);
        if (ev32) atomicAdd(&d.stats[1], ev32);
        if (s) atomicAdd(&d.stats[2], s);
        if (s32) atomicAdd(&d.stats[3], s32);
        if (zooms) atomicAdd(&d.stats[5], zooms);
      }
      d.sp_state[t] = st;
      if (last || st.nbr >= x.K) {
        d.nbr[t] = st.nbr;
        if (st.tfl) atomicOr(&d.tflags[t], st.tfl);
      } else {
        d.sp_act[1 - p][atomicAdd(&d.ctr[C_SP_ACT0 + 1 - p], 1)] = t;
      }
    }
    if (!d.model_lists && (last || st.nbr >= x.K)) {
      int base = 0;
      if (lane == 0 && !(st.tfl & TRACE_SEARCH_UNCONVERGED)) base = atomicAdd(&d.ctr[C_NREFINE], st.nbr);
      base = __shfl_sync(FULL, base, 0);
      if (!(st.tfl & TRACE_SEARCH_UNCONVERGED))
        for (int k = lane; k < st.nbr; k += 32) d.refine_list[base + k] = t * d.KB + k;
    }
    __syncwarp();
  }
}

}  // namespace md200
