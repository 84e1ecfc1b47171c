// bpf_tick.cuh — parts of a plain tick shared by the kernels that keep a filter on the chip from
// tick to tick (the fused small-filter cluster and the resident kernel) and by pass 2: the split
// plan (decision, finish) and the child counts of a chunk of consecutive particles.
#pragma once
#include "bpf_plain.cuh"
#include "bpf_block.cuh"

namespace bpf {

// Tile-frame thresholds of the child count are kept relative to the thread's first
// element and capped here: a thread's 16 fixed-point weights sum to at most 16 * 2^50
// < kThCap, so a capped threshold is never reached, and threshold + c * spacing stays
// below 2^57 for every count c the loop forms.
constexpr unsigned long long kThCap = 1ull << 55;

// Exact count of targets up to element `upto` of a thread's 16 staged log2-weights d:
// #{m >= 0 : R0 + m D <= sum_{i <= upto} floor(2^d_i 2^50)}, at most cap. The rare path of
// the FP32 estimate in pass 2's child count.
static __device__ __noinline__ int exact_count(const float* d, int upto, unsigned long long R0, unsigned long long D,
                                        int cap) {
  unsigned long long l = 0ull;
  for (int i = 0; i <= upto; ++i) l += fix_weight(tile_weight(d[i]));
  if (l < R0) return 0;
  const unsigned long long c = udiv_fp64(l - R0, D) + 1ull;
  return c >= (unsigned long long)cap ? cap : (int)c;
}

// ESS = fl(ss / q) < bound, without the division away from the bound: 2^-48 covers the roundings of the
// quotient and of the products.
__device__ __forceinline__ bool ess_below(double ss, double q, double bound) {
  const double lim = bound * q;
  if (ss < lim * (1.0 - 0x1p-48)) return true;
  if (ss > lim * (1.0 + 0x1p-48)) return false;
  return ss / q < bound;
}

// What the finish of a tick's plan needs from its decision (fused_decide -> fused_finish).
struct FusedTail {
  double tS, tQ, tH, logS_prev_old;
  int nM, degenerate, resample, resampled_prev_old, tick_old;
};


// The tick's decision from its statistics, by one thread: plan_decide's operations on the device-state
// fields that the next tick and the resampling read, in its order; the rest is left to fused_finish
// in tl. The threshold test is a.ess_bound's. APF as TickArgs::apf (the first stage of an auxiliary-filter tick does not advance the tick).
template <int APF = 0>
__device__ __forceinline__ void fused_decide(const TickArgs& a, int nM, double tS, double tQ, double tH,
                                             DevState* st, FusedTail& tl) {
  const bool degenerate = (nM == kNkEmpty) || !(tS > 0.0);
  int resample = 0;
  if (!degenerate) resample = (a.ess_threshold <= 0.0f) || ess_below(tS * tS, tQ, a.ess_bound);
  tl.tS = tS; tl.tQ = tQ; tl.tH = tH; tl.nM = nM;
  tl.degenerate = degenerate ? 1 : 0; tl.resample = resample;
  tl.logS_prev_old = st->logS_prev; tl.resampled_prev_old = st->resampled_prev; tl.tick_old = st->tick;
  const int cur = st->cur;
  if (degenerate) st->error = BPF_ERR_DEGENERATE;
  {
    const int d1 = st->dirs & 1;
    st->dirs = (resample ? d1 : (d1 ^ 1)) | ((d1 ^ 1) << 1);
  }
  if (APF != 1) {
    st->k1 = st->k1 * kPcgMult;
    st->k2 = st->k2 * kPcgMult + 1ull;
    st->tick = tl.tick_old + 1;
  }
  st->do_resample = resample;
  st->nM = nM;
  if (resample) {
    const uint64_t old = st->u_state;
    st->u_state = old * kPcgMult + kHostInc;
    st->u23 = pcg_output(old) >> 9;
    st->logS_prev = a.log_n;
    st->resampled_prev = 1;
    st->resample_count += 1;
    st->src = cur;
    st->cur = cur ^ 1;
  } else if (degenerate) {
    st->logS_prev = a.log_n;
    st->resampled_prev = 1;
  } else {
    st->resampled_prev = 0;
    st->nM_prev = nM;
  }
}

// The finish of that decision, by one thread at any time before the next decision: the FP64 log and
// mean, the record, the running sums and, when the tick keeps its particles, the log of its weight sum.
template <int APF = 0>
__device__ __forceinline__ void fused_finish(const FusedTail& tl, DevState* st, BpfTickRecord* rec_out) {
  constexpr double kLn2d = 0.693147180559945309417232121458;
  double dll = -INFINITY, hm = __longlong_as_double(0x7FF8000000000000LL), L = 0.0, ess = 0.0;
  if (!tl.degenerate) {
    ess = tl.tS * tl.tS / tl.tQ;
    L = log(tl.tS);
    dll = __fma_rn((double)tl.nM, kLn2d, L) - tl.logS_prev_old;
    hm = tl.tH / tl.tS;
  }
  double rec_dll = dll, ll_ref = dll;
  if (APF == 2) rec_dll = st->ll_ref + dll;
  if (APF == 0) ll_ref = (tl.resampled_prev_old ? 0.0 : st->ll_ref) + dll;
  st->ll_ref = ll_ref;
  st->hm = tl.degenerate ? 0.0 : hm;
  if (APF != 1) st->ll_total += rec_dll;
  if (rec_out) {
    BpfTickRecord r;
    r.dloglik = rec_dll; r.loglik_ref = ll_ref; r.loglik_total = st->ll_total;
    r.h_mean = (float)hm; r.ess = (float)ess; r.resampled = tl.resample; r.tick = tl.tick_old;
    *rec_out = r;
  }
  if (!tl.resample && !tl.degenerate) st->logS_prev = L;
}

// A chunk of CH consecutive slots of the tile (slots CH c .. CH c + CH - 1) against the tick's
// targets: its weights, their FP32 sum in order, its first target and tile-frame thresholds
// (th = kThCap: no target is reachable from the chunk).
template <int CH>
struct ChunkTargets {
  float wf[CH];
  float lfT;
  unsigned long long th, D;
  int q, c;
};


// The first target and the tile-frame thresholds of a chunk whose exclusive fixed-point prefix within
// its tile is loc: Pk the tile's prefix in the global frame, r the shift from the tile's frame to it
// (64: the tile has no mass), live: the chunk holds particles.
template <int CH>
__device__ __forceinline__ void chunk_thresholds(int N, unsigned long long loc, unsigned long long Pk, int r, bool live,
                                                 unsigned long long base, unsigned long long delta,
                                                 unsigned long long magic, ChunkTargets<CH>& ct) {
  ct.q = targets_below(Pk + shr64(loc, r), base, delta, magic, N);
  ct.th = kThCap; ct.D = kThCap;
  if (r < 64 && ct.q < N && live) {
    const unsigned long long m = base + (unsigned long long)ct.q * delta - Pk + 1ull;
    if (m <= (~0ull >> r)) ct.th = min((m << r) - loc, kThCap);
    if (delta <= (kThCap >> r)) ct.D = delta << r;
  }
}

// The end of each element's children (output slots [q_{j-1}, q_j), q_{-1} = ct.q): the running count
// c_j = #{m >= 0 : th + m D <= l_j} (l_j the exact fixed-point sum of the chunk's weights up to j)
// estimated in FP32 with pass 2's bound on the estimate's error taken at the chunk's largest sum; near
// a target boundary (one vote per four elements) element i recounts in exact 64-bit integers,
// recount(i) = exact_count of its log2-weights. Whole warps only.
template <int CH, class F>
__device__ __forceinline__ void chunk_child_ends(int N, const ChunkTargets<CH>& ct, int qe[CH], F recount) {
  const unsigned long long R0 = ct.th, D = ct.D;
  const bool none = R0 >= kThCap;
  const float R0w = (float)R0 * 0x1p-50f;
  const float invDw = 1.0f / ((float)D * 0x1p-50f);
  const float R0x = R0w * invDw;
  const float eL = 0x1p-18f * invDw, e0 = fmaf(R0w, eL, 0x1p-44f * invDw);
  const float xT = fmaf(ct.lfT, invDw, -R0x);
  float err = fmaf(ct.lfT, eL, fmaf(fmaxf(fabsf(xT), R0x), 0x1p-21f, e0));
  if (!(xT < 0x1p22f)) err = 1.0f;
  const float err_hi = 1.0f - err;
  const int q0 = ct.q, Kq = 0x4AFFFFFF - q0;
  float lf = 0.0f;
#pragma unroll
  for (int g = 0; g < CH / 4; ++g) {
    int qq[4];
    bool rc[4], any = false;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      lf += ct.wf[4 * g + e];
      const float x = fmaf(lf, invDw, -R0x);
      const float fl = floorf(x);
      const float fr = x - fl;                       // exact
      rc[e] = !none && !(fr > err && fr < err_hi);
      any |= rc[e];
      qq[e] = none ? q0 : min(max(__float_as_int(fl + 0x1p23f) - Kq, q0), N);
    }
    if (__any_sync(0xffffffffu, any)) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (rc[e]) qq[e] = min(q0 + recount(4 * g + e), N);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) qe[4 * g + e] = qq[e];
  }
}

}  // namespace bpf
