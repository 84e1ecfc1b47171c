// bpf_resident.cu — a run of consecutive ticks of a medium filter in one launch, its particles
// resident in shared memory across the GPU (one CTA per SM, up to kResMaxTilesPerCta tiles a CTA).
//
// The tick-per-launch path of such a filter (pass 1, the plan in its last CTA, pass 2) is bound by
// latency, not by work: two dependent launches, a ticket and a one-CTA plan per tick. Here every CTA
// keeps its tiles' particles, log2-weights and the next tick's noise in shared memory from the first
// tick to the last, and the CTAs meet once per tick (twice when the tick resamples):
//   pass 1    the tile arithmetic of pass 1 (kThreads * SPLIT threads a tile, the FP32 partial sums
//             handed along in pass 1's element order), so every tile record is bit for bit pass 1's;
//   exchange  each tile's record {S, Q, H, n_k, E} is published as two 16-byte words that carry the
//             exchange's number, and thread k of every CTA polls tile k's record until the numbers
//             match: barrier and data in one trip through L2. The next tick's noise is formed before
//             the poll, while the records travel;
//   plan      every CTA forms the plan's FP64 sums in the plan kernel's order (one tile a thread, warp
//             butterfly, warps in sequence) and takes the same decision; one CTA (the keeper) also
//             writes the record, whose FP64 log is left to the next tick's exchange;
//   resample  the plan kernel's exact fixed-point rule: the u64 scan over the tile masses in every
//             CTA, then each parent writes its particle to its children's slots: in its own tile's
//             shared memory where they fall there (nearly all do: a tile's outputs drift from its
//             slots by about sqrt(N)), else to the other particle buffer (L2), from which the owner
//             takes them once the CTAs that write there have raised their flags.
// What bounds it: latency, three grid-wide dependencies deep at most, and the issue of 79 thread-instructions
// per particle and tick with two tiles a CTA (99 with one), 186 (223) where the tick resamples, by 16
// warps an SM on 40 to 50% of the cycles (16 particles a thread keep the per-thread overhead small: with
// 1024 threads of 4 the same tick issued 144 per particle). Measured per tick: N = 300000 at
// ESS < 0.5 N 4.0 us (16.4 with a launch per kernel), always resampling 9.1 us (20.8); N = 1000003 at
// ESS < 0.5 N 5.7 us (12.5), always resampling 12.5; N = 2.4 M at ESS < 0.5 N 10.7.
// Results equal the tick-per-launch path's bit for bit.
//
// The CTAs wait on one another, so the launch is cooperative (all resident or none start), and every
// wait gives up after kResWaitNs of polling. A CTA that gives up raises the abort mark, stores none of its
// tiles and sets the state's error itself (the keeper, which writes the rest of the state, leaves that
// word to it): whichever CTA gave up, and however late, the run ends with BPF_ERR_STATE, and a later run
// does not start on such a state.
#include "bpf_tick.cuh"
#include <algorithm>
#include <cstddef>
#include <mutex>
#include <type_traits>

namespace bpf {

constexpr int kResThreads = 512;
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxTiles = 1024;        // records an exchange holds at most (32 sums of 32 tiles)
constexpr int kResHeavy = 16;             // children above which a parent's run is shared by its warp
static_assert(kResMaxTilesPerCta == 4, "four tiles of two groups of threads");

// ---------------------------------------------------------------------------
// Exchange buffer (Plan::xbuf): word 0 the epoch (exchange numbers used so far, advanced by every
// launch's keeper), word 1 the abort mark; then kMail mailboxes, each with a flag per CTA and two
// parities of two 16-byte record words per tile. A record word is read and written as one 128-bit
// access, so its number vouches for its data. Every record and flag is written to all mailboxes and
// CTA b polls mailbox b % kMail: with one mailbox polled by all, the polls of a few hot lines held
// up the records themselves.
// ---------------------------------------------------------------------------
constexpr int kMail = kResMail;
constexpr size_t kXHeader = 256;
__host__ __device__ inline size_t mail_flag_bytes(int G) { return ((size_t)G * 4 + 127) & ~(size_t)127; }
__host__ __device__ inline size_t mail_bytes(int G) { return mail_flag_bytes(G) + (((size_t)G * 64 + 127) & ~(size_t)127); }
size_t resident_xbuf_bytes(int G) { return kXHeader + kMail * mail_bytes(G); }

__device__ __forceinline__ void st_relaxed_b128(void* p, unsigned long long lo, unsigned long long hi) {
  asm volatile("{ .reg .b128 v; mov.b128 v, {%1, %2}; st.relaxed.gpu.global.b128 [%0], v; }" ::"l"(p), "l"(lo), "l"(hi)
               : "memory");
}
__device__ __forceinline__ void ld_relaxed_b128(const void* p, unsigned long long& lo, unsigned long long& hi) {
  asm volatile("{ .reg .b128 v; ld.relaxed.gpu.global.b128 v, [%2]; mov.b128 {%0, %1}, v; }"
               : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Whether a warp's wait goes on (the same answer in every lane): every 256 polls it looks at its budget
// and at the abort mark of this launch. After a no the caller looks at its words once more.
struct Patience {
  WaitBudget budget;
  unsigned spins = 0u;
  __device__ __forceinline__ bool more(const unsigned* abort_word, unsigned mark, unsigned limit) {
    if ((++spins & 255u) != 0u) return true;
    const bool over = budget.over(WaitBudget::clock(global_timer_ns()), limit);
    return __all_sync(0xffffffffu, !over && ld_relaxed_u32(abort_word) != mark);
  }
};

// A tile's particles and log2-weights in shared memory: float4 group i4 sits at swz4(i4), so that a
// warp reading CH consecutive slots a lane (the child counts) falls on distinct banks, as one reading
// consecutive groups (pass 1) does.
__device__ __forceinline__ int swz4(int i4) { return i4 ^ ((i4 >> 3) & 7); }
__device__ __forceinline__ float4 ld4(const float* tile, int i) { return reinterpret_cast<const float4*>(tile)[swz4(i >> 2)]; }
__device__ __forceinline__ void st4(float* tile, int i, float4 v) { reinterpret_cast<float4*>(tile)[swz4(i >> 2)] = v; }
__device__ __forceinline__ float& el(float* tile, int i) { return tile[(swz4(i >> 2) << 2) | (i & 3)]; }

// exact_count on a swizzled tile: the element's chunk starts at slot i0.
static __device__ __noinline__ int exact_count_swz(const float* tile, int i0, int upto, unsigned long long R0,
                                                   unsigned long long D, int cap) {
  unsigned long long l = 0ull;
  for (int i = i0; i <= i0 + upto; ++i) l += fix_weight(tile_weight(tile[(swz4(i >> 2) << 2) | (i & 3)]));
  if (l < R0) return 0;
  const unsigned long long c = udiv_fp64(l - R0, D) + 1ull;
  return c >= (unsigned long long)cap ? cap : (int)c;
}

// Output slots a tile's children are gathered in: a window of kResSteps steps of 128 slots a warp,
// from the tile's first output rounded down to a float4. Children past it are written one by one.
template <int SPLIT> struct ResWindow {
  static constexpr int kSteps = SPLIT == 1 ? 5 : 3;
  static constexpr int kSlots = 8 * SPLIT * kSteps * 128;      // 5120, 6144
};

template <int NT, int SPLIT>
struct ResidentShared {
  static constexpr int NG = kResThreads / (kThreads * SPLIT);
  float h[NT][kTile];                     // particles
  float w[NT][kTile];                     // tile-relative log2-weights
  float z[NT][kTile];                     // state noise of the next propagation
  union {
    struct {
      float part[NT][3][kThreads];        // pass 1's per-thread FP32 partials S, Q, H
      unsigned long long partE[NT][kThreads];
    };
    unsigned short marks[NG][ResWindow<SPLIT>::kSlots];   // resampling: start marks of a tile's children
  };
  float ys[kResThreads];                  // observations of the next ticks
  double wS[32], wQ[32], wH[32];          // record sums of 32 tiles, in their own frame
  unsigned long long wE[32];              // their fixed-point mass, global frame
  unsigned long long wscan[NT][kResWarps];// chunk masses of each warp, by tile
  unsigned long long pre[NT], mass[NT], P[NT];   // own tiles: prefix within their 32 tiles, mass, global prefix
  unsigned long long base, delta, magic;  // the tick's targets
  unsigned long long ustate;              // resampling-uniform PCG32
  int wn[32];                             // frame of each 32 tiles
  int c0[NT], c1[NT];                     // own tiles' first output slots and their ends
  float smax[2][kResWarps];
  unsigned wmax[kResWarps];
  int nexp[NT];
  int resample, degenerate;               // this tick's decision
  __align__(16) DevState st;
  FusedTail tail;
};

// SPLIT threads share a pass-1 thread's sixteen particles; Q tiles per group of kThreads * SPLIT
// threads: (2, 1) for one tile a CTA, (1, 1) for two, (1, 2) for three and four.
template <bool TSTATE, bool GAUSS, bool APF, int SPLIT, int Q>
__global__ void __launch_bounds__(kResThreads, 1)
resident_kernel(Plan p, TickArgs a, ResidentTape tape, ResidentWaits waits, int n_ticks, int nt) {
  constexpr int NG = kResThreads / (kThreads * SPLIT);   // groups
  constexpr int NT = NG * Q;                    // tiles a CTA can hold
  constexpr int GW = 8 * SPLIT;                 // warps of a group
  constexpr int R = 4 / SPLIT;                  // float4 groups of a thread (a tile)
  constexpr int LW = 32 / SPLIT;
  constexpr int CH = 4 * R;                     // consecutive slots of a thread when children are counted
  constexpr int STEPS = ResWindow<SPLIT>::kSteps, WSLOTS = ResWindow<SPLIT>::kSlots;
  extern __shared__ __align__(16) unsigned char res_smem[];
  ResidentShared<NT, SPLIT>& sh = *reinterpret_cast<ResidentShared<NT, SPLIT>*>(res_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = p.N, G = p.G;
  const int first = (int)blockIdx.x * nt;       // this CTA's tiles
  const int nth = min(nt, G - first);
  const bool keeper = blockIdx.x == gridDim.x - 1;
  // this thread's group: tiles grp + NG q; in each, pass-1 thread v's float4 groups s R .. s R + R - 1
  const int grp = warp / GW, gw = warp % GW, gt = tid % (kThreads * SPLIT);
  const int s = lane / LW, v = LW * gw + (lane % LW);
  const int l_first = 4 * (v + kThreads * s * R);        // slot of its first float4; the next is kThreads * 4 on
  const int nwp = (G + 31) >> 5;                // groups of 32 records
  unsigned* xw = reinterpret_cast<unsigned*>(p.xbuf);
  const size_t mail_size = mail_bytes(G);
  const unsigned char* mail = p.xbuf + kXHeader + (blockIdx.x % kMail) * mail_size;   // the one this CTA polls
  const unsigned epoch = ld_relaxed_u32(xw);
  const int Fg = min(kFixF, 62 - ceil_log2_u((unsigned)N));
  const double rcpN = 1.0 / (double)N;

  if (tid < (int)(sizeof(DevState) / 8))
    reinterpret_cast<unsigned long long*>(&sh.st)[tid] = __ldcg(reinterpret_cast<const unsigned long long*>(p.st) + tid);
  __syncthreads();
  if (sh.st.error == BPF_ERR_STATE) n_ticks = 0;         // an earlier run gave up: nothing to go on from
  if (tid == 0) sh.ustate = sh.st.u_state;
  int nk[Q];                                    // the tiles' exponents (previous tick's until pass 1 sets them)
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = grp + NG * q;
    nk[q] = kNkEmpty;
    if (j >= nth) continue;
    const size_t off = (size_t)(first + j) * kTile;
    const float* hg = (sh.st.cur ? p.h1 : p.h0) + off;
    nk[q] = __ldcg(p.nexp + first + j);
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      const int l0 = l_first + 4 * kThreads * rr;
      st4(sh.h[j], l0, __ldcg(reinterpret_cast<const float4*>(hg + l0)));
      st4(sh.w[j], l0, __ldcg(reinterpret_cast<const float4*>(p.w + off + l0)));
    }
  }
  // state noise of this thread's particles for the tick with stream constants (k1, k2): read again
  // only by this thread; half 0 and 1: the first and second half of its groups, 2: all
  auto noise = [&](uint64_t k1, uint64_t k2, int half) {
    const uint64_t k33 = k2 << 33, step2 = 2ull * k2, step_r = (uint64_t)(2 * 4 * kThreads - 8) * k2;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = grp + NG * q;
      if (j >= nth) continue;
      uint64_t sx = k1 + k2 * pcg_inc((uint32_t)((first + j) * kTile + l_first));
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
        if (half == (rr < R / 2 ? 1 : 0)) { sx += 4ull * step2 + step_r; continue; }
        float zz[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float z = icdf_normal_warp(pcg_uniform(pcg_output(sx)));
          if (TSTATE) z *= tstate_scale_warp(sx, k33, a.nu_int, a.nu_state);
          zz[e] = z;
          sx += step2;
        }
        sx += step_r;
        *reinterpret_cast<float4*>(sh.z[j] + l_first + 4 * kThreads * rr) = make_float4(zz[0], zz[1], zz[2], zz[3]);
      }
    }
  };
  uint64_t k1 = sh.st.k1, k2 = sh.st.k2;        // stream constants of the next tick (all threads)
  if (!APF && sh.st.tick > 0) noise(k1, k2, 2);

  // what every thread follows of the device state; the keeper's copy is brought up to date (and the
  // record written) during the next exchange, from the sums its decision left with thread kDecider
  int tick = sh.st.tick, cur = sh.st.cur, nM_prev = sh.st.nM_prev;
  bool carry = sh.st.resampled_prev == 0;
  constexpr int kDecider = kResThreads - 32;
  double dS = 0.0, dQ = 0.0, dH = 0.0;
  int d_nM = 0;
  unsigned xn = 0u;                             // exchanges so far
  bool failed = false;                          // a wait gave up (the same in every thread of the CTA)
  bool pending = false;                         // the keeper's state is one decision behind
  int pending_rec = 0;
  auto settle = [&](int apf_stage, int t) {
    BpfTickRecord* rec = (a.rec && apf_stage != 1) ? a.rec + t : nullptr;
    const int tk = sh.st.tick;
    if (APF && apf_stage == 1) {
      fused_decide<1>(a, d_nM, dS, dQ, dH, &sh.st, sh.tail);
      fused_finish<1>(sh.tail, &sh.st, nullptr);
    } else {
      fused_decide<0>(a, d_nM, dS, dQ, dH, &sh.st, sh.tail);
      if (APF && apf_stage == 2) fused_finish<2>(sh.tail, &sh.st, rec);
      else fused_finish<0>(sh.tail, &sh.st, rec);
    }
    if (tape.aux)
      tape.aux[tk] = sh.tail.degenerate ? make_float2(0.0f, __int_as_float(0))
                                        : make_float2((float)(1.0 / dS), __int_as_float(d_nM));
  };
  const bool ahead = a.ess_threshold <= 0.0f;   // every tick that can resample does
  int stage = 0, prev_stage = 0;                // APF: 0 the first tick of all, else stages 1 and 2 of a tick
  int t = 0;
  while (t < n_ticks) {
    if ((!APF || stage != 2) && (t & (kResThreads - 1)) == 0) {
      __syncthreads();
      if (t + tid < n_ticks) sh.ys[tid] = __ldg(a.y_ptr + t + tid);
      __syncthreads();
    }
    const float y = sh.ys[t & (kResThreads - 1)];
    if (APF && stage != 2) stage = tick > 0 ? 1 : 0;
    ++xn;
    const unsigned xno = epoch + xn;

    // ---- pass 1 ----
    if (grp < nth) {
      ObsModel obs = a.obs;
      obs.y = y;
      const float y2 = y * y;
      const float y2nu = __fmul_rn(y2, obs.inv_nu);
      float x[Q][4 * R];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = grp + NG * q;
        if (j >= nth) continue;
        const int tile0 = (first + j) * kTile;
        float carry_off = 0.0f;
        if (carry) carry_off = (nk[q] == kNkEmpty) ? -INFINITY : (float)(nk[q] - nM_prev);
        const float gauss_c = kGaussLog2C + carry_off;
        const float t_c = __fmul_rn(obs.c_obs, kLog2e) + carry_off;
        auto density = [&](float h) { return GAUSS ? obs_log2pdf_gauss_plus(y2, h, gauss_c) : obs_log2pdf_t_plus(obs, y2nu, h, t_c); };
        float* ck = (tape.ckpt && tick % tape.K == 0) ? tape.ckpt + (size_t)(tick / tape.K) * tape.ckpt_stride + tile0 : nullptr;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
          const int l0 = l_first + 4 * kThreads * rr;
          const float4 h4 = ld4(sh.h[j], l0);
          if (ck) *reinterpret_cast<float4*>(ck + l0) = h4;
          float hh[4] = {h4.x, h4.y, h4.z, h4.w};
          float wp[4] = {0.f, 0.f, 0.f, 0.f}, zz[4] = {0.f, 0.f, 0.f, 0.f};
          if (carry) {
            const float4 w4 = ld4(sh.w[j], l0);
            wp[0] = w4.x; wp[1] = w4.y; wp[2] = w4.z; wp[3] = w4.w;
          }
          if (APF ? stage == 2 : tick > 0) {
            const float4 z4 = *reinterpret_cast<const float4*>(sh.z[j] + l0);
            zz[0] = z4.x; zz[1] = z4.y; zz[2] = z4.z; zz[3] = z4.w;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float h = hh[e], xx;
            if (!APF || stage == 0) {
              if (!APF && tick > 0) h = propagate(h, a.mu, a.rho, a.sigma, zz[e]);
              xx = density(h);
            } else {
              const float m = propagate_mean(h, a.mu, a.rho);
              xx = density(m);
              if (stage == 2) {
                h = fmaf(a.sigma, zz[e], m);
                xx = density(h) - xx;
              }
            }
            if (carry) xx += wp[e];
            hh[e] = h;
            x[q][4 * rr + e] = xx;
          }
          if (!APF || stage != 1) st4(sh.h[j], l0, make_float4(hh[0], hh[1], hh[2], hh[3]));
          if (tape.hist)
            *reinterpret_cast<float4*>(tape.hist + (size_t)tick * tape.ckpt_stride + tile0 + l0) = make_float4(hh[0], hh[1], hh[2], hh[3]);
        }
        if (tile0 + kTile > N) {                     // padding slots carry no weight
#pragma unroll
          for (int i = 0; i < 4 * R; ++i)
            if (tile0 + l_first + 4 * kThreads * (i >> 2) + (i & 3) >= N) x[q][i] = -INFINITY;
        }
        float mx = x[q][0];
#pragma unroll
        for (int e = 1; e < 4 * R; ++e) mx = fmaxf(mx, x[q][e]);
        mx = warp_max_f(mx);
        if (lane == 0) sh.smax[q][warp] = mx;
      }
      asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kThreads * SPLIT) : "memory");
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = grp + NG * q;
        if (j >= nth) continue;
        const float mx = warp_max_f(sh.smax[q][grp * GW + lane % GW]);
        nk[q] = (mx == -INFINITY) ? kNkEmpty : (int)ceilf(fmaxf(mx, -1.0e9f));
        const float fnk = (nk[q] == kNkEmpty) ? INFINITY : (float)nk[q];
        unsigned long long E = 0ull;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
          float dv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            dv[e] = x[q][4 * rr + e] - fnk;
            x[q][4 * rr + e] = tile_weight(dv[e]);       // the weight from here on
            E += fix_weight(x[q][4 * rr + e]);
          }
          st4(sh.w[j], l_first + 4 * kThreads * rr, make_float4(dv[0], dv[1], dv[2], dv[3]));
        }
        // pass 1's per-thread FP32 sums, in its element order, handed along the SPLIT threads
        float aS = 0.f, aQ = 0.f, aH = 0.f;
#pragma unroll
        for (int step = 0; step < SPLIT; ++step) {
          if (SPLIT == 1 || s == step) {
#pragma unroll
            for (int rr = 0; rr < R; ++rr) {
              const float4 h4 = ld4(sh.h[j], l_first + 4 * kThreads * rr);
              const float hv[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float w = x[q][4 * rr + e];
                aS += w;
                aQ = fmaf(w, w, aQ);
                aH = fmaf(w, hv[e], aH);
              }
            }
          }
          if (step + 1 < SPLIT) {
            const float nS = __shfl_up_sync(0xffffffffu, aS, LW);
            const float nQ = __shfl_up_sync(0xffffffffu, aQ, LW);
            const float nH = __shfl_up_sync(0xffffffffu, aH, LW);
            if (s == step + 1) { aS = nS; aQ = nQ; aH = nH; }
          }
        }
#pragma unroll
        for (int o = LW; o < 32; o <<= 1) E += __shfl_xor_sync(0xffffffffu, E, o);
        if (s == SPLIT - 1) { sh.part[j][0][v] = aS; sh.part[j][1][v] = aQ; sh.part[j][2][v] = aH; }
        if (s == 0) sh.partE[j][v] = E;
      }
      asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kThreads * SPLIT) : "memory");
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = grp + NG * q;
        if (gw == q && j < nth) {                      // pass 1's FP64 tile record, published by warp q
          double tS = 0.0, tQ = 0.0, tH = 0.0;
          unsigned long long tE = 0ull;
#pragma unroll
          for (int w = 0; w < kThreads / 32; ++w) {
            tS += (double)sh.part[j][0][lane + 32 * w];
            tQ += (double)sh.part[j][1][lane + 32 * w];
            tH += (double)sh.part[j][2][lane + 32 * w];
            tE += sh.partE[j][lane + 32 * w];
          }
          tS = warp_sum_d(tS); tQ = warp_sum_d(tQ); tH = warp_sum_d(tH);
          tE = warp_sum_u64(tE);
          if ((waits.record_mail >> lane) & 1u) {      // lanes 0 .. kMail - 1 (every lane holds the same sums)
            unsigned char* slot = p.xbuf + kXHeader + lane * mail_size + mail_flag_bytes(G) +
                                  ((size_t)(xn & 1u) * G + first + j) * 32;
            st_relaxed_b128(slot, (unsigned long long)__float_as_uint((float)tS) | ((unsigned long long)__float_as_uint((float)tQ) << 32),
                            (unsigned long long)(unsigned)nk[q] | ((unsigned long long)xno << 32));
            st_relaxed_b128(slot + 16, (unsigned long long)__float_as_uint((float)tH) | (tE << 32),
                            (tE >> 32) | ((unsigned long long)xno << 32));
          }
          if (lane == 0) sh.nexp[j] = nk[q];
        }
      }
    }

    // ---- while the records travel: the next noise, and the keeper's state and record of the last tick ----
    if (!APF || stage != 1) { k1 = k1 * kPcgMult; k2 = k2 * kPcgMult + 1ull; }
    const bool make_noise = APF ? stage == 1 : t + 1 < n_ticks;
    if (make_noise) noise(k1, k2, Q == 1 ? 0 : 2);
    if (keeper && pending && tid == kDecider) settle(prev_stage, pending_rec);

    // ---- exchange: lane l of the warp of 32 tiles takes its tile's record ----
    // (with little noise to form, the first look is issued before its second half: 3% of a tick)
    constexpr int MAXP = (kResMaxTiles + kResThreads - 1) / kResThreads;   // records a thread may take
    auto slot_of = [&](int u) {
      const int k = 32 * (warp + u * kResWarps) + lane;
      return mail + mail_flag_bytes(G) + ((size_t)(xn & 1u) * G + min(k, G - 1)) * 32;
    };
    unsigned long long a0 = 0ull, a1 = 0ull, b0 = 0ull, b1 = 0ull;
    if (warp < nwp) {
      ld_relaxed_b128(slot_of(0), a0, a1);
      ld_relaxed_b128(slot_of(0) + 16, b0, b1);
    }
    if (Q == 1 && make_noise) noise(k1, k2, 1);
    int rn[MAXP];
    unsigned long long rE[MAXP];
    bool bad = false;
#pragma unroll
    for (int u = 0; u < MAXP; ++u) {
      rn[u] = kNkEmpty;
      rE[u] = 0ull;
      const int pw = warp + u * kResWarps;
      if (pw >= nwp) continue;
      const int k = 32 * pw + lane;
      // The loop leaves by a warp vote: a lane that left alone would keep the warp split through the
      // shuffles below (measured 3.5 us for the sums after a spin, 0.13 us together).
      const unsigned char* slot = slot_of(u);
      if (u > 0) { ld_relaxed_b128(slot, a0, a1); ld_relaxed_b128(slot + 16, b0, b1); }
      Patience pt;
      for (;;) {
        const bool ok = (unsigned)(a1 >> 32) == xno && (unsigned)(b1 >> 32) == xno;
        if (__all_sync(0xffffffffu, ok)) break;
        if (!pt.more(xw + 1, epoch + 1u, waits.limit)) {             // the same in every lane
          ld_relaxed_b128(slot, a0, a1);
          ld_relaxed_b128(slot + 16, b0, b1);
          if (!__all_sync(0xffffffffu, (unsigned)(a1 >> 32) == xno && (unsigned)(b1 >> 32) == xno)) bad = true;
          break;
        }
        ld_relaxed_b128(slot, a0, a1);
        ld_relaxed_b128(slot + 16, b0, b1);
      }
      float rS = 0.f, rQ = 0.f, rH = 0.f;
      if (k < G && !bad) {
        rS = __uint_as_float((unsigned)a0); rQ = __uint_as_float((unsigned)(a0 >> 32));
        rn[u] = (int)(unsigned)a1;
        rH = __uint_as_float((unsigned)b0);
        rE[u] = (b0 >> 32) | (b1 << 32);
      }
      // the plan's sums of 32 tiles, in their own frame: scaling by a power of two is exact, so moving
      // them to the global frame afterwards gives the plan's values
      const int nW = __reduce_max_sync(0xffffffffu, rn[u]);
      double S = 0.0, Qs = 0.0, H = 0.0;
      if (rn[u] != kNkEmpty) {
        const double sc = pow2d(rn[u] - nW);
        S = (double)rS * sc; Qs = (double)rQ * (sc * sc); H = (double)rH * sc;
      }
      S = warp_sum_d(S); Qs = warp_sum_d(Qs); H = warp_sum_d(H);
      if (lane == 0) { sh.wn[pw] = nW; sh.wS[pw] = S; sh.wQ[pw] = Qs; sh.wH[pw] = H; }
    }
    if (__syncthreads_or(bad)) { failed = true; break; }

    // ---- decision (the last warp), and beside it, when every tick resamples, the masses ----
    const int nM = __reduce_max_sync(0xffffffffu, lane < nwp ? sh.wn[lane] : kNkEmpty);
    if (warp == kResWarps - 1) {
      double S = 0.0, Qs = 0.0, H = 0.0;
      if (lane < nwp && sh.wn[lane] != kNkEmpty) {
        const double sc = pow2d(sh.wn[lane] - nM);
        S = sh.wS[lane] * sc; Qs = sh.wQ[lane] * sc * sc; H = sh.wH[lane] * sc;
      }
      double tS = 0.0, tQ = 0.0, tH = 0.0;
      for (int w = 0; w < nwp; ++w) {
        tS += __shfl_sync(0xffffffffu, S, w);
        tQ += __shfl_sync(0xffffffffu, Qs, w);
        tH += __shfl_sync(0xffffffffu, H, w);
      }
      dS = tS; dQ = tQ; dH = tH; d_nM = nM;
      if (lane == 0) {
        const bool degenerate = (nM == kNkEmpty) || !(tS > 0.0);
        int resample = 0;
        if (!degenerate) resample = ahead || ess_below(tS * tS, tQ, a.ess_bound);
        sh.resample = resample;
        sh.degenerate = degenerate ? 1 : 0;
      }
      __syncwarp();
    }
    pending = true;
    pending_rec = t;
    prev_stage = stage;
    if (!ahead) __syncthreads();
    if (ahead || sh.resample) {
      // exact fixed-point masses: the tiles' in the global frame, and the own tiles' chunks of CH slots
#pragma unroll
      for (int u = 0; u < MAXP; ++u) {
        const int pw = warp + u * kResWarps;
        if (pw >= nwp) continue;
        const int k = 32 * pw + lane;
        rE[u] = (rn[u] != kNkEmpty) ? shr64(rE[u], nM - rn[u] + kFixF - Fg) : 0ull;
        const unsigned long long incl = warp_incl_scan_add(rE[u], lane);
        if (lane == 31) sh.wE[pw] = incl;
        if (k >= first && k < first + nth) { sh.pre[k - first] = incl - rE[u]; sh.mass[k - first] = rE[u]; }
        rE[u] = incl;                              // the prefix through tile k from here on
      }
      unsigned long long loc[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = grp + NG * q;
        loc[q] = 0ull;
        if (j >= nth) continue;
        unsigned long long e = 0ull;
#pragma unroll
        for (int g = 0; g < CH / 4; ++g) {
          const float4 d4 = ld4(sh.w[j], CH * gt + 4 * g);
          e += fix_weight(tile_weight(d4.x)) + fix_weight(tile_weight(d4.y));
          e += fix_weight(tile_weight(d4.z)) + fix_weight(tile_weight(d4.w));
        }
        const unsigned long long incl = warp_incl_scan_add(e, lane);
        if (lane == 31) sh.wscan[j][gw] = incl;
        loc[q] = incl - e;
      }
      __syncthreads();
      if (sh.resample) {
        // The targets and the own tiles' prefixes by warp 0; the others load their first chunk and clear
        // the marks meanwhile.
        const unsigned long long we = lane < nwp ? sh.wE[lane] : 0ull;
        const unsigned long long winc = warp_incl_scan_add(we, lane);
        if (warp == 0) {
          const unsigned long long total = __shfl_sync(0xffffffffu, winc, 31);
          unsigned long long delta = udiv_fp64_rcp(total, (unsigned long long)N, rcpN);
          const bool zero_spacing = delta == 0ull;
          if (zero_spacing) delta = 1ull;
          const unsigned long long old = sh.ustate;
          const unsigned long long u = pcg_output(old) >> 9;       // the tick's resampling uniform
          const unsigned long long hi = __umul64hi(u, delta), lo = u * delta;
          const unsigned long long base = (hi << 41) | (lo >> 23);   // floor(u * delta / 2^23)
          const unsigned long long magic = udiv_magic_of(delta);
          const int jm = min(lane >> 1, nth - 1);      // lanes 2 j and 2 j + 1: own tile j's first output and its end
          const unsigned long long before = __shfl_sync(0xffffffffu, winc - we, (first + jm) >> 5);
          const unsigned long long Pj = sh.pre[jm] + before;
          const int c = targets_below((lane & 1) ? Pj + sh.mass[jm] : Pj, base, delta, magic, N);
          if (lane < 2 * nth) {
            if (lane & 1) sh.c1[jm] = c;
            else { sh.c0[jm] = c; sh.P[jm] = Pj; }
          }
          __syncwarp();
          if (lane == 0) {
            sh.ustate = old * kPcgMult + kHostInc;
            sh.base = base; sh.delta = delta; sh.magic = magic;
            DevState& st = sh.st;
            if (zero_spacing) st.error = BPF_ERR_DEGENERATE;
            st.base = base; st.delta = delta; st.delta_magic = magic; st.total = total; st.Fg = Fg;
          }
        }
        ChunkTargets<CH> ct;
        unsigned short* mk = sh.marks[grp];
        unsigned long long chunk_loc = 0ull;
        auto load_chunk = [&](int j, unsigned long long lq) {
          ct.c = gt;
          ct.lfT = 0.0f;
#pragma unroll
          for (int g = 0; g < CH / 4; ++g) {
            const float4 d4 = ld4(sh.w[j], CH * gt + 4 * g);
            ct.wf[4 * g] = tile_weight(d4.x); ct.wf[4 * g + 1] = tile_weight(d4.y);
            ct.wf[4 * g + 2] = tile_weight(d4.z); ct.wf[4 * g + 3] = tile_weight(d4.w);
          }
#pragma unroll
          for (int e = 0; e < CH; ++e) ct.lfT += ct.wf[e];
          chunk_loc = lq + warp_sum_u64(lane < gw ? sh.wscan[j][lane] : 0ull);   // its prefix within the tile
          for (int i = gt; i < WSLOTS / 8; i += kThreads * SPLIT) reinterpret_cast<uint4*>(mk)[i] = make_uint4(0u, 0u, 0u, 0u);
        };
        if (grp < nth) load_chunk(grp, loc[0]);
        __syncthreads();
        const unsigned long long base = sh.base, delta = sh.delta, magic = sh.magic;
        float* hdst = cur ? p.h0 : p.h1;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int j = grp + NG * q;
          if (j >= nth) continue;                    // whole groups
          if (q > 0) {
            load_chunk(j, loc[q]);
            asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kThreads * SPLIT) : "memory");   // marks cleared
          }
          const int tk = sh.nexp[j];
          const int r = (tk == kNkEmpty) ? 64 : nM - tk + kFixF - Fg;
          const int own = (first + j) * kTile;
          const int j0 = own + CH * gt;
          chunk_thresholds<CH>(N, chunk_loc, sh.P[j], r, j0 < N, base, delta, magic, ct);
          int qe[CH];
          chunk_child_ends<CH>(N, ct, qe, [&](int upto) { return exact_count_swz(sh.w[j], CH * gt, upto, ct.th, ct.D, N); });
          if (tape.csr) {                            // first child of each parent
            int32_t* cs = tape.csr + (size_t)tick * tape.csr_stride + j0;
#pragma unroll
            for (int g = 0; g < CH / 4; ++g) {
              const int4 f4 = make_int4(g ? qe[4 * g - 1] : ct.q, qe[4 * g], qe[4 * g + 1], qe[4 * g + 2]);
              if (j0 + 4 * g + 4 <= N) {
                *reinterpret_cast<int4*>(cs + 4 * g) = f4;
              } else {
                const int f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) if (j0 + 4 * g + e < N) cs[4 * g + e] = f[e];
              }
            }
          }
          // start marks (slot of a parent's first child: its index in the tile + 1) in the window
          const int c0 = sh.c0[j], c1 = sh.c1[j];
          const int wb = c0 & ~3, we1 = min(c1, wb + WSLOTS);   // window [wb, we1)
#pragma unroll
          for (int e = 0; e < CH; ++e) {
            const int b0 = e ? qe[e - 1] : ct.q;
            if (qe[e] > b0 && b0 < we1) mk[b0 - wb] = (unsigned short)(CH * gt + e + 1);
          }
          if (c1 > we1) {                            // a tile of many children: the rest one by one
            auto put = [&](int o, float hc, int anc) {
              hdst[o] = hc;
              if (a.anc) a.anc[o] = anc;
            };
            float hv[CH];
#pragma unroll
            for (int g = 0; g < CH / 4; ++g) {
              const float4 h4 = ld4(sh.h[j], CH * gt + 4 * g);
              hv[4 * g] = h4.x; hv[4 * g + 1] = h4.y; hv[4 * g + 2] = h4.z; hv[4 * g + 3] = h4.w;
            }
#pragma unroll
            for (int e = 0; e < CH; ++e) {
              const int b0 = max(e ? qe[e - 1] : ct.q, we1), b1 = qe[e];
              if (b1 - b0 <= kResHeavy)
                for (int o = b0; o < b1; ++o) put(o, hv[e], j0 + e);
              unsigned heavy = __ballot_sync(0xffffffffu, b1 - b0 > kResHeavy);
              while (heavy) {                        // long runs are shared by the warp
                const int src = __ffs(heavy) - 1;
                heavy &= heavy - 1u;
                const int h0 = __shfl_sync(0xffffffffu, b0, src), h1 = __shfl_sync(0xffffffffu, b1, src);
                const float hc = __shfl_sync(0xffffffffu, hv[e], src);
                const int an = __shfl_sync(0xffffffffu, j0 + e, src);
                for (int o = h0 + lane; o < h1; o += 32) put(o, hc, an);
              }
            }
          }
          asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kThreads * SPLIT) : "memory");   // marks set
          // Gather: the ancestor of window slot o is the last mark at or before o. Each warp takes a run
          // of slots in steps of 128 (4 per lane); the running maximum of the marks is a lane-local scan,
          // the last marked lane before and a carry from the earlier steps and warps.
          const int nB = we1 - wb;
          const int run = ((nB + GW - 1) / GW + 127) & ~127;
          const int rs = gw * run, re = min(rs + run, nB);
          uint2 mv[STEPS];
          unsigned wm = 0u;
#pragma unroll
          for (int x = 0; x < STEPS; ++x) {
            mv[x] = make_uint2(0u, 0u);
            if (rs + 128 * x < re) mv[x] = reinterpret_cast<const uint2*>(mk + rs + 128 * x)[lane];
            const unsigned m2 = __vmaxu2(mv[x].x, mv[x].y);
            wm = max(wm, max(m2 & 0xffffu, m2 >> 16));
          }
          wm = __reduce_max_sync(0xffffffffu, wm);
          if (lane == 0) sh.wmax[warp] = wm;
          asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kThreads * SPLIT) : "memory");
          unsigned last = __reduce_max_sync(0xffffffffu, lane < gw ? sh.wmax[grp * GW + lane] : 0u);
          float4 out[STEPS];
#pragma unroll
          for (int x = 0; x < STEPS; ++x) {
            out[x] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (rs + 128 * x >= re) continue;
            unsigned am[4];
            am[0] = mv[x].x & 0xffffu;
            am[1] = max(am[0], mv[x].x >> 16);
            am[2] = max(am[1], mv[x].y & 0xffffu);
            am[3] = max(am[2], mv[x].y >> 16);
            unsigned pr, next_last;
            marks_before(am[3], lane, last, pr, next_last);
            last = next_last;
            float hv[4];
            const int o = wb + rs + 128 * x + 4 * lane;          // first of the lane's four slots
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const unsigned jj = max(pr, am[e]);                // 0 before the tile's first child (slot < c0)
              const int src = jj ? (int)jj - 1 : 0;
              hv[e] = el(sh.h[j], src);
              if (a.anc && o + e >= c0 && o + e < we1) a.anc[o + e] = own + src;
            }
            out[x] = make_float4(hv[0], hv[1], hv[2], hv[3]);
            if ((unsigned)(o - own) >= (unsigned)kTile) {        // another tile's slots: to its owner
              if (o >= c0 && o + 4 <= we1) {
                *reinterpret_cast<float4*>(hdst + o) = out[x];
              } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) if (o + e >= c0 && o + e < we1) hdst[o + e] = hv[e];
              }
            }
          }
          asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kThreads * SPLIT) : "memory");   // every parent read
#pragma unroll
          for (int x = 0; x < STEPS; ++x) {
            const int o = wb + rs + 128 * x + 4 * lane;
            if (rs + 128 * x >= re || (unsigned)(o - own) >= (unsigned)kTile) continue;
            if (o >= c0 && o + 4 <= we1) {
              st4(sh.h[j], o - own, out[x]);
            } else {
              const float hv[4] = {out[x].x, out[x].y, out[x].z, out[x].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) if (o + e >= c0 && o + e < we1) el(sh.h[j], o + e - own) = hv[e];
            }
          }
        }
        // every CTA whose children fall into this CTA's slots has written them before they are read
        __syncthreads();
        if (tid < 32 && ((waits.flag_mail >> tid) & 1u))
          st_release_u32(reinterpret_cast<unsigned*>(p.xbuf + kXHeader + tid * mail_size) + blockIdx.x, xno);
        const int slot_lo = first * kTile, slot_hi = (first + nth) * kTile;
        // which CTAs write children into this CTA's slots: bit u, tile 32 (warp + u kResWarps) + lane
        unsigned need = 0u;
#pragma unroll
        for (int u = 0; u < MAXP; ++u) {
          const int pw = warp + u * kResWarps;
          if (pw >= nwp) continue;
          const int k = 32 * pw + lane;
          const unsigned long long before = __shfl_sync(0xffffffffu, winc - we, pw);
          const int o1 = targets_below(before + rE[u], base, delta, magic, N);
          int o0 = __shfl_up_sync(0xffffffffu, o1, 1);
          if (lane == 0) o0 = targets_below(before, base, delta, magic, N);
          if (k < G && o1 > o0 && o0 < slot_hi && o1 > slot_lo && (k < first || k >= first + nth)) need |= 1u << u;
        }
#pragma unroll
        for (int u = 0; u < MAXP; ++u) {
          const bool wait = (need & (1u << u)) != 0u;
          if (!__any_sync(0xffffffffu, wait)) continue;
          const unsigned* flag = reinterpret_cast<const unsigned*>(mail) + (wait ? (32 * (warp + u * kResWarps) + lane) / nt : (int)blockIdx.x);
          Patience pt;
          for (;;) {                              // left by a warp vote, as above
            const bool ok = !wait || (int)(ld_relaxed_u32(flag) - xno) >= 0;
            if (__all_sync(0xffffffffu, ok)) break;
            if (!pt.more(xw + 1, epoch + 1u, waits.limit)) {
              if (!__all_sync(0xffffffffu, !wait || (int)(ld_relaxed_u32(flag) - xno) >= 0)) bad = true;
              break;
            }
          }
          asm volatile("fence.acq_rel.gpu;" ::: "memory");   // acquire (a relaxed poll leaves L1 alone)
        }
        if (__syncthreads_or(bad)) { failed = true; break; }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int j = grp + NG * q;
          if (j >= nth) continue;
          // the slots that the tile's own window did not fill
          const int own = (first + j) * kTile;
          const int c0 = sh.c0[j] - own, c1 = min(sh.c1[j], (sh.c0[j] & ~3) + WSLOTS) - own;
#pragma unroll
          for (int rr = 0; rr < R; ++rr) {
            const int l0 = l_first + 4 * kThreads * rr;
            if (l0 >= c0 && l0 + 4 <= c1) continue;
            const float4 g4 = __ldcg(reinterpret_cast<const float4*>(hdst + own + l0));
            const float hv[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (l0 + e < c0 || l0 + e >= c1) el(sh.h[j], l0 + e) = hv[e];
          }
        }
        cur ^= 1;
        carry = false;
      }
    }
    if (!sh.resample) {
      carry = sh.degenerate == 0;
      if (carry) nM_prev = nM;
    }
    if (!APF || stage != 1) ++tick;
    if (APF && stage == 1) {
      stage = 2;
    } else {
      stage = 0;
      ++t;
    }
  }

  if (tid == kDecider && pending && keeper && !failed) settle(prev_stage, pending_rec);
  __syncthreads();
  if (failed && tid == 0) {
    st_release_u32(xw + 1, epoch + 1u);         // the other CTAs stop waiting
    atomicExch(&p.st->error, BPF_ERR_STATE);
  }
  if (!failed) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = grp + NG * q;
      if (j >= nth) continue;
      const size_t off = (size_t)(first + j) * kTile;
      float* hg = (cur ? p.h1 : p.h0) + off;
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
        const int l0 = l_first + 4 * kThreads * rr;
        *reinterpret_cast<float4*>(hg + l0) = ld4(sh.h[j], l0);
        *reinterpret_cast<float4*>(p.w + off + l0) = ld4(sh.w[j], l0);
      }
      if (gt == 0) p.nexp[first + j] = nk[q];
    }
  }
  if (keeper) {
    if (tid == 0) {
      *reinterpret_cast<volatile unsigned*>(xw) = epoch + 4u * (unsigned)n_ticks + 4u;   // past every number used
      if (sh.st.error == BPF_ERR_DEGENERATE) atomicCAS(&p.st->error, BPF_OK, BPF_ERR_DEGENERATE);
    }
    // every word but the one that holds the error
    if (tid < (int)(sizeof(DevState) / 8) && tid != (int)(offsetof(DevState, error) / 8))
      reinterpret_cast<unsigned long long*>(p.st)[tid] = reinterpret_cast<const unsigned long long*>(&sh.st)[tid];
  }
}
static_assert(offsetof(DevState, error) % 8 == 0 && offsetof(DevState, seed) == offsetof(DevState, error) + 4,
              "the error shares its word with the seed, which no run changes");

// ---------------------------------------------------------------------------
// Launcher
// ---------------------------------------------------------------------------
namespace {

using ResidentKernel = void (*)(Plan, TickArgs, ResidentTape, ResidentWaits, int, int);

template <bool APF, int SPLIT, int Q>
ResidentKernel pick_model(bool tstate, bool gauss, size_t* smem) {
  *smem = sizeof(ResidentShared<kResThreads / (kThreads * SPLIT) * Q, SPLIT>);
  if (tstate) return gauss ? resident_kernel<true, true, APF, SPLIT, Q> : resident_kernel<true, false, APF, SPLIT, Q>;
  return gauss ? resident_kernel<false, true, APF, SPLIT, Q> : resident_kernel<false, false, APF, SPLIT, Q>;
}
template <bool APF>
ResidentKernel pick_shape(int nt, bool tstate, bool gauss, size_t* smem) {
  if (nt <= 1) return pick_model<APF, 2, 1>(tstate, gauss, smem);
  if (nt <= 2) return pick_model<APF, 1, 1>(tstate, gauss, smem);
  return pick_model<APF, 1, 2>(tstate, gauss, smem);
}
ResidentKernel pick(int nt, bool tstate, bool gauss, bool apf, size_t* smem) {
  return apf ? pick_shape<true>(nt, tstate, gauss, smem) : pick_shape<false>(nt, tstate, gauss, smem);
}

constexpr int kMaxConfiguredDevices = 64;
std::mutex g_lock;
int g_sms[kMaxConfiguredDevices] = {};       // 0: not looked at yet, -1: no resident runs on this device
signed char g_ready[kMaxConfiguredDevices][24] = {};   // per kernel: 0 not configured yet, 1 ready, -1 does not fit

}  // namespace

int resident_max_tiles(int device) {
  if (device < 0 || device >= kMaxConfiguredDevices) return 0;
  std::lock_guard<std::mutex> guard(g_lock);
  if (g_sms[device] == 0) {
    int sms = 0, coop = 0;
    const bool ok = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
                    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess && coop != 0 &&
                    sms > 0 && sms * kResMaxTilesPerCta <= kResMaxTiles;
    if (!ok) cudaGetLastError();
    g_sms[device] = ok ? sms : -1;
  }
  return g_sms[device] > 0 ? g_sms[device] * kResMaxTilesPerCta : 0;
}

// Called with `device` current, outside any stream capture; a kernel is loaded and given its shared
// memory when the first filter that runs it asks.
bool resident_ready(int device, int G, int max_tiles, bool tstate, bool gauss, bool apf) {
  if (G < 1 || G > max_tiles || device < 0 || device >= kMaxConfiguredDevices) return false;
  const int sms = max_tiles / kResMaxTilesPerCta, nt = (G + sms - 1) / sms;
  const int shape = nt <= 1 ? 0 : (nt <= 2 ? 1 : 2);
  std::lock_guard<std::mutex> guard(g_lock);
  signed char& state = g_ready[device][shape * 8 + (tstate ? 1 : 0) + (gauss ? 2 : 0) + (apf ? 4 : 0)];
  if (state == 0) {
    size_t smem = 0;
    int per = 0;
    ResidentKernel k = pick(nt, tstate, gauss, apf, &smem);
    const bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kResThreads, smem) == cudaSuccess && per >= 1;
    if (!ok) cudaGetLastError();
    state = ok ? 1 : -1;
  }
  return state > 0;
}

cudaError_t launch_resident(const Plan& p, const TickArgs& a, const ResidentTape& tape, bool apf, int n_ticks,
                            int max_tiles, cudaStream_t s, const ResidentWaits& waits) {
  if (!p.xbuf || p.G < 1 || p.G > max_tiles || p.G > kResMaxTiles || n_ticks < 1 || !a.y_ptr) return cudaErrorInvalidValue;
  if (waits.refused) return cudaErrorCooperativeLaunchTooLarge;
  const int sms = max_tiles / kResMaxTilesPerCta;
  const int nt = (p.G + sms - 1) / sms;
  size_t smem = 0;
  ResidentKernel k = pick(nt, a.nu_int > 0, !(a.obs.nu > 0.0f), apf, &smem);
  cudaLaunchConfig_t cfg = {};
  const int ctas = (p.G + nt - 1) / nt;
  cfg.gridDim = dim3(std::max(1, ctas - (waits.absent ? 1 : 0)));
  cfg.blockDim = dim3(kResThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaSuccess;
  for (int t = 0; t < n_ticks && e == cudaSuccess; t += kResRunTicks) {
    TickArgs run = a;
    run.y_ptr = a.y_ptr + t;
    run.rec = a.rec ? a.rec + t : nullptr;
    e = cudaLaunchKernelEx(&cfg, k, p, run, tape, waits, std::min(kResRunTicks, n_ticks - t), nt);
  }
  return e;
}

}  // namespace bpf
