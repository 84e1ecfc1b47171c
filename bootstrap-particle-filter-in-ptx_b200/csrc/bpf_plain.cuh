// bpf_plain.cuh — device-memory layout and launchers of the plain filter.
//
// HBM layout of one filter of N particles, G = ceil(N/4096) tiles
// (every particle array is padded to G*4096 floats so tile loads never
// leave the allocation):
//   h[2][G*4096]  f32  particle ping-pong (current buffer index in DevState)
//   w[G*4096]     f32  tile-relative log2-weights d_i = x_i - n_k <= 0 (weight 2^d_i)
//   tile records  rec[G] f32x4 {S=sum w, Q=sum w^2, H=sum w h, n_k bits},
//                 nexp[G] i32 (n_k again), E[G] u64 exact fixed-point mass
//   P[G] u64 exclusive tile prefix of the fixed-point CDF, ofirst[G+1] i32
//   items[G + N/8192 + 1] int4 pass-2 work items (tile, first out, end out, flags)
//   DevState      scalars carried from tick to tick
#pragma once
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#include "bpf_alloc.cuh"
#include "bpf_common.cuh"
#include "../../include/gpu_bpf.h"

namespace bpf {

// Scalars that live on the device from tick to tick (no host round trip).
struct DevState {
  uint64_t k1, k2;          // PCG32 stream constants of the next tick t: slot i's state is
                            // k1 + k2 inc_i, k1 = A^t A^2 seed, k2 = A^t (A+1) + sum_{k<t} A^k;
                            // tick to tick k1 <- A k1, k2 <- A k2 + 1
  uint64_t u_state;         // resampling-uniform PCG32 (gpu_bpf_ptx_full.cu:353)
  uint64_t base, delta;     // systematic targets t_i = base + i*delta (fixed point)
  uint64_t delta_magic;     // floor((2^64-1)/delta)
  uint64_t total;           // fixed-point CDF total
  double   logS_prev;       // ln(sum of carried weights) in the carry frame; ln N after a resample
  double   ll_total;        // FP64 running log-likelihood
  double   ll_ref;          // log-evidence since the last resample
  int      tick;            // index of the next tick
  int      cur;             // h buffer holding the current particles
  int      src;             // pass-2 gather source buffer
  int      resampled_prev;  // previous tick resampled (1 before tick 0)
  int      nM_prev;         // global tile exponent of the previous tick
  int      do_resample;     // current tick resamples
  int      nM;              // global tile exponent of the current tick
  int      Fg;              // global-frame fraction bits
  int      n_items;         // pass-2 work items of the current tick
  uint32_t u23;             // resampling uniform of the current tick
  int      resample_count;
  int      dirs;            // tile orders (1 = decreasing): bit 0 the next pass 1, bit 1 this tick's pass 2
  int      error;           // sticky BPF_* error code
  int      seed;            // filter seed (PCG32 streams, resampling uniform)
  double   learn[4];        // online learning sums since the last update: sum_t of
                            // sum W dlw, sum W dlw^2, sum W dlw (h_prev-mu), sum W dlw^2 (h_prev-mu)^2
  double   hm;              // filtered mean of the current tick (FP64): the centre of Silverman jitter
  uint64_t jk1, jk2;        // PCG32 stream constants of the current tick's jitter draw
  float    bw;              // Silverman jitter bandwidth of the current tick
  int      seq;             // host request number of the current tick (copied into the mirror)
};
static_assert(sizeof(DevState) == 200, "DevState layout");

struct Plan {
  int N, G, max_items;
  float* h0; float* h1; float* w;
  int* nexp; unsigned long long* E; float4* rec;
  float4* rec2;              // per tile, online learning only: tile-frame sums of w dlw, w dlw^2, w dlw dh, w dlw^2 dh^2
  unsigned long long* P; int* ofirst; int4* items;
  double* jpart;             // per tile, Silverman jitter only: sum of (h - hm)^2 over the tile's particles
  unsigned* jticket;         // CTAs of the jitter-variance kernel done this tick (the last one resets it)
  unsigned* pticket;         // pass-1 CTAs done this tick when the last one runs the plan (it resets it)
  DevState* st;
  unsigned char* xbuf;       // exchange buffer of resident runs (zeroed once), or null: none
};

// Host-mapped mirror of the state a synchronous tick reads back (zero-copy): written by the
// plan kernel at the end of every tick it is given to, and by pass 2 when it records an error.
struct TickMirror {
  int resample_count;
  int tick;                  // ticks completed
  int error;                 // DevState::error
  int seq;                   // host request number of the tick that wrote it (written last, after a
                             // system fence: the host may take the record once it sees its number)
};

struct TickArgs {
  float mu, rho, sigma;
  float ess_threshold;
  double ess_bound;          // ess_keep_bound(ess_threshold, N): the kernels that hold a filter on the chip compare with it
  double log_n;              // ln N
  ObsModel obs;              // obs.y is used when y_ptr == nullptr
  const float* y_ptr;        // device pointer to this tick's observation, or null
  BpfTickRecord* rec;        // device record slot written by the last pass-1 CTA
  int32_t* anc;              // ancestors of this tick (N ints) or null
  int nu_int;                // Student-t state noise: round(nu_state) degrees of freedom, 0 = Gaussian
  float nu_state;            // Student-t state noise scale parameter
  int learn;                 // accumulate the online-learning score sums of this tick (needs p.rec2)
  int apf;                   // auxiliary particle filter stage: 0 = bootstrap tick, 1 = first stage
                             // (weights p(y | mu + rho (h - mu)), particles unchanged, tick not
                             // advanced), 2 = second stage (propagate, weights p(y|h) / p(y|m))
  // gradient tape (all null outside a taped run)
  float* ckpt;               // copy of the particles pass 1 reads this tick (G*4096 floats) or null
  int32_t* csr;              // on resampling ticks: first child slot of every parent (N ints) or null
  float2* aux;               // {1/S, nM}: normalised weight W_i = 2^(x_i - nM) / S of this tick, or null
  TickMirror* mirror;        // host-mapped mirror of this tick's outcome, or null
  int seq;                   // host request number of this tick (pass 1 stores it in the device state)
  int tail_plan;             // the last pass-1 CTA runs the plan (G <= kTailTiles; no plan launch)
  float silverman;           // Silverman jitter shrink after resampling (0 = off; needs p.jpart)
};

// The smallest double x with x / n >= thr as the plan rounds the quotient (monotone in x), so that the
// test ess / n < thr is the comparison ess < x.
inline double ess_keep_bound(float thr, int n) {
  const double t = (double)thr, d = (double)n;
  double x = t * d;
  if (!(x > 0.0) || std::isinf(x)) return x;
  while (x / d >= t) x = std::nextafter(x, 0.0);
  while (x / d < t) x = std::nextafter(x, INFINITY);
  return x;
}

// Device buffers of a plan for N particles (G, max_items set; DevState included).
cudaError_t plan_alloc(Plan& p, int N);
void plan_free(Plan& p);

// Host-side launchers (stream-ordered, no synchronisation).
// Draws h_0 for `seed` and (re)initialises the DevState on the device.
cudaError_t launch_init(const Plan& p, float mu, float std_stat, int seed, cudaStream_t s);
// pdl = programmatic dependent launch on the previous kernel in the stream.
cudaError_t launch_pass1(const Plan& p, const TickArgs& a, cudaStream_t s, bool pdl);
// Filters of at most kTailTiles tiles may run the plan in pass 1's last CTA (a.tail_plan):
// the same plan code on 256 threads, one tile per thread, so the results equal the plan
// kernel's bit for bit; bootstrap ticks without learning or a gradient tape only.
constexpr int kTailTiles = 256;
bool tail_plan_eligible(const Plan& p, const TickArgs& a);
cudaError_t launch_plan(const Plan& p, const TickArgs& a, cudaStream_t s, bool pdl);
cudaError_t launch_pass2(const Plan& p, const TickArgs& a, int grid, cudaStream_t s, bool pdl);
// Silverman jitter of a resampling tick (both kernels exit at once on other ticks): the bandwidth
// from the resampled particles' spread about the tick's filtered mean, then h += bw z clamped to
// [mu - 8, mu + 8], z from the particle slot's next PCG32 draw.
cudaError_t launch_jitter(const Plan& p, const TickArgs& a, cudaStream_t s, bool pdl);
// Fused small-filter tick (N <= kSmallMaxN): one launch of one CTA runs n_ticks consecutive
// ticks (pass 1, plan and resampling), bit-identical to the three-kernel tick. a.y_ptr and
// a.rec point at the run's first tick (a.obs.y is the observation when y_ptr is null and
// n_ticks is 1). Not for learning, auxiliary-filter, Silverman or taped ticks.
bool small_eligible(const Plan& p, const TickArgs& a);
cudaError_t launch_small(const Plan& p, const TickArgs& a, int n_ticks, cudaStream_t s, bool pdl);
// Resident runs (bpf_resident.cu): n_ticks consecutive ticks of a filter of at most
// resident_max_tiles(device) tiles, bit-identical to the tick-per-launch path, as cooperative launches of
// at most kResRunTicks ticks: a launch holds its SMs from end to end, and this is how long other
// streams' work may have to wait for them (4 to 25 ms; the particles' way in and out of the chip
// between two launches costs a few us). a.y_ptr and a.rec point at the run's first tick; apf:
// auxiliary-filter ticks (threshold 0). Not for learning, Silverman or mirrored ticks. A launch is
// refused where the whole grid does not fit on what the process may use of the device; the caller then
// takes the ticks one by one.
constexpr int kResRunTicks = 1024;
inline int resident_launches(int n_ticks) { return (n_ticks + kResRunTicks - 1) / kResRunTicks; }
struct ResidentTape {        // gradient tape of a taped run from tick 0 (all null otherwise)
  int32_t* csr; size_t csr_stride;     // first child slots, tick t's at csr + t * csr_stride
  float* ckpt; size_t ckpt_stride;     // particles entering every K-th tick
  int K;
  float2* aux;                         // {1/S, nM} per tick
  float* hist;                         // every tick's particles as weighted, at hist + t * ckpt_stride, or null
};
// Waits of resident runs: how long one polls before it gives up and, in tests, one failure made on
// purpose. No wait outlasts its limit.
constexpr unsigned long long kResWaitNs = 2000000000ull;
// Time spent polling against that limit, both in units of 1024 ns, from the clock at one look after
// another. The time between two looks counts as at most a sixteenth of the limit: while the GPU runs
// another program, or the grid is held up as a whole, the clock goes on but nobody could publish what
// the wait is for. (32 bits: the looks are less than an hour apart, and the loops are short of registers.)
struct WaitBudget {
  unsigned last = 0u, spent = 0u;
  static __host__ __device__ __forceinline__ unsigned clock(unsigned long long ns) { return (unsigned)(ns >> 10); }
  __host__ __device__ __forceinline__ bool over(unsigned now, unsigned limit) {
    const unsigned step = now - last, cap = limit / 16u + 1u;
    if (last != 0u) spent += step < cap ? step : cap;
    last = now;
    return spent >= limit;
  }
};
constexpr int kResMail = 16;           // mailboxes of the exchange; CTA b polls mailbox b % kResMail
// Failures for the tests: no record, or no flag of a CTA's children, reaches one of the mailboxes, so the CTAs
// that poll it wait until they give up; the last CTA, with its tiles' records, is absent; or the launch
// is refused on the host, as one that does not fit on the device is.
enum ResidentFault { kFaultNone = 0, kFaultRecords = 1, kFaultFlags = 2, kFaultAbsent = 3, kFaultRefused = 4 };
struct ResidentWaits {
  unsigned limit = (unsigned)(kResWaitNs >> 10);
  unsigned record_mail = (1u << kResMail) - 1u, flag_mail = (1u << kResMail) - 1u;   // mailboxes written to
  bool absent = false, refused = false;
};
inline bool resident_waits_of(int fault, int mailbox, double limit_ms, ResidentWaits* out) {
  if (fault < kFaultNone || fault > kFaultRefused || mailbox < 0 || mailbox >= kResMail ||
      !(limit_ms >= 0.1 && limit_ms <= (double)kResWaitNs * 1e-6))
    return false;
  ResidentWaits w;
  w.limit = (unsigned)(limit_ms * 1e6 / 1024.0);
  if (fault == kFaultRecords) w.record_mail &= ~(1u << mailbox);
  if (fault == kFaultFlags) w.flag_mail &= ~(1u << mailbox);
  w.absent = fault == kFaultAbsent;
  w.refused = fault == kFaultRefused;
  *out = w;
  return true;
}
constexpr int kResMaxTilesPerCta = 4;
size_t resident_xbuf_bytes(int G);
int resident_max_tiles(int device);    // 0: the device takes no resident runs
// Whether the kernel of such a run (G tiles, observation and state noise model) is ready on the device.
bool resident_ready(int device, int G, int max_tiles, bool tstate, bool gauss, bool apf);
cudaError_t launch_resident(const Plan& p, const TickArgs& a, const ResidentTape& tape, bool apf, int n_ticks,
                            int max_tiles, cudaStream_t s, const ResidentWaits& waits = ResidentWaits());
int pass2_grid_size(int device);
// Tiles the fused tick takes on this device (16, else 8; 4 before pass2_grid_size configured it).
int small_max_tiles(int device);
size_t pass2_smem_bytes();
cudaError_t launch_debug_pcg(int seed, int n, int t, uint32_t* d_out, float* d_norm, cudaStream_t s);
// w_out[i] = 2^d_i of the stored tile-relative log2-weights (N floats, device).
cudaError_t launch_tile_weights(const Plan& p, float* w_out, cudaStream_t s);

}  // namespace bpf

// Status and launch bookkeeping shared by the C entry points (bpf_api.cu).
int bpf_record_error(int code);          // sets gpu_bpf_last_error() for this thread, returns code
void bpf_note_launches(long long n);     // adds to gpu_bpf_launch_count()
