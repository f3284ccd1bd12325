// Persistent adaptive DOP853 trajectory of the reduced quartic system, on square tiles, for states
// with a Hermitian density (every density the library or the reference produces).
//
// The equations are those of trajectory.cu (ode_backend.py:170-233, 500-586):
//   dX_c/dt = jac (Qc X_c + X_c Qc^dag + Rc X_c Rc^dag) + src (coef_c (Rc X_s + X_s Rc^dag) + fixed_c).
// Every channel X_c stays Hermitian when rho is, so with Y_c = Qc X_c and P_c = Rc X_c
//   dX_c/dt = jac (Y_c + Y_c^dag + P_c Rc^dag) + src (coef_c (P_s + P_s^dag) + fixed_c),
// and one triangle of it is the whole of it: 2 full products and one on the upper tiles instead of
// 4 full ones (2.5-2.6 D^3 against 4), stage sums, error norms and stage vectors on the upper tiles
// only, and the mirrored entry is written, never computed: X_c is Hermitian to the last bit.
//
// Layout. A matrix is cut into NB x NB tiles of B x B (B = 16 up to DP = 64, 32 above). A team of
// NB^2 CTAs, one cluster, holds one tile each of one channel of a state, or of all seven. CTA (i, j):
//   phase 1: Y_c(i, j) and P_c(i, j): A = [Qc; Rc] rows of block i (shared memory, constant), B = the
//            columns j of X_c;
//   phase 2: T = (P_c Rc^dag)(i, j) when the CTA owns that tile of the channel (i = j, or one of
//            (i, j), (j, i) by the parity of the channel): A = P_c rows of block i, B = Rc^dag columns
//            j (shared memory, constant); k(i, j) from T, Y and the insertion; the stage sum of its
//            own B^2 elements and their mirrors, thread-private from stage to stage.
// A K loop is split over the warps of the CTA, whose partial tiles meet in shared memory. X_c and P_c
// travel through L2 in the order in which a lane reads its MMA fragments, so a fragment is one
// coalesced 512-byte load per warp, straight into registers: no staging buffer, no copy barrier.
// Two cluster barriers per right-hand side (X_c complete, P_c and Y_c complete).
//
// Measured on one B200, a lone random state, per right-hand side, row-block kernel and this one: D = 8
// 10.3 and 2.4 us, D = 32 18.6 and 4.4, D = 64 31.4 and 5.3, Z2 D = 128 161 and 16. At D = 64: MMAs 1.9 us
// (their floor at the DMMA peak 1.2), the two barriers 1.9, operand loads 0.6, partial tiles 0.6.
//
// What bounds it: the chain of dependent right-hand sides of one state. A lone state therefore takes
// one team per channel (7 NB^2 CTAs): the insertion's P_s comes from another team through a flag per
// tile and right-hand side, and only towards the channels that follow in the chains 0 -> 1 -> 2 and
// 6 -> 5 -> 4 -> 3, so a team runs ahead of its followers and nobody waits inside an attempt for a
// team behind it; the teams meet once per attempt at the error norm. Teams of one state wait for one
// another, so such a launch is cooperative. A batch takes one team per state (wide_kernel up to
// DP = 64) when that is faster than a few states at a time (teams_for).
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <type_traits>
#include "capacity.h"
#include "common.cuh"
#include "dop853_device.cuh"
#include "trajectory.h"
#include "trajectory_tile.h"

namespace rcmps {
namespace tile {

constexpr int kChannels = 7;
// insertions coef (R X_s + X_s R^dag) of ode_backend.py:193, and the channel each channel feeds
__constant__ int c_src[kChannels] = {-1, 0, 1, 4, 5, 6, -1};
__constant__ double c_coef[kChannels] = {0.0, 2.0, 3.0, 1.0, 2.0, 3.0, 0.0};
__constant__ int c_feeds[kChannels] = {1, 2, -1, -1, 3, 4, 5};

constexpr int kMaxTiles = 16;
// A record: 0..6 and 7..13 the two error sums by channel; 14..17 the scalar channel's part of the
// proposal, of both error estimates and its k of stage 12; 18 a bounded wait gave up; 19 the device
// clock passed the watchdog. The sums are kept by channel so that every layout adds them in the same
// order (CTAs of a channel, then channels): a state's steps do not depend on the launch it is in.
constexpr int kRec = 20;
constexpr int kPollLimit = 1 << 22;   // polls of a flag (about 0.5 us each) before a wait gives up

// Flags and records through which the teams of one state meet (zeroed before the launch).
struct Sync {
  unsigned pflag[kChannels][kMaxTiles];      // right-hand sides whose P tile is complete
  unsigned rflag[8];                         // attempts whose record is complete, by team
  double rec[kChannels][2][kRec];            // a team's sums, by the attempt's parity
  double crec[kMaxTiles][kRec];              // the CTAs' records of a team whose rank 0 has no room for them
};

template <int DP>
struct TG {
  static constexpr int B = DP <= 64 ? 16 : 32;
  static constexpr int NB = DP / B;
  static constexpr int NR = NB * NB;          // CTAs of a team
  static constexpr int KS = DP / 8;           // k-steps of a product
  static constexpr int KB = B / 8;            // k-steps of one block
  static constexpr int MT = B / 16;           // 16-row tiles of a block
  static constexpr int NTB = B / 8;           // 8-column tiles of a block
  static constexpr int NW = DP == 48 ? 12 : 8;
  static constexpr int NT = 32 * NW;
  static constexpr int OWN = 256;             // threads that own elements
  static constexpr int EPT = B * B / OWN;     // elements each
  static constexpr int BB = B * B;
  static constexpr size_t MAT = (size_t)DP * DP;
  // phase 1: 2 MT row tiles ([Q; R]) x NTB column tiles over NTB x MG1 x S1 warps
  static constexpr int MG1 = DP == 16 ? 2 : 1;
  static constexpr int S1 = NW / (NTB * MG1);
  static constexpr int M1 = 2 * MT / MG1;
  static constexpr int K1 = (KS + S1 - 1) / S1;
  // phase 2: MT x NTB tiles over MG2 x NG2 x S2 warps
  static constexpr int MG2 = MT;
  static constexpr int NG2 = B == 16 ? 2 : 1;
  static constexpr int S2 = DP == 16 ? 2 : NW / (MG2 * NG2);
  static constexpr int N2 = NTB / NG2;
  static constexpr int K2 = (KS + S2 - 1) / S2;
  // partial tiles of 128 values in shared memory. B = 32 folds the upper half of the slices into the
  // lower half first (a full set would not fit beside the panels at DP = 128).
  static constexpr bool FOLD = B == 32;
  static constexpr int SF1 = FOLD ? S1 / 2 : S1, SF2 = FOLD ? S2 / 2 : S2;
  static constexpr int T1 = 2 * MT * NTB, T2 = MT * NTB;
  static constexpr int RED = (SF1 * T1 > SF2 * T2 ? SF1 * T1 : SF2 * T2) * 128;
  // constant operands of one direction, in fragment order
  static constexpr int PANEL = KS * 2 * MT * 128;
  static constexpr int RJ = KS * NTB * 64;
};

// Controller state (kept by the team's rank 0) and the decision it hands to every CTA of the team.
struct Dec {
  double t, h, tn;            // the attempt just judged
  double nt, nh;              // the next attempt
  int accept, dense, stop;
  int spec;                   // the next attempt has sample points in its step: its dense stages are due if accepted
  long long first, last;
};
struct Ctl {
  double h, min_h, max_h, err, y_sc, ksc0;
  long long attempts, accepted, rejected, dense_steps, next_point;
  int status, after_reject;
};
template <int NW>
struct Tail {
  Dec dec;
  Ctl ctl;
  double jac[16], src[16];
  double wk[13][NW];          // warp sums of the scalar channel's trace, by stage
  double tot[kRec];
  int wait_flag, out_of_domain;
};

// Shared memory of tile_kernel (double2 units), one direction's constant operands resident.
template <int DP, bool LONE>
struct Smem {
  using G = TG<DP>;
  static constexpr bool KSM = LONE && G::B == 16;       // stage vectors of the one owned tile
  // a warp of its own for the other teams (B = 32 needs every register of the computing warps)
  static constexpr bool COMM = LONE && G::B == 16;
  static constexpr int IV = COMM ? G::BB : 0;
  static constexpr int THREADS = G::NT + (COMM ? 32 : 0);
  static constexpr int KVEC = KSM ? 18 * G::BB : 0;
  static constexpr int XCH = G::NB == 1 ? 2 * (int)G::MAT : 0;   // X and P of a one-CTA team
  // the CTAs' records at rank 0, and the warps' error sums; at DP = 128 only a lone channel's fit
  static constexpr bool GLOBAL_REC = !LONE && DP == 128;
  static constexpr int NC = LONE ? 1 : kChannels;       // channels whose error sums are kept
  static constexpr int NREC = LONE ? 2 + 6 : kRec;      // doubles of a CTA's record
  static constexpr int GAT = GLOBAL_REC ? 0 : G::NR * NREC / 2;
  static constexpr int WE = 2 * NC * G::NW / 2;
  static constexpr size_t bytes() {
    return ((size_t)(G::PANEL + G::RJ) + G::RED + GAT + (GLOBAL_REC ? 0 : WE) + KVEC + XCH + IV) * 16 + sizeof(Tail<G::NW>);
  }
};

__device__ __forceinline__ void flag_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Bounded wait until *p >= v; a CTA whose wait gave up waits for nothing any more.
__device__ __forceinline__ void flag_wait(const unsigned* p, unsigned v, int* wait_flag) {
  for (int i = 0; i < kPollLimit; ++i) {
    unsigned x;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
    if ((int)(x - v) >= 0) return;
    if (*(volatile int*)wait_flag) return;
  }
  atomicExch(wait_flag, 1);
}

// Offset of entry (row r of block a, column c of block b) in X_c: columns of block b in the order of
// the B fragments [KS][NTB][2][32]; and in P_c: rows of block a in the order of the A fragments
// [KS][MT][4][32].
template <int DP>
__device__ __forceinline__ size_t zoff(int a, int b, int r, int c) {
  using G = TG<DP>;
  return ((size_t)(b * G::KS + a * G::KB + r / 8) * G::NTB + c / 8) * 64 + ((r & 4) << 3) + 4 * (c & 7) + (r & 3);
}
template <int DP>
__device__ __forceinline__ size_t poff(int a, int b, int r, int c) {
  using G = TG<DP>;
  return ((size_t)(a * G::KS + b * G::KB + c / 8) * G::MT + r / 16) * 128 + (((r >> 3) & 1) + 2 * ((c >> 2) & 1)) * 32 +
         4 * (r & 7) + (c & 3);
}
// Entry (r, c) of a 16 x 8 tile in C-fragment order [4][32]; and its place in a partial tile in shared
// memory, where the lanes are permuted so that a warp reads a tile's entries and their mirrors without
// bank conflicts (unpermuted, the mirrors met 8-way).
__device__ __forceinline__ int roff(int r, int c) {
  return (2 * ((r >> 3) & 1) + (c & 1)) * 32 + 4 * (r & 7) + ((c & 7) >> 1);
}

__device__ __forceinline__ int swz(int i, int lane) { return i * 32 + (lane ^ ((lane >> 3) & 3) ^ (4 * (i & 1))); }
__device__ __forceinline__ int soff(int r, int c) {
  return swz(2 * ((r >> 3) & 1) + (c & 1), 4 * (r & 7) + ((c & 7) >> 1));
}

// The CTA's [Qc; Rc] rows of block bi as A fragments [KS][2 MT][4][32], and the columns bj of Rc^dag as
// B fragments [KS][NTB][2][32] (dir 1: the adjoint channels, Qc = Q^dag, Rc = R^dag).
template <int DP>
__device__ void load_panel(const TrajState* st, int dir, int bi, double2* dst) {
  using G = TG<DP>;
  const double2 *Qc = dir ? st->Qh : st->Q, *Rc = dir ? st->Rh : st->R;
  for (int e = threadIdx.x; e < G::PANEL; e += blockDim.x) {
    const int l = e & 31, q = (e >> 5) & 3, m = (e >> 7) % (2 * G::MT), ks = e / (128 * 2 * G::MT);
    const int row = 16 * (m % G::MT) + (l >> 2) + 8 * (q & 1), col = 8 * ks + (l & 3) + 4 * (q >> 1);
    dst[e] = (m < G::MT ? Qc : Rc)[(size_t)(bi * G::B + row) * DP + col];
  }
}
template <int DP>
__device__ void load_rj(const TrajState* st, int dir, int bj, double2* dst) {
  using G = TG<DP>;
  const double2* Rc = dir ? st->Rh : st->R;
  for (int e = threadIdx.x; e < G::RJ; e += blockDim.x) {
    const int l = e & 31, h = (e >> 5) & 1, nt = (e >> 6) % G::NTB, ks = e / (64 * G::NTB);
    const int n = 8 * nt + (l >> 2), k = 8 * ks + (l & 3) + 4 * h;
    dst[e] = zconj(Rc[(size_t)(bj * G::B + n) * DP + k]);
  }
}

// The weight of entry (row, col) of channel c in the error norm: an entry stands for its mirror too;
// a packed state counts one off-diagonal block of an odd channel and both diagonal ones of an even one.
__device__ __forceinline__ double norm_weight(bool packed, int half, int c, int row, int col) {
  const double wt = row == col ? 1.0 : 2.0;
  if (!packed) return wt;
  const bool cross = (row < half) != (col < half);
  if (c & 1) return cross ? 0.0 : wt;
  return cross ? 1.0 : 0.0;
}

// The next attempt from time t with the step h0 (ode_backend.py:500-527).
__device__ __forceinline__ void prepare_attempt(double t, double h0, double endpoint, long long attempts,
                                                long long max_steps, double& h, int& status) {
  const double boundary = t < 0.0 ? 0.0 : endpoint;
  h = fmin(h0, boundary - t);
  if (attempts >= max_steps) status = kMaxSteps;
  else if (!isfinite(h) || h <= 10.0 * fabs(next_up(t) - t)) status = kStepUnderflow;
}

// Whether an attempt from t with step h would step over the sample point `next`.
__device__ __forceinline__ int has_points(double t, double h, double endpoint, const double* points, long long next,
                                          int npoints) {
  const double boundary = t < 0.0 ? 0.0 : endpoint;
  return next < npoints && points[next] <= (h == boundary - t ? boundary : __dadd_rn(t, h));
}

// A warp of rank 0 hands a decision to every CTA of the team.
template <int NR>
__device__ __forceinline__ void share_dec(Dec* shared, const Dec& d) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  if (lane == 0) *shared = d;
  __syncwarp();
  constexpr int words = sizeof(Dec) / 8;
  for (int i = lane; i < words * (NR - 1); i += 32) {
    double* w = reinterpret_cast<double*>(shared) + i % words;
    dsmem_store_f64(w, 1 + i / words, *w);
  }
}

// The first decision of a trajectory (rank 0's warp 0).
template <int NR, class TailT>
__device__ void first_decision(TailT& S, const TrajState* st, const TrajControls& ctl, const double* points,
                               int npoints) {
  Dec d{};
  int status = 0;
  d.nt = -ctl.endpoint;
  prepare_attempt(d.nt, fmin(ctl.initial_h, 2.0 * ctl.endpoint), ctl.endpoint, 0, st->max_steps, d.nh, status);
  d.stop = status ? 1 : 0;
  d.spec = has_points(d.nt, d.nh, ctl.endpoint, points, 0, npoints);
  if ((threadIdx.x & 31) == 0) {
    S.ctl.status = status;
    if (!status) {
      S.ctl.attempts = 1;
      S.ctl.min_h = fmin(S.ctl.min_h, d.nh);
      S.ctl.max_h = fmax(S.ctl.max_h, d.nh);
    }
  }
  share_dec<NR>(&S.dec, d);
}

// The controller (ode_backend.py:529-547; persistent_trajectory_backend.py:109-131) on the state's
// record in S.tot, by one warp of rank 0, every lane alike; pt: the lane's next sample point.
template <int NR, class TailT>
__device__ void decide(TailT& S, const TrajState* st, const TrajControls& ctl, const double* points, int npoints,
                       double pt, double N, double t, double h) {
  const int lane = threadIdx.x & 31;
  Ctl& C = S.ctl;
  const long long next = C.next_point;
  const double k0 = C.ksc0, prop = C.y_sc + (h * c_dop_b[0] * k0 + S.tot[14]);
  const double e5 = c_dop_e5[0] * k0 + S.tot[15], e3 = c_dop_e3[0] * k0 + S.tot[16];
  const double scale = st->atol + st->rtol * fmax(fabs(C.y_sc), fabs(prop));
  double t5 = 0.0, t3 = 0.0;
#pragma unroll
  for (int c = 0; c < kChannels; ++c) {
    t5 += S.tot[c];
    t3 += S.tot[7 + c];
  }
  t5 += (e5 / scale) * (e5 / scale);
  t3 += (e3 / scale) * (e3 / scale);
  const double den = __dadd_rn(t5, __dmul_rn(0.01, t3));
  const double err = den > 0.0 ? __ddiv_rn(__dmul_rn(h, t5), __dsqrt_rn(__dmul_rn(den, N))) : 0.0;
  Dec d{};
  d.t = t;
  d.h = h;
  d.nt = t;
  int status = 0, after = C.after_reject;
  double hn = h, y_sc = C.y_sc, ksc0 = C.ksc0;
  long long rejected = C.rejected, accepted = C.accepted, dense_steps = C.dense_steps, np = next;
  if (S.tot[18] != 0.0) status = kWaitLimit;
  else if (S.tot[19] != 0.0) status = kDeviceTimeout;
  else if (S.out_of_domain) status = kSourceDomain;
  else if (!isfinite(t5) || !isfinite(t3) || !isfinite(err)) status = kNonfiniteError;
  else {
    double factor = err > 0.0 ? fmin(10.0, __dmul_rn(0.9, pow(err, -1.0 / 8.0))) : 10.0;
    if (err > 1.0) {
      ++rejected;
      after = 1;
      hn = __dmul_rn(h, fmax(0.2, factor));
    } else {
      d.accept = 1;
      ++accepted;
      const double boundary = t < 0.0 ? 0.0 : ctl.endpoint;
      d.tn = h == boundary - t ? boundary : __dadd_rn(t, h);
      if (after) factor = fmin(1.0, factor);
      hn = __dmul_rn(h, factor);
      after = 0;
      d.first = next;
      long long last = next;   // the nodes in (t, t_new]
      while (true) {
        const int cnt = __popc(__ballot_sync(0xffffffffu, pt <= d.tn));
        last += cnt;
        if (cnt < 32) break;
        pt = last + lane < npoints ? points[last + lane] : INFINITY;
      }
      d.last = np = last;
      if (last > next) {
        d.dense = 1;
        ++dense_steps;
      }
      d.nt = d.tn;
      y_sc = prop;
      ksc0 = S.tot[17];
    }
    if (d.nt >= ctl.endpoint && np != npoints) status = kMissingSamples;
    if (d.nt < ctl.endpoint && C.attempts >= st->max_steps) status = kMaxSteps;
    if (!status && d.nt < ctl.endpoint)
      prepare_attempt(d.nt, hn, ctl.endpoint, C.attempts, st->max_steps, d.nh, status);
  }
  d.stop = status || d.nt >= ctl.endpoint ? 1 : 0;
  if (!d.stop) d.spec = has_points(d.nt, d.nh, ctl.endpoint, points, np, npoints);
  __syncwarp();
  if (lane == 0) {
    C.err = err;
    C.status = status;
    C.rejected = rejected;
    C.accepted = accepted;
    C.dense_steps = dense_steps;
    C.after_reject = after;
    C.next_point = np;
    C.y_sc = y_sc;
    C.ksc0 = ksc0;
    C.h = d.stop ? hn : d.nh;
    if (!d.stop) {
      ++C.attempts;
      C.min_h = fmin(C.min_h, d.nh);
      C.max_h = fmax(C.max_h, d.nh);
    }
  }
  share_dec<NR>(&S.dec, d);
}

// Entry v of a CTA's record (kRec); we(q, c, i): part i of error sum q of channel c.
template <class TailT, class F>
__device__ double record_entry(const TailT& S, int v, int parts, int c0, int c1, double h, bool late, F we) {
  double x = 0.0;
  if (v < 14) {
    const int c = v % 7, q = v / 7;
    if (c >= c0 && c < c1)
      for (int i = 0; i < parts; ++i) x += we(q, c, i);
  } else if (v < 18) {
    for (int s = 1; s <= 12; ++s) {
      const double w = v == 14 ? (s < 12 ? h * c_dop_b[s] : 0.0) : v == 15 ? c_dop_e5[s]
                       : v == 16 ? c_dop_e3[s] : (s == 12 ? 1.0 : 0.0);
      double k = 0.0;
      for (int i = 0; i < parts; ++i) k += S.wk[s][i];
      x += w * (4.0 * S.src[s] * k);
    }
  } else if (v == 18) {
    x = S.wait_flag ? 1.0 : 0.0;
  } else {
    x = late ? 1.0 : 0.0;
  }
  return x;
}

template <class TailT>
__device__ void init_tail(TailT& S, int parts, double endpoint) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    S.wait_flag = S.out_of_domain = 0;
    Ctl& C = S.ctl;
    C.min_h = INFINITY;
    C.max_h = 0.0;
    C.err = C.y_sc = C.ksc0 = 0.0;
    C.attempts = C.accepted = C.rejected = C.dense_steps = C.next_point = 0;
    C.status = C.after_reject = 0;
    S.jac[0] = 2.0 * endpoint;
    S.src[0] = source_value(-endpoint);
  }
  for (int i = tid; i < 13 * parts; i += blockDim.x) (&S.wk[0][0])[i] = 0.0;
}

// The stage times' Jacobian and source values of an attempt, one stage per thread.
template <class TailT>
__device__ __forceinline__ void stage_times(TailT& S, double t, double h) {
  const int tid = threadIdx.x;
  if (tid >= 1 && tid < 16) {
    const double ts = tid == 12 ? __dadd_rn(t, h) : __dadd_rn(t, __dmul_rn(c_dop_c[tid], h));
    if (fabs(ts) > RCMPS_SOURCE_AMAX * (1.0 + 1e-14)) S.out_of_domain = 1;
    S.jac[tid] = 2.0 * fabs(ts);
    S.src[tid] = source_value(ts);
  }
}

template <class TailT>
__device__ void write_stats(const TailT& S, const TrajState* st, bool packed) {
  const Ctl& C = S.ctl;
  TrajStats* o = st->stats;
  o->status = C.status;
  o->packed = packed ? 1 : 0;
  o->attempts = C.attempts;
  o->accepted = C.accepted;
  o->rejected = C.rejected;
  o->dense_steps = C.dense_steps;
  o->next_point = C.next_point;
  o->t = S.dec.nt;
  o->h = C.h;
  o->min_h = C.min_h;
  o->max_h = C.max_h;
  o->last_error = C.err;
  o->value = C.y_sc;
}

// The order-7 interpolation's coefficients of one entry from its stages kd (rcmps_dop_dense_mask), and
// its value at a node.
__device__ __forceinline__ void dense_coefficients(const double2* kd, double2 yo, double2 yn, double h, double2* cf) {
  const double2 delta = zsub(yn, yo);
  cf[0] = delta;
  cf[1] = zsub(zscale(h, kd[0]), delta);
  cf[2] = zsub(zscale(2.0, delta), zscale(h, zadd(kd[12], kd[0])));
#pragma unroll
  for (int row = 0; row < 4; ++row) {
    double2 v = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if ((rcmps_dop_dense_mask >> j) & 1u) v = zaxpy(h * c_dop_d[16 * row + j], kd[j], v);
    cf[3 + row] = v;
  }
}
__device__ __forceinline__ double2 dense_value(const double2* cf, double2 yo, double2 yn, double node, double t,
                                               double h, double tn) {
  if (node == tn) return yn;
  const double x = (node - t) / h;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < 7; ++i) acc = zscale(i % 2 == 0 ? x : 1.0 - x, zadd(acc, cf[6 - i]));
  return zadd(acc, yo);
}

template <int DP, bool LONE>
__global__ void __launch_bounds__(Smem<DP, LONE>::THREADS, 1)
tile_kernel(const TrajState* __restrict__ states, const double* __restrict__ points, int npoints, TrajControls ctl_in,
            Sync* __restrict__ sync) {
  using G = TG<DP>;
  using SM = Smem<DP, LONE>;
  constexpr int B = G::B, NB = G::NB, NR = G::NR, KS = G::KS, KB = G::KB, MT = G::MT, NTB = G::NTB;
  constexpr int EPT = G::EPT, BB = G::BB;
  constexpr size_t MAT = G::MAT;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = NR == 1 ? 0 : (int)cluster_rank();
  constexpr int teams = LONE ? kChannels : 1;
  const int cid = blockIdx.x / NR;
  const int sidx = cid / teams, team = cid % teams;
  const TrajState* st = states + sidx;
  if (!st->herm || st->z2 < 0) return;    // the state's whole grid of CTAs leaves here
  Sync* sy = sync + sidx;
  const int c0 = LONE ? team : 0, c1 = LONE ? team + 1 : kChannels;   // the team's channels
  const int bi = rank / NB, bj = rank % NB;   // tile (i, j)
  const bool owner_thread = tid < G::OWN;

  double2* sp = reinterpret_cast<double2*>(smem_raw);
  double2* s_panel = sp;                                   // [KS][2 MT][4][32]
  double2* s_rj = s_panel + G::PANEL;                      // [KS][NTB][2][32]
  double2* s_red = s_rj + G::RJ;                           // [RED]
  double* s_gat = reinterpret_cast<double*>(s_red + G::RED);   // [NR][NREC]
  // warp sums of the error norms [2 NC][NW]; without room of their own they take the partial tiles'
  // place, which is idle between a stage's products (other CTAs never write there)
  double* s_we = SM::GLOBAL_REC ? reinterpret_cast<double*>(s_red) : s_gat + 2 * SM::GAT;
  double2* s_k = s_red + G::RED + SM::GAT + (SM::GLOBAL_REC ? 0 : SM::WE);
  double2* s_x = s_k + SM::KVEC;
  double2* s_iv = s_x + SM::XCH;                           // [BB] the insertion of the owned tile
  Tail<G::NW>& S = *reinterpret_cast<Tail<G::NW>*>(s_iv + SM::IV);
  Ctl& C = S.ctl;

  // the barrier of a team: a cluster barrier, or the block's own; and the one of the warps that compute
  auto team_sync = [&]() {
    if constexpr (NR == 1) __syncthreads();
    else cluster_sync();
  };
  auto block_sync = [&]() {
    if constexpr (SM::COMM) asm volatile("bar.sync 1, %0;" ::"n"(G::NT) : "memory");
    else __syncthreads();
  };
  auto xload = [&](const double2* p) -> double2 {   // X and P of a team: L2, or shared memory when NB = 1
    if constexpr (NB == 1) return *p;
    else return __ldcg(p);
  };

  // ---------------------------------------------------------------- routes and ownership
  const bool packed = st->z2 > 0;
  const int half = st->d / 2;
  // packed Z2 state whose halves are whole blocks: structural zeros are skipped
  const bool zskip = packed && st->d == DP && NB % 2 == 0;
  const int ih = zskip && bi * B >= half ? 1 : 0, jh = zskip && bj * B >= half ? 1 : 0;
  auto parity = [](int c) { return (c & 1) ? 0 : 1; };   // F1, F3, A2, A4 are odd
  auto live = [&](int c) { return !zskip || jh == (ih ^ parity(c)); };     // tile (i, j) of X_c, Y_c, T
  auto rlive = [&](int c) { return !zskip || jh == ((1 - ih) ^ parity(c)); };   // tile (i, j) of P_c
  auto owns = [&](int c) {
    if (!live(c)) return false;
    return bi == bj || ((((c + bi + bj) & 1) != 0) == (bi > bj));
  };

  // buffers (trajectory.h): per channel MAT values each
  double2* const gz = NB == 1 ? s_x - (size_t)(LONE ? c0 : 0) * MAT : st->z;             // columns of X_c in B-fragment order
  double2* const gp = NB == 1 ? s_x + (LONE ? 1 : 7) * MAT - (size_t)(LONE ? c0 : 0) * MAT : st->P;   // P_c rows, A-fragment order
  double2* const gy = st->z + (size_t)kChannels * MAT;                                    // Y_c for the tile's owner
  constexpr size_t VEC = (size_t)kChannels * MAT;
  const size_t pstep = teams > 1 && NB > 1 ? VEC : 0;      // P by right-hand side when other teams read it
  // thread-private stage vectors: slot s of channel c, element e of the tile
  double2* const kbase = SM::KSM ? s_k : st->k + (size_t)rank * BB;
  auto kvec = [&](int slot, int c) -> double2* {
    if constexpr (SM::KSM) return s_k + slot * BB;
    else return kbase + (size_t)slot * VEC + (size_t)c * MAT;
  };
  constexpr int kSlotY = 16;   // y and the proposed y: slots 16, 17

  // element e = it * 256 + tid of the tile, in the order of the C fragments: 16 x 8 tile, entry, lane
  auto el_r = [&](int it) { const int e = it * G::OWN + tid; return 16 * (e / (128 * NTB)) + 8 * ((e >> 6) & 1) + ((e >> 2) & 7); };
  auto el_c = [&](int it) { const int e = it * G::OWN + tid; return 8 * ((e / 128) % NTB) + 2 * (e & 3) + ((e >> 5) & 1); };
  auto el_active = [&](int r, int c) { return owner_thread && (bi != bj || r <= c); };
  // ---------------------------------------------------------------- constant operands
  const int dir0 = c0 >= 3 ? 1 : 0;                 // direction of the first channel
  const bool both = c0 < 3 && c1 > 3;
  int panel_dir = dir0, rj_dir = dir0;              // what the resident set holds
  load_panel<DP>(st, dir0, bi, s_panel);
  load_rj<DP>(st, dir0, bj, s_rj);
  auto panel_of = [&](int dir) -> const double2* {
    if (!both) return s_panel;
    if (panel_dir != dir) {
      block_sync();
      load_panel<DP>(st, dir, bi, s_panel);
      block_sync();
      panel_dir = dir;
    }
    return s_panel;
  };
  auto rj_of = [&](int dir) -> const double2* {
    if (!both) return s_rj;
    if (rj_dir != dir) {
      block_sync();
      load_rj<DP>(st, dir, bj, s_rj);
      block_sync();
      rj_dir = dir;
    }
    return s_rj;
  };

  init_tail(S, G::NW, ctl_in.endpoint);
  __syncthreads();

  // The exchange of the records, by one warp of rank 0. post: lane v sums entry v over the team's CTAs
  // and publishes it; collect: the sum over the teams, and the decision on the attempt (t, h).
  const double N = packed ? 10.0 * half * half + 1.0 : (double)kChannels * st->d * st->d + 1.0;
  double team_tot = 0.0;
  auto post = [&](unsigned attempt) {
    const int own = !LONE ? lane : lane >= 14 ? lane - 12 : lane == c0 ? 0 : lane == 7 + c0 ? 1 : -1;
    team_tot = 0.0;
    if (lane < kRec && own >= 0)
      for (int g = 0; g < NR; ++g)
        team_tot += SM::GLOBAL_REC ? __ldcg(&sy->crec[g][own]) : s_gat[SM::NREC * g + own];
    if (teams > 1) {
      if (lane < kRec) sy->rec[team][attempt & 1][lane] = team_tot;
      __syncwarp();
      if (lane == 0) {
        __threadfence();
        flag_release(&sy->rflag[team], attempt);
      }
    }
  };
  auto collect = [&](unsigned attempt, double t, double h) {
    const long long next = C.next_point;
    const double pt = next + lane < npoints ? points[next + lane] : INFINITY;
    double tot = team_tot;
    if (teams > 1) {
      if (lane < teams) flag_wait(&sy->rflag[lane], attempt, &S.wait_flag);
      __syncwarp();
      tot = 0.0;
      if (lane < kRec)
        for (int g = 0; g < teams; ++g) tot += __ldcg(&sy->rec[g][attempt & 1][lane]);
      if (lane == 18 && S.wait_flag) tot = 1.0;
    }
    if (lane < kRec) S.tot[lane] = tot;
    __syncwarp();
    decide<NR>(S, st, ctl_in, points, npoints, pt, N, t, h);
  };

  if constexpr (SM::COMM) {
    // The warp behind the computing ones talks to the other teams, so that no flag's or remote tile's
    // round trip lies on their path: it takes part in every team barrier, brings the insertion of the
    // owned tile to shared memory between the two barriers of a right-hand side, and flags the P tile
    // after the second. Rank 0's also exchanges the records and decides on the attempt: while the
    // other warps go on with the dense stages when the step holds sample points (they are due unless
    // the attempt is rejected, a few in a hundred), so the exchange, 7 to 15 us, is off the path.
    if (warp == G::NW) {
      const int src = c_src[c0], dst = c_feeds[c0];
      const bool takes = src >= 0 && owns(c0);
      unsigned n = 0;
      auto serve = [&](auto&& after) {
        ++n;
        team_sync();
        after();
        if (takes) {
          if (lane < 2) flag_wait(&sy->pflag[src][lane ? bj * NB + bi : rank], n, &S.wait_flag);
          __syncwarp();
          const double2* ps = st->P + (size_t)(n & 31) * kChannels * MAT + (size_t)src * MAT;
          double2 a[BB / 32], b[BB / 32];
#pragma unroll
          for (int q = 0; q < BB / 32; ++q) {   // element q * 32 + lane of the tile
            const int r = 8 * ((q >> 1) & 1) + (lane >> 2), col = 8 * (q >> 2) + 2 * (lane & 3) + (q & 1);
            a[q] = __ldcg(ps + poff<DP>(bi, bj, r, col));
            b[q] = __ldcg(ps + poff<DP>(bj, bi, col, r));
          }
#pragma unroll
          for (int q = 0; q < BB / 32; ++q) s_iv[q * 32 + lane] = zadd(a[q], zconj(b[q]));
        }
        team_sync();
        if (dst >= 0 && lane == 0) {
          __threadfence();
          flag_release(&sy->pflag[c0][rank], n);
        }
      };
      serve([] {});
      team_sync();
      for (unsigned attempt = 1; !S.dec.stop; ++attempt) {
        const double t = S.dec.nt, h = S.dec.nh;
        const bool spec = S.dec.spec != 0;
        for (int s = 1; s <= 12; ++s) serve([] {});
        if (spec) {
          serve([&] { if (rank == 0) post(attempt); });
          serve([] {});
          if (rank == 0) collect(attempt, t, h);
          serve([] {});
        } else {
          team_sync();
          if (rank == 0) {
            post(attempt);
            collect(attempt, t, h);
          }
          team_sync();
        }
      }
      team_sync();
      return;
    }
  }

  int yslot = kSlotY, pslot = kSlotY + 1, k0slot = 0, k12slot = 12;
  auto kslot = [&](int s) { return s == 0 ? k0slot : s == 12 ? k12slot : s; };
  unsigned seq = 0;                      // right-hand sides so far
  double2 yown[LONE ? EPT : 1];          // Y(i, j) (+ its mirror on the diagonal) of the one owned channel

  // ---------------------------------------------------------------- one right-hand side
  // X_c of the team's channels is in gz; k of the owned tiles goes to slot ks_out. during(): work on the
  // thread's own stage vectors, done while the team's barrier completes.
  auto rhs = [&](int ks_out, double jac, double src, auto&& during) {
    ++seq;
    if constexpr (NR == 1 || B == 32) {
      team_sync();
    } else {
      cluster_arrive_release();
      during();
      cluster_wait_acquire();
    }
    double2* const pw = gp + (size_t)(seq & 31) * pstep;
    // ------------------------------------------------ phase 1
    {
      const int nt = warp % NTB, mg = (warp / NTB) % G::MG1, sl = warp / (NTB * G::MG1);
      double2 bz[2 * G::K1];
      auto fetch = [&](int c) {
        const int kh = zskip ? jh ^ parity(c) : 0;
        const int ka = kh * (KS / 2), kn = zskip ? KS / 2 : KS;
        const double2* zc = gz + (size_t)c * MAT + ((size_t)(bj * KS + ka) * NTB + nt) * 64 + lane;
#pragma unroll
        for (int q = 0; q < G::K1; ++q) {
          const int ks = sl + q * G::S1;
          if (ks < kn) {
            bz[2 * q] = xload(zc + (size_t)ks * NTB * 64);
            bz[2 * q + 1] = xload(zc + (size_t)ks * NTB * 64 + 32);
          } else {
            bz[2 * q] = bz[2 * q + 1] = make_double2(0.0, 0.0);
          }
        }
      };
      fetch(c0);
      for (int c = c0; c < c1; ++c) {
        const int dir = c >= 3 ? 1 : 0;
        const bool ql = live(c), rl = rlive(c);
        const int kh = zskip ? jh ^ parity(c) : 0;
        const int ka = kh * (KS / 2), kn = zskip ? KS / 2 : KS;
        const double2* panel = panel_of(dir);
        ZFrag acc[G::M1];
#pragma unroll
        for (int m = 0; m < G::M1; ++m) acc[m].zero();
#pragma unroll
        for (int q = 0; q < G::K1; ++q) {
          const int ks = sl + q * G::S1;
          if (ks < kn) {
            BFrag b;
            b.r[0] = bz[2 * q].x; b.r[1] = bz[2 * q + 1].x;
            b.i[0] = bz[2 * q].y; b.i[1] = bz[2 * q + 1].y;
            b.s[0] = b.r[0] + b.i[0]; b.s[1] = b.r[1] + b.i[1];
            const double2* pa = panel + ((size_t)(ka + ks) * 2 * MT + mg * G::M1) * 128 + lane;
#pragma unroll
            for (int m = 0; m < G::M1; ++m) {
              if (mg * G::M1 + m < MT ? !ql : !rl) continue;
              AFrag a;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const double2 v = pa[m * 128 + 32 * i];
                a.r[i] = v.x;
                a.i[i] = v.y;
                a.s[i] = v.x + v.y;
              }
              zmma(acc[m], a, b);
            }
          }
        }
        if (!LONE && c + 1 < c1) fetch(c + 1);   // in flight while this channel's partial tiles meet
        double2* red = s_red;
        auto deposit = [&](int slot, bool add) {
#pragma unroll
          for (int m = 0; m < G::M1; ++m) {
            double2* p = red + ((size_t)slot * G::T1 + (mg * G::M1 + m) * NTB + nt) * 128;
#pragma unroll
            for (int i = 0; i < 4; ++i) p[swz(i, lane)] = add ? zadd(p[swz(i, lane)], acc[m].value(i)) : acc[m].value(i);
          }
        };
        if constexpr (G::FOLD) {
          if (sl >= G::SF1) deposit(sl - G::SF1, false);
          block_sync();
          if (sl < G::SF1) deposit(sl, true);
        } else {
          deposit(sl, false);
        }
        block_sync();
        if (owner_thread) {
          // sum of the partial tiles at (r, col) of row tile group mq (0: Y, 1: P)
          auto total = [&](int mq, int r, int col) {
            const double2* p = red + ((size_t)(mq * MT + r / 16) * NTB + col / 8) * 128 + soff(r, col);
            double2 v = p[0];
#pragma unroll
            for (int s = 1; s < G::SF1; ++s) v = zadd(v, p[(size_t)s * G::T1 * 128]);
            return v;
          };
          const bool own = owns(c);
#pragma unroll
          for (int it = 0; it < EPT; ++it) {
            const int e = it * G::OWN + tid;
            if (rl) {
              const int l = e & 31, q = (e >> 5) & 3, mt = (e >> 7) % MT, kl = e / (128 * MT);
              const int r = 16 * mt + (l >> 2) + 8 * (q & 1), col = 8 * kl + (l & 3) + 4 * (q >> 1);
              const double2 v = total(1, r, col);
              const size_t off = (size_t)c * MAT + ((size_t)(bi * KS + bj * KB + kl) * MT + mt) * 128 + 32 * q + l;
              pw[off] = v;
              // a one-CTA team publishes P for the team that inserts it
              if (NB == 1 && teams > 1) st->P[(size_t)(seq & 31) * VEC + off] = v;
            }
            if (ql) {
              const int r = el_r(it), col = el_c(it);
              if (own) {
                double2 v = total(0, r, col);
                if (bi == bj) v = zadd(v, zconj(total(0, col, r)));
                if constexpr (LONE) yown[it] = v;
                else gy[VEC + (size_t)c * MAT + (size_t)rank * BB + e] = v;
              } else {
                // the entry whose mirror is element e of the owner's tile (j, i)
                gy[(size_t)c * MAT + (size_t)(bj * NB + bi) * BB + e] = zconj(total(0, col, r));
              }
            }
          }
        }
        if constexpr (!LONE) block_sync();
      }
      if (!SM::COMM && teams > 1) {
        // P tiles that another team inserts: complete, then flagged
        bool feeds = false;
        for (int c = c0; c < c1; ++c) {
          const int f = c_feeds[c];
          feeds |= f >= 0 && (f < c0 || f >= c1);
        }
        if (feeds) {
          block_sync();
          if (tid == 0) {
            __threadfence();
            for (int c = c0; c < c1; ++c) {
              const int f = c_feeds[c];
              if (f >= 0 && (f < c0 || f >= c1)) flag_release(&sy->pflag[c][rank], seq);
            }
          }
        }
      }
    }
    if constexpr (NR == 1) during();
    if constexpr (SM::COMM || NR == 1) {
      team_sync();
    } else {
      // the flags of the tiles that other teams insert are awaited while the barrier completes
      cluster_arrive_release();
      if constexpr (B == 32) during();   // the owners are the last at the first barrier
      for (int c = c0; c < c1; ++c) {
        const int s = c_src[c];
        if (s < 0 || (s >= c0 && s < c1) || !owns(c)) continue;
        if (lane < 2) flag_wait(&sy->pflag[s][lane ? bj * NB + bi : rank], seq, &S.wait_flag);
        __syncwarp();
      }
      cluster_wait_acquire();
    }
    // ------------------------------------------------ phase 2
    {
      const int sl = warp / (G::MG2 * G::NG2), ng = warp % G::NG2, mg = (warp / G::NG2) % G::MG2;
      const bool works = sl < G::S2;
      // P rows of block i: the half with nonzero columns of R^dag's column block j
      const int ka = zskip ? (1 - jh) * (KS / 2) : 0, kn = zskip ? KS / 2 : KS;
      for (int c = c0; c < c1; ++c) {
        if (!owns(c)) continue;
        const int dir = c >= 3 ? 1 : 0;
        const double2* rj = rj_of(dir);
        double2 av[4 * G::K2];
#pragma unroll
        for (int q = 0; q < G::K2; ++q) {
          const int ks = sl + q * G::S2;
          const double2* pa = pw + (size_t)c * MAT + ((size_t)(bi * KS + ka + ks) * MT + mg) * 128 + lane;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            av[4 * q + i] = works && ks < kn ? xload(pa + 32 * i) : make_double2(0.0, 0.0);
        }
        // the epilogue's operands, in flight during the products (B = 32 loads them after: registers)
        const int s = c_src[c];
        const bool remote = !SM::COMM && s >= 0 && (s < c0 || s >= c1);
        const double2* ps = (remote ? st->P + (size_t)(seq & 31) * VEC : pw) + (size_t)(s >= 0 ? s : 0) * MAT;
        const double2* fx = c == 0 ? st->fixed0 : c == 6 ? st->fixed6 : nullptr;
        double2 ev[EPT], iv[EPT];   // Y's other half, the insertion P_s + P_s^dag
        auto operands = [&](int it) {
          const int e = it * G::OWN + tid, r = el_r(it), col = el_c(it);
          double2 v = make_double2(0.0, 0.0);
          if constexpr (LONE) v = yown[it];
          else v = __ldcg(gy + VEC + (size_t)c * MAT + (size_t)rank * BB + e);
          if (bi != bj) {
            const double2 o = __ldcg(gy + (size_t)c * MAT + (size_t)rank * BB + e);
            v = zadd(v, o);
          }
          ev[it] = v;
          v = make_double2(0.0, 0.0);
          if (SM::COMM) {
            if (s >= 0) v = s_iv[e];
          } else if (s >= 0) {
            const double2 *p1 = ps + poff<DP>(bi, bj, r, col), *p2 = ps + poff<DP>(bj, bi, col, r);
            const double2 a = remote ? __ldcg(p1) : xload(p1), b = remote ? __ldcg(p2) : xload(p2);
            v = zadd(a, zconj(b));
          }
          iv[it] = v;
        };
        if (B == 16 && owner_thread) {
#pragma unroll
          for (int it = 0; it < EPT; ++it) operands(it);
        }
        ZFrag acc[G::N2];
#pragma unroll
        for (int n = 0; n < G::N2; ++n) acc[n].zero();
        if (works) {
#pragma unroll
          for (int q = 0; q < G::K2; ++q) {
            const int ks = sl + q * G::S2;
            if (ks < kn) {
              AFrag a;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                a.r[i] = av[4 * q + i].x;
                a.i[i] = av[4 * q + i].y;
                a.s[i] = a.r[i] + a.i[i];
              }
              const double2* pb = rj + ((size_t)(ka + ks) * NTB + ng * G::N2) * 64 + lane;
#pragma unroll
              for (int n = 0; n < G::N2; ++n) {
                BFrag b;
                const double2 v0 = pb[n * 64], v1 = pb[n * 64 + 32];
                b.r[0] = v0.x; b.r[1] = v1.x;
                b.i[0] = v0.y; b.i[1] = v1.y;
                b.s[0] = v0.x + v0.y; b.s[1] = v1.x + v1.y;
                zmma(acc[n], a, b);
              }
            }
          }
        }
        double2* red = s_red;
        auto deposit = [&](int slot, bool add) {
#pragma unroll
          for (int n = 0; n < G::N2; ++n) {
            double2* p = red + ((size_t)slot * G::T2 + mg * NTB + ng * G::N2 + n) * 128;
#pragma unroll
            for (int i = 0; i < 4; ++i) p[swz(i, lane)] = add ? zadd(p[swz(i, lane)], acc[n].value(i)) : acc[n].value(i);
          }
        };
        if constexpr (G::FOLD) {
          if (sl >= G::SF2) deposit(sl - G::SF2, false);
          block_sync();
          if (sl < G::SF2) deposit(sl, true);
        } else {
          if (works) deposit(sl, false);
        }
        block_sync();
        if (owner_thread) {
          if (B == 32) {
#pragma unroll
            for (int it = 0; it < EPT; ++it) operands(it);
          }
          double2* kout = kvec(ks_out, c);
#pragma unroll
          for (int it = 0; it < EPT; ++it) {
            const int e = it * G::OWN + tid, r = el_r(it), col = el_c(it);
            if (!el_active(r, col)) continue;
            const double2* p = red + ((size_t)(r / 16) * NTB + col / 8) * 128 + soff(r, col);
            double2 v = p[0];
#pragma unroll
            for (int q = 1; q < G::SF2; ++q) v = zadd(v, p[(size_t)q * G::T2 * 128]);
            v = zscale(jac, zadd(v, ev[it]));
            if (s >= 0) v = zaxpy(src * c_coef[c], iv[it], v);
            if (fx) v = zaxpy(src, __ldg(fx + (size_t)(bi * B + r) * DP + bj * B + col), v);
            if (bi == bj && r == col) v.y = 0.0;
            kout[e] = v;
          }
        }
        if constexpr (!LONE) block_sync();
      }
    }
  };

  // element e of X_c and its mirror -> gz
  auto put_z = [&](int c, int it, int r, int col, double2 v) {
    double2* z = gz + (size_t)c * MAT;
    z[zoff<DP>(bi, bj, r, col)] = v;
    if (bi != bj || r != col) z[zoff<DP>(bj, bi, col, r)] = zconj(v);
  };

  // Of a stage vector y + h sum_j w_j k_j only the last term waits for the right-hand side before it: the
  // others are summed during that right-hand side, in the same order (a register, or slots 18 and 19).
  // At DP = 128 the stage vectors' loads are the owners' critical path either way and the detour
  // through a slot costs more than the wait hides (Z2 D = 128 16.0 -> 18.2 us, D = 64 6.8 -> 6.1):
  // there the sum is taken when it is used.
  constexpr bool EARLY = DP != 128;
  constexpr int kSlotSum = 18;
  double2 psum[2];
  auto sum_put = [&](int q, int c, int it, double2 v) {
    if constexpr (SM::KSM) psum[q] = v;
    else kvec(kSlotSum + q, c)[it * G::OWN + tid] = v;
  };
  auto sum_get = [&](int q, int c, int it) -> double2 {
    if constexpr (SM::KSM) return psum[q];
    else return kvec(kSlotSum + q, c)[it * G::OWN + tid];
  };
  // y + the first n terms of the weights w (at most MAX) of one entry
  auto entry_sum = [&](const double* w, int n, double h, auto max, int c, int it) -> double2 {
    constexpr int MAX = decltype(max)::value;
    const int e = it * G::OWN + tid;
    double2 kv[MAX];
#pragma unroll
    for (int j = 0; j < MAX; ++j)
      kv[j] = j < n && w[j] != 0.0 ? kvec(kslot(j), c)[e] : make_double2(0.0, 0.0);
    double2 v = kvec(yslot, c)[e];
#pragma unroll
    for (int j = 0; j < MAX; ++j) v = zaxpy(j < n ? h * w[j] : 0.0, kv[j], v);
    return v;
  };
  // both error estimates of one entry without k_12
  auto entry_errors = [&](int c, int it, double2& e5, double2& e3) {
    double2 kv[12];
#pragma unroll
    for (int j = 0; j < 12; ++j) kv[j] = kvec(kslot(j), c)[it * G::OWN + tid];
    e5 = e3 = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      e5 = zaxpy(c_dop_e5[j], kv[j], e5);
      e3 = zaxpy(c_dop_e3[j], kv[j], e3);
    }
  };
  auto partial_sum = [&](const double* w, int n, double h, auto max) {
    if constexpr (EARLY) {
      for (int c = c0; c < c1; ++c) {
        if (!owns(c) || !owner_thread) continue;
#pragma unroll
        for (int it = 0; it < EPT; ++it) sum_put(0, c, it, entry_sum(w, n, h, max, c, it));
      }
    }
  };
  auto partial_errors = [&]() {
    if constexpr (EARLY) {
      for (int c = c0; c < c1; ++c) {
        if (!owns(c) || !owner_thread) continue;
#pragma unroll
        for (int it = 0; it < EPT; ++it) {
          double2 e5, e3;
          entry_errors(c, it, e5, e3);
          sum_put(0, c, it, e5);
          sum_put(1, c, it, e3);
        }
      }
    }
  };

  // ---------------------------------------------------------------- start: y = 0, k0 = f(-a, 0)
  for (int c = c0; c < c1; ++c) {
    if (!owns(c) || !owner_thread) continue;
#pragma unroll
    for (int it = 0; it < EPT; ++it) {
      const int r = el_r(it), col = el_c(it);
      if (!el_active(r, col)) continue;
      const double2 z0 = make_double2(0.0, 0.0);
      kvec(yslot, c)[it * G::OWN + tid] = z0;
      put_z(c, it, r, col, z0);
    }
  }
  rhs(k0slot, S.jac[0], S.src[0], [] {});

  const double atol = st->atol, rtol = st->rtol;
  const unsigned long long t_start = global_ns();
  if (rank == 0 && warp == 0) first_decision<NR>(S, st, ctl_in, points, npoints);
  team_sync();

  unsigned attempt = 0;
  bool stop = S.dec.stop != 0;
  while (!stop) {
    ++attempt;
    const double t = S.dec.nt, h = S.dec.nh;
    const bool spec = S.dec.spec != 0;
    block_sync();
    stage_times(S, t, h);
    block_sync();
    // ------------------------------------------------------------ stages 1..12
    for (int s = 1; s <= 12; ++s) {
      const double* w = s == 12 ? c_dop_b : c_dop_a + 16 * s;
      double part = 0.0;
      for (int c = c0; c < c1; ++c) {
        if (!owns(c) || !owner_thread) continue;
#pragma unroll
        for (int it = 0; it < EPT; ++it) {
          const int e = it * G::OWN + tid, r = el_r(it), col = el_c(it);
          if (!el_active(r, col)) continue;
          double2 base;
          if constexpr (EARLY) base = s == 1 ? kvec(yslot, c)[e] : sum_get(0, c, it);
          else base = entry_sum(w, s - 1, h, std::integral_constant<int, 11>(), c, it);
          const double2 v = zaxpy(h * w[s - 1], kvec(kslot(s - 1), c)[e], base);
          put_z(c, it, r, col, v);
          if (s == 12) kvec(pslot, c)[e] = v;
          if (c == 2) {
            const double2 sv = __ldg(st->S + (size_t)(bi * B + r) * DP + bj * B + col);
            part += (bi == bj && r == col ? 1.0 : 2.0) * (v.x * sv.x - v.y * sv.y);
          }
        }
      }
      if (c0 <= 2 && 2 < c1) {
        part = warp_sum(part);
        if (lane == 0) S.wk[s][warp] = part;
      }
      rhs(kslot(s), S.jac[s], S.src[s], [&] {
        if (s < 12) partial_sum(s == 11 ? c_dop_b : c_dop_a + 16 * (s + 1), s, h, std::integral_constant<int, 11>());
        else partial_errors();
      });
    }
    // ------------------------------------------------------------ error norms
    if constexpr (SM::GLOBAL_REC) block_sync();   // the last stage's partial tiles have been read
    for (int c = c0; c < c1; ++c) {
      double s5 = 0.0, s3 = 0.0;
      if (owns(c) && owner_thread) {
#pragma unroll
      for (int it = 0; it < EPT; ++it) {
        const int e = it * G::OWN + tid, r = el_r(it), col = el_c(it);
        if (!el_active(r, col)) continue;
        const int row = bi * B + r, cl = bj * B + col;
        const double wt = norm_weight(packed, half, c, row, cl);
        if (wt == 0.0) continue;
        const double2 k12 = kvec(kslot(12), c)[e];
        double2 e5, e3;
        if constexpr (EARLY) {
          e5 = sum_get(0, c, it);
          e3 = sum_get(1, c, it);
        } else {
          entry_errors(c, it, e5, e3);
        }
        e5 = zaxpy(c_dop_e5[12], k12, e5);
        e3 = zaxpy(c_dop_e3[12], k12, e3);
        const double2 yo = kvec(yslot, c)[e], yn = kvec(pslot, c)[e];
        const double scale = atol + rtol * fmax(hypot(yo.x, yo.y), hypot(yn.x, yn.y));
        s5 += wt * (zabs2(e5) / (scale * scale));
        s3 += wt * (zabs2(e3) / (scale * scale));
      }
      }
      s5 = warp_sum(s5);
      s3 = warp_sum(s3);
      if (lane == 0) {
        s_we[(LONE ? 0 : c) * G::NW + warp] = s5;
        s_we[(SM::NC + (LONE ? 0 : c)) * G::NW + warp] = s3;
      }
    }
    block_sync();
    // the CTA's record (kRec; a lone channel's: both error sums, then 14..19) into rank 0
    if (tid < SM::NREC) {
      const int v = !LONE ? tid : tid < 2 ? 7 * tid + c0 : tid + 12;
      const double x = record_entry(S, v, G::NW, c0, c1, h, ctl_in.max_ns && global_ns() - t_start >= ctl_in.max_ns,
                                    [&](int q, int c, int i) { return s_we[(q * SM::NC + (LONE ? 0 : c)) * G::NW + i]; });
      if constexpr (SM::GLOBAL_REC) sy->crec[rank][tid] = x;
      else if constexpr (NR == 1) s_gat[tid] = x;
      else dsmem_store_f64(s_gat + rank * SM::NREC + tid, 0, x);
    }
    bool dense = SM::COMM && spec;
    if constexpr (SM::COMM) {
      if (!spec) {
        team_sync();
        team_sync();
      }
    } else {
      team_sync();
      if (rank == 0 && warp == 0) {
        post(attempt);
        collect(attempt, t, h);
      }
      team_sync();
      dense = S.dec.accept && S.dec.dense;
    }
    if (dense) {
        // dense stages 13..15
        partial_sum(c_dop_a + 16 * 13, 12, h, std::integral_constant<int, 12>());
        for (int s = 13; s < 16; ++s) {
          for (int c = c0; c < c1; ++c) {
            if (!owns(c) || !owner_thread) continue;
#pragma unroll
            for (int it = 0; it < EPT; ++it) {
              const int e = it * G::OWN + tid, r = el_r(it), col = el_c(it);
              if (!el_active(r, col)) continue;
              double2 base;
              if constexpr (EARLY) base = sum_get(0, c, it);
              else base = entry_sum(c_dop_a + 16 * s, s - 1, h, std::integral_constant<int, 14>(), c, it);
              put_z(c, it, r, col, zaxpy(h * c_dop_a[16 * s + s - 1], kvec(kslot(s - 1), c)[e], base));
            }
          }
          rhs(s, S.jac[s], S.src[s], [&] {
            if (s < 15) partial_sum(c_dop_a + 16 * (s + 1), s, h, std::integral_constant<int, 14>());
          });
        }
    }
    stop = S.dec.stop != 0;
    if (S.dec.accept) {
      if (dense) {
        // order-7 interpolation at the nodes in (t, t_new]
        const double tn = S.dec.tn;
        const long long first = S.dec.first, last = S.dec.last;
        for (int c = c0; c < c1; ++c) {
          if (!owner_thread) continue;
          if (!owns(c)) continue;
#pragma unroll 1
          for (int it = 0; it < EPT; ++it) {
            const int e = it * G::OWN + tid, r = el_r(it), col = el_c(it);
            if (!el_active(r, col)) continue;
            double2 kd[16];
#pragma unroll
            for (int j = 0; j < 16; ++j)
              kd[j] = ((rcmps_dop_dense_mask >> j) & 1u) ? kvec(kslot(j), c)[e] : make_double2(0.0, 0.0);
            const double2 yo = kvec(yslot, c)[e], yn = kvec(pslot, c)[e];
            double2 cf[7];
            dense_coefficients(kd, yo, yn, h, cf);
            double2* o1 = st->samples + (size_t)c * MAT + (size_t)(bi * B + r) * DP + bj * B + col;
            double2* o2 = st->samples + (size_t)c * MAT + (size_t)(bj * B + col) * DP + bi * B + r;
            for (long long node = first; node < last; ++node) {
              const double2 v = dense_value(cf, yo, yn, points[node], t, h, tn);
              o1[(size_t)node * VEC] = v;
              if (bi != bj || r != col) o2[(size_t)node * VEC] = zconj(v);
            }
          }
        }
      }
      // commit: y <- proposed, f <- k12
      int x = yslot;
      yslot = pslot;
      pslot = x;
      x = k0slot;
      k0slot = k12slot;
      k12slot = x;
    }
  }
  if (rank == 0 && team == 0 && tid == 0) write_stats(S, st, packed);
  team_sync();   // no CTA leaves while another may still write into its shared memory
}

// ---------------------------------------------------------------- one team per state, B = 16
// The same tiles for a batch that fills the GPU: one team holds all seven channels, and each channel's
// 16 x 8 half tile is one warp's (DP 48, 64) or both are (DP 16, 32, where two CTAs share an SM). All
// channels go through a phase side by side, so a right-hand side exposes each latency once and not
// once per channel. The columns j of every X_c, and later the rows i of the owned P_c, land in shared
// memory by one bulk copy per channel (they are contiguous in fragment order). A warp sums its K slices
// in the order in which tile_kernel's warps meet, and keeps the same partial sums of the error norm:
// the two kernels give the same bits. 32 x D = 64 (16 of them Z2): 24 us per right-hand side of a random
// state on 16 CTAs, 8 states at once, against 119 us on 4 CTAs in the row-block kernel with 32 at once;
// bound by the MMAs (13.5 of the 24 us; 9.4 at the DMMA peak) and, between them, by barriers and the stage
// vectors' round trips to L2 (its bandwidth is at 10%; two CTAs per SM at D = 32: 17%).
template <int DP>
struct Wide {
  using G = TG<DP>;
  static_assert(G::B == 16 && G::MT == 1 && G::NTB == 2, "16 x 16 tiles");
  static constexpr int NPT = DP <= 32 ? 2 : 1;          // column tiles per warp
  static constexpr int NW = 2 * kChannels / NPT;
  static constexpr int NT = 32 * NW;
  static constexpr int XC = 16 * DP;                    // columns of X_c or rows of P_c
  static constexpr int PARTS = 8;                       // partial sums of a tile: column tile, entry
  static constexpr int XB = kChannels * XC * (G::NB == 1 ? 2 : 1);
  static constexpr int GAT = G::NR * kRec / 2, WE = kChannels * PARTS;
  static constexpr size_t BYTES = (size_t)(2 * (G::PANEL + G::RJ) + XB + GAT + WE) * 16 + sizeof(Tail<PARTS>) + 64;
  static_assert(BYTES <= (DP <= 32 ? 232448 / 2 - 1024 : 232448), "shared memory per CTA");
};

// tot = sum over S slices of K-steps (slice, slice + S, ..) of the 16 x 8 product, slice by slice.
// A: fragments [kstep][sa], B: [kstep][sb] (double2 strides per k-step), lane offset included.
template <int S, int K>
__device__ __forceinline__ void slice_product(const double2* A, int sa, const double2* Bf, int sb, int kn, double2* tot) {
#pragma unroll
  for (int sl = 0; sl < S; ++sl) {
    ZFrag acc;
    acc.zero();
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const int ks = sl + q * S;
      if (ks < kn) {
        AFrag a;
        BFrag b;
        const double2 *pa = A + ks * sa, *pb = Bf + ks * sb;
        const double2 b0 = pb[0], b1 = pb[32];
        b.r[0] = b0.x; b.r[1] = b1.x;
        b.i[0] = b0.y; b.i[1] = b1.y;
        b.s[0] = b0.x + b0.y; b.s[1] = b1.x + b1.y;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double2 v = pa[32 * i];
          a.r[i] = v.x;
          a.i[i] = v.y;
          a.s[i] = v.x + v.y;
        }
        zmma(acc, a, b);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) tot[i] = sl == 0 ? acc.value(i) : zadd(tot[i], acc.value(i));
  }
}

template <int DP>
__global__ void __launch_bounds__(Wide<DP>::NT, DP <= 32 ? 2 : 1)
wide_kernel(const TrajState* __restrict__ states, const double* __restrict__ points, int npoints, TrajControls ctl_in) {
  using G = TG<DP>;
  using W = Wide<DP>;
  constexpr int B = 16, NB = G::NB, NR = G::NR, KS = G::KS, BB = G::BB, NPT = W::NPT;
  constexpr size_t MAT = G::MAT, VEC = (size_t)kChannels * MAT;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = NR == 1 ? 0 : (int)cluster_rank();
  const TrajState* st = states + blockIdx.x / NR;
  if (!st->herm || st->z2 < 0) return;    // the whole cluster leaves here
  const int bi = rank / NB, bj = rank % NB;

  double2* sp = reinterpret_cast<double2*>(smem_raw);
  double2* s_panel = sp;                                 // [2][KS][2][4][32]
  double2* s_rj = s_panel + 2 * G::PANEL;                // [2][KS][2][2][32]
  double2* s_x = s_rj + 2 * G::RJ;                       // [7][XC] (NB = 1: X, then P)
  double* s_gat = reinterpret_cast<double*>(s_x + W::XB);   // [NR][kRec]
  double* s_we = s_gat + 2 * W::GAT;                     // [2][7][PARTS]
  Tail<W::PARTS>& S = *reinterpret_cast<Tail<W::PARTS>*>(s_we + 2 * W::WE);
  uint64_t* s_full = reinterpret_cast<uint64_t*>(&S + 1);   // [7] a channel's copy landed

  auto team_sync = [&]() {
    if constexpr (NR == 1) __syncthreads();
    else cluster_sync();
  };
  const bool packed = st->z2 > 0;
  const int half = st->d / 2;
  const bool zskip = packed && st->d == DP && NB % 2 == 0;
  const int ih = zskip && bi * B >= half ? 1 : 0, jh = zskip && bj * B >= half ? 1 : 0;
  const int kn = zskip ? KS / 2 : KS;
  auto parity = [](int c) { return (c & 1) ? 0 : 1; };
  auto live = [&](int c) { return !zskip || jh == (ih ^ parity(c)); };
  auto owns = [&](int c) { return live(c) && (bi == bj || ((((c + bi + bj) & 1) != 0) == (bi > bj))); };

  // the warp's channel and what the CTA does with it
  const int c = NPT == 2 ? warp : warp >> 1, nt0 = NPT == 2 ? 0 : warp & 1;
  const int dir = c >= 3 ? 1 : 0, src_ch = c_src[c];
  const bool ql = live(c), rl = !zskip || jh == ((1 - ih) ^ parity(c)), own = owns(c);
  const int kx = zskip ? (jh ^ parity(c)) * (KS / 2) : 0;   // first k-step of phase 1
  const int kp = zskip ? (1 - jh) * (KS / 2) : 0;           // and of phase 2
  const double coef = c_coef[c];
  const double2* fx = c == 0 ? st->fixed0 : c == 6 ? st->fixed6 : nullptr;

  double2* const gz = NB == 1 ? s_x : st->z;
  double2* const gp = NB == 1 ? s_x + kChannels * W::XC : st->P;
  double2* const gy = st->z + VEC;          // mirrored Y entries for the tile's owner
  double2* const gyo = gy + VEC + (size_t)c * MAT + (size_t)rank * BB;   // the owner's Y, thread-private
  double2* const gyx = gy + (size_t)c * MAT + (size_t)rank * BB;
  double2* const kb = st->k + (size_t)c * MAT + (size_t)rank * BB;       // thread-private stage vectors
  auto kvec = [&](int slot) { return kb + (size_t)slot * VEC; };
  // entry i of column tile nt: row, column, index in C-fragment order
  auto el_r = [&](int i) { return 8 * (i >> 1) + (lane >> 2); };
  auto el_c = [&](int nt, int i) { return 8 * nt + 2 * (lane & 3) + (i & 1); };
  auto el_e = [&](int nt, int i) { return (nt * 4 + i) * 32 + lane; };
  auto active = [&](int r, int col) { return bi != bj || r <= col; };

  load_panel<DP>(st, 0, bi, s_panel);
  load_panel<DP>(st, 1, bi, s_panel + G::PANEL);
  load_rj<DP>(st, 0, bj, s_rj);
  load_rj<DP>(st, 1, bj, s_rj + G::RJ);
  const double2* const panel = s_panel + dir * G::PANEL + lane;
  const double2* const rj = s_rj + dir * G::RJ + lane;
  init_tail(S, W::PARTS, ctl_in.endpoint);
  for (int i = tid; i < 2 * W::WE; i += W::NT) s_we[i] = 0.0;
  if (NB > 1 && tid == 0) {
    for (int i = 0; i < kChannels; ++i) mbar_init(&s_full[i], 1);
    fence_mbar_init();
  }
  __syncthreads();

  int yslot = 16, pslot = 17, k0slot = 0, k12slot = 12;
  auto kslot = [&](int s) { return s == 0 ? k0slot : s == 12 ? k12slot : s; };
  unsigned seq = 0;
  uint32_t phase = 0;       // of the channel's barrier
  auto landed = [&]() {
    if constexpr (NB > 1) {
      if (!*(volatile int*)&S.wait_flag) mbar_wait(&s_full[c], phase, &S.wait_flag);
      phase ^= 1;
    }
  };

  auto rhs = [&](int ks_out, double jac, double src, auto&& during) {   // during(): as in tile_kernel
    ++seq;
    if constexpr (NR == 1) {
      during();
      team_sync();
    } else {
      fence_proxy_async_global();
      cluster_arrive_release();
      during();
      cluster_wait_acquire();
    }
    if (NB > 1 && tid == 0) {
      fence_proxy_async_global();
      fence_proxy_async_shared();
      for (int q = 0; q < kChannels; ++q) {
        const int ka = zskip ? (jh ^ parity(q)) * (KS / 2) : 0;
        mbar_expect_tx(&s_full[q], kn * 128 * 16);
        bulk_g2s(s_x + q * W::XC, gz + (size_t)q * MAT + (size_t)(bj * KS + ka) * 128, kn * 128 * 16, &s_full[q]);
      }
    }
    landed();
#pragma unroll
    for (int it = 0; it < NPT; ++it) {
      const int nt = nt0 + it;
      const double2* xb = s_x + c * W::XC + nt * 64 + lane;
      if (ql) {
        double2 y[4];
        slice_product<G::S1, G::K1>(panel + kx * 256, 256, xb, 128, kn, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = el_r(i), col = el_c(nt, i);
          if (own) gyo[el_e(nt, i)] = y[i];
          // the mirror entry, in the order of the owner's tile (j, i)
          if (!own || bi == bj) gy[(size_t)c * MAT + (size_t)(bj * NB + bi) * BB + (r / 8) * 128 + roff(col, r)] = zconj(y[i]);
        }
      }
      if (rl) {
        double2 p[4];
        slice_product<G::S1, G::K1>(panel + kx * 256 + 128, 256, xb, 128, kn, p);
#pragma unroll
        for (int i = 0; i < 4; ++i) gp[(size_t)c * MAT + poff<DP>(bi, bj, el_r(i), el_c(nt, i))] = p[i];
      }
    }
    if constexpr (NB > 1) fence_proxy_async_global();
    team_sync();
    if (NB > 1 && tid == 0) {
      fence_proxy_async_global();
      fence_proxy_async_shared();
      for (int q = 0; q < kChannels; ++q) {
        if (!owns(q)) continue;
        mbar_expect_tx(&s_full[q], kn * 128 * 16);
        bulk_g2s(s_x + q * W::XC, gp + (size_t)q * MAT + (size_t)(bi * KS + kp) * 128, kn * 128 * 16, &s_full[q]);
      }
    }
    if (own) {
      // the epilogue's operands first: they cross L2 while the rows of P land
      double2 ev[NPT][4], iv[NPT][4];
#pragma unroll
      for (int it = 0; it < NPT; ++it)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int nt = nt0 + it, r = el_r(i), col = el_c(nt, i), e = el_e(nt, i);
          ev[it][i] = zadd(__ldcg(gyo + e), __ldcg(gyx + e));
          iv[it][i] = make_double2(0.0, 0.0);
          if (src_ch >= 0) {
            const double2 *p1 = gp + (size_t)src_ch * MAT + poff<DP>(bi, bj, r, col),
                          *p2 = gp + (size_t)src_ch * MAT + poff<DP>(bj, bi, col, r);
            if constexpr (NB == 1) iv[it][i] = zadd(*p1, zconj(*p2));
            else iv[it][i] = zadd(__ldcg(p1), zconj(__ldcg(p2)));
          }
        }
      landed();
      double2* kout = kvec(ks_out);
#pragma unroll
      for (int it = 0; it < NPT; ++it) {
        const int nt = nt0 + it;
        const double2* pb = (NB == 1 ? gp + (size_t)c * MAT : s_x + c * W::XC) + lane;
        double2 tt[4];
        slice_product<G::S2, G::K2>(pb, 128, rj + kp * 128 + nt * 64, 128, kn, tt);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = el_r(i), col = el_c(nt, i);
          double2 v = zscale(jac, zadd(tt[i], ev[it][i]));
          if (src_ch >= 0) v = zaxpy(src * coef, iv[it][i], v);
          if (fx) v = zaxpy(src, __ldg(fx + (size_t)(bi * B + r) * DP + bj * B + col), v);
          if (bi == bj && r == col) v.y = 0.0;
          if (active(r, col)) kout[el_e(nt, i)] = v;
        }
      }
    }
  };
  auto put_z = [&](int r, int col, double2 v) {
    double2* z = gz + (size_t)c * MAT;
    z[zoff<DP>(bi, bj, r, col)] = v;
    if (bi != bj || r != col) z[zoff<DP>(bj, bi, col, r)] = zconj(v);
  };

  // Stage sums and error estimates as in tile_kernel: with one column tile per warp all but the last
  // term is summed during the right-hand side before (slots 18 and 19); with two, where two CTAs share an
  // SM and the stage vectors' L2 round trips set the pace, when it is used.
  constexpr bool EARLY = NPT == 1;
  auto entry_sum = [&](const double* w, int n, double h, auto max, int e) -> double2 {
    constexpr int MAX = decltype(max)::value;
    double2 kv[MAX];
#pragma unroll
    for (int j = 0; j < MAX; ++j) kv[j] = j < n && w[j] != 0.0 ? kvec(kslot(j))[e] : make_double2(0.0, 0.0);
    double2 v = kvec(yslot)[e];
#pragma unroll
    for (int j = 0; j < MAX; ++j) v = zaxpy(j < n ? h * w[j] : 0.0, kv[j], v);
    return v;
  };
  auto entry_errors = [&](int e, double2& e5, double2& e3) {
    double2 kv[12];
#pragma unroll
    for (int j = 0; j < 12; ++j) kv[j] = kvec(kslot(j))[e];
    e5 = e3 = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      e5 = zaxpy(c_dop_e5[j], kv[j], e5);
      e3 = zaxpy(c_dop_e3[j], kv[j], e3);
    }
  };
  auto partial_sum = [&](const double* w, int n, double h, auto max) {
    if constexpr (EARLY) {
      if (!own) return;
#pragma unroll 2
      for (int i = 0; i < 4; ++i)
        if (active(el_r(i), el_c(nt0, i))) kvec(18)[el_e(nt0, i)] = entry_sum(w, n, h, max, el_e(nt0, i));
    }
  };
  auto partial_errors = [&]() {
    if constexpr (EARLY) {
      if (!own) return;
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        double2 e5, e3;
        entry_errors(el_e(nt0, i), e5, e3);
        kvec(18)[el_e(nt0, i)] = e5;
        kvec(19)[el_e(nt0, i)] = e3;
      }
    }
  };

  // ---------------------------------------------------------------- start: y = 0, k0 = f(-a, 0)
  if (own) {
#pragma unroll
    for (int it = 0; it < NPT; ++it)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int nt = nt0 + it, r = el_r(i), col = el_c(nt, i);
        if (!active(r, col)) continue;
        kvec(yslot)[el_e(nt, i)] = make_double2(0.0, 0.0);
        put_z(r, col, make_double2(0.0, 0.0));
      }
  }
  rhs(k0slot, S.jac[0], S.src[0], [] {});

  const double atol = st->atol, rtol = st->rtol;
  const double N = packed ? 10.0 * half * half + 1.0 : (double)kChannels * st->d * st->d + 1.0;
  const unsigned long long t_start = global_ns();
  if (rank == 0 && warp == 0) first_decision<NR>(S, st, ctl_in, points, npoints);
  team_sync();

  bool stop = S.dec.stop != 0;
  while (!stop) {
    const double t = S.dec.nt, h = S.dec.nh;
    __syncthreads();
    stage_times(S, t, h);
    __syncthreads();
    for (int s = 1; s <= 12; ++s) {
      const double* w = s == 12 ? c_dop_b : c_dop_a + 16 * s;
      if (own) {
#pragma unroll
        for (int it = 0; it < NPT; ++it)
#pragma unroll (EARLY ? 4 : 2)
          for (int i = 0; i < 4; ++i) {
            const int nt = nt0 + it, r = el_r(i), col = el_c(nt, i), e = el_e(nt, i);
            double part = 0.0;
            if (active(r, col)) {
              double2 base;
              if constexpr (EARLY) base = kvec(s == 1 ? yslot : 18)[e];
              else base = entry_sum(w, s - 1, h, std::integral_constant<int, 11>(), e);
              const double2 v = zaxpy(h * w[s - 1], kvec(kslot(s - 1))[e], base);
              put_z(r, col, v);
              if (s == 12) kvec(pslot)[e] = v;
              if (c == 2) {
                const double2 sv = __ldg(st->S + (size_t)(bi * B + r) * DP + bj * B + col);
                part += (bi == bj && r == col ? 1.0 : 2.0) * (v.x * sv.x - v.y * sv.y);
              }
            }
            if (c == 2) {
              part = warp_sum(part);
              if (lane == 0) S.wk[s][nt * 4 + i] = part;
            }
          }
      }
      rhs(kslot(s), S.jac[s], S.src[s], [&] {
        if (s < 12) partial_sum(s == 11 ? c_dop_b : c_dop_a + 16 * (s + 1), s, h, std::integral_constant<int, 11>());
        else partial_errors();
      });
    }
    // ------------------------------------------------------------ error norms
    if (own) {
#pragma unroll
      for (int it = 0; it < NPT; ++it)
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
          const int nt = nt0 + it, r = el_r(i), col = el_c(nt, i), e = el_e(nt, i);
          double s5 = 0.0, s3 = 0.0;
          const double wt = active(r, col) ? norm_weight(packed, half, c, bi * B + r, bj * B + col) : 0.0;
          if (wt != 0.0) {
            const double2 k12 = kvec(kslot(12))[e];
            double2 e5, e3;
            if constexpr (EARLY) {
              e5 = kvec(18)[e];
              e3 = kvec(19)[e];
            } else {
              entry_errors(e, e5, e3);
            }
            e5 = zaxpy(c_dop_e5[12], k12, e5);
            e3 = zaxpy(c_dop_e3[12], k12, e3);
            const double2 yo = kvec(yslot)[e], yn = kvec(pslot)[e];
            const double scale = atol + rtol * fmax(hypot(yo.x, yo.y), hypot(yn.x, yn.y));
            s5 += wt * (zabs2(e5) / (scale * scale));
            s3 += wt * (zabs2(e3) / (scale * scale));
          }
          s5 = warp_sum(s5);
          s3 = warp_sum(s3);
          if (lane == 0) {
            s_we[c * W::PARTS + nt * 4 + i] = s5;
            s_we[(kChannels + c) * W::PARTS + nt * 4 + i] = s3;
          }
        }
    }
    __syncthreads();
    if (tid < kRec) {
      const double x = record_entry(S, tid, W::PARTS, 0, kChannels, h, ctl_in.max_ns && global_ns() - t_start >= ctl_in.max_ns,
                                    [&](int q, int ch, int i) { return s_we[(q * kChannels + ch) * W::PARTS + i]; });
      if constexpr (NR == 1) s_gat[tid] = x;
      else dsmem_store_f64(s_gat + rank * kRec + tid, 0, x);
    }
    team_sync();
    if (rank == 0 && warp == 0) {
      double tot = 0.0;
      if (lane < kRec)
        for (int g = 0; g < NR; ++g) tot += s_gat[kRec * g + lane];
      const long long next = S.ctl.next_point;
      const double pt = next + lane < npoints ? points[next + lane] : INFINITY;
      if (lane < kRec) S.tot[lane] = tot;
      __syncwarp();
      decide<NR>(S, st, ctl_in, points, npoints, pt, N, t, h);
    }
    team_sync();
    stop = S.dec.stop != 0;
    if (S.dec.accept) {
      if (S.dec.dense) {
        partial_sum(c_dop_a + 16 * 13, 12, h, std::integral_constant<int, 12>());
        for (int s = 13; s < 16; ++s) {
          if (own) {
#pragma unroll
            for (int it = 0; it < NPT; ++it)
#pragma unroll 1
              for (int i = 0; i < 4; ++i) {
                const int nt = nt0 + it, r = el_r(i), col = el_c(nt, i), e = el_e(nt, i);
                if (!active(r, col)) continue;
                double2 base;
                if constexpr (EARLY) base = kvec(18)[e];
                else base = entry_sum(c_dop_a + 16 * s, s - 1, h, std::integral_constant<int, 14>(), e);
                put_z(r, col, zaxpy(h * c_dop_a[16 * s + s - 1], kvec(kslot(s - 1))[e], base));
              }
          }
          rhs(s, S.jac[s], S.src[s], [&] {
            if (s < 15) partial_sum(c_dop_a + 16 * (s + 1), s, h, std::integral_constant<int, 14>());
          });
        }
        const double tn = S.dec.tn;
        const long long first = S.dec.first, last = S.dec.last;
        if (own) {
#pragma unroll
          for (int it = 0; it < NPT; ++it)
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
              const int nt = nt0 + it, r = el_r(i), col = el_c(nt, i), e = el_e(nt, i);
              if (!active(r, col)) continue;
              double2 kd[16];
#pragma unroll
              for (int j = 0; j < 16; ++j)
                kd[j] = ((rcmps_dop_dense_mask >> j) & 1u) ? kvec(kslot(j))[e] : make_double2(0.0, 0.0);
              const double2 yo = kvec(yslot)[e], yn = kvec(pslot)[e];
              double2 cf[7];
              dense_coefficients(kd, yo, yn, h, cf);
              double2* o1 = st->samples + (size_t)c * MAT + (size_t)(bi * B + r) * DP + bj * B + col;
              double2* o2 = st->samples + (size_t)c * MAT + (size_t)(bj * B + col) * DP + bi * B + r;
              for (long long node = first; node < last; ++node) {
                const double2 v = dense_value(cf, yo, yn, points[node], t, h, tn);
                o1[(size_t)node * VEC] = v;
                if (bi != bj || r != col) o2[(size_t)node * VEC] = zconj(v);
              }
            }
        }
      }
      int x = yslot;
      yslot = pslot;
      pslot = x;
      x = k0slot;
      k0slot = k12slot;
      k12slot = x;
    }
  }
  if (rank == 0 && tid == 0) write_stats(S, st, packed);
  if (NB > 1 && tid == 0 && S.wait_flag) {
    // a copy whose wait gave up may still be in flight: wait (bounded) for each channel's last one
    for (int q = 0; q < kChannels; ++q) mbar_wait(&s_full[q], (seq * (owns(q) ? 2u : 1u) - 1u) & 1u, nullptr);
  }
  team_sync();   // no CTA leaves while another may still write into its shared memory
}

// The structurally zero tiles of a packed Z2 state's samples (channel c at every node): the tile
// kernel never writes them.
__global__ void zero_samples_kernel(const TrajState* states, int dp, int npoints) {
  const TrajState* st = states + blockIdx.y;
  const int half = dp / 2;
  if (!st->herm || st->z2 <= 0 || st->d != dp) return;
  const size_t mat = (size_t)dp * dp;
  for (long long m = blockIdx.x; m < (long long)npoints * kChannels; m += gridDim.x) {
    const int c = (int)(m % kChannels);
    const bool odd = c % 2 == 0;
    double2* out = st->samples + (size_t)m * mat;
    for (int e = threadIdx.x; e < dp * dp; e += blockDim.x) {
      const bool cross = (e / dp < half) != (e % dp < half);
      if (cross != odd) out[e] = make_double2(0.0, 0.0);
    }
  }
}

// A launch of clusters of TG<DP>::NR CTAs.
template <int DP, class K>
static cudaError_t configure(K kern, int nclusters, int threads, size_t smem, bool cooperative, cudaStream_t stream,
                             cudaLaunchAttribute* attr, cudaLaunchConfig_t& cfg) {
  cfg = {};
  cfg.gridDim = dim3(nclusters * TG<DP>::NR, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = TG<DP>::NR;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cooperative ? 2 : 1;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

// Clusters of a kernel that the device holds at once (0: it cannot place one; -1: the query failed).
template <int DP, class K>
static int resident_clusters(K kern, int threads, size_t smem) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg;
  int n = 0;
  if (configure<DP>(kern, 1, threads, smem, false, nullptr, attr, cfg) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return n;
}

// The current device's capacity, a constant of device and kernel.
template <class F>
static int per_device(std::atomic<int> (&known)[64], F ask) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return std::max(0, ask());
  return capacity_once(known[dev], ask);
}
// States whose seven teams are resident at once, and those of the one-team kernel.
template <int DP>
static int lone_states() {
  static_assert(Smem<DP, true>::bytes() <= 232448, "shared memory per CTA");
  static std::atomic<int> known[64];
  return per_device(known, [] {
    const int n = resident_clusters<DP>(tile_kernel<DP, true>, Smem<DP, true>::THREADS, Smem<DP, true>::bytes());
    return n < 0 ? n : n / kChannels;
  });
}
template <int DP>
static int batch_states() {
  static std::atomic<int> known[64];
  return per_device(known, [] {
    if constexpr (TG<DP>::B == 16) {
      return resident_clusters<DP>(wide_kernel<DP>, Wide<DP>::NT, Wide<DP>::BYTES);
    } else {
      static_assert(Smem<DP, false>::bytes() <= 232448, "shared memory per CTA");
      return resident_clusters<DP>(tile_kernel<DP, false>, TG<DP>::NT, Smem<DP, false>::bytes());
    }
  });
}

// Seven teams per state, a few states per launch one launch after another, or one team per state, as
// many states at once as fit: the former while its rounds number at most 4 (DP <= 64) or 6 times the
// latter's. Measured per right-hand side, one round of either: D = 16 2.8 against 14 us, D = 32 4.5
// against 25, D = 48 5.3 against 21, D = 64 5.6 against 24, D = 96 20 against 130, D = 128 26 against 190.
template <int DP>
static int teams_for(int nstates) {
  const int lone = lone_states<DP>(), batch = batch_states<DP>();
  const long long rounds = lone ? (nstates + lone - 1) / lone : 0, waves = batch ? (nstates + batch - 1) / batch : 0;
  if (lone && (!batch || rounds <= (TG<DP>::B == 16 ? 4 : 6) * waves)) return kChannels;
  return batch ? 1 : 0;
}

template <int DP>
static int ctas_for(int nstates) {
  const int teams = teams_for<DP>(nstates);
  return TG<DP>::NR * teams * std::min(nstates, teams == kChannels ? lone_states<DP>() : batch_states<DP>());
}

template <int DP>
static cudaError_t launch(const TrajState* d_states, int nstates, const double* d_points, int npoints,
                          const TrajControls& ctl, void* sync, int teams, cudaStream_t stream) {
  using G = TG<DP>;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg;
  cudaError_t e;
  Sync* sy = static_cast<Sync*>(sync);
  if (teams == kChannels) {
    e = cudaMemsetAsync(sync, 0, (size_t)nstates * sizeof(Sync), stream);
    const int lone = lone_states<DP>();
    for (int s = 0; e == cudaSuccess && s < nstates; s += lone) {
      note_launch();
      e = configure<DP>(tile_kernel<DP, true>, std::min(lone, nstates - s) * kChannels, Smem<DP, true>::THREADS,
                        Smem<DP, true>::bytes(), true, stream, attr, cfg);
      if (e == cudaSuccess)
        e = cudaLaunchKernelEx(&cfg, tile_kernel<DP, true>, d_states + s, d_points, npoints, ctl, sy + s);
    }
    return e;
  }
  note_launch();
  if constexpr (G::B == 16) {
    e = configure<DP>(wide_kernel<DP>, nstates, Wide<DP>::NT, Wide<DP>::BYTES, false, stream, attr, cfg);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, wide_kernel<DP>, d_states, d_points, npoints, ctl);
  } else {
    e = configure<DP>(tile_kernel<DP, false>, nstates, G::NT, Smem<DP, false>::bytes(), false, stream, attr, cfg);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, tile_kernel<DP, false>, d_states, d_points, npoints, ctl, sy);
  }
}

}  // namespace tile

cudaError_t tile_trajectory_init() { return dop853_upload(); }

static int lone_states_for(int dp) {
  switch (dp) {
    case 16: return tile::lone_states<16>();
    case 32: return tile::lone_states<32>();
    case 48: return tile::lone_states<48>();
    case 64: return tile::lone_states<64>();
    case 96: return tile::lone_states<96>();
    case 128: return tile::lone_states<128>();
    default: return 0;
  }
}

static Admission& admission(int device) {
  static Admission all[64];
  return all[device & 63];
}
void TilePass::enter(int device, int dp, int nstates, cudaStream_t stream) {
  const int capacity = lone_states_for(dp);
  states_ = std::min(nstates, capacity);   // the rest follow in later rounds
  admission_ = &admission(device);
  stream_ = stream;
  admission_->enter(dp, states_, capacity);
}
void TilePass::leave(cudaEvent_t done) {
  if (!admission_) return;
  cudaEventSynchronize(done);
  admission_->leave(states_);
  admission_ = nullptr;
}
TilePass::~TilePass() {
  if (!admission_) return;
  cudaStreamSynchronize(stream_);
  admission_->leave(states_);
}
size_t tile_sync_bytes() { return sizeof(tile::Sync); }

int tile_trajectory_teams(int dp, int nstates) {
  switch (dp) {
    case 16: return tile::teams_for<16>(nstates);
    case 32: return tile::teams_for<32>(nstates);
    case 48: return tile::teams_for<48>(nstates);
    case 64: return tile::teams_for<64>(nstates);
    case 96: return tile::teams_for<96>(nstates);
    case 128: return tile::teams_for<128>(nstates);
    default: return 0;
  }
}

int tile_trajectory_ctas(int dp, int nstates) {
  switch (dp) {
    case 16: return tile::ctas_for<16>(nstates);
    case 32: return tile::ctas_for<32>(nstates);
    case 48: return tile::ctas_for<48>(nstates);
    case 64: return tile::ctas_for<64>(nstates);
    case 96: return tile::ctas_for<96>(nstates);
    case 128: return tile::ctas_for<128>(nstates);
    default: return 0;
  }
}

cudaError_t tile_trajectory_launch(int dp, const TrajState* d_states, int nstates, const double* d_points, int npoints,
                                   const TrajControls& ctl, void* sync, int teams, bool zero_samples,
                                   cudaStream_t stream) {
  if (zero_samples) {
    note_launch();
    tile::zero_samples_kernel<<<dim3(512, nstates), 256, 0, stream>>>(d_states, dp, npoints);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  switch (dp) {
    case 16: return tile::launch<16>(d_states, nstates, d_points, npoints, ctl, sync, teams, stream);
    case 32: return tile::launch<32>(d_states, nstates, d_points, npoints, ctl, sync, teams, stream);
    case 48: return tile::launch<48>(d_states, nstates, d_points, npoints, ctl, sync, teams, stream);
    case 64: return tile::launch<64>(d_states, nstates, d_points, npoints, ctl, sync, teams, stream);
    case 96: return tile::launch<96>(d_states, nstates, d_points, npoints, ctl, sync, teams, stream);
    case 128: return tile::launch<128>(d_states, nstates, d_points, npoints, ctl, sync, teams, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace rcmps
