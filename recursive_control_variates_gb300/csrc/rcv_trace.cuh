// Persistent tracer loop with deferred expensive events.
//
// Every warp pulls batches of path indices from one global counter and hands
// them to idle lanes.  A lane is always in one of these phases:
//   kStart    path (or adjoint replay pass) waiting to be initialised
//   kMain     walking the main path: up to kWalkSteps free-flight steps per
//             iteration
//   kScatter  real scattering event waiting to be processed (albedo lookups,
//             phase and NEE direction sampling, adjoint scatter)
//   kNee      walking the NEE shadow ray (ratio tracking)
//   kNeeAdj   adjoint replay only: walking the shadow ray again to scatter
//             its gradients
// Path starts and scattering events cost 100-200 instructions while a
// free-flight step costs a few dozen; executing them as soon as one lane
// needs them would leave the other 31 lanes waiting in almost every
// iteration.  Lanes that reach one park in kStart / kScatter and the warp runs
// that branch only when at least `defer` lanes wait (or when no lane can walk),
// so the expensive branches run with many lanes and the free-flight step
// stays converged.  The per-path random-number order is unchanged, so results
// do not depend on the schedule.
//
// Adjoint (path replay backpropagation, Vicini et al. 2021) in two launches.
// The gradient of an event is dL . L_rem times a factor of the event, where
// L_rem = L - (radiance gathered before the event) is only known once the
// path has ended.
//   kAdjoint  radiance pass: traces the path on `new`, stores its total
//             radiance L and, at every real scattering event, a 64-byte
//             checkpoint (random-number state, position, depth, throughput,
//             radiance so far, NEE contribution).
//   kReplay   a queue of replay tasks: the segment of every path from the
//             camera to its first scattering event, then one task per
//             checkpoint (that scattering event, its NEE shadow ray and the
//             segment to the next event).  Each task replays its segment with
//             the same random numbers and scatters the gradients; a task
//             stops at the next scattering event, which has its own task.
// A path whose checkpoints did not fit is replayed whole by its camera task.
//   kForward  the same replay tasks for forward-mode derivatives: at each
//             event where kReplay scatters dL . L_rem times a factor into the
//             grid gradient, it adds L_rem times the factor applied to the
//             tangent field to the task's image derivative, which goes to its
//             pixel at the end of the task.
// Replaying segments instead of whole paths keeps every task short, so the
// launch does not end on a few paths that scatter dozens of times.
//   kTape     the radiance pass without checkpoints: it records every
//             gradient event of the path (main-walk null collisions, real
//             scattering events, shadow-walk steps) on a tape, as its
//             position and a reference to the path or to the record of its
//             scattering event (radiance gathered before it, NEE
//             contribution).  The gradient is then one flat pass over the
//             tape (rcv_tape.cu), which recomputes each event's factor from
//             the medium; paths whose events did not fit are replayed whole
//             by kReplay over the lost list.
#pragma once
#include "rcv_volume.cuh"

namespace rcv {

enum PathPhase { kIdle = 0, kStart = 1, kMain = 2, kScatter = 3, kNee = 4, kNeeAdj = 5 };

// Replay task kinds.
enum TaskKind { kTaskSegment = 0, kTaskWhole = 1, kTaskCheckpoint = 2 };

// Checkpoint record (4 float4): [path, depth, rng.state lo, hi] [p, bn.x]
// [bn.y, bn.z, Lacc.x, Lacc.y] [Lacc.z, cn]; Lacc = radiance gathered before
// the event's NEE contribution cn.
__device__ __forceinline__ void write_checkpoint(float4* rec, uint32_t path, int depth, uint64_t state,
                                                 const V3& p, const V3& bn, const V3& lacc, const V3& cn) {
  rec[0] = make_float4(__uint_as_float(path), __int_as_float(depth), __uint_as_float((uint32_t)state),
                       __uint_as_float((uint32_t)(state >> 32)));
  rec[1] = make_float4(p.x, p.y, p.z, bn.x);
  rec[2] = make_float4(bn.y, bn.z, lacc.x, lacc.y);
  rec[3] = make_float4(lacc.z, cn.x, cn.y, cn.z);
}

// Job of a global path index: binary search in the launch's job table.
__device__ __forceinline__ const VolJob& job_of(const Queue& Q, int64_t path) {
  int lo = 0, hi = Q.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (Q.jobs[mid].path_begin <= path)
      lo = mid;
    else
      hi = mid - 1;
  }
  return Q.jobs[lo];
}

// Warps per tracer block (the cooperative walk keeps 3 x 32 floats per warp in
// shared memory).
constexpr int kTraceWarps = 4;
constexpr int kTraceBlock = 32 * kTraceWarps;

// Cooperative walk of a warp's last paths.
//
// Once the path queue is empty a warp runs until its longest path ends, and
// that path's free-flight steps form one chain of dependent lookups: at full
// size the last paths of a launch (up to 64 scattering events, each with a
// shadow walk) keep a few warps busy for 40 % of the launch time.  A run of
// null collisions of the main walk, or of ratio-tracking steps of the shadow
// walk, needs no result of one step to place the next except the position,
// and the random numbers of step k are at a known offset in the path's stream
// (3 draws per main step below the roulette depth: roulette, distance,
// real/null; 1 per shadow step).  So a group of G lanes evaluates the next G
// steps of one walking path at once: lane k jumps the stream to step k, takes
// its distance, and looks the densities up at its tentative point, assuming
// all earlier steps of the group were null (main) or did not end the shadow
// walk.  The first step that is something else (a real collision, leaving the
// segment, a zero throughput or transmittance) ends the run; the owner lane
// takes the steps before it, and the regular step code then executes that
// step itself.  Positions, remaining distances, null-collision weights and
// transmittances are accumulated in step order with the operations of the
// regular step, so a path gives the same bits whether it walks alone or with
// helpers.  `m` holds the walking lanes (at most 16: G = 32 / 16 / 8 / 4 / 2 for
// 1 / 2 / 3-4 / 5-8 / 9-16 paths; a limit of 4 / 8 / 16 gave 822 / 766 / 711 us
// for the paired launch of five 107 x 83 views, 202 / 181 / 180 us at 128^2); `org`, `dir`, `tmax` are the walk's ray and
// remaining distance, `c1`, `c2` its throughputs (main: bn, bo) or
// transmittances (shadow: trn, tro in .x); `s_t`, `s_w1`, `s_w2` are the
// warp's 32-float shared arrays for the steps' distances and weights.
// Returns the number of steps the calling lane's path took (0 for lanes that
// own no walking path).  kTape: every step taken is a gradient event, which
// the lane that evaluated it appends to the tape with the owner's reference
// `ref`; `lost` is set on an owner whose events did not fit.
template <int kMode, bool kTable>
__device__ __forceinline__ int coop_walk(unsigned m, bool main_walk, const VolJob& single, const VolJob* Jp,
                                         Pcg32& rng, float mu, float inv_mu, float half_inv_mu, V3& org,
                                         const V3& dir, float& tmax, V3& c1, V3& c2, float* s_t, float* s_w1,
                                         float* s_w2, const Queue& Q, TapeCursor& tc, uint32_t ref, bool& lost) {
  constexpr unsigned kFull = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const int n = __popc(m);
  const int G = coop_group(n);
  const int grp = (int)lane / G;
  const int k = (int)lane & (G - 1);
  const int base = grp * G;
  const bool busy = grp < n;
  // owner of this lane's group: the grp-th walking lane (lanes of idle groups
  // read their own registers and touch no memory)
  const int owner = coop_owner(m, grp, (int)lane);

  const bool g_main = __shfl_sync(kFull, (int)main_walk, owner) != 0;
  const VolJob& J = kTable ? *(const VolJob*)__shfl_sync(kFull, (unsigned long long)Jp, owner) : single;
  Pcg32 r;
  r.state = __shfl_sync(kFull, (unsigned long long)rng.state, owner);
  r.inc = __shfl_sync(kFull, (unsigned long long)rng.inc, owner);
  // (every path of a single job has its majorant)
  const float g_mu = kTable ? __shfl_sync(kFull, mu, owner) : mu;
  const float g_inv = kTable ? __shfl_sync(kFull, inv_mu, owner) : inv_mu;
  const float g_hinv = kTable ? __shfl_sync(kFull, half_inv_mu, owner) : half_inv_mu;
  // throughputs (transmittances in .x) before the group's first step
  V3 b1{__shfl_sync(kFull, c1.x, owner), 0.0f, 0.0f}, b2{0.0f, 0.0f, 0.0f};
  if (kMode == kTwoState) {
    b1.y = __shfl_sync(kFull, c1.y, owner);
    b1.z = __shfl_sync(kFull, c1.z, owner);
    b2 = V3{__shfl_sync(kFull, c2.x, owner), __shfl_sync(kFull, c2.y, owner), __shfl_sync(kFull, c2.z, owner)};
  }
  const V3 dv{__shfl_sync(kFull, dir.x, owner), __shfl_sync(kFull, dir.y, owner), __shfl_sync(kFull, dir.z, owner)};
  float px = __shfl_sync(kFull, org.x, owner), py = __shfl_sync(kFull, org.y, owner);
  float pz = __shfl_sync(kFull, org.z, owner), tr = __shfl_sync(kFull, tmax, owner);

  // this lane's step: its draws, distance and real/null variable
  const ulonglong2 jump = __ldg(reinterpret_cast<const ulonglong2*>(kCoopJumps.j) + (g_main ? 3 * k : k));
  r.state = jump.x * r.state + jump.y * r.inc;
  if (g_main) pcg_skip1(r);  // roulette draw, unused below the roulette depth
  const float t = free_flight(next1d(r), g_mu, g_inv);
  const float ur = g_main ? next1d(r) : 0.0f;
  s_t[lane] = t;
  __syncwarp();
  // position and remaining distance before this lane's step, in step order
#pragma unroll 4
  for (int j = 0; j < k; ++j) {
    const float tj = s_t[base + j];
    px = fmaf(tj, dv.x, px);
    py = fmaf(tj, dv.y, py);
    pz = fmaf(tj, dv.z, pz);
    tr = tr - tj;
  }
  const bool valid = busy && t <= tr;
  const V3 x{fmaf(t, dv.x, px), fmaf(t, dv.y, py), fmaf(t, dv.z, pz)};
  float st_o = 0.0f, st_n = 0.0f;
  if (valid) {
    const Lookup lk = locate(J, x);
    float rho_o = 0.0f, rho_n;
    if (kMode == kTwoState)
      density2(J, lk, rho_o, rho_n);
    else
      rho_n = density_new(J, lk);
    st_o = J.scale * rho_o;
    st_n = J.scale * rho_n;
  }
  bool term;
  float w1 = 1.0f, w2 = 1.0f;  // main: null-collision weights (two-state); shadow: transmittance factors
  if (g_main) {
    const float prob = kMode == kTwoState ? (st_n + st_o) * g_hinv : st_n * g_inv;
    term = !(valid && ur >= prob);
    if (kMode == kTwoState) {
      const float sn_o = g_mu - st_o, sn_n = g_mu - st_n;
      w1 = (2.0f * sn_n) / (sn_n + sn_o);
      w2 = 2.0f - w1;
    }
  } else {
    term = !valid;
    w1 = (g_mu - st_n) * g_inv;
    if (kMode == kTwoState) w2 = (g_mu - st_o) * g_inv;
  }
  s_w1[lane] = w1;
  if (kMode == kTwoState) s_w2[lane] = w2;
  __syncwarp();
  // throughputs before and after this lane's step, in step order (the owner
  // alone took them one after the other while the group waited); a step is
  // not taken when the regular one would end the path before it (throughput
  // zero) or the shadow walk with it (transmittance zero)
#pragma unroll 4
  for (int j = 0; j < k; ++j) {
    const float x1 = s_w1[base + j];
    b1.x *= x1;
    if (kMode == kTwoState) {
      const float x2 = s_w2[base + j];
      b1.y *= x1;
      b1.z *= x1;
      b2 = V3{b2.x * x2, b2.y * x2, b2.z * x2};
    }
  }
  if (kMode == kTwoState && g_main) term = term || !nonzero<kMode>(b1, b2);
  b1 = V3{b1.x * w1, b1.y * w1, b1.z * w1};
  if (kMode == kTwoState) b2 = V3{b2.x * w2, b2.y * w2, b2.z * w2};
  if (!g_main) term = term || (b1.x == 0.0f && (kMode != kTwoState || b2.x == 0.0f));
  const unsigned tb_all = __ballot_sync(kFull, term);

  // the owner takes the steps before the first one that is not
  const bool own = (m >> lane) & 1u;
  int f = 0, src = (int)lane;
  const int ob = __popc(m & ((1u << lane) - 1u)) * G;
  const unsigned gmask = G == 32 ? kFull : ((1u << G) - 1u);
  if (own) {
    const unsigned tb = (tb_all >> ob) & gmask;
    f = tb != 0u ? __ffs(tb) - 1 : G;
    if (f > 0) src = ob + f - 1;
  }
  // state after f steps: position, remaining distance and stream after step
  // f - 1 of the group's lane that took it
  const V3 xs{__shfl_sync(kFull, x.x, src), __shfl_sync(kFull, x.y, src), __shfl_sync(kFull, x.z, src)};
  const float ts = __shfl_sync(kFull, tr - t, src);
  const unsigned long long ss = __shfl_sync(kFull, (unsigned long long)r.state, src);
  b1.x = __shfl_sync(kFull, b1.x, src);
  if (kMode == kTwoState) {
    b1.y = __shfl_sync(kFull, b1.y, src);
    b1.z = __shfl_sync(kFull, b1.z, src);
    b2 = V3{__shfl_sync(kFull, b2.x, src), __shfl_sync(kFull, b2.y, src), __shfl_sync(kFull, b2.z, src)};
  }
  if (kMode == kTape) {
    // the group's steps before the first that ends the run are events
    const int fg = __shfl_sync(kFull, f, owner);
    const uint32_t rg = __shfl_sync(kFull, ref, owner);
    // sigma_n of each step (the cooperative walk runs on the global majorant)
    const bool ok = tape_append(Q, tc, busy && k < fg, x, rg, g_mu - st_n);
    const unsigned bad = __ballot_sync(kFull, !ok);
    if (own && ((bad >> ob) & gmask) != 0u) lost = true;
  }
  if (f == 0) return 0;
  org = xs;
  tmax = ts;
  rng.state = ss;
  c1.x = b1.x;
  if (kMode == kTwoState) {
    c2.x = b2.x;
    if (main_walk) {
      c1 = b1;
      c2 = b2;
    }
  }
  return f;
}

// dLoss/dL of one path of pixel `pix` (the pixel value is the mean of its
// samples), as the replay uses it.
__device__ __forceinline__ V3 pixel_dL(const VolJob& J, int pix) {
  const float* g = J.grad_img + (int64_t)pix * 3;
  const float fs = (float)J.spp;
  return V3{g[0] / fs, g[1] / fs, g[2] / fs};
}

// Environment map seen along the box direction d (made a unit world
// direction first): radiance, and the pdf of sampling that direction for NEE.
__device__ __forceinline__ V3 env_radiance_dir(const VolJob& J, const V3& d, float& pdf) {
  V3 wd{d.x * J.box.x, d.y * J.box.y, d.z * J.box.z};
  const float inv_len = 1.0f / sqrtf(fmaf(wd.z, wd.z, fmaf(wd.y, wd.y, wd.x * wd.x)));
  wd = V3{wd.x * inv_len, wd.y * inv_len, wd.z * inv_len};
  float u, v, st;
  env_uv(wd, u, v, st);
  pdf = env_pdf(J.env, u, v, st);
  return env_eval_uv(J.env, u, v);
}

// kSG: the launch may contain media with a majorant supergrid.  kCount: the
// launch accumulates the RCV_COUNTER_* event counts (off, the counters cost
// no registers).
// kEnv: the launch's job has an environment map (else the constant white
// environment; the two are separate kernels so that the constant one carries
// none of the map's code).  kTable: the paths belong to the jobs of Q.jobs.
// Without a table every field of the job is an operand in the kernel's
// parameter bank; behind a pointer that may lead to a table entry, the walk
// would load its grid size, scale, cell address and depth limits again in
// every step and hold the pointer in two registers (2 to 3 % of a step).
template <int kMode, bool kSG, bool kCount, bool kEnv, bool kTable>
__device__ void trace_persistent(const VolJob& single, const Queue& Q, Counts& cnt) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  const float mis = 0.5f;  // power heuristic between two equal 1/(4 pi) pdfs
  const float emit_weight = 1.0f / kInvFourPi;
  const unsigned defer = (unsigned)Q.defer;
  // replay tasks, scattering the image gradient (kReplay) or gathering a
  // tangent field (kForward)
  constexpr bool kRep = kMode == kReplay || kMode == kForward;
  // radiance passes of the adjoint (checkpoints or tape)
  constexpr bool kRad = kMode == kAdjoint || kMode == kTape;
  constexpr bool kCoop = kMode == kTwoState || kMode == kSingle || kRad;
  __shared__ float s_coop[kCoop ? kTraceWarps * 96 : 1];  // cooperative walk: distances, weights
  // Cold state of each lane, [word][thread] (no bank conflicts): what a walk
  // does not touch from one of its ends to the next waits here instead of in
  // registers.  A lane walks one ray at a time, so the registers hold one
  // position, direction and distance; during a shadow walk the vertex and the
  // next segment are cold.
  enum { cP = 0, cWo = 3, cT = 6, cLn = 7, cLo = 10, cSid = 13, cPix, cPath, cIter0, cScn, cSco, cBn, cBo, cPathHi, cCk, cEnv = cCk + 2,
         cWords = cEnv + 3 };
  constexpr int kColdWords = kEnv ? int(cWords) : (kMode == kAdjoint ? int(cEnv) : int(cCk));
  __shared__ float s_cold[kColdWords * kTraceBlock];
  float* const cold = s_cold + threadIdx.x;
  const auto F = [cold](int i) -> float& { return cold[i * kTraceBlock]; };
  const auto U = [cold](int i) -> uint32_t& { return reinterpret_cast<uint32_t*>(cold)[i * kTraceBlock]; };
  const auto get3 = [cold](int i) {
    return V3{cold[i * kTraceBlock], cold[(i + 1) * kTraceBlock], cold[(i + 2) * kTraceBlock]};
  };
  const auto put3 = [cold](int i, const V3& v) {
    cold[i * kTraceBlock] = v.x;
    cold[(i + 1) * kTraceBlock] = v.y;
    cold[(i + 2) * kTraceBlock] = v.z;
  };
  // next path of the warp's claimed batch (its paths left are in `left`)
  __shared__ unsigned long long s_next[kTraceWarps];
  unsigned long long* const next = s_next + (threadIdx.x >> 5);
  unsigned left = 0u;
  bool queue_empty = false;
  const VolJob* Jp = kTable ? Q.jobs : nullptr;
  int phase = kIdle;
  float mu = 0.0f, inv_mu = 0.0f;  // half of inv_mu is recomputed where needed (one register less)
  const auto job_majorant = [&](const VolJob& J) {
    const float mu_old = J.scale * bits_to_float(__ldg(J.maxbits + 0));
    const float mu_new = J.scale * bits_to_float(__ldg(J.maxbits + 1));
    mu = (kMode == kTwoState) ? fmaxf(mu_old, mu_new) : mu_new;
    inv_mu = 1.0f / mu;
  };
  if (!kTable) job_majorant(single);  // the same for every path
  V3 dL{0.0f, 0.0f, 0.0f};  // kForward: the task's image derivative
  // kReplay: dL . L_rem with dL = dLoss/dL of the pixel; it changes only with
  // L_rem, and dL itself is recomputed from the image gradient at the events
  // that need it per channel (fewer registers live through the walk)
  float s_main = 0.0f;

  // (defined from the start: left undefined, a state would carry from one
  // tracer of a paired launch into the next and cost registers there)
  Pcg32 rng{0ull, 0ull};
  // whole-path replay: state of the stream of the second shadow walk (its
  // increment is rng.inc)
  uint64_t nee_state = 0;
  // the walk: position, direction and distance left of the main path or of
  // its shadow ray; throughputs
  V3 x{0, 0, 0}, dir{0, 0, 0};
  float rem = 0.0f;
  V3 bo{1, 1, 1}, bn{1, 1, 1};
  int depth = 0;
  // transmittances of the shadow ray (the throughputs' .x is cold meanwhile)
  float& trn = bn.x;
  float& tro = bo.x;
  bool ck_lost = false;  // a checkpoint (kTape: an event or event record) of this path did not fit
  // kTape: reference of the path's next events (kind << 30 | entered path or
  // event record), and the warp's tape chunk
  uint32_t tref = 0;
  TapeCursor tc{0u, 0u};
  // replay: radiance the path gathers after its current point,
  // L_rem = L - (radiance gathered so far), kept instead of L and the sum so far
  V3 Lrem{0, 0, 0}, cn_task{0, 0, 0};
  uint32_t ck_slot = 0;  // replay checkpoint task: its record (the NEE contribution is re-read there)
  float s_nee = 0.0f;
  int task = kTaskSegment;
  bool own_event = false;  // checkpoint task: its scattering event is still to be processed
  // loop iterations: a path's length is n_iter - its cold start when it ends
  uint32_t n_iter = 0;

  while (true) {
    ++n_iter;
    // ------------------------------------------- hand new paths to idle lanes
    unsigned need = __ballot_sync(0xffffffffu, phase == kIdle);
    while (need != 0u && !queue_empty) {
      if (left == 0u) {
        if (lane == 0) {
          // replay: camera tasks [0, paths) (after a tape pass: the paths on
          // the lost list), then the checkpoints that were written
          const int64_t total = !kRep ? Q.total
                                      : (Q.lost_list != nullptr ? (int64_t)*Q.lost_count
                                                                : Q.total + min((int64_t)*Q.ckpt_count, Q.ckpt_cap));
          const int64_t b = (int64_t)atomicAdd(Q.counter, (unsigned long long)Q.batch);
          if (b < total) {
            *next = (unsigned long long)b;
            left = (unsigned)min((int64_t)Q.batch, total - b);
          }
        }
        left = __shfl_sync(0xffffffffu, left, 0);
        if (left == 0u) {
          queue_empty = true;
          break;
        }
      }
      __syncwarp();  // lane 0's last write of *next, seen by all (a shuffle or ballot orders no memory)
      const unsigned take = min((unsigned)__popc(need), left);
      const unsigned rank = (unsigned)__popc(need & lt_mask);
      if (((need >> lane) & 1u) && rank < take) {
        const uint64_t path = *next + rank;
        U(cPath) = (uint32_t)path;
        U(cPathHi) = (uint32_t)(path >> 32);
        phase = kStart;
      }
      __syncwarp();
      if (lane == 0) *next += take;
      left -= take;
      need = __ballot_sync(0xffffffffu, phase == kIdle);
    }
    const unsigned m_start = __ballot_sync(0xffffffffu, phase == kStart);
    const unsigned m_scat = __ballot_sync(0xffffffffu, phase == kScatter);
    // (`need` holds the idle lanes: every other lane walks)
    const unsigned m_walk = ~(need | m_start | m_scat);
    if (queue_empty && (m_start | m_scat | m_walk) == 0u) break;
    // Once the queue is empty no new lanes arrive to fill a deferred branch;
    // waiting would only make the warp's last paths take turns.
    const unsigned need_lanes = queue_empty ? 1u : defer;
    const bool run_start =
        (unsigned)__popc(m_start) >= need_lanes || (m_walk == 0u && m_scat == 0u && m_start != 0u);
    const bool run_scat = (unsigned)__popc(m_scat) >= need_lanes || (m_walk == 0u && m_scat != 0u);

    bool finished = false;  // the lane's current path (or task) ends this iteration
    // the shadow walk ends in this iteration (handled below, after the tape)
    bool nee_done = false;
    // kTape: the scattering event at the cold vertex processed in this iteration,
    // with its sigma_t
    float ev_sf = 0.0f;
    bool ev_scat = false;

    // ------------------------------------------------------------ path start
    if (run_start && phase == kStart) {
      U(cIter0) = n_iter;
      int64_t path = (int64_t)((uint64_t)U(cPath) | ((uint64_t)U(cPathHi) << 32));
      // replay: a checkpoint task resumes at its scattering event
      const bool resume = kRep && Q.lost_list == nullptr && path >= Q.total;
      float4 r0, r1, r2, r3;
      if (resume) {
        ck_slot = (uint32_t)(path - Q.total);
        const float4* rec = Q.ckpt + (path - Q.total) * 4;
        r0 = rec[0];
        r1 = rec[1];
        r2 = rec[2];
        r3 = rec[3];
        path = (int64_t)__float_as_uint(r0.x);
      } else if (kRep && Q.lost_list != nullptr) {
        path = (int64_t)Q.lost_list[path];  // a path the tape could not hold
      }
      U(cPath) = (uint32_t)path;
      if (kTable) Jp = &job_of(Q, path);
      const VolJob& J = kTable ? *Jp : single;
      if (kTable) job_majorant(J);
      // k-th pixel of the job's hand-out order, sample s of that pixel
      // 32-bit index arithmetic: a job has fewer than 2^32 paths
      const uint32_t local = (uint32_t)(path - J.path_begin);
      const uint32_t uspp = (uint32_t)J.spp;
      const uint32_t k = local / uspp;
      const uint32_t smp = local - k * uspp;
      const int pix = J.pixel_order != nullptr ? (int)__ldg(J.pixel_order + k) : (int)k;
      const uint32_t sid = (uint32_t)pix * (uint32_t)J.spp + smp;  // sample index within the job
      U(cPix) = (uint32_t)pix;
      U(cSid) = sid;
      seed_lane(rng, J.seed, sid);
      bo = V3{1, 1, 1};
      bn = V3{1, 1, 1};
      put3(cLn, V3{0, 0, 0});
      if (kMode == kTwoState) put3(cLo, V3{0, 0, 0});
      depth = 0;
      if (kRad) ck_lost = false;
      if (kMode == kTape) tref = kTapeEmpty;  // until the path enters the medium
      if (kRep) {
        if (kMode == kForward) dL = V3{0.0f, 0.0f, 0.0f};
        const float4 lt = Q.path_ltot[path];
        Lrem = V3{lt.x, lt.y, lt.z};
        task = resume ? kTaskCheckpoint : (lt.w != 0.0f ? kTaskWhole : kTaskSegment);
      }
      if (resume) {
        if (task != kTaskCheckpoint || Q.path_ltot[path].w != 0.0f) {
          finished = true;  // the path is replayed whole by its camera task
        } else {
          depth = __float_as_int(r0.y);
          rng.state = (uint64_t)__float_as_uint(r0.z) | ((uint64_t)__float_as_uint(r0.w) << 32);
          x = V3{r1.x, r1.y, r1.z};
          bn = V3{r1.w, r2.x, r2.y};
          const V3 Ln{r2.z, r2.w, r3.x};
          put3(cLn, Ln);
          Lrem = V3{Lrem.x - Ln.x, Lrem.y - Ln.y, Lrem.z - Ln.z};
          if (kMode == kForward) cn_task = V3{r3.y, r3.z, r3.w};
          F(cScn) = J.scale * density_new(J, locate(J, x));
          own_event = true;
          phase = kScatter;
        }
      } else {
        const float u0 = next1d(rng), u1 = next1d(rng);
        V3 o;
        const uint32_t py = (uint32_t)pix / (uint32_t)J.width;
        camera_ray(J, (int)((uint32_t)pix - py * (uint32_t)J.width), (int)py, u0, u1, o, dir);
        (void)next1d(rng);  // colour channel for free-flight sampling (grey extinction)
        if (!roulette<kMode>(J, rng, depth, bn, bo)) {
          finished = true;
        } else {
          const V3 inv_d = recip(dir);
          float tn, tf;
          slab(o, inv_d, tn, tf);
          if (!(tn <= tf && tf > 0.0f)) {
            // camera ray misses the cube: environment seen directly
            if (!J.hide_emitters) {
              if (kEnv) {
                float pdf;
                const V3 Le = env_radiance_dir(J, dir, pdf);
                put3(cLn, V3{bn.x * Le.x, bn.y * Le.y, bn.z * Le.z});
                if (kMode == kTwoState) put3(cLo, V3{bo.x * Le.x, bo.y * Le.y, bo.z * Le.z});
              } else {
                put3(cLn, bn);
                if (kMode == kTwoState) put3(cLo, bo);
              }
            }
            finished = true;
          } else {
            // null BSDF of the cube boundary: its 1D + 2D sample is drawn and discarded
            pcg_skip3(rng);
            x = advance(o, fmaxf(tn, 0.0f), dir);
            float a;
            slab(x, inv_d, a, rem);
            phase = kMain;
            if (kMode == kTape) {
              const uint32_t k = (uint32_t)atomicAdd(Q.entered_count, 1ull);
              __stcs(Q.entered + (kTable ? 2u * k : k), (uint32_t)path);
              tref = (kEvCamera << 30) | k;
            }
          }
        }
      }
    }

    if (kMode == kReplay && run_start && phase != kIdle && U(cIter0) == n_iter) {
      const V3 g = pixel_dL(kTable ? *Jp : single, (int)U(cPix));  // the task started in this iteration
      s_main = (g.x * Lrem.x + g.y * Lrem.y) + g.z * Lrem.z;
    }

    // ------------------------------------------------- real scattering event
    if (run_scat && phase == kScatter) {
      const VolJob& J = kTable ? *Jp : single;
      if (kRep && task == kTaskSegment) {
        finished = true;  // the event has its own checkpoint task
      } else if (kRep && task == kTaskCheckpoint && !own_event) {
        finished = true;
      } else {
        const Lookup lk = locate(J, x);
        const AlbedoLookup alk = albedo_lookup(J, lk, x);
        const float st_n = F(cScn), st_o = kMode == kTwoState ? F(cSco) : 0.0f;
        const V3 an = albedo_at(J, alk, 1);
        const V3 ss_n{st_n * an.x, st_n * an.y, st_n * an.z};
        if (kMode == kTwoState) {
          // plugins/twostatevolpath.py:259-260
          const V3 ao = albedo_at(J, alk, 0);
          const V3 ss_o{st_o * ao.x, st_o * ao.y, st_o * ao.z};
          // one division: 2 / (st_n + st_o) equals 1 / st_n exactly for equal
          // states, so those keep the single-state weights bit for bit
          const float k2 = 2.0f / (st_n + st_o);
          bn = V3{bn.x * (ss_n.x * k2), bn.y * (ss_n.y * k2), bn.z * (ss_n.z * k2)};
          bo = V3{bo.x * (ss_o.x * k2), bo.y * (ss_o.y * k2), bo.z * (ss_o.z * k2)};
        } else {
          if (kMode == kReplay) {
            // d log(sigma_s) / d density and d log(albedo) / d albedo at the event
            const V3 Lr = Lrem;
            const V3 g = pixel_dL(J, (int)U(cPix));
            const float sd = s_main;  // (g . Lr)
            scatter_density(J, lk, (J.scale * sd) / st_n);
            if (kCount) ++cnt.grad_events;
            if (J.grad_albedo != nullptr) {
              if (kCount) ++cnt.albedo_events;
              const V3 ga{(g.x * Lr.x) / fmaxf(an.x, 1e-8f), (g.y * Lr.y) / fmaxf(an.y, 1e-8f),
                          (g.z * Lr.z) / fmaxf(an.z, 1e-8f)};
              scatter_albedo(J, alk, ga);
            }
          } else if (kMode == kForward) {
            // the same terms applied to the tangent field: L_rem times
            // d log(sigma_s) along the tangent, per channel
            const V3 Lr = Lrem;
            const float f = (J.scale * tangent_density(J, lk)) / st_n;
            dL = V3{dL.x + Lr.x * f, dL.y + Lr.y * f, dL.z + Lr.z * f};
            if (kCount) ++cnt.grad_events;
            if (J.grad_albedo != nullptr) {
              if (kCount) ++cnt.albedo_events;
              const V3 ta = tangent_albedo(J, alk);
              dL = V3{dL.x + Lr.x * (ta.x / fmaxf(an.x, 1e-8f)), dL.y + Lr.y * (ta.y / fmaxf(an.y, 1e-8f)),
                      dL.z + Lr.z * (ta.z / fmaxf(an.z, 1e-8f))};
            }
          }
          // a checkpoint already holds the throughput after the event
          if (!(kRep && task == kTaskCheckpoint)) {
            const float k1 = 1.0f / st_n;
            bn = V3{bn.x * (ss_n.x * k1), bn.y * (ss_n.y * k1), bn.z * (ss_n.z * k1)};
          }
        }
        if (kMode == kAdjoint) {  // random-number state at the event, for its checkpoint
          U(cCk) = (uint32_t)rng.state;
          U(cCk + 1) = (uint32_t)(rng.state >> 32);
        }
        if (kMode == kTape && !ck_lost) {
          // the event's record, written when its shadow walk ends; the walk's
          // steps refer to it (a path without one is replayed instead)
          const unsigned long long k = atomicAdd(Q.ckpt_count, 1ull);
          if ((int64_t)k < Q.ckpt_cap) {
            tref = (kEvShadow << 30) | (uint32_t)k;
            ev_scat = true;  // the event itself
            ev_sf = st_n;
          } else {
            ck_lost = true;  // its events are not recorded any more
          }
        }
        // isotropic phase sample (1D unused + 2D), plugins/twostatevolpath.py:275
        pcg_skip1(rng);
        const float pu0 = next1d(rng), pu1 = next1d(rng);
        put3(cP, x);
        {
          // the next segment, needed when the NEE walk ends; its exit
          // distance is computed here, where many lanes run together
          const V3 wo = to_box(J, uniform_sphere(pu0, pu1));
          float a, t_next;
          slab(x, recip(wo), a, t_next);
          put3(cWo, wo);
          F(cT) = t_next;
        }
        // NEE towards the environment, then ratio tracking
        const float nu0 = next1d(rng), nu1 = next1d(rng);
        if (kEnv) {
          // NEE towards the environment map (plugins/twostatevolpath.py:315-344):
          // importance-sampled direction, power-heuristic weight against the
          // phase function's pdf
          V3 Le;
          float pdf;
          dir = to_box(J, env_sample(J.env, nu0, nu1, Le, pdf));
          float k = 0.0f;
          if (pdf > 0.0f && pdf < kInf) k = (kInvFourPi * env_mis(pdf, kInvFourPi)) / pdf;
          // NEE weight of the pending shadow ray (Le / pdf * phase * MIS)
          put3(cEnv, V3{Le.x * k, Le.y * k, Le.z * k});
        } else {
          dir = to_box(J, uniform_sphere(nu0, nu1));
        }
        {
          float a;
          slab(x, recip(dir), a, rem);
        }
        F(cBn) = bn.x;
        trn = 1.0f;
        if (kMode == kTwoState) {
          F(cBo) = bo.x;
          tro = 1.0f;
        }
        phase = kNee;
        if (kRep) {
          if (task == kTaskCheckpoint) {
            // NEE contribution known from the radiance pass: one shadow walk
            // on the main stream scatters its gradient (gathers the tangent)
            V3 cn = cn_task;
            if (kMode == kReplay) {
              const float4 r3 = Q.ckpt[(int64_t)ck_slot * 4 + 3];
              cn = V3{r3.y, r3.z, r3.w};
            }
            Lrem = V3{Lrem.x - cn.x, Lrem.y - cn.y, Lrem.z - cn.z};
            if (kMode == kReplay) {
              const V3 g = pixel_dL(J, (int)U(cPix));
              s_nee = (g.x * cn.x + g.y * cn.y) + g.z * cn.z;
              s_main = (g.x * Lrem.x + g.y * Lrem.y) + g.z * Lrem.z;
            }
            own_event = false;
            phase = kNeeAdj;
          } else {
            nee_state = rng.state;  // whole-path replay: walk for the transmittance, then again
          }
        }
      }
    }

    // ------------------------- cooperative walk of the last paths (see above)
    bool many = false;  // too many lanes walk for it
    if (kCoop && queue_empty) {
      const VolJob& J = kTable ? *Jp : single;
      bool elig = false;
      if (!finished) {
        if (phase == kNee) {
          elig = true;
        } else if (phase == kMain) {
          bool alive = bn.x != 0.0f || bn.y != 0.0f || bn.z != 0.0f;
          if (kMode == kTwoState) alive = alive || (bo.x != 0.0f || bo.y != 0.0f || bo.z != 0.0f);
          elig = alive && depth <= J.rr_depth;
        }
        if (kSG && elig && J.sg[0] > 0) elig = false;
      }
      const unsigned m_coop = __ballot_sync(0xffffffffu, elig);
      const int n_coop = __popc(m_coop);
      many = n_coop > kCoopMost;
      if (n_coop >= 1 && n_coop <= kCoopMost) {
        const bool mw = phase == kMain;
        float* s = s_coop + (threadIdx.x >> 5) * 96;
        const int f = coop_walk<kMode, kTable>(m_coop, mw, single, Jp, rng, mu, inv_mu, 0.5f * inv_mu, x, dir, rem, bn,
                                               bo, s, s + 32, s + 64, Q, tc, tref, ck_lost);
        if (f > 0) {
          if (kCount) {
            if (mw)
              cnt.lookups += (unsigned)f;
            else
              cnt.nee_lookups += (unsigned)f;
          }
          U(cIter0) -= (uint32_t)f;  // the path's cost counts its steps
        }
      }
    }

    // --------------------------------------------------- free-flight step
    const int steps = kRep || kSG || (queue_empty && !many) ? 1 : kWalkSteps;
#pragma unroll 1
    for (int sub = 1;; ++sub) {
      // kTape: this step's event, appended where the warp has reconverged (null
      // collision or shadow-walk step at x), with its reference and sigma_n
      bool ev_walk = false;
      uint32_t ev_ref = 0;
      float ev_f = 0.0f;
      if (!finished && !nee_done && (phase == kMain || phase == kNee || phase == kNeeAdj)) {
        const VolJob& J = kTable ? *Jp : single;
        // whole-path replay: the second shadow walk draws from the saved stream
        // (chosen by value, not through a pointer, which would put both
        // streams in local memory)
        const bool nee_stream = kRep && phase == kNeeAdj && task == kTaskWhole;
        if (phase == kMain && !roulette<kMode>(J, rng, depth, bn, bo)) {
          finished = true;
        } else {
          // majorant of this collision: global, or the supergrid cell it lies in
          float mu_c = mu, inv_c = inv_mu, hinv_c = 0.5f * inv_mu;
          float t;
          if (kSG && J.sg[0] > 0) {
            const float tau = -log_unit(1.0f - (nee_stream ? next1d_state(nee_state, rng.inc) : next1d(rng)));
            t = supergrid_flight(J, kMode == kTwoState ? J.sg_two : J.sg_new, x, dir, rem, tau, mu_c);
            inv_c = 1.0f / mu_c;
            hinv_c = 0.5f * inv_c;
          } else {
            t = free_flight(nee_stream ? next1d_state(nee_state, rng.inc) : next1d(rng), mu, inv_mu);
          }
          const bool valid = t <= rem;
          Lookup lk;
          float rho_o = 0.0f, rho_n = 0.0f;
          if (valid) {
            x = advance(x, t, dir);  // the step's end, whatever happens there
            lk = locate(J, x);
            if (kMode == kTwoState)
              density2(J, lk, rho_o, rho_n);
            else
              rho_n = density_new(J, lk);
            if (kCount) {
              if (phase == kMain)
                ++cnt.lookups;
              else
                ++cnt.nee_lookups;
            }
          }
          const float st_o = J.scale * rho_o, st_n = J.scale * rho_n;

          bool walk_done = false;  // the shadow walk ends
          if (valid) {
            // factors of the step if it is not a scattering event: ratio
            // tracking of a shadow ray (plugins/twostatevolpath.py:443-452), or
            // the weights of a null collision (:227-231, 256-257; they sum to 2,
            // equal states give exactly 1)
            const float sn_n = mu_c - st_n;
            float fn = sn_n * inv_c, fo = kMode == kTwoState ? (mu_c - st_o) * inv_c : 1.0f;
            bool null = true;
            if (phase == kMain) {
              const float ur = next1d(rng);
              // real-collision probability: mean of both states' sigma_t / mu
              // (plugins/twostatevolpath.py:222-225); equal states give exactly
              // the single-state sigma_t / mu
              float prob;
              if (kMode == kTwoState)
                prob = (st_n + st_o) * hinv_c;
              else
                prob = st_n * inv_c;
              null = ur >= prob;
              fn = 1.0f;
              if (kMode == kTwoState) {
                const float den = sn_n + (mu_c - st_o);
                fn = (2.0f * sn_n) / den;
                fo = 2.0f - fn;
              }
            }
            if (null) {
              bn.x *= fn;  // (of a shadow ray: its transmittance)
              if (kMode == kTwoState) {
                bo.x *= fo;
                const float gn = phase == kMain ? fn : 1.0f, go = phase == kMain ? fo : 1.0f;
                bn.y *= gn;
                bn.z *= gn;
                bo.y *= go;
                bo.z *= go;
              }
              if (kRep && phase != kNee && (phase == kMain || sn_n > 0.0f)) {
                if (kMode == kForward) {
                  const V3 Lr = phase == kMain ? Lrem : cn_task;
                  const float f = -(J.scale * tangent_density(J, lk)) / sn_n;
                  dL = V3{dL.x + Lr.x * f, dL.y + Lr.y * f, dL.z + Lr.z * f};
                } else {
                  scatter_density(J, lk, -(J.scale * (phase == kMain ? s_main : s_nee)) / sn_n);
                }
                if (kCount) ++cnt.grad_events;
              }
              rem = rem - t;
              if (kMode == kTape) {
                ev_walk = true;
                ev_ref = tref;
                ev_f = sn_n;
              }
              walk_done = phase != kMain && ((kMode == kTwoState) ? (trn == 0.0f && tro == 0.0f) : (trn == 0.0f));
            } else {
              // real scattering event (plugins/twostatevolpath.py:249-253)
              depth += 1;
              if (depth >= J.max_depth) {
                finished = true;
              } else {
                if (kCount) ++cnt.scatters;
                F(cScn) = st_n;
                if (kMode == kTwoState) F(cSco) = st_o;
                phase = kScatter;
              }
            }
          } else if (phase == kMain) {
            // leaves the cube: null BSDF sample, outside iteration RR, environment
            pcg_skip3(rng);
            if (roulette<kMode>(J, rng, depth, bn, bo) && !(J.hide_emitters && depth == 0)) {
              V3 Ln = get3(cLn), Lo{0, 0, 0};
              if (kMode == kTwoState) Lo = get3(cLo);
              if (kEnv) {
                // environment map hit after a phase sample: power heuristic
                // against NEE (plugins/twostatevolpath.py:288-308)
                float pdf;
                const V3 Le = env_radiance_dir(J, dir, pdf);
                const float k = depth == 0 ? 1.0f : env_mis(kInvFourPi, pdf);
                Ln = V3{Ln.x + (bn.x * Le.x) * k, Ln.y + (bn.y * Le.y) * k, Ln.z + (bn.z * Le.z) * k};
                if (kMode == kTwoState)
                  Lo = V3{Lo.x + (bo.x * Le.x) * k, Lo.y + (bo.y * Le.y) * k, Lo.z + (bo.z * Le.z) * k};
              } else {
                const float k = depth == 0 ? 1.0f : mis;
                Ln = V3{Ln.x + bn.x * k, Ln.y + bn.y * k, Ln.z + bn.z * k};
                if (kMode == kTwoState) Lo = V3{Lo.x + bo.x * k, Lo.y + bo.y * k, Lo.z + bo.z * k};
              }
              put3(cLn, Ln);
              if (kMode == kTwoState) put3(cLo, Lo);
            }
            finished = true;
          } else {
            walk_done = true;
          }
          if (!kRep || phase == kNee) {
            nee_done = walk_done;
          } else if (walk_done) {
            // kNeeAdj: the shadow walk with gradients ends
            bn.x = F(cBn);
            x = get3(cP);
            dir = get3(cWo);
            rem = F(cT);
            phase = kMain;
          }
        }
      }
      if (kMode == kTape && !tape_append(Q, tc, ev_walk && !ck_lost, x, ev_ref, ev_f)) ck_lost = true;
      if (sub >= steps) break;
      ++n_iter;  // (a path's cost counts its steps, and those of its last round)
    }

    if (kMode == kTape && run_scat) {
      if (!tape_append(Q, tc, ev_scat && !ck_lost, get3(cP), (kEvScatter << 30) | (tref & kTapeIndexMask), ev_sf))
        ck_lost = true;
    }

    // -------------------------------------------------- end of the shadow walk
    if (nee_done) {
      const VolJob& J = kTable ? *Jp : single;
      const V3 p = get3(cP);
      const float tn = trn, to = tro;
      bn.x = F(cBn);
      if (kMode == kTwoState) bo.x = F(cBo);
      V3 Ln = get3(cLn);
      V3 cn;
      if (kEnv) {
        const V3 e = get3(cEnv);
        cn = V3{(bn.x * e.x) * tn, (bn.y * e.y) * tn, (bn.z * e.z) * tn};
      } else {
        const float en = emit_weight * tn;
        cn = V3{((bn.x * kInvFourPi) * mis) * en, ((bn.y * kInvFourPi) * mis) * en,
                ((bn.z * kInvFourPi) * mis) * en};
      }
      if (kMode == kAdjoint && !ck_lost) {
        const unsigned long long slot = atomicAdd(Q.ckpt_count, 1ull);
        if ((int64_t)slot < Q.ckpt_cap)
          write_checkpoint(Q.ckpt + slot * 4, U(cPath), depth, (uint64_t)U(cCk) | ((uint64_t)U(cCk + 1) << 32), p, bn,
                           Ln, cn);
        else
          ck_lost = true;
      }
      if (kMode == kTape && (tref >> 30) == kEvShadow) {
        // the scattering event's record: its path, the radiance gathered
        // before its NEE contribution, and that contribution; the event
        // itself goes on the tape, and the next segment's null
        // collisions refer to the record too
        const uint32_t k = tref & kTapeIndexMask;
        float4* rec = Q.ckpt + (int64_t)k * 2;
        __stcs(rec, make_float4(__uint_as_float(U(cPath)), Ln.x, Ln.y, Ln.z));
        __stcs(rec + 1, make_float4(cn.x, cn.y, cn.z, 0.0f));
        tref = (kEvSegment << 30) | k;
      }
      Ln = V3{Ln.x + cn.x, Ln.y + cn.y, Ln.z + cn.z};
      put3(cLn, Ln);
      if (kRep) Lrem = V3{Lrem.x - cn.x, Lrem.y - cn.y, Lrem.z - cn.z};
      if (kMode == kTwoState) {
        V3 Lo = get3(cLo);
        if (kEnv) {
          const V3 e = get3(cEnv);
          Lo = V3{Lo.x + (bo.x * e.x) * to, Lo.y + (bo.y * e.y) * to, Lo.z + (bo.z * e.z) * to};
        } else {
          const float eo = emit_weight * to;
          Lo = V3{Lo.x + ((bo.x * kInvFourPi) * mis) * eo, Lo.y + ((bo.y * kInvFourPi) * mis) * eo,
                  Lo.z + ((bo.z * kInvFourPi) * mis) * eo};
        }
        put3(cLo, Lo);
      }
      x = p;
      if (kRep) {
        // whole-path replay: walk the shadow ray again (saved stream) to
        // back-propagate through its transmittance
        if (kMode == kReplay) {
          const V3 g = pixel_dL(J, (int)U(cPix));
          s_nee = (g.x * cn.x + g.y * cn.y) + g.z * cn.z;
          s_main = (g.x * Lrem.x + g.y * Lrem.y) + g.z * Lrem.z;
        } else {
          cn_task = cn;
        }
        float a;
        slab(x, recip(dir), a, rem);
        trn = 1.0f;  // bn.x is still cold
        phase = kNeeAdj;
      } else {
        dir = get3(cWo);
        rem = F(cT);
        phase = kMain;
      }
    }

    // -------------------------------------------------------------- path end
    if (finished) {
      const VolJob& J = kTable ? *Jp : single;
      if (kMode == kTwoState || kMode == kSingle) {
        float4* o = Q.path_out + (J.path_begin + U(cSid)) * (kMode == kTwoState ? 2 : 1);
        __stcs(o, make_float4(F(cLn), F(cLn + 1), F(cLn + 2), 0.0f));
        if (kMode == kTwoState) __stcs(o + 1, make_float4(F(cLo), F(cLo + 1), F(cLo + 2), 0.0f));
      }
      // (no event refers to a path that did not enter the medium)
      if (kRad && (kMode != kTape || tref != kTapeEmpty))
        __stcs(Q.path_ltot + U(cPath), make_float4(F(cLn), F(cLn + 1), F(cLn + 2), ck_lost ? 1.0f : 0.0f));
      if (kMode == kTape && ck_lost) Q.lost_list[atomicAdd(Q.lost_count, 1ull)] = U(cPath);
      if (kMode == kForward && (dL.x != 0.0f || dL.y != 0.0f || dL.z != 0.0f)) {
        // the task's share of its pixel's derivative (the pixel value is the
        // mean of its samples)
        const float fs = (float)J.spp;
        float* o = J.out_img + (int64_t)U(cPix) * 3;
        atomicAdd(o + 0, dL.x / fs);
        atomicAdd(o + 1, dL.y / fs);
        atomicAdd(o + 2, dL.z / fs);
      }
      if (kCount && !kRep) ++cnt.paths;
      if (J.pixel_cost != nullptr) red_add_u32(J.pixel_cost + U(cPix), n_iter - U(cIter0));
      phase = kIdle;
    }
  }
  if (kMode == kTape) tape_close(Q, tc);  // the unused slots of the warp's last chunk
}

}  // namespace rcv
