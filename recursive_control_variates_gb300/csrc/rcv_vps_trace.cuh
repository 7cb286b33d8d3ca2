// Persistent tracers of the volpathsimple adjoint (rcv_vps.cu).
//
// One thread per path (Vps::backward_path) leaves most lanes of a warp
// waiting: every lane is at another point of three nested loops (free flight
// inside a segment, segments of a path, the paths traced twice and a third
// one for differential ratio tracking).  At 512^2, 16 spp, depth 64 that
// launch took 13.1 ms at a few lanes per instruction.  Here the adjoint is
// two persistent launches with a few free-flight steps per loop iteration for
// every lane, whatever its phase (as in rcv_trace.cuh), and two flat passes;
// on the same film 0.82 + 0.70 + 0.21 + 0.08 ms (GB300, launches one at a
// time).  The tracers are
// bound by the issue of divergent instructions and end on their longest
// paths (a DRT path that follows its first path in the same lane and launch
// gave 2.0 ms for the two tracers where two launches took 1.74), the flat
// passes by the vector reductions into the gradient:
//   kVpsTape  traces each path once.  It records every segment (64 bytes:
//             the path, the NEE radiance gathered before it, its ray, its
//             length, the NEE contribution at its end) and every step of a
//             shadow walk (16 + 4 bytes on the warp's tape), keeps the
//             reservoir of differential ratio tracking, and writes the
//             path's radiance and, if its reservoir holds a segment, a task.
//   kVpsDrt   one path per task: the truncated-exponential distance on the
//             kept segment, its transmittance, and the radiance scattered in
//             at that point.
//   the flat passes (rcv_vps.cu) turn records, tasks and tape into the
//   gradient, now that each path's radiance is known.
// The radiance that remains at a segment is L - (NEE radiance before it), as
// in the tape of rcv_trace.cuh; the replay subtracts the contributions one by
// one (the difference is the rounding of that sum).  Every path takes the
// random numbers, positions and decisions of backward_path bit for bit: the
// second stream draws a fixed number per segment (one for the reservoir, four
// for the transmittance samples), so its state at any segment is a jump away.
#pragma once
#include "rcv_volume.cuh"

namespace rcv {

enum VpsMode { kVpsTape = 0, kVpsDrt = 1 };

constexpr int kVpsWarps = 4;
constexpr int kVpsBlock = 32 * kVpsWarps;
// Segment record (4 float4): [path, Lacc] [o, interval] [d, k << 1 | escaped]
// [NEE contribution at its end, 0].
constexpr int kVpsRec = 4;
// Task (3 float4): [path, record, depth, segments of the path] [reservoir
// weight, -] [-]; the tracer leaves [path, Li] [reservoir weight, distance
// weight] [x, 0].
constexpr int kVpsTask = 3;

struct VpsParams {
  int32_t use_nee, use_drt, use_drt_subsampling, use_drt_mis;
  uint32_t alt_seed;   // seed of the adjoint's second stream
  int32_t draws;       // second-stream draws per segment
  float4* path_out;    // primal: per-path radiance
  float4* task;        // kVpsDrt tasks
  unsigned long long* task_count;
  const uint32_t* lost_list;  // vps_kernel: only these streams (pixel * spp + sample), or null for all
  const unsigned long long* lost_count;
};

__device__ __forceinline__ uint64_t pack64(uint32_t lo, uint32_t hi) { return (uint64_t)lo | ((uint64_t)hi << 32); }

// Pixel of a path in the launch's hand-out order, and its random stream.
__device__ __forceinline__ uint32_t vps_sid(const VolJob& J, uint32_t path, int& pix) {
  const uint32_t local = path - (uint32_t)J.path_begin;
  const uint32_t k = local / (uint32_t)J.spp;
  pix = J.pixel_order != nullptr ? (int)__ldg(J.pixel_order + k) : (int)k;
  return (uint32_t)pix * (uint32_t)J.spp + (local - k * (uint32_t)J.spp);
}

// Cooperative walk of a warp's last paths (see coop_walk in rcv_trace.cuh):
// groups of lanes take the next steps of one path each, with this tracer's two
// draws per main step, its quotients and its walked distance `acc` (of a shadow
// walk: its transmittance).
template <int kMode>
__device__ __forceinline__ void vps_coop(unsigned m, bool main_walk, const VolJob& J, Pcg32& rng, float mu,
                                         float inv_mu, V3& org, const V3& dir, float& tmax, float& acc, float* s_t,
                                         float* s_w, const Queue& Q, TapeCursor& tc, uint32_t rec, bool& lost) {
  constexpr unsigned kFull = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const int n = __popc(m), G = coop_group(n);
  const int grp = (int)lane / G, k = (int)lane & (G - 1), base = grp * G;
  const bool busy = grp < n;
  const int owner = coop_owner(m, grp, (int)lane);
  const bool g_main = __shfl_sync(kFull, (int)main_walk, owner) != 0;
  Pcg32 r;
  r.state = __shfl_sync(kFull, (unsigned long long)rng.state, owner);
  r.inc = __shfl_sync(kFull, (unsigned long long)rng.inc, owner);
  const V3 dv{__shfl_sync(kFull, dir.x, owner), __shfl_sync(kFull, dir.y, owner), __shfl_sync(kFull, dir.z, owner)};
  float px = __shfl_sync(kFull, org.x, owner), py = __shfl_sync(kFull, org.y, owner);
  float pz = __shfl_sync(kFull, org.z, owner), tr = __shfl_sync(kFull, tmax, owner);
  float a = __shfl_sync(kFull, acc, owner);

  const ulonglong2 jump = __ldg(reinterpret_cast<const ulonglong2*>(kCoopJumps.j) + (g_main ? 2 * k : k));
  r.state = jump.x * r.state + jump.y * r.inc;
  const float t = free_flight(next1d(r), mu, inv_mu);
  const float ur = g_main ? next1d(r) : 0.0f;
  s_t[lane] = t;
  __syncwarp();
#pragma unroll 4
  for (int j = 0; j < k; ++j) {
    const float tj = s_t[base + j];
    px = fmaf(tj, dv.x, px);
    py = fmaf(tj, dv.y, py);
    pz = fmaf(tj, dv.z, pz);
    tr = tr - tj;
    if (g_main) a = a + tj;
  }
  const bool valid = busy && t <= tr;
  const V3 x{fmaf(t, dv.x, px), fmaf(t, dv.y, py), fmaf(t, dv.z, pz)};
  const float st = valid ? J.scale * density_new(J, locate(J, x)) : 0.0f;
  const float sn = mu - st;
  bool term = !valid;
  float w = 1.0f;
  if (g_main)
    term = term || ur < (mu != 0.0f ? div_by(st, mu, inv_mu) : 0.0f);
  else
    w = mu != 0.0f ? div_by(sn, mu, inv_mu) : sn;
  s_w[lane] = w;
  __syncwarp();
  if (!g_main) {
#pragma unroll 4
    for (int j = 0; j < k; ++j) a *= s_w[base + j];
  }
  a = g_main ? a + t : a * w;
  term = term || (!g_main && a == 0.0f);
  const unsigned tb_all = __ballot_sync(kFull, term);

  const bool own = (m >> lane) & 1u;
  const int ob = __popc(m & ((1u << lane) - 1u)) * G;
  const unsigned gmask = G == 32 ? kFull : ((1u << G) - 1u);
  int f = 0, src = (int)lane;
  if (own) {
    const unsigned tb = (tb_all >> ob) & gmask;
    f = tb != 0u ? __ffs(tb) - 1 : G;
    if (f > 0) src = ob + f - 1;
  }
  const V3 xs{__shfl_sync(kFull, x.x, src), __shfl_sync(kFull, x.y, src), __shfl_sync(kFull, x.z, src)};
  const float ts = __shfl_sync(kFull, tr - t, src), as = __shfl_sync(kFull, a, src);
  const unsigned long long ss = __shfl_sync(kFull, (unsigned long long)r.state, src);
  if (kMode == kVpsTape) {
    const int fg = __shfl_sync(kFull, f, owner);
    const uint32_t rg = __shfl_sync(kFull, rec, owner);
    const bool kept = __shfl_sync(kFull, (int)lost, owner) == 0;
    const bool ok = tape_append(Q, tc, busy && kept && k < fg && !g_main && w > 0.0f, x, rg, sn);
    const unsigned bad = __ballot_sync(kFull, !ok);
    if (own && ((bad >> ob) & gmask) != 0u) lost = true;
  }
  if (f == 0) return;
  org = xs;
  tmax = ts;
  acc = as;
  rng.state = ss;
}

template <int kMode, bool kSG, bool kEnv>
__device__ void trace_vps(const VolJob& J, const VpsParams& P, const Queue& Q) {
  constexpr bool kDrt = kMode == kVpsDrt;
  enum { kVIdle = 0, kVStart, kVMain, kVNee, kVVertex, kVEscape, kVDir };
  // per-lane values that only the segment ends need, out of the registers
  // that the walk keeps: [word][thread]
  constexpr int kCold = (kDrt ? 5 : 13) + (kEnv ? 3 : 0);
  __shared__ float s_cold[kCold * kVpsBlock];
  float* cold = s_cold + threadIdx.x;
  const auto F = [cold](int i) -> float& { return cold[i * kVpsBlock]; };
  const auto U = [cold](int i) -> uint32_t& { return reinterpret_cast<uint32_t*>(cold)[i * kVpsBlock]; };
  // kVpsTape: second stream (state, increment), reservoir sum, kept weight, kept record, kept depth
  constexpr int cAlt = 0, cSum = 4, cCur = 7, cKeep = 10, cKeepDepth = 11, cMax = 12;
  // kVpsDrt: task, NEE at the resampled point, its distance
  constexpr int cTask = 0, cNee = 1, cDist = 4;
  constexpr int cEnv = kDrt ? 5 : 13;

  __shared__ float s_coop[kSG ? 1 : kVpsWarps * 64];
  const unsigned lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
  const unsigned defer = (unsigned)Q.defer;
  const float mu = J.scale * bits_to_float(__ldg(J.maxbits + 1)), inv_mu = 1.0f / mu;

  __shared__ unsigned s_next[kVpsWarps];  // next path of the warp's claimed batch
  unsigned* const next = s_next + (threadIdx.x >> 5);
  unsigned left = 0u;  // paths left in it
  bool queue_empty = false;
  uint32_t path = 0;
  int phase = kVIdle, depth = 0;
  int stage = 0;  // kVpsDrt: 0 distance on the kept segment, 1 NEE there, 2 the path from there
  Pcg32 rng{0ull, 0ull};
  V3 xo{0, 0, 0}, sd{0, 0, 0}, p{0, 0, 0}, w{0, 0, 0};          // segment origin and direction; walk position and direction
  float rem = 0.0f, acc = 0.0f;  // distance left; distance walked (segment) or transmittance (shadow)
  V3 thr{1, 1, 1}, L{0, 0, 0};
  bool lost = false;
  uint32_t rec = 0, nseg = 0;
  TapeCursor tc{0u, 0u};

  while (true) {
    unsigned need = __ballot_sync(0xffffffffu, phase == kVIdle);
    while (need != 0u && !queue_empty) {
      if (left == 0u) {
        if (lane == 0) {
          const int64_t total = kDrt ? (int64_t)*P.task_count : Q.total;
          const int64_t b = (int64_t)atomicAdd(Q.counter, (unsigned long long)Q.batch);
          if (b < total) {
            *next = (unsigned)b;
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
        path = *next + rank;
        phase = kVStart;
      }
      __syncwarp();
      if (lane == 0) *next += take;
      left -= take;
      need = __ballot_sync(0xffffffffu, phase == kVIdle);
    }
    const unsigned m_start = __ballot_sync(0xffffffffu, phase == kVStart);
    const unsigned m_turn = __ballot_sync(0xffffffffu, phase >= kVVertex);
    const unsigned m_walk = __ballot_sync(0xffffffffu, phase == kVMain || phase == kVNee);
    if (queue_empty && (m_start | m_turn | m_walk) == 0u) break;
    const unsigned need_lanes = queue_empty ? 1u : defer;
    const bool run_start =
        (unsigned)__popc(m_start) >= need_lanes || (m_walk == 0u && m_turn == 0u && m_start != 0u);
    const bool run_turn = (unsigned)__popc(m_turn) >= need_lanes || (m_walk == 0u && m_turn != 0u);
    bool finished = false;
    bool begin = false;  // the lane's segment (xo, sd, rem) starts: roulette at the end of the turn

    // ------------------------------------------------------------ path start
    if (run_start && phase == kVStart) {
      int pix;
      thr = V3{1, 1, 1};
      L = V3{0, 0, 0};
      if (kDrt) {
        // last task first: the first launch's longest paths ended last, and
        // theirs are the tasks that take longest
        path = (uint32_t)*P.task_count - 1u - path;
        U(cTask) = path;
        const float4 t0 = P.task[(int64_t)path * kVpsTask];
        const float4* r = Q.ckpt + (int64_t)__float_as_uint(t0.y) * kVpsRec;
        const float4 r1 = r[1], r2 = r[2];
        path = __float_as_uint(t0.x);
        depth = __float_as_int(t0.z);
        const uint32_t sid = vps_sid(J, path, pix);
        seed_lane(rng, P.alt_seed, sid);
        rng.state = pcg_jump(rng.state, rng.inc, (uint32_t)P.draws * __float_as_uint(t0.w));
        xo = V3{r1.x, r1.y, r1.z};
        sd = V3{r2.x, r2.y, r2.z};
        float tn, tmax;
        slab(xo, recip(sd), tn, tmax);
        stage = 0;
        if (!(mu > 0.0f)) {
          phase = kVIdle;  // the flat pass skips the tasks of an empty medium
        } else {
          const float e = exp_nonpos(-(mu * tmax));
          const float u = next1d(rng);
          const float tp = -log_unit(1.0f - u * (1.0f - e)) / mu;
          F(cDist) = tp;
          p = xo;
          w = sd;
          rem = tp;
          acc = 1.0f;
          phase = kVNee;
        }
      } else {
        const uint32_t sid = vps_sid(J, path, pix);
        seed_lane(rng, J.seed, sid);
        depth = 0;
        lost = false;
        nseg = 0;
        const float u0 = next1d(rng), u1 = next1d(rng);
        V3 o, d;
        const uint32_t py = (uint32_t)pix / (uint32_t)J.width;
        camera_ray(J, (int)((uint32_t)pix - py * (uint32_t)J.width), (int)py, u0, u1, o, d);
        pcg_skip1(rng);
        const V3 inv_d = recip(d);
        float tn, tf;
        slab(o, inv_d, tn, tf);
        if (!(tn <= tf && tf > 0.0f)) {
          phase = kVIdle;  // misses the medium: no gradient, nothing to record
        } else {
          pcg_skip1(rng);  // the draw that seeds the second stream
          xo = advance(o, fmaxf(tn, 0.0f), d);
          sd = d;
          float a;
          slab(xo, inv_d, a, rem);
          begin = true;
          Pcg32 alt;
          seed_lane(alt, P.alt_seed, sid);
          U(cAlt) = (uint32_t)alt.state;
          U(cAlt + 1) = (uint32_t)(alt.state >> 32);
          U(cAlt + 2) = (uint32_t)alt.inc;
          U(cAlt + 3) = (uint32_t)(alt.inc >> 32);
          F(cSum) = F(cSum + 1) = F(cSum + 2) = 0.0f;
          U(cKeep) = 0xffffffffu;
        }
      }
    }

    // ------------------- segment ends, scattering events, next directions
    if (run_turn && phase >= kVVertex) {
      bool do_nee = false, do_dir = phase == kVDir;
      if (!kDrt && phase != kVDir) {
        // the segment that ended: reservoir and record
        const bool escaped = phase == kVEscape;
        const unsigned long long k64 = atomicAdd(Q.ckpt_count, 1ull);
        if ((int64_t)k64 < Q.ckpt_cap) {
          rec = (uint32_t)k64;
          float4* r = Q.ckpt + (int64_t)rec * kVpsRec;
          __stcs(r, make_float4(__uint_as_float(path), L.x, L.y, L.z));
          __stcs(r + 1, make_float4(xo.x, xo.y, xo.z, escaped ? F(cMax) : acc));
          __stcs(r + 2, make_float4(sd.x, sd.y, sd.z, __uint_as_float((nseg << 1) | (escaped ? 1u : 0u))));
          __stcs(r + 3, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
        } else {
          lost = true;
        }
        ++nseg;
        if (P.use_drt) {
          Pcg32 alt{pack64(U(cAlt), U(cAlt + 1)), pack64(U(cAlt + 2), U(cAlt + 3))};
          const float pick = next1d(alt);
          // the four transmittance draws are taken by the flat pass
          pcg_skip3(alt);
          pcg_skip1(alt);
          U(cAlt) = (uint32_t)alt.state;
          U(cAlt + 1) = (uint32_t)(alt.state >> 32);
          const V3 s{F(cSum) + thr.x, F(cSum + 1) + thr.y, F(cSum + 2) + thr.z};
          F(cSum) = s.x;
          F(cSum + 1) = s.y;
          F(cSum + 2) = s.z;
          const float ratio = ((thr.x / s.x + thr.y / s.y) + thr.z / s.z) / 3.0f;
          if (pick <= ratio) {
            F(cCur) = thr.x;
            F(cCur + 1) = thr.y;
            F(cCur + 2) = thr.z;
            U(cKeep) = rec;
            U(cKeepDepth) = (uint32_t)depth;
          }
        }
      }
      if (phase == kVEscape) {
        finished = true;
        if (!(depth <= 0 && J.hide_emitters)) {
          const bool weigh = P.use_nee && (kDrt || depth > 0);
          if (kEnv) {
            float pdf;
            V3 wd{sd.x * J.box.x, sd.y * J.box.y, sd.z * J.box.z};
            const float inv_len = 1.0f / sqrtf(fmaf(wd.z, wd.z, fmaf(wd.y, wd.y, wd.x * wd.x)));
            wd = V3{wd.x * inv_len, wd.y * inv_len, wd.z * inv_len};
            float u, v, st;
            env_uv(wd, u, v, st);
            pdf = env_pdf(J.env, u, v, st);
            const V3 Le = env_eval_uv(J.env, u, v);
            const float k = weigh ? env_mis(kInvFourPi, pdf) : 1.0f;
            L = V3{L.x + (thr.x * Le.x) * k, L.y + (thr.y * Le.y) * k, L.z + (thr.z * Le.z) * k};
          } else {
            const float k = weigh ? 0.5f : 1.0f;
            L = V3{L.x + thr.x * k, L.y + thr.y * k, L.z + thr.z * k};
          }
        }
      } else if (phase == kVVertex) {
        if (kDrt && stage == 0) {
          // the resampled point of the kept segment, with its weight T / pdf
          const float tp = F(cDist);
          float tn, tmax;
          slab(xo, recip(sd), tn, tmax);
          const float e = exp_nonpos(-(mu * tmax));
          const float pdf = (mu * exp_nonpos(-(mu * tp))) / (1.0f - e);
          xo = advance(xo, tp, sd);
          float4* t = P.task + (int64_t)U(cTask) * kVpsTask;
          reinterpret_cast<float*>(t + 1)[3] = acc / pdf;
          __stcs(t + 2, make_float4(xo.x, xo.y, xo.z, 0.0f));
          F(cNee) = F(cNee + 1) = F(cNee + 2) = 0.0f;
          stage = 1;
          do_nee = P.use_nee != 0;
          do_dir = !do_nee;
        } else {
          const V3 x = advance(xo, acc, sd);
          const Lookup lx = locate(J, x);
          const V3 a = albedo_at(J, albedo_lookup(J, lx, x), 1);
          thr = V3{thr.x * a.x, thr.y * a.y, thr.z * a.z};
          depth += 1;
          xo = x;
          if (depth >= J.max_depth) {
            finished = true;
          } else {
            do_nee = P.use_nee != 0;
            do_dir = !do_nee;
          }
        }
      }
      if (do_nee || do_dir) {
        if (do_dir) pcg_skip1(rng);
        const float u0 = next1d(rng), u1 = next1d(rng);
        V3 dir;
        if (kEnv && do_nee) {
          V3 Le;
          float pdf;
          dir = env_sample(J.env, u0, u1, Le, pdf);
          float k = 0.0f;
          if (pdf > 0.0f && pdf < kInf) k = (kInvFourPi * env_mis(pdf, kInvFourPi)) / pdf;
          F(cEnv) = Le.x * k;
          F(cEnv + 1) = Le.y * k;
          F(cEnv + 2) = Le.z * k;
        } else {
          dir = uniform_sphere(u0, u1);
        }
        dir = to_box(J, dir);
        float tn, tf;
        slab(xo, recip(dir), tn, tf);
        if (do_nee) {
          w = dir;
          p = xo;
          rem = tf;
          acc = 1.0f;
          phase = kVNee;
        } else {
          sd = dir;
          rem = tf;
          bool active = tf > 0.0f;  // else an accidental escape (:279-283)
          if (kDrt && stage == 1) {
            // the recursive path: its depth and its (unused) seeding draw (:103)
            stage = 2;
            depth += 1;
            active = active && depth < J.max_depth;
            if (active) pcg_skip1(rng);
          }
          begin = active;
          finished = !active;
        }
      }
    }

    // ------------------------------- a segment begins: Russian roulette
    if (begin) {
      const float q = fminf(fmaxf(fmaxf(thr.x, thr.y), thr.z), 0.99f);
      const bool rr = depth > J.rr_depth;
      const bool alive = thr.x != 0.0f || thr.y != 0.0f || thr.z != 0.0f;
      const float u = next1d(rng);
      if (!alive || (rr && !(u < q))) {
        finished = true;
      } else {
        if (rr) {
          const float iq = 1.0f / q;
          thr = V3{thr.x * iq, thr.y * iq, thr.z * iq};
        }
        p = xo;
        w = sd;
        acc = 0.0f;
        if (!kDrt) F(cMax) = rem;
        phase = kVMain;
      }
    }

    // ------------------------------ cooperative walk of the warp's last paths
    bool many = false;  // too many lanes walk for it
    if (!kSG && queue_empty) {
      const unsigned m_coop = __ballot_sync(0xffffffffu, !finished && (phase == kVMain || phase == kVNee));
      many = __popc(m_coop) > kCoopMost;
      if (m_coop != 0u && __popc(m_coop) <= kCoopMost) {
        float* s = s_coop + (threadIdx.x >> 5) * 64;
        vps_coop<kMode>(m_coop, phase == kVMain, J, rng, mu, inv_mu, p, w, rem, acc, s, s + 32, Q, tc, rec, lost);
      }
    }

    // ---------------------------------------------------- free-flight step
    // (several before the next look at the lanes that wait, see kWalkSteps)
    const int steps = kSG || (queue_empty && !many) ? 1 : kWalkSteps;
#pragma unroll 1
    for (int sub = 1;; ++sub) {
      bool ev = false;  // kVpsTape: a shadow-walk step with a gradient, at p
      float ev_sn = 0.0f;
      if (!finished && (phase == kVMain || phase == kVNee)) {
        float m = mu, inv_m = inv_mu, t;
        const float uf = next1d(rng);
        if (kSG) {
          m = mu;
          t = supergrid_flight(J, J.sg_new, p, w, rem, -log_unit(1.0f - uf), m);
          inv_m = 1.0f / m;
        } else {
          t = free_flight(uf, mu, inv_mu);
        }
        const bool valid = t <= rem;
        float st = 0.0f;
        V3 x;
        if (valid) {
          x = advance(p, t, w);
          st = J.scale * density_new(J, locate(J, x));
        }
        if (phase == kVMain) {
          if (valid) {
            const float ratio = m != 0.0f ? div_by(st, m, inv_m) : 0.0f;
            const float u = next1d(rng);
            acc = acc + t;
            if (u < ratio) {
              phase = kVVertex;
            } else {
              p = x;
              rem = rem - t;
            }
          } else {
            phase = kVEscape;
          }
        } else {
          bool done = !valid;
          if (valid) {
            const float sn = m - st;
            const float contrib = m != 0.0f ? div_by(sn, m, inv_m) : sn;
            acc = acc * contrib;
            p = x;
            rem = rem - t;
            if (!kDrt) {
              ev = contrib > 0.0f && !lost;
              ev_sn = sn;
            }
            done = acc == 0.0f;
          }
          if (done) {
            if (kDrt && stage == 0) {
              phase = kVVertex;
            } else {
              V3 c;
              if (kEnv) {
                c = V3{(thr.x * F(cEnv)) * acc, (thr.y * F(cEnv + 1)) * acc, (thr.z * F(cEnv + 2)) * acc};
              } else {
                const float mis = 0.5f, en = (1.0f / kInvFourPi) * acc;
                c = V3{((thr.x * kInvFourPi) * mis) * en, ((thr.y * kInvFourPi) * mis) * en,
                       ((thr.z * kInvFourPi) * mis) * en};
              }
              if (kDrt && stage == 1) {
                F(cNee) = c.x;
                F(cNee + 1) = c.y;
                F(cNee + 2) = c.z;
              } else {
                L = V3{L.x + c.x, L.y + c.y, L.z + c.z};
                if (!kDrt && !lost)
                  __stcs(Q.ckpt + (int64_t)rec * kVpsRec + 3, make_float4(c.x, c.y, c.z, 0.0f));
              }
              phase = kVDir;
            }
          }
        }
      }
      if (!kDrt && !tape_append(Q, tc, ev, p, rec, ev_sn)) lost = true;
      if (sub >= steps) break;
    }

    // -------------------------------------------------------------- path end
    if (finished) {
      if (kDrt) {
        P.task[(int64_t)U(cTask) * kVpsTask] =
            make_float4(__uint_as_float(path), F(cNee) + L.x, F(cNee + 1) + L.y, F(cNee + 2) + L.z);
      } else {
        __stcs(Q.path_ltot + path, make_float4(L.x, L.y, L.z, lost ? 1.0f : 0.0f));
        if (lost) {
          int unused;
          Q.lost_list[atomicAdd(Q.lost_count, 1ull)] = vps_sid(J, path, unused);
        } else if (P.use_drt && U(cKeep) != 0xffffffffu) {
          const V3 cur{F(cCur), F(cCur + 1), F(cCur + 2)};
          const float dmean = ((cur.x + cur.y) + cur.z) / 3.0f;
          if (dmean != 0.0f) {
            const float wmean = ((F(cSum) + F(cSum + 1)) + F(cSum + 2)) / 3.0f;
            float4* t = P.task + (int64_t)atomicAdd(P.task_count, 1ull) * kVpsTask;
            t[0] = make_float4(__uint_as_float(path), __uint_as_float(U(cKeep)), __uint_as_float(U(cKeepDepth)),
                               __uint_as_float(nseg));
            t[1] = make_float4((wmean * cur.x) / dmean, (wmean * cur.y) / dmean, (wmean * cur.z) / dmean, 0.0f);
          }
        }
      }
      phase = kVIdle;
    }
  }
  if (!kDrt) tape_close(Q, tc);
}

}  // namespace rcv
