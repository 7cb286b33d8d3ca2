// volpathsimple (plugins/volpathsimple.py): the reference's simplified
// volumetric path tracer and its differential-ratio-tracking adjoint, the
// `adjoint_integrator` of every grid experiment (experiments.py:131,245,364).
//
// Primal (VolpathSimpleIntegrator.sample, :53-327), per loop iteration:
// Russian roulette (1D); a real interaction by delta tracking
// (sample_real_interaction, :349-395: per collision a free-flight 1D and,
// inside the segment, a real/null 1D); NEE towards the environment (2D + one
// 1D per ratio-tracking step, :398-491); the phase sample (1D + 2D).  A path
// that leaves the cube sees the environment with the MIS weight of its last
// scattering event (:296-321).  After reaching the medium, one 1D seeds the
// adjoint's second stream (:103-113).
//
// Adjoint: a primal pass gives L; a replay with L_rem = L - (NEE so far)
// back-propagates
//   - the scattering term at each real interaction, MIS weight s^2/(1+s^2),
//     s = sigma_t (:160-186);
//   - the transmittance of each last segment by 4 uniform samples (:597-620);
//   - each NEE shadow ray by replaying its ratio tracking (:412-422, :481-505);
//   - differential ratio tracking: for every segment (escaping or not) a
//     reservoir keeps one, weighted by the throughput (:743-778); at the end a
//     distance is resampled on it in proportion to the transmittance and a
//     recursive path estimates the in-scattered radiance, MIS 1/(1+s^2)
//     (:508-594, :623-668).  Without subsampling this runs at every segment.
// The extra random numbers come from a second stream seeded with
// sample_tea_32(bits of lane 0's seeding draw, 1) (:108-113).
// sample_interaction_drt belongs to the Mitsuba fork the reference depends
// on; it is restated as a distance from the majorant's exponential truncated
// to the segment, weight = ratio-tracking transmittance / pdf.
//
// The arithmetic follows the oracle's float sequence.  The adjoint runs as
// two persistent tracers and two flat gradient passes over what they record
// (rcv_vps_trace.cuh); vps_kernel, one thread per path, renders the primal and
// takes the adjoints whose second stream has no fixed number of draws per
// segment (DRT without subsampling), the paths that a recording lost, and
// callers without a workspace.
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "rcv_common.h"
#include "rcv_pack.cuh"
#include "rcv_vps_trace.cuh"

namespace rcv {

struct VpsSeg {
  V3 o, d;
  float tmax;
};

// kEnv: the job has an environment map (else the constant white environment).
template <bool kEnv>
struct Vps {
  const VolJob& J;
  const VpsParams& P;
  float mu, inv_mu;  // global majorant of `new` (scale * max density) and 1/mu

  __device__ float flight(Pcg32& r, const V3& o, const V3& d, float tmax, float& m) const {
    const float u = next1d(r);
    m = mu;
    if (J.sg[0] > 0) {
      const float tau = -log_unit(1.0f - u);
      return supergrid_flight(J, J.sg_new, o, d, tmax, tau, m);
    }
    return free_flight(u, mu, inv_mu);
  }

  __device__ float sigma_t(const Lookup& l) const { return J.scale * density_new(J, l); }

  __device__ float real_interaction(Pcg32& r, const VpsSeg& seg) const {
    V3 p = seg.o;
    float rem = seg.tmax, t_acc = 0.0f;
    for (;;) {
      float m;
      const float t = flight(r, p, seg.d, rem, m);
      if (!(t <= rem)) return kInf;
      const V3 x = advance(p, t, seg.d);
      const float st = sigma_t(locate(J, x));
      const float ratio = m != 0.0f ? st / m : 0.0f;
      const float u = next1d(r);
      t_acc = t_acc + t;
      if (u < ratio) return t_acc;
      p = x;
      rem = rem - t;
    }
  }

  // Ratio tracking from o along w to tmax; with `adj`, scatters adj . dlog T.
  __device__ float transmittance(Pcg32& r, const V3& o, const V3& w, float tmax, const V3* adj) const {
    V3 q = o;
    float rem = tmax, tr = 1.0f;
    for (;;) {
      float m;
      const float t = flight(r, q, w, rem, m);
      if (!(t <= rem)) break;
      const V3 x = advance(q, t, w);
      const Lookup l = locate(J, x);
      const float sn = m - sigma_t(l);
      const float contrib = m != 0.0f ? sn / m : sn;
      if (adj != nullptr && contrib > 0.0f) {
        const float wn = (adj->x + adj->y) + adj->z;
        scatter_density(J, l, -(J.scale * wn) / sn);
      }
      tr = tr * contrib;
      q = x;
      rem = rem - t;
      if (tr == 0.0f) break;
    }
    return tr;
  }

  __device__ float exit_distance(const V3& o, const V3& d) const {
    float tn, tf;
    slab(o, recip(d), tn, tf);
    return tf;
  }

  // NEE towards the environment (sample_emitter_for_nee, :393-417): the
  // constant one sampled uniformly (MIS 1/2 against the phase function), a
  // map by importance with the power heuristic.
  __device__ V3 nee(Pcg32& r, const V3& x, const V3& thr, const V3* dL) const {
    Pcg32 replay = r;
    const float u0 = next1d(r), u1 = next1d(r);
    V3 w, e{0.0f, 0.0f, 0.0f};
    if (kEnv) {
      V3 Le;
      float pdf;
      w = to_box(J, env_sample(J.env, u0, u1, Le, pdf));
      float k = 0.0f;
      if (pdf > 0.0f && pdf < kInf) k = (kInvFourPi * env_mis(pdf, kInvFourPi)) / pdf;
      e = V3{Le.x * k, Le.y * k, Le.z * k};
    } else {
      w = to_box(J, uniform_sphere(u0, u1));
    }
    const float tf = exit_distance(x, w);
    const float tr = transmittance(r, x, w, tf, nullptr);
    V3 c;
    if (kEnv) {
      c = V3{(thr.x * e.x) * tr, (thr.y * e.y) * tr, (thr.z * e.z) * tr};
    } else {
      const float mis = 0.5f;
      const float en = (1.0f / kInvFourPi) * tr;
      c = V3{((thr.x * kInvFourPi) * mis) * en, ((thr.y * kInvFourPi) * mis) * en,
             ((thr.z * kInvFourPi) * mis) * en};
    }
    if (dL != nullptr) {
      const V3 adj{dL->x * c.x, dL->y * c.y, dL->z * c.z};
      pcg_skip1(replay);
      pcg_skip1(replay);
      transmittance(replay, x, w, tf, &adj);
    }
    return c;
  }

  __device__ V3 primal_from(Pcg32& r, VpsSeg seg, int depth, bool has_scattered, bool active) const {
    V3 L{0, 0, 0}, thr{1, 1, 1};
    bool escaped = false;
    while (active) {
      const float q = fminf(fmaxf(fmaxf(thr.x, thr.y), thr.z), 0.99f);
      const bool rr = depth > J.rr_depth;
      const bool alive = thr.x != 0.0f || thr.y != 0.0f || thr.z != 0.0f;
      const float u = next1d(r);
      if (!alive || (rr && !(u < q))) break;
      if (rr) {
        const float iq = 1.0f / q;
        thr = V3{thr.x * iq, thr.y * iq, thr.z * iq};
      }
      const float t = real_interaction(r, seg);
      if (!(t < kInf)) {
        escaped = true;
        break;
      }
      const V3 x = advance(seg.o, t, seg.d);
      const Lookup lx = locate(J, x);
      const V3 a = albedo_at(J, albedo_lookup(J, lx, x), 1);
      has_scattered = true;
      thr = V3{thr.x * a.x, thr.y * a.y, thr.z * a.z};
      depth += 1;
      if (depth >= J.max_depth) break;
      if (P.use_nee) {
        const V3 c = nee(r, x, thr, nullptr);
        L = V3{L.x + c.x, L.y + c.y, L.z + c.z};
      }
      pcg_skip1(r);
      const float pu0 = next1d(r), pu1 = next1d(r);
      seg.o = x;
      seg.d = to_box(J, uniform_sphere(pu0, pu1));
      const float tf = exit_distance(seg.o, seg.d);
      if (!(tf > 0.0f)) break;  // accidental escape (:279-283)
      seg.tmax = tf;
    }
    if (escaped && !(depth <= 0 && J.hide_emitters)) {
      if (kEnv) {
        // map hit: power heuristic against NEE after a scattering event (:280-298)
        float pdf;
        const V3 Le = env_along(seg.d, pdf);
        const float k = (P.use_nee && has_scattered) ? env_mis(kInvFourPi, pdf) : 1.0f;
        L = V3{L.x + (thr.x * Le.x) * k, L.y + (thr.y * Le.y) * k, L.z + (thr.z * Le.z) * k};
      } else {
        const float k = (P.use_nee && has_scattered) ? 0.5f : 1.0f;
        L = V3{L.x + thr.x * k, L.y + thr.y * k, L.z + thr.z * k};
      }
    }
    return L;
  }

  // Radiance of the environment map along a box direction and the pdf of
  // sampling it (the direction made a unit world direction first).
  __device__ V3 env_along(const V3& d, float& pdf) const {
    V3 wd{d.x * J.box.x, d.y * J.box.y, d.z * J.box.z};
    const float inv_len = 1.0f / sqrtf(fmaf(wd.z, wd.z, fmaf(wd.y, wd.y, wd.x * wd.x)));
    wd = V3{wd.x * inv_len, wd.y * inv_len, wd.z * inv_len};
    float u, v, st;
    env_uv(wd, u, v, st);
    pdf = env_pdf(J.env, u, v, st);
    return env_eval_uv(J.env, u, v);
  }

  // Camera ray, colour-channel draw, medium entry (reach_medium, :329-346);
  // `d` is the camera ray (for the environment when it misses the medium).
  __device__ bool camera(Pcg32& r, int pix, VpsSeg& seg, V3& d) const {
    const float u0 = next1d(r), u1 = next1d(r);
    V3 o;
    camera_ray(J, pix % J.width, pix / J.width, u0, u1, o, d);
    pcg_skip1(r);
    const V3 inv_d = recip(d);
    float tn, tf;
    slab(o, inv_d, tn, tf);
    if (!(tn <= tf && tf > 0.0f)) return false;
    seg.o = advance(o, fmaxf(tn, 0.0f), d);
    seg.d = d;
    float a;
    slab(seg.o, inv_d, a, seg.tmax);
    return true;
  }

  __device__ V3 render_path(uint32_t sid, int pix) const {
    Pcg32 r;
    seed_lane(r, J.seed, sid);
    VpsSeg seg;
    V3 d;
    if (!camera(r, pix, seg, d)) {
      if (J.hide_emitters) return V3{0.0f, 0.0f, 0.0f};
      if (kEnv) {
        float pdf;
        return env_along(d, pdf);
      }
      return V3{1.0f, 1.0f, 1.0f};
    }
    pcg_skip1(r);  // seeds the adjoint's second stream
    return primal_from(r, seg, 0, false, true);
  }

  __device__ void drt(Pcg32& alt, const VpsSeg& seg, int depth, const V3& adj) const {
    if (!(mu > 0.0f)) return;
    const float e = exp_nonpos(-(mu * seg.tmax));
    const float u = next1d(alt);
    const float tp = -log_unit(1.0f - u * (1.0f - e)) / mu;
    const float pdf = (mu * exp_nonpos(-(mu * tp))) / (1.0f - e);
    const float tr = transmittance(alt, seg.o, seg.d, tp, nullptr);
    const float wdrt = tr / pdf;
    const V3 x = advance(seg.o, tp, seg.d);
    const Lookup l = locate(J, x);
    const AlbedoLookup al = albedo_lookup(J, l, x);
    const float st = sigma_t(l);
    const V3 a = albedo_at(J, al, 1);
    V3 Li{0, 0, 0};
    if (P.use_nee) Li = nee(alt, x, V3{1, 1, 1}, nullptr);
    pcg_skip1(alt);
    const float pu0 = next1d(alt), pu1 = next1d(alt);
    VpsSeg next{x, to_box(J, uniform_sphere(pu0, pu1)), 0.0f};
    const float tf = exit_distance(next.o, next.d);
    const bool ok = tf > 0.0f;
    next.tmax = tf;
    const int next_depth = depth + 1;
    const bool active = ok && next_depth < J.max_depth;
    if (active) pcg_skip1(alt);  // the recursive call's seeding draw (:103)
    const V3 Lr = primal_from(alt, next, next_depth, true, active);
    Li = V3{Li.x + Lr.x, Li.y + Lr.y, Li.z + Lr.z};
    const float mis = P.use_drt_mis ? 1.0f / (1.0f + st * st) : 1.0f;
    const float k0 = mis * wdrt;
    const V3 k{(k0 * adj.x) * Li.x, (k0 * adj.y) * Li.y, (k0 * adj.z) * Li.z};
    scatter_density(J, l, J.scale * ((k.x * a.x + k.y * a.y) + k.z * a.z));
    if (J.grad_albedo != nullptr) scatter_albedo(J, al, V3{k.x * st, k.y * st, k.z * st});
  }

  __device__ void backward_path(uint32_t sid, int pix, const V3& dL) const {
    const V3 Ltot = render_path(sid, pix);
    Pcg32 r, alt;
    seed_lane(r, J.seed, sid);
    seed_lane(alt, P.alt_seed, sid);
    VpsSeg seg;
    V3 d;
    if (!camera(r, pix, seg, d)) return;
    pcg_skip1(r);
    V3 res = Ltot, thr{1, 1, 1};
    int depth = 0;
    V3 wsum{0, 0, 0}, cur{0, 0, 0};
    bool have = false;
    VpsSeg keep{};
    int keep_depth = 0;
    for (;;) {
      const float q = fminf(fmaxf(fmaxf(thr.x, thr.y), thr.z), 0.99f);
      const bool rr = depth > J.rr_depth;
      const bool alive = thr.x != 0.0f || thr.y != 0.0f || thr.z != 0.0f;
      const float u = next1d(r);
      if (!alive || (rr && !(u < q))) break;
      if (rr) {
        const float iq = 1.0f / q;
        thr = V3{thr.x * iq, thr.y * iq, thr.z * iq};
      }
      const float t = real_interaction(r, seg);
      const bool escape = !(t < kInf);
      if (P.use_drt) {
        if (P.use_drt_subsampling) {
          wsum = V3{wsum.x + thr.x, wsum.y + thr.y, wsum.z + thr.z};
          const float pick = next1d(alt);
          const float ratio = ((thr.x / wsum.x + thr.y / wsum.y) + thr.z / wsum.z) / 3.0f;
          if (pick <= ratio) {
            cur = thr;
            keep = seg;
            keep_depth = depth;
            have = true;
          }
        } else {
          drt(alt, seg, depth, V3{dL.x * thr.x, dL.y * thr.y, dL.z * thr.z});
        }
      }
      if (!escape) {
        const V3 x = advance(seg.o, t, seg.d);
        const Lookup l = locate(J, x);
        const AlbedoLookup al = albedo_lookup(J, l, x);
        const float st = sigma_t(l);
        const V3 a = albedo_at(J, al, 1);
        if (!P.use_drt || P.use_drt_mis) {
          const float mis = P.use_drt ? (st * st) / (1.0f + st * st) : 1.0f;
          const float inv_pdf = 1.0f / st;
          const V3 k{((mis * dL.x) * (res.x / fmaxf(1e-8f, a.x))) * inv_pdf,
                     ((mis * dL.y) * (res.y / fmaxf(1e-8f, a.y))) * inv_pdf,
                     ((mis * dL.z) * (res.z / fmaxf(1e-8f, a.z))) * inv_pdf};
          scatter_density(J, l, J.scale * ((k.x * a.x + k.y * a.y) + k.z * a.z));
          if (J.grad_albedo != nullptr) scatter_albedo(J, al, V3{k.x * st, k.y * st, k.z * st});
        }
      }
      {
        const float interval = escape ? seg.tmax : t;
        const float w = (dL.x * res.x + dL.y * res.y) + dL.z * res.z;
        const float coef = -(w * (interval * 0.25f));
        for (int j = 0; j < 4; ++j) {
          const float tj = next1d(alt) * interval;
          scatter_density(J, locate(J, advance(seg.o, tj, seg.d)), J.scale * coef);
        }
      }
      if (escape) break;
      const V3 x = advance(seg.o, t, seg.d);
      const Lookup lx = locate(J, x);
      const V3 a = albedo_at(J, albedo_lookup(J, lx, x), 1);
      thr = V3{thr.x * a.x, thr.y * a.y, thr.z * a.z};
      depth += 1;
      if (depth >= J.max_depth) break;
      if (P.use_nee) {
        const V3 c = nee(r, x, thr, &dL);
        res = V3{res.x - c.x, res.y - c.y, res.z - c.z};
      }
      pcg_skip1(r);
      const float pu0 = next1d(r), pu1 = next1d(r);
      seg.o = x;
      seg.d = to_box(J, uniform_sphere(pu0, pu1));
      const float tf = exit_distance(seg.o, seg.d);
      if (!(tf > 0.0f)) break;
      seg.tmax = tf;
    }
    if (P.use_drt && P.use_drt_subsampling && have) {
      const float dmean = ((cur.x + cur.y) + cur.z) / 3.0f;
      if (dmean != 0.0f) {
        const float wmean = ((wsum.x + wsum.y) + wsum.z) / 3.0f;
        const V3 sw{(wmean * cur.x) / dmean, (wmean * cur.y) / dmean, (wmean * cur.z) / dmean};
        drt(alt, keep, keep_depth, V3{sw.x * dL.x, sw.y * dL.y, sw.z * dL.z});
      }
    }
  }
};

template <bool kAdj, bool kEnv>
__global__ void __launch_bounds__(128) vps_kernel(const __grid_constant__ VolJob J,
                                                  const __grid_constant__ VpsParams P) {
  const float mu = J.scale * bits_to_float(__ldg(J.maxbits + 1));
  const Vps<kEnv> v{J, P, mu, 1.0f / mu};
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const bool listed = kAdj && P.lost_list != nullptr;
  const int64_t n = listed ? (int64_t)*P.lost_count : J.path_count;
  for (int64_t path = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; path < n; path += stride) {
    const uint32_t sid = listed ? P.lost_list[path] : (uint32_t)path;  // pixel * spp + sample
    const int pix = (int)(sid / (uint32_t)J.spp);
    if (kAdj) {
      const float* g = J.grad_img + (int64_t)pix * 3;
      const float fs = (float)J.spp;
      v.backward_path(sid, pix, V3{g[0] / fs, g[1] / fs, g[2] / fs});
    } else {
      const V3 L = v.render_path(sid, pix);
      P.path_out[path] = make_float4(L.x, L.y, L.z, 0.0f);
    }
  }
}

// Resident blocks per SM: 7 without spills for the DRT paths (72 registers), 6
// for the first (80; at 7, which spills, a DRT step is 2 % slower).
template <int kMode, bool kSG, bool kEnv>
__global__ void __launch_bounds__(kVpsBlock, kMode == kVpsDrt ? 7 : 6) vps_trace_kernel(const __grid_constant__ VolJob J,
                                                                 const __grid_constant__ VpsParams P,
                                                                 const __grid_constant__ Queue Q) {
  trace_vps<kMode, kSG, kEnv>(J, P, Q);
}

__device__ __forceinline__ V3 vps_dL(const VolJob& J, int pix) {
  const float* g = J.grad_img + (int64_t)pix * 3;
  const float fs = (float)J.spp;
  return V3{g[0] / fs, g[1] / fs, g[2] / fs};
}

// Flat pass over the segment records and the DRT tasks: the transmittance
// term of every segment (4 uniform samples of the second stream), the
// scattering term at its end, the weight of its shadow walk (for the pass
// over the tape), and the DRT term of every task.
__global__ void __launch_bounds__(256, 4) vps_segments_kernel(const __grid_constant__ VolJob J,
                                                           const __grid_constant__ VpsParams P,
                                                           const __grid_constant__ Queue Q, float* __restrict__ wn) {
  const int64_t nrec = min((int64_t)*Q.ckpt_count, Q.ckpt_cap), ntask = P.use_drt ? (int64_t)*P.task_count : 0;
  // (whole warps: the reductions go pairwise)
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int64_t first = int64_t(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u);
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t base = first; base < nrec; base += stride) {
    const int64_t i = base + lane;
    bool on = false, event = false;  // the record counts; it ends at a scattering event
    V3 o{0, 0, 0}, d{0, 0, 0}, ga{0, 0, 0};
    float interval = 0.0f, coef = 0.0f, ge = 0.0f;
    Pcg32 alt{0ull, 0ull};
    Lookup l{};
    AlbedoLookup al{};
    if (i < nrec) {
      const float4* r = Q.ckpt + i * kVpsRec;
      const float4 r0 = __ldcs(r), r1 = __ldcs(r + 1), r2 = __ldcs(r + 2), r3 = __ldcs(r + 3);
      const uint32_t path = __float_as_uint(r0.x);
      const float4 lt = __ldg(Q.path_ltot + path);
      on = lt.w == 0.0f;
      if (!on) {  // lost: the path is taken whole by vps_kernel
        wn[i] = 0.0f;
      } else {
        int pix;
        const uint32_t sid = vps_sid(J, path, pix);
        const V3 dL = vps_dL(J, pix);
        const V3 res{lt.x - r0.y, lt.y - r0.z, lt.z - r0.w};
        wn[i] = (dL.x * r3.x + dL.y * r3.y) + dL.z * r3.z;
        o = V3{r1.x, r1.y, r1.z};
        d = V3{r2.x, r2.y, r2.z};
        interval = r1.w;
        const uint32_t kf = __float_as_uint(r2.w);
        event = (kf & 1u) == 0u && (!P.use_drt || P.use_drt_mis);
        if (event) {
          const V3 x = advance(o, interval, d);
          l = locate(J, x);
          al = albedo_lookup(J, l, x);
          const float st = J.scale * density_new(J, l);
          const V3 a = albedo_at(J, al, 1);
          const float mis = P.use_drt ? (st * st) / (1.0f + st * st) : 1.0f;
          const float inv_pdf = 1.0f / st;
          const V3 k{((mis * dL.x) * (res.x / fmaxf(1e-8f, a.x))) * inv_pdf,
                     ((mis * dL.y) * (res.y / fmaxf(1e-8f, a.y))) * inv_pdf,
                     ((mis * dL.z) * (res.z / fmaxf(1e-8f, a.z))) * inv_pdf};
          ge = J.scale * ((k.x * a.x + k.y * a.y) + k.z * a.z);
          ga = V3{k.x * st, k.y * st, k.z * st};
        }
        seed_lane(alt, P.alt_seed, sid);
        alt.state = pcg_jump(alt.state, alt.inc, (uint32_t)P.draws * (kf >> 1) + (uint32_t)(P.draws - 4));
        const float w = (dL.x * res.x + dL.y * res.y) + dL.z * res.z;
        coef = -(w * (interval * 0.25f));
      }
    }
    if (__any_sync(0xffffffffu, event)) {
      scatter_density_warp(event, J.grad_cells, l, ge);
      if (J.grad_albedo != nullptr) scatter_albedo_warp(event, albedo_record(J, al), al, ga);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float tj = next1d(alt) * interval;
      scatter_density_warp(on, J.grad_cells, locate(J, advance(o, tj, d)), J.scale * coef);
    }
  }
  if (!(J.scale * bits_to_float(__ldg(J.maxbits + 1)) > 0.0f)) return;  // empty medium: no DRT
  for (int64_t base = first; base < ntask; base += stride) {
    const int64_t i = base + lane;
    const bool on = i < ntask;
    Lookup l{};
    AlbedoLookup al{};
    float ge = 0.0f;
    V3 ga{0, 0, 0};
    if (on) {
      const float4* t = P.task + i * kVpsTask;
      const float4 t0 = __ldcs(t), t1 = __ldcs(t + 1), t2 = __ldcs(t + 2);
      int pix;
      vps_sid(J, __float_as_uint(t0.x), pix);
      const V3 dL = vps_dL(J, pix), x{t2.x, t2.y, t2.z};
      l = locate(J, x);
      al = albedo_lookup(J, l, x);
      const float st = J.scale * density_new(J, l);
      const V3 a = albedo_at(J, al, 1);
      const float mis = P.use_drt_mis ? 1.0f / (1.0f + st * st) : 1.0f;
      const float k0 = mis * t1.w;
      const V3 k{(k0 * (t1.x * dL.x)) * t0.y, (k0 * (t1.y * dL.y)) * t0.z, (k0 * (t1.z * dL.z)) * t0.w};
      ge = J.scale * ((k.x * a.x + k.y * a.y) + k.z * a.z);
      ga = V3{k.x * st, k.y * st, k.z * st};
    }
    scatter_density_warp(on, J.grad_cells, l, ge);
    if (J.grad_albedo != nullptr) scatter_albedo_warp(on, albedo_record(J, al), al, ga);
  }
}

// Flat pass over the shadow-walk steps on the tape: -(weight of the walk) /
// sigma_n at each.
__global__ void __launch_bounds__(256, 6) vps_shadow_kernel(const __grid_constant__ VolJob J,
                                                         const __grid_constant__ Queue Q,
                                                         const float* __restrict__ wn) {
  const int64_t n = min((int64_t)*Q.tape_count, Q.tape_cap);
  const int64_t first = int64_t(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u);
  for (int64_t base = first; base < n; base += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = base + (threadIdx.x & 31u);
    const float4 ev = i < n ? __ldcs(Q.tape + i) : make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(kTapeEmpty));
    const uint32_t ref = __float_as_uint(ev.w);
    const float w = ref != kTapeEmpty ? __ldg(wn + ref) : 0.0f;
    const bool on = w != 0.0f;
    float g = 0.0f;
    if (on) g = -(J.scale * w) / __ldcs(Q.tape_f + i);
    scatter_density_warp(on, J.grad_cells, locate(J, V3{ev.x, ev.y, ev.z}), g);
  }
}

// Workspace of the recorded adjoint over `paths` paths at a time (256-byte
// aligned sections): counters (hand-out of both tracers, records, tape slots,
// lost paths, tasks) | order buckets | pixel order | per-path radiance |
// segment records | their shadow weights | tape (16 + 4 bytes a slot) | tasks
// | lost list.
// Room per path: 6 segments and 48 shadow steps.  A path of a medium that
// fills the view takes about 3 segments and 20 steps at the albedos and
// depths of the test scenes; what does not fit is traced by vps_kernel.
constexpr int kVpsRecsPerPath = 6, kVpsSlotsPerPath = 48;
constexpr int64_t kVpsMaxPaths = int64_t(1) << 22;  // 6 GB of workspace: larger films go in several passes
constexpr int64_t kVpsMinPaths = int64_t(1) << 16;

struct VpsLayout {
  uint64_t counters, buckets, order, ltot, rec, wn, tape, task, lost, total;
};

static VpsLayout vps_layout(int64_t npix, int64_t paths) {
  VpsLayout L;
  const uint64_t n = (uint64_t)paths;
  L.counters = 0;
  L.buckets = 256;
  L.order = align256(kRenderHeadBytes);
  L.ltot = align256(L.order + uint64_t(npix) * sizeof(uint32_t));
  L.rec = align256(L.ltot + n * 16u);
  L.wn = align256(L.rec + n * kVpsRecsPerPath * 64u);
  L.tape = align256(L.wn + n * kVpsRecsPerPath * 4u);
  L.task = align256(L.tape + uint64_t(tape_capacity(paths, kVpsSlotsPerPath)) * 20u);
  L.lost = align256(L.task + n * kVpsTask * 16u);
  L.total = align256(L.lost + n * 4u);
  return L;
}

// Paths that a workspace of `bytes` takes at a time (0: too small).
static int64_t vps_paths_for(int64_t npix, int64_t paths, uint64_t bytes) {
  int64_t n = paths < kVpsMaxPaths ? paths : kVpsMaxPaths;
  while (vps_layout(npix, n).total > bytes) {
    if (n <= kVpsMinPaths) return 0;
    n = n / 2 > kVpsMinPaths ? n / 2 : kVpsMinPaths;
  }
  return n;
}

using VpsKernel = void (*)(VolJob, VpsParams, Queue);
static const VpsKernel kVpsKernels[2][4] = {
    {vps_trace_kernel<kVpsTape, false, false>, vps_trace_kernel<kVpsTape, true, false>,
     vps_trace_kernel<kVpsTape, false, true>, vps_trace_kernel<kVpsTape, true, true>},
    {vps_trace_kernel<kVpsDrt, false, false>, vps_trace_kernel<kVpsDrt, true, false>,
     vps_trace_kernel<kVpsDrt, false, true>, vps_trace_kernel<kVpsDrt, true, true>}};

static int vps_resident(int mode, int variant) {
  static std::once_flag once;
  static int blocks[2][4];
  std::call_once(once, [] {
    for (int k = 0; k < 8; ++k) {
      int& b = blocks[k / 4][k % 4];
      b = 1;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kVpsKernels[k / 4][k % 4], kVpsBlock, 0);
      if (b < 1) b = 1;
    }
  });
  return blocks[mode][variant];
}

// sample_tea_32(bits of lane 0's fourth draw, 1)[0] (:108-113).
static uint32_t vps_alt_seed(uint32_t seed) {
  Pcg32 r;
  seed_lane(r, seed, 0u);
  next1d(r);
  next1d(r);
  next1d(r);
  const float u = next1d(r);
  uint32_t bits;
  std::memcpy(&bits, &u, 4);
  uint32_t a, b;
  tea(bits, 1u, 4, a, b);
  return a;
}

static int vps_setup(const rcv_medium* m, const rcv_sensor* s, const rcv_volpath_options* o,
                     const rcv_volpathsimple_flags* f, uint32_t seed, int spp, VolJob* J, VpsParams* P) {
  int rc = make_volume_job(m, s, o, seed, spp, J);
  if (rc) return rc;
  std::memset(P, 0, sizeof(*P));
  const rcv_volpathsimple_flags def{1, 1, 1, 1};
  const rcv_volpathsimple_flags& F = f ? *f : def;
  P->use_nee = F.use_nee != 0;
  P->use_drt = F.use_drt != 0;
  P->use_drt_subsampling = F.use_drt_subsampling != 0;
  P->use_drt_mis = F.use_drt_mis != 0;
  P->alt_seed = vps_alt_seed(seed);
  return RCV_OK;
}

// Grid-stride launch: at most 16 blocks of 128 threads per SM.
static unsigned vps_grid(int64_t paths) {
  static std::once_flag once;
  static int sms = 1;
  std::call_once(once, [] {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms < 1) sms = 1;
  });
  int64_t blocks = (paths + 127) / 128;
  if (blocks > int64_t(sms) * 16) blocks = int64_t(sms) * 16;
  return (unsigned)(blocks < 1 ? 1 : blocks);
}

static int vps_whole(const VolJob& J, const VpsParams& P, unsigned grid, cudaStream_t st) {
  if (J.env.valid)
    vps_kernel<true, true><<<grid, 128, 0, st>>>(J, P);
  else
    vps_kernel<true, false><<<grid, 128, 0, st>>>(J, P);
  return launched("volpathsimple adjoint launch");
}

// The recorded adjoint of all paths, `chunk` at a time.
static int vps_recorded(VolJob J, VpsParams P, const rcv_volpath_options* o, char* ws, int64_t npix, int64_t chunk,
                        cudaStream_t st) {
  const VpsLayout L = vps_layout(npix, chunk);
  unsigned long long* qc = reinterpret_cast<unsigned long long*>(ws + L.counters);
  int rc = RCV_OK;
  if (o->order != RCV_ORDER_ROW_MAJOR) {
    // by the estimate: the path lengths of an earlier call would order a little
    // better but would tie the scratch to the caller
    OrderJob O;
    O.J = J;
    O.head = ws;
    O.npix = (int32_t)npix;
    O.buckets = reinterpret_cast<uint32_t*>(ws + L.buckets);
    O.order = reinterpret_cast<uint32_t*>(ws + L.order);
    O.cost = nullptr;
    O.chord = o->order == RCV_ORDER_LONGEST_FIRST;
    rc = order_pixels(&O, 1, st);
    if (rc) return rc;
    J.pixel_order = O.order;
  }
  P.draws = P.use_drt ? 5 : 4;
  P.task = reinterpret_cast<float4*>(ws + L.task);
  P.task_count = qc + 5;
  Queue Q;
  std::memset(&Q, 0, sizeof(Q));
  Q.ckpt = reinterpret_cast<float4*>(ws + L.rec);
  Q.ckpt_count = qc + 2;
  Q.ckpt_cap = chunk * kVpsRecsPerPath;
  Q.tape = reinterpret_cast<float4*>(ws + L.tape);
  Q.tape_f = reinterpret_cast<float*>(ws + L.tape + uint64_t(tape_capacity(chunk, kVpsSlotsPerPath)) * 16u);
  Q.tape_count = qc + 3;
  const int per_path = o->tape_events_per_path;
  Q.tape_cap = tape_capacity(chunk, per_path >= 1 && per_path < kVpsSlotsPerPath ? per_path : kVpsSlotsPerPath);
  Q.path_ltot = reinterpret_cast<float4*>(ws + L.ltot);
  Q.lost_list = reinterpret_cast<uint32_t*>(ws + L.lost);
  Q.lost_count = qc + 4;
  // launch options beyond a warp's means are brought into range (the adjoint
  // of one thread per path ignored them)
  Q.defer = o->defer > 0 ? (o->defer < 32 ? o->defer : 32) : 8;
  float* wn = reinterpret_cast<float*>(ws + L.wn);
  const int variant = (J.sg[0] > 0 ? 1 : 0) + (J.env.valid ? 2 : 0);
  const int sms = tracer_sm_count();
  for (int64_t base = 0; base < J.path_count; base += chunk) {
    const int64_t n = J.path_count - base < chunk ? J.path_count - base : chunk;
    J.path_begin = -base;  // path p of the pass is path base + p of the film
    if (base > 0 || J.pixel_order == nullptr)
      RCV_TRY_CUDA(cudaMemsetAsync(qc, 0, 8 * sizeof(unsigned long long), st), "counters reset");
    for (int mode = kVpsTape; mode <= (P.use_drt ? kVpsDrt : kVpsTape); ++mode) {
      Q.counter = qc + mode;
      Q.total = n;
      const int64_t cap = int64_t(sms) * vps_resident(mode, variant);
      const int64_t batch = paths_per_fetch(n);
      Q.batch = (int32_t)batch;
      int64_t blocks = (n + batch * kVpsWarps - 1) / (batch * kVpsWarps);
      if (blocks > cap) blocks = cap;
      kVpsKernels[mode][variant]<<<(unsigned)blocks, kVpsBlock, 0, st>>>(J, P, Q);
      rc = launched("volpathsimple tracer launch");
      if (rc) return rc;
    }
    // as many blocks as are resident, so that the pass goes through its records
    // once (8 blocks per SM in two waves: DRT step of 512^2 x 16 spp 2978 us, so 2923)
    vps_segments_kernel<<<(unsigned)sms * 4u, 256, 0, st>>>(J, P, Q, wn);
    rc = launched("volpathsimple segments launch");
    if (rc) return rc;
    vps_shadow_kernel<<<(unsigned)sms * 6u, 256, 0, st>>>(J, Q, wn);
    rc = launched("volpathsimple shadow launch");
    if (rc) return rc;
    VpsParams R = P;
    R.lost_list = Q.lost_list;
    R.lost_count = Q.lost_count;
    rc = vps_whole(J, R, vps_grid(n) < (unsigned)sms ? vps_grid(n) : (unsigned)sms * 4u, st);
    if (rc) return rc;
  }
  return RCV_OK;
}

}  // namespace rcv

using namespace rcv;

extern "C" uint64_t rcv_volpathsimple_workspace_bytes(int32_t width, int32_t height, int32_t spp) {
  if (width <= 0 || height <= 0 || spp <= 0) return 0;
  return align256(uint64_t(width) * height * spp * 16u);
}

extern "C" int rcv_render_volpathsimple(const rcv_medium* m, const rcv_sensor* s, const rcv_volpath_options* o,
                                        const rcv_volpathsimple_flags* f, uint32_t seed, int32_t spp, float* img,
                                        void* workspace, void* stream) {
  RCV_REQUIRE(img != nullptr && workspace != nullptr, "image / workspace are NULL");
  RCV_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, "workspace must be 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  VolJob J;
  VpsParams P;
  int rc = vps_setup(m, s, o, f, seed, spp, &J, &P);
  if (rc) return rc;
  P.path_out = static_cast<float4*>(workspace);
  if (J.env.valid)
    vps_kernel<false, true><<<vps_grid(J.path_count), 128, 0, st>>>(J, P);
  else
    vps_kernel<false, false><<<vps_grid(J.path_count), 128, 0, st>>>(J, P);
  rc = launched("volpathsimple launch");
  if (rc) return rc;
  return launch_reduce(false, P.path_out, 0, int64_t(J.width) * J.height, J.spp, img, nullptr, st);
}

extern "C" int rcv_render_backward_volpathsimple(const rcv_medium* m, const rcv_sensor* s,
                                                 const rcv_volpath_options* o, const rcv_volpathsimple_flags* f,
                                                 uint32_t seed, int32_t spp, const float* grad_img,
                                                 float* grad_density, float* grad_albedo, void* stream) {
  return rcv_render_backward_volpathsimple_ws(m, s, o, f, seed, spp, grad_img, grad_density, grad_albedo, nullptr, 0,
                                              stream);
}

extern "C" uint64_t rcv_volpathsimple_adjoint_workspace_bytes(int32_t width, int32_t height, int32_t spp) {
  if (width <= 0 || height <= 0 || spp <= 0) return 0;
  const int64_t npix = int64_t(width) * height, paths = npix * spp;
  return vps_layout(npix, paths < kVpsMaxPaths ? paths : kVpsMaxPaths).total;
}

extern "C" int rcv_render_backward_volpathsimple_ws(const rcv_medium* m, const rcv_sensor* s,
                                                    const rcv_volpath_options* o, const rcv_volpathsimple_flags* f,
                                                    uint32_t seed, int32_t spp, const float* grad_img,
                                                    float* grad_density, float* grad_albedo, void* workspace,
                                                    uint64_t workspace_bytes, void* stream) {
  RCV_REQUIRE(grad_img != nullptr && grad_density != nullptr, "gradient buffers are NULL");
  RCV_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, "workspace must be 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  VolJob J;
  VpsParams P;
  int rc = vps_setup(m, s, o, f, seed, spp, &J, &P);
  if (rc) return rc;
  const bool want_albedo = grad_albedo != nullptr && m->albedo_old != nullptr;
  rc = reset_gradients(m, want_albedo, st);
  if (rc) return rc;
  if (!want_albedo) J.grad_albedo = nullptr;
  J.grad_img = grad_img;
  const int64_t npix = int64_t(J.width) * J.height;
  const bool recorded = workspace != nullptr && (!P.use_drt || P.use_drt_subsampling);
  const int64_t chunk = recorded ? vps_paths_for(npix, J.path_count, workspace_bytes) : 0;
  if (chunk > 0)
    rc = vps_recorded(J, P, o, static_cast<char*>(workspace), npix, chunk, st);
  else
    rc = vps_whole(J, P, vps_grid(J.path_count), st);
  if (rc) return rc;
  return launch_fold(m, grad_density, want_albedo ? grad_albedo : nullptr, st);
}
