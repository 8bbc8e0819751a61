// Volumetric progressive photon mapping: photon emission, photon tree,
// per-pixel gather and the progressive N / R / flux update in FP64, or the
// reference's ray-marched estimate with one global radius per pass.
//
// Reference: PPM_PT.comp (main :452-489, interactWithMedium :393-447,
// depositPhoton :304-321), PPM_PE.comp (samplePhotonMap :304-375, ray march
// :443-546), RenderTechniquePPM.cpp (RecordDrawCommands :229-300,
// UpdateRadius :302-312), KDTree.{h,cpp} (a stub in the reference).
//
// The reference deposits photons into a 100^3 x 32-slot grid hash (extra
// photons dropped) and shrinks one global radius per pass; this build keeps
// every photon, orders them along a 30-bit Morton curve and builds a binary
// radix tree over them (the LBVH of the beam pipeline, with point leaves:
// a spatial median-style subdivision standing in for the kd-tree), and
// keeps per-pixel statistics as stochastic progressive photon mapping
// does: each pass one measurement point per pixel (a delta-tracked
// collision along the camera ray), M photons within the pixel's radius R,
//   N' = N + alpha M,  ratio = (N + alpha M) / (N + M),
//   R' = R ratio^(1/3),  tau' = (tau + Phi) ratio,
// with Phi = sum_p f(w_p . -w_cam) Phi_p / sigma_t(x), and the estimate
//   L = background / k + albedo tau / (4/3 pi R^3 k).
// Photons are stored at every real collision with the power arriving there,
// so direct and multiple scattering both come from the photon map.
#include <cmath>

#include "track.cuh"
#include "sort.cuh"
#include "ppb.cuh"
#include "ppm.cuh"

namespace vcr {

vcr_status lbvh_build(vcr_ctx* ctx, const uint32_t* codes, int n, uint32_t* left, uint32_t* right, cudaStream_t st);
size_t lbvh_cluster_bytes(size_t n);
vcr_status lbvh_build_refit(vcr_ctx* ctx, const uint32_t* codes, const uint32_t* order, const float4* seg_a,
                            const float4* seg_b, int n, uint32_t* left, uint32_t* right, float4* clusters,
                            float4* leaf_lo, float4* leaf_hi, float4* node_lo, float4* node_hi, cudaStream_t st,
                            float4* node_pk);

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* sums, uint32_t* d_total,
                               cudaStream_t st);
constexpr uint32_t kPlacePhotons = 1u << 21;  // exclusive_scan_u32's limit

// Photon box entry and power: the same sun / constant-sky emission as the
// beams (see ppb.cu).
__device__ __forceinline__ float ppm_box_entry(const SceneView& s, f3 d, Rng& rng, f3& o) {
  f3 e = s.b1 - s.b0;
  float ax = fabsf(d.x) * (e.y * e.z), ay = fabsf(d.y) * (e.x * e.z), az = fabsf(d.z) * (e.x * e.y);
  float at = (ax + ay) + az;
  float sel = rng_next(rng) * at;
  float u = rng_next(rng), v = rng_next(rng);
  if (sel < ax) o = mk(d.x > 0.0f ? s.b0.x : s.b1.x, s.b0.y + u * e.y, s.b0.z + v * e.z);
  else if (sel < ax + ay) o = mk(s.b0.x + u * e.x, d.y > 0.0f ? s.b0.y : s.b1.y, s.b0.z + v * e.z);
  else o = mk(s.b0.x + u * e.x, s.b0.y + v * e.y, d.z > 0.0f ? s.b0.z : s.b1.z);
  return at;
}

// Persistent photon tracing: a lane takes the next photon (one atomic per
// warp on the launch's cursor) whenever its photon has ended, so the lanes
// of a warp whose photons end early keep working while the warp's longest
// path runs.  Deposits at every real collision go to a shared buffer
// through one atomic per warp and round (order fixed later by uid; a
// photon's path, and so every deposit, is the same whichever lane traces
// it).  n_events[p] is the number of photon p's deposits.
__device__ __forceinline__ void ppm_start_photon(const SceneView& s, uint32_t p, uint32_t photons, uint32_t seed,
                                                 uint32_t pass, Rng& rng, f3& o, f3& d, f3& power) {
  rng = rng_pcg(seed ^ kPpmEmitSalt, p, pass);
  const float inv = 1.0f / ((float)photons * 0.5f);
  bool sun = rng_next(rng) < 0.5f;
  if (sun) {
    d = s.sun;
  } else {
    float z = 1.0f - 2.0f * rng_next(rng);
    float sn, cs;
    vsincos2pi(rng_next(rng), &sn, &cs);
    float rr = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    d = mk(rr * cs, rr * sn, z);
  }
  float at = ppm_box_entry(s, d, rng, o);
  if (sun) {
    float f = (s.light * at) * inv;
    power = mk(f, f, f);
  } else {
    power = s.sky * (((4.0f * kPI) * at) * inv);
  }
}

__global__ void __launch_bounds__(128) ppm_emit_kernel(GridView g, SceneView s, uint32_t photons, uint32_t seed,
                                                       uint32_t pass, uint32_t cap, float4* __restrict__ pos,
                                                       float4* __restrict__ pw, float4* __restrict__ dir,
                                                       uint32_t* __restrict__ uid, uint32_t* __restrict__ count,
                                                       uint32_t* __restrict__ n_events, Counters cnt) {
  const uint32_t lane = threadIdx.x & 31u;
  bool alive = false, exhausted = false;
  uint32_t p = 0, events = 0;
  uint32_t started = 0, lookups = 0, cells = 0, deposits = 0;
  Rng rng{0u, 0u};
  f3 o = mk(0.f, 0.f, 0.f), d = o, power = o;
  while (true) {
    const bool need = !alive && !exhausted;
    const uint32_t want = __ballot_sync(0xffffffffu, need);
    if (want) {
      const uint32_t leader = __ffs(want) - 1;
      uint32_t base = 0;
      if (lane == leader) base = (uint32_t)atomicAdd(cnt.c + 4, (unsigned long long)__popc(want));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const uint32_t id = base + __popc(want & ((1u << lane) - 1u));
        if (id >= photons) {
          exhausted = true;
        } else {
          p = id;
          events = 0;
          ++started;
          ppm_start_photon(s, p, photons, seed, pass, rng, o, d, power);
          alive = true;
        }
      }
    }
    if (__all_sync(0xffffffffu, !alive && exhausted)) break;
    bool dep = false;
    if (alive) {
      float t;
      if (free_flight(g, s, o, d, rng, t, lookups, cells)) {
        o = along(o, d, t);
        dep = true;
      } else {
        alive = false;
        n_events[p] = events;
      }
    }
    const uint32_t m = __ballot_sync(0xffffffffu, dep);
    if (m) {
      const uint32_t leader = __ffs(m) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (dep) {
        const uint32_t slot = base + __popc(m & ((1u << lane) - 1u));
        if (slot < cap) {
          pos[slot] = make_float4(o.x, o.y, o.z, 0.0f);
          pw[slot] = make_float4(power.x, power.y, power.z, 0.0f);
          dir[slot] = make_float4(d.x, d.y, d.z, 0.0f);
          uid[slot] = p * kPpmMaxEvents + events;
        }
        ++events;
        ++deposits;
        power = power * s.albedo;
        if ((s.max_events && events >= s.max_events) || events >= kPpmMaxEvents) {
          alive = false;
          n_events[p] = events;
        } else {
          d = hg_sample(s.ph, d, rng, true);
        }
      }
    }
  }
  flush_counters(cnt, started, lookups, deposits, cells);
}

__device__ __forceinline__ uint32_t ppm_code(const SceneView& s, float4 p) {
  f3 e = s.b1 - s.b0;
  float qx = fminf(fmaxf(((p.x - s.b0.x) / e.x) * 1024.0f, 0.0f), 1023.0f);
  float qy = fminf(fmaxf(((p.y - s.b0.y) / e.y) * 1024.0f, 0.0f), 1023.0f);
  float qz = fminf(fmaxf(((p.z - s.b0.z) / e.z) * 1024.0f, 0.0f), 1023.0f);
  return (morton_expand10((uint32_t)qx) << 2) | (morton_expand10((uint32_t)qy) << 1) | morton_expand10((uint32_t)qz);
}

// Morton key of each photon in uid order: photon p's event e is number
// first[p] + e of them (first: the exclusive sums of the photons' deposits).
// A sort by uid gives the same order in four passes: 150 us for 3.2 M
// photons, the sums and this kernel 51 us.
__global__ void ppm_place_kernel(SceneView s, const float4* __restrict__ pos, const uint32_t* __restrict__ uid,
                                 const uint32_t* __restrict__ first, uint32_t n, uint32_t* __restrict__ codes,
                                 uint32_t* __restrict__ idx) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t u = uid[i], at = first[u / kPpmMaxEvents] + u % kPpmMaxEvents;
  codes[at] = ppm_code(s, pos[i]);
  idx[at] = i;
}

// Morton key of each photon in uid order (order = photons sorted by uid).
__global__ void ppm_keys_kernel(SceneView s, const float4* __restrict__ pos, const uint32_t* __restrict__ by_uid,
                                uint32_t n, uint32_t* __restrict__ codes, uint32_t* __restrict__ idx) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t ph = by_uid[i];
  codes[i] = ppm_code(s, pos[ph]);
  idx[i] = ph;
}

// ratio^(1/3) for ratio in [alpha, 1]: six Newton steps from 1 (converged
// to double precision for ratio >= 0.05), so host and device agree exactly.
__host__ __device__ __forceinline__ double ppm_cbrt_ratio(double r) {
  double y = 1.0;
  for (int i = 0; i < 6; ++i) y = y - (y * y * y - r) / (3.0 * y * y);
  return y;
}

// Photon powers and directions in the tree's leaf order: leaf i holds
// photon order[i] (the march, which visits every leaf's photon).
__global__ void ppm_leaf_order_kernel(const uint32_t* __restrict__ order, const float4* __restrict__ pw,
                                      const float4* __restrict__ dir, uint32_t n, float4* __restrict__ leaf_pw,
                                      float4* __restrict__ leaf_dir) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t ph = order[i];
    leaf_pw[i] = pw[ph];
    leaf_dir[i] = dir[ph];
  }
}

// Boxes over 8 consecutive photons of the leaf order (level 0), over 8 of
// those (level 1), ... up to the first level of at most 8; box i of a level
// at box[2 (first + i)] (low corner) and the next (high corner).
constexpr int kOctLevels = 10;  // 8^10 = 2^30 > 2^28 photons
struct OctLayout {
  uint32_t first[kOctLevels];  // the level's first box
  uint32_t count[kOctLevels];
  uint32_t total;
  int levels;
};
static OctLayout oct_layout(uint32_t photons) {
  OctLayout o{};
  uint32_t n = photons;
  do {
    n = (n + 7u) / 8u;
    o.count[o.levels] = n;
    o.first[o.levels++] = o.total;
    o.total += n;
  } while (n > 8u && o.levels < kOctLevels);
  return o;
}

// Three levels at a time, from the level `below` (its boxes, or the photons
// in their order, whose positions the first call also copies): a CTA's 512
// inputs make 64 boxes, 8 of the next level and one of the third.
constexpr int kOctThreads = 512;
__device__ __forceinline__ void oct_union(float4& lo, float4& hi) {  // of 8 neighbouring lanes
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
  }
}
__global__ void __launch_bounds__(kOctThreads) oct_kernel(const uint32_t* __restrict__ order,
                                                          const float4* __restrict__ pos,
                                                          float4* __restrict__ leaf_pos, float4* __restrict__ box,
                                                          OctLayout ol, int level, uint32_t n) {
  __shared__ float4 s_lo[kOctThreads / 8], s_hi[kOctThreads / 8];
  uint32_t i = blockIdx.x * kOctThreads + threadIdx.x;
  const float4 none_lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
  const float4 none_hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
  float4 lo = none_lo, hi = none_hi;
  if (i < n) {
    if (level == 0) {
      lo = hi = pos[order[i]];
      leaf_pos[i] = lo;
    } else {
      const float4* b = box + 2 * (size_t)(ol.first[level - 1] + i);
      lo = b[0];
      hi = b[1];
    }
  }
  uint32_t t = threadIdx.x;
#pragma unroll
  for (int k = 0; k < 3; ++k) {  // inputs of step k: threads t < 512 / 8^k
    oct_union(lo, hi);
    n = (n + 7u) / 8u;
    i >>= 3;
    const uint32_t width = kOctThreads >> (3 * k);
    if (t < width && (t & 7u) == 0u) {
      if (level + k < ol.levels && i < n) {
        float4* b = box + 2 * (size_t)(ol.first[level + k] + i);
        b[0] = lo;
        b[1] = hi;
      }
      s_lo[t >> 3] = lo;
      s_hi[t >> 3] = hi;
    }
    __syncthreads();
    lo = t < width / 8u ? s_lo[t] : none_lo;
    hi = t < width / 8u ? s_hi[t] : none_hi;
    i = (blockIdx.x * kOctThreads >> (3 * (k + 1))) + t;
    __syncthreads();
  }
}

// What the march reads: photon powers and directions in the tree's leaf
// order (leaf i holds photon order[i]), the leaf positions, and the internal
// nodes packed as (low corner, left child bits) (high corner, right child
// bits).  The gather: the leaf positions, the boxes of 8 above them, and the
// photons by their order.
struct PpmGatherView {
  const float4* pw;
  const float4* dir;
  const float4* leaf_lo;
  const float4* node_pk;
  const uint32_t* order;
  const float4* box;
  OctLayout ol;
  // pixels with a measurement point: their number, the points with sigma_t, the pixels
  uint32_t* points;
  float4* point;
  uint32_t* point_pix;
  int n;
  double* stats;  // per pixel: N, R, tau rgb, background rgb
  float alpha;
  uint32_t seed, pass;
};

__device__ __forceinline__ float box_dist2(f3 x, float4 lo, float4 hi) {
  float dx = fmaxf(fmaxf(lo.x - x.x, 0.0f), x.x - hi.x);
  float dy = fmaxf(fmaxf(lo.y - x.y, 0.0f), x.y - hi.y);
  float dz = fmaxf(fmaxf(lo.z - x.z, 0.0f), x.z - hi.z);
  return (dx * dx + dy * dy) + dz * dz;
}

// The progressive update of a pixel (FP64): M photons of summed contribution
// phi, background bg of the pass; then the current estimate, expressed as a
// sum over the passes so far.
__device__ __forceinline__ void ppm_update(const PpmGatherView& v, const SceneView& s, uint32_t pix, uint32_t M, f3 phi,
                                           f3 bg, double* __restrict__ sum) {
  double* st = v.stats + 8 * (size_t)pix;
  double N = st[0], R = st[1];
  double tau[3] = {st[2], st[3], st[4]};
  if (M > 0) {
    double am = (double)v.alpha * (double)M;
    double ratio = (N + am) / (N + (double)M);
    st[0] = N + am;
    st[1] = R * ppm_cbrt_ratio(ratio);
    tau[0] = (tau[0] + (double)phi.x) * ratio;
    tau[1] = (tau[1] + (double)phi.y) * ratio;
    tau[2] = (tau[2] + (double)phi.z) * ratio;
    st[2] = tau[0];
    st[3] = tau[1];
    st[4] = tau[2];
  }
  st[5] += (double)bg.x;
  st[6] += (double)bg.y;
  st[7] += (double)bg.z;
  double Rn = st[1];
  double vol = (4.0 / 3.0) * 3.14159265358979323846 * Rn * Rn * Rn;
  double a = (double)s.albedo / vol;
  double* o3 = sum + 3 * (size_t)pix;
  o3[0] = st[5] + a * tau[0];
  o3[1] = st[6] + a * tau[1];
  o3[2] = st[7] + a * tau[2];
}

// One thread a pixel: the camera ray's collision.  Pixels that have one leave
// their measurement point (with its sigma_t) in a list for the gather, the
// others are done.
__global__ void __launch_bounds__(128) ppm_camera_kernel(const __grid_constant__ GridView g,
                                                         const __grid_constant__ SceneView s,
                                                         const __grid_constant__ CamView cam,
                                                         const __grid_constant__ PassView pv,
                                                         const __grid_constant__ PpmGatherView v,
                                                         double* __restrict__ sum, Counters cnt) {
  const uint32_t lane = threadIdx.x & 31u, id = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = id < pv.cw * pv.ch;
  uint32_t lookups = 0, cells = 0, pix = 0;
  float4 point = make_float4(0.f, 0.f, 0.f, 0.f);
  bool query = false;
  if (in) {
    const uint32_t cy = id / pv.cw, cx = id - cy * pv.cw;
    const int x = (int)(pv.x0 + cx), y = (int)(pv.y0 + cy);
    pix = (uint32_t)y * pv.width + (uint32_t)x;
    f3 o, rd, bg = mk(0.f, 0.f, 0.f);
    camera_ray(cam, x, y, o, rd);
    float tmin, tmax;
    if (!slab(o, rd, s.b0, s.b1, tmin, tmax) || tmax < 0.0f || !(s.ds > 0.0f)) {
      bg = sky(s, rd);
    } else {
      f3 entry = along(o, rd, fmaxf(tmin, 0.0f));
      Rng rng = rng_pcg(v.seed ^ kPpmGatherSalt, pix, v.pass);
      float t;
      if (!free_flight(g, s, entry, rd, rng, t, lookups, cells)) {
        bg = sky(s, rd);
      } else if (v.n > 0) {
        const f3 xm = along(entry, rd, t);
        point = make_float4(xm.x, xm.y, xm.z, s.k_sigma * density_at(g, s, xm));
        ++lookups;
        query = true;
      }
    }
    if (!query) ppm_update(v, s, pix, 0u, mk(0.f, 0.f, 0.f), bg, sum);
  }
  const uint32_t m = __ballot_sync(0xffffffffu, query);
  uint32_t base = 0;
  if (m && lane == 0) base = atomicAdd(v.points, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (query) {
    const uint32_t at = base + __popc(m & ((1u << lane) - 1u));
    v.point[at] = point;
    v.point_pix[at] = pix;
  }
  flush_counters(cnt, in ? 1ull : 0ull, lookups, 0, cells);
}

// What a warp of the gather shares: its measurement points, the boxes of each
// level still to open, and the photons found but not yet evaluated.
constexpr uint32_t kPpmChunk = 8;  // measurement points a warp takes at a time
struct PpmWarp {
  float4 x[kPpmChunk];            // measurement point, radius^2
  float4 wo[kPpmChunk];           // direction toward the camera
  uint32_t open[kOctLevels][32];  // per level: boxes the sphere meets, in order
  uint8_t next[kOctLevels], count[kOctLevels];
  uint32_t leaf[64];              // ring of found photons (their leaves), and whose they are
  uint8_t of[64];
  float c[3][32];                 // contributions of a group of them
  uint32_t own[kPpmChunk];        // each point's photons in the group
};

// The photons within the radius of each measurement point.  A warp takes
// eight points from the list and looks them up one after the other: a round
// opens the next four boxes of a level and tests their 32 children (boxes or
// photons), one lane each; those that the sphere meets, in order, are opened
// before the level's other boxes.  A photon within the radius lies in boxes
// within the radius, so the boxes do not change what is found.  The photons
// found are evaluated (phase toward the camera times power) 32 at a time,
// whichever points they belong to, and a lane adds its point's in leaf order:
// the same floats as a walk that visits the leaves in order.
constexpr int kPpmGatherThreads = 128;

__global__ void __launch_bounds__(kPpmGatherThreads, 8)
    ppm_gather_kernel(const __grid_constant__ SceneView s, const __grid_constant__ CamView cam,
                      const __grid_constant__ PassView pv, const __grid_constant__ PpmGatherView v,
                      double* __restrict__ sum, Counters cnt, unsigned long long* __restrict__ tested) {
  __shared__ PpmWarp s_w[kPpmGatherThreads / 32];
  PpmWarp& w = s_w[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, slot = lane >> 3, oct = lane & 7u;
  const uint32_t n = (uint32_t)v.n, points = *v.points;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const int top = v.ol.levels - 1;
  uint32_t found_total = 0, cand = 0;
  for (uint32_t chunk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; chunk * kPpmChunk < points; chunk += warps) {
    const uint32_t here = min(kPpmChunk, points - chunk * kPpmChunk);
    uint32_t pix = 0, M = 0;
    float sigma_t = 0.0f;
    f3 phi = mk(0.f, 0.f, 0.f);
    if (lane < here) {
      const float4 p = v.point[chunk * kPpmChunk + lane];
      pix = v.point_pix[chunk * kPpmChunk + lane];
      sigma_t = p.w;
      const float r = (float)v.stats[8 * (size_t)pix + 1];
      f3 o, rd;
      camera_ray(cam, (int)(pix % pv.width), (int)(pix / pv.width), o, rd);
      w.x[lane] = make_float4(p.x, p.y, p.z, r * r);
      w.wo[lane] = make_float4(-rd.x, -rd.y, -rd.z, 0.f);
    }
    __syncwarp();
    uint32_t qh = 0, qn = 0;  // the ring's head and count, warp-uniform
    const auto evaluate = [&]() {  // a group of up to 32 photons, one lane each
      const uint32_t m = min(qn, 32u);
      if (lane < kPpmChunk) w.own[lane] = 0u;
      __syncwarp();
      f3 c = mk(0.f, 0.f, 0.f);
      uint32_t key = 32u + lane;
      if (lane < m) {
        const uint32_t at = (qh + lane) & 63u, ph = v.order[w.leaf[at]];
        key = w.of[at];
        const float4 d = v.dir[ph], pw = v.pw[ph], wo = w.wo[key];
        c = mk(pw.x, pw.y, pw.z) * hg_pdf(s.ph, dot(mk(d.x, d.y, d.z), mk(wo.x, wo.y, wo.z)));
      }
      const uint32_t peers = __match_any_sync(0xffffffffu, key);
      if (lane < m && (peers & lt) == 0u) w.own[key] = peers;
      w.c[0][lane] = c.x;
      w.c[1][lane] = c.y;
      w.c[2][lane] = c.z;
      __syncwarp();
      if (lane < kPpmChunk)
        for (uint32_t b = w.own[lane]; b; b &= b - 1u) {
          const int j = __ffs(b) - 1;
          phi = phi + mk(w.c[0][j], w.c[1][j], w.c[2][j]);
        }
      __syncwarp();
      qh += m;
      qn -= m;
    };
    for (uint32_t j = 0; j < here; ++j) {
      const float4 q = w.x[j];
      const f3 x = mk(q.x, q.y, q.z);
      // the top level's boxes (at most 8)
      int lev = top;
      uint32_t next = 0, count = 0;  // of the current level's open boxes
      {
        bool hit = false;
        if (lane < v.ol.count[top]) {
          const float4* b = v.box + 2 * (size_t)(v.ol.first[top] + lane);
          hit = box_dist2(x, b[0], b[1]) <= q.w;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        if (hit) w.open[top][__popc(m & lt)] = lane;
        count = __popc(m);
        __syncwarp();
      }
      while (true) {
        if (next >= count) {
          if (lev == top) break;
          ++lev;
          next = w.next[lev];
          count = w.count[lev];
          __syncwarp();  // before lane 0 writes them again
          continue;
        }
        if (lev > 0) {
          const uint32_t k = next + slot, child = k < count ? 8u * w.open[lev][k] + oct : 0xFFFFFFFFu;
          if (lane == 0) {
            w.next[lev] = (uint8_t)(next + 4u);
            w.count[lev] = (uint8_t)count;
          }
          --lev;
          bool hit = false;
          if (child < v.ol.count[lev]) {
            const float4* b = v.box + 2 * (size_t)(v.ol.first[lev] + child);
            hit = box_dist2(x, b[0], b[1]) <= q.w;
          }
          const uint32_t m = __ballot_sync(0xffffffffu, hit);
          if (hit) w.open[lev][__popc(m & lt)] = child;
          next = 0;
          count = __popc(m);
          __syncwarp();
        } else {
          // up to eight boxes of photons: two rounds' loads together
          uint32_t leaf[2];
          float4 p[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t k = next + 4u * i + slot;
            leaf[i] = k < count ? 8u * w.open[0][k] + oct : 0xFFFFFFFFu;
            if (leaf[i] < n) p[i] = v.leaf_lo[leaf[i]];
          }
          next += 8u;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            bool hit = false;
            if (leaf[i] < n) {
              ++cand;
              const f3 dq = mk(p[i].x, p[i].y, p[i].z) - x;
              hit = dot(dq, dq) <= q.w;
            }
            const uint32_t found = __ballot_sync(0xffffffffu, hit);
            if (hit) {
              const uint32_t at = (qh + qn + __popc(found & lt)) & 63u;
              w.leaf[at] = leaf[i];
              w.of[at] = (uint8_t)j;
            }
            qn += __popc(found);
            if (lane == j) M += __popc(found);
            if (qn >= 32u) evaluate();
          }
          __syncwarp();
        }
      }
    }
    if (qn) evaluate();
    if (lane < here) {
      phi = sigma_t > 0.0f ? mk(phi.x / sigma_t, phi.y / sigma_t, phi.z / sigma_t) : mk(0.f, 0.f, 0.f);
      ppm_update(v, s, pix, M, phi, mk(0.f, 0.f, 0.f), sum);
      found_total += M;
    }
    __syncwarp();  // the points are written again
  }
  flush_counters(cnt, 0ull, 0ull, found_total, 0ull);
  warp_count(tested, cand);
}

// ---------------------------------------------------------------------------
// The reference's estimate: a ray march with one global radius
// (PPM_PE.comp main :443-546, samplePhotonMap :304-375)
// ---------------------------------------------------------------------------
constexpr uint32_t kPpmMarchSalt = 0x5F356495u;
constexpr uint32_t kMarchCap = 1u << 20;  // march and ambient steps of one pixel
constexpr float kPI4_3 = kPI * 4.0f / 3.0f;

// samplePhotonMap at x: the photons within the global radius r, phase
// toward wo times power, in the tree's depth-first leaf order, over the
// sphere volume times sigma_s.  Like the reference it draws one random
// number when the sum is positive (its unused six-tap density average).
__device__ f3 march_photon_map(const PpmGatherView& v, const SceneView& s, f3 x, f3 wo, float r, float scatter,
                               Rng& rng, uint32_t& cand) {
  f3 phi = mk(0.f, 0.f, 0.f);
  if (scatter == 0.0f || v.n <= 0) return phi;
  const float r2 = r * r;
  uint32_t stack[kGatherStack];
  int sp = 0;
  uint32_t node = v.n == 1 ? kLeafBit : 0u;
  while (true) {
    if (node & kLeafBit) {
      const uint32_t lf = node & ~kLeafBit;
      ++cand;
      const float4 q = v.leaf_lo[lf];
      const f3 dq = mk(q.x, q.y, q.z) - x;
      if (dot(dq, dq) <= r2) {
        const float4 w = v.dir[lf], pw = v.pw[lf];
        const float f = hg_pdf(s.ph, dot(wo, mk(w.x, w.y, w.z)));
        phi = phi + mk(f * pw.x, f * pw.y, f * pw.z);
      }
    } else {
      const float4 lo = v.node_pk[2 * (size_t)node], hi = v.node_pk[2 * (size_t)node + 1];
      if (box_dist2(x, lo, hi) <= r2) {
        if (sp < kGatherStack) stack[sp++] = __float_as_uint(hi.w);
        node = __float_as_uint(lo.w);
        continue;
      }
    }
    if (sp == 0) break;
    node = stack[--sp];
  }
  if ((phi.x + phi.y) + phi.z <= 0.0f) return mk(0.f, 0.f, 0.f);
  rng_next(rng);
  const float den = ((kPI4_3 * r) * r2) * scatter;
  return mk(phi.x / den, phi.y / den, phi.z / den);
}

__global__ void __launch_bounds__(128) ppm_march_kernel(GridView g, SceneView s, CamView cam, SvView sv, PassView pv,
                                                        PpmGatherView v, float radius, float step, float amb_step,
                                                        double* __restrict__ sum, Counters cnt,
                                                        unsigned long long* __restrict__ tested) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t lookups = 0, cand = 0;
  if (id < pv.cw * pv.ch) {
    const uint32_t cy = id / pv.cw, cx = id - cy * pv.cw;
    const int x = (int)(pv.x0 + cx), y = (int)(pv.y0 + cy);
    const uint32_t pix = (uint32_t)y * pv.width + (uint32_t)x;
    Rng rng = s.rng_mode == 1 ? rng_xorshift(pv.seed * ((uint32_t)x + (uint32_t)y * pv.padded_w))
                              : rng_pcg(pv.seed ^ kPpmMarchSalt, pix, pv.pass);
    f3 pos, rd;
    camera_ray(cam, x, y, pos, rd);
    f3 L = sky(s, rd);
    float tmin, tmax;
    if (slab(pos, rd, s.b0, s.b1, tmin, tmax) && s.ds > 0.0f) {
      const f3 closest = along(pos, rd, tmin);
      pos = along(pos, rd, tmax - step * rng_next(rng));
      const float max_d = length(pos - closest);
      const f3 wo = -rd;
      float cur = 0.0f;
      for (uint32_t it = 0; cur < max_d && it < kMarchCap; ++it) {
        pos = pos - rd * step;
        cur = cur + step;
        const float ext = (density_at(g, s, pos) * s.ds) / s.bs;
        ++lookups;
        const float scatter = s.albedo * ext;
        const float pdf = hg_pdf(s.ph, dot(wo, s.sun));
        const float dl = (s.light * pdf) * sv_lookup(sv, pos);
        f3 direct = mk(dl, dl, dl);
        // ambient: the sky along a phase-sampled direction, attenuated by
        // the mean extinction of a coarse march to the box
        const f3 adir = hg_sample(s.ph, rd, rng, false);
        f3 ap = pos;
        float acc = 0.0f, adist = 0.0f;
        uint32_t n = 0;
        f3 amb = sky(s, adir);
        while (in_box(ap, s.b0, s.b1) && n < kMarchCap) {
          ap = ap + adir * amb_step;
          acc = acc + density_at(g, s, ap);
          adist = adist + amb_step;
          ++n;
        }
        lookups += n;
        if (n > 0) {
          acc = acc * (s.ds / s.bs);
          const float att = vexp(((-adist) * acc) / (float)n);
          amb = amb * att;
          if (amb.x > 0.0f) direct = direct + amb;
        }
        const f3 ind = march_photon_map(v, s, pos, wo, radius, scatter, rng, cand) * s.albedo;
        const float a = vexp((-step) * ext);
        const f3 src = direct + ind;
        L = L * a + mk((scatter * src.x) * step, (scatter * src.y) * step, (scatter * src.z) * step);
      }
    }
    write_result(pv, sum, pix, L);
  }
  flush_counters(cnt, id < pv.cw * pv.ch ? 1ull : 0ull, lookups, 0, 0);
  warp_count(tested, cand);
}

__global__ void ppm_init_stats_kernel(double* __restrict__ stats, size_t pixels, double r0) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pixels) return;
  double* st = stats + 8 * i;
  st[0] = 0.0;
  st[1] = r0;
  for (int k = 2; k < 8; ++k) st[k] = 0.0;
}

void ppm_free(vcr_ctx* ctx) {
  PpmState* st = ctx->ppm;
  if (!st) return;
  void* ptrs[] = {st->pos, st->pw, st->dir, st->uid, st->count, st->by_uid, st->uid_sorted, st->codes, st->idx,
                  st->codes_sorted, st->order, st->left, st->right, st->tree_clusters,
                  st->leaf_lo, st->leaf_hi, st->node_lo, st->node_hi, st->node_pk, st->leaf_pw, st->leaf_dir,
                  st->box, st->stats, st->iota, st->points, st->point, st->point_pix,
                  st->deposits, st->first, st->scan_sums};
  for (void* p : ptrs) cudaFree(p);
  probe_free(st->gather);
  delete st;
  ctx->ppm = nullptr;
}

__global__ void iota_kernel(uint32_t* __restrict__ v, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = i;
}

vcr_status ppm_setup(vcr_ctx* ctx, const vcr_ppm_params* p) {
  if (!p || p->photons == 0 || p->photons > (1u << 26) || p->capacity < 2 || p->capacity > (1u << 28) ||
      !(p->radius > 0.0f) || !(p->alpha > 0.0f && p->alpha <= 1.0f) || p->estimator > VCR_PPM_MARCH ||
      (p->estimator == VCR_PPM_MARCH && !(p->march_step > 0.0f && p->ambient_step > 0.0f)))
    return fail(ctx, VCR_ERR_INVALID,
                "ppm params: photons 1..2^26, capacity 2..2^28, radius > 0, alpha in (0,1], estimator "
                "VCR_PPM_GATHER or VCR_PPM_MARCH (with march_step > 0, ambient_step > 0)");
  if (!ctx->d_sum) return fail(ctx, VCR_ERR_STATE, "vcr_ppm_setup needs a frame (vcr_set_frame)");
  ppm_free(ctx);
  PpmState* st = new PpmState();
  ctx->ppm = st;
  st->prm = *p;
  size_t C = p->capacity;
#define VCR_ALLOC(ptr, bytes) VCR_CUDA(ctx, cudaMalloc(reinterpret_cast<void**>(&(ptr)), (bytes)))
  VCR_ALLOC(st->pos, C * 16);
  VCR_ALLOC(st->pw, C * 16);
  VCR_ALLOC(st->dir, C * 16);
  VCR_ALLOC(st->uid, C * 4);
  VCR_ALLOC(st->count, 4);
  VCR_ALLOC(st->by_uid, C * 4);
  VCR_ALLOC(st->uid_sorted, C * 4);
  VCR_ALLOC(st->codes, C * 4);
  VCR_ALLOC(st->idx, C * 4);
  VCR_ALLOC(st->codes_sorted, C * 4);
  VCR_ALLOC(st->order, C * 4);
  VCR_ALLOC(st->left, C * 4);
  VCR_ALLOC(st->right, C * 4);
  VCR_ALLOC(st->leaf_lo, C * 16);
  VCR_ALLOC(st->box, (size_t)oct_layout(p->capacity).total * 32 + 8 * 32);  // a visit reads 8 boxes
  if (p->estimator == VCR_PPM_MARCH) {  // the march walks the tree's boxes and leaf-order photons
    VCR_ALLOC(st->tree_clusters, lbvh_cluster_bytes(C));
    VCR_ALLOC(st->leaf_hi, C * 16);
    VCR_ALLOC(st->node_lo, C * 16);
    VCR_ALLOC(st->node_hi, C * 16);
    VCR_ALLOC(st->node_pk, 2 * C * 16);
    VCR_ALLOC(st->leaf_pw, C * 16);
    VCR_ALLOC(st->leaf_dir, C * 16);
  }
  VCR_ALLOC(st->iota, C * 4);
  VCR_ALLOC(st->deposits, (size_t)p->photons * 4);
  VCR_ALLOC(st->first, (size_t)p->photons * 4);
  VCR_ALLOC(st->scan_sums, 4096 * 4);
  size_t px = (size_t)ctx->width * ctx->height;
  VCR_ALLOC(st->stats, px * 8 * sizeof(double));
  VCR_ALLOC(st->points, 4);
  VCR_ALLOC(st->point, px * 16);
  VCR_ALLOC(st->point_pix, px * 4);
#undef VCR_ALLOC
  iota_kernel<<<(unsigned)((C + 255) / 256), 256>>>(st->iota, (uint32_t)C);
  ppm_init_stats_kernel<<<(unsigned)((px + 255) / 256), 256>>>(st->stats, px, (double)p->radius);
  VCR_CUDA(ctx, cudaGetLastError());
  st->pixels = px;
  return ensure_scratch(ctx, sort_scratch_bytes(p->capacity));
}

// RenderTechniquePPM::UpdateRadius (:302-312) for frame k + 1 (pass k):
// r_1 = R0, r_n = r_(n-1) ((n - 1 + alpha) / n)^0.33333, in float.
float ppm_global_radius(float r0, float alpha, uint32_t pass) {
  float r = r0;
  for (uint32_t n = 2; n <= pass + 1; ++n) r = r * std::pow(((float)(n - 1) + alpha) / (float)n, 0.33333f);
  return r;
}

static SvView sv_view(const vcr_ctx* ctx) {
  SvView sv{};
  sv.tex = ctx->d_sv;
  sv.n = (int)ctx->sv.voxel_axis_count;
  sv.b0 = mk(ctx->sv.bounds_min[0], ctx->sv.bounds_min[1], ctx->sv.bounds_min[2]);
  const f3 e = mk(ctx->sv.bounds_max[0], ctx->sv.bounds_max[1], ctx->sv.bounds_max[2]) - sv.b0;
  for (int i = 0; i < 9; ++i) sv.B[i] = ctx->sv.basis_change[i];
  sv.ext.x = (sv.B[0] * e.x + sv.B[1] * e.y) + sv.B[2] * e.z;
  sv.ext.y = (sv.B[3] * e.x + sv.B[4] * e.y) + sv.B[5] * e.z;
  sv.ext.z = (sv.B[6] * e.x + sv.B[7] * e.y) + sv.B[8] * e.z;
  return sv;
}

vcr_status ppm_pass_launch(vcr_ctx* ctx, const vcr_pass_desc* pass, cudaStream_t cs) {
  PpmState* st = ctx->ppm;
  if (!st) return fail(ctx, VCR_ERR_STATE, "vcr_ppm_pass needs vcr_ppm_setup");
  if (!ctx->has_grid || !ctx->has_cloud || !ctx->has_cam || !ctx->has_params || !ctx->d_sum)
    return fail(ctx, VCR_ERR_STATE, "vcr_ppm_pass needs a grid, cloud, camera, params and frame");
  if ((size_t)ctx->width * ctx->height != st->pixels)
    return fail(ctx, VCR_ERR_STATE, "the frame changed since vcr_ppm_setup");
  const bool march = st->prm.estimator == VCR_PPM_MARCH;
  if (ctx->params.rng_mode != VCR_RNG_PCG && !march)
    return fail(ctx, VCR_ERR_UNSUPPORTED, "the gather estimate uses PCG streams");
  if (march && !ctx->has_sv)
    return fail(ctx, VCR_ERR_STATE, "the march estimate needs vcr_shadow_volume_build first");
  PassView pv;
  vcr_status vs = make_pass_view(ctx, pass, pv);
  if (vs) return vs;
  if (pv.spp != 1 || (pv.flags & VCR_PASS_NO_ACCUMULATE))
    return fail(ctx, VCR_ERR_UNSUPPORTED, "photon mapping keeps its own statistics: spp 1, accumulating passes");
  GridView g = grid_view(ctx);
  SceneView s = scene_view(ctx);
  const uint32_t P = st->prm.photons, C = st->prm.capacity;
  Counters cnt{ctx->d_counters};
  VCR_CUDA(ctx, cudaMemsetAsync(ctx->d_counters, 0, 5 * sizeof(unsigned long long), cs));
  VCR_CUDA(ctx, cudaMemsetAsync(st->count, 0, 4, cs));
  {  // persistent: as many CTAs as fit, up to one lane a photon
    int per_sm = 0;
    VCR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ppm_emit_kernel, 128, 0));
    const uint32_t blocks = std::min<uint32_t>((uint32_t)(ctx->sm_count * std::max(per_sm, 1)), (P + 127) / 128);
    ppm_emit_kernel<<<blocks, 128, 0, cs>>>(g, s, P, pass->seed, pass->pass_index, C, st->pos, st->pw, st->dir,
                                            st->uid, st->count, st->deposits, cnt);
  }
  VCR_CUDA(ctx, cudaGetLastError());
  uint32_t total = 0;
  VCR_CUDA(ctx, cudaMemcpyAsync(&total, st->count, 4, cudaMemcpyDeviceToHost, cs));
  VCR_CUDA(ctx, cudaStreamSynchronize(cs));
  uint32_t n = std::min(total, C);
  st->photons_stored = n;
  st->dropped = total - n;
  // deterministic order: by (photon, event) uid, then stable along the Morton
  // curve
  if (total <= C && P <= kPlacePhotons) {
    VCR_CUDA(ctx, exclusive_scan_u32(st->deposits, st->first, P, st->scan_sums, nullptr, cs));
    if (n) {
      ppm_place_kernel<<<(n + 255) / 256, 256, 0, cs>>>(s, st->pos, st->uid, st->first, n, st->codes, st->idx);
      VCR_CUDA(ctx, cudaGetLastError());
    }
  } else {
    // more photons than the scan takes, or deposits that were dropped: a sort
    // by uid, over the bits a uid of this photon count uses
    uint32_t uid_bits = 1;
    while (uid_bits < 32 && (1ull << uid_bits) <= (uint64_t)P * kPpmMaxEvents + kPpmMaxEvents) ++uid_bits;
    VCR_CUDA(ctx, sort_pairs_enqueue(ctx->sm_count, ctx->d_error, ctx->d_scratch, st->uid, st->iota, st->uid_sorted,
                                     st->by_uid, n, 0, uid_bits, cs));
    if (n) {
      ppm_keys_kernel<<<(n + 255) / 256, 256, 0, cs>>>(s, st->pos, st->by_uid, n, st->codes, st->idx);
      VCR_CUDA(ctx, cudaGetLastError());
    }
  }
  VCR_CUDA(ctx, sort_pairs_enqueue(ctx->sm_count, ctx->d_error, ctx->d_scratch, st->codes, st->idx,
                                   st->codes_sorted, st->order, n, 0, 30, cs));
  PpmGatherView gv{};
  gv.leaf_lo = st->leaf_lo;
  gv.n = (int)n;
  gv.stats = st->stats;
  gv.alpha = st->prm.alpha;
  gv.seed = pass->seed;
  gv.pass = pass->pass_index;
  if (march) {
    vs = lbvh_build_refit(ctx, st->codes_sorted, st->order, st->pos, st->pos, (int)n, st->left, st->right,
                          st->tree_clusters, st->leaf_lo, st->leaf_hi, st->node_lo, st->node_hi, cs, st->node_pk);
    if (vs) return vs;
    if (n) {  // powers and directions in leaf order, read with the leaf's position
      ppm_leaf_order_kernel<<<ctx->sm_count * 8, 256, 0, cs>>>(st->order, st->pw, st->dir, n, st->leaf_pw,
                                                               st->leaf_dir);
      VCR_CUDA(ctx, cudaGetLastError());
    }
    gv.pw = st->leaf_pw;
    gv.dir = st->leaf_dir;
    gv.node_pk = st->node_pk;
  } else {  // the tree's topology (vcr_ppm_read's alone: 87 us of 3.2 M photons), and the boxes the gather descends
    vs = lbvh_build(ctx, st->codes_sorted, (int)n, st->left, st->right, cs);
    if (vs) return vs;
    gv.ol = oct_layout(n);
    uint32_t inputs = n;
    for (int level = 0; level < gv.ol.levels && n; level += 3) {
      oct_kernel<<<(inputs + kOctThreads - 1) / kOctThreads, kOctThreads, 0, cs>>>(st->order, st->pos, st->leaf_lo,
                                                                                 st->box, gv.ol, level, inputs);
      VCR_CUDA(ctx, cudaGetLastError());
      for (int k = 0; k < 3; ++k) inputs = (inputs + 7u) / 8u;
    }
    gv.pw = st->pw;
    gv.dir = st->dir;
    gv.order = st->order;
    gv.box = st->box;
    gv.points = st->points;
    gv.point = st->point;
    gv.point_pix = st->point_pix;
  }
  uint32_t pixels = pv.cw * pv.ch;
  vcr_status ps = probe_begin(ctx, st->gather, cs);
  if (ps) return ps;
  if (march) {
    ppm_march_kernel<<<(pixels + 127) / 128, 128, 0, cs>>>(
        g, s, cam_view(ctx->cam), sv_view(ctx), pv, gv, ppm_global_radius(st->prm.radius, st->prm.alpha, pv.pass),
        st->prm.march_step, st->prm.ambient_step, ctx->d_sum, cnt, st->gather.d_count);
  } else {
    VCR_CUDA(ctx, cudaMemsetAsync(st->points, 0, 4, cs));
    ppm_camera_kernel<<<(pixels + 127) / 128, 128, 0, cs>>>(g, s, cam_view(ctx->cam), pv, gv, ctx->d_sum, cnt);
    VCR_CUDA(ctx, cudaGetLastError());
    const uint32_t blocks = std::min<uint32_t>((uint32_t)ctx->sm_count * 8u,
                                               (pixels + kPpmGatherThreads / 32 * kPpmChunk - 1) /
                                                   (kPpmGatherThreads / 32 * kPpmChunk));
    ppm_gather_kernel<<<blocks, kPpmGatherThreads, 0, cs>>>(s, cam_view(ctx->cam), pv, gv, ctx->d_sum, cnt,
                                                            st->gather.d_count);
  }
  VCR_CUDA(ctx, cudaGetLastError());
  ps = probe_end(ctx, st->gather, cs);
  if (ps) return ps;
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, cs));
  // the sums hold the running estimate times the pass count
  ctx->passes += 1;
  ctx->samples += 1;
  return VCR_OK;
}

}  // namespace vcr

using namespace vcr;

extern "C" VCR_API vcr_status vcr_ppm_setup(vcr_ctx* ctx, const vcr_ppm_params* p) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  vcr_status st = ppm_setup(ctx, p);
  if (st) return st;
  VCR_CUDA(ctx, cudaDeviceSynchronize());
  return vcr_reset_accumulation(ctx);
}

extern "C" VCR_API vcr_status vcr_ppm_free(vcr_ctx* ctx) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaDeviceSynchronize();
  ppm_free(ctx);
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_ppm_pass(vcr_ctx* ctx, const vcr_pass_desc* pass, void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!pass) return fail(ctx, VCR_ERR_INVALID, "null pass");
  return ppm_pass_launch(ctx, pass, (cudaStream_t)stream);
}

extern "C" VCR_API vcr_status vcr_ppm_info(vcr_ctx* ctx, vcr_ppm_info_t* out) {
  if (!ctx || !out) return fail(ctx, VCR_ERR_INVALID, "null argument");
  if (!ctx->ppm) return fail(ctx, VCR_ERR_STATE, "no photon-map state");
  out->photons_stored = ctx->ppm->photons_stored;
  out->dropped = ctx->ppm->dropped;
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_ppm_gather_stats(vcr_ctx* ctx, uint64_t* count, float* ms) {
  if (!ctx || !count || !ms) return fail(ctx, VCR_ERR_INVALID, "null argument");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->ppm) return fail(ctx, VCR_ERR_STATE, "no photon-map state");
  return probe_read(ctx, ctx->ppm->gather, *count, *ms);
}

extern "C" VCR_API vcr_status vcr_ppm_read(vcr_ctx* ctx, vcr_ppm_buffer which, void* host, size_t bytes) {
  if (!ctx || !host) return fail(ctx, VCR_ERR_INVALID, "null argument");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  PpmState* st = ctx->ppm;
  if (!st) return fail(ctx, VCR_ERR_STATE, "no photon-map state");
  VCR_CUDA(ctx, cudaEventSynchronize(ctx->work_done));
  size_t n = st->photons_stored;
  const void* src = nullptr;
  size_t want = 0;
  switch (which) {
    case VCR_PPM_STATS: src = st->stats; want = st->pixels * 8 * sizeof(double); break;
    case VCR_PPM_POS: src = st->pos; want = n * 16; break;
    case VCR_PPM_POWER: src = st->pw; want = n * 16; break;
    case VCR_PPM_DIR: src = st->dir; want = n * 16; break;
    case VCR_PPM_UID: src = st->uid; want = n * 4; break;
    case VCR_PPM_ORDER: src = st->order; want = n * 4; break;
    case VCR_PPM_LEFT: src = st->left; want = n > 1 ? (n - 1) * 4 : 0; break;
    case VCR_PPM_RIGHT: src = st->right; want = n > 1 ? (n - 1) * 4 : 0; break;
    default: return fail(ctx, VCR_ERR_INVALID, "unknown photon buffer %d", (int)which);
  }
  if (bytes != want) return fail(ctx, VCR_ERR_INVALID, "photon buffer %d is %zu bytes, not %zu", (int)which, want, bytes);
  if (want) VCR_CUDA(ctx, cudaMemcpy(host, src, want, cudaMemcpyDeviceToHost));
  return VCR_OK;
}
