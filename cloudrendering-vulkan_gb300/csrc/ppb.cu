// Progressive photon beams: emission, beam segments, LBVH and its boxes,
// camera-ray beam gather.
//
// Reference: PPB_PT.comp (main :506-539, generateSunRay :396-430,
// generateAmbientRay :432-445, interactWithMedium :453-501,
// depositPhotonBeam :334-393), PPB_GenerateHierarchy.comp (:62-168),
// PPB_CalculateAABB.comp (:64-120), PPB_PE.comp (traverseTree :408-466,
// accumulateRadiance :362-404), RenderTechniquePPB.cpp (RecordDrawCommands
// :436-519, UpdateRadius :530-546).
//
// Differences from the shipped shaders, all deliberate (the reference's PPB
// never ran end to end): the sun-face choice has its missing `else`
// (PPB_PT.comp:413); beam capacity is enforced; the radius schedule is the
// intended product r_{k+1} = r_k (k + alpha) / (k + 1) (the shader host sums,
// RenderTechniquePPB.cpp:538-544); LBVH leaves keep their primitive and the
// split uses index-augmented prefixes for equal Morton codes; the boxes'
// maxima are of the upper bounds (PPB_CalculateAABB.comp:90 used bounds[0]); the
// estimator is the beam x beam 1D one (normalised biweight, 1/sin theta)
// with camera transmittance from 16 free-flight samples along the camera ray,
// the way each beam carries 16 along itself.
//
// Determinism: every photon writes its beams into its own slots; a prefix
// sum over photons places the segments, so the segment order, the sort and
// the BVH are identical from run to run.
#include "track.cuh"
#include "sort.cuh"
#include "ppb.cuh"

namespace vcr {

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* sums, uint32_t* d_total,
                               cudaStream_t st);

// ---------------------------------------------------------------------------
// emission
// ---------------------------------------------------------------------------
constexpr uint32_t kEmitWarps = 20;  // warps of the emission an SM holds
struct PpbEmitView {
  float* slots;         // [P * K * kSlotFloats]
  uint32_t* nbeams;     // [P]
  uint32_t* slot_segs;  // [P * K] segments of each beam
  uint32_t* slot_off;   // [P * K] exclusive prefix inside the photon
  uint32_t* photon_segs;// [P]
  float* reach;         // [P * K] the farthest of each beam's transmittance distances
  uint32_t photons, K, lanes;  // lanes: photons a warp
  float radius;
  uint32_t seed, pass;
};

__device__ __forceinline__ uint32_t segments_of(float len, float r) {
  float q = len / r;
  uint32_t n = q < (float)(kMaxSegPerBeam - 1) ? (uint32_t)q + 1u : kMaxSegPerBeam;
  return n;
}

// Origin on the box face the direction enters through, uniform over the
// projected area; returns the projected area.  Face weights are |d_a| times
// the face area (generateSunRay, PPB_PT.comp:396-430, with the else-if).
__device__ __forceinline__ float box_entry(const SceneView& s, f3 d, Rng& rng, f3& o) {
  f3 e = s.b1 - s.b0;
  float ax = fabsf(d.x) * (e.y * e.z), ay = fabsf(d.y) * (e.x * e.z), az = fabsf(d.z) * (e.x * e.y);
  float at = (ax + ay) + az;
  float sel = rng_next(rng) * at;
  float u = rng_next(rng), v = rng_next(rng);
  if (sel < ax) {
    o = mk(d.x > 0.0f ? s.b0.x : s.b1.x, s.b0.y + u * e.y, s.b0.z + v * e.z);
  } else if (sel < ax + ay) {
    o = mk(s.b0.x + u * e.x, d.y > 0.0f ? s.b0.y : s.b1.y, s.b0.z + v * e.z);
  } else {
    o = mk(s.b0.x + u * e.x, s.b0.y + v * e.y, d.z > 0.0f ? s.b0.z : s.b1.z);
  }
  return at;
}

// One lane a photon, v.lanes photons a warp.  The flights of all of a
// photon's beams (16 transmittance distances and the interaction each) follow
// one another in one loop over tentative collisions, so a lane whose flight
// ends early goes on with its next one.
__device__ __forceinline__ void emit_photons(const GridView& g, const SceneView& s, const PpbEmitView& v,
                                             const Counters& cnt) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t p = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * v.lanes + lane;
  const bool mine = lane < v.lanes && p < v.photons;
  uint32_t lookups = 0, cells = 0, events = 0, beams = 0;
  if (mine) {
    Rng rng = rng_pcg(v.seed ^ kEmitSalt, p, v.pass);
    f3 d, power;
    const float inv = 1.0f / ((float)v.photons * 0.5f);
    bool sun = rng_next(rng) < 0.5f;
    if (sun) {
      d = s.sun;
    } else {  // uniform direction for the constant sky
      float z = 1.0f - 2.0f * rng_next(rng);
      float sn, cs;
      vsincos2pi(rng_next(rng), &sn, &cs);
      float rr = sqrtf(fmaxf(0.0f, 1.0f - z * z));
      d = mk(rr * cs, rr * sn, z);
    }
    f3 o;
    float at = box_entry(s, d, rng, o);
    if (sun) {
      float f = (s.light * at) * inv;
      power = mk(f, f, f);
    } else {
      float f = ((4.0f * kPI) * at) * inv;
      power = s.sky * f;
    }
    uint32_t seg_total = 0;
    int flight = 0;  // of the beam: 16 distances, then the interaction
    bool beam = true, fresh = true;  // a beam begins; a flight begins
    float reach = 0.0f;
    float* sl = nullptr;
    Track tr;
    while (true) {
      if (beam) {
        float tmin, tmax;
        if (beams >= v.K || !slab(o, d, s.b0, s.b1, tmin, tmax) || !finite_pos(tmax)) break;
        // deposit a beam from o to the box exit (depositPhotonBeam, PPB_PT.comp:334-393)
        const size_t slot = (size_t)p * v.K + beams;
        sl = v.slots + slot * kSlotFloats;
        sl[0] = o.x; sl[1] = o.y; sl[2] = o.z;
        sl[3] = d.x; sl[4] = d.y; sl[5] = d.z;
        sl[6] = tmax;
        sl[7] = power.x; sl[8] = power.y; sl[9] = power.z;
        const uint32_t ns = segments_of(tmax, v.radius);
        v.slot_segs[slot] = ns;
        v.slot_off[slot] = seg_total;
        seg_total += ns;
        ++beams;
        reach = 0.0f;
        flight = 0;
        beam = false;
        fresh = true;
      }
      if (fresh) track_init(tr, g, s, g.majorants, o, d, cells);
      fresh = false;
      float tau = -vlog(rng_next(rng));
      bool ended = true, hit = false;
      if (track_walk(tr, g.majorants, s.k_sigma, tau, cells, 0xFFFFFFFFu) == kCandidate) {
        const float rho = density_at(g, s, along(o, d, tr.t));
        ++lookups;
        if (rng_next(rng) * tr.m < rho) hit = true;
        else ended = lookups + cells > kPathWorkCap;  // runaway guard (non-finite input)
      }
      if (!ended) continue;
      fresh = true;
      if (flight < kBeamDists) {
        const float e = hit ? tr.t : kEscaped;
        sl[10 + flight] = e;
        reach = fmaxf(reach, e);
        if (++flight == kBeamDists) v.reach[(size_t)p * v.K + beams - 1u] = reach;
        continue;
      }
      // next interaction (interactWithMedium, PPB_PT.comp:453-501)
      if (!hit) break;
      o = along(o, d, tr.t);
      ++events;
      power = power * s.albedo;
      if (s.max_events && events >= s.max_events) break;
      d = hg_sample(s.ph, d, rng, true);
      beam = true;
    }
    v.nbeams[p] = beams;
    v.photon_segs[p] = seg_total;
  }
  flush_counters(cnt, mine ? 1ull : 0ull, lookups, events, cells);
}

// Each beam split into equal segments of about the radius, with the 30-bit
// Morton code of each midpoint.  A warp takes a photon's beams one after the
// other, a lane a segment, so that the stores of neighbouring segments are
// neighbours (a thread a beam, each on its own run of segments: 431 us for
// 9.6 M segments, 127 so; their 44 bytes each take 62).
__global__ void __launch_bounds__(128) ppb_segment_kernel(
    SceneView s, const float* __restrict__ slots, const uint32_t* __restrict__ nbeams,
    const uint32_t* __restrict__ slot_segs, const uint32_t* __restrict__ slot_off,
    const uint32_t* __restrict__ photon_off, uint32_t photons, uint32_t K, float radius, uint32_t cap,
    float4* __restrict__ seg_a, float4* __restrict__ seg_b, uint32_t* __restrict__ seg_beam,
    uint32_t* __restrict__ codes, uint32_t* __restrict__ idx) {
  const uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
  if (p >= photons) return;  // warp-uniform
  const uint32_t beams = nbeams[p], first = photon_off[p];
  const f3 e = s.b1 - s.b0;
  for (uint32_t k = 0; k < beams; ++k) {
    const size_t slot = (size_t)p * K + k;
    const float* sl = slots + slot * kSlotFloats;
    const f3 o = mk(sl[0], sl[1], sl[2]), d = mk(sl[3], sl[4], sl[5]);
    const uint32_t ns = slot_segs[slot], base = first + slot_off[slot];
    const float segl = sl[6] / (float)ns;
    for (uint32_t j = lane; j < ns; j += 32u) {
      const uint32_t gi = base + j;
      if (gi >= cap) break;
      float off = (float)j * segl;
      f3 a = along(o, d, off);
      f3 b = along(a, d, segl);
      seg_a[gi] = make_float4(a.x, a.y, a.z, radius);
      seg_b[gi] = make_float4(b.x, b.y, b.z, off);
      seg_beam[gi] = (uint32_t)slot;
      f3 m = (a + b) * 0.5f;
      float qx = fminf(fmaxf(((m.x - s.b0.x) / e.x) * 1024.0f, 0.0f), 1023.0f);
      float qy = fminf(fmaxf(((m.y - s.b0.y) / e.y) * 1024.0f, 0.0f), 1023.0f);
      float qz = fminf(fmaxf(((m.z - s.b0.z) / e.z) * 1024.0f, 0.0f), 1023.0f);
      codes[gi] = (morton_expand10((uint32_t)qx) << 2) | (morton_expand10((uint32_t)qy) << 1) |
                  morton_expand10((uint32_t)qz);
      idx[gi] = gi;
    }
  }
}

// ---------------------------------------------------------------------------
// LBVH (Karras, "Maximizing Parallelism in the Construction of BVHs,
// Octrees, and k-d Trees", HPG 2012) over sorted 30-bit keys
// ---------------------------------------------------------------------------
__device__ __forceinline__ int lbvh_delta(const uint32_t* __restrict__ keys, int n, int i, int j) {
  if (j < 0 || j > n - 1) return -1;
  uint32_t a = keys[i], b = keys[j];
  if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
  return __clz(a ^ b);
}

// Children and leaf range [first, last] of internal node i.
__device__ __forceinline__ void lbvh_node(const uint32_t* __restrict__ keys, int n, int i, uint32_t& left,
                                          uint32_t& right, int& first, int& last) {
  int d = lbvh_delta(keys, n, i, i + 1) - lbvh_delta(keys, n, i, i - 1) > 0 ? 1 : -1;
  int dmin = lbvh_delta(keys, n, i, i - d);
  int lmax = 2;
  while (lbvh_delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (lbvh_delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = lbvh_delta(keys, n, i, j);
  int s = 0;
  for (int div = 2;; div <<= 1) {
    int t = (l + div - 1) / div;
    if (lbvh_delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    if (t == 1) break;
  }
  int gamma = i + s * d + (d < 0 ? -1 : 0);
  first = min(i, j);
  last = max(i, j);
  left = first == gamma ? (uint32_t)gamma | kLeafBit : (uint32_t)gamma;
  right = last == gamma + 1 ? (uint32_t)(gamma + 1) | kLeafBit : (uint32_t)(gamma + 1);
}

__global__ void lbvh_build_kernel(const uint32_t* __restrict__ keys, int n, uint32_t* __restrict__ left,
                                  uint32_t* __restrict__ right) {
  int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n - 1) return;
  uint32_t l, r;
  int first, last;
  lbvh_node(keys, n, i, l, r, first, last);
  left[i] = l;
  right[i] = r;
}

// Capped-cylinder AABB of a segment (calculateBeamBounds,
// PPB_CalculateAABB.comp:64-80): e = r sqrt(1 - a^2/|a|^2) per axis.
__device__ __forceinline__ void segment_box(float4 A, float4 B, float4& lo, float4& hi) {
  f3 pa = mk(A.x, A.y, A.z), pb = mk(B.x, B.y, B.z);
  float r = A.w;
  f3 a = pb - pa;
  float dd = dot(a, a);
  f3 e;
  if (dd > 0.0f) {
    e.x = r * sqrtf(fmaxf(0.0f, 1.0f - (a.x * a.x) / dd));
    e.y = r * sqrtf(fmaxf(0.0f, 1.0f - (a.y * a.y) / dd));
    e.z = r * sqrtf(fmaxf(0.0f, 1.0f - (a.z * a.z) / dd));
  } else {
    e = mk(r, r, r);
  }
  lo = make_float4(fminf(pa.x - e.x, pb.x - e.x), fminf(pa.y - e.y, pb.y - e.y), fminf(pa.z - e.z, pb.z - e.z), 0.f);
  hi = make_float4(fmaxf(pa.x + e.x, pb.x + e.x), fmaxf(pa.y + e.y, pb.y + e.y), fmaxf(pa.z + e.z, pb.z + e.z), 0.f);
}

// Boxes that cover `leaves` leaves, 2^log2_per_box leaves a box.
__device__ __forceinline__ uint32_t boxes_above(uint32_t leaves, uint32_t log2_per_box) {
  return (uint32_t)(((uint64_t)leaves + (1ull << log2_per_box) - 1ull) >> log2_per_box);
}

// Union of a warp's boxes, in every lane.
__device__ __forceinline__ void warp_box(float4& lo, float4& hi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
  }
}

// Which leaves can contribute to any pixel, 32 leaves (a cluster of the
// Morton order) a warp: a segment past the farthest of its beam's 16
// transmittance distances has none of them left, and where every majorant
// cell its box touches is zero the density at the closest point is; both
// factors of the estimate are then exactly 0.  A cell's majorant bounds the
// trilinear lookups inside it, unless the grid has texels below zero (or that
// are no number): then every leaf is live.  The points looked up lie within the radius of
// the segment; its box is grown by that, and by a hundredth of a cell against
// the rounding of the cell index.
struct LiveView {
  const uint32_t* order;
  const float4* seg_a;
  const float4* seg_b;
  const uint32_t* seg_beam;
  const float* reach;
  const float* maj;  // a pyramid level, or nullptr: every leaf is live
  int mnb[3];
  f3 b0, icell;
};
__device__ __forceinline__ bool segment_meets_density(const LiveView& v, float4 A, float4 B) {
  const float r = A.w;
  const float l[3] = {(fminf(A.x, B.x) - r - v.b0.x) * v.icell.x, (fminf(A.y, B.y) - r - v.b0.y) * v.icell.y,
                      (fminf(A.z, B.z) - r - v.b0.z) * v.icell.z};
  const float h[3] = {(fmaxf(A.x, B.x) + r - v.b0.x) * v.icell.x, (fmaxf(A.y, B.y) + r - v.b0.y) * v.icell.y,
                      (fmaxf(A.z, B.z) + r - v.b0.z) * v.icell.z};
  int c0[3], c1[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float top = (float)(v.mnb[a] - 1);
    c0[a] = (int)clampf(floorf(l[a] - 0.01f), 0.0f, top);
    c1[a] = (int)clampf(floorf(h[a] + 0.01f), 0.0f, top);
  }
  if ((c1[0] - c0[0] + 1) * (c1[1] - c0[1] + 1) * (c1[2] - c0[2] + 1) > 64) return true;  // not worth the walk
  for (int z = c0[2]; z <= c1[2]; ++z)
    for (int y = c0[1]; y <= c1[1]; ++y)
      for (int x = c0[0]; x <= c1[0]; ++x)
        if (!(__ldg(v.maj + ((size_t)x + (size_t)v.mnb[0] * ((size_t)y + (size_t)v.mnb[1] * z))) == 0.0f)) return true;
  return false;
}
__global__ void __launch_bounds__(256) ppb_live_kernel(const __grid_constant__ LiveView v, uint32_t n,
                                                       uint32_t* __restrict__ masks, uint32_t* __restrict__ counts) {
  const uint32_t lane = threadIdx.x & 31u, c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= (n + 31u) / 32u) return;  // warp-uniform
  const uint32_t i = c * 32u + lane;
  bool live = false;
  if (i < n) {
    const uint32_t sid = v.order[i];
    const float4 B = v.seg_b[sid];
    live = !v.maj || (v.reach[v.seg_beam[sid]] >= B.w && segment_meets_density(v, v.seg_a[sid], B));
  }
  const uint32_t m = __ballot_sync(0xffffffffu, live);
  if (lane == 0) {
    masks[c] = m;
    counts[c] = __popc(m);
  }
}

// The gather's leaves: the live ones in leaf order, segments and boxes side
// by side with their neighbours'.
struct GatherLeaves {
  float4* a;
  float4* b;
  float4* lo;
  float4* hi;
  uint32_t* beam;
};
__global__ void __launch_bounds__(256) ppb_compact_kernel(const uint32_t* __restrict__ order,
                                                          const float4* __restrict__ seg_a,
                                                          const float4* __restrict__ seg_b,
                                                          const uint32_t* __restrict__ seg_beam,
                                                          const float4* __restrict__ leaf_lo,
                                                          const float4* __restrict__ leaf_hi, uint32_t n,
                                                          const uint32_t* __restrict__ masks,
                                                          const uint32_t* __restrict__ offsets, GatherLeaves out) {
  const uint32_t lane = threadIdx.x & 31u, c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= (n + 31u) / 32u) return;  // warp-uniform
  const uint32_t m = masks[c];
  if (!((m >> lane) & 1u)) return;
  const uint32_t i = c * 32u + lane, sid = order[i], at = offsets[c] + __popc(m & ((1u << lane) - 1u));
  out.a[at] = seg_a[sid];
  out.b[at] = seg_b[sid];
  out.beam[at] = seg_beam[sid];
  out.lo[at] = leaf_lo[i];
  out.hi[at] = leaf_hi[i];
}

// A cluster level: box c over boxes [32 c, 32 c + 32) of the level below,
// which has ceil(*leaves / per_box) of them (the live leaves' count is on
// the device; the launch covers the most there can be).
__global__ void __launch_bounds__(256) ppb_cluster_kernel(const float4* __restrict__ lo_in,
                                                          const float4* __restrict__ hi_in,
                                                          const uint32_t* __restrict__ leaves, uint32_t log2_per_box,
                                                          float4* __restrict__ clo, float4* __restrict__ chi) {
  const uint32_t n = boxes_above(*leaves, log2_per_box);
  const uint32_t lane = threadIdx.x & 31u, c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= (n + 31u) / 32u) return;  // warp-uniform
  const uint32_t i = c * 32u + lane;
  float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
  if (i < n) {
    lo = lo_in[i];
    hi = hi_in[i];
  }
  warp_box(lo, hi);
  if (lane == 0) {
    clo[c] = lo;
    chi[c] = hi;
  }
}

// A node's box is the union of the leaf boxes of its range, whatever the tree
// between them looks like, so the nodes need not wait for one another: short
// ranges are read leaf by leaf, longer ones are taken by the whole warp from
// boxes over 32, 32^2 and 32^3 leaves (clusters).  Minima and maxima: the
// values of a walk from the leaves up.  9.6 M leaves, topology and boxes: 774 us,
// bound by the loads of the searches and ranges (1,254 us with the second
// child to arrive at a node, by an atomic counter, taking its box up).
constexpr int kLbvhLevels = 4;   // leaves, and three levels of clusters
constexpr int kLbvhShort = 32;   // leaves a lane reads itself (8 / 16 / 32 / 64: 700 / 619 / 606 / 630 us)
struct LbvhBoxes {
  const float4* lo[kLbvhLevels];
  const float4* hi[kLbvhLevels];
};

__device__ __forceinline__ void box_add(float4& lo, float4& hi, const float4 l, const float4 h) {
  lo.x = fminf(lo.x, l.x);
  lo.y = fminf(lo.y, l.y);
  lo.z = fminf(lo.z, l.z);
  hi.x = fmaxf(hi.x, h.x);
  hi.y = fmaxf(hi.y, h.y);
  hi.z = fmaxf(hi.z, h.z);
}

// Leaf boxes, and the clusters of 32 and of 1,024 of them.
__global__ void __launch_bounds__(1024) lbvh_leaf_kernel(const float4* __restrict__ seg_a,
                                                         const float4* __restrict__ seg_b,
                                                         const uint32_t* __restrict__ order, int n,
                                                         float4* __restrict__ leaf_lo, float4* __restrict__ leaf_hi,
                                                         float4* __restrict__ lo1, float4* __restrict__ hi1,
                                                         float4* __restrict__ lo2, float4* __restrict__ hi2) {
  __shared__ float4 s_lo[32], s_hi[32];
  const int g = (int)(blockIdx.x * blockDim.x + threadIdx.x), lane = (int)(threadIdx.x & 31u);
  const int warp = (int)(threadIdx.x >> 5);
  const uint32_t sid = order[min(g, n - 1)];  // past the end: the last leaf again
  float4 lo, hi;
  segment_box(seg_a[sid], seg_b[sid], lo, hi);
  if (g < n) {
    leaf_lo[g] = lo;
    leaf_hi[g] = hi;
  }
  if (!lo1) return;
  warp_box(lo, hi);
  if (lane == 0) {
    if (g < n) {
      lo1[g >> 5] = lo;
      hi1[g >> 5] = hi;
    }
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  if (warp != 0) return;
  lo = s_lo[lane];
  hi = s_hi[lane];
  warp_box(lo, hi);
  if (lane == 0) {
    lo2[blockIdx.x] = lo;
    hi2[blockIdx.x] = hi;
  }
}

// Clusters of 32 boxes, a warp each.
__global__ void lbvh_cluster_kernel(const float4* __restrict__ lo_in, const float4* __restrict__ hi_in, int n,
                                    float4* __restrict__ lo_out, float4* __restrict__ hi_out) {
  const int lane = (int)(threadIdx.x & 31u), c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (c * 32 >= n) return;  // warp-uniform
  const int i = min(c * 32 + lane, n - 1);
  float4 lo = lo_in[i], hi = hi_in[i];
  warp_box(lo, hi);
  if (lane == 0) {
    lo_out[c] = lo;
    hi_out[c] = hi;
  }
}

__global__ void __launch_bounds__(256) lbvh_node_kernel(const uint32_t* __restrict__ keys, int n, LbvhBoxes b,
                                                        uint32_t* __restrict__ left, uint32_t* __restrict__ right,
                                                        float4* __restrict__ node_lo, float4* __restrict__ node_hi,
                                                        float4* __restrict__ node_pk) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x), lane = (int)(threadIdx.x & 31u);
  const bool mine = i < n - 1;
  uint32_t l = 0, r = 0;
  int first = 0, last = 0;
  float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
  if (mine) {
    lbvh_node(keys, n, i, l, r, first, last);
    if (last - first < kLbvhShort) {
      lo = b.lo[0][first];
      hi = b.hi[0][first];
      for (int k = first + 1; k <= last; ++k) box_add(lo, hi, b.lo[0][k], b.hi[0][k]);
    }
  }
  for (uint32_t todo = __ballot_sync(0xffffffffu, mine && last - first >= kLbvhShort); todo; todo &= todo - 1u) {
    const int src = __ffs(todo) - 1;
    int p = __shfl_sync(0xffffffffu, first, src), e = __shfl_sync(0xffffffffu, last, src) + 1;
    // the range's ends at a level that a cluster of the next does not cover,
    // then the clusters between them
    float4 wl = b.lo[0][p], wh = b.hi[0][p];
#pragma unroll
    for (int level = 0; level < kLbvhLevels; ++level) {
      const float4* bl = b.lo[level];
      const float4* bh = b.hi[level];
      if (level + 1 == kLbvhLevels || e - p <= 64) {
        for (int k = p + lane; k < e; k += 32) box_add(wl, wh, bl[k], bh[k]);
        break;
      }
      const int up = (p + 31) & ~31, down = e & ~31;  // up <= down: the range is longer than 64
      if (p + lane < up) box_add(wl, wh, bl[p + lane], bh[p + lane]);
      if (down + lane < e) box_add(wl, wh, bl[down + lane], bh[down + lane]);
      p = up >> 5;
      e = down >> 5;
    }
    warp_box(wl, wh);
    if (lane == src) {
      lo = wl;
      hi = wh;
    }
  }
  if (!mine) return;
  left[i] = l;
  right[i] = r;
  node_lo[i] = make_float4(lo.x, lo.y, lo.z, 0.f);
  node_hi[i] = make_float4(hi.x, hi.y, hi.z, 0.f);
  if (node_pk) {  // box and children together: one 32-byte sector per node for the gathers
    node_pk[2 * (size_t)i] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(l));
    node_pk[2 * (size_t)i + 1] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(r));
  }
}

// ---------------------------------------------------------------------------
// gather
// ---------------------------------------------------------------------------
// Boxes over 32 consecutive leaves of the Morton order (level 0), over 32 of
// those (level 1), ... up to the first level of at most 32 boxes.
constexpr int kClusterLevels = 6;  // 32^6 leaves > 2^26
struct ClusterLayout {
  uint32_t count[kClusterLevels];  // boxes of each level when every leaf is live
  uint32_t first[kClusterLevels];  // the level's first box in the arrays
  int levels;
  uint32_t total;
};
static ClusterLayout cluster_layout(uint32_t leaves) {
  ClusterLayout c{};
  uint32_t n = leaves;
  do {
    n = (n + 31u) / 32u;
    c.count[c.levels] = n;
    c.first[c.levels++] = c.total;
    c.total += n;
  } while (n > 32u && c.levels < kClusterLevels);
  return c;
}

// What the gather reads: the live segments in the LBVH's leaf order, their
// boxes and the cluster boxes above them, the beam slots and each pixel's
// camera free flights.
struct PpbGatherView {
  GatherLeaves leaf;
  const uint32_t* n_live;
  const float* slots;
  const float4* cluster_lo;
  const float4* cluster_hi;
  float* cam_dist;
  ClusterLayout cl;
  float radius;
  bool every_pair;  // not without the pairs that give exactly 0: the grid may hold texels that are no number
  uint32_t seed, pass;
};

// Ray-box overlap of [t0, t1] with the slab interval.
__device__ __forceinline__ bool ray_box(f3 o, f3 inv, float t0, float t1, float4 lo, float4 hi) {
  float ax = (lo.x - o.x) * inv.x, bx = (hi.x - o.x) * inv.x;
  float ay = (lo.y - o.y) * inv.y, by = (hi.y - o.y) * inv.y;
  float az = (lo.z - o.z) * inv.z, bz = (hi.z - o.z) * inv.z;
  float tn = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fmaxf(fminf(az, bz), t0));
  float tf = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fminf(fmaxf(az, bz), t1));
  return tn <= tf;
}

// Camera ray of a crop pixel clipped to the cloud's box; false: it sees the
// sky alone.
__device__ __forceinline__ bool gather_ray(const SceneView& s, const CamView& cam, const PassView& pv, uint32_t cx,
                                           uint32_t cy, f3& o, f3& rd, float& t_in, float& t_out) {
  camera_ray(cam, (int)(pv.x0 + cx), (int)(pv.y0 + cy), o, rd);
  float tmin, tmax;
  if (!slab(o, rd, s.b0, s.b1, tmin, tmax) || tmax < 0.0f || !(s.ds > 0.0f)) return false;
  t_in = fmaxf(tmin, 0.0f);
  t_out = tmax;
  return true;
}

// Ascending order of 16 values (Batcher's bitonic sort, 80 exchanges): how
// many of them are at least x is then a binary search.
__device__ __forceinline__ void sort16(float (&v)[kBeamDists]) {
#pragma unroll
  for (int size = 2; size <= kBeamDists; size *= 2)
#pragma unroll
    for (int stride = size / 2; stride > 0; stride /= 2)
#pragma unroll
      for (int i = 0; i < kBeamDists; ++i) {
        const int j = i ^ stride;
        if (j < i) continue;
        const float a = fminf(v[i], v[j]), b = fmaxf(v[i], v[j]);
        v[i] = (i & size) == 0 ? a : b;
        v[j] = (i & size) == 0 ? b : a;
      }
}

// The 16 free flights along each pixel's camera ray, stored in ascending
// order.  One thread a pixel; its flights follow one another in one loop
// over tentative collisions, so lanes whose flights end early go on with
// their next one instead of waiting for the warp's longest.
__device__ __forceinline__ void camera_flights(const GridView& g, const SceneView& s, const CamView& cam,
                                               const PassView& pv, const PpbGatherView& v, const Counters& cnt,
                                               uint32_t id) {
  uint32_t lookups = 0, cells = 0;
  if (id < pv.cw * pv.ch) {
    const uint32_t cy = id / pv.cw, cx = id - cy * pv.cw;
    f3 o, rd;
    float t_in, t_out;
    if (gather_ray(s, cam, pv, cx, cy, o, rd, t_in, t_out)) {
      const uint32_t pix = (pv.y0 + cy) * pv.width + pv.x0 + cx;
      const f3 entry = along(o, rd, t_in);
      Rng rng = rng_pcg(v.seed ^ kGatherSalt, pix, v.pass);
      float d[kBeamDists];
#pragma unroll
      for (int i = 0; i < kBeamDists; ++i) d[i] = kEscaped;
      Track tr;
      int i = 0;
      bool fresh = true;
      while (i < kBeamDists) {
        if (fresh) track_init(tr, g, s, g.majorants, entry, rd, cells);
        fresh = false;
        float tau = -vlog(rng_next(rng));
        bool ended = true;
        float t = kEscaped;
        if (track_walk(tr, g.majorants, s.k_sigma, tau, cells, 0xFFFFFFFFu) == kCandidate) {
          const float rho = density_at(g, s, along(entry, rd, tr.t));
          ++lookups;
          if (rng_next(rng) * tr.m < rho) t = tr.t;
          else ended = lookups + cells > kPathWorkCap;  // runaway guard (non-finite input)
        }
        if (ended) {
#pragma unroll
          for (int k = 0; k < kBeamDists; ++k)
            if (k == i) d[k] = t;  // constant indices: the values stay in registers
          ++i;
          fresh = true;
        }
      }
      sort16(d);
      float4* out = reinterpret_cast<float4*>(v.cam_dist + (size_t)id * kBeamDists);
#pragma unroll
      for (int k = 0; k < kBeamDists / 4; ++k) out[k] = make_float4(d[4 * k], d[4 * k + 1], d[4 * k + 2], d[4 * k + 3]);
    }
  }
  flush_counters(cnt, 0ull, lookups, 0, cells);
}

// The two need nothing of each other: the camera's CTAs follow the emission's
// in one launch and fill the SMs as its longest photons end.  What bounds the
// emission is its longest photon, some thousand flights one after the other:
// the fewer photons share its warp, the shorter its turns, so a warp takes no
// more of them than put every warp on the SMs at once (20 an SM).  A whole
// pass, with one launch after the other and 32 photons a warp, and now:
// 1280x720, 60,741 photons 23.98 -> 23.54 ms; 640x360, 20,000 photons 5.62 ->
// 5.20; 160x90, 5,000 photons 2.35 -> 1.49 (12 warps an SM 1.58, 26 the first
// 23.93).  Photons from a cursor, 1 to 3 CTAs an SM: 25.6 to 23.9 ms, 2.72 the
// small one.
__global__ void __launch_bounds__(128) ppb_trace_kernel(const __grid_constant__ GridView g,
                                                        const __grid_constant__ SceneView s,
                                                        const __grid_constant__ PpbEmitView ev, uint32_t emit_blocks,
                                                        const __grid_constant__ CamView cam,
                                                        const __grid_constant__ PassView pv,
                                                        const __grid_constant__ PpbGatherView v, Counters cnt) {
  if (blockIdx.x < emit_blocks) emit_photons(g, s, ev, cnt);
  else camera_flights(g, s, cam, pv, v, cnt, (blockIdx.x - emit_blocks) * blockDim.x + threadIdx.x);
}

// A pixel tile's view of the scene, for finding the tile's pixels whose rays
// can meet a box.  A point p lies on the ray of the pixel (a, b) away from
// the tile's centre where A(p - apex) = a W(p - apex) and B(p - apex) = b
// W(p - apex), with the three linear forms of the camera's basis.  The box
// is grown by `grow` (1e-5 of the scene's coordinates: the rounding of the
// exact ray-box test) and the pixel range by `slack` (1/32 pixel and the
// forms' own rounding, which grows with the tile's distance from the image
// centre), so every pixel whose ray meets the box is in the range.
struct TileView {
  f3 apex, W, A, B;
  float grow, slack, far;
};
__device__ __forceinline__ TileView tile_view(const CamView& c, const SceneView& s, int x0, int y0, int w, int h) {
  const f3 F = c.fwd * c.near_plane, R = c.right * c.px, U = -(c.up * c.py);
  const f3 ru = cross(R, U), uf = cross(U, F), fr = cross(F, R);
  const float inv = 1.0f / dot(F, ru);
  TileView t;
  t.apex = c.pos;
  t.W = ru * inv;
  // pixels relative to the tile's centre
  const float ac = (float)(x0 - c.hw) + 0.5f * (float)(w - 1), bc = (float)(y0 - c.hh) + 0.5f * (float)(h - 1);
  t.A = uf * inv - t.W * ac;
  t.B = fr * inv - t.W * bc;
  t.far = INFINITY;
  t.slack = 0.03125f + 4e-6f * (fabsf(ac) + fabsf(bc));
  t.grow = 1e-5f * fmaxf(fmaxf(fmaxf(fabsf(c.pos.x), fabsf(c.pos.y)), fabsf(c.pos.z)),
                         fmaxf(fmaxf(fmaxf(fabsf(s.b0.x), fabsf(s.b0.y)), fabsf(s.b0.z)),
                               fmaxf(fmaxf(fabsf(s.b1.x), fabsf(s.b1.y)), fabsf(s.b1.z))));
  return t;
}
// The pixels (bit x + kW y) of the tile that the box may cover: all of them
// where the box reaches the camera's plane or a form is not finite.
template <uint32_t kW, uint32_t kH>
__device__ __forceinline__ uint32_t tile_pixels(const TileView& t, float4 lo, float4 hi) {
  const float cx = 0.5f * (lo.x + hi.x), cy = 0.5f * (lo.y + hi.y), cz = 0.5f * (lo.z + hi.z);
  const float ex = hi.x - cx + t.grow, ey = hi.y - cy + t.grow, ez = hi.z - cz + t.grow;
  const float rx = cx - t.apex.x, ry = cy - t.apex.y, rz = cz - t.apex.z;
  const float wc = fmaf(t.W.x, rx, fmaf(t.W.y, ry, t.W.z * rz));
  const float we = fmaf(fabsf(t.W.x), ex, fmaf(fabsf(t.W.y), ey, fabsf(t.W.z) * ez));
  const float ac = fmaf(t.A.x, rx, fmaf(t.A.y, ry, t.A.z * rz));
  const float ae = fmaf(fabsf(t.A.x), ex, fmaf(fabsf(t.A.y), ey, fabsf(t.A.z) * ez));
  const float bc = fmaf(t.B.x, rx, fmaf(t.B.y, ry, t.B.z * rz));
  const float be = fmaf(fabsf(t.B.x), ex, fmaf(fabsf(t.B.y), ey, fabsf(t.B.z) * ez));
  const float near_w = wc - we;
  if (near_w > t.far) return 0u;  // behind every ray's end
  constexpr uint32_t kRows = 1u | (kH > 1u ? 1u << kW : 0u) | (kH > 2u ? 1u << 2u * kW | 1u << 3u * kW : 0u);
  static_assert((kH == 1u || kH == 2u || kH == 4u) && kW * kH <= 32u, "tile shapes");
  constexpr uint32_t kAll = (kW * kH == 32u) ? 0xFFFFFFFFu : (1u << (kW * kH)) - 1u;
  const float in = 1.0f / near_w, fn = 1.0f / (wc + we);
  constexpr float hx = 0.5f * (float)(kW - 1u), hy = 0.5f * (float)(kH - 1u);
  const float a0 = ac - ae, a1 = ac + ae, b0 = bc - be, b1 = bc + be;
  const float x0 = ceilf(a0 * (a0 < 0.0f ? in : fn) + (hx - t.slack));
  const float x1 = floorf(a1 * (a1 > 0.0f ? in : fn) + (hx + t.slack));
  const float y0 = ceilf(b0 * (b0 < 0.0f ? in : fn) + (hy - t.slack));
  const float y1 = floorf(b1 * (b1 > 0.0f ? in : fn) + (hy + t.slack));
  if (!(near_w > 0.0f) || !(x0 == x0 && x1 == x1 && y0 == y0 && y1 == y1)) return kAll;
  if (x1 < 0.0f || y1 < 0.0f || x0 > (float)(kW - 1u) || y0 > (float)(kH - 1u) || x1 < x0 || y1 < y0) return 0u;
  const uint32_t xa = (uint32_t)fmaxf(x0, 0.0f), xb = (uint32_t)fminf(x1, (float)(kW - 1u));
  const uint32_t ya = (uint32_t)fmaxf(y0, 0.0f), yb = (uint32_t)fminf(y1, (float)(kH - 1u));
  const uint32_t row = (2u << xb) - (1u << xa);
  return row * ((kRows << (kW * ya)) & (kRows >> (kW * (kH - 1u - yb))));
}

// The pixels of the tile whose rays can come within r of the segment (start
// pa, unit direction bd, length segl) at a point between its ends: the pixels
// beam_closest can pass, and few others.  With the ray of pixel (a, b) from
// the apex along q = Q + a R + b U (not normalised) and w the apex relative to
// an end of the segment, the two lines are |q . (bd x w)| / |q x bd| apart,
// and their closest points lie past that end of the segment, along bd, where
// (q x w) . (q x bd) > 0.  The first is linear in (a, b) with the right-hand
// side bounded over the tile; the second is quadratic, its linear part at the
// tile's centre and a bound of the rest are used.  Margins over the rounding
// here and in beam_closest: there t and sb are off by some 1e-6 |w| / den,
// which is 1e-6 |w| |q|^2 of (q x w) . (q x bd) whatever den is (2e-5 allowed);
// distances by 1e-7 of the coordinates (grow: 1e-5).  A form that is not
// finite leaves the pixel in.
//
// A segment is about as long as its radius, so its box covers five times the
// pixels that pass.  1280x720, 60,741 photons: 2.31 G (leaf, pixel) pairs of
// the boxes' ranges become 0.64 G, of which 0.44 G pass; gather 25.1 -> 20.6 ms.
__device__ __forceinline__ float sum_abs(f3 v) { return (fabsf(v.x) + fabsf(v.y)) + fabsf(v.z); }
__device__ __forceinline__ f3 fcross(f3 a, f3 b) {
  return mk(fmaf(a.y, b.z, -(a.z * b.y)), fmaf(a.z, b.x, -(a.x * b.z)), fmaf(a.x, b.y, -(a.y * b.x)));
}
__device__ __forceinline__ float fdot(f3 a, f3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
template <uint32_t kW, uint32_t kH>
__device__ __forceinline__ uint32_t near_pixels(const CamView& cam, float grow, int x0, int y0, f3 pa, float r, f3 bd,
                                                float segl) {
  constexpr float hx = 0.5f * (float)(kW - 1u), hy = 0.5f * (float)(kH - 1u);
  const f3 R = cam.right * cam.px, U = -(cam.up * cam.py);
  const f3 Q = cam.fwd * cam.near_plane + R * ((float)(x0 - cam.hw) + hx) + U * ((float)(y0 - cam.hh) + hy);
  const f3 w = cam.pos - pa;
  const float qn = sum_abs(Q) + hx * sum_abs(R) + hy * sum_abs(U), wn = sum_abs(w) + segl;
  const f3 c = fcross(Q, bd), cR = fcross(R, bd), cU = fcross(U, bd), m = fcross(bd, w);
  const float dc = hx * sum_abs(cR) + hy * sum_abs(cU);  // q x bd is within this of c
  // |f| <= F
  const float fR = fdot(R, m), fU = fdot(U, m);
  const float F = fmaf(fmaf(r, 1.0001f, grow), fmaf(sqrtf(fdot(c, c)), 1.0001f, dc), 4e-6f * (qn * wn));
  // g0 >= -G0 at the start, g1 <= G1 at the end (w - segl bd)
  const f3 e = fcross(Q, w), eR = fcross(R, w), eU = fcross(U, w);
  const float g0R = fdot(eR, c) + fdot(e, cR), g0U = fdot(eU, c) + fdot(e, cU);
  const float round = (qn * qn) * fmaf(2e-5f, wn, grow);
  const float G0 = fmaf(1.01f * (hx * sum_abs(eR) + hy * sum_abs(eU)), dc, round);
  const float G1 = fmaf(1.01f * segl * dc, dc, G0);
  const float cc = fdot(c, c), g1R = fmaf(-2.0f * segl, fdot(c, cR), g0R), g1U = fmaf(-2.0f * segl, fdot(c, cU), g0U);
  float f = fmaf(-hx, fR, fmaf(-hy, fU, fdot(Q, m)));
  float g0 = fmaf(-hx, g0R, fmaf(-hy, g0U, fdot(e, c)));
  float g1 = fmaf(-hx, g1R, fmaf(-hy, g1U, fmaf(-segl, cc, fdot(e, c))));
  uint32_t pixels = 0;
#pragma unroll
  for (uint32_t y = 0; y < kH; ++y) {
    float a = f, b = g0, d = g1;
#pragma unroll
    for (uint32_t x = 0; x < kW; ++x) {
      if (!(fabsf(a) > F || b < -G0 || d > G1)) pixels |= 1u << (y * kW + x);
      a += fR;
      b += g0R;
      d += g1R;
    }
    f += fU;
    g0 += g0U;
    g1 += g1U;
  }
  return pixels;
}

// Beam x beam (1D) estimate of one segment (accumulateRadiance,
// PPB_PE.comp:362-404, with the fixes named at the top of the file), in two
// steps.  The first, for every (ray, segment) pair: the closest points of
// the camera ray (o, rd) and the segment (start pa, unit direction bd,
// length segl), at t along the ray and sb along the segment; false where the
// pair contributes nothing.  The distance is compared squared, with a margin
// over the rounding of the square root; the second step decides with it.
// (A segment of no length has no direction: the caller leaves it out.)
__device__ __forceinline__ float closest_limit(float r) {
  const float r2 = r * r;
  return r2 > 1e-30f ? r2 * 1.000001f : INFINITY;
}
__device__ __forceinline__ bool beam_closest(f3 pa, float limit, f3 bd, float segl, f3 o, f3 rd, float t_in,
                                             float t_far, float& t, float& sb) {
  float b = dot(rd, bd);
  float den = 1.0f - b * b;
  if (!(den > 1e-6f)) return false;  // (nearly) parallel
  f3 w0 = o - pa;
  float dw = dot(rd, w0), ew = dot(bd, w0);
  t = (b * ew - dw) / den;
  sb = ew + t * b;
  if (t < t_in || t > t_far || sb < 0.0f || sb > segl) return false;
  const f3 e = along(o, rd, t) - along(pa, bd, sb);
  return dot(e, e) < limit;
}

// The second step: the contribution of a pair the first one kept.  off: the
// segment's distance from its beam's origin; dist: the pixel's 16 ascending
// camera flights.
__device__ __forceinline__ f3 beam_contribution(const GridView& g, const SceneView& s, const float* __restrict__ sl,
                                                f3 pa, float r, f3 bd, float off, f3 o, f3 rd, float t_in, float t,
                                                float sb, const float* __restrict__ dist16, uint32_t& lookups) {
  f3 xc = along(o, rd, t);
  f3 xb = along(pa, bd, sb);
  float dist = length(xc - xb);
  if (!(dist < r)) return mk(0.f, 0.f, 0.f);
  float b = dot(rd, bd);
  float den = 1.0f - b * b;
  float u = dist / r;
  float q = 1.0f - u * u;
  float kern = ((0.9375f * q) * q) / r;  // 15/16 (1 - u^2)^2 / r
  float rho = density_at(g, s, xc);
  ++lookups;
  float sigma_s = (s.albedo * s.k_sigma) * rho;
  float sbeam = sb + off;  // distance from the beam origin
  const float2* s2 = reinterpret_cast<const float2*>(sl);  // slots are 112 B: 8-byte aligned pairs
  uint32_t cb = 0;
#pragma unroll
  for (int i = 0; i < kBeamDists / 2; ++i) {
    const float2 e = __ldg(s2 + 5 + i);
    cb += (e.x >= sbeam ? 1u : 0u) + (e.y >= sbeam ? 1u : 0u);
  }
  const float2 p0 = __ldg(s2 + 3), p12 = __ldg(s2 + 4);  // (length, power r), (power g, power b)
  float tc = t - t_in;
  uint32_t below = 0;  // camera flights shorter than tc
#pragma unroll
  for (int i = 0; i < kBeamDists / 4; ++i) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(dist16) + i);
    below += (q.x < tc ? 1u : 0u) + (q.y < tc ? 1u : 0u) + (q.z < tc ? 1u : 0u) + (q.w < tc ? 1u : 0u);
  }
  uint32_t cc = (uint32_t)kBeamDists - below;
  float tb = (float)cb * (1.0f / kBeamDists), tcam = (float)cc * (1.0f / kBeamDists);
  float ph = hg_pdf(s.ph, dot(bd, -rd));
  float w = ((((kern * sigma_s) * tcam) * tb) * ph) / sqrtf(den);
  return mk(p0.y * w, p12.x * w, p12.y * w);
}

// Per-pixel gather.  A warp takes a tile of P pixels and finds the leaves
// whose boxes its rays may meet by descending the 32-wide cluster boxes, one
// lane a box (coalesced loads; the box's pixel range in the tile by three
// linear forms).  The leaves it finds are queued and taken 32 at a time, one
// lane a leaf, for the direction and length of the segment and the pixels it
// can contribute to (near_pixels).  The (leaf, pixel) pairs of a batch are
// listed and tested 32 at a time, one lane a pair, for the closest points;
// those that pass are queued and evaluated 32 at a time, again one lane a
// pair, if the ray meets the leaf's box (the single-ray walk of the LBVH
// visits exactly the leaves whose boxes the ray meets, since a ray that meets
// a box meets every box around it).  A pixel adds its pairs' contributions in
// queue order, which is ascending leaf order: the order of the depth-first
// walk, so the sums are the same floats.
//
// Bound by the evaluation's instructions (divisions, square roots, gathers:
// half of all) and by what the L1 holds beside the warps' shared memory: the
// leaf slots keep only what the pair test reads (2 KB a warp instead of 4:
// 21.3 -> 19.9 ms with the camera's kernel; queuing the pairs' distances as
// well, 0.5 KB more, took 1.7 ms).  1280x720, 60,741 photons, 9.6 M segments of
// radius 0.015: 18.8 ms for 0.64 G pairs; 27.5 with a box test of each of 2.3 G
// pairs before the closest points; 71.9 with the leaves and ray ends that give
// exactly 0 (ppb_live_kernel, t_far); 129 with one lane a pixel for the closest
// points and the evaluation, 12 lanes of 32 at work.
constexpr int kGatherThreads = 128;
constexpr int kGatherWarps = kGatherThreads / 32;
constexpr int kLeafBatch = 64;  // leaf slots of a warp; a batch is tested once more than 32 are filled
__host__ __device__ constexpr uint32_t gather_w(int P) { return P == 32 ? 8u : P >= 8 ? 4u : 2u; }

template <int P>
struct __align__(16) GatherWarp {
  float4 leaf[kLeafBatch][2];  // (start, number of the leaf) (direction, length)
  float4 ray[P][3];            // (origin, t_in) (direction, t_far) (1 / direction, t_box)
  float2 q_t[64];              // queued pairs: (t, sb)
  uint32_t q_id[64];           // leaf slot << 5 | pixel
  uint32_t pixels[kLeafBatch]; // the tile's pixels a leaf's box may cover
  float c[3][32];              // contributions of a group of pairs
  uint32_t own[P];             // each pixel's pairs in the group
  uint2 cand[64];              // leaves whose boxes the tile meets: leaf, pixels of the box
  uint32_t mask[kClusterLevels], base[kClusterLevels];
  uint16_t pair[32 * P];       // the pairs of 32 leaves: leaf slot << 5 | pixel
};

template <int P>
__global__ void __launch_bounds__(kGatherThreads, 6) ppb_gather_kernel(const __grid_constant__ GridView g,
                                                                    const __grid_constant__ SceneView s,
                                                                    const __grid_constant__ CamView cam,
                                                                    const __grid_constant__ PassView pv,
                                                                    const __grid_constant__ PpbGatherView v,
                                                                    double* __restrict__ sum, Counters cnt,
                                                                    unsigned long long* __restrict__ evaluated) {
  constexpr uint32_t kW = gather_w(P), kH = (uint32_t)P / kW;
  extern __shared__ __align__(16) unsigned char s_raw[];
  GatherWarp<P>& w = reinterpret_cast<GatherWarp<P>*>(s_raw)[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t tiles_x = (pv.cw + kW - 1u) / kW;
  const uint32_t tx0 = (wid % tiles_x) * kW, ty0 = (wid / tiles_x) * kH;
  const uint32_t cx = tx0 + lane % kW, cy = ty0 + lane / kW;  // lane p < P owns pixel p of the tile
  const bool valid = lane < (uint32_t)P && cx < pv.cw && cy < pv.ch;
  uint32_t lookups = 0, segs = 0;
  f3 L = mk(0.f, 0.f, 0.f);
  bool trav = false;
  float depth = -INFINITY;  // W of the tile's farthest ray end
  const uint32_t n = *v.n_live;
  const float limit = closest_limit(v.radius);  // every segment's radius
  TileView view = tile_view(cam, s, (int)(pv.x0 + tx0), (int)(pv.y0 + ty0), (int)kW, (int)kH);
  if (valid) {
    f3 o, rd;
    float t_in, t_out;
    if (!gather_ray(s, cam, pv, cx, cy, o, rd, t_in, t_out)) {
      L = sky(s, rd);
    } else {
      const float4* d = reinterpret_cast<const float4*>(v.cam_dist + (size_t)(cy * pv.cw + cx) * kBeamDists);
      const float through = t_out - t_in;
      uint32_t cexit = 0;
#pragma unroll
      for (int i = 0; i < kBeamDists / 4; ++i) {
        const float4 q = d[i];
        cexit += (q.x >= through ? 1u : 0u) + (q.y >= through ? 1u : 0u) + (q.z >= through ? 1u : 0u) +
                 (q.w >= through ? 1u : 0u);
      }
      L = sky(s, rd) * ((float)cexit * (1.0f / kBeamDists));
      trav = n > 0u;
      // past the farthest flight (d[3].w) the camera transmittance is 0 (the
      // margin is over the rounding of t - t_in); the boxes are looked for
      // some radii further, as a closest point may lie before its box
      const float t_far = v.every_pair ? t_out : fminf(t_out, (t_in + d[kBeamDists / 4 - 1].w) * 1.0001f);
      const float t_box = fminf(t_out, t_far + 8.0f * v.radius);
      depth = fmaf(view.W.x, fmaf(t_box, rd.x, o.x - view.apex.x),
                   fmaf(view.W.y, fmaf(t_box, rd.y, o.y - view.apex.y),
                        view.W.z * fmaf(t_box, rd.z, o.z - view.apex.z)));
      w.ray[lane][0] = make_float4(o.x, o.y, o.z, t_in);
      w.ray[lane][1] = make_float4(rd.x, rd.y, rd.z, t_far);
      w.ray[lane][2] = make_float4(1.0f / rd.x, 1.0f / rd.y, 1.0f / rd.z, t_box);
    }
  }
  const uint32_t rays = __ballot_sync(0xffffffffu, trav);
  if (rays) {
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) depth = fmaxf(depth, __shfl_xor_sync(0xffffffffu, depth, k));
    view.far = depth;
    const int top = v.cl.levels - 1;
    int lev = top;  // warp-uniform, as are filled and the masks
    uint32_t filled = 0, ch = 0, cn = 0;  // leaf slots; first candidate and their number
    bool done = false;
    {
      bool see = false;
      if (lane < boxes_above(n, 5u * (uint32_t)v.cl.levels))
        see = (rays & tile_pixels<kW, kH>(view, v.cluster_lo[v.cl.first[top] + lane],
                                          v.cluster_hi[v.cl.first[top] + lane])) != 0u;
      const uint32_t m = __ballot_sync(0xffffffffu, see);
      if (lane == 0) {
        w.mask[top] = m;
        w.base[top] = 0u;
      }
      __syncwarp();
    }
    while (true) {
      // ---- descend until more than 32 leaves are at hand ----------------
      while (filled <= 32u && !(done && cn == 0u)) {
        if (cn >= 32u || done) {  // 32 candidates, a lane each: the segment's own pixels
          const uint32_t take = min(cn, 32u);
          float4 A = make_float4(0.f, 0.f, 0.f, 0.f), B = A;
          f3 ax = mk(0.f, 0.f, 0.f);
          float segl = 0.0f;
          uint32_t leaf = 0, covers = 0;
          if (lane < take) {
            const uint2 q = w.cand[(ch + lane) & 63u];
            leaf = q.x;
            A = v.leaf.a[leaf];
            B = v.leaf.b[leaf];
            ax = mk(B.x, B.y, B.z) - mk(A.x, A.y, A.z);
            segl = length(ax);
            ax = mk(ax.x / segl, ax.y / segl, ax.z / segl);
            covers = q.y & near_pixels<kW, kH>(cam, view.grow, (int)(pv.x0 + tx0), (int)(pv.y0 + ty0),
                                               mk(A.x, A.y, A.z), v.radius, ax, segl);
            if (!(segl > 0.0f)) covers = 0u;
          }
          const uint32_t cm = __ballot_sync(0xffffffffu, covers != 0u);
          if (covers) {
            const uint32_t at = filled + __popc(cm & lt);
            float4* f = w.leaf[at];
            f[0] = make_float4(A.x, A.y, A.z, __uint_as_float(leaf));
            f[1] = make_float4(ax.x, ax.y, ax.z, segl);
            w.pixels[at] = covers;
          }
          filled += __popc(cm);
          ch += take;
          cn -= take;
          __syncwarp();
          continue;
        }
        const uint32_t m = w.mask[lev];
        const uint32_t node = w.base[lev] + __ffs(m) - 1u;
        __syncwarp();
        if (m == 0u) {
          if (lev == top) done = true;
          else ++lev;
          continue;
        }
        if (lane == 0) w.mask[lev] = m & (m - 1u);
        const uint32_t child = node * 32u + lane;
        if (lev > 0) {
          --lev;
          bool see = false;
          if (child < boxes_above(n, 5u * (uint32_t)(lev + 1)))
            see = (rays & tile_pixels<kW, kH>(view, v.cluster_lo[v.cl.first[lev] + child],
                                              v.cluster_hi[v.cl.first[lev] + child])) != 0u;
          const uint32_t cm = __ballot_sync(0xffffffffu, see);
          if (lane == 0) {
            w.mask[lev] = cm;
            w.base[lev] = node * 32u;
          }
        } else {
          uint32_t covers = 0u;
          if (child < n) covers = rays & tile_pixels<kW, kH>(view, v.leaf.lo[child], v.leaf.hi[child]);
          const uint32_t cm = __ballot_sync(0xffffffffu, covers != 0u);
          if (covers) w.cand[(ch + cn + __popc(cm & lt)) & 63u] = make_uint2(child, covers);
          cn += __popc(cm);
        }
        __syncwarp();
      }
      if (filled == 0u) break;
      // ---- the batch's pairs, in leaf order -------------------------------
      uint32_t qh = 0, qn = 0;
      for (uint32_t half = 0; half < filled; half += 32u) {
        uint32_t pm = half + lane < filled ? w.pixels[half + lane] : 0u;
        uint32_t at = __popc(pm);  // inclusive prefix of the lanes' pair counts
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
          const uint32_t x = __shfl_up_sync(0xffffffffu, at, k);
          if (lane >= (uint32_t)k) at += x;
        }
        const uint32_t pairs = __shfl_sync(0xffffffffu, at, 31);
        at -= __popc(pm);
        segs += __popc(pm);
        for (; pm; pm &= pm - 1u) w.pair[at++] = (uint16_t)(((half + lane) << 5) | (__ffs(pm) - 1u));
        __syncwarp();
        for (uint32_t i = 0; i < pairs; i += 32u) {
          bool pass = false;
          float t = 0.0f, sb = 0.0f;
          uint32_t id = 0;
          if (i + lane < pairs) {
            id = w.pair[i + lane];
            const float4 r0 = w.ray[id & 31u][0], r1 = w.ray[id & 31u][1];
            const float4 a = w.leaf[id >> 5][0], d = w.leaf[id >> 5][1];
            pass = beam_closest(mk(a.x, a.y, a.z), limit, mk(d.x, d.y, d.z), d.w, mk(r0.x, r0.y, r0.z),
                                mk(r1.x, r1.y, r1.z), r0.w, r1.w, t, sb);
          }
          const uint32_t acc = __ballot_sync(0xffffffffu, pass);
          if (pass) {
            const uint32_t k = (qh + qn + __popc(acc & lt)) & 63u;
            w.q_id[k] = id;
            w.q_t[k] = make_float2(t, sb);
          }
          qn += __popc(acc);
          const bool last = i + 32u >= pairs && half + 32u >= filled;  // the leaf slots are refilled after it
          while (qn >= 32u || (last && qn)) {
            // ---- a group of up to 32 pairs, one lane each ------------------
            const uint32_t m = min(qn, 32u);
            if (lane < (uint32_t)P) w.own[lane] = 0u;
            __syncwarp();
            f3 c = mk(0.f, 0.f, 0.f);
            uint32_t key = 32u + lane;
            if (lane < m) {
              const uint32_t k = (qh + lane) & 63u, e = w.q_id[k];
              const float2 ts = w.q_t[k];
              key = e & 31u;
              const float4* f = w.leaf[e >> 5];
              const float4 a = f[0], d = f[1];
              const uint32_t leaf = __float_as_uint(a.w), beam = v.leaf.beam[leaf];
              const float4 lo = v.leaf.lo[leaf], hi = v.leaf.hi[leaf];
              const float off = v.leaf.b[leaf].w;
              const float4 r0 = w.ray[key][0], r1 = w.ray[key][1], r2 = w.ray[key][2];
              const f3 o = mk(r0.x, r0.y, r0.z);
              if (ray_box(o, mk(r2.x, r2.y, r2.z), r0.w, r2.w, lo, hi)) {
                const uint32_t pixel = (ty0 + key / kW) * pv.cw + tx0 + key % kW;
                c = beam_contribution(g, s, v.slots + (size_t)beam * kSlotFloats, mk(a.x, a.y, a.z), v.radius,
                                      mk(d.x, d.y, d.z), off, o, mk(r1.x, r1.y, r1.z), r0.w, ts.x, ts.y,
                                      v.cam_dist + (size_t)pixel * kBeamDists, lookups);
              } else {
                key = 32u + lane;  // no pair after all
              }
            }
            const uint32_t peers = __match_any_sync(0xffffffffu, key);
            if (key < 32u && (peers & lt) == 0u) w.own[key] = peers;  // a pixel: not a lane without a pair
            w.c[0][lane] = c.x;
            w.c[1][lane] = c.y;
            w.c[2][lane] = c.z;
            __syncwarp();
            if (lane < (uint32_t)P)
              for (uint32_t b = w.own[lane]; b; b &= b - 1u) {
                const int j = __ffs(b) - 1;
                L = L + mk(w.c[0][j], w.c[1][j], w.c[2][j]);
              }
            __syncwarp();
            qh += m;
            qn -= m;
          }
        }
        __syncwarp();
      }
      filled = 0;
      if (done && cn == 0u) break;
    }
  }
  if (valid) write_result(pv, sum, (pv.y0 + cy) * pv.width + pv.x0 + cx, L);
  flush_counters(cnt, valid ? 1ull : 0ull, lookups, 0, 0);
  warp_count(evaluated, segs);
}

template <int P>
static vcr_status gather_launch_t(vcr_ctx* ctx, const GridView& g, const SceneView& s, const CamView& cam,
                                  const PassView& pv, const PpbGatherView& gv, Counters cnt,
                                  unsigned long long* d_count, cudaStream_t st) {
  constexpr uint32_t kW = gather_w(P), kH = (uint32_t)P / kW;
  constexpr size_t smem = kGatherWarps * sizeof(GatherWarp<P>);
  static_assert(smem <= 48 * 1024, "static shared memory limit");
  const uint32_t tiles = ((pv.cw + kW - 1u) / kW) * ((pv.ch + kH - 1u) / kH);
  ppb_gather_kernel<P><<<(tiles + kGatherWarps - 1) / kGatherWarps, kGatherThreads, smem, st>>>(
      g, s, cam, pv, gv, ctx->d_sum, cnt, d_count);
  VCR_CUDA(ctx, cudaGetLastError());
  return VCR_OK;
}

// The largest tile that still gives the SMs 84 tiles each, three and a half
// rounds of the 24 warps an SM holds: a larger tile shares a leaf's set-up
// among more pixels, a smaller one leaves less work to the longest warp.
// Measured (ms with the camera's kernel, 256^3 cloud, twice and half that
// many tiles): 1280x720, 9.6 M segments 20.0 at 32 pixels, 21.0 at 16; 640x360,
// 3.1 M segments 3.57 / 3.27 / 4.46 at 32 / 16 / 8; 320x180 2.56 / 1.89 / 2.27
// at 16 / 8 / 4; 160x90 1.55 / 1.30 / 1.30 at 8 / 4 / 2.
static vcr_status gather_launch(vcr_ctx* ctx, const GridView& g, const SceneView& s, const CamView& cam,
                                const PassView& pv, const PpbGatherView& gv, Counters cnt,
                                unsigned long long* d_count, cudaStream_t st) {
  const auto fits = [&](uint32_t w, uint32_t h) {
    return (uint64_t)((pv.cw + w - 1u) / w) * ((pv.ch + h - 1u) / h) >= 84ull * (uint32_t)ctx->sm_count;
  };
  if (fits(8, 4)) return gather_launch_t<32>(ctx, g, s, cam, pv, gv, cnt, d_count, st);
  if (fits(4, 4)) return gather_launch_t<16>(ctx, g, s, cam, pv, gv, cnt, d_count, st);
  if (fits(4, 2)) return gather_launch_t<8>(ctx, g, s, cam, pv, gv, cnt, d_count, st);
  if (fits(2, 2)) return gather_launch_t<4>(ctx, g, s, cam, pv, gv, cnt, d_count, st);
  return gather_launch_t<2>(ctx, g, s, cam, pv, gv, cnt, d_count, st);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static void ppb_release(PpbState* st) {
  void* ptrs[] = {st->slots,      st->nbeams,      st->slot_segs,   st->slot_off,   st->photon_segs,
                  st->photon_off, st->scan_sums,   st->total,       st->seg_a,      st->seg_b,
                  st->leaf_a,     st->leaf_b,      st->leaf_beam,   st->cluster_lo, st->seg_beam,
                  st->codes,      st->idx,         st->codes_sorted, st->idx_sorted, st->left,
                  st->right,      st->tree_clusters, st->live_counts, st->leaf_lo,
                  st->leaf_hi,    st->node_lo,     st->node_hi,     st->cluster_hi, st->cam_dist,
                  st->live_lo,    st->live_hi,     st->live_mask,   st->live_off,   st->reach};
  for (void* p : ptrs) cudaFree(p);
  probe_free(st->gather);
}

void ppb_free(vcr_ctx* ctx) {
  if (!ctx->ppb) return;
  ppb_release(ctx->ppb);
  delete ctx->ppb;
  ctx->ppb = nullptr;
}

// r_k = r_0 prod_{i=1..k} (i + alpha) / (i + 1), in double (the intended
// per-pass reduction of RenderTechniquePPB::UpdateRadius).
float ppb_radius_at(float r0, float alpha, uint32_t pass) {
  double r = r0;
  for (uint32_t i = 1; i <= pass; ++i) r *= ((double)i + (double)alpha) / ((double)i + 1.0);
  return (float)r;
}

// Cluster boxes of a tree of n leaves.
static int lbvh_count(int n, int level) { return (int)(((int64_t)n + (1ll << (5 * level)) - 1) >> (5 * level)); }
size_t lbvh_cluster_bytes(size_t n) {
  size_t boxes = 0;
  for (int l = 1; l < kLbvhLevels; ++l) boxes += (n + ((size_t)1 << (5 * l)) - 1) >> (5 * l);
  return boxes * 2 * sizeof(float4);
}

vcr_status ppb_setup(vcr_ctx* ctx, const vcr_ppb_params* p) {
  if (!p || p->photons == 0 || p->photons > (1u << 21) || p->capacity < 2 || p->capacity > (1u << 26) ||
      !(p->radius > 0.0f) || !(p->alpha > 0.0f && p->alpha <= 1.0f))
    return fail(ctx, VCR_ERR_INVALID, "ppb params: photons 1..2^21, capacity 2..2^26, radius > 0, alpha in (0,1]");
  ppb_free(ctx);
  PpbState* st = new PpbState();
  ctx->ppb = st;
  st->prm = *p;
  uint32_t K = ctx->params.max_events ? std::min<uint32_t>(ctx->params.max_events + 1u, kMaxBeamsPerPhoton)
                                      : kMaxBeamsPerPhoton;
  st->K = K;
  size_t P = p->photons, C = p->capacity;
#define VCR_ALLOC(ptr, bytes) VCR_CUDA(ctx, cudaMalloc(reinterpret_cast<void**>(&(ptr)), (bytes)))
  VCR_ALLOC(st->slots, P * K * kSlotFloats * sizeof(float));
  VCR_ALLOC(st->nbeams, P * 4);
  VCR_ALLOC(st->slot_segs, P * K * 4);
  VCR_ALLOC(st->slot_off, P * K * 4);
  VCR_ALLOC(st->photon_segs, P * 4);
  VCR_ALLOC(st->photon_off, P * 4);
  VCR_ALLOC(st->scan_sums, 4096 * 4);
  VCR_ALLOC(st->total, 4);
  VCR_ALLOC(st->seg_a, C * sizeof(float4));
  VCR_ALLOC(st->seg_b, C * sizeof(float4));
  VCR_ALLOC(st->live_lo, C * sizeof(float4));
  VCR_ALLOC(st->live_hi, C * sizeof(float4));
  VCR_ALLOC(st->live_mask, (C + 31) / 32 * 4);
  VCR_ALLOC(st->live_off, (C + 31) / 32 * 4);
  VCR_ALLOC(st->reach, P * K * 4);
  VCR_ALLOC(st->cluster_lo, cluster_layout((uint32_t)C).total * sizeof(float4));
  VCR_ALLOC(st->cluster_hi, cluster_layout((uint32_t)C).total * sizeof(float4));
  VCR_ALLOC(st->leaf_a, C * sizeof(float4));
  VCR_ALLOC(st->leaf_b, C * sizeof(float4));
  VCR_ALLOC(st->leaf_beam, C * 4);
  VCR_ALLOC(st->seg_beam, C * 4);
  VCR_ALLOC(st->codes, C * 4);
  VCR_ALLOC(st->idx, C * 4);
  VCR_ALLOC(st->codes_sorted, C * 4);
  VCR_ALLOC(st->idx_sorted, C * 4);
  VCR_ALLOC(st->left, C * 4);
  VCR_ALLOC(st->right, C * 4);
  VCR_ALLOC(st->tree_clusters, lbvh_cluster_bytes(C));
  VCR_ALLOC(st->live_counts, (C + 31) / 32 * 4);
  VCR_ALLOC(st->leaf_lo, C * sizeof(float4));
  VCR_ALLOC(st->leaf_hi, C * sizeof(float4));
  VCR_ALLOC(st->node_lo, C * sizeof(float4));
  VCR_ALLOC(st->node_hi, C * sizeof(float4));
#undef VCR_ALLOC
  return ensure_scratch(ctx, sort_scratch_bytes(p->capacity));
}

vcr_status lbvh_build(vcr_ctx* ctx, const uint32_t* codes, int n, uint32_t* left, uint32_t* right, cudaStream_t st) {
  if (n <= 1) return VCR_OK;
  lbvh_build_kernel<<<(n - 1 + 255) / 256, 256, 0, st>>>(codes, n, left, right);
  VCR_CUDA(ctx, cudaGetLastError());
  return VCR_OK;
}

vcr_status lbvh_build_refit(vcr_ctx* ctx, const uint32_t* codes, const uint32_t* order, const float4* seg_a,
                            const float4* seg_b, int n, uint32_t* left, uint32_t* right, float4* clusters,
                            float4* leaf_lo, float4* leaf_hi, float4* node_lo, float4* node_hi, cudaStream_t st,
                            float4* node_pk) {
  if (n <= 0) return VCR_OK;
  LbvhBoxes b{};
  float4 *lo[kLbvhLevels] = {leaf_lo}, *hi[kLbvhLevels] = {leaf_hi};
  const bool clustered = n > 64;  // shorter ranges are read leaf by leaf
  for (int l = 1; l < kLbvhLevels && clustered; ++l) {
    lo[l] = clusters;
    hi[l] = clusters + lbvh_count(n, l);
    clusters += 2 * (size_t)lbvh_count(n, l);
  }
  lbvh_leaf_kernel<<<lbvh_count(n, 2), 1024, 0, st>>>(seg_a, seg_b, order, n, leaf_lo, leaf_hi, lo[1], hi[1], lo[2], hi[2]);
  VCR_CUDA(ctx, cudaGetLastError());
  if (clustered) {
    const int boxes = lbvh_count(n, 2);
    lbvh_cluster_kernel<<<(lbvh_count(n, 3) + 7) / 8, 256, 0, st>>>(lo[2], hi[2], boxes, lo[3], hi[3]);
    VCR_CUDA(ctx, cudaGetLastError());
  }
  if (n == 1) return VCR_OK;
  for (int l = 0; l < kLbvhLevels; ++l) {
    b.lo[l] = lo[l];
    b.hi[l] = hi[l];
  }
  lbvh_node_kernel<<<(n - 1 + 255) / 256, 256, 0, st>>>(codes, n, b, left, right, node_lo, node_hi, node_pk);
  VCR_CUDA(ctx, cudaGetLastError());
  return VCR_OK;
}

vcr_status ppb_pass_launch(vcr_ctx* ctx, const vcr_pass_desc* pass, cudaStream_t st_) {
  PpbState* st = ctx->ppb;
  if (!st) return fail(ctx, VCR_ERR_STATE, "vcr_ppb_pass needs vcr_ppb_setup");
  if (!ctx->has_grid || !ctx->has_cloud || !ctx->has_cam || !ctx->has_params || !ctx->d_sum)
    return fail(ctx, VCR_ERR_STATE, "vcr_ppb_pass needs a grid, cloud, camera, params and frame");
  if (ctx->params.rng_mode != VCR_RNG_PCG) return fail(ctx, VCR_ERR_UNSUPPORTED, "photon beams use PCG streams");
  PassView pv;
  vcr_status vs = make_pass_view(ctx, pass, pv);
  if (vs) return vs;
  if (pv.spp != 1) return fail(ctx, VCR_ERR_UNSUPPORTED, "photon beams gather one estimate per pixel and pass");
  GridView g = grid_view(ctx);
  SceneView s = scene_view(ctx);
  const uint32_t P = st->prm.photons, K = st->K, C = st->prm.capacity;
  st->radius = ppb_radius_at(st->prm.radius, st->prm.alpha, pass->pass_index);
  Counters cnt{ctx->d_counters};
  VCR_CUDA(ctx, cudaMemsetAsync(ctx->d_counters, 0, 5 * sizeof(unsigned long long), st_));
  PpbEmitView ev{st->slots, st->nbeams, st->slot_segs, st->slot_off, st->photon_segs, st->reach, P, K, 32u, st->radius,
                 pass->seed, pass->pass_index};
  const size_t pixels = (size_t)pv.cw * pv.ch;
  if (st->cam_pixels < pixels) {  // kept for the next pass; frames may grow after the set-up
    cudaFree(st->cam_dist);
    st->cam_dist = nullptr;
    st->cam_pixels = 0;
    VCR_CUDA(ctx, cudaMalloc(reinterpret_cast<void**>(&st->cam_dist), pixels * kBeamDists * sizeof(float)));
    st->cam_pixels = pixels;
  }
  PpbGatherView gv{};
  gv.cam_dist = st->cam_dist;
  gv.seed = pass->seed;
  gv.pass = pass->pass_index;
  while (ev.lanes > 1u && P <= (ev.lanes / 2u) * kEmitWarps * (uint32_t)ctx->sm_count) ev.lanes /= 2u;
  const uint32_t emit_blocks = (P + 4u * ev.lanes - 1u) / (4u * ev.lanes);
  ppb_trace_kernel<<<emit_blocks + (unsigned)((pixels + 127) / 128), 128, 0, st_>>>(g, s, ev, emit_blocks,
                                                                                   cam_view(ctx->cam), pv, gv, cnt);
  VCR_CUDA(ctx, cudaGetLastError());
  VCR_CUDA(ctx, exclusive_scan_u32(st->photon_segs, st->photon_off, P, st->scan_sums, st->total, st_));
  uint32_t total = 0;
  VCR_CUDA(ctx, cudaMemcpyAsync(&total, st->total, 4, cudaMemcpyDeviceToHost, st_));
  VCR_CUDA(ctx, cudaStreamSynchronize(st_));
  uint32_t n = std::min(total, C);
  st->segments = n;
  st->dropped = total - n;
  ppb_segment_kernel<<<(P + 3u) / 4u, 128, 0, st_>>>(
      s, st->slots, st->nbeams, st->slot_segs, st->slot_off, st->photon_off, P, K, st->radius, C, st->seg_a, st->seg_b,
      st->seg_beam, st->codes, st->idx);
  VCR_CUDA(ctx, cudaGetLastError());
  VCR_CUDA(ctx, sort_pairs_enqueue(ctx->sm_count, ctx->d_error, ctx->d_scratch, st->codes, st->idx, st->codes_sorted,
                                   st->idx_sorted, n, 0, 30, st_));
  // the tree and its boxes; the gather reads the leaf boxes, vcr_ppb_read the
  // nodes (606 us of 9.6 M leaves)
  vs = lbvh_build_refit(ctx, st->codes_sorted, st->idx_sorted, st->seg_a, st->seg_b, (int)n, st->left, st->right,
                        st->tree_clusters, st->leaf_lo, st->leaf_hi, st->node_lo, st->node_hi, st_, nullptr);
  if (vs) return vs;
  // the gather's leaves and clusters
  gv.cl = cluster_layout(n);
  gv.leaf = GatherLeaves{st->leaf_a, st->leaf_b, st->live_lo, st->live_hi, st->leaf_beam};
  gv.n_live = st->total;  // n's copy is on the host by now
  if (n) {
    LiveView lv{st->idx_sorted, st->seg_a, st->seg_b, st->seg_beam, st->reach, nullptr, {0, 0, 0}, s.b0, f3{}};
    // the finest majorant level whose cells are at least as wide as a
    // segment's box is thick: the box then spans few of them
    int level = 0;
    const f3 ext = s.b1 - s.b0;
    f3 cell{};
    for (;; ++level) {
      const float voxels = (float)(kBrick << level);
      cell = mk(ext.x / (float)ctx->gdesc.size[0] * voxels, ext.y / (float)ctx->gdesc.size[1] * voxels,
                ext.z / (float)ctx->gdesc.size[2] * voxels);
      if (level == 3 || std::min(cell.x, std::min(cell.y, cell.z)) >= 2.0f * st->radius) break;
    }
    if (!ctx->below_zero) lv.maj = ctx->d_majorants + ctx->moff[level];
    for (int a = 0; a < 3; ++a) lv.mnb[a] = ctx->mnb[level][a];
    lv.icell = mk(1.0f / cell.x, 1.0f / cell.y, 1.0f / cell.z);
    const uint32_t c = (n + 31u) / 32u;
    ppb_live_kernel<<<(c + 7u) / 8u, 256, 0, st_>>>(lv, n, st->live_mask, st->live_counts);
    VCR_CUDA(ctx, cudaGetLastError());
    VCR_CUDA(ctx, exclusive_scan_u32(st->live_counts, st->live_off, c, st->scan_sums, st->total, st_));
    ppb_compact_kernel<<<(c + 7u) / 8u, 256, 0, st_>>>(st->idx_sorted, st->seg_a, st->seg_b, st->seg_beam,
                                                       st->leaf_lo, st->leaf_hi, n, st->live_mask, st->live_off,
                                                       gv.leaf);
    VCR_CUDA(ctx, cudaGetLastError());
    for (int l = 0; l < gv.cl.levels; ++l) {
      const float4* lo_in = l ? st->cluster_lo + gv.cl.first[l - 1] : st->live_lo;
      const float4* hi_in = l ? st->cluster_hi + gv.cl.first[l - 1] : st->live_hi;
      ppb_cluster_kernel<<<(gv.cl.count[l] + 7u) / 8u, 256, 0, st_>>>(lo_in, hi_in, gv.n_live, 5u * (uint32_t)l,
                                                                     st->cluster_lo + gv.cl.first[l],
                                                                     st->cluster_hi + gv.cl.first[l]);
      VCR_CUDA(ctx, cudaGetLastError());
    }
  }
  gv.slots = st->slots;
  gv.radius = st->radius;
  gv.every_pair = ctx->below_zero;
  gv.cluster_lo = st->cluster_lo;
  gv.cluster_hi = st->cluster_hi;
  vcr_status ps = probe_begin(ctx, st->gather, st_);
  if (ps) return ps;
  vs = gather_launch(ctx, g, s, cam_view(ctx->cam), pv, gv, cnt, st->gather.d_count, st_);
  if (vs) return vs;
  ps = probe_end(ctx, st->gather, st_);
  if (ps) return ps;
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, st_));
  if (!(pv.flags & VCR_PASS_NO_ACCUMULATE)) {
    ctx->passes += 1;
    ctx->samples += 1;
  }
  return VCR_OK;
}

}  // namespace vcr

using namespace vcr;

extern "C" VCR_API vcr_status vcr_ppb_setup(vcr_ctx* ctx, const vcr_ppb_params* p) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  return ppb_setup(ctx, p);
}

extern "C" VCR_API vcr_status vcr_ppb_free(vcr_ctx* ctx) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaDeviceSynchronize();
  ppb_free(ctx);
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_ppb_pass(vcr_ctx* ctx, const vcr_pass_desc* pass, void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!pass) return fail(ctx, VCR_ERR_INVALID, "null pass");
  return ppb_pass_launch(ctx, pass, (cudaStream_t)stream);
}

extern "C" VCR_API vcr_status vcr_ppb_info(vcr_ctx* ctx, vcr_ppb_info_t* out) {
  if (!ctx || !out) return fail(ctx, VCR_ERR_INVALID, "null argument");
  if (!ctx->ppb) return fail(ctx, VCR_ERR_STATE, "no photon-beam state");
  out->segments = ctx->ppb->segments;
  out->dropped = ctx->ppb->dropped;
  out->radius = ctx->ppb->radius;
  out->beam_slots = ctx->ppb->K;
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_ppb_gather_stats(vcr_ctx* ctx, uint64_t* count, float* ms) {
  if (!ctx || !count || !ms) return fail(ctx, VCR_ERR_INVALID, "null argument");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->ppb) return fail(ctx, VCR_ERR_STATE, "no photon-beam state");
  return probe_read(ctx, ctx->ppb->gather, *count, *ms);
}

// Copies of the last pass's beam data (test and debug access).
extern "C" VCR_API vcr_status vcr_ppb_read(vcr_ctx* ctx, vcr_ppb_buffer which, void* host, size_t bytes) {
  if (!ctx || !host) return fail(ctx, VCR_ERR_INVALID, "null argument");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  PpbState* st = ctx->ppb;
  if (!st) return fail(ctx, VCR_ERR_STATE, "no photon-beam state");
  VCR_CUDA(ctx, cudaEventSynchronize(ctx->work_done));
  size_t n = st->segments, P = st->prm.photons, K = st->K;
  const void* src = nullptr;
  size_t want = 0;
  switch (which) {
    case VCR_PPB_SLOTS: src = st->slots; want = P * K * kSlotFloats * 4; break;
    case VCR_PPB_NBEAMS: src = st->nbeams; want = P * 4; break;
    case VCR_PPB_SEG_A: src = st->seg_a; want = n * 16; break;
    case VCR_PPB_SEG_B: src = st->seg_b; want = n * 16; break;
    case VCR_PPB_SEG_BEAM: src = st->seg_beam; want = n * 4; break;
    case VCR_PPB_CODES: src = st->codes; want = n * 4; break;
    case VCR_PPB_ORDER: src = st->idx_sorted; want = n * 4; break;
    case VCR_PPB_LEFT: src = st->left; want = n > 1 ? (n - 1) * 4 : 0; break;
    case VCR_PPB_RIGHT: src = st->right; want = n > 1 ? (n - 1) * 4 : 0; break;
    case VCR_PPB_NODE_LO: src = st->node_lo; want = n > 1 ? (n - 1) * 16 : 0; break;
    case VCR_PPB_NODE_HI: src = st->node_hi; want = n > 1 ? (n - 1) * 16 : 0; break;
    case VCR_PPB_LEAF_LO: src = st->leaf_lo; want = n * 16; break;
    case VCR_PPB_LEAF_HI: src = st->leaf_hi; want = n * 16; break;
    default: return fail(ctx, VCR_ERR_INVALID, "unknown beam buffer %d", (int)which);
  }
  if (bytes != want) return fail(ctx, VCR_ERR_INVALID, "beam buffer %d is %zu bytes, not %zu", (int)which, want, bytes);
  if (want) VCR_CUDA(ctx, cudaMemcpy(host, src, want, cudaMemcpyDeviceToHost));
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_lbvh_build(vcr_ctx* ctx, const uint32_t* d_sorted_codes, const uint32_t* d_order,
                                             const float* d_seg_a, const float* d_seg_b, uint32_t n,
                                             uint32_t* d_left, uint32_t* d_right, float* d_node_lo, float* d_node_hi,
                                             float* d_leaf_lo, float* d_leaf_hi, void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  if (n == 0) return VCR_OK;
  if (n > (1u << 30)) return fail(ctx, VCR_ERR_UNSUPPORTED, "LBVH of %u leaves", n);
  if (!d_sorted_codes || !d_order || !d_seg_a || !d_seg_b || !d_leaf_lo || !d_leaf_hi ||
      (n > 1 && (!d_left || !d_right || !d_node_lo || !d_node_hi)))
    return fail(ctx, VCR_ERR_INVALID, "null LBVH buffer");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  vcr_status vs = ensure_scratch(ctx, lbvh_cluster_bytes(n));
  if (vs) return vs;
  cudaStream_t st = (cudaStream_t)stream;
  vs = lbvh_build_refit(ctx, d_sorted_codes, d_order, reinterpret_cast<const float4*>(d_seg_a),
                        reinterpret_cast<const float4*>(d_seg_b), (int)n, d_left, d_right,
                        reinterpret_cast<float4*>(ctx->d_scratch), reinterpret_cast<float4*>(d_leaf_lo),
                        reinterpret_cast<float4*>(d_leaf_hi), reinterpret_cast<float4*>(d_node_lo),
                        reinterpret_cast<float4*>(d_node_hi), st, nullptr);
  if (vs) return vs;
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, st));
  return VCR_OK;
}
