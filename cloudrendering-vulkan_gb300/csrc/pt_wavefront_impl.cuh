// Persistent DDA wavefront path tracer: kernel and launcher.
//
// Same light transport as the per-pixel tracker (PathTracer.comp:366-425)
// with two changes of method the target asks for: free flights walk a
// pyramid level of per-cell majorants with a 3D DDA (instead of one global
// majorant, PathTracer.comp:338), and sun NEE is unbiased ratio tracking
// (instead of the shadow-volume lookup, PathTracer.comp:406-411).
//
// Schedule: persistent warps, each with a pool of paths in shared memory.
// A lane flies one path's ray at a time: a step of the loop draws an optical
// depth, walks a bounded number of majorant cells (resumable: the depth left
// over is kept) and takes at most one density lookup.  A flight lasts two
// lookups on average, and what stands between two flights - the light of a
// finished sun ray and a new direction, a finished path's result, a new
// camera path - is longer code that few lanes of a warp need at the same
// time: done in the lanes, those parts ran in nearly every step at 4 to 6 of
// 32 lanes.  So the lane stores the path's few words in the pool, queues it
// for its part and takes another path that is ready to fly; a part runs once
// 32 paths wait for it (or when nothing else can be done), and lanes take
// new rays (one DDA set-up site) once kRefillAt of them are without one.
// New paths come from a global cursor, 32 neighbouring ones at a time.  One
// launch may render several consecutive passes (pv.passes): its work items
// run through the passes in order, each with its pass's random streams, so
// that one pass's longest paths overlap the next one's.
//
// Bound by instruction issue (70 % of the slots, 17 of 32 lanes an
// instruction at 24 warps an SM; the cell walk at 10 lanes is what is left).
// 8 passes of 1920x1080 over the 1024x512x1024 cloud: 8.1 -> 4.8 ms, 12
// views of the 512^3 cloud: 12.3 -> 7.2 ms against one path a lane with
// those parts in the lanes (8 lanes an instruction).
//
// When the selected majorant level fits, one thread stages it into shared
// memory with a TMA bulk copy (cp.async.bulk + mbarrier) at CTA start and
// every DDA cell visit reads shared memory.  The arithmetic per path is
// identical to the oracle's sequential loop, so results are bit-exact with
// it.
//
// This file is compiled twice: by pt_wavefront.cu into namespace
// vcr::exact (device code built with -fmad=false and the library's own
// transcendental series, bit-exact with the oracle) and by
// pt_wavefront_fast.cu into vcr::fast (contracted multiply-adds and the
// hardware approximations of log, exp and sincos; selected by
// vcr_tuning.fast_math).  VCR_WF_NS names the namespace.
#include "track.cuh"
#include "nrc.cuh"

#ifndef VCR_WF_NS
#error "VCR_WF_NS must name the namespace of this instantiation"
#endif

namespace vcr {
namespace VCR_WF_NS {

// Where paths that end in the radiance cache leave their query.
struct NrcSink {
  NrcRecord* rec;
  uint32_t* count;
  uint32_t capacity;
};

constexpr uint32_t kMbarDrain = kDefaultStageWait;  // wait for a copy in flight after a timeout

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(phase)
      : "memory");
  return ok != 0u;
}

// Copy `bytes` (multiple of 16, 16-byte aligned both sides) from global to
// this CTA's shared memory with one bulk copy; every thread waits (at most
// `polls` polls).  Returns false (error word set) if the copy did not
// complete in time; the copy in flight is then waited for once more (at
// most kMbarDrain polls) so that no copy lands after the CTA stops using
// the buffer, and the caller copies the majorants with plain loads.
__device__ bool stage_to_smem(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint32_t polls, int* err) {
  const uint32_t b = smem_u32(bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(b)
                 : "memory");
  }
  bool ok = false;
  for (uint32_t i = 0; i < polls; ++i) {
    if (mbar_try_wait(b, 0u)) {
      ok = true;
      break;
    }
  }
  if (!ok) {
    atomicExch(err, 3);  // staging wait ran out; wait (bounded) once more for the copy in flight
    for (uint32_t i = 0; i < kMbarDrain; ++i)
      if (mbar_try_wait(b, 0u)) break;
  }
  return __syncthreads_and(ok ? 1 : 0) != 0;
}

// Rarely-taken bodies live out of line: the persistent loop then stays small
// enough for the instruction cache (a fully inlined loop stalled on
// instruction fetch more than on memory).  They take and return values, not
// references, so the path state they touch stays in registers instead of
// being stored to the stack around each call; the kernel's struct
// parameters are __grid_constant__ so that passing them by const reference
// does not copy them to local memory.
struct DirRng {
  f3 d;
  Rng r;
};
__device__ __noinline__ DirRng sample_direction(const Phase& ph, f3 dir, Rng rng) {
  DirRng o;
  o.d = hg_sample(ph, dir, rng, true);
  o.r = rng;
  return o;
}

__device__ __noinline__ f3 escape_radiance(const SceneView& s, f3 dir) { return sky(s, dir); }

// Camera ray of a path; returns false (L = sky) if it misses the cloud.
struct PathStart {
  f3 pos, dir, L;
  bool hit;
};
__device__ __noinline__ PathStart start_path(const CamView& cam, const SceneView& s, int x, int y) {
  PathStart o;
  camera_ray(cam, x, y, o.pos, o.dir);
  o.L = mk(0.f, 0.f, 0.f);
  float tmin, tmax;
  if (!slab(o.pos, o.dir, s.b0, s.b1, tmin, tmax) || tmax < 0.0f || !(s.ds > 0.0f)) {
    o.L = sky(s, o.dir);
    o.hit = false;
    return o;
  }
  o.pos = along(o.pos, o.dir, tmax < tmin ? tmax : tmin);
  o.hit = true;
  return o;
}

// A training path's radiance is final: turn the recorded radiance-before
// and throughput-before of each of its vertices into the target
// (L - L_before) / beta_before, walking the chain of its record slots.
__device__ __noinline__ void finish_training(const NrcTrainSink& ts, uint32_t slot, f3 L) {
  for (int i = 0; i < kNrcRecordEvents && slot != kNrcNoSlot; ++i) {
    NrcRecord* r = ts.rec + slot;
    float inv = 1.0f / __uint_as_float(r->pad[0]);
    r->w0 = (L.x - r->w0) * inv;
    r->w1 = (L.y - r->w1) * inv;
    r->w2 = (L.z - r->w2) * inv;
    slot = r->pad[1];
  }
}

// Append a training vertex; returns the slot (or the previous one if full).
__device__ __noinline__ uint32_t record_training(const NrcTrainSink& ts, const SceneView& s, f3 pos, f3 dir, f3 L,
                                                 float beta, uint32_t prev) {
  uint32_t q = atomicAdd(ts.count, 1u);
  if (q >= ts.capacity) return prev;
  NrcRecord r;
  r.px = pos.x; r.py = pos.y; r.pz = pos.z;
  r.vx = -dir.x; r.vy = -dir.y; r.vz = -dir.z;
  r.sx = s.sun.x; r.sy = s.sun.y; r.sz = s.sun.z;
  r.w0 = L.x; r.w1 = L.y; r.w2 = L.z;
  r.pix = kNrcNoSlot;
  r.pad[0] = __float_as_uint(beta);
  r.pad[1] = prev;
  r.pad[2] = 0u;
  ts.rec[q] = r;
  return q;
}

constexpr uint32_t kTrainPath = 0x80000000u;  // pid flag of a training path

// Russian roulette of a training path's continuation: survive with
// probability p and carry weight 1/p.
struct Roulette {
  Rng r;
  float beta;
  bool alive;
};
__device__ __noinline__ Roulette roulette(Rng rng, float p, float beta) {
  Roulette o;
  o.alive = rng_next(rng) < p;
  o.r = rng;
  o.beta = o.alive ? beta / p : beta;
  return o;
}
__device__ __forceinline__ bool roulette_survives(Rng& rng, float p, float& beta) {
  Roulette o = roulette(rng, p, beta);
  rng = o.r;
  beta = o.beta;
  return o.alive;
}

// 768 threads an SM: 80 registers a thread, nothing spilled.  (1,024 at 64:
// 74 B spilled and less L1 beside the pools, 15-20 % slower; 896 at 72 in
// CTAs of 128: the same time.)
constexpr int kThreadsPerSm = 768;
// Lanes without a ray before new ones are set up: 6 to 16 measured within 3 %.
constexpr uint32_t kRefillAt = 10;
// Training paths run to their end (64 events) where camera paths of the
// cached tracker end at their second event: each is a chain of dependent
// steps, and the longest decides when the launch ends.  So they come first,
// and apart from camera paths: one warp for every kTrainShare of them starts
// on the training paths' own cursor, takes 32 neighbouring ones at a time like
// any warp (a pool's worth in all, so that some of these warps find none
// left), and camera paths once the cursor has run out.  45 k of them with
// 4.1 M camera paths: 1,213 us a frame with mixed warps, 976 with a warp for
// every 8 to 32, 1,020 for every 96.
constexpr uint32_t kTrainShare = 16;
// The paths a warp holds, in shared memory: the lanes fly 32 of them at a
// time, the others wait in one of the queues.  With 80 the parts ran at 15
// to 19 lanes and the passes above took 3 % longer; 128 leave two CTAs an SM.
constexpr int kPool = 96;   // paths of a warp
constexpr int kRing = 128;  // a power of two of at least kPool entries
struct PathPool {
  float px[kPool], py[kPool], pz[kPool];  // the current vertex (or the entry point)
  float dx[kPool], dy[kPool], dz[kPool];  // direction of travel into / from it
  float L[kPool], beta[kPool];            // radiance (grey until the sky is added) and throughput
  float T[kPool];                         // transmittance of a finished sun ray; 1 / 0: escaped or not (finished paths)
  uint32_t rng[kPool], pix[kPool], pid[kPool], events[kPool], lookups[kPool], cells[kPool];
  unsigned long long totals[4];  // paths, lookups, events, cells of the warp's paths so far
  uint8_t ready[kRing];   // ring: a new flight along (dx, dy, dz) can start
  uint8_t shade[kRing];   // ring: the sun ray is done, a new direction is due
  uint8_t done[kPool];    // stack: finished paths
  uint8_t free_[kPool];   // stack: unused slots
};

__host__ __device__ constexpr uint32_t align16(uint32_t b) { return (b + 15u) & ~15u; }

enum : uint32_t { kIdle = 0, kAim = 1, kFly = 2 };  // lane: no path; path with a new ray to set up; in flight

// What the radiance cache takes from a path's collision at `o` (direction of
// travel d): a training path's record, or the query that ends a camera path
// at its nrc_events-th event (returns true).  The event is counted, and the
// throughput takes the albedo, when the path's sun ray is done.
__device__ __forceinline__ bool cache_vertex(PathPool& pool, uint32_t slot, const SceneView& s, const NrcSink& nq,
                                          const NrcTrainSink& ts, f3 o, f3 d) {
  const uint32_t ev = pool.events[slot] + 1u;
  const float beta = pool.beta[slot];
  if (pool.pid[slot] & kTrainPath) {
    if (ev <= (uint32_t)kNrcRecordEvents) {
      const float l = pool.L[slot];
      pool.pix[slot] = record_training(ts, s, o, d, mk(l, l, l), beta, pool.pix[slot]);
    }
    return false;
  }
  if (!s.nrc_events || ev != s.nrc_events) return false;
  pool.events[slot] = ev;
  const uint32_t q = atomicAdd(nq.count, 1u);
  if (q < nq.capacity) {  // it predicts what leaves this vertex
    NrcRecord rec;
    rec.px = o.x; rec.py = o.y; rec.pz = o.z;
    rec.vx = -d.x; rec.vy = -d.y; rec.vz = -d.z;
    rec.sx = s.sun.x; rec.sy = s.sun.y; rec.sz = s.sun.z;
    rec.w0 = beta; rec.w1 = beta; rec.w2 = beta;
    rec.pix = pool.pix[slot];
    rec.pad[0] = rec.pad[1] = rec.pad[2] = 0u;
    nq.rec[q] = rec;
  }
  return true;
}

// Work items [0, ts.paths) are training paths (their pid carries kTrainPath
// and their pix the slot of their last record); the pass's camera paths
// follow.  kBatch: the camera paths are those of bt's views (pid holds the
// view, whose sun the path uses), the view table sits in shared memory
// after the staged majorants, and the pass index adds *bt.pass_ctr (so a
// replayed graph renders consecutive passes).  kCache: the launch has training
// paths, or its camera paths end in cache queries.  kCorners: the grid has
// corner blocks.
template <int kThreads, bool kStage, bool kBatch, bool kCache, bool kCorners>
__global__ void __launch_bounds__(kThreads, kThreadsPerSm / kThreads)
    pt_wavefront_kernel(const __grid_constant__ GridView g, const __grid_constant__ SceneView s,
                        const __grid_constant__ CamView cam, const __grid_constant__ PassView pv,
                        double* __restrict__ sum, uint32_t* __restrict__ stats, Counters cnt, uint32_t total,
                        uint32_t dda_steps, uint32_t cap, uint32_t train_warps, uint32_t maj_bytes,
                        uint32_t stage_polls, const __grid_constant__ NrcSink nq,
                        const __grid_constant__ NrcTrainSink ts, const __grid_constant__ BatchSink bt,
                        int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ __align__(8) uint64_t s_bar;
  float* s_maj = reinterpret_cast<float*>(s_raw);
  const float* maj = kStage ? s_maj : g.majorants;
  if (kStage && !stage_to_smem(s_maj, g.majorants, maj_bytes, &s_bar, stage_polls, err)) {
    for (uint32_t i = threadIdx.x; i < maj_bytes / 4u; i += blockDim.x) s_maj[i] = __ldg(g.majorants + i);
    __syncthreads();
  }
  unsigned char* s_next = s_raw + (kStage ? align16(maj_bytes) : 0u);
  BatchView* s_views = reinterpret_cast<BatchView*>(s_next);
  uint32_t pass = pv.pass;
  if (kBatch) {
    const uint2* src = reinterpret_cast<const uint2*>(bt.views);
    uint2* dst = reinterpret_cast<uint2*>(s_views);
    const uint32_t words = bt.count * (uint32_t)(sizeof(BatchView) / 8);
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    pass += *bt.pass_ctr;
    s_next += bt.count * sizeof(BatchView);
    __syncthreads();
  }
  PathPool& pool = reinterpret_cast<PathPool*>(s_next)[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t per_pass = pv.cw * pv.ch * pv.spp;  // camera paths of one pass
  const float k = s.k_sigma;
  const f3 lsun0 = -s.sun;
  // warp-uniform queue state
  const uint32_t slots = cap < 32u ? cap : (uint32_t)kPool;
  uint32_t n_free = slots, n_done = 0, n_ready = 0, h_ready = 0, n_shade = 0, h_shade = 0;
  bool exhausted = false;
  const uint32_t n_train = kCache ? ts.paths : 0u;
  bool serving = kCache && (threadIdx.x >> 5) * gridDim.x + blockIdx.x < train_warps;
  for (uint32_t i = lane; i < (uint32_t)kPool; i += 32u) pool.free_[i] = (uint8_t)i;
  if (lane < 4u) pool.totals[lane] = 0ull;
  __syncwarp();
  // the lane's flight
  uint32_t mode = kIdle, slot = 0;
  bool sun_ray = false, walking = false;
  float tau = 0.0f, T = 1.0f;
  uint32_t lookups = 0, cells = 0;
  uint32_t rs = 0;  // the path's random state
  f3 o = mk(0.f, 0.f, 0.f), rd = mk(0.f, 0.f, 1.f);
  Track tr;

  while (true) {
    const uint32_t flying = __ballot_sync(0xffffffffu, mode == kFly);
    // (with no new paths to come only what waits is worth a look, at once)
    const bool look = exhausted ? n_ready + n_shade != 0u || n_done >= 32u || __any_sync(0xffffffffu, mode == kAim)
                                : 32u - __popc(flying) >= kRefillAt;
    if (flying == 0u || look) {
      // ---- hand the lanes without a path one that waits -------------------
      const uint32_t idle = __ballot_sync(0xffffffffu, mode == kIdle);
      const uint32_t n_idle = __popc(idle);
      while (n_ready < n_idle || n_done >= 32u) {
        if (n_done >= 32u || (n_done && n_ready == 0u && n_shade == 0u && n_free < slots && (exhausted || n_free == 0u))) {
          // ---- finished paths: results --------------------------------------
          const uint32_t m = min(n_done, 32u);
          uint32_t ev = 0, lk = 0, ce = 0;
          if (lane < m) {
            const uint32_t q = pool.done[n_done - 1u - lane];
            const uint32_t pid = pool.pid[q], pix = pool.pix[q];
            ev = pool.events[q];
            lk = pool.lookups[q];
            ce = pool.cells[q];
            const float l = pool.L[q];
            f3 L = mk(l, l, l);
            if (pool.T[q] != 0.0f)
              L = L + escape_radiance(s, mk(pool.dx[q], pool.dy[q], pool.dz[q])) * pool.beta[q];
            if (kCache && (pid & kTrainPath)) {
              finish_training(ts, pix, L);
            } else {
              write_result(pv, sum, pix, L);
              if (stats && (pid % pv.spp) == 0) {
                uint32_t* st = stats + 4 * (size_t)pix;
                st[0] = ev; st[1] = lk; st[2] = pv.pass; st[3] = ce;
              }
            }
            pool.free_[n_free + lane] = (uint8_t)q;
          }
          // a path counts < 2^27 (the work cap): 32 of them fit 32 bits
          const uint32_t a_look = __reduce_add_sync(0xffffffffu, lk), a_ev = __reduce_add_sync(0xffffffffu, ev),
                         a_cells = __reduce_add_sync(0xffffffffu, ce);
          if (lane == 0) {
            pool.totals[1] += a_look;
            pool.totals[2] += a_ev;
            pool.totals[3] += a_cells;
          }
          n_free += m;
          n_done -= m;
        } else if (n_shade >= 32u || (n_shade && n_ready == 0u && (exhausted || n_free < 32u))) {
          // ---- finished sun rays: their light, and a new direction ----------
          const uint32_t m = min(n_shade, 32u);
          bool go = false, end = false;
          uint32_t q = 0;
          if (lane < m) {
            q = pool.shade[(h_shade + lane) & (kRing - 1)];
            const f3 dir = mk(pool.dx[q], pool.dy[q], pool.dz[q]);
            const uint32_t pid = pool.pid[q], ev = pool.events[q] + 1u;  // the collision the ray started at
            float beta = pool.beta[q] * s.albedo;
            pool.events[q] = ev;
            const f3 lsun = kBatch ? -s_views[pid].sun : lsun0;
            const float phase = hg_pdf(s.ph, dot(-dir, -lsun));
            const float c = ((s.light * phase) * pool.T[q]) * beta;
            pool.L[q] = pool.L[q] + c;
            Rng rng{pool.rng[q], 0u};
            if (s.max_events && ev >= s.max_events) {
              end = true;
            } else if (kCache && (pid & kTrainPath) && ts.survival > 0.0f && ev >= (uint32_t)kNrcRecordEvents &&
                       !roulette_survives(rng, ts.survival, beta)) {
              end = true;  // past the recorded vertices: Russian roulette
            } else if (pool.lookups[q] + pool.cells[q] > kPathWorkCap) {  // runaway guard (non-finite input)
              end = true;
            } else {
              const DirRng nd = sample_direction(s.ph, dir, rng);
              pool.dx[q] = nd.d.x;
              pool.dy[q] = nd.d.y;
              pool.dz[q] = nd.d.z;
              pool.rng[q] = nd.r.state;
              pool.beta[q] = beta;
              go = true;
            }
            if (end) pool.T[q] = 0.0f;
          }
          const uint32_t mg = __ballot_sync(0xffffffffu, go), me = __ballot_sync(0xffffffffu, end);
          if (go) pool.ready[(h_ready + n_ready + __popc(mg & lt)) & (kRing - 1)] = (uint8_t)q;
          if (end) pool.done[n_done + __popc(me & lt)] = (uint8_t)q;
          h_shade += m;
          n_shade -= m;
          n_ready += __popc(mg);
          n_done += __popc(me);
        } else if (!exhausted && n_free != 0u && (n_free >= 32u || n_ready == 0u)) {
          // ---- new paths ----------------------------------------------------
          const uint32_t take = min(min(n_free, cap), 32u);
          uint32_t base = 0;
          if (lane == 0) base = (uint32_t)atomicAdd(cnt.c + (serving ? kTrainCursor : kWorkCursor), (unsigned long long)take);
          base = __shfl_sync(0xffffffffu, base, 0) + (serving || !kCache || !train_warps ? 0u : n_train);
          const uint32_t end = serving ? n_train : total + n_train;
          exhausted = base + take >= end;
          uint32_t id = base + lane, pid = 0, pix = 0;
          bool hit = false;
          const bool fresh = lane < take && id < end;
          Rng rng{0u, 0u};
          PathStart ps;
          if (fresh) {
            if (kBatch) {  // camera path of a view: the last view with path0 <= id
              uint32_t lo = 0, hi = bt.count - 1u;
              while (lo < hi) {
                uint32_t mid = (lo + hi + 1u) >> 1;
                if (s_views[mid].path0 <= id) lo = mid;
                else hi = mid - 1u;
              }
              const BatchView& bv = s_views[lo];
              uint32_t local = id - bv.path0;
              uint32_t per_row = bv.width * pv.spp;
              uint32_t cy = local / per_row, rem = local - cy * per_row;
              uint32_t cx = rem / pv.spp, sp = rem - cx * pv.spp;
              uint32_t lp = cy * bv.width + cx;
              pid = lo;
              pix = bv.pix0 + lp;
              rng = rng_pcg(pv.seed + kViewSeedStep * lo, lp * pv.spp + sp, pass);
              ps = start_path(bv.cam, s, (int)cx, (int)cy);
              if (!ps.hit) write_result(pv, sum, pix, ps.L);
            } else if (kCache && id < n_train) {  // training path from a uniformly drawn pixel of the crop
              rng = rng_pcg(pv.seed ^ kNrcTrainSalt, id, pass);
              uint32_t pp = (uint32_t)(rng_next(rng) * (float)(pv.cw * pv.ch));
              pp = min(pp, pv.cw * pv.ch - 1u);
              pid = kTrainPath;
              pix = kNrcNoSlot;
              ps = start_path(cam, s, (int)(pv.x0 + pp % pv.cw), (int)(pv.y0 + pp / pv.cw));
            } else {
              id -= n_train;
              uint32_t pq = pass;  // a launch of several passes: item id / per_pass is the pass offset
              if (pv.passes > 1u) {
                const uint32_t q = id / per_pass;
                id -= q * per_pass;
                pq += q;
              }
              pid = id;
              uint32_t per_row = pv.cw * pv.spp;
              uint32_t cy = id / per_row, rem = id - cy * per_row;
              uint32_t cx = rem / pv.spp, sp = rem - cx * pv.spp;
              int x = (int)(pv.x0 + cx), y = (int)(pv.y0 + cy);
              pix = (uint32_t)y * pv.width + (uint32_t)x;
              rng = rng_pcg(pv.seed, pix * pv.spp + sp, pq);
              ps = start_path(cam, s, x, y);
              if (!ps.hit) {
                write_result(pv, sum, pix, ps.L);
                if (stats && sp == 0) {
                  uint32_t* st = stats + 4 * (size_t)pix;
                  st[0] = 0; st[1] = 0; st[2] = pv.pass; st[3] = 0;
                }
              }
            }
            hit = ps.hit;
          }
          const uint32_t m = __ballot_sync(0xffffffffu, hit), n_new = __popc(__ballot_sync(0xffffffffu, fresh));
          if (lane == 0) pool.totals[0] += n_new;
          if (hit) {
            const uint32_t r = __popc(m & lt), q = pool.free_[n_free - 1u - r];
            pool.px[q] = ps.pos.x;
            pool.py[q] = ps.pos.y;
            pool.pz[q] = ps.pos.z;
            pool.dx[q] = ps.dir.x;
            pool.dy[q] = ps.dir.y;
            pool.dz[q] = ps.dir.z;
            pool.L[q] = 0.0f;
            pool.beta[q] = 1.0f;
            pool.rng[q] = rng.state;
            pool.pix[q] = pix;
            pool.pid[q] = pid;
            pool.events[q] = 0u;
            pool.lookups[q] = 0u;
            pool.cells[q] = 0u;
            pool.ready[(h_ready + n_ready + r) & (kRing - 1)] = (uint8_t)q;
          }
          n_free -= __popc(m);
          n_ready += __popc(m);
        } else {
          break;
        }
        __syncwarp();
      }
      const uint32_t m = min(n_idle, n_ready), r = __popc(idle & lt);
      if (mode == kIdle && r < m) {
        slot = pool.ready[(h_ready + r) & (kRing - 1)];
        o = mk(pool.px[slot], pool.py[slot], pool.pz[slot]);
        rd = mk(pool.dx[slot], pool.dy[slot], pool.dz[slot]);
        rs = pool.rng[slot];
        lookups = pool.lookups[slot];
        cells = pool.cells[slot];
        sun_ray = false;
        mode = kAim;
      }
      h_ready += m;
      n_ready -= m;
      // ---- the one DDA set-up site (camera ray, sun ray, scattered ray) -----
      if (mode == kAim) {
        track_init(tr, g, s, maj, o, rd, cells);
        walking = false;
        mode = kFly;
      }
      __syncwarp();
      if (!__any_sync(0xffffffffu, mode == kFly)) {
        // nothing waits either unless it is finished paths
        if (n_done == 0u) {
          if (!kCache || !serving) break;
          serving = false;  // its training paths are done: camera paths from now on
          exhausted = total == 0u;
        }
        continue;
      }
    }
    // ---- one bounded walk ---------------------------------------------------
    int r = kPending;
    if (mode == kFly) {
      if (!walking) {
        Rng rng{rs, 0u};
        tau = -vlog(rng_next(rng));
        rs = rng.state;
        walking = true;
      }
      r = track_walk(tr, maj, k, tau, cells, dda_steps);
    }
    __syncwarp();
    // ---- at most one density lookup (the candidate lanes together) ---------
    f3 p = o;
    float rho = 0.0f;
    if (r == kCandidate) {
      p = along(o, rd, tr.t);
      rho = density_from<kCorners>(g, s, p);
    }
    __syncwarp();
    // ---- collision, escape and path bookkeeping -----------------------------
    bool to_shade = false, to_done = false;
    if (r != kPending) {
      walking = false;
      bool nee_done = false, escaped = false, end = false;
      if (r == kCandidate) {
        ++lookups;
        if (sun_ray) T = T * (1.0f - rho / tr.m);
        float xi = 0.0f;  // the acceptance test's draw, or the roulette's on a dim sun ray
        if (!sun_ray || T < 0.05f) {
          Rng rng{rs, 0u};
          xi = rng_next(rng);
          rs = rng.state;
        }
        if (sun_ray) {
          if (T < 0.05f) {
            nee_done = xi >= 0.5f;
            T = nee_done ? 0.0f : T * 2.0f;
          }
        } else if (xi * tr.m < rho) {  // real collision (xi < rho / m): start the sun ray
          o = p;
          pool.px[slot] = o.x;
          pool.py[slot] = o.y;
          pool.pz[slot] = o.z;
          if (kCache) end = cache_vertex(pool, slot, s, nq, ts, o, rd);
          T = 1.0f;
          sun_ray = true;
          rd = kBatch ? -s_views[pool.pid[slot]].sun : lsun0;
          mode = kAim;
        }
      } else if (!sun_ray) {
        escaped = true;
        end = true;
      } else {
        nee_done = true;
      }
      if (lookups + cells > kPathWorkCap && !nee_done && !end) {  // runaway guard (non-finite input)
        if (mode == kAim) pool.events[slot] += 1u;
        end = true;
      }
      if (nee_done || end) {
        pool.T[slot] = nee_done ? T : (escaped ? 1.0f : 0.0f);
        pool.rng[slot] = rs;
        pool.lookups[slot] = lookups;
        pool.cells[slot] = cells;
        mode = kIdle;
        to_shade = nee_done;
        to_done = !nee_done;
      }
    }
    const uint32_t ms = __ballot_sync(0xffffffffu, to_shade), md = __ballot_sync(0xffffffffu, to_done);
    if (to_shade) pool.shade[(h_shade + n_shade + __popc(ms & lt)) & (kRing - 1)] = (uint8_t)slot;
    if (to_done) pool.done[n_done + __popc(md & lt)] = (uint8_t)slot;
    n_shade += __popc(ms);
    n_done += __popc(md);
    __syncwarp();
  }
  if (lane < 4u && pool.totals[lane]) atomicAdd(cnt.c + lane, pool.totals[lane]);
}



// A level is staged where the CTAs of 768 threads an SM still fit beside
// each other's pools (and some L1 is left): up to 16 KB for each of three
// CTAs of 256 threads, half of that for each of six of 128.  12 views of the
// 512^3 cloud over 16 KB of level-2 cells: 7.5 ms staged, 7.8 ms not.  Larger
// levels come through the L1; against one path a lane with up to 96 KB staged, 4
// passes of 1280x720 over 32 KB took 2.41 ms and take 1.65, over 86 KB 3.49 and
// 1.82 (at 128 threads 5.81 and 1.82), over 128 KB 2.61 and 1.90.  A batch's view
// table shares the room: 64, 128 and 256 views 18.0, 15.6 and 18.8 ms before,
// 10.3, 11.3 and 13.3 now.
constexpr uint32_t max_staged_bytes(uint32_t threads) { return 64u * threads; }

template <int kThreads, bool kStage, bool kBatch, bool kCache, bool kCorners>
static vcr_status launch_t(vcr_ctx* ctx, const GridView& g, const SceneView& s, const CamView& cam,
                           const PassView& pv, uint32_t* stats, Counters cnt, uint32_t total, uint32_t maj_bytes,
                           const NrcTrainSink& ts, const BatchSink& bt, double* sum, cudaStream_t st) {
  auto kern = pt_wavefront_kernel<kThreads, kStage, kBatch, kCache, kCorners>;
  constexpr uint32_t kWarps = kThreads / 32;
  const size_t pools = kWarps * sizeof(PathPool);
  size_t smem = pools + (kStage ? align16(maj_bytes) : 0u) + (kBatch ? bt.count * sizeof(BatchView) : 0u);
  // the attribute is per device, so it is set on every launch (a host-side call)
  VCR_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(pools + max_staged_bytes(kThreads) + kMaxBatchViews * sizeof(BatchView))));
  int per_sm = 0;
  VCR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem));
  if (per_sm < 1) per_sm = 1;
  const uint64_t paths = (uint64_t)total + ts.paths;
  if (paths == 0) return VCR_OK;
  uint32_t blocks = (uint32_t)(ctx->sm_count * per_sm);
  // a launch of few paths spreads them over all the warps that fit: a warp
  // with one path runs only that path's parts (64x64 pixels: 166 -> 126 us)
  uint32_t cap = (uint32_t)std::min<uint64_t>((paths + (uint64_t)blocks * kWarps - 1) / ((uint64_t)blocks * kWarps), 32u);
  blocks = std::min<uint32_t>(blocks, (uint32_t)((paths + (uint64_t)cap * kWarps - 1) / ((uint64_t)cap * kWarps)));
  const uint32_t train_warps = cap == 32u && total ? (ts.paths + kTrainShare - 1u) / kTrainShare : 0u;
  NrcSink nq{nullptr, nullptr, 0u};
  if (s.nrc_events && ctx->nrc) nq = NrcSink{ctx->nrc->query, ctx->nrc->query_count, ctx->nrc->query_capacity};
  kern<<<blocks, kThreads, smem, st>>>(g, s, cam, pv, sum, stats, cnt, total, ctx->tuning.dda_steps, cap, train_warps, maj_bytes,
                                       wait_limits().stage_wait, nq, ts, bt, ctx->d_error);
  VCR_CUDA(ctx, cudaGetLastError());
  return VCR_OK;
}

template <bool kBatch, bool kCache, bool kCorners>
static vcr_status launch_c(vcr_ctx* ctx, const GridView& g, const SceneView& s, const CamView& cam,
                           const PassView& pv, uint32_t* stats, Counters cnt, uint32_t total, uint32_t bytes,
                           bool stage, const NrcTrainSink& ts, const BatchSink& bt, double* sum, cudaStream_t st) {
  if (ctx->tuning.block_threads == 128)
    return stage ? launch_t<128, true, kBatch, kCache, kCorners>(ctx, g, s, cam, pv, stats, cnt, total, bytes, ts, bt, sum, st)
                 : launch_t<128, false, kBatch, kCache, kCorners>(ctx, g, s, cam, pv, stats, cnt, total, bytes, ts, bt, sum, st);
  return stage ? launch_t<256, true, kBatch, kCache, kCorners>(ctx, g, s, cam, pv, stats, cnt, total, bytes, ts, bt, sum, st)
               : launch_t<256, false, kBatch, kCache, kCorners>(ctx, g, s, cam, pv, stats, cnt, total, bytes, ts, bt, sum, st);
}

template <bool kBatch, bool kCache>
static vcr_status launch_b(vcr_ctx* ctx, const GridView& g, const SceneView& s, const CamView& cam,
                           const PassView& pv, uint32_t* stats, Counters cnt, uint32_t total, uint32_t bytes,
                           bool stage, const NrcTrainSink& ts, const BatchSink& bt, double* sum, cudaStream_t st) {
  return g.corners ? launch_c<kBatch, kCache, true>(ctx, g, s, cam, pv, stats, cnt, total, bytes, stage, ts, bt, sum, st)
                   : launch_c<kBatch, kCache, false>(ctx, g, s, cam, pv, stats, cnt, total, bytes, stage, ts, bt, sum, st);
}

vcr_status wavefront_launch(vcr_ctx* ctx, const GridView& g, const SceneView& s, const CamView& cam,
                            const PassView& pv, uint32_t* stats, Counters cnt, uint32_t total, cudaStream_t st,
                            const NrcTrainSink* train, const BatchSink* batch, double* sum) {
  const vcr_tuning& t = ctx->tuning;
  NrcTrainSink ts{nullptr, nullptr, 0u, 0u, 0.0f};
  if (train) ts = *train;
  BatchSink bt{nullptr, 0u, nullptr};
  if (batch) bt = *batch;
  if ((uint64_t)total + ts.paths >= (uint64_t)kTrainPath)
    return fail(ctx, VCR_ERR_UNSUPPORTED, "more than 2^31 paths in one launch");
  if (batch && (train || bt.count == 0 || bt.count > kMaxBatchViews || !bt.views || !bt.pass_ctr))
    return fail(ctx, VCR_ERR_INVALID, "a batch launch needs 1..%u views and no training paths", kMaxBatchViews);
  size_t cells = (size_t)g.mnb[0] * g.mnb[1] * g.mnb[2];
  uint32_t bytes = (uint32_t)(((cells + 3) & ~(size_t)3) * sizeof(float));  // padded level: 16-byte multiple
  bool stage = t.stage_majorants && bytes <= max_staged_bytes(t.block_threads);
  if (!sum) sum = ctx->d_sum;
  // a launch with neither queries nor training paths takes a kernel without
  // their parts, whose shorter loop is fetched faster: 8 passes of 1920x1080
  // 5.29 -> 4.98 ms, 12 views 7.49 -> 7.12, 64x64 pixels 192 -> 174 us with the
  // call's host time (batches refuse the cache).  The texel gathers of grids
  // without corner blocks are left out in the same way (5.06 -> 4.70 ms, 7.26 ->
  // 6.99 ms, a 512x512 frame 260 -> 248 us, an online cached frame 961 -> 913 us)
  if (batch) return launch_b<true, false>(ctx, g, s, cam, pv, stats, cnt, total, bytes, stage, ts, bt, sum, st);
  return s.nrc_events || ts.paths
             ? launch_b<false, true>(ctx, g, s, cam, pv, stats, cnt, total, bytes, stage, ts, bt, sum, st)
             : launch_b<false, false>(ctx, g, s, cam, pv, stats, cnt, total, bytes, stage, ts, bt, sum, st);
}

}  // namespace VCR_WF_NS
}  // namespace vcr
