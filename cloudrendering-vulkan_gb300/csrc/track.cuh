// DDA free-flight tracking over a majorant pyramid level, shared by the
// path tracer, the photon-beam emitter and the photon emitter.
#pragma once

#include "pt_common.cuh"

namespace vcr {

// A ray's walk over the majorant cells: the steps and cells of dda_advance /
// dda_linear (vcr_device.cuh) in a form with fewer instructions a cell.  The
// cell is its linear index, an axis's step the index difference, and the
// cells left before the grid's side are counted down in 10 bits an axis (an
// axis has at most 1024 cells).
struct Track {
  float tmax[3];  // ray t of the next boundary per axis
  float tdel[3];  // t per cell along the axis (+inf: the axis never advances)
  int step[3];    // index difference of a step along the axis
  uint32_t cell;  // linear index of the current cell
  uint32_t left;  // cells left along the ray per axis, 10 bits each
  float t, t_end, m;
};

__device__ __forceinline__ void track_axis(float o, float d, float inv, float b0, float cs, int c, int nc, float& tmax,
                                           float& tdel, uint32_t& left) {
  const bool up = d > 0.0f, moves = up || d < 0.0f;
  const float edge = b0 + (float)(up ? c + 1 : c) * cs;
  tmax = moves ? (edge - o) * inv : INFINITY;
  tdel = moves ? fabsf(cs * inv) : INFINITY;
  left = (uint32_t)(up ? nc - 1 - c : c);
}

__device__ __forceinline__ void track_init(Track& tr, const GridView& g, const SceneView& s, const float* maj, f3 o,
                                           f3 d, uint32_t& cells) {
  float tmin, tmax;
  const f3 inv = recip(d);
  if (!slab_inv(o, inv, s.b0, s.b1, tmin, tmax) || !finite_pos(tmax)) tmax = 0.0f;
  tr.t = 0.0f;
  tr.t_end = tmax;
  const int cx = cell_of(o.x, s.b0.x, s.icell.x, g.mnb[0]), cy = cell_of(o.y, s.b0.y, s.icell.y, g.mnb[1]),
            cz = cell_of(o.z, s.b0.z, s.icell.z, g.mnb[2]);
  uint32_t lx, ly, lz;
  track_axis(o.x, d.x, inv.x, s.b0.x, s.cell.x, cx, g.mnb[0], tr.tmax[0], tr.tdel[0], lx);
  track_axis(o.y, d.y, inv.y, s.b0.y, s.cell.y, cy, g.mnb[1], tr.tmax[1], tr.tdel[1], ly);
  track_axis(o.z, d.z, inv.z, s.b0.z, s.cell.z, cz, g.mnb[2], tr.tmax[2], tr.tdel[2], lz);
  tr.left = lx | (ly << 10) | (lz << 20);
  const int sy = g.mnb[0], sz = g.mnb[0] * g.mnb[1];
  tr.step[0] = d.x < 0.0f ? -1 : 1;
  tr.step[1] = d.y < 0.0f ? -sy : sy;
  tr.step[2] = d.z < 0.0f ? -sz : sz;
  tr.cell = (uint32_t)(cx + sy * cy + sz * cz);
  tr.m = maj[tr.cell];
  ++cells;
}

enum : int { kPending = 0, kCandidate = 1, kExit = 2 };

// Up to `steps` cells of one free flight: consume the optical depth `tau`
// cell by cell (dtau = (m k)(min(exit, t_end) - t)); a tentative collision
// lands at t + tau/(m k) inside the cell where tau runs out.  The lanes of a
// warp leave the loop after different cell counts, so the collision's
// division stands behind it, once for all of them (inside, every group that
// left took its own), and the axis is selected instead of branched to.
__device__ __forceinline__ int track_walk(Track& tr, const float* maj, float k, float& tau, uint32_t& cells,
                                          uint32_t steps) {
  int r = kPending;
  float sig = 0.0f;
  for (uint32_t i = 0; i < steps; ++i) {
    const float e = fminf(fminf(tr.tmax[0], tr.tmax[1]), tr.tmax[2]);
    const float se = fminf(e, tr.t_end);
    sig = tr.m * k;
    const float dtau = sig * (se - tr.t);
    if (dtau > tau) {
      r = kCandidate;
      break;
    }
    tau = tau - dtau;
    tr.t = se;
    const bool x = tr.tmax[0] <= tr.tmax[1] && tr.tmax[0] <= tr.tmax[2];
    const bool y = !x && tr.tmax[1] <= tr.tmax[2];
    const uint32_t field = x ? 0x3FFu : y ? 0x3FFu << 10 : 0x3FFu << 20;
    if (e >= tr.t_end || (tr.left & field) == 0u) {  // the ray's end, or the grid's side
      r = kExit;
      break;
    }
    tr.left -= field & 0x00100401u;
    tr.cell += (uint32_t)(x ? tr.step[0] : y ? tr.step[1] : tr.step[2]);
    if (x) tr.tmax[0] = tr.tmax[0] + tr.tdel[0];
    if (y) tr.tmax[1] = tr.tmax[1] + tr.tdel[1];
    if (!x && !y) tr.tmax[2] = tr.tmax[2] + tr.tdel[2];
    tr.m = maj[tr.cell];
    ++cells;
  }
  if (r == kCandidate) tr.t = tr.t + tau / sig;
  return r;
}

// One delta-tracking free flight from o along unit d (DDA majorants):
// true with the distance t of the first real collision, false on escape
// (t = distance to the box exit).  Draw order: per tentative collision one
// uniform for the optical depth, then one for the acceptance test.
__device__ __forceinline__ bool free_flight(const GridView& g, const SceneView& s, f3 o, f3 d, Rng& rng, float& t,
                                            uint32_t& lookups, uint32_t& cells) {
  Track tr;
  track_init(tr, g, s, g.majorants, o, d, cells);
  while (true) {
    float tau = -vlog(rng_next(rng));
    if (track_walk(tr, g.majorants, s.k_sigma, tau, cells, 0xFFFFFFFFu) != kCandidate) {
      t = tr.t_end;
      return false;
    }
    float rho = density_at(g, s, along(o, d, tr.t));
    ++lookups;
    if (rng_next(rng) * tr.m < rho) {  // xi < rho / m without the division
      t = tr.t;
      return true;
    }
    if (lookups + cells > kPathWorkCap) {  // runaway guard (non-finite input)
      t = tr.t_end;
      return false;
    }
  }
}

}  // namespace vcr
