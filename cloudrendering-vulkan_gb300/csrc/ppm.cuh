// Photon-map state owned by a context (RenderTechniquePPM's photon map and
// collision map, RenderTechniquePPM.cpp:115-156, plus per-pixel statistics).
#pragma once

#include "vcr_internal.h"

namespace vcr {

constexpr uint32_t kPpmMaxEvents = 64;  // deposits per photon path (uid = photon * 64 + event)
constexpr uint32_t kPpmEmitSalt = 0x27D4EB2Fu;
constexpr uint32_t kPpmGatherSalt = 0x165667B1u;

struct PpmState {
  vcr_ppm_params prm{};
  size_t pixels = 0;
  uint32_t photons_stored = 0, dropped = 0;
  float4 *pos = nullptr, *pw = nullptr, *dir = nullptr;
  uint32_t *uid = nullptr, *count = nullptr, *by_uid = nullptr, *uid_sorted = nullptr, *codes = nullptr,
           *idx = nullptr, *codes_sorted = nullptr, *order = nullptr, *iota = nullptr;
  uint32_t *deposits = nullptr, *first = nullptr, *scan_sums = nullptr;  // per emitted photon: deposits, their sums
  uint32_t *left = nullptr, *right = nullptr;
  float4* tree_clusters = nullptr;  // the march's tree: boxes over 32, 32^2 and 32^3 leaves while it is built
  float4 *leaf_lo = nullptr, *leaf_hi = nullptr, *node_lo = nullptr, *node_hi = nullptr;
  // the march's tree walk: internal nodes packed as (lo, left), (hi, right),
  // photon powers and directions in leaf order
  float4* node_pk = nullptr;
  float4* leaf_pw = nullptr;
  float4* leaf_dir = nullptr;
  float4* box = nullptr;  // the gather's boxes over 8 consecutive leaves, over 8 of those, ...
  // the pass's measurement points: their number, position and sigma_t, pixel
  uint32_t *points = nullptr, *point_pix = nullptr;
  float4* point = nullptr;
  double* stats = nullptr;  // per pixel: N, R, tau rgb, background rgb
  GatherProbe gather;       // photons the last gather tested, its device time
};

}  // namespace vcr
