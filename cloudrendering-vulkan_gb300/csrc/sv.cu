// Shadow volume: a light-aligned n^3 grid of approximate sun transmittance,
// exp(-(z+1) * voxelSize * mean density along the column), the
// reference-parity NEE term.
//
// Reference: ShadowVolume.comp:77-93 (one invocation per (x,y) column marching z),
// calculateVoxelPosition (Tests.cpp:104-110 restates it on the CPU),
// dispatch RenderTechniqueSV.cpp:102-113.
#include "vcr_internal.h"

namespace vcr {

struct SvBuild {
  f3 b0, right, up, light;
  float vs;
  int n;
};

// A CTA takes 32 columns (consecutive x: the z slices' stores are coalesced)
// and kSlab z at a time.  The lookups of a slab do not depend on one another:
// its warps share them.  Only the running sums along z are a chain of adds
// (in the order of the march, so the same floats), which one warp walks, a
// column a lane; the exponentials are spread over the warps again.  A thread
// marching its column alone, a dependent load and an add a step, left the
// 128^3 volume to 64 CTAs: 102 us, now 22 us (2.1 M lookups and stores).
constexpr int kSlab = 64;
constexpr int kSvWarps = 8;

__global__ void __launch_bounds__(32 * kSvWarps) sv_build_kernel(GridView g, SceneView s, SvBuild b,
                                                                 float* __restrict__ out) {
  __shared__ float s_acc[kSlab][32], s_dist[kSlab];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t n = (uint32_t)b.n, col = blockIdx.x * 32u + lane;
  const bool in = col < n * n;
  const uint32_t x = in ? col % n : 0u, y = in ? col / n : 0u;
  const size_t plane = (size_t)n * n;
  const float fx = (float)x * b.vs, fy = (float)y * b.vs;
  float acc = 0.0f, dist = 0.0f;  // warp 0: the column's sums so far
  for (uint32_t z0 = 0; z0 < n; z0 += kSlab) {
    const uint32_t nz = min((uint32_t)kSlab, n - z0);
    for (uint32_t k = warp; k < nz; k += kSvWarps) {
      const float fz = (float)(z0 + k) * b.vs;
      f3 p;
      p.x = ((b.b0.x + fx * b.right.x) + fy * b.up.x) + fz * b.light.x;
      p.y = ((b.b0.y + fx * b.right.y) + fy * b.up.y) + fz * b.light.y;
      p.z = ((b.b0.z + fx * b.right.z) + fy * b.up.z) + fz * b.light.z;
      s_acc[k][lane] = in && in_box(p, s.b0, s.b1) ? (density_at(g, s, p) * s.ds) / s.bs : 0.0f;
    }
    __syncthreads();
    if (warp == 0) {
      for (uint32_t k = 0; k < nz; ++k) {
        acc = acc + s_acc[k][lane];
        s_acc[k][lane] = acc;
        dist = dist + b.vs;
        if (lane == 0) s_dist[k] = dist;
      }
    }
    __syncthreads();
    if (in)
      for (uint32_t k = warp; k < nz; k += kSvWarps)
        out[(size_t)col + plane * (z0 + k)] = vexp(((-s_dist[k]) * s_acc[k][lane]) / (float)(z0 + k + 1u));
    __syncthreads();
  }
}

vcr_status sv_build_launch(vcr_ctx* ctx, const vcr_shadow_volume* sv, cudaStream_t st) {
  if (!ctx->has_grid || !ctx->has_cloud) return fail(ctx, VCR_ERR_STATE, "shadow volume needs a grid and a cloud");
  uint32_t n = sv->voxel_axis_count;
  if (n < 2 || n > 1024) return fail(ctx, VCR_ERR_INVALID, "shadow volume axis count %u outside [2, 1024]", n);
  size_t bytes = (size_t)n * n * n * sizeof(float);
  if (!ctx->has_sv || ctx->sv.voxel_axis_count != n) {
    cudaFree(ctx->d_sv);
    ctx->d_sv = nullptr;
    ctx->has_sv = false;
    VCR_CUDA(ctx, cudaMalloc(&ctx->d_sv, bytes));
  }
  SvBuild b;
  b.b0 = mk(sv->bounds_min[0], sv->bounds_min[1], sv->bounds_min[2]);
  b.right = mk(sv->right[0], sv->right[1], sv->right[2]);
  b.up = mk(sv->up[0], sv->up[1], sv->up[2]);
  b.light = mk(sv->light_dir[0], sv->light_dir[1], sv->light_dir[2]);
  b.vs = sv->voxel_size;
  b.n = (int)n;
  uint32_t cols = n * n;
  sv_build_kernel<<<(cols + 31) / 32, 32 * kSvWarps, 0, st>>>(grid_view(ctx), scene_view(ctx), b, ctx->d_sv);
  VCR_CUDA(ctx, cudaGetLastError());
  ctx->sv = *sv;
  ctx->has_sv = true;
  return VCR_OK;
}

}  // namespace vcr
