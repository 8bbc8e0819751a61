// Neural radiance cache: a 64 -> 5x64 (ReLU) -> 3 MLP that predicts the
// radiance leaving a scattering vertex toward the previous vertex, trained
// online on paths the tracer itself produces and queried where paths
// terminate into it.  No reference counterpart.
//
// Tensor cores, BF16 operands, FP32 accumulation.  Queries: a
// register-resident forward (mma.sync m16n8k16, nrc_mma.cuh) — each warp
// runs 16-sample tiles whose activations stay in the MMA fragments, the CTA
// shares only the BF16 weights.  Training: one CTA per SM holds
// the BF16 weights and, for a 128-sample tile, the activation tiles and the
// gradient ping-pong in padded shared memory (215 KB); its warps have roles:
// the forward and the backward's dY_l W_l^T run register-resident on the same
// mma.sync fragments, ldmatrix.trans feeds X_l^T dY_l over the tile to warps
// of their own, and others encode the next tile's inputs.  The weight gradient
// stays in the warps' accumulator fragments across all the CTA's tiles; at
// the end each CTA stores it into its own slot and one kernel sums the
// slots in a fixed order and takes the Adam step (one atomic add per
// weight per CTA cost as much as the tiles themselves).  Adam runs on FP32
// master weights and refreshes the BF16 copies (training weights, and the
// moving average the queries use).
#include <cmath>
#include <cstring>

#include "nrc.cuh"
#include "nrc_mma.cuh"
#include "track.cuh"

namespace vcr {

using bf16 = __nv_bfloat16;

// Training CTA: 4 chain warps (forward and backward, 32 records each), 4
// gradient warps and 4 encoder warps, one 128-record tile at a time.
constexpr int kTrainRole = 4 * 32;  // threads of a role
constexpr int kTrainThreads = 3 * kTrainRole;
constexpr int kTrainTile = 128;

constexpr int kTileX = kTrainTile * kLdX;                                  // one activation tile

struct NrcView {
  const bf16* wb;   // training weights
  const bf16* wbi;  // inference weights (the moving average, or wb)
  f3 b0, inv_ext;
  int levels;       // position-encoding levels the network sees (the rest are 0)
  // grid encoding (nullptr: the frequency encoding): the tables training
  // reads, the tables queries read (their moving average, or gtab), and the
  // tables' gradient accumulator
  const float* gtab;
  const float* gtab_i;
  float* ggrad;
};

// ---------------------------------------------------------------------------
// inference: sum[pix] += throughput * max(cache(x, view, sun), 0); out (if
// given) receives the 3 outputs.  Register-resident forward (nrc_mma.cuh):
// every warp runs whole 16-sample tiles, the CTA shares only the weights.
// ---------------------------------------------------------------------------
constexpr int kInferThreads = 256;

__global__ void __launch_bounds__(kInferThreads, 3) nrc_infer_kernel(NrcView v, const NrcRecord* __restrict__ recs,
                                                                     const uint32_t* __restrict__ count_ptr,
                                                                     uint32_t capacity, double* __restrict__ sum,
                                                                     float* __restrict__ out) {
  extern __shared__ __align__(128) unsigned char smem[];
  bf16* W = reinterpret_cast<bf16*>(smem);
  float* dirs = reinterpret_cast<float*>(W + kWs);  // 16 level directions
  load_weights<kInferThreads>(v.wbi, W);
  load_level_dirs(dirs);
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t count = min(*count_ptr, capacity);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile * 16u < count; tile += warps) {
    const uint32_t i0 = tile * 16u + (uint32_t)g, i1 = i0 + 8u;
    NrcRecord r0{}, r1{};
    if (i0 < count) r0 = recs[i0];
    if (i1 < count) r1 = recs[i1];
    uint32_t a[4][4];
    encode_a(r0, i0 < count, v.b0, v.inv_ext, dirs, t, 0, a, v.levels, v.gtab_i);
    encode_a(r1, i1 < count, v.b0, v.inv_ext, dirs, t, 1, a, v.levels, v.gtab_i);
    float yg[3], yh[3];
    mlp_forward_mma(W, a, lane, yg, yh);
    if (t == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t idx = h ? i1 : i0;
        if (idx >= count) continue;
        const NrcRecord& r = h ? r1 : r0;
        const float* y = h ? yh : yg;
        if (out) {
          out[3 * idx] = y[0];
          out[3 * idx + 1] = y[1];
          out[3 * idx + 2] = y[2];
        }
        if (sum) {
          double* o = sum + 3 * (size_t)r.pix;
          atomicAdd(o + 0, (double)(r.w0 * fmaxf(y[0], 0.0f)));
          atomicAdd(o + 1, (double)(r.w1 * fmaxf(y[1], 0.0f)));
          atomicAdd(o + 2, (double)(r.w2 * fmaxf(y[2], 0.0f)));
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// training: relative L2 loss sum_c (y - t)^2 / (sg(y)^2 + 0.01) / (3 B)
// ---------------------------------------------------------------------------

// Launched with launch_overlapped, a kernel may be set up on the device while
// the one before it in its stream still runs; grid_wait waits for that one's
// end, and comes before any access to memory.  grid_trigger lets the next one
// be set up.  A training step is two short kernels: 41.7 -> 41.0 us.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

// Registers a thread of each role, a launch with 168 in all: 3 x 168 = 504.
constexpr int kRegsChain = 216, kRegsGrad = 224, kRegsEncode = 64;
static_assert(kRegsChain + kRegsGrad + kRegsEncode <= 3 * 168, "register split");
template <int kRegs>
__device__ __forceinline__ void set_regs_up() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void set_regs_down() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// k-tile kt of the B fragments of a hidden layer, W_l as [in][out] (the
// forward) and as [out][in] (the backward); NP 16-wide tiles.
template <int NP>
__device__ __forceinline__ void load_in_out(const bf16* Wl, int ld, int kt, uint32_t (&b)[4][4], int lane) {
  const int rr = lane & 7, q = lane >> 3;
#pragma unroll
  for (int np = 0; np < NP; ++np) ldsm_x4_t(b[np], Wl + (kt * 16 + rr + 8 * (q & 1)) * ld + np * 16 + 8 * (q >> 1));
}
__device__ __forceinline__ void load_out_in(const bf16* Wl, int ld, int kt, uint32_t (&b)[4][4], int lane) {
  const int rr = lane & 7, q = lane >> 3;
#pragma unroll
  for (int np = 0; np < 4; ++np) ldsm_x4(b[np], Wl + (np * 16 + rr + 8 * (q >> 1)) * ld + kt * 16 + 8 * (q & 1));
}

// mma_bf16 with zero for the accumulators' old values.
__device__ __forceinline__ void mma_bf16_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

// One layer of one fragment of 16 records, acc = a b over KT k-tiles.  After
// each pair of MMAs comes other(kt, np), a sixteenth of what the last layer of
// the warp's other fragment leaves to do: its scalar work fills the issue
// slots between the MMAs.  After k-tile kt comes reload(kt), for b[kt] is not
// needed any more.
template <int KT, class Reload, class Other>
__device__ __forceinline__ void chain_phase(float (&acc)[8][4], const uint32_t (&a)[4][4], uint32_t (&b)[4][4][4],
                                            Reload reload, Other other) {
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      if (kt == 0) {
        mma_bf16_zero(acc[2 * np], a[kt], b[kt][np][0], b[kt][np][1]);
        mma_bf16_zero(acc[2 * np + 1], a[kt], b[kt][np][2], b[kt][np][3]);
      } else if (kt < KT) {
        mma_bf16(acc[2 * np], a[kt], b[kt][np][0], b[kt][np][1]);
        mma_bf16(acc[2 * np + 1], a[kt], b[kt][np][2], b[kt][np][3]);
      }
      other(kt, np);
    }
    reload(kt);
  }
}

// Word p of k-tile kt of a fragment to its rows of a tile.
__device__ __forceinline__ void store_word(bf16* T, int row, int t, int kt, int p, uint32_t w) {
  *reinterpret_cast<uint32_t*>(T + (row + 8 * (p & 1)) * kLdX + kt * 16 + 8 * (p >> 1) + 2 * t) = w;
}

// ReLU and BF16 of word p of accumulator tiles 2 kt, 2 kt + 1: the A fragment
// of the next layer's k-tile kt (the maximum after the rounding is the
// rounding of the maximum, and takes a NaN to 0 like fmaxf).
__device__ __forceinline__ uint32_t relu_word(const float (&acc)[8][4], int kt, int p) {
  const float* y = &acc[2 * kt + (p >> 1)][2 * (p & 1)];
  const __nv_bfloat162 r = __hmax2(__floats2bfloat162_rn(y[0], y[1]), __floats2bfloat162_rn(0.0f, 0.0f));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// The same for the backward: the accumulators times 1 where the layer's input
// x is above zero, else times 0.
__device__ __forceinline__ uint32_t mask_word(const float (&acc)[8][4], int kt, int p, uint32_t x) {
  const float* y = &acc[2 * kt + (p >> 1)][2 * (p & 1)];
  const __nv_bfloat162 one = __hgt2(*reinterpret_cast<const __nv_bfloat162*>(&x), __floats2bfloat162_rn(0.0f, 0.0f));
  const __nv_bfloat162 r = __hmul2(__floats2bfloat162_rn(y[0], y[1]), one);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// A fragment of 16 records of a [record][feature] tile, by the address of the
// lane's row of it.
__device__ __forceinline__ void load_fragment(const bf16* p, uint32_t (&a)[4][4]) {
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) ldsm_x4(a[kt], p + kt * 16);
}

// Half of the 64 inputs of one record as its row of X_0 (nrc_encode's order):
// eight levels and one direction; zeros for a row without a record.
template <bool kGrid>
__device__ __forceinline__ void encode_half(const NrcRecord* rec, int half, const NrcView& v, const float* dirs,
                                            bf16* row) {
  uint4* out = reinterpret_cast<uint4*>(row) + 2 * half;
  if (!rec) {
    out[0] = out[1] = out[4] = out[5] = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  float ux, uy, uz;
  nrc_box_coords(*rec, v.b0, v.inv_ext, ux, uy, uz);
  const float* d = half ? &rec->sx : &rec->vx;
  const float dx = d[0], dy = d[1], dz = d[2];
#pragma unroll 1
  for (int j = 0; j < 2; ++j) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int l = 8 * half + 4 * j + i;
      float sn = 0.0f, cs = 0.0f;
      if (l < v.levels) {
        if (kGrid) nrc_grid_level(v.gtab, l, ux, uy, uz, &sn, &cs);
        else nrc_encode_level_dir(l, dirs[3 * l], dirs[3 * l + 1], dirs[3 * l + 2], ux, uy, uz, &sn, &cs);
      }
      w[i] = pack_bf16(sn, cs);
    }
    out[j] = make_uint4(w[0], w[1], w[2], w[3]);
  }
  float sh[16];
  nrc_sh16(dx, dy, dz, sh);
#pragma unroll
  for (int j = 0; j < 2; ++j)
    out[4 + j] = make_uint4(pack_bf16(sh[8 * j], sh[8 * j + 1]), pack_bf16(sh[8 * j + 2], sh[8 * j + 3]),
                            pack_bf16(sh[8 * j + 4], sh[8 * j + 5]), pack_bf16(sh[8 * j + 6], sh[8 * j + 7]));
}

// Named barriers of the training CTA (0 is __syncthreads).  Each is arrived
// at by one role and waited for by another; a pair is used in turn, so a role
// never arrives twice at one barrier before the other has passed it.
enum TrainBar : int {
  kBarFull = 1,   // +0, +1: dY_l (and X_l) of every row stored; chain -> gradient
  kBarEmpty = 3,  // +0, +1: dW_l added up, its dY buffer and X_l free; gradient -> chain
  kBarInput = 5,  // +0, +1: X_0 of a tile encoded; encoders -> chain
  kBarSpare = 7,  // +0, +1: dW_0 added up, its buffer of X_0 free; gradient -> encoders
  kBarFirst = 9,  // X_0 of the first tile; encoders and gradient -> chain
  kBarDirs = 10,  // the level directions; encoders and gradient
  kBarChain = 11, // the weights; the chain warps alone
};
template <int kRoles>
__device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kRoles * kTrainRole) : "memory");
}
template <int kRoles>
__device__ __forceinline__ void bar_wait(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kRoles * kTrainRole) : "memory");
}

// One CTA per SM, a 128-record tile at a time, in three roles of 4 warps, one
// of each on every scheduler.
//
// Chain warps own 32 records each, as two fragments of 16 that are half a
// layer apart: while the tensor pipe works on one, the other's activations
// are rounded and stored.  The forward keeps the activations in MMA fragments
// (as the queries do) and stores each layer's input X_l once, as BF16, into
// the tile's shared [record][feature] buffers; the backward runs dY_l W_l^T
// in registers as well (the dY A fragments of one layer are the masked
// accumulators of the last), so only X_l and dY_l go
// through shared memory.
//
// Gradient warps add up dW_l = X_l^T dY_l over all 128 records as soon as
// dY_l is stored, while the chain warps work on dY_{l-1}.  Warp w owns the
// 32 x 32 block (rows 32(w/2).., columns 32(w%2)..) of every 64x64
// hidden-layer gradient and rows 16w.. of the 64x16 output layer's, in
// registers across the CTA's tiles; X_l^T and dY_l fragments come from
// ldmatrix.trans.  At the end each CTA stores its gradient into its own slot
// of gpart.
//
// Encoder warps write the next tile's inputs, a record a lane (X_0 has two
// buffers).
//
// What bounds it: a tile's 3,840 MMAs take 7,700 cycles of the four tensor
// pipes (8.1 each; FMA-pipe instructions go to the same port, so the masks and
// maxima are packed BF16), its operands 9,600 wavefronts of shared memory; it
// takes 13,300 cycles, the forward at the chain's latency, the backward at
// both pipes (1,500 cycles a layer).  65,536 records, 8 steps: 431 us with
// eight warps that did everything in turn (two barriers a layer, 11,200
// wavefronts a tile), 382 with eight chain and eight gradient warps, 333 so
// (348 with eight gradient warps of half the block: more wavefronts).
//
// kGrid (the grid encoding): the backward also forms dX_0 = dY_0 W_0^T for
// the 32 position inputs in registers and adds, for every record, level and
// feature, the 8 trilinear shares of it into the tables' gradient (float
// atomics, so their order, and the last bits of the sums, vary).  They bound
// it: an entry's two features in one vector atomic 131 us for 65.9 k records,
// one by one 215.
template <bool kGrid>
__global__ void __launch_bounds__(kTrainThreads, 1) nrc_train_kernel(NrcView v, const NrcRecord* __restrict__ recs,
                                                                     const uint32_t* __restrict__ count_ptr,
                                                                     uint32_t capacity, uint32_t first_rec,
                                                                     float* __restrict__ gpart, float* __restrict__ loss) {
  extern __shared__ __align__(128) unsigned char smem[];
  bf16* W = reinterpret_cast<bf16*>(smem);              // [in][out], rows of ldw(l)
  bf16* X = W + kWs;                                     // X_1 .. X_5 of the tile at l * kTileX, X_0 of two tiles at 0 and 6
  bf16* D = X + (kNrcLayers + 1) * kTileX;               // dY ping-pong: dY_5, dY_3, dY_1 in buffer 0
  float* dirs = reinterpret_cast<float*>(D + 2 * kTileX);  // 16 position-level directions
  // records [first_rec, first_rec + capacity) of the *count_ptr written; a
  // CTA without a tile leaves its slot alone (the reduction reads the slots
  // of the first ceil(count / kTrainTile) CTAs only)
  grid_wait();
  grid_trigger();
  const uint32_t total = *count_ptr;
  const int role = threadIdx.x / kTrainRole;  // 0 chain, 1 gradient, 2 encoders
  const int k = threadIdx.x & (kTrainRole - 1);
  // what does not depend on the records, while the count is on its way
  if (role == 0) {
    load_weights<kTrainRole>(v.wb, W);
    bar_wait<1>(kBarChain);
  } else {
    if (role == 2 && k < kNrcPosLevels) nrc_level_dir(k, dirs[3 * k], dirs[3 * k + 1], dirs[3 * k + 2]);
    bar_wait<2>(kBarDirs);
  }
  const uint32_t count = total > first_rec ? min(total - first_rec, capacity) : 0u;
  if (blockIdx.x * kTrainTile >= count) return;
  const int warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rr = lane & 7, q = lane >> 3;
  const uint32_t start = blockIdx.x * kTrainTile, stride = gridDim.x * kTrainTile;
  recs += first_rec;

  if (role == 2) {
    set_regs_down<kRegsEncode>();
    uint32_t tile = 0;
#pragma unroll 1
    for (uint32_t first = start; first < count; first += stride, ++tile) {
      const int at = tile & 1;
      if (tile >= 2) bar_wait<2>(kBarSpare + at);  // dW_0 of the tile before the last
      const uint32_t idx = first + (uint32_t)k;
      const NrcRecord* rec = idx < count ? recs + idx : nullptr;
      bf16* out = X + (at ? kNrcLayers * kTileX : 0) + k * kLdX;
#pragma unroll 1
      for (int half = 0; half < (tile ? 2 : 1); ++half) encode_half<kGrid>(rec, half, v, dirs, out);
      if (tile) bar_arrive<2>(kBarInput + at);
      else bar_arrive<3>(kBarFirst);
    }
    return;
  }

  if (role == 1) {
    set_regs_up<kRegsGrad>();
    // half of the first tile's inputs: there is nothing else to do yet
    encode_half<kGrid>(start + (uint32_t)k < count ? recs + start + k : nullptr, 1, v, dirs, X + k * kLdX);
    bar_arrive<3>(kBarFirst);
    const int m0 = (warp >> 1) * 32, n0 = (warp & 1) * 32;  // the warp's gradient blocks
    float dwh[kNrcHidden][2][4][4], dwo[2][4];
#pragma unroll
    for (int l = 0; l < kNrcHidden; ++l)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          dwh[l][i][j][0] = dwh[l][i][j][1] = dwh[l][i][j][2] = dwh[l][i][j][3] = 0.0f;
#pragma unroll
    for (int j = 0; j < 2; ++j) dwo[j][0] = dwo[j][1] = dwo[j][2] = dwo[j][3] = 0.0f;
    uint32_t tile = 0;
#pragma unroll 1
    for (uint32_t first = start; first < count; first += stride, ++tile) {
      const int at = tile & 1;
      const bool more = count - first > stride;                     // a next tile
      const bool spare = more && count - first - stride > stride;  // and one after it
#pragma unroll
      for (int l = kNrcLayers - 1; l >= 0; --l) {  // unrolled: the gradient blocks are indexed by layer
        const int buf = (kNrcLayers - 1 - l) & 1;
        const bf16* Xl = X + (l == 0 && at ? kNrcLayers : l) * kTileX;
        const bf16* Dl = D + buf * kTileX;
        bar_wait<2>(kBarFull + buf);  // X_l and dY_l complete for every row
        // dW_l += X_l^T dY_l over the tile's 128 records (k); the fragments of
        // 16 records are loaded while the last 16's are used
        // X_l^T: features by records 16kt..; dY_l: records 16kt.. by columns
        const bf16* xr = Xl + (rr + 8 * (q >> 1)) * kLdX + 8 * (q & 1) + (l == kNrcLayers - 1 ? warp * 16 : m0);
        const bf16* dr = Dl + (rr + 8 * (q & 1)) * kLdX + 8 * (q >> 1) + (l == kNrcLayers - 1 ? 0 : n0);
        uint32_t xa[2][2][4], b[2][2][4];
        auto load = [&](int kt) {
#pragma unroll
          for (int i = 0; i < (l == kNrcLayers - 1 ? 1 : 2); ++i) {
            ldsm_x4_t(xa[kt & 1][i], xr + kt * 16 * kLdX + 16 * i);
            ldsm_x4_t(b[kt & 1][i], dr + kt * 16 * kLdX + 16 * i);
          }
        };
        load(0);
#pragma unroll
        for (int kt = 0; kt < kTrainTile / 16; ++kt) {
          if (kt + 1 < kTrainTile / 16) load(kt + 1);
          const int u = kt & 1;
          if (l == kNrcLayers - 1) {
            mma_bf16(dwo[0], xa[u][0], b[u][0][0], b[u][0][1]);
            mma_bf16(dwo[1], xa[u][0], b[u][0][2], b[u][0][3]);
          } else {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                mma_bf16(dwh[l < kNrcHidden ? l : 0][i][j], xa[u][i], b[u][j >> 1][2 * (j & 1)],
                         b[u][j >> 1][2 * (j & 1) + 1]);
          }
        }
        if (l > 1 || more) bar_arrive<2>(kBarEmpty + buf);  // nobody waits for the CTA's last two
      }
      if (spare) bar_arrive<2>(kBarSpare + at);
    }
    // the CTA's gradient ([in][out] layout per layer) into its own slot of
    // gpart, every weight written (the warps' blocks cover each layer once);
    // nrc_grad_reduce_kernel sums the slots in a fixed order
    float* slot = gpart + (size_t)blockIdx.x * kNrcWeightCount;
#pragma unroll
    for (int l = 0; l < kNrcHidden; ++l)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float* base = slot + nrc_layer_offset(l) + (m0 + 16 * i + g) * kNrcWidth + n0 + j * 8 + 2 * t;
          *reinterpret_cast<float2*>(base) = make_float2(dwh[l][i][j][0], dwh[l][i][j][1]);
          *reinterpret_cast<float2*>(base + 8 * kNrcWidth) = make_float2(dwh[l][i][j][2], dwh[l][i][j][3]);
        }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float* base = slot + nrc_layer_offset(kNrcHidden) + (warp * 16 + g) * kNrcOutPad + j * 8 + 2 * t;
      *reinterpret_cast<float2*>(base) = make_float2(dwo[j][0], dwo[j][1]);
      *reinterpret_cast<float2*>(base + 8 * kNrcOutPad) = make_float2(dwo[j][2], dwo[j][3]);
    }
    return;
  }

  // chain warps
  set_regs_up<kRegsChain>();
  const bf16* xf = X + (warp * 32 + rr + 8 * (q & 1)) * kLdX + 8 * (q >> 1);  // the lane's rows of its warp's fragments
  const int row = warp * 32 + g;  // the lane's tile rows: row + 8 h, h = 0 .. 3 (fragment h / 2)
  const float inv_n = 1.0f / (3.0f * (float)max(count, 1u));
  float loss_local = 0.0f;
  uint32_t tile = 0;
#pragma unroll 1
  for (uint32_t first = start; first < count; first += stride, ++tile) {
    const int at = tile & 1;
    // the targets of the lane's output columns, for the loss below
    float target[4][2];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const float* tp = &recs[min(first + (uint32_t)row + 8u * h, count - 1u)].w0;
      target[h][0] = tp[t == 1 ? 2 : 0];
      target[h][1] = tp[1];
    }
    if (tile) bar_wait<2>(kBarInput + at);
    else bar_wait<3>(kBarFirst);
    uint32_t a[2][4][4];
    load_fragment(xf + (at ? kNrcLayers : 0) * kTileX, a[0]);
    load_fragment(xf + (at ? kNrcLayers : 0) * kTileX + 16 * kLdX, a[1]);
    uint32_t b[4][4][4];
    float acc[2][8][4];
    const auto none = [](int, int = 0) {};
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) load_in_out<4>(W, ldw(0), kt, b[kt], lane);
    chain_phase<4>(acc[0], a[0], b, none, none);
    if (tile > 0) bar_wait<2>(kBarEmpty + 0);  // the last tile's dW_1: X_1 .. X_5 and dY buffer 0 are free
    // turn l: fragment 1's layer l, then fragment 0's layer l + 1
#pragma unroll 1
    for (int l = 0; l < kNrcHidden - 1; ++l) {
      bf16* Xn = X + (l + 1) * kTileX;
      chain_phase<4>(
          acc[1], a[1], b, [&](int kt) { load_in_out<4>(W + woff(l + 1), ldw(0), kt, b[kt], lane); },
          [&](int kt, int p) {
            a[0][kt][p] = relu_word(acc[0], kt, p);
            store_word(Xn, row, t, kt, p, a[0][kt][p]);
          });
      chain_phase<4>(acc[0], a[0], b, none, [&](int kt, int p) {
        a[1][kt][p] = relu_word(acc[1], kt, p);
        store_word(Xn, row + 16, t, kt, p, a[1][kt][p]);
      });
    }
    {
      bf16* Xn = X + kNrcHidden * kTileX;
      chain_phase<4>(
          acc[1], a[1], b, [&](int kt) { load_in_out<1>(W + woff(kNrcHidden), ldw(kNrcHidden), kt, b[kt], lane); },
          [&](int kt, int p) {
            a[0][kt][p] = relu_word(acc[0], kt, p);
            store_word(Xn, row, t, kt, p, a[0][kt][p]);
          });
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        a[1][i >> 2][i & 3] = relu_word(acc[1], i >> 2, i & 3);
        store_word(Xn, row + 16, t, i >> 2, i & 3, a[1][i >> 2][i & 3]);
      }
    }
    // output layer (columns 0..7 of 16: the rest is padding) and the loss
    // gradient dY_5 (columns 0..2)
    float out[2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      out[m][0] = out[m][1] = out[m][2] = out[m][3] = 0.0f;
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) mma_bf16(out[m], a[m][kt], b[kt][0][0], b[kt][0][1]);
    }
    load_out_in(W + woff(kNrcHidden), ldw(kNrcHidden), 0, b[0], lane);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      float d5[4];  // (row, 2t), (row, 2t+1), (row+8, 2t), (row+8, 2t+1)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t idx = first + (uint32_t)row + 16u * m + 8u * h;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = 2 * t + e;
          float gval = 0.0f;
          if (c < kNrcOut && idx < count) {
            const float y = out[m][2 * h + e];
            const float den = y * y + 0.01f;
            const float diff = y - target[2 * m + h][e];
            const float rel = diff / den;
            loss_local += (diff * rel) * inv_n;
            gval = (2.0f * rel) * inv_n;
          }
          d5[2 * h + e] = gval;
        }
      }
      a[m][0][0] = pack_bf16(d5[0], d5[1]);
      a[m][0][1] = pack_bf16(d5[2], d5[3]);
      a[m][0][2] = 0u;  // columns 8..15: padding
      a[m][0][3] = 0u;
#pragma unroll
      for (int p = 0; p < 4; ++p) store_word(D, row + 16 * m, t, 0, p, a[m][0][p]);  // dY_5 in buffer 0
    }
    bar_arrive<2>(kBarFull + 0);
    // backward, from here a holds dY: dY_{l-1} = (dY_l W_l^T) * (X_l > 0) for
    // the warp's rows; layer 5 has one k-tile
    chain_phase<1>(acc[0], a[0], b, none, none);
    if (tile > 0) bar_wait<2>(kBarEmpty + 1);  // the last tile's dW_0
    {
      uint32_t x[4][4];  // X_5
      load_fragment(xf + kNrcHidden * kTileX, x);
      chain_phase<1>(
          acc[1], a[1], b, [&](int kt) { load_out_in(W + woff(kNrcHidden - 1), ldw(0), kt, b[kt], lane); },
          [&](int kt, int p) {
            a[0][kt][p] = mask_word(acc[0], kt, p, x[kt][p]);
            store_word(D + kTileX, row, t, kt, p, a[0][kt][p]);
          });
    }
    // turn l: dY_{l-1} of fragment 0, while dY_l of fragment 1 is finished,
    // then dY_{l-1} of fragment 1
#pragma unroll 1
    for (int l = kNrcHidden - 1; l >= 1; --l) {
      const int buf = (kNrcLayers - l) & 1;  // of dY_{l-1}
      uint32_t x[4][4];  // X_{l+1} of fragment 1, then X_l of fragment 0
      load_fragment(xf + (l + 1) * kTileX + 16 * kLdX, x);
      chain_phase<4>(acc[0], a[0], b, none, [&](int kt, int p) {
        a[1][kt][p] = mask_word(acc[1], kt, p, x[kt][p]);
        store_word(D + (buf ^ 1) * kTileX, row + 16, t, kt, p, a[1][kt][p]);
      });
      load_fragment(xf + l * kTileX, x);
      bar_arrive<2>(kBarFull + (buf ^ 1));  // dY_l
      bar_wait<2>(kBarEmpty + buf);         // the buffer's last reader, dW_{l+1}
      chain_phase<4>(
          acc[1], a[1], b,
          [&](int kt) {
            if (l > 1) load_out_in(W + woff(l - 1), ldw(0), kt, b[kt], lane);
          },
          [&](int kt, int p) {
            a[0][kt][p] = mask_word(acc[0], kt, p, x[kt][p]);
            store_word(D + buf * kTileX, row, t, kt, p, a[0][kt][p]);
          });
    }
    {
      uint32_t x[4][4];  // X_1
      load_fragment(xf + kTileX + 16 * kLdX, x);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        a[1][i >> 2][i & 3] = mask_word(acc[1], i >> 2, i & 3, x[i >> 2][i & 3]);
        store_word(D + kTileX, row + 16, t, i >> 2, i & 3, a[1][i >> 2][i & 3]);  // dY_0 in buffer 1
      }
      bar_arrive<2>(kBarFull + 1);
    }
    if (kGrid) {
      // dX_0 for inputs 0..31 (n-tiles 0..3): acc[nt] holds (row, 8nt+2t+e)
      // and (row+8, 8nt+2t+e), i.e. level 4nt+t, feature e
      const bf16* W0 = W + woff(0);
#pragma unroll 1
      for (int m = 0; m < 2; ++m) {
        float dx[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) dx[nt][0] = dx[nt][1] = dx[nt][2] = dx[nt][3] = 0.0f;
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
          uint32_t d0[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) d0[p] = m ? a[1][kt][p] : a[0][kt][p];
#pragma unroll
          for (int np = 0; np < 2; ++np) {
            uint32_t b0[4];
            ldsm_x4(b0, W0 + (np * 16 + rr + 8 * (q >> 1)) * ldw(0) + kt * 16 + 8 * (q & 1));
            mma_bf16(dx[2 * np], d0, b0[0], b0[1]);
            mma_bf16(dx[2 * np + 1], d0, b0[2], b0[3]);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t idx = first + (uint32_t)row + 16u * m + 8u * h;
          if (idx >= count) continue;
          const NrcRecord& rec = recs[idx];
          float ux, uy, uz;
          nrc_box_coords(rec, v.b0, v.inv_ext, ux, uy, uz);
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const int lv = 4 * nt + t;
            if (lv >= v.levels) continue;
            const float d0 = dx[nt][2 * h], d1 = dx[nt][2 * h + 1];
            const int n = nrc_grid_res(lv);
            const NrcGridCell c = nrc_grid_cell(n, ux, uy, uz);
            float* gl = v.ggrad + (size_t)lv * kNrcGridTable * 2;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const uint32_t e = nrc_grid_index(n, c.x + (k & 1), c.y + ((k >> 1) & 1), c.z + (k >> 2));
              const float w = nrc_grid_weight(c, k);
              atomicAdd(reinterpret_cast<float2*>(gl) + e, make_float2(w * d0, w * d1));
            }
          }
        }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) loss_local += __shfl_xor_sync(0xffffffffu, loss_local, o);
  if (lane == 0) atomicAdd(loss, loss_local);
}

// The optimiser state Adam updates, and the hyper-parameters of one step
// (bias corrections c1 = 1 - b1^t, c2 = 1 - b2^t; moving-average decay).
struct AdamView {
  float* w;
  bf16* wb;
  float* m;
  float* v;
  float* ema;
  bf16* wbi;
};
struct AdamStep {
  float lr, b1, b2, eps, c1, c2, decay;
};

constexpr int kReduceCols = 64;    // weights per reduction CTA
constexpr int kReduceGroups = 4;   // slot groups per weight (b mod 4)
constexpr int kReduceUnroll = 8;   // independent loads in flight per thread
static_assert(kNrcWeightCount % kReduceCols == 0, "reduction tiling");

// Sums the slots of the CTAs that had records (the first
// ceil(count / kTrainTile)) in a fixed order: thread group g adds slots
// g, g+4, g+8, ... into eight partial sums (slot g + 4u + 32k into sum u),
// combined pairwise, then the four groups in order.  Without kAdam the sum
// is added to grad; with kAdam the Adam step follows on grad + sum and grad
// is cleared.  One launch of kNrcWeightCount / 64 CTAs: every weight's 152
// loads are spread over four threads with eight in flight each.  Its first
// thread also moves the step's loss sum to loss[1] and clears loss[0] for
// the next step's training kernel.
template <bool kAdam>
__global__ void __launch_bounds__(kReduceCols * kReduceGroups)
    nrc_grad_reduce_kernel(const float* __restrict__ gpart, int blocks, const uint32_t* __restrict__ count_ptr,
                           uint32_t capacity, uint32_t first_rec, float* __restrict__ grad, AdamView a, AdamStep h,
                           float* __restrict__ loss) {
  __shared__ float part[kReduceGroups][kReduceCols];
  grid_wait();
  grid_trigger();
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // the step's loss, and a zero sum for the next step
    loss[1] = loss[0];
    loss[0] = 0.0f;
  }
  const int col = threadIdx.x % kReduceCols, grp = threadIdx.x / kReduceCols;
  const int i = blockIdx.x * kReduceCols + col;
  const uint32_t total = *count_ptr;
  const uint32_t count = total > first_rec ? min(total - first_rec, capacity) : 0u;
  const int active = (int)min((uint32_t)blocks, (count + kTrainTile - 1) / kTrainTile);
  float s[kReduceUnroll];
#pragma unroll
  for (int u = 0; u < kReduceUnroll; ++u) s[u] = 0.0f;
  constexpr int kStride = kReduceGroups * kReduceUnroll;
  int b = grp;
  for (; b + kStride - kReduceGroups < active; b += kStride) {
    float x[kReduceUnroll];
#pragma unroll
    for (int u = 0; u < kReduceUnroll; ++u) x[u] = gpart[(size_t)(b + kReduceGroups * u) * kNrcWeightCount + i];
#pragma unroll
    for (int u = 0; u < kReduceUnroll; ++u) s[u] += x[u];
  }
#pragma unroll
  for (int u = 0; u < kReduceUnroll; ++u)  // the last slots of the group: < 8 of them
    if (b + kReduceGroups * u < active) s[u] += gpart[(size_t)(b + kReduceGroups * u) * kNrcWeightCount + i];
  part[grp][col] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
  __syncthreads();
  if (grp != 0) return;
  const float sum = (part[0][col] + part[1][col]) + (part[2][col] + part[3][col]);
  if (!kAdam) {
    grad[i] += sum;
    return;
  }
  const float gi = grad[i] + sum;
  const float mi = h.b1 * a.m[i] + (1.0f - h.b1) * gi;
  const float vi = h.b2 * a.v[i] + (1.0f - h.b2) * gi * gi;
  a.m[i] = mi;
  a.v[i] = vi;
  const float wi = a.w[i] - h.lr * (mi / h.c1) / (sqrtf(vi / h.c2) + h.eps);
  a.w[i] = wi;
  a.wb[i] = __float2bfloat16_rn(wi);
  grad[i] = 0.0f;
  if (a.ema) {
    const float e = h.decay * a.ema[i] + (1.0f - h.decay) * wi;
    a.ema[i] = e;
    a.wbi[i] = __float2bfloat16_rn(e);
  }
}

__global__ void nrc_copy_weights_kernel(const float* __restrict__ w, float* __restrict__ ema, bf16* __restrict__ wbi) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kNrcWeightCount) {
    ema[i] = w[i];
    wbi[i] = __float2bfloat16_rn(w[i]);
  }
}

__global__ void nrc_to_bf16_kernel(const float* __restrict__ w, bf16* __restrict__ wb) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kNrcWeightCount) wb[i] = __float2bfloat16_rn(w[i]);
}

// Adam step on the grid encoding's tables (step size h.lr x
// kNrcGridLrScale), clearing their gradient; the moving average as for the
// weights.
__global__ void nrc_grid_adam_kernel(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                                     float* __restrict__ grad, float* __restrict__ ema, AdamStep h) {
  const float lr = h.lr * kNrcGridLrScale;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < kNrcGridParams;
       i += (size_t)gridDim.x * blockDim.x) {
    const float gi = grad[i];
    const float mi = h.b1 * m[i] + (1.0f - h.b1) * gi;
    const float vi = h.b2 * v[i] + (1.0f - h.b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / h.c1) / (sqrtf(vi / h.c2) + h.eps);
    w[i] = wi;
    grad[i] = 0.0f;
    if (ema) ema[i] = h.decay * ema[i] + (1.0f - h.decay) * wi;
  }
}

// The tables' initial values: uniform in [-1e-4, 1e-4] from a seeded hash
// (the moving average starts equal).
__global__ void nrc_grid_init_kernel(float* __restrict__ w, float* __restrict__ ema, uint32_t seed) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < kNrcGridParams;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t hsh = pcg_hash(seed ^ 0x9E3779B9u ^ pcg_hash((uint32_t)i));
    const float u = (float)(hsh >> 8) * 5.96046448e-08f;  // [0,1)
    const float x = (2.0f * u - 1.0f) * 1e-4f;
    w[i] = x;
    if (ema) ema[i] = x;
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static size_t infer_smem() { return (size_t)kWs * 2 + kNrcPosLevels * 3 * sizeof(float); }
static size_t train_smem() {
  return (size_t)kWs * 2 + (size_t)(kNrcLayers + 3) * kTileX * 2 + kNrcPosLevels * 3 * sizeof(float);
}

size_t nrc_param_count(const NrcState* st) {
  return (size_t)kNrcWeightCount + (st && st->gw ? kNrcGridParams : 0);
}

NrcView nrc_view(const vcr_ctx* ctx) {
  NrcView v;
  v.wb = reinterpret_cast<const bf16*>(ctx->nrc->wb);
  v.wbi = reinterpret_cast<const bf16*>(ctx->nrc->wbi ? ctx->nrc->wbi : ctx->nrc->wb);
  const vcr_cloud& c = ctx->cloud;
  v.b0 = mk(c.bounds_min[0], c.bounds_min[1], c.bounds_min[2]);
  v.inv_ext = mk(1.0f / (c.bounds_max[0] - c.bounds_min[0]), 1.0f / (c.bounds_max[1] - c.bounds_min[1]),
                 1.0f / (c.bounds_max[2] - c.bounds_min[2]));
  v.levels = kNrcPosLevels - (int)ctx->nrc->prm.position_drop;
  const NrcState* st = ctx->nrc;
  v.gtab = st->gw;
  v.gtab_i = st->gema ? st->gema : st->gw;
  v.ggrad = st->ggrad;
  return v;
}

void nrc_free(vcr_ctx* ctx) {
  NrcState* st = ctx->nrc;
  if (!st) return;
  void* ptrs[] = {st->w,      st->wb,          st->m,     st->v,           st->grad, st->gpart, st->ema,
                  st->wbi,    st->loss,        st->train, st->train_count, st->query, st->query_count,
                  st->gw,     st->gm,          st->gv,    st->ggrad,       st->gema};
  for (void* p : ptrs) cudaFree(p);
  delete st;
  ctx->nrc = nullptr;
}

// Kaiming-uniform initial weights from a seeded hash (host).
static void nrc_init_weights(std::vector<float>& w, uint32_t seed) {
  w.assign(kNrcWeightCount, 0.0f);
  uint32_t c = 0;
  for (int l = 0; l < kNrcLayers; ++l) {
    int cols = nrc_layer_cols(l);
    float bound = l < kNrcHidden ? sqrtf(6.0f / (float)kNrcWidth) : sqrtf(1.0f / (float)kNrcWidth);
    for (int i = 0; i < kNrcWidth; ++i)
      for (int o = 0; o < cols; ++o) {
        uint32_t hsh = pcg_hash(seed ^ pcg_hash(c++));
        float u = (float)(hsh >> 8) * 5.96046448e-08f;  // [0,1)
        w[(size_t)nrc_layer_offset(l) + (size_t)i * cols + o] =
            (l == kNrcLayers - 1 && o >= kNrcOut) ? 0.0f : (2.0f * u - 1.0f) * bound;
      }
  }
}

vcr_status nrc_setup(vcr_ctx* ctx, const vcr_nrc_params* p) {
  if (!p || p->train_samples == 0 || p->train_samples > (1u << 22) || !(p->learning_rate > 0.0f) ||
      p->query_capacity == 0 || !(p->ema_decay >= 0.0f && p->ema_decay < 1.0f) ||
      !(p->tail_survival >= 0.0f && p->tail_survival < 1.0f) || p->query_kernel > VCR_NRC_QUERY_TCGEN05 ||
      p->position_drop > (uint32_t)kNrcPosLevels || p->encoding > VCR_NRC_ENCODING_GRID)
    return fail(ctx, VCR_ERR_INVALID,
                "nrc params: train_samples 1..2^22, learning_rate > 0, query_capacity > 0, ema_decay and "
                "tail_survival in [0,1), query_kernel a VCR_NRC_QUERY_* value, position_drop 0..16, encoding a "
                "VCR_NRC_ENCODING_* value");
  nrc_free(ctx);
  NrcState* st = new NrcState();
  ctx->nrc = st;
  st->prm = *p;
  st->query_capacity = p->query_capacity;
  st->train_cap = 2 * p->train_samples;
#define VCR_ALLOC(ptr, bytes) VCR_CUDA(ctx, cudaMalloc(reinterpret_cast<void**>(&(ptr)), (bytes)))
  VCR_ALLOC(st->w, kNrcWeightCount * 4);
  VCR_ALLOC(st->wb, kNrcWeightCount * 2);
  VCR_ALLOC(st->m, kNrcWeightCount * 4);
  VCR_ALLOC(st->v, kNrcWeightCount * 4);
  VCR_ALLOC(st->grad, kNrcWeightCount * 4);
  st->gpart_blocks = ctx->sm_count;
  VCR_ALLOC(st->gpart, (size_t)st->gpart_blocks * kNrcWeightCount * 4);
  VCR_ALLOC(st->loss, 8);
  VCR_ALLOC(st->train, (size_t)st->train_cap * sizeof(NrcRecord));
  if (p->ema_decay > 0.0f) {
    VCR_ALLOC(st->ema, kNrcWeightCount * 4);
    VCR_ALLOC(st->wbi, kNrcWeightCount * 2);
  }
  VCR_ALLOC(st->train_count, 4);
  VCR_ALLOC(st->query, (size_t)p->query_capacity * sizeof(NrcRecord));
  VCR_ALLOC(st->query_count, 4);
  if (p->encoding == VCR_NRC_ENCODING_GRID) {
    VCR_ALLOC(st->gw, kNrcGridParams * 4);
    VCR_ALLOC(st->gm, kNrcGridParams * 4);
    VCR_ALLOC(st->gv, kNrcGridParams * 4);
    VCR_ALLOC(st->ggrad, kNrcGridParams * 4);
    if (p->ema_decay > 0.0f) VCR_ALLOC(st->gema, kNrcGridParams * 4);
  }
#undef VCR_ALLOC
  VCR_CUDA(ctx, cudaMemset(st->train_count, 0, 4));
  VCR_CUDA(ctx, cudaMemset(st->loss, 0, 8));
  std::vector<float> w;
  nrc_init_weights(w, p->seed);
  VCR_CUDA(ctx, cudaMemcpy(st->w, w.data(), kNrcWeightCount * 4, cudaMemcpyHostToDevice));
  VCR_CUDA(ctx, cudaMemset(st->m, 0, kNrcWeightCount * 4));
  VCR_CUDA(ctx, cudaMemset(st->v, 0, kNrcWeightCount * 4));
  VCR_CUDA(ctx, cudaMemset(st->grad, 0, kNrcWeightCount * 4));
  VCR_CUDA(ctx, cudaMemset(st->query_count, 0, 4));
  nrc_to_bf16_kernel<<<(kNrcWeightCount + 255) / 256, 256>>>(st->w, reinterpret_cast<bf16*>(st->wb));
  VCR_CUDA(ctx, cudaGetLastError());
  if (st->ema) {
    nrc_copy_weights_kernel<<<(kNrcWeightCount + 255) / 256, 256>>>(st->w, st->ema, reinterpret_cast<bf16*>(st->wbi));
    VCR_CUDA(ctx, cudaGetLastError());
  }
  if (st->gw) {
    VCR_CUDA(ctx, cudaMemset(st->gm, 0, kNrcGridParams * 4));
    VCR_CUDA(ctx, cudaMemset(st->gv, 0, kNrcGridParams * 4));
    VCR_CUDA(ctx, cudaMemset(st->ggrad, 0, kNrcGridParams * 4));
    nrc_grid_init_kernel<<<ctx->sm_count * 8, 256>>>(st->gw, st->gema, p->seed);
    VCR_CUDA(ctx, cudaGetLastError());
  }
  VCR_CUDA(ctx, cudaFuncSetAttribute(nrc_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)infer_smem()));
  VCR_CUDA(ctx, cudaFuncSetAttribute(nrc_train_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)train_smem()));
  VCR_CUDA(ctx, cudaFuncSetAttribute(nrc_train_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)train_smem()));
  return VCR_OK;
}

template <class... P, class... A>
static cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                     A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Gradient of the loss over records [first, first + capacity) of the
// *d_count written (device): added to grad, or (adam) followed by one Adam
// step in the same reduction launch.
static vcr_status nrc_grad(vcr_ctx* ctx, const NrcRecord* recs, const uint32_t* d_count, uint32_t capacity,
                           cudaStream_t s, uint32_t first, bool adam) {
  NrcState* st = ctx->nrc;
  const int blocks = st->gpart_blocks;
  const auto train = st->gw ? nrc_train_kernel<true> : nrc_train_kernel<false>;
  VCR_CUDA(ctx, cudaFuncSetAttribute(train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem()));
  VCR_CUDA(ctx, launch_overlapped(train, dim3(blocks), dim3(kTrainThreads), train_smem(), s, nrc_view(ctx), recs, d_count,
                                  capacity, first, st->gpart, st->loss));
  AdamView a{st->w, reinterpret_cast<bf16*>(st->wb), st->m, st->v, st->ema, reinterpret_cast<bf16*>(st->wbi)};
  AdamStep h{};
  if (adam) {
    st->step += 1;
    h.lr = st->prm.learning_rate;
    h.b1 = 0.9f;
    h.b2 = 0.99f;
    h.eps = 1e-8f;
    h.c1 = 1.0f - (float)std::pow(0.9, (double)st->step);
    h.c2 = 1.0f - (float)std::pow(0.99, (double)st->step);
    // moving-average decay ramps up over the first steps: min(d, (1+k)/(10+k))
    h.decay = std::min(st->prm.ema_decay, (1.0f + (float)st->step) / (10.0f + (float)st->step));
  }
  const dim3 grid(kNrcWeightCount / kReduceCols), block(kReduceCols * kReduceGroups);
  const auto reduce = adam ? nrc_grad_reduce_kernel<true> : nrc_grad_reduce_kernel<false>;
  VCR_CUDA(ctx, launch_overlapped(reduce, grid, block, 0, s, st->gpart, blocks, d_count, capacity, first, st->grad, a, h,
                                  st->loss));
  if (adam && st->gw) {
    nrc_grid_adam_kernel<<<ctx->sm_count * 8, 256, 0, s>>>(st->gw, st->gm, st->gv, st->ggrad, st->gema, h);
    VCR_CUDA(ctx, cudaGetLastError());
  }
  return VCR_OK;
}

// BF16 copies from the FP32 master weights and their moving average (after
// the FP32 state was written from outside, e.g. a checkpoint).
vcr_status nrc_refresh_copies(vcr_ctx* ctx) {
  NrcState* st = ctx->nrc;
  nrc_to_bf16_kernel<<<(kNrcWeightCount + 255) / 256, 256>>>(st->w, reinterpret_cast<bf16*>(st->wb));
  VCR_CUDA(ctx, cudaGetLastError());
  if (st->ema) {
    nrc_to_bf16_kernel<<<(kNrcWeightCount + 255) / 256, 256>>>(st->ema, reinterpret_cast<bf16*>(st->wbi));
    VCR_CUDA(ctx, cudaGetLastError());
  }
  return VCR_OK;
}

uint32_t nrc_query_capacity(const vcr_ctx* ctx) { return ctx->nrc ? ctx->nrc->query_capacity : 0u; }

vcr_status nrc_reset_queries(vcr_ctx* ctx, cudaStream_t s) {
  VCR_CUDA(ctx, cudaMemsetAsync(ctx->nrc->query_count, 0, 4, s));
  return VCR_OK;
}

// Which kernel serves the queries (vcr_nrc_params.query_kernel).
static bool use_tc(const NrcState* st) { return st->prm.query_kernel == VCR_NRC_QUERY_TCGEN05; }

vcr_status nrc_infer_queries(vcr_ctx* ctx, cudaStream_t s) {
  NrcState* st = ctx->nrc;
  if (use_tc(st)) {
    const NrcView v = nrc_view(ctx);
    return nrc_infer_tc_launch(ctx, v.wbi, v.b0, v.inv_ext, v.levels, v.gtab_i, st->query, st->query_count,
                               st->query_capacity, ctx->d_sum, nullptr, s);
  }
  VCR_CUDA(ctx, cudaFuncSetAttribute(nrc_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)infer_smem()));
  int per_sm = 0;
  VCR_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, nrc_infer_kernel, kInferThreads, infer_smem()));
  int blocks = ctx->sm_count * std::max(per_sm, 1);
  nrc_infer_kernel<<<blocks, kInferThreads, infer_smem(), s>>>(nrc_view(ctx), st->query, st->query_count,
                                                               st->query_capacity, ctx->d_sum, nullptr);
  VCR_CUDA(ctx, cudaGetLastError());
  return VCR_OK;
}

static vcr_status nrc_check_scene(vcr_ctx* ctx, const char* who) {
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "%s needs vcr_nrc_setup", who);
  if (!ctx->has_grid || !ctx->has_cloud || !ctx->has_cam || !ctx->has_params || !ctx->d_sum)
    return fail(ctx, VCR_ERR_STATE, "%s needs a grid, cloud, camera, params and frame", who);
  return VCR_OK;
}

static bool nrc_calibrated(const vcr_ctx* ctx) {
  const NrcState* st = ctx->nrc;
  return st->npaths && !memcmp(&st->calib_cam, &ctx->cam, sizeof(vcr_camera)) &&
         !memcmp(&st->calib_cloud, &ctx->cloud, sizeof(vcr_cloud)) && st->calib_w == ctx->width &&
         st->calib_h == ctx->height;
}

// Training paths: extended paths from uniformly drawn pixels that record
// the radiance leaving each of their first kNrcRecordEvents scattering
// vertices toward the previous vertex, target_i = (L_total - L_before_i) /
// beta_i.  They run in the persistent wavefront kernel, alone
// (vcr_nrc_train_step) or as the first work items of a pass (vcr_nrc_frame),
// where their long paths overlap the pass's short ones.  The first step for
// a camera/cloud/frame calibrates the path count so that a step yields
// about train_samples records (synchronises once; deterministic, as the
// yield of a seeded launch is).  A step with pass.spp = S > 1 traces S
// sets of paths in its one launch: a training-only launch is as long as
// its longest path, so S sets take far less than S launches (0.95 ms for
// four sets against 0.65 ms for one on the 1920x1080 cloud scene).
static NrcTrainSink nrc_sink(vcr_ctx* ctx) {
  NrcState* st = ctx->nrc;
  return NrcTrainSink{st->train, st->train_count, st->train_cap, st->npaths, st->prm.tail_survival};
}

static vcr_status nrc_launch_training(vcr_ctx* ctx, const PassView& pv, uint32_t paths, cudaStream_t s) {
  NrcTrainSink ts = nrc_sink(ctx);
  ts.paths = paths;
  VCR_CUDA(ctx, cudaMemsetAsync(ts.count, 0, 4, s));
  VCR_CUDA(ctx, cudaMemsetAsync(ctx->d_counters, 0, kPassCounterBytes, s));
  return wavefront_launch(ctx, grid_view(ctx), scene_view(ctx), cam_view(ctx->cam), pv, nullptr,
                          Counters{ctx->d_counters}, 0u, s, &ts);
}

static vcr_status nrc_calibrate(vcr_ctx* ctx, const PassView& pv, cudaStream_t s) {
  NrcState* st = ctx->nrc;
  const uint32_t want = st->prm.train_samples, paths = std::max(1u, want / 2);
  vcr_status vs = nrc_launch_training(ctx, pv, paths, s);
  if (vs) return vs;
  uint32_t got = 0;
  VCR_CUDA(ctx, cudaMemcpyAsync(&got, st->train_count, 4, cudaMemcpyDeviceToHost, s));
  VCR_CUDA(ctx, cudaStreamSynchronize(s));
  double n = std::ceil((double)paths * (double)want / (double)std::max(got, 1u));
  st->npaths = (uint32_t)std::min(std::max(n, (double)std::max(1u, want / 4)), 16.0 * (double)want);
  st->calib_cam = ctx->cam;
  st->calib_cloud = ctx->cloud;
  st->calib_w = ctx->width;
  st->calib_h = ctx->height;
  return VCR_OK;
}

// Loss gradient over the step's records, then Adam.
static vcr_status nrc_update(vcr_ctx* ctx, cudaStream_t s, uint32_t first = 0, uint32_t limit = 0) {
  NrcState* st = ctx->nrc;
  return nrc_grad(ctx, st->train, st->train_count, limit ? limit : st->train_cap, s, first, true);
}

// Record room for `sets` training sets; growing the buffer synchronises.
static vcr_status nrc_reserve_sets(vcr_ctx* ctx, uint32_t sets) {
  NrcState* st = ctx->nrc;
  const uint64_t cap = 2ull * st->prm.train_samples * sets;
  if (sets > kNrcMaxSets || cap > (1ull << 25))
    return fail(ctx, VCR_ERR_INVALID, "training sets (pass.spp) 1..%u with sets x train_samples <= 2^24", kNrcMaxSets);
  if (cap <= st->train_cap) return VCR_OK;
  VCR_CUDA(ctx, cudaDeviceSynchronize());
  VCR_CUDA(ctx, cudaFree(st->train));
  st->train = nullptr;
  st->train_cap = 0;
  VCR_CUDA(ctx, cudaMalloc(reinterpret_cast<void**>(&st->train), (size_t)cap * sizeof(NrcRecord)));
  st->train_cap = (uint32_t)cap;
  return VCR_OK;
}

vcr_status nrc_train_step(vcr_ctx* ctx, const vcr_pass_desc* pass, cudaStream_t s) {
  vcr_status vs = nrc_check_scene(ctx, "vcr_nrc_train_step");
  if (vs) return vs;
  PassView pv;
  vs = make_pass_view(ctx, pass, pv);
  if (vs) return vs;
  const uint32_t sets = pv.spp;
  vs = nrc_reserve_sets(ctx, sets);
  if (vs) return vs;
  NrcState* st = ctx->nrc;
  if (!nrc_calibrated(ctx)) {
    vs = nrc_calibrate(ctx, pv, s);  // its records serve a one-set step
    if (!vs && sets > 1) vs = nrc_launch_training(ctx, pv, st->npaths * sets, s);
  } else {
    vs = nrc_launch_training(ctx, pv, st->npaths * sets, s);
  }
  if (vs) return vs;
  st->records = true;
  st->sets = sets;
  // one set: a step over all its records; several: over the first
  // train_samples, and vcr_nrc_train_more continues after them
  vs = sets == 1 ? nrc_update(ctx, s) : nrc_update(ctx, s, 0, st->prm.train_samples);
  if (vs) return vs;
  st->cursor = sets == 1 ? 0u : st->prm.train_samples;
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, s));
  return VCR_OK;
}

// One frame of the cached tracker: one wavefront launch runs this frame's
// training paths first and the pass's camera paths after them (the latter
// end in the cache at nrc_events, queried with the weights before this
// frame's update), then the loss gradient and Adam.  Same result as
// vcr_pt_pass followed by vcr_nrc_train_step with the same pass.
vcr_status nrc_frame(vcr_ctx* ctx, const vcr_pass_desc* pass, cudaStream_t s) {
  vcr_status vs = nrc_check_scene(ctx, "vcr_nrc_frame");
  if (vs) return vs;
  if (ctx->params.nrc_events == 0 || ctx->params.tracker != VCR_TRACKER_DDA)
    return fail(ctx, VCR_ERR_STATE, "vcr_nrc_frame needs the DDA tracker and params.nrc_events > 0");
  PassView pv;
  vs = make_pass_view(ctx, pass, pv);
  if (vs) return vs;
  if (!nrc_calibrated(ctx)) {  // the calibration synchronises: training launch first, then the pass
    vs = nrc_calibrate(ctx, pv, s);
    if (vs) return vs;
    vs = pt_pass_launch(ctx, pass, s);
  } else {
    NrcTrainSink ts = nrc_sink(ctx);
    VCR_CUDA(ctx, cudaMemsetAsync(ts.count, 0, 4, s));
    vs = pt_pass_launch(ctx, pass, s, &ts);
  }
  if (vs) return vs;
  ctx->nrc->records = true;
  ctx->nrc->sets = 1;
  ctx->nrc->cursor = 0;
  vs = nrc_update(ctx, s);
  if (vs) return vs;
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, s));
  return VCR_OK;
}

}  // namespace vcr

using namespace vcr;

extern "C" VCR_API vcr_status vcr_nrc_setup(vcr_ctx* ctx, const vcr_nrc_params* p) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  vcr_status st = nrc_setup(ctx, p);
  if (st) return st;
  VCR_CUDA(ctx, cudaDeviceSynchronize());
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_nrc_free(vcr_ctx* ctx) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaDeviceSynchronize();
  nrc_free(ctx);
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_nrc_train_step(vcr_ctx* ctx, const vcr_pass_desc* pass, void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!pass) return fail(ctx, VCR_ERR_INVALID, "null pass");
  return nrc_train_step(ctx, pass, (cudaStream_t)stream);
}

extern "C" VCR_API vcr_status vcr_nrc_train_more(vcr_ctx* ctx, uint32_t steps, uint32_t max_records,
                                                 void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  if (!ctx->nrc->records)
    return fail(ctx, VCR_ERR_STATE, "no training records (vcr_nrc_train_step or vcr_nrc_frame first)");
  cudaStream_t s = (cudaStream_t)stream;
  NrcState* st = ctx->nrc;
  const uint32_t want = st->prm.train_samples * st->sets;
  const uint32_t batch = (max_records && max_records < want) ? max_records : 0u;
  for (uint32_t k = 0; k < steps; ++k) {
    // consecutive steps, and consecutive calls, walk through the records
    // batch by batch, from the start again after the last whole batch
    if (batch && st->cursor + batch > want) st->cursor = 0;
    vcr_status vs = batch ? nrc_update(ctx, s, st->cursor, batch) : nrc_update(ctx, s);
    if (vs) return vs;
    if (batch) st->cursor += batch;
  }
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, s));
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_nrc_set_learning_rate(vcr_ctx* ctx, float learning_rate) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  if (!(learning_rate > 0.0f) || !std::isfinite(learning_rate))
    return fail(ctx, VCR_ERR_INVALID, "learning rate must be finite and > 0");
  ctx->nrc->prm.learning_rate = learning_rate;  // read on the host when the next step is enqueued
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_nrc_frame(vcr_ctx* ctx, const vcr_pass_desc* pass, void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!pass) return fail(ctx, VCR_ERR_INVALID, "null pass");
  return nrc_frame(ctx, pass, (cudaStream_t)stream);
}

extern "C" VCR_API vcr_status vcr_nrc_info(vcr_ctx* ctx, vcr_nrc_info_t* out) {
  if (!ctx || !out) return fail(ctx, VCR_ERR_INVALID, "null argument");
  NrcState* st = ctx->nrc;
  if (!st) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  VCR_CUDA(ctx, cudaEventSynchronize(ctx->work_done));
  float loss = 0.0f;
  uint32_t ntrain = 0, nq = 0;
  VCR_CUDA(ctx, cudaMemcpy(&loss, st->loss + 1, 4, cudaMemcpyDeviceToHost));
  VCR_CUDA(ctx, cudaMemcpy(&ntrain, st->train_count, 4, cudaMemcpyDeviceToHost));
  VCR_CUDA(ctx, cudaMemcpy(&nq, st->query_count, 4, cudaMemcpyDeviceToHost));
  out->steps = st->step;
  out->last_loss = loss;
  out->train_records = std::min(ntrain, st->train_cap);
  out->queries = std::min(nq, st->query_capacity);
  out->weights = (uint32_t)nrc_param_count(st);
  return VCR_OK;
}

// `count` is the network's weight count, or (grid encoding) the full
// parameter count with the tables after the weights.
static vcr_status nrc_check_count(vcr_ctx* ctx, size_t count) {
  const size_t all = nrc_param_count(ctx->nrc);
  if (count != (size_t)kNrcWeightCount && count != all)
    return fail(ctx, VCR_ERR_INVALID, "the cache has %d weights (%zu parameters with the grid tables)",
                kNrcWeightCount, all);
  return VCR_OK;
}

// Weights: FP32 master copy in the layer layout of vcr_nrc_params.
extern "C" VCR_API vcr_status vcr_nrc_get_weights(vcr_ctx* ctx, float* host, size_t count) {
  if (!ctx || !host) return fail(ctx, VCR_ERR_INVALID, "null argument");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  vcr_status cs = nrc_check_count(ctx, count);
  if (cs) return cs;
  VCR_CUDA(ctx, cudaEventSynchronize(ctx->work_done));
  VCR_CUDA(ctx, cudaMemcpy(host, ctx->nrc->w, kNrcWeightCount * 4, cudaMemcpyDeviceToHost));
  if (count > (size_t)kNrcWeightCount)
    VCR_CUDA(ctx, cudaMemcpy(host + kNrcWeightCount, ctx->nrc->gw, kNrcGridParams * 4, cudaMemcpyDeviceToHost));
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_nrc_set_weights(vcr_ctx* ctx, const float* host, size_t count) {
  if (!ctx || !host) return fail(ctx, VCR_ERR_INVALID, "null argument");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  vcr_status cs = nrc_check_count(ctx, count);
  if (cs) return cs;
  VCR_CUDA(ctx, cudaDeviceSynchronize());
  VCR_CUDA(ctx, cudaMemcpy(ctx->nrc->w, host, kNrcWeightCount * 4, cudaMemcpyHostToDevice));
  if (count > (size_t)kNrcWeightCount) {
    VCR_CUDA(ctx, cudaMemcpy(ctx->nrc->gw, host + kNrcWeightCount, kNrcGridParams * 4, cudaMemcpyHostToDevice));
    if (ctx->nrc->gema)
      VCR_CUDA(ctx, cudaMemcpy(ctx->nrc->gema, ctx->nrc->gw, kNrcGridParams * 4, cudaMemcpyDeviceToDevice));
  }
  nrc_to_bf16_kernel<<<(kNrcWeightCount + 255) / 256, 256>>>(ctx->nrc->w, reinterpret_cast<bf16*>(ctx->nrc->wb));
  VCR_CUDA(ctx, cudaGetLastError());
  if (ctx->nrc->ema) {
    nrc_copy_weights_kernel<<<(kNrcWeightCount + 255) / 256, 256>>>(ctx->nrc->w, ctx->nrc->ema,
                                                                     reinterpret_cast<bf16*>(ctx->nrc->wbi));
    VCR_CUDA(ctx, cudaGetLastError());
  }
  VCR_CUDA(ctx, cudaDeviceSynchronize());
  return VCR_OK;
}

// Evaluate the cache on n records (device NrcRecord array, 64 B each);
// writes 3 floats per record to d_out.  For tests and tools.
extern "C" VCR_API vcr_status vcr_nrc_forward(vcr_ctx* ctx, const void* d_records, uint32_t n, float* d_out,
                                              void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  if (n == 0) return VCR_OK;
  if (!d_records || !d_out) return fail(ctx, VCR_ERR_INVALID, "null buffer");
  if (!ctx->has_cloud) return fail(ctx, VCR_ERR_STATE, "the encoding needs the cloud box (vcr_set_cloud)");
  cudaStream_t s = (cudaStream_t)stream;
  vcr_status vs = ensure_scratch(ctx, 4);
  if (vs) return vs;
  uint32_t* d_n = reinterpret_cast<uint32_t*>(ctx->d_scratch);
  VCR_CUDA(ctx, cudaMemcpyAsync(d_n, &n, 4, cudaMemcpyHostToDevice, s));
  if (use_tc(ctx->nrc)) {
    const NrcView v = nrc_view(ctx);
    vs = nrc_infer_tc_launch(ctx, v.wbi, v.b0, v.inv_ext, v.levels, v.gtab_i,
                             reinterpret_cast<const NrcRecord*>(d_records), d_n, n, nullptr, d_out, s);
    if (vs) return vs;
  } else {
    VCR_CUDA(ctx, cudaFuncSetAttribute(nrc_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)infer_smem()));
    nrc_infer_kernel<<<ctx->sm_count * 3, kInferThreads, infer_smem(), s>>>(
        nrc_view(ctx), reinterpret_cast<const NrcRecord*>(d_records), d_n, n, nullptr, d_out);
    VCR_CUDA(ctx, cudaGetLastError());
  }
  VCR_CUDA(ctx, cudaStreamSynchronize(s));
  return VCR_OK;
}

// `steps` Adam steps on n caller records (targets in w0..w2).
extern "C" VCR_API vcr_status vcr_nrc_fit(vcr_ctx* ctx, const void* d_records, uint32_t n, uint32_t steps,
                                          void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  if (!d_records || n == 0) return fail(ctx, VCR_ERR_INVALID, "bad fit arguments");
  if (!ctx->has_cloud) return fail(ctx, VCR_ERR_STATE, "the encoding needs the cloud box (vcr_set_cloud)");
  cudaStream_t s = (cudaStream_t)stream;
  vcr_status vs = ensure_scratch(ctx, 4);
  if (vs) return vs;
  uint32_t* d_n = reinterpret_cast<uint32_t*>(ctx->d_scratch);
  VCR_CUDA(ctx, cudaMemcpyAsync(d_n, &n, 4, cudaMemcpyHostToDevice, s));
  for (uint32_t k = 0; k < steps; ++k) {
    vs = nrc_grad(ctx, reinterpret_cast<const NrcRecord*>(d_records), d_n, n, s, 0, true);
    if (vs) return vs;
  }
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, s));
  return VCR_OK;
}

// Loss gradient over n records (targets in w0..w2), without an update:
// copies the gradient to host (count = weight count) and returns the loss.
extern "C" VCR_API vcr_status vcr_nrc_gradient(vcr_ctx* ctx, const void* d_records, uint32_t n, float* host_grad,
                                               size_t count, float* out_loss) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->nrc) return fail(ctx, VCR_ERR_STATE, "no radiance cache");
  if (!d_records || !host_grad || n == 0) return fail(ctx, VCR_ERR_INVALID, "bad gradient arguments");
  vcr_status cs = nrc_check_count(ctx, count);
  if (cs) return cs;
  if (!ctx->has_cloud) return fail(ctx, VCR_ERR_STATE, "the encoding needs the cloud box (vcr_set_cloud)");
  vcr_status vs = ensure_scratch(ctx, 4);
  if (vs) return vs;
  uint32_t* d_n = reinterpret_cast<uint32_t*>(ctx->d_scratch);
  VCR_CUDA(ctx, cudaMemcpy(d_n, &n, 4, cudaMemcpyHostToDevice));
  NrcState* st = ctx->nrc;
  VCR_CUDA(ctx, cudaMemset(st->grad, 0, kNrcWeightCount * 4));
  if (st->ggrad) VCR_CUDA(ctx, cudaMemset(st->ggrad, 0, kNrcGridParams * 4));
  vs = nrc_grad(ctx, reinterpret_cast<const NrcRecord*>(d_records), d_n, n, 0, 0, false);
  if (vs) return vs;
  VCR_CUDA(ctx, cudaDeviceSynchronize());
  VCR_CUDA(ctx, cudaMemcpy(host_grad, st->grad, kNrcWeightCount * 4, cudaMemcpyDeviceToHost));
  if (count > (size_t)kNrcWeightCount)
    VCR_CUDA(ctx, cudaMemcpy(host_grad + kNrcWeightCount, st->ggrad, kNrcGridParams * 4, cudaMemcpyDeviceToHost));
  if (out_loss) VCR_CUDA(ctx, cudaMemcpy(out_loss, st->loss + 1, 4, cudaMemcpyDeviceToHost));
  VCR_CUDA(ctx, cudaMemset(st->grad, 0, kNrcWeightCount * 4));
  if (st->ggrad) VCR_CUDA(ctx, cudaMemset(st->ggrad, 0, kNrcGridParams * 4));
  return VCR_OK;
}
