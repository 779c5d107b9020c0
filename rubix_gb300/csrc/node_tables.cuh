// Shared parts of the node-by-node forward and its adjoint: the cut of the SSP grid into
// slices, the T' table over the Doppler factor, a particle's place on both, a warp's staged
// records and its view of the telescope grid, and the hand-over of flagged spaxels to the
// general kernels.  Everything lives in an anonymous namespace: each translation unit that
// includes this header gets its own copy of the kernels.
#pragma once

#include "cube_nodes.cuh"

namespace rubix {
namespace {

constexpr int kExt = 512;        // virtual telescope samples on either side
constexpr int kMaxBins = 224;    // samples of one (item, slice) row: 7 per lane
constexpr int kWin = 768;        // samples of a slice's window over all alpha
constexpr int kMaxSlices = 128;
constexpr int kMaxWaves = 64;
constexpr int kSub = 256;        // particles sorted together
constexpr int kAlphaBits = 18;
constexpr float kAlphaStep = 1.0f / (1 << kAlphaBits);
constexpr float kAlphaMax = 2040.f * kAlphaStep;       // |alpha - 1| covered (2333 km/s)
// |alpha - 1| covered by the T' table (949 km/s): the few faster stars of a galaxy have their T'
// summed directly, 2 ns each, where every tile of rows costs 4 us and 340 kB.
constexpr int kAlphaHalf = 832;                        // alpha rows on either side of 1
constexpr float kTableMax = 830.f * kAlphaStep;
constexpr int kAlphaTile = 64;                         // rows computed together
constexpr int kAlphaTiles = 2 * kAlphaHalf / kAlphaTile + 1;
constexpr int kAlphaRows = kAlphaTiles * kAlphaTile;
static_assert(kAlphaTiles <= 32, "a word of tiles");
constexpr int kStage = 33;       // staged records of a warp: 32 and one of weight zero
constexpr int kRuns = 4;
constexpr int kDustMost = 8;     // samples between two nodes that a lane holds with dust

struct NodeCtrl {
  int flagged;                  // spaxels left to the general kernel
  // their items by place in its list: of several-chunk spaxels, of large ones, of the rest
  int left[3], listed[3];
  unsigned e_lo, e_hi;          // bits of max(-e), max(e) of the dust exponents, >= 0
  unsigned tile_mask;           // tiles of alpha rows that some star needs
  unsigned tile_sel;            // the same without the screened spaxels' stars
  unsigned a_min_inv, a_max;    // ~bits, bits of the smallest and largest alpha, approximate
  int fast, screened;           // a star beyond the table; flags set before the items
  unsigned dz_inv, dt_inv;      // ~bits of the smallest SSP / telescope spacing
  unsigned dz_max, dt_max;      // bits of the largest (3e38: not ascending)
  unsigned run_max[kRuns], run_min_inv[kRuns];  // extent of own_nodes(r) + 1, + 0 intervals
  int k_first;                  // 1 + node below the telescope range at any alpha
  int k_last_inv;               // n_wave - node above it
  unsigned fmax;                // bits of max |flux| (above inf: NaN)
  int n_rough;                  // particles in the list of rough ones
  int n_items, n_multi;         // work items with particles; those of several-item spaxels
  int next[kMaxWaves][kMaxSlices];
};

// A spaxel is left to the general kernel: its flag, and its items counted for that kernel's list
// (work items of `chunk` particles as in cube_prepare).
struct NodeFlags {
  int* flags;
  NodeCtrl* ctrl;
  const int* seg_off;
  int chunk, big;
  // Place in the list's order and number of a spaxel's items.
  __device__ __forceinline__ int place(int s, int& items) const {
    const int cnt = seg_off[s + 1] - seg_off[s];
    items = (cnt + chunk - 1) / chunk;
    return items > 1 ? 0 : (cnt >= big ? 1 : 2);
  }
  __device__ __forceinline__ void leave(int s) const {
    if (atomicExch(&flags[s], 1) != 0) return;
    int items;
    const int p = place(s, items);
    atomicAdd(&ctrl->left[p], items);
    ctrl->flagged = 1;
  }
  // The counts of spaxels that a block has flagged itself.
  __device__ __forceinline__ void add(const int* s_left) const {
    const int tid = threadIdx.x;
    if (tid < 3 && s_left[tid] > 0) {
      atomicAdd(&ctrl->left[tid], s_left[tid]);
      ctrl->flagged = 1;
    }
  }
};

// A slice has 32, 16, 8 or 4 nodes; all but its first and last are its own.
__host__ __device__ constexpr int own_nodes(int r) { return (32 >> r) - 2; }

// Slices that the workspace provides rows for.
__host__ __device__ inline int max_slices_of(int n_wave) {
  const int s = (n_wave + 30) / 31 + 1;
  return s > kMaxSlices ? kMaxSlices : (s < 48 ? 48 : s);
}

struct NodePlan {
  int ok;
  int k_first, k_last, n_own, n_slices;  // first and last node, nodes of a slice, slices
  int w;                         // samples that a node may cross within a group of particles
  float dt_min, window;          // samples that an item's alpha range may span
  int most;                      // samples between two nodes at most
};

// How the grids are cut into slices, from the extrema; every block derives the same plan.
__device__ __forceinline__ NodePlan node_plan(const NodeCtrl* c, int n_wave, float x_last,
                                              bool dust) {
  NodePlan p;
  const float dz = __uint_as_float(~c->dz_inv), dt = __uint_as_float(~c->dt_inv);
  const float dtm = __uint_as_float(c->dt_max), fm = __uint_as_float(c->fmax);
  p.k_first = max(c->k_first - 1, 0);
  const int k_last = p.k_last = min(n_wave - c->k_last_inv, n_wave - 1);
  p.dt_min = dt;
  p.ok = 0;
  p.n_own = 0;
  p.w = 1;
  p.most = 0;
  p.n_slices = 0;
  p.window = 0.f;
  // lambda' spacing >= alpha*dz minus two roundings of lambda' (|lambda'| < 2^14): at
  // least one sample between two nodes; float32 exact enough to order samples and nodes
  if (!(dz * (1.f - kAlphaMax) - 4.0e-3f > dtm) || !(dt > 2.0e-2f) || !(dtm < 1e30f) ||
      !(__uint_as_float(c->dz_max) < 1e30f) || !(x_last < 16384.f) || !(fm < 1e30f) ||
      k_last <= p.k_first)
    return p;
  const float ratio = (dz * (1.f - kAlphaMax) - 4.0e-3f) / dtm;
  p.w = ratio > 2.f ? 2 : 1;
  p.most = (int)(__uint_as_float(c->dz_max) * (1.f + kAlphaMax) / dt + 1.01f);
  // with dust every sample is evaluated: fewer than two of them between nodes, or more than
  // a lane holds, are the general kernel's
  if (dust && (p.w < 2 || p.most > kDustMost)) return p;
  const float swing = 2.f * kAlphaMax * x_last / dt;  // samples a node moves over all alpha
  for (int r = 0; r < kRuns; ++r) {
    const float hi = __uint_as_float(c->run_max[r]) * (1.f + kAlphaMax) / dt;
    const float lo = __uint_as_float(~c->run_min_inv[r]) * (1.f - kAlphaMax) / dtm;
    const float win = fminf((float)kMaxBins - hi, lo) - 4.f;
    if (win < 24.f || hi + swing + 8.f > (float)(kExt - 16) ||
        hi + swing + 8.f > (float)(kWin - 8))
      continue;
    p.n_own = own_nodes(r);
    p.window = win;
    p.n_slices = (k_last - p.k_first + p.n_own) / p.n_own;  // k_last too has an owner
    p.ok = p.n_slices <= max_slices_of(n_wave);
    return p;
  }
  return p;
}

// SSP wavelength k, continued with the end spacings beyond the grid.
__device__ __forceinline__ float lam_ext(const float* __restrict__ wz, int n, int k) {
  if (k < 0) return wz[0] + (float)k * (wz[1] - wz[0]);
  if (k >= n) return wz[n - 1] + (float)(k - n + 1) * (wz[n - 1] - wz[n - 2]);
  return wz[k];
}

// Telescope sample e of the extended grid (e = t + kExt), continued with the end spacings.
__device__ __forceinline__ float x_ext(const float* __restrict__ wt, int n, int e) {
  const int t = e - kExt;
  if (t < 0) return wt[0] + (float)t * (wt[1] - wt[0]);
  if (t >= n) return wt[n - 1] + (float)(t - n + 1) * (wt[n - 1] - wt[n - 2]);
  return wt[t];
}

// alpha - 1 of a velocity, to 1e-7.
__device__ __forceinline__ float approx_am1(float v) {
  const float z = v * (float)(1.0 / kSpeedOfLight);
  return z * (1.f + 0.5f * z * (1.f + (1.f / 3.f) * z));
}

// The tiles of alpha rows on either side of it, up to a row beyond the limit that node_particle
// checks on the rounded alpha; false beyond.
__device__ __forceinline__ bool alpha_tiles(float am1, int& a, int& b) {
  if (!(fabsf(am1) <= kTableMax + kAlphaStep)) return false;
  const int r = (int)floorf(am1 * (float)(1 << kAlphaBits)) + kAlphaHalf;
  a = max(r - 1, 0) / kAlphaTile;
  b = min(r + 2, kAlphaRows - 1) / kAlphaTile;
  return true;
}

// Grid extrema, and the rows of alpha that the particles' velocities fall on.
__global__ void __launch_bounds__(256) node_setup_kernel(
    const float* __restrict__ wz, int n_wave, const float* __restrict__ wt, int n_t,
    const float* __restrict__ vel, long long vel_stride, int vel_comp, long long n,
    const float* __restrict__ dust_e, NodeCtrl* __restrict__ ctrl) {
  const long long gtid = blockIdx.x * 256LL + threadIdx.x, gsz = gridDim.x * 256LL;
  if (gtid < n_t - 1) {
    float d = wt[gtid + 1] - wt[gtid];
    const bool bad = !(d > 0.f);
    atomicMax(&ctrl->dt_max, bad ? __float_as_uint(3e38f) : __float_as_uint(d));
    if (!bad) atomicMax(&ctrl->dt_inv, ~__float_as_uint(d));
  }
  if (dust_e && gtid < n_t) {
    const float e = dust_e[gtid];
    // a value that is not finite makes the limit infinite: every star is flagged
    atomicMax(&ctrl->e_hi, __float_as_uint(isfinite(e) ? fmaxf(e, 0.f) : kFltMax));
    atomicMax(&ctrl->e_lo, __float_as_uint(isfinite(e) ? fmaxf(-e, 0.f) : kFltMax));
  }
  const float x0 = wt[0], x1 = wt[n_t - 1];
  const float hi = 1.f + kAlphaMax, lo = 1.f - kAlphaMax;
  if (gtid < n_wave - 1) {
    const int k = (int)gtid;
    const float a = wz[k], b = wz[k + 1];
    if (a * hi <= x0 && !(b * hi <= x0)) ctrl->k_first = k + 1;
    if (!(a * lo > x1) && b * lo > x1) ctrl->k_last_inv = n_wave - (k + 1);
    const float d = b - a;
    const bool bad = !(d > 0.f);
    const bool seen = bad || (b * 1.05f >= x0 && a * 0.95f <= x1);
    if (seen) {
      atomicMax(&ctrl->dz_max, bad ? __float_as_uint(3e38f) : __float_as_uint(d));
      atomicMax(&ctrl->dz_inv, ~__float_as_uint(bad ? 0.f : d));
    }
#pragma unroll
    for (int r = 0; r < kRuns; ++r) {
      const float e0 = lam_ext(wz, n_wave, k + own_nodes(r)) - a;
      const float e1 = lam_ext(wz, n_wave, k + own_nodes(r) + 1) - a;
      if (seen && e0 >= 0.f && e1 >= 0.f) {
        atomicMax(&ctrl->run_max[r], __float_as_uint(e1));
        atomicMax(&ctrl->run_min_inv[r], ~__float_as_uint(e0));
      }
    }
  }
  __shared__ unsigned s_mask, s_min_inv, s_max;
  __shared__ int s_fast;
  if (threadIdx.x == 0) {
    s_mask = s_min_inv = s_max = 0u;
    s_fast = 0;
  }
  __syncthreads();
  unsigned mask = 0u;
  bool fast = false;
  float amin = 2.f, amax = 0.f;
  for (long long i = gtid; i < n; i += gsz) {
    const float am1 = approx_am1(vel[i * vel_stride + vel_comp]);
    fast = fast || !(fabsf(am1) <= kAlphaMax - kAlphaStep);
    amin = fminf(amin, 1.f + am1);
    amax = fmaxf(amax, 1.f + am1);
    int a, b;
    if (!alpha_tiles(am1, a, b)) continue;
    mask |= (1u << a) | (1u << b);
  }
  mask = __reduce_or_sync(0xffffffffu, mask);
  const unsigned lo_inv = __reduce_max_sync(0xffffffffu, ~__float_as_uint(amin));
  const unsigned hi_bits = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_min_inv, lo_inv);
    atomicMax(&s_max, hi_bits);
    atomicOr(&s_mask, mask);
  }
  if (fast) s_fast = 1;
  __syncthreads();
  if (threadIdx.x == 0 && s_mask) atomicOr(&ctrl->tile_mask, s_mask);
  if (threadIdx.x == 0) {
    atomicMax(&ctrl->a_min_inv, s_min_inv);
    atomicMax(&ctrl->a_max, s_max);
    if (s_fast) ctrl->fast = 1;
  }
}

__device__ __forceinline__ bool tile_used(const NodeCtrl* c, int tile) {
  return ((c->screened ? c->tile_sel : c->tile_mask) >> tile) & 1u;
}

// Whether the call's velocities may flag a spaxel: where no star is beyond the table and all of
// them together fit an item's window, none is screened.
__device__ __forceinline__ bool screen_wanted(const NodeCtrl* c, const NodePlan& p, float x1) {
  const float spread = __uint_as_float(c->a_max) - __uint_as_float(~c->a_min_inv) + 1e-6f;
  return !p.ok || c->fast || spread * x1 / (1.f - kAlphaMax) > p.window * p.dt_min;
}

// Whether an item's range of alpha is wider than the rows of its slices.
__device__ __forceinline__ bool too_wide(const NodePlan& p, float amin, float amax, float x1) {
  return (amax - amin) * x1 / (1.f - kAlphaMax) > p.window * p.dt_min;
}

// What the velocities of one item's stars say, by a warp: whether they flag their spaxel, and
// the tiles of their alpha rows.  On alpha to 1e-7 in float32 (the exact one takes 64-bit
// products, 0.7 ms for 2 10^5 stars on one SM), so it flags what is beyond the gather's conditions
// by more than that and leaves the rest to them.
__device__ __forceinline__ bool screen_item(const CubeInputs& in, const NodePlan& p, int jb,
                                            int je, float x1, unsigned& mask) {
  float lo = 1.f, hi = -1.f, far = 0.f;
#pragma unroll 4
  for (int j = jb + (threadIdx.x & 31); j < je; j += 32) {
    const float am1 = approx_am1(in.vel[(long long)in.perm[j] * in.vel_stride + in.vel_comp]);
    int a, b;
    if (alpha_tiles(am1, a, b)) mask |= (1u << a) | (1u << b);
    lo = fminf(lo, am1);
    hi = fmaxf(hi, am1);
    far = fmaxf(far, isnan(am1) ? 1.f : fabsf(am1));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    far = fmaxf(far, __shfl_xor_sync(0xffffffffu, far, o));
  }
  return far > kAlphaMax + kAlphaStep || too_wide(p, lo + 1e-6f, hi, x1);
}

// Particles of each spaxel that the node path renders, to count(s, particles), by the whole grid
// and before there are work items.  Where velocities rule spaxels out, or the grids all of
// them, they are flagged here and count nothing, and only the other stars' tiles are built:
// with a dispersion of 1000 km/s, where nearly every spaxel is flagged, the table product
// alone took 270 us.
template <class F>
__device__ __forceinline__ void screened_counts(const CubeInputs& in, const NodeFlags& flags,
                                                bool dust, int item, F count) {
  constexpr int kLarge = 256;  // stars of a spaxel that a whole block screens
  __shared__ NodePlan s_plan;
  __shared__ int s_left[3], s_large[32], s_large_n, s_flag;
  __shared__ unsigned s_sel, s_mask;
  const float x1 = in.wave_t[in.n_wave_t - 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  const int gtid = blockIdx.x * blockDim.x + tid, gsz = gridDim.x * blockDim.x;
  if (tid == 0) {
    s_plan = node_plan(flags.ctrl, in.n_wave, x1, dust);
    s_sel = 0u;
  }
  if (tid < 3) s_left[tid] = 0;
  int own = gtid < in.n_seg ? in.seg_off[gtid + 1] - in.seg_off[gtid] : 0;  // loaded meanwhile
  __syncthreads();
  const NodePlan plan = s_plan;
  const bool screen = screen_wanted(flags.ctrl, plan, x1);
  auto leave = [&](int s) {
    int items;
    const int p = flags.place(s, items);
    atomicAdd(&s_left[p], items);
    flags.flags[s] = 1;
    count(s, 0);
  };
  if (!screen || !plan.ok) {
    for (int s = gtid; s < in.n_seg; s += gsz) {
      if (s != gtid) own = in.seg_off[s + 1] - in.seg_off[s];
      if (screen && own > 0) leave(s);
      else count(s, own);
    }
  } else {
    // a spaxel per warp, the large ones among them by the block together
    if (gtid == 0) flags.ctrl->screened = 1;
    for (int s0 = blockIdx.x * warps; s0 < in.n_seg; s0 += gridDim.x * warps) {
      if (tid == 0) s_large_n = 0;
      __syncthreads();
      const int s = s0 + warp;
      if (s < in.n_seg) {
        const int jb = in.seg_off[s], je = in.seg_off[s + 1];
        if (je - jb > kLarge) {
          if (lane == 0) s_large[atomicAdd(&s_large_n, 1)] = s;
        } else {
          unsigned mask = 0u;
          const bool flag = screen_item(in, plan, jb, je, x1, mask);
          mask = __reduce_or_sync(0xffffffffu, mask);
          if (lane == 0) {
            if (flag) leave(s);
            else count(s, je - jb);
            if (!flag && mask) atomicOr(&s_sel, mask);
          }
        }
      }
      __syncthreads();
      const int n_large = s_large_n;
      for (int q = 0; q < n_large; ++q) {
        if (tid == 0) {
          s_flag = 0;
          s_mask = 0u;
        }
        __syncthreads();
        const int big = s_large[q], jb = in.seg_off[big], je = in.seg_off[big + 1];
        unsigned mask = 0u;
        bool flag = false;
        for (int c = jb + warp * item; c < je; c += warps * item)
          flag = screen_item(in, plan, c, min(c + item, je), x1, mask) || flag;
        mask = __reduce_or_sync(0xffffffffu, mask);
        if (lane == 0) {
          if (flag) s_flag = 1;
          atomicOr(&s_mask, mask);
        }
        __syncthreads();
        if (tid == 0) {
          if (s_flag) {
            leave(big);
          } else {
            count(big, je - jb);
            s_sel |= s_mask;
          }
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
  flags.add(s_left);
  if (tid == 0 && s_sel) atomicOr(&flags.ctrl->tile_sel, s_sel);
}

// The work items are made by one block for few spaxels and stars (it screens 2 10^5 stars in 0.4
// ms), else in a launch each for counts, scans and list: 8.8 us for 4489 spaxels, where one
// block takes 10 without counting.
constexpr long long kItemsOneBlockStars = 1 << 16;
inline bool items_one_block(int n_seg, long long n) {
  return n_seg <= kItemsOneBlock && n <= kItemsOneBlockStars;
}

// The two resampling weights that interval [k, k + 1] gives its nodes at one alpha: the
// samples x_t inside it at distance d from node k weigh dx_t (1 - d / len) and dx_t d / len.
// The nodes are lambda_z * alpha unrounded, as float pairs; the few samples of an interval
// are summed directly.
__device__ __forceinline__ float2 interval_weights(const float* __restrict__ wz,
                                                   const float* __restrict__ wt, int n_t, int k,
                                                   float alpha, float x0, float inv) {
  const float z0 = wz[k], z1 = wz[k + 1];
  const float ah = __fmul_rn(z0, alpha), al = fmaf(z0, alpha, -ah);
  const float bh = __fmul_rn(z1, alpha), bl = fmaf(z1, alpha, -bh);
  int t = min(max((int)((ah - x0) * inv), 0), n_t - 1);
  while (t > 0 && (wt[t - 1] - ah) - al >= 0.f) --t;
  while (t < n_t && (wt[t] - ah) - al < 0.f) ++t;
  float s0 = 0.f, s1 = 0.f, prev = t > 0 ? wt[t - 1] : x0;
  for (; t < n_t; ++t) {
    const float x = wt[t];
    if ((x - bh) - bl >= 0.f) break;
    const float dx = t > 0 ? x - prev : 0.f;
    s0 += dx;
    s1 = fmaf(dx, (x - ah) - al, s1);
    prev = x;
  }
  const float rise = s1 / ((bh - ah) + (bl - al));
  return make_float2(s0 - rise, rise);
}

constexpr int kWeightBlocks = 1024;

// Largest roughness that the table is read with, relative to T': its error is then below 6e-7,
// 1e-7 rms, the size of float32's own in a sum of 3721 products.  The synthetic templates
// (absorption lines of 2 to 8 A) have up to 4.4e-7, 7.5e-7 on the 700 bluest samples; noise of
// 10 % from node to node has 1.4e-6, emission lines of 100 A equivalent width 1e-5.
constexpr float kRoughLimit = 1e-6f;

// How far the interpolated T' of a template may be from the sum on its shifted grid, for
// kRoughLimit.  T'(alpha) has a kink where a node passes a sample (bin width times the jump
// of the template's slope at the node), of which linear interpolation over one alpha step cuts
// off at most a quarter step; and the table's nodes are not rounded to float32, which moves a
// node by up to lambda 2^-24 and T' by that times the mean step of the flux beside it.  Both
// have either sign from node to node: the root of the sum of the squares over the nodes in
// range.  Against float64 (templates with noise, absorption lines, emission lines of 1.5 and
// 3 A, a single node; 400 velocities each) the largest error is 0.38 to 0.62 of this on 1.25 A
// samples, 0.14 on 5 A ones, the rms error 0.03 to 0.14 of it.
__device__ __forceinline__ float node_roughness(const float* __restrict__ f,
                                                const float* __restrict__ wz, int k, float dt_max,
                                                float scale) {
  const float z = wz[k], f1 = f[k], up = (f[k + 1] - f1) * scale, dn = (f1 - f[k - 1]) * scale;
  const float jump = __fdividef(up, wz[k + 1] - z) - __fdividef(dn, z - wz[k - 1]);
  const float kink = dt_max * z * (0.25f * kAlphaStep) * jump;
  const float round = z * 5.9604645e-8f * (0.5f * (fabsf(up) + fabsf(dn)));
  return fmaf(kink, kink, round * round);
}

// Per template (block b < rows): float64 prefix sums, max |F| and the roughness.
// The remaining blocks: the resampling weights of T' at alpha_i, h_k = sum_t dlambda_t
// hat_k(x_t) with hat_k the hat function of node k, one alpha row of a used tile at a time.
// Nodes are stored from k_first on, kpad to a row, zero beyond the last.
__global__ void __launch_bounds__(kPrefixThreads) node_tables_kernel(
    const float* __restrict__ flux, int rows, int n_wave, const float* __restrict__ wz,
    const float* __restrict__ wt, int n_t, double* __restrict__ prefix, float* __restrict__ h,
    int kpad, float* __restrict__ rough, bool dust, NodeCtrl* __restrict__ ctrl,
    CubeCtrl* __restrict__ cc) {
  if ((int)blockIdx.x == rows + kWeightBlocks) {  // for the general kernel's tables
    if (threadIdx.x == 0) {
      bucket_params(wt, n_t, cc->lnq0, cc->h);
      cc->inv_h = 1.0 / cc->h;
      cc->bmax = (float)(kVmaxKms / kSpeedOfLight / cc->h);
    }
    return;
  }
  const int k_first = max(ctrl->k_first - 1, 0);
  const int k_last = min(n_wave - ctrl->k_last_inv, n_wave - 1);
  if ((int)blockIdx.x < rows) {
    const double total = prefix_row(flux, blockIdx.x, n_wave, wz, prefix);
    __shared__ float s_sum[kPrefixThreads / 32];
    const float* f = flux + (long long)blockIdx.x * n_wave;
    const float dt_max = __uint_as_float(ctrl->dt_max);
    // squares of fluxes in any unit: relative to the total (0: any value is rough)
    const float scale = (float)(1.0 / fmax(fabs(total), 1e-37));
    unsigned m = 0u;
    float sum = 0.f;
    for (int k = threadIdx.x; k < n_wave; k += kPrefixThreads) {
      m = max(m, __float_as_uint(f[k]) & 0x7fffffffu);
      if (k >= max(k_first, 1) && k <= min(k_last, n_wave - 2))
        sum += node_roughness(f, wz, k, dt_max, scale);
    }
    m = __reduce_max_sync(0xffffffffu, m);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&ctrl->fmax, m);
      s_sum[threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kPrefixThreads / 32; ++w) sum += s_sum[w];
      rough[blockIdx.x] = sqrtf(sum) / scale;
    }
    return;
  }
  // nothing reads the weights of a grid that does not qualify (fmax, still being formed, can
  // only rule it out)
  if (!node_plan(ctrl, n_wave, wt[n_t - 1], dust).ok) return;
  __shared__ float s_rise[kPrefixThreads + 1];
  const int tid = threadIdx.x;
  const int count = k_last - k_first + 1;
  const float x0 = wt[0], inv = (float)(n_t - 1) / (wt[n_t - 1] - x0);
  for (int u = blockIdx.x - rows;; u += kWeightBlocks) {
    // row u of the used tiles
    int tile = 0, left = u / kAlphaTile;
    while (tile < kAlphaTiles && (!tile_used(ctrl, tile) || left-- > 0)) ++tile;
    if (tile == kAlphaTiles) return;
    const int row = tile * kAlphaTile + u % kAlphaTile;
    const float alpha = 1.f + (float)(row - kAlphaHalf) * kAlphaStep;  // exact
    if (tid == 0) s_rise[0] = 0.f;
    for (int q0 = 0; q0 < kpad; q0 += kPrefixThreads) {
      const int q = q0 + tid;
      float2 w = make_float2(0.f, 0.f);
      if (q < count - 1) w = interval_weights(wz, wt, n_t, k_first + q, alpha, x0, inv);
      s_rise[tid + 1] = w.y;
      __syncthreads();
      if (q < kpad) h[(long long)row * kpad + q] = w.x + s_rise[tid];
      __syncthreads();
      if (tid == kPrefixThreads - 1) s_rise[0] = w.y;
    }
    __syncthreads();
  }
}

// H[i][c] = sum_k h[i][k] F[c][k]: 64 alpha rows x 32 templates per block of 128 threads,
// 4 x 4 per thread, 32 nodes staged at a time.  Sums of 32 products are added with Kahan's
// compensation: a plain float32 sum over ~740 nodes would be 5e-7 off, this one is 1e-8.
// NaN for a template too rough to be read from the table.
// 106 us at 10^7 particles (800 alpha rows x 1302 templates; 129 with padded tiles, whose
// transposing stores fell in 8 banks).
// Bound by FMA issue: 1 GFMA for 1025 rows of a 1326-template grid, 40 TFMA/s on the chip.
__global__ void __launch_bounds__(128) node_table_product_kernel(
    const float* __restrict__ h, int kpad, const float* __restrict__ flux, int n_templ,
    int n_wave, const float* __restrict__ wt, int n_t, bool dust,
    const float* __restrict__ rough, const NodeCtrl* __restrict__ ctrl, float* __restrict__ H) {
  constexpr int BK = 32, BM = kAlphaTile, BN = 32;
  const int tile = blockIdx.y;
  if (!tile_used(ctrl, tile)) return;
  const NodePlan p = node_plan(ctrl, n_wave, wt[n_t - 1], dust);
  if (!p.ok) return;
  const int K = min(p.k_last - p.k_first + 1, kpad);
  // columns permuted by the node (column ^ 4 (k / 4 mod 8)): the transposing stores of a warp
  // fall in 32 banks and the 16-byte loads stay whole
  __shared__ __align__(16) float sa[2][BK][BM];
  __shared__ __align__(16) float sb[2][BK][BN];
  const int tid = threadIdx.x;
  const int r0 = tile * BM, c0 = blockIdx.x * BN;
  const int tr = (tid >> 3) * 4, tc = (tid & 7) * 4;
  // loads: a thread takes 4 consecutive nodes of h in 4 rows, and of F node `lane` in 8
  const int lr = tid >> 3, lk = (tid & 7) * 4, lane = tid & 31, warp = tid >> 5;
  float4 ra[4];
  float rb[8];
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      ra[i] = *reinterpret_cast<const float4*>(h + (long long)(r0 + lr + 16 * i) * kpad + k0 + lk);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = c0 + warp * 8 + j;
      rb[j] = (k0 + lane < K && c < n_templ)
                  ? flux[(long long)c * n_wave + p.k_first + k0 + lane] : 0.f;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int col = (lr + 16 * i) ^ lk;  // lk = 4 (k / 4)
      sa[buf][lk][col] = ra[i].x;
      sa[buf][lk + 1][col] = ra[i].y;
      sa[buf][lk + 2][col] = ra[i].z;
      sa[buf][lk + 3][col] = ra[i].w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sb[buf][lane][(warp * 8 + j) ^ (lane & 28)] = rb[j];
  };
  float sum[4][4], comp[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[i][j] = comp[i][j] = 0.f;
  const int steps = (K + BK - 1) / BK;  // kpad is a multiple of BK
  load(0);
  store(0);
  __syncthreads();
  for (int s = 0; s < steps; ++s) {
    if (s + 1 < steps) load((s + 1) * BK);
    float acc[4][4];
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&sa[s & 1][k][tr ^ (k & 28)]);
      const float4 b = *reinterpret_cast<const float4*>(&sb[s & 1][k][tc ^ (k & 28)]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] = k == 0 ? av[i] * bv[j] : fmaf(av[i], bv[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float y = acc[i][j] - comp[i][j];
        const float t = sum[i][j] + y;
        comp[i][j] = (t - sum[i][j]) - y;
        sum[i][j] = t;
      }
    if (s + 1 < steps) store((s + 1) & 1);
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (c0 + tc + j >= n_templ) continue;
    const float e = rough[c0 + tc + j];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      H[(long long)(r0 + tr + i) * n_templ + c0 + tc + j] =
          e <= kRoughLimit * fabsf(sum[i][j]) ? sum[i][j] : __int_as_float(0x7fffffff);
  }
}

// Last SSP wavelength k with lambda'_k <= x (-1: none), on an ascending grid (where it is not,
// the plan flags every spaxel): a linear guess, right to one node on a uniform grid, else the
// search, whose ten dependent loads a block waited for (node_gather_kernel 194 -> 173 us at
// 10^6 particles, 10.5 -> 7.8 at 2000; the adjoint's gather alike).
__device__ __forceinline__ int last_below(const float* __restrict__ wz, int n, float alpha,
                                          float x) {
  if (n < 2) return count_le_scaled(wz, n, alpha, x) - 1;
  const float z0 = wz[0], inv = (float)(n - 1) / (wz[n - 1] - z0);
  const int k = (int)fminf(fmaxf((x / alpha - z0) * inv, 0.f), (float)(n - 2));
  const float a = __fmul_rn(wz[k], alpha), b = __fmul_rn(wz[k + 1], alpha);
  if (x < a) {
    if (k > 0 && __fmul_rn(wz[k - 1], alpha) <= x) return k - 1;
  } else if (x < b) {
    return k;
  } else if (k + 2 < n && x < __fmul_rn(wz[k + 2], alpha)) {
    return k + 1;
  }
  return count_le_scaled(wz, n, alpha, x) - 1;
}

// 1 / x by the hardware's reciprocal (relative error about 2^-23); x is a positive normal.
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

constexpr int kRoughThreads = 512;
constexpr int kRoughBlocks = 2;  // per SM
constexpr int kRoughUnroll = 2;

// Samples before each sample, for sums over the samples of an interval: entry t holds
// (x_{t-1}, sum_{q < t} dx_q x_q as a float pair, x_t), t = 0 .. n_t, with dx_0 = 0.
// Returns whether a linear guess of a sample's place is right to half a sample everywhere.
__device__ __forceinline__ bool sample_table(const float* __restrict__ wt, int n_t, float4* tab) {
  __shared__ double s_warp[kRoughThreads / 32];
  const int per = (n_t + kRoughThreads) / kRoughThreads, tid = threadIdx.x;
  const int t0 = min(tid * per, n_t + 1), t1 = min(t0 + per, n_t + 1);
  const float x0 = wt[0], inv = (float)(n_t - 1) / (wt[n_t - 1] - x0);
  auto term = [&](int q) {
    return q >= 1 && q < n_t ? (double)(wt[q] - wt[q - 1]) * (double)wt[q] : 0.0;
  };
  double sum = 0.0;
  bool even = true;
  for (int t = t0; t < t1; ++t) {
    sum += term(t);
    if (t < n_t) even = even && fabsf((wt[t] - x0) * inv - (float)t) <= 0.5f;
  }
  double run = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, run, d);
    if ((tid & 31) >= d) run += y;
  }
  if ((tid & 31) == 31) s_warp[tid >> 5] = run;
  __syncthreads();
  run -= sum;
  for (int w = 0; w < (tid >> 5); ++w) run += s_warp[w];
  for (int t = t0; t < t1; ++t) {
    const float hi = (float)run;
    tab[t] = make_float4(wt[max(t - 1, 0)], hi, (float)(run - (double)hi),
                         t < n_t ? wt[t] : kFltMax);
    run += term(t);
  }
  return __syncthreads_and(even);
}

size_t rough_smem(int n_t) { return sizeof(float4) * (size_t)(n_t + 1); }

// Entry of the first sample >= a.  Even samples: a linear guess, corrected by one; else a search.
template <bool kEven>
__device__ __forceinline__ float4 first_sample(const float4* tab, int n_t, float a, float x0,
                                               float inv) {
  if constexpr (kEven) {
    const int t = min(max((int)((a - x0) * inv), 0), n_t - 1) + 1;
    float4 e = tab[t];
    const bool before = !(e.x < a), after = e.w < a;
    if (before || after) e = tab[before ? t - 1 : t + 1];
    return e;
  } else {
    int lo = 0, hi = n_t;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (tab[mid].w < a) lo = mid + 1; else hi = mid;
    }
    return tab[lo];
  }
}

// T' of one particle summed over its own shifted nodes by a warp, a lane per node (31 intervals
// at a time): what the general kernel sums, without the table.  An interval's samples enter by
// differences of the sample table: the sum of dx, exact, and that of dx (x - a), whose
// large parts cancel exactly in the product-sum.
template <bool kEven>
__device__ __forceinline__ float direct_tprime(const float* __restrict__ f, int n_age, int n_wave,
                                               const float* __restrict__ wz, const float4* tab,
                                               int n_t, int k_first, int k_last, float alpha,
                                               const float (&w)[4]) {
  const int lane = threadIdx.x & 31;
  const float* f1 = f + (long long)n_age * n_wave;  // corners 00, 10, 01, 11
  const float* f2 = f + n_wave;
  const float* f3 = f1 + n_wave;
  const float x0 = tab[0].w, inv = (float)(n_t - 1) / (tab[n_t].x - x0);
  float sum = 0.f;
  constexpr int kUnroll = kEven ? kRoughUnroll : 1;
#pragma unroll kUnroll
  for (int k0 = k_first; k0 < k_last; k0 += 31) {
    const int k = min(k0 + lane, k_last);
    const float a = __fmul_rn(wz[k], alpha);
    float G = w[0] * f[k];
    G = fmaf(w[1], f1[k], G);
    G = fmaf(w[2], f2[k], G);
    G = fmaf(w[3], f3[k], G);
    const float4 e = first_sample<kEven>(tab, n_t, a, x0, inv);
    const float b = __shfl_down_sync(0xffffffffu, a, 1);
    const float G1 = __shfl_down_sync(0xffffffffu, G, 1);
    const float s0 = __shfl_down_sync(0xffffffffu, e.x, 1) - e.x;
    const float hi = __shfl_down_sync(0xffffffffu, e.y, 1) - e.y;
    const float lo = __shfl_down_sync(0xffffffffu, e.z, 1) - e.z;
    const float s1 = fmaf(-a, s0, hi) + lo;
    // past the last node nothing is added: a == b there
    if (lane < 31 && k0 + lane < k_last) sum += fmaf(s1 * fast_rcp(b - a), G1 - G, s0 * G);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum;
}

// One particle on the tables: the corner weights, T (and, for the gradients, its corner
// values), T', and whether the general kernel has to take it.
struct NodeParticle {
  float alpha, T, Tp;
  float w[4];      // corners 00, 10, 01, 11 as (metallicity, age)
  double dT[4];    // in-range flux sum of each, over alpha
  float tz, ta, dzg, dag;
  int row;         // template 00
  bool outside, bad;
  bool rough;      // T' is not in the table (NaN): to be summed directly
};

__device__ __forceinline__ void corner_weights(float tz, float ta, float (&w)[4]) {
  w[0] = (1.f - tz) * (1.f - ta);
  w[1] = tz * (1.f - ta);
  w[2] = (1.f - tz) * ta;
  w[3] = tz * ta;
}

// Whether T / T' is unusual and left to the general kernel.
__device__ __forceinline__ bool bad_scale(float T, float Tp) {
  const float sc = T / Tp;
  return !(sc > 0.25f && sc < 4.f);
}

__device__ __forceinline__ NodeParticle node_particle(const CubeInputs& in,
                                                      const double* __restrict__ prefix,
                                                      const float* __restrict__ H, long long i) {
  NodeParticle p;
  const float x0 = in.wave_t[0], x1 = in.wave_t[in.n_wave_t - 1];
  const int n_templ = in.n_met * in.n_age;
  const float Z = in.met[i], A = in.age[i];
  p.alpha = doppler_factor(in.vel[i * in.vel_stride + in.vel_comp]);
  p.outside = (Z < in.ssp_met[0]) || (Z > in.ssp_met[in.n_met - 1]) || (A < in.ssp_age[0]) ||
              (A > in.ssp_age[in.n_age - 1]);
  p.bad = p.rough = false;
  p.row = 0;
  p.T = p.Tp = p.tz = p.ta = p.dzg = p.dag = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    p.w[c] = 0.f;
    p.dT[c] = 0.0;
  }
  if (!(fabsf(p.alpha - 1.f) <= kAlphaMax)) {
    p.bad = true;
    p.alpha = 1.f;
    return p;
  }
  if (p.outside) return p;
  const int iz = min(max(count_le(in.ssp_met, in.n_met, Z), 1), in.n_met - 1);
  const int ia = min(max(count_le(in.ssp_age, in.n_age, A), 1), in.n_age - 1);
  p.dzg = in.ssp_met[iz] - in.ssp_met[iz - 1];
  p.dag = in.ssp_age[ia] - in.ssp_age[ia - 1];
  p.tz = p.dzg == 0.f ? 0.f : (Z - in.ssp_met[iz - 1]) / p.dzg;
  p.ta = p.dag == 0.f ? 0.f : (A - in.ssp_age[ia - 1]) / p.dag;
  const int ks = last_below(in.ssp_wave_z, in.n_wave, p.alpha, x0);
  const int ke = last_below(in.ssp_wave_z, in.n_wave, p.alpha, x1);
  p.row = (iz - 1) * in.n_age + (ia - 1);
  if (ks < 0 || ke + 1 > in.n_wave - 1) {
    p.bad = true;
    return p;
  }
  corner_weights(p.tz, p.ta, p.w);
  const int rr[4] = {p.row, p.row + in.n_age, p.row + 1, p.row + in.n_age + 1};
  // T: in-range flux sum, entries ka..ke with x0 <= lambda'_k <= x1, k >= 1
  int ka = __fmul_rn(in.ssp_wave_z[ks], p.alpha) >= x0 ? ks : ks + 1;
  ka = max(ka, 1);
  const float u = (p.alpha - 1.f) * (float)(1 << kAlphaBits);  // exact
  const int r = (int)floorf(u) + kAlphaHalf;
  const float fr = u - floorf(u);
  const bool tabled = fabsf(p.alpha - 1.f) <= kTableMax;
  const float* h0 = H + (long long)r * n_templ;
  const float* h1 = h0 + n_templ;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const double* pf = prefix + (long long)rr[c] * in.n_wave;
    if (ka <= ke) p.dT[c] = pf[ke] - pf[ka - 1];
    p.T = fmaf(p.w[c], (float)p.dT[c], p.T);
    if (tabled) p.Tp = fmaf(p.w[c], fmaf(fr, h1[rr[c]] - h0[rr[c]], h0[rr[c]]), p.Tp);
  }
  p.T *= p.alpha;
  p.rough = !tabled || isnan(p.Tp);
  if (!p.rough && bad_scale(p.T, p.Tp)) p.bad = true;
  return p;
}

// A place in the list of rough particles, taken by the calling lanes of a warp together.
__device__ __forceinline__ int rough_place(NodeCtrl* ctrl) {
  const unsigned on = __activemask();
  const int lane = threadIdx.x & 31, lead = __ffs(on) - 1;
  int base = 0;
  if (lane == lead) base = atomicAdd(&ctrl->n_rough, __popc(on));
  return __shfl_sync(on, base, lead) + __popc(on & ((1u << lane) - 1u));
}

// T' of a rough particle by a warp: alpha and the byte offset of its corner row in the slice
// table (as in the records), its corner weights.
__device__ __forceinline__ float rough_tprime(const CubeInputs& in, const NodePlan& plan,
                                              const float4* tab, bool even, float2 rec,
                                              const float (&w)[4]) {
  const float* f = in.ssp_flux + (long long)(__float_as_int(rec.y) / 128) * in.n_wave;
  return even ? direct_tprime<true>(f, in.n_age, in.n_wave, in.ssp_wave_z, tab, in.n_wave_t,
                                    plan.k_first, plan.k_last, rec.x, w)
              : direct_tprime<false>(f, in.n_age, in.n_wave, in.ssp_wave_z, tab, in.n_wave_t,
                                     plan.k_first, plan.k_last, rec.x, w);
}

// Rank of this thread's key (alpha's bits) among the m of the block's run, ties by place.
__device__ __forceinline__ int run_rank(const unsigned* s_key, int m, int tid) {
  const unsigned key = s_key[tid];
  int rank = 0;
  for (int q = 0; q < m; q += 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(&s_key[q]);
    rank += (v.x < key || (v.x == key && q < tid)) + (v.y < key || (v.y == key && q + 1 < tid)) +
            (v.z < key || (v.z == key && q + 2 < tid)) + (v.w < key || (v.w == key && q + 3 < tid));
  }
  return rank;
}

// The records that a warp has staged, one array per value: a step reads one word of NPL
// records at a time, one wavefront each (16-byte loads of the same take four).
struct StagedRecs {
  float w[4][kStage];  // corner weights times beta
  float alpha[kStage];
  int row[kStage];     // byte offset of the first corner's row in the slice table
};

struct SliceShared {
  const float* tab;  // [template][32]
  const float* xw;   // window of the extended telescope grid, kWin samples
  const float* ew;   // with dust: the exponents of the window's samples
  StagedRecs* st;    // this warp's staged records
  float* st_av;      // with dust: their columns
  float* f;          // this warp's samples, kMaxBins
  float inv;         // samples per Angstrom over the window
};

// Smallest window index j with xw[j] >= x: a linear guess, right to one sample on a uniform
// grid and corrected by steps on others.
__device__ __forceinline__ int sample_at(const SliceShared& s, float x) {
  int j = min(max((int)((x - s.xw[0]) * s.inv), 1), kWin - 2);
  const float x0 = s.xw[j - 1], x1 = s.xw[j], x2 = s.xw[j + 1];
  if (x0 < x && x <= x2) return x <= x1 ? j : j + 1;
  while (j > 1 && s.xw[j - 1] >= x) --j;
  while (j < kWin - 1 && s.xw[j] < x) ++j;
  return j;
}

// First sample of a slice's window: a few below the lowest place of its first node (lambda
// before the Doppler shift), by a 32-way search of one warp.
__device__ __forceinline__ int window_start(const float* __restrict__ wt, int n_t, float lambda,
                                            int lane) {
  const float x = lambda * (1.f - kAlphaMax);
  int lo = 0, hi = n_t + 2 * kExt;  // the first sample >= x is in [lo, hi]
  while (hi - lo > 0) {
    const int step = (hi - lo + 31) / 32;
    const int e = lo + lane * step;
    const unsigned below = __ballot_sync(0xffffffffu, e < hi && x_ext(wt, n_t, e) < x);
    const int k = __popc(below);  // samples lo, lo + step, .. below x
    const int new_hi = min(hi, lo + k * step);
    lo = k == 0 ? lo : lo + (k - 1) * step + 1;
    hi = k == 0 ? lo : new_hi;
  }
  return max(lo - 3, 0);
}

// The slice with the most items left, if more than `least`; -1 else.
__device__ __forceinline__ int busiest_slice(const int* next, int n_slices, int total, int least) {
  int best = -1, most = least;
  for (int q = 0; q < n_slices; ++q) {
    const int left = total - *(volatile const int*)&next[q];
    if (left > most) {
      most = left;
      best = q;
    }
  }
  return best;
}

int rough_blocks(long long n) {
  return (int)std::min<long long>((n + kRoughThreads / 32 - 1) / (kRoughThreads / 32),
                                  (long long)sm_count() * kRoughBlocks);
}

int kpad_of(int n_wave) { return (n_wave + 31) / 32 * 32; }

// Grid extrema and used alpha rows.
int node_setup(const CubeInputs& in, const float* dust_e, NodeCtrl* ctrl, cudaStream_t st) {
  const long long work = std::max<long long>(std::max(in.n_wave_t, in.n_wave), in.n);
  const int g = (int)std::min<long long>((work + 255) / 256, (long long)sm_count() * 8);
  const int need = (std::max(in.n_wave_t, in.n_wave) + 255) / 256;
  node_setup_kernel<<<std::max(g, need), 256, 0, st>>>(in.ssp_wave_z, in.n_wave, in.wave_t,
                                                       in.n_wave_t, in.vel, in.vel_stride,
                                                       in.vel_comp, in.n, dust_e, ctrl);
  RUBIX_LAUNCH_CHECK("node_setup_kernel");
  return RUBIX_OK;
}

// Prefix sums and resampling weights, the T' table: two launches.
int node_build_tables(const CubeInputs& in, const float* dust_e, double* prefix, float* h,
                      float* H, float* rough, NodeCtrl* ctrl, CubeCtrl* cc, cudaStream_t st) {
  const int n_templ = in.n_met * in.n_age, nW = in.n_wave, kpad = kpad_of(nW);
  node_tables_kernel<<<n_templ + kWeightBlocks + 1, kPrefixThreads, 0, st>>>(
      in.ssp_flux, n_templ, nW, in.ssp_wave_z, in.wave_t, in.n_wave_t, prefix, h, kpad, rough,
      dust_e != nullptr, ctrl, cc);
  RUBIX_LAUNCH_CHECK("node_tables_kernel");
  node_table_product_kernel<<<dim3((n_templ + 31) / 32, kAlphaTiles), 128, 0, st>>>(
      h, kpad, in.ssp_flux, n_templ, nW, in.wave_t, in.n_wave_t, dust_e != nullptr, rough, ctrl, H);
  RUBIX_LAUNCH_CHECK("node_table_product_kernel");
  return RUBIX_OK;
}

// The workspace of what is left to the general kernels (grad: the adjoint's, which has no
// partial spectra).
NodeFallback carve_fallback(Carve& c, const CubeInputs& in, int chunk, bool grad) {
  NodeFallback f{};
  f.At = c.take<float>((size_t)in.n_wave_t);
  f.bucket = c.take<int2>(kBuckets);
  f.ct = c.take<float4>((size_t)(in.n_met - 1) * (in.n_age - 1) * in.n_wave);
  f.rec = c.take<ParticleRec>((size_t)in.n);
  f.done = c.take<int>((size_t)in.n_seg);
  f.slot_start = c.take<int>((size_t)in.n_seg);
  f.chunk = chunk;
  f.alo = (float)std::exp(-kVmaxKms / kSpeedOfLight);
  f.ahi = (float)std::exp(kVmaxKms / kSpeedOfLight);
  f.items = c.take<int2>((size_t)max_slots(in.n, chunk) + in.n_seg);
  if (!grad)
    f.partials = c.take<float>((size_t)max_slots(in.n, chunk) * in.n_wave_t);
  return f;
}

size_t fallback_bytes(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk,
                      bool grad) {
  CubeInputs in{};
  in.n_met = nZ;
  in.n_age = nA;
  in.n_wave = nW;
  in.n_wave_t = n_t;
  in.n_seg = n_seg;
  in.n = n;
  Carve c(nullptr);
  carve_fallback(c, in, chunk, grad);
  return c.off;
}

// What the general kernel reads (cube_prepare's setup passes), when a spaxel is flagged: the
// tables over the grids, the flagged spaxels' items and the records of their particles.
__global__ void __launch_bounds__(256) node_fallback_kernel(CubeInputs in, NodeFallback f,
                                                            const double* __restrict__ prefix,
                                                            NodeFlags flags,
                                                            CubeCtrl* __restrict__ ctrl,
                                                            bool grad) {
  const NodeCtrl* nc = flags.ctrl;
  if (!nc->flagged) return;
  __shared__ int s_cnt[3], s_at[3];
  const int tid = threadIdx.x;
  const int gtid = blockIdx.x * 256 + tid, gsz = gridDim.x * 256;
  const double lnq0 = ctrl->lnq0, h = ctrl->h;
  for (int t = gtid; t < in.n_wave_t; t += gsz)
    f.At[t] = (float)((log((double)in.wave_t[t]) - lnq0) / h);
  for (int b = gtid; b < kBuckets; b += gsz)
    f.bucket[b] = bucket_entry(in.ssp_wave_z, in.n_wave, lnq0, h, b);
  const int at1 = nc->left[0], at2 = at1 + nc->left[1];
  if (gtid == 0) ctrl->n_items = at2 + nc->left[2];
  // 256 spaxels at a time: places within the block, then the block's in the list
  for (long long s0 = blockIdx.x * 256LL; s0 < in.n_seg; s0 += gsz) {
    const long long s = s0 + tid;
    const bool on = s < in.n_seg && flags.flags[s];
    int n = 0, p = 0, at = 0;
    if (on) p = flags.place((int)s, n);
    __syncthreads();
    if (tid < 3) s_cnt[tid] = 0;
    __syncthreads();
    if (on) at = atomicAdd(&s_cnt[p], n);
    __syncthreads();
    if (tid < 3 && s_cnt[tid] > 0) s_at[tid] = atomicAdd(&flags.ctrl->listed[tid], s_cnt[tid]);
    __syncthreads();
    if (on) {
      at += s_at[p] + (p == 0 ? 0 : (p == 1 ? at1 : at2));
      f.slot_start[s] = at;
      f.done[s] = 0;
      for (int c = 0; c < n; ++c) f.items[at + c] = make_int2((int)s, c);
    }
  }
  corner_table(in.ssp_flux, in.n_met, in.n_age, in.n_wave, f.ct, gtid, gsz);
  const long long n_valid = in.seg_off[in.n_seg];
  for (long long j = gtid; j < n_valid && j < in.n; j += gsz) {
    int lo = 0, hi = in.n_seg - 1;  // the spaxel of place j: the last that starts at or before it
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (in.seg_off[mid] <= j) lo = mid; else hi = mid - 1;
    }
    if (!flags.flags[lo]) continue;
    gather_records(in.mass, in.met, in.age, in.vel, in.vel_stride, in.vel_comp, in.perm,
                   in.seg_off, in.n_seg, in.ssp_met, in.n_met, in.ssp_age, in.n_age,
                   in.ssp_wave_z, in.n_wave, in.wave_t, in.n_wave_t, prefix, ctrl->inv_h,
                   ctrl->bmax, __uint_as_float(~nc->dz_inv), __uint_as_float(nc->dt_max), f.rec,
                   grad ? 1 : 0, in.av, f.alo, f.ahi, j, j + 1, 1);
  }
}

}  // namespace
}  // namespace rubix
