// The datacube accumulated node by node: the forward of kernel (b) for template grids
// that fit an SM's shared memory, wavelength slice by wavelength slice.
//
// A particle adds beta * I(x_t) to its spaxel, with I the piecewise-linear interpolant of
// its mixed template on the shifted grid lambda'_k = fl32(lambda_z,k * alpha) and
// beta = m T / T' (rubix/spectra/ifu.py:224-266).  Two properties of the path make the
// work per particle proportional to the SSP nodes inside the telescope range (737 at
// MUSE's 3721 bins on a 1221-node template) instead of to the telescope bins:
//
//   * T' = sum_t I_t dlambda_t is linear in the template, T' = sum_c w_c H_c(alpha) over
//     the four corners c, and H_c(alpha) is smooth in alpha.  H is tabulated at
//     alpha_i = 1 + i 2^-18 (1.1 km/s apart, exact in float32) for every template by one
//     small matrix product and interpolated linearly: 2e-8 of T' rms on the synthetic
//     templates (lines of 45 % depth, 2-8 A wide), below float32 rounding.  The error grows
//     with a template's kinks; it is bounded template by template, and a particle of a rougher
//     one (emission lines) has its T' summed on its own grid.  beta is then known before any
//     spectrum is formed.
//   * Inside one SSP interval the particle's spectrum is A + B (x - x_j).  A lane owns an
//     SSP node; while alpha moves by less than one telescope bin the samples strictly
//     between two nodes stay the same, so the lane sums (A, B) of its interval over all
//     particles in registers and only the sample at the node itself needs a choice of
//     side.  The sums are spread over the 4-5 samples of the interval once per group of
//     particles instead of once per particle.
//
// Measured (221 x 6 x 1221 templates, 3721 samples, LSF fused, one GB300): 10^7 particles on
// 300 x 300 spaxels, whole render 12.3 ms against 40.2 ms with every particle evaluated at
// every sample (this file's slice kernel 8.4 ms of it, cube_main_kernel 38.5 ms); 10^6 on
// 150 x 150, 1.67 ms against 4.46 ms.  Relative 2-norm error against float64 7.6e-8, as before.
//
// Stages: grid extrema and the velocity range; the work-item list, without the spaxels that
// velocities rule out; prefix sums of the templates, their roughness and the resampling
// weights at alpha_i; H; records of every item sorted by alpha, and those of rough
// templates; the slice kernel; the merge of the slices (and chunks) of a spaxel with the
// optional LSF.  A spaxel with any particle that the tables do not cover
// (a shifted grid that does not span the telescope range, |v| above 2300 km/s, values
// that are not finite or that may overflow) is flagged and left to cube_main_kernel, as
// is everything when the grids themselves do not qualify.  Within the path every decision
// depends on the configuration and the spaxel's own particles only, so a spaxel's result does
// not depend on what else is rendered with it; whether a call takes the path at all is chosen
// by its sizes (cube_nodes_worth).
#include "cube_nodes.cuh"
#include "node_tables.cuh"

#include <type_traits>

namespace rubix {
namespace {

constexpr int kItem = 4 * kSub;  // particles of a work item
// Warps of a slice block: 20 where the sums fit 102 registers (2 % over 16), 16 where every
// sample is held (1505 us with 20 against 1402 for 5 10^5 dusty particles).
template <bool kDust>
constexpr int kNodeWarps = kDust ? 16 : 20;

// Work items: ranges of up to kItem particles of one spaxel; empty and flagged spaxels have
// none.  Spaxels of several items first (item index = row), then those with many particles.
__device__ __forceinline__ void node_count(const CubeInputs& in, const NodeFlags& flags, bool dust,
                                           int big, int* multi, int* large, int* small) {
  screened_counts(in, flags, dust, kItem, [&](int s, int cnt) {
    multi[s] = cnt > kItem ? (cnt + kItem - 1) / kItem : 0;
    large[s] = (cnt <= kItem && cnt >= big) ? 1 : 0;
    small[s] = (cnt < big && cnt > 0) ? 1 : 0;
  });
}

__global__ void __launch_bounds__(256) node_count_kernel(CubeInputs in, NodeFlags flags, bool dust,
                                                         int big, int* multi, int* large,
                                                         int* small) {
  node_count(in, flags, dust, big, multi, large, small);
}

// Item index of chunk 0 of a spaxel (its chunks follow one another).
__device__ __forceinline__ int first_item(int s, int cnt, int big, int n_seg, const int* multi,
                                          const int* large, const int* small) {
  if (cnt > kItem) return multi[s];
  if (cnt >= big) return multi[n_seg] + large[s];
  return multi[n_seg] + large[n_seg] + small[s];
}

__device__ __forceinline__ void node_fill_items(const int* seg_off, const int* flags, int n_seg,
                                                int big, const int* multi, const int* large,
                                                const int* small, int2* items, NodeCtrl* ctrl) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n_seg; s += gridDim.x * blockDim.x) {
    const int cnt = seg_off[s + 1] - seg_off[s];
    if (cnt == 0 || flags[s]) continue;
    const int i0 = first_item(s, cnt, big, n_seg, multi, large, small);
    for (int c = 0; c * kItem < cnt; ++c) items[i0 + c] = make_int2(s, c);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctrl->n_multi = multi[n_seg];
    ctrl->n_items = multi[n_seg] + large[n_seg] + small[n_seg];
  }
}

__global__ void node_fill_items_kernel(const int* seg_off, const int* flags, int n_seg, int big,
                                       const int* multi, const int* large, const int* small,
                                       int2* items, NodeCtrl* ctrl) {
  node_fill_items(seg_off, flags, n_seg, big, multi, large, small, items, ctrl);
}

// All three steps by one block.
__global__ void __launch_bounds__(1024) node_items_kernel(CubeInputs in, NodeFlags flags,
                                                          bool dust, int big, int* multi,
                                                          int* large, int* small, int2* items) {
  node_count(in, flags, dust, big, multi, large, small);
  __syncthreads();
  scan_exclusive_block(multi, in.n_seg, 1);
  scan_exclusive_block(large, in.n_seg, 1);
  scan_exclusive_block(small, in.n_seg, 1);
  __syncthreads();
  node_fill_items(in.seg_off, flags.flags, in.n_seg, big, multi, large, small, items, flags.ctrl);
}

struct GatherArgs {
  CubeInputs in;
  const double* prefix;
  const float* H;
  NodeCtrl* ctrl;
  const int2* items;
  float4* rec_w;
  float2* rec_a;
  float* rec_av;  // dust only
  NodeFlags flags;
  int4* desc;
  int2* rough;  // records of rough particles, and their spaxels
};

// Largest dust transmission that a column lets through (2^(e A_V) over all wavelengths).
__device__ __forceinline__ float dust_top(const GatherArgs& a, float av) {
  if (!a.rec_av) return 1.f;
  const float up = fmaxf(__uint_as_float(a.ctrl->e_hi) * av, -__uint_as_float(a.ctrl->e_lo) * av);
  return isfinite(av) ? exp2f(fmaxf(up, 0.f)) : kFltMax;
}

// The record of a particle (beta times the corner weights); true: its spaxel is left to the
// general kernel.
__device__ __forceinline__ bool node_record(const GatherArgs& a, const NodeParticle& q,
                                            long long i, float av, float4& w) {
  const float mass = a.in.mass[i];
  const float beta = mass != 0.f ? mass * (q.T / q.Tp) : 0.f;
  const float top = fabsf(beta) * __uint_as_float(a.ctrl->fmax);  // without dust dust_top is 1
  // what the general kernel treats specially, or what may leave float32's range; a
  // particle outside the templates has no spectrum unless 0 times its mass or its
  // transmission is not 0
  if (q.outside && !q.bad) return !isfinite(mass) || !(dust_top(a, av) < 1e30f);
  w = make_float4(beta * q.w[0], beta * q.w[1], beta * q.w[2], beta * q.w[3]);
  return q.bad || !(top * dust_top(a, av) < 1e30f) || (beta != 0.f && !(top > 1e-25f));
}

// One block per work item: the record of each particle (beta times the four corner
// weights; alpha and the byte offset of its first corner row in the slice table), sorted
// by alpha within runs of kSub (ties by input order: the order is a function of the
// spaxel's particles alone).  Latency-bound on the gathers through the permutation.
// A particle of a rough template leaves what node_rough_kernel needs in the record's place.
__global__ void __launch_bounds__(kSub) node_gather_kernel(GatherArgs a) {
  __shared__ __align__(16) unsigned s_key[kSub];
  __shared__ float s_lo[kSub / 32], s_hi[kSub / 32];
  __shared__ NodePlan s_plan;
  __shared__ int s_flag;
  const CubeInputs& in = a.in;
  const int tid = threadIdx.x;
  const float x1 = in.wave_t[in.n_wave_t - 1];
  if (tid == 0) s_plan = node_plan(a.ctrl, in.n_wave, x1, a.rec_av != nullptr);
  __syncthreads();
  const NodePlan plan = s_plan;
  const int n_items = a.ctrl->n_items;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int2 it = a.items[item];
    const int seg_b = in.seg_off[it.x], seg_e = in.seg_off[it.x + 1];
    const int jb = seg_b + it.y * kItem;
    const int je = min(jb + kItem, seg_e);
    float amin = 2.f, amax = 0.f;
    if (tid == 0) s_flag = !plan.ok;
    __syncthreads();
    for (int j0 = jb; j0 < je && plan.ok; j0 += kSub) {
      const int m = min(kSub, je - j0);
      float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
      float alpha = 1.f, av = 0.f;
      int row = 0;
      bool rough = false;
      if (tid < m) {
        const long long i = in.perm[j0 + tid];
        const NodeParticle q = node_particle(in, a.prefix, a.H, i);
        if (a.rec_av) av = in.av[i];
        alpha = q.alpha;
        row = q.row;
        rough = q.rough;
        if (rough) {
          w = make_float4(q.tz, q.ta, q.T, __int_as_float((int)i));
        } else if (node_record(a, q, i, av, w)) {
          s_flag = 1;
        }
      }
      s_key[tid] = tid < m ? __float_as_uint(alpha) : 0xffffffffu;
      __syncthreads();
      if (tid < m) {
        amin = fminf(amin, alpha);
        amax = fmaxf(amax, alpha);
        const int at = j0 + run_rank(s_key, m, tid);
        a.rec_w[at] = w;
        a.rec_a[at] = make_float2(alpha, __int_as_float(row * 128));
        if (a.rec_av) a.rec_av[at] = av;
        if (rough) a.rough[rough_place(a.ctrl)] = make_int2(at, it.x);
      }
      __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      amin = fminf(amin, __shfl_xor_sync(0xffffffffu, amin, o));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    }
    if ((tid & 31) == 0) {
      s_lo[tid >> 5] = amin;
      s_hi[tid >> 5] = amax;
    }
    __syncthreads();
    if (tid == 0) {
      for (int q = 1; q < kSub / 32; ++q) {
        amin = fminf(amin, s_lo[q]);
        amax = fmaxf(amax, s_hi[q]);
      }
      a.desc[item] = make_int4(jb, je - jb, __float_as_int(amin), __float_as_int(amax));
      // the samples a node crosses within the item must fit the row
      if (s_flag || too_wide(plan, amin, amax, x1)) a.flags.leave(it.x);
    }
    __syncthreads();
  }
}

// The records of rough particles, a warp each.  Bound by issue (0.63 per cycle) and shared-memory
// wavefronts (69 %) together, about 1600 instructions a particle of 740 nodes: 2.0 ms for 10^6
// (all of them rough: forward 1.94 -> 4.0 ms, where the general path takes 4.05), with two
// blocks an SM and two rounds of nodes in flight; 2.2 with one, 2.0 with three blocks or four
// rounds.  One warp summed a
// whole sorted run's in the gather before: 18 ms.
__global__ void __launch_bounds__(kRoughThreads, kRoughBlocks) node_rough_kernel(GatherArgs a) {
  const int n = a.ctrl->n_rough;
  if (n == 0) return;
  extern __shared__ __align__(16) float4 s_tab4[];
  __shared__ NodePlan s_plan;
  const CubeInputs& in = a.in;
  if (threadIdx.x == 0)
    s_plan = node_plan(a.ctrl, in.n_wave, in.wave_t[in.n_wave_t - 1], a.rec_av != nullptr);
  const bool even = sample_table(in.wave_t, in.n_wave_t, s_tab4);
  const NodePlan plan = s_plan;
  for (int e = (blockIdx.x * kRoughThreads + threadIdx.x) >> 5; e < n;
       e += gridDim.x * (kRoughThreads / 32)) {
    const int2 at = a.rough[e];
    const float4 rec = a.rec_w[at.x];
    NodeParticle q;
    corner_weights(rec.x, rec.y, q.w);
    q.T = rec.z;
    q.Tp = rough_tprime(in, plan, s_tab4, even, a.rec_a[at.x], q.w);
    q.outside = false;
    q.bad = bad_scale(q.T, q.Tp);
    const long long i = __float_as_int(rec.w);
    float4 w;
    const bool bad = node_record(a, q, i, a.rec_av ? in.av[i] : 0.f, w);
    if ((threadIdx.x & 31) == 0) {
      a.rec_w[at.x] = w;
      if (bad) a.flags.leave(at.y);
    }
  }
}

struct SliceArgs {
  const float* flux;
  const float* wz;
  const float* wt;
  int n_templ, n_age, n_wave, n_t;
  const int4* desc;  // per item: first record, records, smallest and largest alpha
  const float4* rec_w;
  const float2* rec_a;
  const float* rec_av;  // dust only, with the exponents per telescope wavelength
  const float* dust_e;
  float* rows;    // [row][slice][kMaxBins]
  int2* row_pos;  // [row][slice]: first extended sample, samples
  NodeCtrl* ctrl;
  int wave, multi_rows, n_seg;
  long long slice_rows;  // rows of kMaxBins samples in the workspace
};

// Single-item spaxels of a wave: as many as the rows left by the others hold.
__device__ __forceinline__ int wave_size(long long slice_rows, int n_slices, int multi_rows,
                                         int n_seg) {
  return (int)min((long long)n_seg, slice_rows / n_slices - multi_rows);
}

// Items [i0, i1) of a wave: wave 0 holds every item of a several-item spaxel and the first
// wave_items others, wave w the next wave_items.  Item i uses row i when it is one of
// several, else the row of its place in the wave.
__device__ __forceinline__ void wave_range(const NodeCtrl* c, int wave, int wave_items, int& i0,
                                           int& i1) {
  const int s0 = c->n_multi + wave * wave_items;
  i0 = wave == 0 ? 0 : min(s0, c->n_items);
  i1 = min(s0 + wave_items, c->n_items);
}
__device__ __forceinline__ int item_row(int item, int n_multi, int wave, int wave_items,
                                        int multi_rows) {
  return item < n_multi ? item : multi_rows + (item - n_multi - wave * wave_items);
}

// One item by one warp on one slice: NPL nodes per lane (two or four, in packed pairs), NPL
// particles at a time, each on 32 / NPL lanes.
//
// A group holds particles whose alpha differ by less than W telescope bins.  With j the
// first sample at or right of node l at the group's first alpha, node l (1..n_own of the
// slice) fills the samples from j to the next node's; with t = x_j - lambda'_l it sums
//   A = sum (G_l + s_l t), B = sum s_l    the right interval's line, the value from j+W on
//   D_m = sum (s_{l-1} - s_l) min(t, -d_m), m < W, d_m = x_{j+m} - x_j: the samples that the
//         node crosses lie on the left line (slope sum B of node l - 1) while t < -d_m, so
//         f_{j+m} = A + D_m + d_m B_{l-1}.
// The groups are the same for every slice: neighbours agree on who fills a sample.
template <int NPL, int W>
struct SliceItem {
  static constexpr int LPG = 32 / NPL;  // lanes of a particle
  static constexpr int PR = NPL / 2;    // packed pairs of nodes
  const SliceShared& sh;
  const int lane, i, g, own, nxt_lane, prv_lane;
  const bool mine;
  const float lam_own;
  float2 nlam[PR];  // minus the wavelengths: -lambda' comes from one packed product
  float nlam_r;
  const char* tab;

  __device__ __forceinline__ SliceItem(const SliceShared& s, int lane_, int n_own,
                                       const float* __restrict__ lam)
      : sh(s), lane(lane_), i(lane_ & (LPG - 1)), g(lane_ / LPG), own(i * NPL + g),
        nxt_lane((((own + 1) % NPL) * LPG + (own + 1) / NPL) & 31),
        prv_lane(own == 0 ? 0 : ((own - 1) % NPL) * LPG + (own - 1) / NPL),
        mine(own >= 1 && own <= n_own), lam_own(lam[own]) {
#pragma unroll
    for (int q = 0; q < PR; ++q)
      nlam[q] = make_float2(-lam[i * NPL + 2 * q], -lam[i * NPL + 2 * q + 1]);
    nlam_r = -lam[i * NPL + NPL];
    tab = reinterpret_cast<const char*>(s.tab) + i * (4 * NPL);
  }

  int j;
  float xo, xo1;                   // samples j and (W > 1) j + 1 of the node this lane collects
  float2 xj[PR], dm[PR], A[PR], B[PR], D[W][PR];

  // Reduction over the particle groups; lane (g, i) ends with the sum of node i*NPL + g.
  __device__ __forceinline__ float collect(const float2 (&v)[PR]) const {
    if constexpr (NPL == 2) {
      return (g ? v[0].y : v[0].x) + __shfl_xor_sync(0xffffffffu, g ? v[0].x : v[0].y, 16);
    } else {
      const bool h = g & 2, l = g & 1;
      const float a0 =
          (h ? v[1].x : v[0].x) + __shfl_xor_sync(0xffffffffu, h ? v[0].x : v[1].x, 16);
      const float a1 =
          (h ? v[1].y : v[0].y) + __shfl_xor_sync(0xffffffffu, h ? v[0].y : v[1].y, 16);
      return (l ? a1 : a0) + __shfl_xor_sync(0xffffffffu, l ? a0 : a1, 8);
    }
  }
  // The owner lanes' value for every node of this lane.
  __device__ __forceinline__ void spread(float v, float2 (&o)[PR]) const {
#pragma unroll
    for (int q = 0; q < PR; ++q) {
      o[q].x = __shfl_sync(0xffffffffu, v, 2 * q * LPG + i);
      o[q].y = __shfl_sync(0xffffffffu, v, (2 * q + 1) * LPG + i);
    }
  }

  __device__ __forceinline__ void open(float alpha) {
    j = sample_at(sh, __fmul_rn(lam_own, alpha));
    xo = sh.xw[j];
    spread(xo, xj);
    if constexpr (W > 1) {
      xo1 = sh.xw[j + 1];
      spread(xo - xo1, dm);
    }
#pragma unroll
    for (int q = 0; q < PR; ++q) {
      A[q] = B[q] = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < W; ++m) D[m][q] = make_float2(0.f, 0.f);
    }
  }

  // The group's sums to this warp's samples.  Every sample has one lane.
  __device__ __forceinline__ void flush(int jb) {
    const float s0 = collect(A), s1 = collect(B);
    const float p0 = s0 + collect(D[0]);
    float p1 = 0.f;
    if constexpr (W > 1) p1 = s0 + collect(D[1]);
    const int jn = __shfl_sync(0xffffffffu, j, nxt_lane);
    if constexpr (W > 1) {
      const float left = __shfl_sync(0xffffffffu, s1, prv_lane);
      p1 = fmaf(xo1 - xo, left, p1);
    }
    if (mine) {
      float* f = sh.f - jb;
      const int e1 = min(jn, jb + kMaxBins);  // the window checks keep every sample inside
      constexpr int U = 4;                    // samples inside the interval taken together
      float v[U], x[U];
      const bool in = j + W <= e1;
      const float f0 = in ? f[j] : 0.f;
      const float f1 = in && W > 1 ? f[j + 1] : 0.f;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = j + W + u;
        v[u] = e < e1 ? f[e] : 0.f;
        x[u] = e < e1 ? sh.xw[e] : 0.f;
      }
      if (in) {
        f[j] = f0 + p0;
        if (W > 1) f[j + 1] = f1 + p1;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = j + W + u;
        if (e < e1) f[e] = v[u] + fmaf(s1, x[u] - xo, s0);
      }
      for (int e = j + W + U; e < e1; ++e) f[e] += fmaf(s1, sh.xw[e] - xo, s0);
    }
    __syncwarp();
  }

  // What a step reads of its NPL particles, loaded a step ahead; r: this lane's record.
  struct Loaded {
    float2 c[4][PR];
    float w[4], alpha;
  };
  __device__ __forceinline__ void load(int r, int zoff, Loaded& v) const {
    const StagedRecs& st = *sh.st;
    const char* t0 = tab + st.row[r];
    const char* t1 = t0 + zoff;
    const char* tc[4] = {t0, t1, t0 + 128, t1 + 128};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v.w[k] = st.w[k][r];
      if constexpr (NPL == 2) {
        v.c[k][0] = *reinterpret_cast<const float2*>(tc[k]);
      } else {
        const float4 x = *reinterpret_cast<const float4*>(tc[k]);
        v.c[k][0] = make_float2(x.x, x.y);
        v.c[k][PR - 1] = make_float2(x.z, x.w);
      }
    }
    v.alpha = st.alpha[r];
  }
  __device__ __forceinline__ void step(const Loaded& v) {
    float2 G[PR];
    const float2 w0 = make_float2(v.w[0], v.w[0]), w1 = make_float2(v.w[1], v.w[1]);
    const float2 w2 = make_float2(v.w[2], v.w[2]), w3 = make_float2(v.w[3], v.w[3]);
    const float2 al = make_float2(v.alpha, v.alpha);
    const auto& c = v.c;
    float2 nlp[PR], s[PR];
#pragma unroll
    for (int q = 0; q < PR; ++q) {
      G[q] = __fmul2_rn(w0, c[0][q]);
      G[q] = __ffma2_rn(w1, c[1][q], G[q]);
      G[q] = __ffma2_rn(w2, c[2][q], G[q]);
      G[q] = __ffma2_rn(w3, c[3][q], G[q]);
      nlp[q] = __fmul2_rn(nlam[q], al);
    }
    const float G_r = __shfl_down_sync(0xffffffffu, G[0].x, 1, LPG);
    const float nlp_r = __fmul_rn(nlam_r, al.x);
#pragma unroll
    for (int q = 0; q < PR; ++q) {
      const float Gn = q + 1 < PR ? G[q + 1 < PR ? q + 1 : 0].x : G_r;
      const float ln = q + 1 < PR ? nlp[q + 1 < PR ? q + 1 : 0].x : nlp_r;
      const float2 r = make_float2(fast_rcp(nlp[q].x - nlp[q].y), fast_rcp(nlp[q].y - ln));
      s[q] = __fmul2_rn(make_float2(G[q].y - G[q].x, Gn - G[q].y), r);
    }
    const float s_l = __shfl_up_sync(0xffffffffu, s[PR - 1].y, 1, LPG);
#pragma unroll
    for (int q = 0; q < PR; ++q) {
      const float2 t = __fadd2_rn(xj[q], nlp[q]);
      const float sp = q > 0 ? s[q > 0 ? q - 1 : 0].y : s_l;
      const float2 d = make_float2(sp - s[q].x, s[q].x - s[q].y);
      D[0][q] = __ffma2_rn(d, make_float2(fminf(t.x, 0.f), fminf(t.y, 0.f)), D[0][q]);
      if constexpr (W > 1)
        D[1][q] = __ffma2_rn(d, make_float2(fminf(t.x, dm[q].x), fminf(t.y, dm[q].y)), D[1][q]);
      A[q] = __fadd2_rn(A[q], __ffma2_rn(s[q], t, G[q]));
      B[q] = __fadd2_rn(B[q], s[q]);
    }
  }
};

// The same with a dust column in front of every particle: its spectrum is multiplied by
// 2^(e_t A_V) (spectra/dust/dust_baseclasses.py:163-164), so every sample is evaluated, one
// node and its up to M samples per lane, one particle at a time.  The group's samples, their
// exponents and sums stay in registers.  Bound by the 2^x rate (16 a cycle and SM) and issue:
// about 60 instructions and 7 multi-function ones per particle and 32 nodes.
template <int M>
struct DustItem {
  static constexpr int W = 2;
  const SliceShared& sh;
  const int lane;
  const bool mine;
  const float lam, lam_r;
  const char* tab;
  int j;
  float xo, d[M], e[M], acc[M];

  __device__ __forceinline__ DustItem(const SliceShared& s, int lane_, int n_own,
                                      const float* __restrict__ l)
      : sh(s), lane(lane_), mine(lane_ >= 1 && lane_ <= n_own), lam(l[lane_]),
        lam_r(l[lane_ + 1]), tab(reinterpret_cast<const char*>(s.tab) + 4 * lane_) {}

  __device__ __forceinline__ void open(float alpha) {
    j = sample_at(sh, __fmul_rn(lam, alpha));
    xo = sh.xw[j];
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int q = min(j + m, kWin - 1);
      d[m] = sh.xw[q] - xo;
      e[m] = sh.ew[q];
      acc[m] = 0.f;
    }
  }

  __device__ __forceinline__ void flush(int jb) {
    const int jn = __shfl_down_sync(0xffffffffu, j, 1);
    if (mine) {
      float* f = sh.f - jb;
      const int e1 = min(jn, jb + kMaxBins);
      float v[M];
#pragma unroll
      for (int m = 0; m < M; ++m) v[m] = j + m < e1 ? f[j + m] : 0.f;
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (j + m < e1) f[j + m] = v[m] + acc[m];
    }
    __syncwarp();
  }

  struct Loaded {
    float c[4], w[4], alpha, av;
  };
  __device__ __forceinline__ void load(int r, int zoff, Loaded& v) const {
    const StagedRecs& st = *sh.st;
    const char* t0 = tab + st.row[r];
    v.c[0] = *reinterpret_cast<const float*>(t0);
    v.c[1] = *reinterpret_cast<const float*>(t0 + zoff);
    v.c[2] = *reinterpret_cast<const float*>(t0 + 128);
    v.c[3] = *reinterpret_cast<const float*>(t0 + zoff + 128);
#pragma unroll
    for (int k = 0; k < 4; ++k) v.w[k] = st.w[k][r];
    v.alpha = st.alpha[r];
    v.av = sh.st_av[r];
  }
  __device__ __forceinline__ void step(const Loaded& v) {
    float G = v.w[0] * v.c[0];
    G = fmaf(v.w[1], v.c[1], G);
    G = fmaf(v.w[2], v.c[2], G);
    G = fmaf(v.w[3], v.c[3], G);
    const float lp = __fmul_rn(lam, v.alpha);
    const float G_r = __shfl_down_sync(0xffffffffu, G, 1);
    const float s = (G_r - G) * fast_rcp(__fmul_rn(lam_r, v.alpha) - lp);
    const float s_l = __shfl_up_sync(0xffffffffu, s, 1);
    const float t = xo - lp;
    const float base = fmaf(s, t, G);
    const float c = s_l - s;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float y = fmaf(s, d[m], base);
      if (m < W) y = fmaf(c, fminf(t + d[m], 0.f), y);
      acc[m] = fmaf(y, dust_transmission(e[m], v.av), acc[m]);
    }
  }
};

template <class T>
struct TypeOf {
  using type = T;
};

// Item of a warp: its first record and record count, its smallest and largest alpha.
struct ItemDesc {
  int p0, np;
  float lo, hi;
};

// The slice kernel: a block holds one slice (32 nodes) of every template in shared memory
// and its warps take the work items in turn, so a particle's corners cost four shared
// loads per 32 nodes (13 KB per particle in all, 40 TB/s over the chip) instead of the same
// bytes from L2.  Bound by shared-memory wavefronts (63 % of the pipe) and issue (0.65 per
// cycle) together at 409 us for 4 10^5 particles on 60 x 60 spaxels; a step's operands are
// loaded one step ahead (483 us without), 20 warps hide more latency than 16 or 12 (+2 %,
// +15 %), four nodes a lane beat two by 6 % and one by 8 %, W = 2 needs half the flushes of
// W = 1, W = 3 costs more per step than it saves.  A warp's next item, its description and its first records are fetched while the one before
// is processed.  A block whose slice has no items left takes the slice with the most.
template <class Item, int NPL, bool kDust>
__device__ __forceinline__ void slice_items(const SliceArgs& a, const SliceShared& sh,
                                            const float* s_lam, int n_own, int lane, int slice,
                                            int n_slices, int i0, int total, int e0, float w_seg,
                                            int n_multi, int wave_items, int* __restrict__ next) {
  Item w(sh, lane, n_own, s_lam);
  const int grp = lane / (32 / NPL);  // the lane's particle of a step
  const int zoff = a.n_age * 128;
  const float lam_lo = s_lam[1], lam_hi = s_lam[n_own + 1];
  auto take = [&]() { return lane == 0 ? atomicAdd(next, 1) : 0; };
  auto describe = [&](int cur) {
    ItemDesc d{0, 0, 1.f, 1.f};
    if (cur < total) {
      const int4 v = a.desc[i0 + cur];
      d = ItemDesc{v.x, v.y, __int_as_float(v.z), __int_as_float(v.w)};
    }
    return d;
  };
  float4 rw = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 ra = make_float2(1.f, 0.f);
  float rv = 0.f;
  auto fetch = [&](int p, int n) {
    rw = make_float4(0.f, 0.f, 0.f, 0.f);
    ra = make_float2(1.f, 0.f);
    if (lane < n) {
      if (kDust) rv = a.rec_av[(long long)p + lane];
      rw = a.rec_w[(long long)p + lane];
      ra = a.rec_a[(long long)p + lane];
    }
  };
  int cur = __shfl_sync(0xffffffffu, take(), 0);
  int nxt = __shfl_sync(0xffffffffu, take(), 0);
  ItemDesc d = describe(cur), dn = describe(nxt);
  int nxt2_raw = take();
  fetch(d.p0, d.np);
  while (d.np > 0) {
    const int nxt2 = __shfl_sync(0xffffffffu, nxt2_raw, 0);
    const ItemDesc dn2 = describe(nxt2);
    nxt2_raw = take();
    const int jb = sample_at(sh, __fmul_rn(lam_lo, d.lo));
    bool open = false;
    float a_lim = 0.f;  // alpha at which the sample windows have to move
    for (int base = 0; base < d.np; base += 32) {
      const int cnt = min(32, d.np - base);
      __syncwarp();
      sh.st->w[0][lane] = rw.x;
      sh.st->w[1][lane] = rw.y;
      sh.st->w[2][lane] = rw.z;
      sh.st->w[3][lane] = rw.w;
      sh.st->alpha[lane] = ra.x;
      sh.st->row[lane] = __float_as_int(ra.y);
      if (kDust) sh.st_av[lane] = rv;
      const float al = ra.x;
      __syncwarp();
      if (base + 32 < d.np) fetch(d.p0 + base + 32, d.np - base - 32);
      else fetch(dn.p0, dn.np);
      bool fresh = (base & (kSub - 1)) == 0;  // a new sorted run
      int pos = 0;
      while (pos < cnt) {
        const float a0 = __shfl_sync(0xffffffffu, al, pos);
        if (!open || a0 >= a_lim || fresh) {
          if (open) w.flush(jb);
          w.open(a0);
          a_lim = a0 + w_seg;
          open = true;
          fresh = false;
        }
        const unsigned past =
            __ballot_sync(0xffffffffu, lane > pos && lane < cnt && al >= a_lim);
        const int end = past ? __ffs(past) - 1 : cnt;
        typename Item::Loaded v;
        w.load(pos + grp < end ? pos + grp : 32, zoff, v);  // 32: a record of weight zero
        for (int p = pos + NPL; p < end; p += NPL) {
          const typename Item::Loaded u = v;
          w.load(p + grp < end ? p + grp : 32, zoff, v);
          w.step(u);
        }
        w.step(v);
        pos = end;
      }
    }
    if (open) w.flush(jb);
    const int nb = min(sample_at(sh, __fmul_rn(lam_hi, d.hi)) - jb, kMaxBins);
    const long long row =
        (long long)item_row(i0 + cur, n_multi, a.wave, wave_items, a.multi_rows) * n_slices +
        slice;
    float* out = a.rows + row * kMaxBins;
    for (int b = lane; b < nb; b += 32) {
      out[b] = sh.f[b];
      sh.f[b] = 0.f;
    }
    if (lane == 0) a.row_pos[row] = make_int2(e0 + jb, nb);
    __syncwarp();
    cur = nxt;
    nxt = nxt2;
    d = dn;
    dn = dn2;
  }
}

template <bool kDust>
__global__ void __launch_bounds__(32 * kNodeWarps<kDust>, 1) node_slice_kernel(SliceArgs a) {
  constexpr int kWarps = kNodeWarps<kDust>, kThreads = 32 * kWarps;
  extern __shared__ __align__(16) unsigned char smem[];
  float* s_tab = reinterpret_cast<float*>(smem);
  float* s_xw = s_tab + (size_t)a.n_templ * 32;
  StagedRecs* s_st = reinterpret_cast<StagedRecs*>(s_xw + kWin);
  float* s_f = reinterpret_cast<float*>(s_st + kWarps);
  float* s_ew = s_f + kWarps * kMaxBins;  // dust only
  float* s_av = s_ew + kWin;
  __shared__ float s_lam[36];
  __shared__ NodePlan s_plan;
  __shared__ int s_slice, s_e0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float x_last = a.wt[a.n_t - 1];
  if (tid == 0) s_plan = node_plan(a.ctrl, a.n_wave, x_last, kDust);
  __syncthreads();
  const NodePlan plan = s_plan;
  if (!plan.ok) return;
  int i0, i1;
  const int wave_items = wave_size(a.slice_rows, plan.n_slices, a.multi_rows, a.n_seg);
  wave_range(a.ctrl, a.wave, wave_items, i0, i1);
  const int total = i1 - i0;
  if (total <= 0) return;
  SliceShared sh;
  sh.tab = s_tab;
  sh.xw = s_xw;
  sh.st = s_st + warp;
  sh.f = s_f + warp * kMaxBins;
  sh.ew = s_ew;
  sh.st_av = s_av + warp * kStage;
  if (lane == 0) {
    if (kDust) sh.st_av[32] = 0.f;
    for (int k = 0; k < 4; ++k) sh.st->w[k][32] = 0.f;
    sh.st->alpha[32] = 1.f;
    sh.st->row[32] = 0;
  }
  for (int b = lane; b < kMaxBins; b += 32) sh.f[b] = 0.f;
  int* next = a.ctrl->next[a.wave];
  int slice = (int)((long long)blockIdx.x * plan.n_slices / gridDim.x);
  const float w_seg =
      (float)plan.w * 0.98f * plan.dt_min * (1.f - kAlphaMax) / x_last - 2.4e-7f;

  for (;;) {
    const int k0 = plan.k_first - 1 + slice * plan.n_own;  // node of lane 0
    for (int r = warp; r < a.n_templ; r += kWarps) {
      const int k = k0 + lane;
      s_tab[r * 32 + lane] =
          (lane <= plan.n_own + 1 && k >= 0 && k < a.n_wave)
              ? a.flux[(long long)r * a.n_wave + k] : 0.f;
    }
    if (tid < 36) s_lam[tid] = lam_ext(a.wz, a.n_wave, k0 + tid);
    if (warp == 0) {
      const int e = window_start(a.wt, a.n_t, lam_ext(a.wz, a.n_wave, k0), lane);
      if (lane == 0) s_e0 = e;
    }
    __syncthreads();
    const int e0 = s_e0;
    for (int q = tid; q < kWin; q += kThreads) {
      s_xw[q] = x_ext(a.wt, a.n_t, e0 + q);
      if (kDust) s_ew[q] = a.dust_e[min(max(e0 + q - kExt, 0), a.n_t - 1)];
    }
    __syncthreads();
    sh.inv = (float)(kWin - 1) / (s_xw[kWin - 1] - s_xw[0]);
    auto run = [&](auto item, auto npl) {
      slice_items<typename decltype(item)::type, decltype(npl)::value, kDust>(
          a, sh, s_lam, plan.n_own, lane, slice, plan.n_slices, i0, total, e0, w_seg,
          a.ctrl->n_multi, wave_items, next + slice);
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    using I4 = std::integral_constant<int, 4>;
    if constexpr (kDust) {
      if (plan.most <= 4) run(TypeOf<DustItem<4>>{}, I1{});
      else if (plan.most <= 6) run(TypeOf<DustItem<6>>{}, I1{});
      else run(TypeOf<DustItem<kDustMost>>{}, I1{});
    } else {
      if (plan.w == 1) run(TypeOf<SliceItem<2, 1>>{}, I2{});
      else run(TypeOf<SliceItem<4, 2>>{}, I4{});
    }
    __syncthreads();
    if (tid == 0) s_slice = busiest_slice(next, plan.n_slices, total, 2 * kWarps);
    __syncthreads();
    slice = s_slice;
    if (slice < 0) return;
  }
}

struct MergeArgs {
  const int* seg_off;
  const int* multi;
  const int* large;
  const int* small;
  int n_seg, big, n_t, n_wave;
  const float* wt;
  const int* flags;
  const float* rows;
  const int2* row_pos;
  const NodeCtrl* ctrl;
  int wave, multi_rows;
  bool dust;
  long long slice_rows;
  float* cube;
  long long stride;
  int lsf_k, lsf_crop;
  float lsf[kMaxLsfTaps + 1];
};

constexpr int kMergeThreads = 256;

// One block per spaxel: the slices of its items summed (neighbouring slices share only the
// samples around their common node: even slices first, then odd ones; items with Kahan's
// compensation), then the LSF (rubix/telescope/lsf/lsf.py:29-105) and the store.  Empty
// spaxels are zero.  Bound by HBM: the rows once, the cube once.
template <int R>
__global__ void __launch_bounds__(kMergeThreads) node_merge_kernel(MergeArgs a) {
  extern __shared__ float s_buf[];
  __shared__ NodePlan s_plan;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_plan = node_plan(a.ctrl, a.n_wave, a.wt[a.n_t - 1], a.dust);
  __syncthreads();
  const int n_slices = s_plan.n_slices;
  const int K = a.lsf_k, n_t = a.n_t;
  const int lead = K > 0 ? K - 1 - a.lsf_crop : 0;
  const int pad = R * kMergeThreads + (K > 0 ? K : 0);  // s_spec: lead + n_t + zeros
  float* s_spec = s_buf;
  float* s_comp = s_buf + pad;
  int i0 = 0, i1 = 0, wave_items = 0;
  if (s_plan.ok) {
    wave_items = wave_size(a.slice_rows, n_slices, a.multi_rows, a.n_seg);
    wave_range(a.ctrl, a.wave, wave_items, i0, i1);
  }
  const int n_multi = a.ctrl->n_multi;
  if (a.wave > 0 && i0 >= i1) return;
  // The block's spaxels kMergeThreads at a time, one looked up per thread: a lookup is a chain
  // of three loads, about 1 us a spaxel when the block waited for each (this kernel 180 ->
  // 144 us at 22 500 spaxels, 1124 -> 915 at 90 000 and 10^7 particles).
  __shared__ int s_cnt[kMergeThreads], s_it[kMergeThreads];
  for (int b = 0, s = blockIdx.x; s < a.n_seg; ++b, s += gridDim.x) {
    if (b % kMergeThreads == 0) {
      const long long mine = s + (long long)tid * gridDim.x;
      int n = -1, it = 0;  // -1: nothing to do
      if (mine < a.n_seg) {
        n = a.seg_off[mine + 1] - a.seg_off[mine];
        if (n == 0) {
          if (a.wave != 0) n = -1;
        } else if (a.flags[mine]) {
          n = -1;
        } else {
          it = first_item((int)mine, n, a.big, a.n_seg, a.multi, a.large, a.small);
          if (it < i0 || it >= i1) n = -1;
        }
      }
      __syncthreads();  // the last batch is done with the lists
      s_cnt[tid] = n;
      s_it[tid] = it;
      __syncthreads();
    }
    const int cnt = s_cnt[b % kMergeThreads];
    if (cnt < 0) continue;
    float* out = a.cube + (long long)s * a.stride;
    if (cnt == 0) {
      for (int t = tid; t < n_t; t += kMergeThreads) out[t] = 0.f;
      continue;
    }
    const int it0 = s_it[b % kMergeThreads];
    const int chunks = (cnt + kItem - 1) / kItem;
    for (int i = tid; i < pad; i += kMergeThreads) s_spec[i] = 0.f;
    if (chunks > 1)
      for (int i = tid; i < n_t; i += kMergeThreads) s_comp[i] = 0.f;
    __syncthreads();
    for (int c = 0; c < chunks; ++c) {
      const long long row0 =
          (long long)item_row(it0 + c, n_multi, a.wave, wave_items, a.multi_rows) * n_slices;
#pragma unroll
      for (int parity = 0; parity < 2; ++parity) {
        for (int q = 2 * warp + parity; q < n_slices; q += 2 * (kMergeThreads / 32)) {
          const int2 pos = a.row_pos[row0 + q];
          const float* src = a.rows + (row0 + q) * kMaxBins;
          float v[kMaxBins / 32];
#pragma unroll
          for (int u = 0; u < kMaxBins / 32; ++u)
            v[u] = 32 * u + lane < pos.y ? src[32 * u + lane] : 0.f;
#pragma unroll
          for (int u = 0; u < kMaxBins / 32; ++u) {
            const int t = pos.x - kExt + 32 * u + lane;
            if (32 * u + lane < pos.y && t >= 0 && t < n_t) {
              float* d = s_spec + lead + t;
              if (chunks == 1) {
                *d += v[u];
              } else {
                const float y = v[u] - s_comp[t];
                const float z = *d + y;
                s_comp[t] = (z - *d) - y;
                *d = z;
              }
            }
          }
        }
        __syncthreads();
      }
    }
    if (K > 0) {
      float o[R];
      const int t0 = tid * R;
      if (K == 25) {  // rubix's LSF: 2 * 12 + 1 taps (telescope/lsf/lsf.py:12-26)
        float win[R + 24];
#pragma unroll
        for (int i = 0; i < R + 24; ++i) win[i] = s_spec[t0 + i];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          o[r] = 0.f;
#pragma unroll
          for (int j = 0; j < 25; ++j) o[r] = fmaf(a.lsf[j], win[r + 24 - j], o[r]);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) o[r] = 0.f;
        for (int j = 0; j < K; ++j) {
          const float w = a.lsf[j];
#pragma unroll
          for (int r = 0; r < R; ++r) o[r] = fmaf(w, s_spec[t0 + r + K - 1 - j], o[r]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; ++r) s_spec[t0 + r] = o[r];
      __syncthreads();
    }
    for (int t = tid; t < n_t; t += kMergeThreads) out[t] = s_spec[t];
    __syncthreads();
  }
}

// Shared memory of the kernel without dust; the one with it has four warps fewer.
size_t slice_smem(int n_templ) {
  constexpr int kW = kNodeWarps<false>;
  return sizeof(float) * ((size_t)n_templ * 32 + kWin + kW * kMaxBins) + sizeof(StagedRecs) * kW +
         sizeof(float) * (kWin + kW * kStage);
}

size_t row_bytes(int n_wave) {
  return (size_t)max_slices_of(n_wave) * (kMaxBins * sizeof(float) + sizeof(int2));
}

// Rows of the items of spaxels with more than kItem particles: at most n / kItem full ones
// and one partial one for each such spaxel.
long long multi_row_count(long long n) { return 2 * n / kItem + 1; }

struct NodeLayout {
  NodeCtrl* ctrl;
  int* flags;
  int *multi, *large, *small;
  int2* items;
  int4* desc;
  double* prefix;
  // not used before the last merge by the fallback, nor after it by the slices
  float* h;
  float* H;
  float* rough_of;
  float4* rec_w;
  float2* rec_a;
  float* rec_av;
  int2* rough;
  float* rows;
  int2* row_pos;
  size_t shared_off, fixed;  // start of the shared region; bytes without rows
};

NodeLayout carve_nodes(void* ws, long long n, int n_seg, int nZ, int nA, int nW) {
  Carve c(ws);
  NodeLayout L;
  c.take<CubeCtrl>(1);
  L.ctrl = c.take<NodeCtrl>(1);
  L.flags = c.take<int>((size_t)n_seg);
  L.multi = c.take<int>((size_t)n_seg + 1);
  L.large = c.take<int>((size_t)n_seg + 1);
  L.small = c.take<int>((size_t)n_seg + 1);
  L.items = c.take<int2>((size_t)(multi_row_count(n) + n_seg));
  L.desc = c.take<int4>((size_t)(multi_row_count(n) + n_seg));
  L.prefix = c.take<double>((size_t)nZ * nA * nW);
  L.shared_off = c.off;
  L.h = c.take<float>((size_t)kAlphaRows * kpad_of(nW));
  L.H = c.take<float>((size_t)kAlphaRows * nZ * nA);
  L.rough_of = c.take<float>((size_t)nZ * nA);
  L.rec_w = c.take<float4>((size_t)n);
  L.rec_a = c.take<float2>((size_t)n);
  L.rec_av = c.take<float>((size_t)n);
  L.rough = c.take<int2>((size_t)n);
  L.fixed = c.off;
  L.rows = nullptr;
  L.row_pos = nullptr;
  return L;
}

constexpr size_t kRowBudget = (size_t)2 << 30;  // rows of single-item spaxels at a time

long long min_wave_items(int n_seg) {
  return std::max<long long>((n_seg + kMaxWaves - 1) / kMaxWaves, std::min(n_seg, 256));
}

}  // namespace

bool cube_nodes_supported(int nZ, int nA, int nW, int n_t) {
  return n_t >= 2 && nW >= 2 && slice_smem(nZ * nA) <= 227 * 1024;
}

// Rows for the single-item spaxels of a wave: all of them, or what kRowBudget holds.
namespace {
long long full_wave(int n_seg, int nW) {
  return std::max(min_wave_items(n_seg),
                  std::min<long long>(n_seg, (long long)(kRowBudget / row_bytes(nW))));
}
}  // namespace

size_t cube_nodes_bytes(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk) {
  const NodeLayout L = carve_nodes(nullptr, n, n_seg, nZ, nA, nW);
  return std::max(L.fixed + (size_t)(multi_row_count(n) + full_wave(n_seg, nW)) * row_bytes(nW),
                  L.shared_off + fallback_bytes(n, n_seg, nZ, nA, nW, n_t, chunk, false));
}

bool cube_nodes_fit(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk,
                    size_t bytes) {
  const NodeLayout L = carve_nodes(nullptr, n, n_seg, nZ, nA, nW);
  const long long wave = std::max(min_wave_items(n_seg), (full_wave(n_seg, nW) + 1) / 2);
  return bytes >= L.fixed + (size_t)(multi_row_count(n) + wave) * row_bytes(nW) &&
         bytes >= L.shared_off + fallback_bytes(n, n_seg, nZ, nA, nW, n_t, chunk, false);
}

int cube_nodes_launches(long long n, int n_seg, int nZ, int nA, int nW, size_t bytes) {
  const NodeLayout L = carve_nodes(nullptr, n, n_seg, nZ, nA, nW);
  const long long fit = (long long)((bytes - L.fixed) / row_bytes(nW)) - multi_row_count(n);
  const long long wave = std::min<long long>(n_seg, fit);
  return (items_one_block(n_seg, n) ? 7 : 9) + 2 * (int)((n_seg + wave - 1) / wave);
}

int cube_nodes_forward(const CubeInputs& in, const float* dust_e, const float* lsf_taps, int n_lsf, int lsf_crop,
                       const CubeTuning& tune, float* cube, long long stride, void* ws,
                       size_t ws_bytes, NodeFallback* fb, cudaStream_t st) {
  NodeLayout L = carve_nodes(ws, in.n, in.n_seg, in.n_met, in.n_age, in.n_wave);
  const int big_item = tune.big_item;
  const NodeFlags flags{L.flags, L.ctrl, in.seg_off, tune.chunk, big_item};
  const int n_templ = in.n_met * in.n_age, nW = in.n_wave;
  const size_t rb = row_bytes(nW);
  const long long multi_rows = multi_row_count(in.n);
  const long long fit = (long long)((ws_bytes - L.fixed) / rb) - multi_rows;
  const int wave_items = (int)std::min<long long>(in.n_seg, fit);
  const int waves = (in.n_seg + wave_items - 1) / wave_items;
  const size_t total_rows = (size_t)(multi_rows + wave_items) * max_slices_of(nW);
  char* base = static_cast<char*>(ws) + L.fixed;
  L.rows = reinterpret_cast<float*>(base);
  L.row_pos = reinterpret_cast<int2*>(base + total_rows * kMaxBins * sizeof(float));

  // control block, counters and flags are contiguous
  RUBIX_CUDA_TRY(cudaMemsetAsync(ws, 0, (size_t)((char*)(L.flags + in.n_seg) - (char*)ws), st));
  {
    const int rc = node_setup(in, dust_e, L.ctrl, st);
    if (rc != RUBIX_OK) return rc;
  }
  const bool dust = dust_e != nullptr;
  if (items_one_block(in.n_seg, in.n)) {
    node_items_kernel<<<1, 1024, 0, st>>>(in, flags, dust, big_item, L.multi, L.large, L.small,
                                          L.items);
    RUBIX_LAUNCH_CHECK("node_items_kernel");
  } else {
    const long long work = std::max<long long>(in.n_seg, in.n / 8);  // if screened, a warp a spaxel
    const int g = (int)std::min<long long>((work + 255) / 256, (long long)sm_count() * 8);
    node_count_kernel<<<g, 256, 0, st>>>(in, flags, dust, big_item, L.multi, L.large, L.small);
    RUBIX_LAUNCH_CHECK("node_count_kernel");
    scan_exclusive_3<<<3, 1024, 0, st>>>(L.multi, L.large, L.small, in.n_seg);
    RUBIX_LAUNCH_CHECK("scan_exclusive_3");
    node_fill_items_kernel<<<g, 256, 0, st>>>(in.seg_off, L.flags, in.n_seg, big_item, L.multi,
                                              L.large, L.small, L.items, L.ctrl);
    RUBIX_LAUNCH_CHECK("node_fill_items_kernel");
  }
  {
    const int rc = node_build_tables(in, dust_e, L.prefix, L.h, L.H, L.rough_of, L.ctrl,
                                     static_cast<CubeCtrl*>(ws), st);
    if (rc != RUBIX_OK) return rc;
  }
  const long long items_max = multi_rows + std::min<long long>(in.n_seg, in.n);
  {
    GatherArgs g{in, L.prefix, L.H, L.ctrl, L.items, L.rec_w, L.rec_a,
                 dust_e ? L.rec_av : nullptr, flags, L.desc, L.rough};
    const int blocks = (int)std::min<long long>(items_max, (long long)sm_count() * 8);
    node_gather_kernel<<<blocks, kSub, 0, st>>>(g);
    RUBIX_LAUNCH_CHECK("node_gather_kernel");
    const size_t smem = rough_smem(in.n_wave_t);
    if (smem > 48 * 1024)
      RUBIX_CUDA_TRY(cudaFuncSetAttribute(
          node_rough_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    node_rough_kernel<<<rough_blocks(in.n), kRoughThreads, smem, st>>>(g);
    RUBIX_LAUNCH_CHECK("node_rough_kernel");
  }
  const size_t smem = slice_smem(n_templ);
  const auto slice_kernel = dust_e ? node_slice_kernel<true> : node_slice_kernel<false>;
  RUBIX_CUDA_TRY(cudaFuncSetAttribute(slice_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
  MergeArgs m;
  m.seg_off = in.seg_off;
  m.multi = L.multi;
  m.large = L.large;
  m.small = L.small;
  m.n_seg = in.n_seg;
  m.big = big_item;
  m.n_t = in.n_wave_t;
  m.n_wave = nW;
  m.wt = in.wave_t;
  m.flags = L.flags;
  m.rows = L.rows;
  m.row_pos = L.row_pos;
  m.ctrl = L.ctrl;
  m.multi_rows = (int)multi_rows;
  m.dust = dust_e != nullptr;
  m.slice_rows = (long long)total_rows;
  m.cube = cube;
  m.stride = stride;
  m.lsf_k = n_lsf;
  m.lsf_crop = lsf_crop;
  for (int i = 0; i <= kMaxLsfTaps; ++i) m.lsf[i] = i < n_lsf ? lsf_taps[i] : 0.f;
  for (int w = 0; w < waves; ++w) {
    const SliceArgs a{in.ssp_flux, in.ssp_wave_z, in.wave_t, n_templ, in.n_age, nW, in.n_wave_t,
                      L.desc, L.rec_w, L.rec_a, L.rec_av, dust_e, L.rows, L.row_pos, L.ctrl, w, (int)multi_rows, in.n_seg, (long long)total_rows};
    slice_kernel<<<sm_count(), 32 * (dust_e ? kNodeWarps<true> : kNodeWarps<false>), smem, st>>>(a);
    RUBIX_LAUNCH_CHECK("node_slice_kernel");
    m.wave = w;
    const int blocks = (int)std::min<long long>(in.n_seg, (long long)sm_count() * 8);
    auto launch = [&](auto r) -> int {
      constexpr int R = decltype(r)::value;
      // at most 33 KB: no opt-in
      const size_t ms = sizeof(float) * ((size_t)R * kMergeThreads + std::max(n_lsf, 0) + in.n_wave_t);
      node_merge_kernel<R><<<blocks, kMergeThreads, ms, st>>>(m);
      RUBIX_LAUNCH_CHECK("node_merge_kernel");
      return RUBIX_OK;
    };
    const int need = (in.n_wave_t + kMergeThreads - 1) / kMergeThreads;
    int rc;
    if (need <= 4) rc = launch(std::integral_constant<int, 4>{});
    else if (need <= 8) rc = launch(std::integral_constant<int, 8>{});
    else if (need <= 15) rc = launch(std::integral_constant<int, 15>{});
    else rc = launch(std::integral_constant<int, 16>{});
    if (rc != RUBIX_OK) return rc;
  }
  // The flagged spaxels, if any, in the region that the slices no longer need.
  Carve c(static_cast<char*>(ws) + L.shared_off);
  *fb = carve_fallback(c, in, tune.chunk, false);
  node_fallback_kernel<<<sm_count() * 8, 256, 0, st>>>(
      in, *fb, L.prefix, flags, static_cast<CubeCtrl*>(ws), false);
  RUBIX_LAUNCH_CHECK("node_fallback_kernel");
  return RUBIX_OK;
}

}  // namespace rubix
