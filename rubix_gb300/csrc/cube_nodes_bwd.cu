// Adjoint of the node-by-node forward (see cube_nodes.cu): the gradients of
// L = <adj, cube> with respect to every particle's mass, metallicity, age and velocity.
//
// The forward adds beta I_t to the spaxel, so with a_t the spaxel's adjoint (formulas and
// conventions of adjoint.cu)
//   gamma = sum_t a_t I_t, H_Z, H_A = the same of the interpolants' Z and age derivatives,
//   D_Z, D_A = those against dx_t, H_v = sum_t a_t x_t slope_t, D_v = sum_t dx_t x_t slope_t
// and T' comes from the H table.  (D_A from the table would be a difference of neighbouring
// templates' entries, 6e-6 off.)  All seven sums run over SSP nodes: gamma = sum_k G_k u_k,
// H_Z = sum_k (dG/dZ)_k u_k, ..., where u_k, the adjoint gathered to node k, is common to
// them.  Over a group of particles of similar alpha the samples of an interval are the same
// but for the two next to its node, so the sums of a_t, a_t (x_t - x_j), a_t x_t, dx_t, ...
// over them are formed once per group and lane, and a particle costs the node arithmetic
// (about 75 instructions per 32 nodes) instead of eight sums over every telescope bin.
//
// Measured (one GB300): 2 10^5 particles, 50 x 50 x 3721, 221 x 6 x 1221 templates: this
// adjoint 0.82 ms with its tables (the slice kernel 0.59) against 1.43 ms of the general one,
// a whole fit step 2.82 -> 2.15 ms; eight ragged galaxies (7 10^5 particles) 8.53 -> 6.10 ms.
// The slice kernel is bound by issue (0.68 per cycle) and shared-memory wavefronts (60 %).
// Relative 2-norm errors against float64 as the general path's (3.5e-7).
//
// Work items are runs of up to 256 particles of one spaxel, slices and blocks as in the
// forward; each (item, slice) writes seven sums per particle, and a last pass adds the slices
// and writes the gradients.  Fixed order everywhere: deterministic.  Flagged spaxels (also
// those whose adjoint is not finite or may overflow) are left to cube_adjoint_kernel.
#include "cube_nodes.cuh"
#include "node_tables.cuh"

#include <type_traits>

namespace rubix {
namespace {

constexpr int kAdjItem = kSub;  // particles of a work item: one sorted run
constexpr int kNodeAdjWarps = 16;
constexpr int kNodeAdjThreads = 32 * kNodeAdjWarps;
constexpr int kNodeSums = 7;

// What the last pass needs of a particle, in sorted order.
struct __align__(16) AdjFinal {
  float4 a;  // T, T', dT/dZ, dT/dage
  float4 b;  // 1 / dZ, 1 / dage of the cell, mass, index of the particle (bits)
};

__device__ __forceinline__ void adj_count(const CubeInputs& in, const NodeFlags& flags,
                                          int* chunks) {
  screened_counts(in, flags, false, kAdjItem, [&](int s, int cnt) {
    chunks[s] = (cnt + kAdjItem - 1) / kAdjItem;
  });
}

// Items in the order of their particles, so that a wave of particles is a range of items.
__device__ __forceinline__ void adj_fill(int n_seg, const int* chunks, int2* items,
                                         NodeCtrl* ctrl) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n_seg; s += gridDim.x * blockDim.x) {
    const int n = chunks[s + 1] - chunks[s];
    for (int c = 0; c < n; ++c) items[chunks[s] + c] = make_int2(s, c);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->n_items = chunks[n_seg];
}

__global__ void __launch_bounds__(256) node_adj_count_kernel(CubeInputs in, NodeFlags flags,
                                                             int* chunks) {
  adj_count(in, flags, chunks);
}
__global__ void node_adj_fill_kernel(int n_seg, const int* chunks, int2* items, NodeCtrl* ctrl) {
  adj_fill(n_seg, chunks, items, ctrl);
}

// All three steps by one block.
__global__ void __launch_bounds__(1024) node_adj_items_kernel(CubeInputs in, NodeFlags flags,
                                                              int* chunks, int2* items) {
  adj_count(in, flags, chunks);
  __syncthreads();
  scan_exclusive_block(chunks, in.n_seg, 1);
  __syncthreads();
  adj_fill(in.n_seg, chunks, items, flags.ctrl);
}

struct AdjGatherArgs {
  CubeInputs in;
  const double* prefix;
  const float* H;
  NodeCtrl* ctrl;
  const int2* items;
  float2* rec_w;  // place in the cell: tz, ta
  float2* rec_a;
  AdjFinal* fin;
  NodeFlags flags;
  int4* desc;  // first record, records, smallest and largest alpha
  int* rough;  // records of rough particles
};

// One block per work item, as node_gather_kernel, without beta.  T' of a rough particle holds
// its spaxel until it is summed.
__global__ void __launch_bounds__(kSub) node_adj_gather_kernel(AdjGatherArgs a) {
  __shared__ __align__(16) unsigned s_key[kSub];
  __shared__ unsigned s_lo, s_hi;
  __shared__ NodePlan s_plan;
  __shared__ int s_flag;
  const CubeInputs& in = a.in;
  const int tid = threadIdx.x;
  const float x1 = in.wave_t[in.n_wave_t - 1];
  if (tid == 0) s_plan = node_plan(a.ctrl, in.n_wave, x1, false);
  __syncthreads();
  const NodePlan plan = s_plan;
  const int n_items = a.ctrl->n_items;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int2 it = a.items[item];
    const int jb = in.seg_off[it.x] + it.y * kAdjItem;
    const int m = min(kAdjItem, in.seg_off[it.x + 1] - jb);
    if (tid == 0) {
      s_flag = !plan.ok;
      s_lo = 0xffffffffu;
      s_hi = 0u;
    }
    __syncthreads();
    NodeParticle q;
    q.alpha = 1.f;
    float mass = 0.f;
    long long i = 0;
    const bool on = tid < m && plan.ok;
    if (on) {
      i = in.perm[jb + tid];
      q = node_particle(in, a.prefix, a.H, i);
      mass = in.mass[i];
      if (q.bad || !(fabsf(mass) < 1e30f)) s_flag = 1;
      atomicMin(&s_lo, __float_as_uint(q.alpha));
      atomicMax(&s_hi, __float_as_uint(q.alpha));
    }
    s_key[tid] = on ? __float_as_uint(q.alpha) : 0xffffffffu;
    __syncthreads();
    if (on) {
      const int j = jb + run_rank(s_key, m, tid);
      AdjFinal f;
      const float izw = q.dzg == 0.f ? 0.f : 1.f / q.dzg, iaw = q.dag == 0.f ? 0.f : 1.f / q.dag;
      const float tz = q.tz, ta = q.ta;
      const double tZ = (double)q.alpha * (double)izw *
                        ((1.0 - ta) * (q.dT[1] - q.dT[0]) + (double)ta * (q.dT[3] - q.dT[2]));
      const double tA = (double)q.alpha * (double)iaw *
                        ((1.0 - tz) * (q.dT[2] - q.dT[0]) + (double)tz * (q.dT[3] - q.dT[1]));
      f.a = make_float4(q.T, q.Tp, (float)tZ, (float)tA);
      f.b = make_float4(izw, iaw, mass, __int_as_float((int)i));
      a.fin[j] = f;
      a.rec_w[j] = make_float2(tz, ta);
      a.rec_a[j] = make_float2(q.alpha, __int_as_float(q.row * 128));
      if (q.rough) {
        a.fin[j].a.y = __int_as_float(it.x);
        a.rough[rough_place(a.ctrl)] = j;
      }
    }
    __syncthreads();
    if (tid == 0) {
      const float lo = __uint_as_float(s_lo), hi = __uint_as_float(s_hi);
      a.desc[item] = make_int4(jb, m, (int)s_lo, (int)s_hi);
      if (s_flag || too_wide(plan, lo, hi, x1)) a.flags.leave(it.x);
    }
    __syncthreads();
  }
}

// T' of rough particles, a warp each (as node_rough_kernel).
__global__ void __launch_bounds__(kRoughThreads, kRoughBlocks) node_adj_rough_kernel(AdjGatherArgs a) {
  const int n = a.ctrl->n_rough;
  if (n == 0) return;
  extern __shared__ __align__(16) float4 s_tab4[];
  __shared__ NodePlan s_plan;
  const CubeInputs& in = a.in;
  if (threadIdx.x == 0)
    s_plan = node_plan(a.ctrl, in.n_wave, in.wave_t[in.n_wave_t - 1], false);
  const bool even = sample_table(in.wave_t, in.n_wave_t, s_tab4);
  const NodePlan plan = s_plan;
  for (int e = (blockIdx.x * kRoughThreads + threadIdx.x) >> 5; e < n;
       e += gridDim.x * (kRoughThreads / 32)) {
    const int j = a.rough[e];
    const float4 f = a.fin[j].a;
    const float2 z = a.rec_w[j];
    float w[4];
    corner_weights(z.x, z.y, w);
    const float Tp = rough_tprime(in, plan, s_tab4, even, a.rec_a[j], w);
    if ((threadIdx.x & 31) == 0) {
      a.fin[j].a.y = Tp;
      if (bad_scale(f.x, Tp)) a.flags.leave(__float_as_int(f.y));
    }
  }
}

// Items [i0, i1) and first record of a wave of `per` particles: those that start in it.
__device__ __forceinline__ int items_from(const int4* __restrict__ desc, int n_items,
                                          long long start) {
  int lo = 0, hi = n_items;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((long long)desc[mid].x < start) lo = mid + 1; else hi = mid;
  }
  return lo;
}

struct AdjSliceArgs {
  const float* flux;
  const float* wz;
  const float* wt;
  int n_templ, n_age, n_wave, n_t;
  const int4* desc;
  const int2* items;
  const float2* rec_w;
  const float2* rec_a;
  const float* adj;
  long long adj_stride;
  NodeFlags flags;
  float* part;  // [slice][kNodeSums][per + kAdjItem]
  NodeCtrl* ctrl;
  int wave;
  long long per;
};

// A warp's item on one slice, two nodes per lane and two particles at a time (16 lanes each).
// Lane (g, i) owns node 2 i + g when samples are summed; every lane then holds both nodes'.
struct AdjItem {
  static constexpr int LPG = 16;
  const SliceShared& sh;
  const float* dx;  // window: dlambda of every sample, 0 outside the telescope grid
  const int lane, i, g, own, nxt_lane;
  const float lam_own;
  float2 nlam;
  float nlam_r;
  const char* tab;
  float2 on;  // 1 for the slice's own nodes
  float2 xj, d1, h0, h1, e0, e1, H0, H1, V, E0, E1, X;

  __device__ __forceinline__ AdjItem(const SliceShared& s, const float* dx_, int lane_, int n_own,
                                     const float* __restrict__ lam)
      : sh(s), dx(dx_), lane(lane_), i(lane_ & 15), g(lane_ >> 4), own(2 * i + g),
        nxt_lane(g == 0 ? i + 16 : ((i + 1) & 15)), lam_own(lam[own]),
        nlam(make_float2(-lam[2 * i], -lam[2 * i + 1])), nlam_r(-lam[2 * i + 2]),
        tab(reinterpret_cast<const char*>(s.tab) + 8 * i) {
    on.x = (2 * i >= 1 && 2 * i <= n_own) ? 1.f : 0.f;
    on.y = (2 * i + 1 >= 1 && 2 * i + 1 <= n_own) ? 1.f : 0.f;
  }

  __device__ __forceinline__ float2 spread(float v) const {
    return make_float2(__shfl_sync(0xffffffffu, v, i), __shfl_sync(0xffffffffu, v, 16 + i));
  }

  // The group's sums over the samples of each interval (window sample j is at h[j - jb]).
  __device__ __forceinline__ void open(float alpha, int jb, int nb) {
    const int j = sample_at(sh, __fmul_rn(lam_own, alpha));
    const int jn = __shfl_sync(0xffffffffu, j, nxt_lane);
    const float* h = sh.f - jb;
    const int top = jb + nb;
    const float xo = sh.xw[j];
    const int j1 = min(j + 1, kWin - 1);
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f, s4 = 0.f, s5 = 0.f;
    for (int q = j; q < jn && q < top; ++q) {
      const float x = sh.xw[q], v = h[q], e = dx[q];
      s0 += v;
      s1 = fmaf(v, x - xo, s1);
      s2 = fmaf(v, x, s2);
      s3 = fmaf(e, x, s3);
      s4 += e;
      s5 = fmaf(e, x - xo, s5);
    }
    xj = spread(xo);
    d1 = spread(sh.xw[j1] - xo);
    h0 = spread(j < top ? h[j] : 0.f);
    h1 = spread(j1 < top ? h[j1] : 0.f);
    e0 = spread(dx[j]);
    e1 = spread(dx[j1]);
    H0 = spread(s0);
    H1 = spread(s1);
    V = spread(s2);
    X = spread(s3);
    E0 = spread(s4);
    E1 = spread(s5);
  }

  struct Loaded {
    float2 c[4];
    float tz, ta, alpha;
  };
  __device__ __forceinline__ void load(int r, int zoff, Loaded& v) const {
    const StagedRecs& st = *sh.st;
    const char* t0 = tab + st.row[r];
    v.c[0] = *reinterpret_cast<const float2*>(t0);
    v.c[1] = *reinterpret_cast<const float2*>(t0 + zoff);
    v.c[2] = *reinterpret_cast<const float2*>(t0 + 128);
    v.c[3] = *reinterpret_cast<const float2*>(t0 + zoff + 128);
    v.tz = st.w[0][r];
    v.ta = st.w[1][r];
    v.alpha = st.alpha[r];
  }

  // Seven sums of this lane's particle over its 16 lanes, sum i / 2 in its lane i (even).
  template <int W>
  __device__ __forceinline__ float step(const Loaded& v) const {
    // G as the forward mixes it (a slope is a difference of two G: with another rounding it
    // would be 1e-5 off the forward's), its derivatives in tz and ta from differences
    const float2 neg = make_float2(-1.f, -1.f);
    const float2 tz = make_float2(v.tz, v.tz), ta = make_float2(v.ta, v.ta);
    const float2 uz = make_float2(1.f - v.tz, 1.f - v.tz), ua = make_float2(1.f - v.ta, 1.f - v.ta);
    float2 G = __fmul2_rn(__fmul2_rn(uz, ua), v.c[0]);
    G = __ffma2_rn(__fmul2_rn(tz, ua), v.c[1], G);
    G = __ffma2_rn(__fmul2_rn(uz, ta), v.c[2], G);
    G = __ffma2_rn(__fmul2_rn(tz, ta), v.c[3], G);
    const float2 GZ = __ffma2_rn(ta, __ffma2_rn(neg, v.c[2], v.c[3]),
                                 __fmul2_rn(ua, __ffma2_rn(neg, v.c[0], v.c[1])));
    const float2 GA = __ffma2_rn(tz, __ffma2_rn(neg, v.c[1], v.c[3]),
                                 __fmul2_rn(uz, __ffma2_rn(neg, v.c[0], v.c[2])));
    const float2 nlp = __fmul2_rn(nlam, make_float2(v.alpha, v.alpha));
    const float nlp_r = __fmul_rn(nlam_r, v.alpha);
    const float G_r = __shfl_down_sync(0xffffffffu, G.x, 1, LPG);
    const float2 r = make_float2(fast_rcp(nlp.x - nlp.y), fast_rcp(nlp.y - nlp_r));
    const float2 s = __fmul2_rn(make_float2(G.y - G.x, G_r - G.y), r);
    const float2 t = __fadd2_rn(xj, nlp);
    // samples j (and j + 1) lie on the left interval's line while t (t + d1) < 0
    const float2 m0 = make_float2(fminf(t.x, 0.f), fminf(t.y, 0.f));
    float2 Q = __fmul2_rn(h0, m0), R = __fmul2_rn(e0, m0);
    const float2 x0 = xj;
    const float2 f0 = make_float2(t.x < 0.f ? x0.x : 0.f, t.y < 0.f ? x0.y : 0.f);
    float2 U = __fmul2_rn(h0, f0), Y = __fmul2_rn(e0, f0);
    if constexpr (W > 1) {
      const float2 t1 = __fadd2_rn(t, d1), x1 = __fadd2_rn(xj, d1);
      const float2 m1 = make_float2(fminf(t1.x, 0.f), fminf(t1.y, 0.f));
      Q = __ffma2_rn(h1, m1, Q);
      R = __ffma2_rn(e1, m1, R);
      const float2 f1 = make_float2(t1.x < 0.f ? x1.x : 0.f, t1.y < 0.f ? x1.y : 0.f);
      U = __ffma2_rn(h1, f1, U);
      Y = __ffma2_rn(e1, f1, Y);
    }
    const float Q_r = __shfl_down_sync(0xffffffffu, Q.x, 1, LPG);
    const float R_r = __shfl_down_sync(0xffffffffu, R.x, 1, LPG);
    const float U_r = __shfl_down_sync(0xffffffffu, U.x, 1, LPG);
    const float Y_r = __shfl_down_sync(0xffffffffu, Y.x, 1, LPG);
    // z: what an interval's slope takes from its samples, over its length; u: what a node's
    // value takes (from the adjoint, from dx)
    const float2 za = __fmul2_rn(
        r, __fadd2_rn(__ffma2_rn(H0, t, H1), make_float2(Q.y - Q.x, Q_r - Q.y)));
    const float2 ze = __fmul2_rn(
        r, __fadd2_rn(__ffma2_rn(E0, t, E1), make_float2(R.y - R.x, R_r - R.y)));
    const float za_l = __shfl_up_sync(0xffffffffu, za.y, 1, LPG);
    const float ze_l = __shfl_up_sync(0xffffffffu, ze.y, 1, LPG);
    const float2 u = __fmul2_rn(on, __fadd2_rn(H0, make_float2(za_l - za.x, za.x - za.y)));
    const float2 ue = __fmul2_rn(on, __fadd2_rn(E0, make_float2(ze_l - ze.x, ze.x - ze.y)));
    const float2 so = __fmul2_rn(on, s);
    const float2 av = __fadd2_rn(V, make_float2(U.y - U.x, U_r - U.y));
    const float2 ax = __fadd2_rn(X, make_float2(Y.y - Y.x, Y_r - Y.y));
    auto pair = [](float2 x, float2 y) { return fmaf(x.y, y.y, x.x * y.x); };
    const float q[8] = {pair(G, u),   pair(GZ, u),  pair(GA, u), pair(GZ, ue),
                        pair(GA, ue), pair(so, av), pair(so, ax), 0.f};
    // transposed butterfly over the 16 lanes: lane bits 3, 2, 1 choose the sum, bit 0 is added
    const bool b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
    float p[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      p[k] = (b3 ? q[4 + k] : q[k]) + __shfl_xor_sync(0xffffffffu, b3 ? q[k] : q[4 + k], 8);
    const float a0 = (b2 ? p[2] : p[0]) + __shfl_xor_sync(0xffffffffu, b2 ? p[0] : p[2], 4);
    const float a1 = (b2 ? p[3] : p[1]) + __shfl_xor_sync(0xffffffffu, b2 ? p[1] : p[3], 4);
    float o = (b1 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, b1 ? a0 : a1, 2);
    o += __shfl_xor_sync(0xffffffffu, o, 1);
    return o;
  }
  // The sum that a lane holds after step, or -1.
  __device__ __forceinline__ int place() const {
    const int k = (lane & 15) >> 1;
    return (lane & 1) || k >= kNodeSums ? -1 : k;
  }
};

struct AdjShared {
  float sums[kNodeSums][32];  // of a staged batch
};

template <int W>
__device__ __forceinline__ void adj_items(const AdjSliceArgs& a, const SliceShared& sh,
                                          const float* dx, AdjShared* so, const float* s_lam,
                                          int n_own, int lane, int slice, int i0, int total,
                                          int e0, float w_seg, float h_max,
                                          int* __restrict__ next) {
  AdjItem w(sh, dx, lane, n_own, s_lam);
  const int zoff = a.n_age * 128;
  const float lam_lo = s_lam[0], lam_hi = s_lam[n_own + 1];
  const int grp = lane >> 4, place = w.place();
  const long long first = a.wave * a.per, pitch = a.per + kAdjItem;
  float* part = a.part + (long long)slice * kNodeSums * pitch;
  auto take = [&]() { return lane == 0 ? atomicAdd(next, 1) : 0; };
  int cur = __shfl_sync(0xffffffffu, take(), 0);
  while (cur < total) {
    const int nxt = take();
    const int4 d = a.desc[i0 + cur];
    const int2 it = a.items[i0 + cur];
    const int p0 = d.x, np = d.y;
    const int jb = sample_at(sh, __fmul_rn(lam_lo, __int_as_float(d.z)));
    const int nb = min(sample_at(sh, __fmul_rn(lam_hi, __int_as_float(d.w))) + 2 - jb, kMaxBins);
    const float* adj = a.adj + (long long)it.x * a.adj_stride;
    bool bad = false;
    for (int b = lane; b < nb; b += 32) {
      const int t = e0 + jb + b - kExt;
      const float h = (t >= 0 && t < a.n_t) ? adj[t] : 0.f;
      bad |= !(fabsf(h) < h_max);
      sh.f[b] = h;
    }
    if (bad) a.flags.leave(it.x);
    bool open = false;
    float a_lim = 0.f;
    for (int base = 0; base < np; base += 32) {
      const int cnt = min(32, np - base);
      float2 rw = make_float2(0.f, 0.f), ra = make_float2(1.f, 0.f);
      if (lane < cnt) {
        rw = a.rec_w[(long long)p0 + base + lane];
        ra = a.rec_a[(long long)p0 + base + lane];
      }
      __syncwarp();
      sh.st->w[0][lane] = rw.x;
      sh.st->w[1][lane] = rw.y;
      sh.st->alpha[lane] = ra.x;
      sh.st->row[lane] = __float_as_int(ra.y);
      const float al = ra.x;
      __syncwarp();
      int pos = 0;
      while (pos < cnt) {
        const float al0 = __shfl_sync(0xffffffffu, al, pos);
        if (!open || al0 >= a_lim) {
          w.open(al0, jb, nb);
          a_lim = al0 + w_seg;
          open = true;
        }
        const unsigned past =
            __ballot_sync(0xffffffffu, lane > pos && lane < cnt && al >= a_lim);
        const int end = past ? __ffs(past) - 1 : cnt;
        AdjItem::Loaded v;
        w.load(pos + grp < end ? pos + grp : 32, zoff, v);
        for (int p = pos; p < end; p += 2) {
          const AdjItem::Loaded u = v;
          if (p + 2 < end) w.load(p + 2 + grp < end ? p + 2 + grp : 32, zoff, v);
          const float o = w.template step<W>(u);
          if (place >= 0 && p + grp < end) so->sums[place][p + grp] = o;
        }
        pos = end;
      }
      __syncwarp();
      if (lane < cnt) {
        const long long at = (long long)p0 - first + base + lane;
#pragma unroll
        for (int k = 0; k < kNodeSums; ++k) part[k * pitch + at] = so->sums[k][lane];
      }
    }
    __syncwarp();
    cur = __shfl_sync(0xffffffffu, nxt, 0);
  }
}

size_t adj_slice_smem(int n_templ) {
  return sizeof(float) * ((size_t)n_templ * 32 + 2 * kWin + kNodeAdjWarps * kMaxBins) +
         (sizeof(StagedRecs) + sizeof(AdjShared)) * kNodeAdjWarps;
}

// As node_slice_kernel, with the adjoint's window in the place of the sums.
__global__ void __launch_bounds__(kNodeAdjThreads, 1) node_adj_slice_kernel(AdjSliceArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  float* s_tab = reinterpret_cast<float*>(smem);
  float* s_xw = s_tab + (size_t)a.n_templ * 32;
  float* s_dx = s_xw + kWin;
  float* s_f = s_dx + kWin;
  StagedRecs* s_st = reinterpret_cast<StagedRecs*>(s_f + kNodeAdjWarps * kMaxBins);
  AdjShared* s_so = reinterpret_cast<AdjShared*>(s_st + kNodeAdjWarps);
  __shared__ float s_lam[36];
  __shared__ NodePlan s_plan;
  __shared__ int s_slice, s_e0, s_i0, s_i1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float x_last = a.wt[a.n_t - 1];
  if (tid == 0) {
    s_plan = node_plan(a.ctrl, a.n_wave, x_last, false);
    const int n = a.ctrl->n_items;
    s_i0 = items_from(a.desc, n, a.wave * a.per);
    s_i1 = items_from(a.desc, n, (a.wave + 1) * a.per);
  }
  __syncthreads();
  const NodePlan plan = s_plan;
  const int i0 = s_i0, total = s_i1 - s_i0;
  if (!plan.ok || total <= 0) return;
  const float fm = __uint_as_float(a.ctrl->fmax);
  const float h_max = fm > 0.f ? fminf(1e28f / fm, 1e28f) : 1e28f;
  SliceShared sh;
  sh.tab = s_tab;
  sh.xw = s_xw;
  sh.ew = nullptr;
  sh.st_av = nullptr;
  sh.st = s_st + warp;
  sh.f = s_f + warp * kMaxBins;
  if (lane == 0) {
    sh.st->w[0][32] = sh.st->w[1][32] = 0.f;
    sh.st->alpha[32] = 1.f;
    sh.st->row[32] = 0;
  }
  int* next = a.ctrl->next[a.wave];
  int slice = (int)((long long)blockIdx.x * plan.n_slices / gridDim.x);
  const float w_seg =
      (float)plan.w * 0.98f * plan.dt_min * (1.f - kAlphaMax) / x_last - 2.4e-7f;
  for (;;) {
    const int k0 = plan.k_first - 1 + slice * plan.n_own;  // node of lane 0
    for (int r = warp; r < a.n_templ; r += kNodeAdjWarps) {
      const int k = k0 + lane;
      s_tab[r * 32 + lane] = (lane <= plan.n_own + 1 && k >= 0 && k < a.n_wave)
                                 ? a.flux[(long long)r * a.n_wave + k] : 0.f;
    }
    if (tid < 36) s_lam[tid] = lam_ext(a.wz, a.n_wave, k0 + tid);
    if (warp == 0) {
      const int e = window_start(a.wt, a.n_t, lam_ext(a.wz, a.n_wave, k0), lane);
      if (lane == 0) s_e0 = e;
    }
    __syncthreads();
    const int e0 = s_e0;
    for (int q = tid; q < kWin; q += kNodeAdjThreads) {
      const int t = e0 + q - kExt;
      s_xw[q] = x_ext(a.wt, a.n_t, e0 + q);
      s_dx[q] = (t > 0 && t < a.n_t) ? a.wt[t] - a.wt[t - 1] : 0.f;
    }
    __syncthreads();
    sh.inv = (float)(kWin - 1) / (s_xw[kWin - 1] - s_xw[0]);
    if (plan.w == 1)
      adj_items<1>(a, sh, s_dx, s_so + warp, s_lam, plan.n_own, lane, slice, i0, total, e0, w_seg,
                   h_max, next + slice);
    else
      adj_items<2>(a, sh, s_dx, s_so + warp, s_lam, plan.n_own, lane, slice, i0, total, e0, w_seg,
                   h_max, next + slice);
    __syncthreads();
    if (tid == 0) s_slice = busiest_slice(next, plan.n_slices, total, 2 * kNodeAdjWarps);
    __syncthreads();
    slice = s_slice;
    if (slice < 0) return;
  }
}

struct AdjMergeArgs {
  const int2* items;
  const int4* desc;
  const AdjFinal* fin;
  const float* part;
  const int* flags;
  const NodeCtrl* ctrl;
  const float* wt;
  int n_wave, n_t, wave;
  long long per;
  float *g_mass, *g_met, *g_age, *g_vlos;
};

// One block per work item: the slices' sums of each particle, then its gradients
// (adjoint.cu's formulas).  Bound by HBM: 28 bytes per particle and slice.
__global__ void __launch_bounds__(kAdjItem) node_adj_merge_kernel(AdjMergeArgs a) {
  __shared__ NodePlan s_plan;
  __shared__ int s_i0, s_i1;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_plan = node_plan(a.ctrl, a.n_wave, a.wt[a.n_t - 1], false);
    const int n = a.ctrl->n_items;
    s_i0 = items_from(a.desc, n, a.wave * a.per);
    s_i1 = items_from(a.desc, n, (a.wave + 1) * a.per);
  }
  __syncthreads();
  if (!s_plan.ok) return;
  const int n_slices = s_plan.n_slices;
  const long long first = a.wave * a.per, pitch = a.per + kAdjItem;
  for (int item = s_i0 + blockIdx.x; item < s_i1; item += gridDim.x) {
    if (a.flags[a.items[item].x]) continue;
    const int4 d = a.desc[item];
    if (tid >= d.y) continue;
    const long long j = (long long)d.x + tid;
    const float* p = a.part + (j - first);
    float q[kNodeSums];
#pragma unroll
    for (int k = 0; k < kNodeSums; ++k) q[k] = 0.f;
#pragma unroll 4
    for (int s = 0; s < n_slices; ++s)
#pragma unroll
      for (int k = 0; k < kNodeSums; ++k) q[k] += p[((long long)s * kNodeSums + k) * pitch];
    const AdjFinal f = a.fin[j];
    const float T = f.a.x, Tp = f.a.y, TZ = f.a.z, TA = f.a.w, m = f.b.z;
    const float HZ = f.b.x * q[1], HA = f.b.y * q[2], DZ = f.b.x * q[3], DA = f.b.y * q[4];
    const float gamma = q[0], HV = q[5], DV = q[6];
    const long long i = __float_as_int(f.b.w);
    const float sc = T / Tp;
    float gm = 0.f, gz = 0.f, ga = 0.f, gv = 0.f;
    if (Tp != 0.f && isfinite(sc)) {
      const float beta = m * sc, k = m / Tp;
      const float inv_c = (float)(1.0 / kSpeedOfLight);
      gm = sc * gamma;
      gz = fmaf(beta, HZ, gamma * k * (TZ - sc * DZ));
      ga = fmaf(beta, HA, gamma * k * (TA - sc * DA));
      gv = fmaf(-beta * inv_c, HV, gamma * k * inv_c * (T + sc * DV));
    }
    if (a.g_mass) a.g_mass[i] = gm;
    if (a.g_met) a.g_met[i] = gz;
    if (a.g_age) a.g_age[i] = ga;
    if (a.g_vlos) a.g_vlos[i] = gv;
  }
}

struct AdjNodeLayout {
  NodeCtrl* ctrl;
  int* flags;
  int* chunks;
  int2* items;
  int4* desc;
  double* prefix;
  float *h, *H, *rough_of;
  float2* rec_w;  // place in the cell: tz, ta
  float2* rec_a;
  AdjFinal* fin;
  int* rough;
  float* part;
  size_t shared_off, fixed;
};

long long adj_items_max(long long n, int n_seg) { return n / kAdjItem + std::min<long long>(n, n_seg); }

AdjNodeLayout carve_adj(void* ws, long long n, int n_seg, int nZ, int nA, int nW) {
  Carve c(ws);
  AdjNodeLayout L;
  c.take<CubeCtrl>(1);
  L.ctrl = c.take<NodeCtrl>(1);
  L.flags = c.take<int>((size_t)n_seg);
  L.chunks = c.take<int>((size_t)n_seg + 1);
  L.items = c.take<int2>((size_t)adj_items_max(n, n_seg));
  L.desc = c.take<int4>((size_t)adj_items_max(n, n_seg));
  L.prefix = c.take<double>((size_t)nZ * nA * nW);
  L.shared_off = c.off;
  L.h = c.take<float>((size_t)kAlphaRows * kpad_of(nW));
  L.H = c.take<float>((size_t)kAlphaRows * nZ * nA);
  L.rough_of = c.take<float>((size_t)nZ * nA);
  L.rec_w = c.take<float2>((size_t)n);
  L.rec_a = c.take<float2>((size_t)n);
  L.fin = c.take<AdjFinal>((size_t)n);
  L.rough = c.take<int>((size_t)n);
  L.fixed = c.off;
  L.part = ws ? reinterpret_cast<float*>(static_cast<char*>(ws) + L.fixed) : nullptr;
  return L;
}

constexpr size_t kPartBudget = (size_t)2 << 30;

size_t part_bytes(long long per, int n_wave) {
  return sizeof(float) * (size_t)max_slices_of(n_wave) * kNodeSums * (size_t)(per + kAdjItem);
}

// Particles of a wave that a part region of `bytes` holds.
long long part_particles(size_t bytes, int n_wave) {
  return (long long)(bytes / (sizeof(float) * max_slices_of(n_wave) * kNodeSums)) - kAdjItem;
}

long long min_wave_particles(long long n) {
  return std::max<long long>((n + kMaxWaves - 1) / kMaxWaves, std::min<long long>(n, 4096));
}

}  // namespace

bool cube_nodes_bwd_supported(int nZ, int nA, int nW, int n_t) {
  return n_t >= 2 && nW >= 2 && adj_slice_smem(nZ * nA) <= 227 * 1024;
}

namespace {
// Particles of a wave: all of them, or what kPartBudget holds.
long long full_wave_particles(long long n, int nW) {
  return std::max(min_wave_particles(n), std::min(n, part_particles(kPartBudget, nW)));
}
}  // namespace

size_t cube_nodes_bwd_bytes(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk) {
  const AdjNodeLayout L = carve_adj(nullptr, n, n_seg, nZ, nA, nW);
  return std::max(L.fixed + part_bytes(full_wave_particles(n, nW), nW),
                  L.shared_off + fallback_bytes(n, n_seg, nZ, nA, nW, n_t, chunk, true));
}

bool cube_nodes_bwd_fit(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk,
                        size_t bytes) {
  const AdjNodeLayout L = carve_adj(nullptr, n, n_seg, nZ, nA, nW);
  const long long per = std::max(min_wave_particles(n), (full_wave_particles(n, nW) + 1) / 2);
  return bytes >= L.fixed + part_bytes(per, nW) &&
         bytes >= L.shared_off + fallback_bytes(n, n_seg, nZ, nA, nW, n_t, chunk, true);
}

int cube_nodes_bwd_launches(long long n, int n_seg, int nZ, int nA, int nW, size_t bytes) {
  const AdjNodeLayout L = carve_adj(nullptr, n, n_seg, nZ, nA, nW);
  const long long per = std::min(n, part_particles(bytes - L.fixed, nW));
  return (items_one_block(n_seg, n) ? 7 : 9) + 2 * (int)((n + per - 1) / per);
}

int cube_nodes_backward(const CubeInputs& in, const float* adj, long long adj_stride,
                        const CubeTuning& tune, float* const* grads, void* ws, size_t ws_bytes,
                        NodeFallback* fb, cudaStream_t st) {
  const AdjNodeLayout L = carve_adj(ws, in.n, in.n_seg, in.n_met, in.n_age, in.n_wave);
  const NodeFlags flags{L.flags, L.ctrl, in.seg_off, tune.chunk, tune.big_item};
  const int n_templ = in.n_met * in.n_age, nW = in.n_wave;
  RUBIX_CUDA_TRY(cudaMemsetAsync(ws, 0, (size_t)((char*)(L.flags + in.n_seg) - (char*)ws), st));
  {
    const int rc = node_setup(in, nullptr, L.ctrl, st);
    if (rc != RUBIX_OK) return rc;
  }
  if (items_one_block(in.n_seg, in.n)) {
    node_adj_items_kernel<<<1, 1024, 0, st>>>(in, flags, L.chunks, L.items);
    RUBIX_LAUNCH_CHECK("node_adj_items_kernel");
  } else {
    const long long work = std::max<long long>(in.n_seg, in.n / 8);  // if screened, a warp a spaxel
    const int g = (int)std::min<long long>((work + 255) / 256, (long long)sm_count() * 8);
    node_adj_count_kernel<<<g, 256, 0, st>>>(in, flags, L.chunks);
    RUBIX_LAUNCH_CHECK("node_adj_count_kernel");
    scan_exclusive_1block<<<1, 1024, 0, st>>>(L.chunks, in.n_seg, 1);
    RUBIX_LAUNCH_CHECK("scan_exclusive_1block");
    node_adj_fill_kernel<<<g, 256, 0, st>>>(in.n_seg, L.chunks, L.items, L.ctrl);
    RUBIX_LAUNCH_CHECK("node_adj_fill_kernel");
  }
  {
    const int rc = node_build_tables(in, nullptr, L.prefix, L.h, L.H, L.rough_of, L.ctrl,
                                     static_cast<CubeCtrl*>(ws), st);
    if (rc != RUBIX_OK) return rc;
  }
  const int blocks =
      (int)std::min<long long>(adj_items_max(in.n, in.n_seg), (long long)sm_count() * 8);
  {
    const AdjGatherArgs g{in,      L.prefix, L.H,   L.ctrl, L.items,
                          L.rec_w, L.rec_a,  L.fin, flags, L.desc, L.rough};
    node_adj_gather_kernel<<<blocks, kSub, 0, st>>>(g);
    RUBIX_LAUNCH_CHECK("node_adj_gather_kernel");
    const size_t smem = rough_smem(in.n_wave_t);
    if (smem > 48 * 1024)
      RUBIX_CUDA_TRY(cudaFuncSetAttribute(
          node_adj_rough_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    node_adj_rough_kernel<<<rough_blocks(in.n), kRoughThreads, smem, st>>>(g);
    RUBIX_LAUNCH_CHECK("node_adj_rough_kernel");
  }
  const long long per = std::min(in.n, part_particles(ws_bytes - L.fixed, nW));
  const int waves = (int)((in.n + per - 1) / per);
  const size_t smem = adj_slice_smem(n_templ);
  RUBIX_CUDA_TRY(cudaFuncSetAttribute(node_adj_slice_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (int w = 0; w < waves; ++w) {
    const AdjSliceArgs a{in.ssp_flux, in.ssp_wave_z, in.wave_t, n_templ, in.n_age, nW,
                         in.n_wave_t, L.desc,        L.items,   L.rec_w, L.rec_a,  adj,
                         adj_stride,  flags,         L.part,    L.ctrl,  w,        per};
    node_adj_slice_kernel<<<sm_count(), kNodeAdjThreads, smem, st>>>(a);
    RUBIX_LAUNCH_CHECK("node_adj_slice_kernel");
    const AdjMergeArgs m{L.items, L.desc, L.fin, L.part,   L.flags,  L.ctrl,   in.wave_t, nW,
                         in.n_wave_t, w, per, grads[0], grads[1], grads[2], grads[3]};
    node_adj_merge_kernel<<<blocks, kAdjItem, 0, st>>>(m);
    RUBIX_LAUNCH_CHECK("node_adj_merge_kernel");
  }
  Carve c(static_cast<char*>(ws) + L.shared_off);
  *fb = carve_fallback(c, in, tune.chunk, true);
  node_fallback_kernel<<<sm_count() * 8, 256, 0, st>>>(
      in, *fb, L.prefix, flags, static_cast<CubeCtrl*>(ws), true);
  RUBIX_LAUNCH_CHECK("node_fallback_kernel");
  return RUBIX_OK;
}

}  // namespace rubix
