// Kernel (a): aperture mask, spaxel assignment and a stable LSD radix sort of the
// particles by spaxel index, ending in per-spaxel segment offsets.
//
// The radix sort is written from the published LSD scheme: per pass, a per-tile
// digit histogram, one exclusive scan over (digit, tile), and a stable scatter in
// which each tile ranks its keys with warp-level match/popc and per-warp digit
// counters.  No float atomics anywhere; the result is deterministic.
#include "common.cuh"
#include "particle_frame.cuh"
#include "radix.cuh"
#include "scan.cuh"

#include <type_traits>

namespace rubix {
namespace {

constexpr int kMaxSmemEdges = 8192;

// Smallest and largest edge, by one warp (fminf and fmaxf skip NaN in any order).
__device__ __forceinline__ void edge_range(const float* __restrict__ edges, int n, float& s_lo,
                                           float& s_hi) {
  const int lane = threadIdx.x;
  float lo = edges[min(lane, n - 1)], hi = lo;
  for (int i = lane; i < n; i += 32) {
    lo = fminf(lo, edges[i]);
    hi = fmaxf(hi, edges[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) {
    s_lo = lo;
    s_hi = hi;
  }
}

__global__ void aperture_mask_kernel(const float* __restrict__ coords, long long n,
                                     long long stride, const float* __restrict__ edges,
                                     int n_edges, unsigned char* __restrict__ mask) {
  __shared__ float s_lo, s_hi;
  if (threadIdx.x < 32) edge_range(edges, n_edges, s_lo, s_hi);
  __syncthreads();
  const float lo = s_lo, hi = s_hi;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    mask[i] = inside_aperture(coords[i * stride], coords[i * stride + 1], lo, hi) ? 1 : 0;
  }
}

// spaxel_index on the block's edges.  On ascending edges the count of edges <= x does not
// depend on how it is found: a linear guess, right to one edge on an even grid, takes 3 loads
// where the search takes 9 for 301 edges (85 -> 49 us for 10^7 particles).  Edges that are not
// even to half a step (the guess and the search: 168 us, the search alone 88), and few of them (5
// edges: 86 and 45 us), are searched.
constexpr int kGuessEdges = 24;

struct EdgeBins {
  const float* e;
  const int n, nb;
  const bool guess;
  const float e0, inv;
  __device__ __forceinline__ EdgeBins(const float* e_, int n_, bool guess_)
      : e(e_), n(n_), nb(n_ - 1), guess(guess_), e0(e_[0]),
        inv((float)(n_ - 1) / (e_[n_ - 1] - e_[0])) {}
  // Whether edge i allows the guess.
  static __device__ __forceinline__ bool even(const float* __restrict__ edges, int n, int i) {
    const float v = edges[i], e0 = edges[0], inv = (float)(n - 1) / (edges[n - 1] - e0);
    return fabsf((v - e0) * inv - (float)i) <= 0.5f && (i + 1 == n || v <= edges[i + 1]);
  }
  __device__ __forceinline__ int bin(float x) const {
    if (guess) {
      // clamped before the conversion: NaN becomes 0, a far x stays an index
      int c = (int)fminf(fmaxf((x - e0) * inv, 0.f), (float)(nb - 1)) + 1;
      c = min(c, nb);
      if (c < nb && e[c] <= x) ++c;
      if (c > 1 && e[c - 1] > x) --c;
      // the clipped bin c - 1: below the first edge and above the last count as its ends
      if ((c == 1 || e[c - 1] <= x) && (c == nb || e[c] > x)) return c - 1;
    }
    return min(max(count_le(e, n, x) - 1, 0), nb - 1);
  }
  __device__ __forceinline__ int flat(float x, float y) const { return bin(x) + nb * bin(y); }
};

__global__ void spaxel_assign_kernel(const float* __restrict__ coords, long long n,
                                     long long stride, const float* __restrict__ edges,
                                     int n_edges, int* __restrict__ idx_out) {
  extern __shared__ float s_edges[];
  const bool in_smem = n_edges <= kMaxSmemEdges;
  const float* e = in_smem ? s_edges : edges;
  bool even = n_edges >= kGuessEdges;
  for (int i = threadIdx.x; i < n_edges; i += blockDim.x) {
    if (in_smem) s_edges[i] = edges[i];
    even = even && EdgeBins::even(edges, n_edges, i);
  }
  even = __syncthreads_and(even);
  const EdgeBins bins(e, n_edges, even);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    idx_out[i] = bins.flat(coords[i * stride], coords[i * stride + 1]);
}

constexpr int kMaxFrameFields = 8;

// Per-particle float32 fields copied with the particles outside the aperture set to 0.
struct FrameFields {
  const float* in[kMaxFrameFields];
  float* out[kMaxFrameFields];
  int width[kMaxFrameFields];
  int n;
};

// rotate_galaxy + filter_particles + spaxel_assignment in one pass over the particles:
// coordinates and velocities turned by M (when rotate), the aperture mask of the turned
// coordinates, the masked copies of the fields, and the flat spaxel index.  The same
// per-particle arithmetic as rotate_kernel, aperture_mask_kernel and spaxel_assign_kernel.
__global__ void frame_assign_kernel(const float* coords, const float* velocity, long long n,
                                    int rotate, Mat3 M, float* coords_out, float* velocity_out,
                                    const float* __restrict__ edges, int n_edges, FrameFields F,
                                    unsigned char* __restrict__ mask_out,
                                    int* __restrict__ idx_out) {
  extern __shared__ float s_edges[];
  __shared__ float s_lo, s_hi;
  const bool in_smem = n_edges <= kMaxSmemEdges;
  const float* e = in_smem ? s_edges : edges;
  bool even = n_edges >= kGuessEdges;
  for (int i = threadIdx.x; i < n_edges; i += blockDim.x) {
    if (in_smem) s_edges[i] = edges[i];
    even = even && EdgeBins::even(edges, n_edges, i);
  }
  if (threadIdx.x < 32) edge_range(edges, n_edges, s_lo, s_hi);
  even = __syncthreads_and(even);
  const EdgeBins bins(e, n_edges, even);
  const float lo = s_lo, hi = s_hi;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float x = coords[3 * i], y = coords[3 * i + 1], z = coords[3 * i + 2];
    if (rotate) {
      rotate_row(x, y, z, M, x, y, z);
      coords_out[3 * i] = x;
      coords_out[3 * i + 1] = y;
      coords_out[3 * i + 2] = z;
      float vx, vy, vz;
      rotate_row(velocity[3 * i], velocity[3 * i + 1], velocity[3 * i + 2], M, vx, vy, vz);
      velocity_out[3 * i] = vx;
      velocity_out[3 * i + 1] = vy;
      velocity_out[3 * i + 2] = vz;
    }
    const bool inside = inside_aperture(x, y, lo, hi);
    if (mask_out) mask_out[i] = inside ? 1 : 0;
    for (int f = 0; f < F.n; ++f) {
      const int w = F.width[f];
      for (int k = 0; k < w; ++k) F.out[f][i * w + k] = inside ? F.in[f][i * w + k] : 0.f;
    }
    idx_out[i] = bins.flat(x, y);
  }
}

// key = idx if kept and inside [0, n_segments), else n_segments (sorts last); value = place.
struct SpaxelSource {
  const int* idx;
  const unsigned char* keep;
  int n_segments;
  __device__ __forceinline__ unsigned key(long long e) const {
    const int k = idx[e];
    const bool ok = (k >= 0) && (k < n_segments) && (keep == nullptr || keep[e] != 0);
    return ok ? (unsigned)k : (unsigned)n_segments;
  }
  __device__ __forceinline__ int val(long long e) const { return (int)e; }
};

// seg_offsets[s] = first sorted position whose key >= s, for s in [0, n_segments].
__global__ void seg_offsets_kernel(const unsigned* __restrict__ keys, long long n,
                                   int n_segments, int* __restrict__ offsets) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j <= n;
       j += (long long)gridDim.x * blockDim.x) {
    long long lo = (j == 0) ? 0 : (long long)keys[j - 1] + 1;
    long long hi = (j == n) ? n_segments : min((long long)keys[j], (long long)n_segments);
    for (long long s = lo; s <= hi; ++s) offsets[s] = (int)j;
  }
}

// The same by one binary search per segment, for many keys and segments: whatever the gaps
// between occupied segments (the pass over the keys writes a gap with one thread: 98 us for a
// disk of 10^7 stars that leaves most of 90 000 spaxels empty, this 13 us).  A chain of some 20
// loads: for fewer keys or segments the pass is the faster one (10^5 keys of 3600 segments,
// whole sort: 55.6 us with the search, 51.6 with the pass; 10^6 of 16 segments 37.4, 33.2).
__global__ void seg_search_kernel(const unsigned* __restrict__ keys, int n, int n_segments,
                                  int* __restrict__ offsets) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s <= n_segments;
       s += gridDim.x * blockDim.x) {
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = lo + ((hi - lo) >> 1);
      if (keys[mid] < (unsigned)s) lo = mid + 1; else hi = mid;
    }
    offsets[s] = lo;
  }
}

int grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  long long cap = (long long)sm_count() * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

// Bits of the keys 0..n_segments, and passes of up to nine: 10^7 keys of 90 000 spaxels (17
// bits) take two passes of 9 and 8 bits, 0.29 ms in all with the offsets, where three of 8 bits
// after a pass that wrote the keys took 0.50; the bits are spread evenly, as fewer digits make longer runs.
constexpr int kSpaxelDigits = 512;
int key_bits(int n_segments) {
  int bits = 1;
  while (bits < 32 && ((unsigned)n_segments >> bits) != 0) ++bits;
  return bits;
}

}  // namespace
}  // namespace rubix

using namespace rubix;

extern "C" int rubix_aperture_mask(const float* coords, int64_t n, int64_t coord_stride,
                                   const float* edges, int32_t n_edges, uint8_t* mask_out,
                                   void* stream) {
  RUBIX_REQUIRE(n >= 0, RUBIX_E_INVALID, "rubix_aperture_mask: n < 0");
  RUBIX_REQUIRE(n_edges >= 1, RUBIX_E_SHAPE, "rubix_aperture_mask: need at least one edge");
  RUBIX_REQUIRE(coord_stride >= 2, RUBIX_E_SHAPE, "rubix_aperture_mask: coord_stride < 2");
  if (n == 0) return RUBIX_OK;
  RUBIX_REQUIRE(coords && edges && mask_out, RUBIX_E_INVALID,
                "rubix_aperture_mask: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  aperture_mask_kernel<<<grid_for(n, 256), 256, 0, st>>>(coords, n, coord_stride, edges,
                                                          n_edges, mask_out);
  RUBIX_LAUNCH_CHECK("aperture_mask_kernel");
  return RUBIX_OK;
}

extern "C" int rubix_spaxel_assign(const float* coords, int64_t n, int64_t coord_stride,
                                   const float* edges, int32_t n_edges, int32_t* idx_out,
                                   void* stream) {
  RUBIX_REQUIRE(n >= 0, RUBIX_E_INVALID, "rubix_spaxel_assign: n < 0");
  RUBIX_REQUIRE(n_edges >= 2, RUBIX_E_SHAPE, "rubix_spaxel_assign: need at least two edges");
  RUBIX_REQUIRE((long long)(n_edges - 1) * (n_edges - 1) < (1LL << 31), RUBIX_E_SHAPE,
                "rubix_spaxel_assign: (n_edges-1)^2 overflows int32");
  RUBIX_REQUIRE(coord_stride >= 2, RUBIX_E_SHAPE, "rubix_spaxel_assign: coord_stride < 2");
  if (n == 0) return RUBIX_OK;
  RUBIX_REQUIRE(coords && edges && idx_out, RUBIX_E_INVALID,
                "rubix_spaxel_assign: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  size_t smem = n_edges <= kMaxSmemEdges ? (size_t)n_edges * sizeof(float) : 0;
  spaxel_assign_kernel<<<grid_for(n, 256), 256, smem, st>>>(coords, n, coord_stride, edges,
                                                             n_edges, idx_out);
  RUBIX_LAUNCH_CHECK("spaxel_assign_kernel");
  return RUBIX_OK;
}

extern "C" int rubix_orient_filter_assign(const float* coords, const float* velocity,
                                          int64_t n, const double* matrix9, float* coords_out,
                                          float* velocity_out, const float* edges,
                                          int32_t n_edges, int32_t n_fields,
                                          const float* const* fields_in,
                                          float* const* fields_out,
                                          const int32_t* field_widths, uint8_t* mask_out,
                                          int32_t* idx_out, void* stream) {
  RUBIX_REQUIRE(n >= 0, RUBIX_E_INVALID, "rubix_orient_filter_assign: n < 0");
  RUBIX_REQUIRE(n_edges >= 2, RUBIX_E_SHAPE,
                "rubix_orient_filter_assign: need at least two edges");
  RUBIX_REQUIRE((long long)(n_edges - 1) * (n_edges - 1) < (1LL << 31), RUBIX_E_SHAPE,
                "rubix_orient_filter_assign: (n_edges-1)^2 overflows int32");
  RUBIX_REQUIRE(n_fields >= 0 && n_fields <= kMaxFrameFields, RUBIX_E_INVALID,
                "rubix_orient_filter_assign: n_fields must be in [0, %d]", kMaxFrameFields);
  RUBIX_REQUIRE(n_fields == 0 || (fields_in && fields_out && field_widths), RUBIX_E_INVALID,
                "rubix_orient_filter_assign: null field arrays");
  RUBIX_REQUIRE(n_fields == 0 || mask_out, RUBIX_E_INVALID,
                "rubix_orient_filter_assign: filtered fields need mask_out");
  FrameFields F;
  F.n = n_fields;
  for (int f = 0; f < kMaxFrameFields; ++f) {
    F.in[f] = nullptr;
    F.out[f] = nullptr;
    F.width[f] = 0;
  }
  for (int f = 0; f < n_fields; ++f) {
    RUBIX_REQUIRE(field_widths[f] >= 1, RUBIX_E_SHAPE,
                  "rubix_orient_filter_assign: field %d has width < 1", f);
    RUBIX_REQUIRE(n == 0 || (fields_in[f] && fields_out[f]), RUBIX_E_INVALID,
                  "rubix_orient_filter_assign: field %d has a null pointer", f);
    F.in[f] = fields_in[f];
    F.out[f] = fields_out[f];
    F.width[f] = field_widths[f];
  }
  if (n == 0) return RUBIX_OK;
  RUBIX_REQUIRE(coords && edges && idx_out, RUBIX_E_INVALID,
                "rubix_orient_filter_assign: null pointer");
  Mat3 M;
  for (int i = 0; i < 9; ++i) M.m[i] = matrix9 ? matrix9[i] : (i % 4 == 0 ? 1.0 : 0.0);
  if (matrix9)
    RUBIX_REQUIRE(velocity && coords_out && velocity_out, RUBIX_E_INVALID,
                  "rubix_orient_filter_assign: a rotation needs velocity, coords_out and "
                  "velocity_out");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  size_t smem = n_edges <= kMaxSmemEdges ? (size_t)n_edges * sizeof(float) : 0;
  frame_assign_kernel<<<grid_for(n, 256), 256, smem, st>>>(
      coords, velocity, n, matrix9 ? 1 : 0, M, coords_out, velocity_out, edges, n_edges, F,
      mask_out, idx_out);
  RUBIX_LAUNCH_CHECK("frame_assign_kernel");
  return RUBIX_OK;
}

extern "C" size_t rubix_spaxel_sort_workspace_size(int64_t n, int32_t n_segments) {
  if (n < 0 || n_segments < 0) return 0;
  long long n_tiles = (n + kSortTile - 1) / kSortTile;
  if (n_tiles < 1) n_tiles = 1;
  Carve c(nullptr);
  c.take<unsigned>((size_t)n);               // keys A
  c.take<unsigned>((size_t)n);               // keys B
  c.take<int>((size_t)n);                    // vals scratch
  c.take<int>((size_t)kSpaxelDigits * (n_tiles + 1));  // histogram + digit totals
  return c.off;
}

extern "C" int rubix_spaxel_sort(const int32_t* idx, const uint8_t* keep, int64_t n,
                                 int32_t n_segments, int32_t* perm_out,
                                 int32_t* seg_offsets_out, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  RUBIX_REQUIRE(n >= 0 && n < (1LL << 31), RUBIX_E_SHAPE,
                "rubix_spaxel_sort: n must be in [0, 2^31)");
  RUBIX_REQUIRE(n_segments >= 0 && n_segments < 0x7fffffff, RUBIX_E_SHAPE,
                "rubix_spaxel_sort: bad n_segments");
  RUBIX_REQUIRE(seg_offsets_out != nullptr, RUBIX_E_INVALID,
                "rubix_spaxel_sort: seg_offsets_out is null");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n == 0) {
    RUBIX_CUDA_TRY(cudaMemsetAsync(seg_offsets_out, 0, sizeof(int) * ((size_t)n_segments + 1), st));
    return RUBIX_OK;
  }
  RUBIX_REQUIRE(idx && perm_out, RUBIX_E_INVALID, "rubix_spaxel_sort: null pointer");
  size_t need = rubix_spaxel_sort_workspace_size(n, n_segments);
  RUBIX_REQUIRE(workspace != nullptr && workspace_bytes >= need, RUBIX_E_WORKSPACE,
                "rubix_spaxel_sort: workspace of %zu bytes needed, %zu given", need,
                workspace_bytes);
  const int n_tiles = (int)((n + kSortTile - 1) / kSortTile);
  Carve c(workspace);
  unsigned* keys_a = c.take<unsigned>((size_t)n);
  unsigned* keys_b = c.take<unsigned>((size_t)n);
  int* vals_ws = c.take<int>((size_t)n);
  int* hist = c.take<int>((size_t)kSpaxelDigits * (n_tiles + 1));
  int* totals = hist + (long long)kSpaxelDigits * n_tiles;  // per-digit totals of a pass

  const int bits = key_bits(n_segments);
  const int passes = (bits + 8) / 9;
  const int per = (bits + passes - 1) / passes;
  unsigned* kin = keys_b;
  unsigned* kout = keys_a;
  int* vin = nullptr;
  for (int p = 0; p < passes; ++p) {
    const int shift = p * per;
    const int digits = 1 << std::min(per, bits - shift);
    const unsigned dmask = (unsigned)(digits - 1);
    // the last pass writes perm_out; the ones before it alternate
    int* vout = ((passes - 1 - p) % 2 == 0) ? perm_out : vals_ws;
    auto pass = [&](auto src, auto width) -> int {
      constexpr int kD = decltype(width)::value;
      radix_hist_kernel<kD><<<n_tiles, kSortThreads, 0, st>>>(src, n, shift, dmask, n_tiles, hist);
      RUBIX_LAUNCH_CHECK("radix_hist_kernel");
      radix_rowscan_kernel<<<digits, kSortThreads, 0, st>>>(hist, n_tiles, totals);
      RUBIX_LAUNCH_CHECK("radix_rowscan_kernel");
      radix_scatter_kernel<kD><<<n_tiles, kSortThreads, 0, st>>>(src, kout, vout, n, shift, dmask,
                                                                 n_tiles, hist, totals);
      RUBIX_LAUNCH_CHECK("radix_scatter_kernel");
      return RUBIX_OK;
    };
    using D256 = std::integral_constant<int, 256>;
    using D512 = std::integral_constant<int, kSpaxelDigits>;
    const SpaxelSource first{idx, keep, n_segments};
    const PairSource next{kin, vin};
    int rc;
    if (digits <= 256) rc = p == 0 ? pass(first, D256{}) : pass(next, D256{});
    else rc = p == 0 ? pass(first, D512{}) : pass(next, D512{});
    if (rc != RUBIX_OK) return rc;
    std::swap(kin, kout);
    vin = vout;
  }
  if (n > (1 << 19) && n_segments >= 1024 && n_segments < n / 2) {
    seg_search_kernel<<<grid_for((long long)n_segments + 1, 256), 256, 0, st>>>(
        kin, (int)n, n_segments, seg_offsets_out);
    RUBIX_LAUNCH_CHECK("seg_search_kernel");
    return RUBIX_OK;
  }
  seg_offsets_kernel<<<grid_for(n + 1, 256), 256, 0, st>>>(kin, n, n_segments, seg_offsets_out);
  RUBIX_LAUNCH_CHECK("seg_offsets_kernel");
  return RUBIX_OK;
}
