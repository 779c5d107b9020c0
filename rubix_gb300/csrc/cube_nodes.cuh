// Interface of the node-by-node forward (cube_nodes.cu) to the entry points of kernel (b).
#pragma once

#include "cube_common.cuh"

namespace rubix {

// What the node path leaves for cube_main_kernel: the work items of the flagged spaxels
// (their number in the workspace's CubeCtrl, 0 when none is flagged) and its inputs.
struct NodeFallback {
  int chunk;
  float alo, ahi;  // alpha at -kVmaxKms and kVmaxKms
  int2* items;  // items of several-chunk spaxels (item index = partial slot), then others
  int* slot_start;
  float* At;
  int2* bucket;
  float4* ct;
  ParticleRec* rec;
  int* done;
  float* partials;
};

// Runs the node path: the cube of every spaxel that is not flagged, and *fb for the rest.
// dust_e: dust exponents per telescope wavelength (with in.av), or null.  tune: the work items
// of the general kernel.
int cube_nodes_forward(const CubeInputs& in, const float* dust_e, const float* lsf_taps, int n_lsf, int lsf_crop,
                       const CubeTuning& tune, float* cube, long long stride, void* ws,
                       size_t ws_bytes, NodeFallback* fb, cudaStream_t st);

// Which path a call takes by its sizes: kPathAuto the node path where it is the faster one.
enum CubePath { kPathAuto, kPathGeneral, kPathNodes };
bool cube_nodes_worth(long long n, int n_seg, int nZ, int nA, int nW, int n_t);

// Whether the host-side sizes qualify (the template slice fits shared memory).
bool cube_nodes_supported(int nZ, int nA, int nW, int n_t);
// Workspace of the node path, and whether a workspace of `bytes` holds it (with as little as half
// the rows at a time; with fewer, in more waves, it is slower than the general path);
// chunk: of the general kernel's work items.
size_t cube_nodes_bytes(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk);
bool cube_nodes_fit(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk,
                    size_t bytes);

// Kernels that cube_nodes_forward launches.
int cube_nodes_launches(long long n, int n_seg, int nZ, int nA, int nW, size_t bytes);
// The adjoint of cube_nodes_forward without dust (cube_nodes_bwd.cu): grads are dL/dmass,
// dL/dZ, dL/dage and dL/dv_los (zeroed by the caller, null where not wanted).
int cube_nodes_backward(const CubeInputs& in, const float* adj, long long adj_stride,
                        const CubeTuning& tune, float* const* grads, void* ws, size_t ws_bytes, NodeFallback* fb,
                        cudaStream_t st);
bool cube_nodes_bwd_supported(int nZ, int nA, int nW, int n_t);
size_t cube_nodes_bwd_bytes(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk);
bool cube_nodes_bwd_fit(long long n, int n_seg, int nZ, int nA, int nW, int n_t, int chunk,
                        size_t bytes);
int cube_nodes_bwd_launches(long long n, int n_seg, int nZ, int nA, int nW, size_t bytes);
// Workspace of the path without it (accumulate.cu).
size_t cube_general_workspace(int64_t n, int32_t n_segments, int32_t n_wave_t, int32_t n_met,
                              int32_t n_age, int32_t n_wave);

}  // namespace rubix
