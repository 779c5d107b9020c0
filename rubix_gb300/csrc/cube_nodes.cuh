// Interface of the node-by-node forward (cube_nodes.cu) to the entry points of kernel (b).
#pragma once

#include "cube_common.cuh"

namespace rubix {

// What the node path leaves for cube_main_kernel: the flagged spaxels and its inputs
// (built only when some spaxel is flagged; all pointers are device memory).
struct NodeFallback {
  const int* gate;  // work items: of several-chunk spaxels, of the others
  int2* items;      // the former from 0, the latter from split
  int split, chunk;
  int* slot_start;
  float* At;
  int2* bucket;
  float4* ct;
  ParticleRec* rec;
  int* done;
  float* partials;
};

// Runs the node path: the cube of every spaxel that is not flagged, and *fb for the rest.
int cube_nodes_forward(const CubeInputs& in, const float* lsf_taps, int n_lsf, int lsf_crop,
                       int big_item, float* cube, long long stride, void* ws, size_t ws_bytes,
                       NodeFallback* fb, cudaStream_t st);

// Whether the host-side sizes qualify (the template slice fits shared memory).
bool cube_nodes_supported(int nZ, int nA, int nW, int n_t);
// Workspace of the node path, and whether a workspace of `bytes` holds it (with fewer rows
// at a time in a smaller one).
size_t cube_nodes_bytes(long long n, int n_seg, int nZ, int nA, int nW, int n_t);
bool cube_nodes_fit(long long n, int n_seg, int nZ, int nA, int nW, int n_t, size_t bytes);

// Kernels that cube_nodes_forward launches.
int cube_nodes_launches(long long n, int n_seg, int nZ, int nA, int nW, size_t bytes);
// Workspace of the path without it (accumulate.cu).
size_t cube_general_workspace(int64_t n, int32_t n_segments, int32_t n_wave_t, int32_t n_met,
                              int32_t n_age, int32_t n_wave);

}  // namespace rubix
