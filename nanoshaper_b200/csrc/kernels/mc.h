// Vertex assembly and marching-cubes kernels (mc.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "lookback.cuh"
#include "pipeline.h"

namespace nsg {

// Item counts of a triangulation, kept on the device (int64 each): the passes read the counts of
// the passes before them there, and the host reads them once, at the end.
enum { kMcAnalytic = 0, kMcActive = 1, kMcMidpoint = 2, kMcTriangle = 3, kMcLowFace = 4, kMcCounts = 8 };

// Both argument blocks cover a whole batch: ray ordinals, cube rows, active cubes and vertices
// are batch-wide; every structure's bit grid starts at its word_base in `bits`.  The output arrays
// have capacities (items): a pass drops what exceeds them and the passes after it do nothing, and
// the host, which sees the counts, enlarges the arrays and runs the passes again.
struct VertArgs {
  BatchDev B;
  int64_t nrays;                 // accurate-triangulation rays of the three panels, all structures
  const int64_t* ray_pair_off;
  const int32_t* ray_pair_cnt;
  const double* pairs;
  const uint32_t* bits;
  double* vpos;                  // 3 per vertex
  int4* vkey;                    // ix, iy, iz, dir per vertex
  int32_t* vstruct;              // structure of every vertex
  int64_t cap;                   // vertices
  const int2* pair_pid;          // gradient mode: patches of the pair ends, else null
  int32_t* vpid;                 // gradient mode: patch of every analytic vertex
  int64_t* voff;                 // first analytic vertex of every structure (n+1)
  int64_t* counts;
  LookBack lb;
};

struct MCArgs {
  BatchDev B;
  const uint32_t* bits;
  double* vpos;
  int4* vkey;
  int32_t* vstruct;              // structure of every vertex
  int64_t cap_vert, cap_active, cap_tri;
  int64_t nwords_map;            // entries of the active-cube map
  int4* act_rec;                 // i, j, k, case | structure << 11
  int32_t* tri_cnt;              // triangles per active cube (interior cubes: from the classification)
  int32_t* bnd_list;             // active cubes on the low faces of the cube range
  // active-cube map, one entry per 32 cubes of a cube row (W = ceil((NX-2)/32) per row, rows of a
  // structure from its aword_base): the cubes' active bits and the active index of the first
  // active cube of the word
  int2* amap;
  int32_t* cube_vl;              // 12 per active cube: the vertex of each cut edge it reads
  bool clear_slots;              // the classification clears the slots (a batch of one chunk)
  int32_t* tris;
  double* cube_area;
  const int64_t* voff;           // first analytic vertex of every structure (n+1)
  int64_t* aoff;                 // first active cube of every structure (n+1)
  int64_t* counts;
  LookBack lb_rows, lb_mid, lb_tris;
  // gradient mode (vgrad null otherwise): d area / d (analytic vertex position along its ray),
  // then d area / d patch parameters
  const int32_t* vpid;
  double* vgrad;
  double* garea;
  const double* f64;
  const int32_t* i32;
  double probe;
};

// Look-back tickets of the four passes over so many rays, map words and (at most) active cubes.
struct McTickets {
  int64_t vert, rows, mid, tris;
};
McTickets mc_tickets(int64_t rays, int64_t words, int64_t cubes);
cudaError_t launch_vert(const VertArgs& A, cudaStream_t s);
cudaError_t launch_mc_rows(const MCArgs& A, cudaStream_t s);
// Slots of the active cubes of structures [b0, b1) to -1; `cubes` (about as many) sizes the grid.
cudaError_t launch_mc_clear(const MCArgs& A, int b0, int b1, int64_t cubes, cudaStream_t s);
cudaError_t launch_mc_mid(const MCArgs& A, cudaStream_t s);
// blocks_per_sm: 4 (64 registers a thread) or 3 (80 registers).
cudaError_t launch_mc_tris(const MCArgs& A, int blocks_per_sm, cudaStream_t s);
// Analytic vertices of structures [b0, b1) (about `vertices` of them): the first vertex of each
// grid edge is written into the vertex slots of the (up to four) active cubes that share the edge.
cudaError_t launch_mc_push(const MCArgs& A, int b0, int b1, int64_t vertices, cudaStream_t s);
// Triangle counts of the listed low-face cubes, once the midpoint vertices are in place.
cudaError_t launch_mc_tris_bnd(const MCArgs& A, cudaStream_t s);
// Analytic normal of every analytic vertex v < n_analytic from its patch vpid[v] (zero for patch
// kinds without one, e.g. mesh triangles); 3 doubles per vertex.
cudaError_t launch_vertex_normals(const double* vpos, const int32_t* vpid, int64_t n_analytic, const double* f64,
                                  const int32_t* i32, double probe, double* normals, cudaStream_t s);
// d area / d patch parameters from the per-vertex derivatives (gradient mode).
cudaError_t launch_grad_vert(const MCArgs& A, int64_t vertices, cudaStream_t s);

}  // namespace nsg
