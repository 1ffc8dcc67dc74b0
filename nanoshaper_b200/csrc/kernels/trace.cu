// Patch windows, candidates, torus screen, intersections and interval fill of the ray caster.
//
// The reference is patch-centric: every patch loops over the pixels of its bounding window,
// tests the rays and pushes hits into per-pixel heap lists that are then sorted
// (ConnollySurface::getPatchIntersectionData src/ConnollySurface.cpp:4319-4590,
// Surface::countPixelIntersections/copyPatchIntersections/reorderPatchIntersections
// src/Surface.cpp:4941-5095) and consumed by setVerticesAndGridsWithIntersectionData
// (src/Surface.cpp:5101-6251).  Here the (ray, patch) candidates of a ray set are listed first, tested
// one per thread, and the hits of a ray are sorted and paired by the warp that owns its tile of 32x4
// pixels; the kernels are described at their places below.  The candidate set of a ray is the
// reference's: pixel inside the patch window, inside the bounding box, inside the equatorial disc.
// Only rays with more than 32 hits go through per-tile patch lists, one thread per ray.
#include <limits.h>

#include "pipeline.h"
#include "ray_math.cuh"
#include "ray_math_mixed.cuh"
#include "grad.cuh"
#include "isect.cuh"
#include "lookback.cuh"
#include "../torus_screen.h"

namespace nsg {

namespace {

// Pixel window of every patch (start, end per axis; -1 when culled) and the screen record of the torus
// patches, with the panels' window-area sums (out[0..2], out[3..5] for the torus patches) and the
// patch kinds present (out[6]) of the same pass.  The sums go through one atomic per block, word and
// kind: one per warp is 5 ns each on the same address, 169 us for 340,000 mesh triangles (-> 50).
constexpr int kWinThreads = 256;
__global__ void __launch_bounds__(kWinThreads) k_windows(PatchDev P, int32_t* win, float4* screen, BatchDev B,
                                                         unsigned long long* out) {
  __shared__ unsigned long long s_sum[kWindowSums];
  if (threadIdx.x < kWindowSums) s_sum[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  unsigned long long area[3] = {0, 0, 0}, tor[3] = {0, 0, 0};
  unsigned kinds = 0;
  for (int64_t p = blockIdx.x * (int64_t)kWinThreads + threadIdx.x; p < P.n; p += (int64_t)gridDim.x * kWinThreads) {
    const GridDev& g = B.s[B.patch_struct[p]].g;
    const double* f = P.f64 + (int64_t)NS_PATCH_F64 * p;
    const int32_t* ir = P.i32 + NS_PATCH_I32 * p;
    const double r = f[3];
    double down[3], up[3];
    bool cull = false;
    const int kind = ir[0];
    const bool skin = ns_has_box(kind), torus = kind == NS_EDGE_REG || kind == NS_EDGE_SING;
    kinds |= 1u << kind;
    for (int d = 0; d < 3; d++) {
      // SES: the bounding sphere's box; skin cells and mesh triangles: their stored box
      // (src/SkinSurface.cpp:3470-3500, src/MeshSurface.cpp:447-472)
      down[d] = skin ? f[NS_SKIN_LO + d] : f[d] - r;
      up[d] = skin ? f[NS_SKIN_HI + d] : f[d] + r;
      if (down[d] > g.mx[d] + NS_EPS_INT) cull = true;
    }
    for (int d = 0; d < 3; d++)
      if (up[d] < g.mn[d] - (g.hside - NS_DELTA + NS_EPS_INT)) cull = true;
    int32_t* w = win + 6 * p;
    unsigned long long size[3] = {0, 0, 0};
    for (int d = 0; d < 3; d++) {
      int64_t s = -1, e = -1;
      if (!cull) {
        s = (int64_t)rintp(fmax(0., down[d] - g.mn[d]) * g.scale);
        e = (int64_t)rintp(fmax(0., up[d] - g.mn[d]) * g.scale);
        if (e >= g.n[d]) e = g.n[d] - 1;
        if (e >= s) size[d] = (unsigned long long)(e - s + 1);
      }
      w[d] = (int32_t)s;
      w[3 + d] = (int32_t)e;
    }
    const unsigned long long win_area[3] = {size[1] * size[2], size[0] * size[1], size[0] * size[2]};
    for (int q = 0; q < 3; q++) {
      area[q] += win_area[q];
      if (torus) tor[q] += win_area[q];
    }
    if (torus && screen) {
      float rec[kTorusScreen];
      const int first = ir[1], cnt = ir[2];
      const bool wedge = cnt == 2 && P.flag[first] != 0;
      torus_screen_record(f, wedge ? (const double*)(P.pool + first) : nullptr, wedge, P.probe, rec);
      float4* o = screen + (kTorusScreen / 4) * p;
#pragma unroll
      for (int q = 0; q < kTorusScreen / 4; q++)
        o[q] = make_float4(rec[4 * q], rec[4 * q + 1], rec[4 * q + 2], rec[4 * q + 3]);
    }
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    for (int o = 16; o; o >>= 1) {
      area[q] += __shfl_xor_sync(0xffffffffu, area[q], o);
      tor[q] += __shfl_xor_sync(0xffffffffu, tor[q], o);
    }
    if (lane == 0 && area[q]) atomicAdd(s_sum + q, area[q]);
    if (lane == 0 && tor[q]) atomicAdd(s_sum + 3 + q, tor[q]);
  }
  kinds = __reduce_or_sync(0xffffffffu, kinds);
  if (lane == 0 && kinds) atomicOr(s_sum + 6, (unsigned long long)kinds);
  __syncthreads();
  if (threadIdx.x < 6 && s_sum[threadIdx.x]) atomicAdd(out + threadIdx.x, s_sum[threadIdx.x]);
  if (threadIdx.x == 6 && s_sum[6]) atomicOr(out + 6, s_sum[6]);
}

// Patch-local FP32 copies of the pool entries (and of the skin quadrics).  A warp takes 32 patches and
// spreads their entries over its lanes, in pool order: consecutive patches' entries are neighbours,
// so loads and stores are coalesced (a patch per lane: 110 us for 2.9 M entries -> 64 us).
__global__ void k_pool32(PatchDev P, float4* out, float4* quad32, double4* quadl) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = p < P.n;
  const double* f = P.f64 + (int64_t)NS_PATCH_F64 * (valid ? p : 0);
  const int32_t* ir = P.i32 + NS_PATCH_I32 * (valid ? p : 0);
  const int kind = ir[0];
  const bool skin = ns_is_skin(kind);
  {
    const int lane = threadIdx.x & 31;
    const int cnt = valid ? ir[2] : 0, first = ir[1];
    const double c0 = f[0], c1 = f[1], c2 = f[2];
    const int incl = warp_incl(cnt);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int e0 = 0; e0 < total; e0 += 32) {
      const int e = e0 + lane;
      const int l = owner_lane(incl, e < total ? e : total - 1);
      const int q = __shfl_sync(0xffffffffu, first, l) + (e - __shfl_sync(0xffffffffu, incl - cnt, l));
      const int k = __shfl_sync(0xffffffffu, kind, l);
      const double o0 = __shfl_sync(0xffffffffu, c0, l), o1 = __shfl_sync(0xffffffffu, c1, l),
                   o2 = __shfl_sync(0xffffffffu, c2, l);
      if (e >= total) continue;
      const double4 w = P.pool[q];
      if (k == NS_POINT) {
        out[q] = make_float4((float)(w.x - o0), (float)(w.y - o1), (float)(w.z - o2), (float)w.w);
      } else {
        // planes about the local origin; the skin's (partly unnormalised) planes are scaled to unit
        // normals so that the FP32 value is a distance (the scale does not change a sign)
        const double inv = ns_is_skin(k) ? 1.0 / sqrt(w.x * w.x + w.y * w.y + w.z * w.z) : 1.0;
        out[q] = make_float4((float)(w.x * inv), (float)(w.y * inv), (float)(w.z * inv),
                             (float)((w.w + (w.x * o0 + w.y * o1 + w.z * o2)) * inv));
      }
    }
  }
  if (!valid) return;
  if (skin && quad32) {
    // the quadric about the local origin c: A, bl = A c + b, cl = f(c)
    const double* Q = f + NS_SKIN_Q;
    const double A[3][3] = {{Q[0], Q[4], Q[7]}, {Q[4], Q[1], Q[5]}, {Q[7], Q[5], Q[2]}};
    const double b[3] = {Q[9], Q[8], Q[6]};
    double bl[3];
    for (int i = 0; i < 3; i++) bl[i] = (A[i][0] * f[0] + A[i][1] * f[1] + A[i][2] * f[2]) + b[i];
    const double cl = (f[0] * (bl[0] + b[0]) + f[1] * (bl[1] + b[1]) + f[2] * (bl[2] + b[2])) + Q[3];
    quad32[3 * p] = make_float4((float)A[0][0], (float)A[1][1], (float)A[2][2], (float)A[0][1]);
    quad32[3 * p + 1] = make_float4((float)A[1][2], (float)A[0][2], (float)bl[0], (float)bl[1]);
    quad32[3 * p + 2] = make_float4((float)bl[2], (float)cl, 0.f, 0.f);
    quadl[p] = make_double4(bl[0], bl[1], bl[2], cl);
  }
}

__global__ void k_bin(PatchDev P, BatchDev B, int set, int32_t* tile_cnt, const int64_t* tile_off,
                      int32_t* tile_cursor, int32_t* tile_list) {
  int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= P.n) return;
  const int32_t* w = P.win + 6 * p;
  if (w[0] < 0) return;
  const StructDev& S = B.s[B.patch_struct[p]];
  const RaySet rs = make_ray_set(set, S.g);
  int64_t ntm = (rs.nb + kTileM - 1) / kTileM;
  int m0 = w[rs.fd] / kTileM, m1 = w[3 + rs.fd] / kTileM;
  int n0 = w[rs.ld] / kTileN, n1 = w[3 + rs.ld] / kTileN;
  for (int tn = n0; tn <= n1; tn++)
    for (int tm = m0; tm <= m1; tm++) {
      int64_t t = S.tile_base[rs.panel] + (int64_t)tn * ntm + tm;
      if (tile_list == nullptr) {
        atomicAdd(tile_cnt + t, 1);
      } else {
        int pos = atomicAdd(tile_cursor + t, 1);
        tile_list[tile_off[t] + pos] = (int32_t)p;
      }
    }
}

// Candidate test of the reference's pixel loop: the ray origin lies inside the patch's bounding
// box and equatorial disc (src/ConnollySurface.cpp:4469-4502); the pixel window test is done by
// the caller.
__device__ __forceinline__ bool candidate(const double* f, const RaySet& rs, const double* pa) {
  int fd = rs.fd, ld = rs.ld;
  double r = f[kR];
  if (pa[fd] < f[fd] - r || pa[fd] > f[fd] + r) return false;
  if (pa[ld] < f[ld] - r || pa[ld] > f[ld] + r) return false;
  double dx = f[fd] - pa[fd];
  double dy = f[ld] - pa[ld];
  return !(dx * dx + dy * dy > r * r);
}

// Double-precision intersection of a candidate: hits in t[0..n-1] (ray parameter units).
__device__ __forceinline__ int intersect_f64(const double* f, int kind, int first, int cnt, const PatchDev& P,
                                             const RaySet& rs, const double* pa, const double* dir, double ray_dir,
                                             double* t) {
  int vc = rs.vc;
  if (!ray_sphere_f64(pa, dir, f, f[kR], &t[0], &t[1])) return 0;
  int numInt = 2;
  if (kind == NS_EDGE_REG || kind == NS_EDGE_SING) numInt = ray_torus_f64(f, P.probe, vc, pa, ray_dir, t);
  int out = 0;
  for (int i = 0; i < numInt; i++) {
    double ip[3] = {pa[0], pa[1], pa[2]};
    ip[vc] += t[i] * ray_dir;
    if (feasible_f64(f, kind, first, cnt, P.pool, P.flag, ip)) t[out++] = t[i];
  }
  return out;
}

// Tests one (ray, patch) candidate and reports the feasible hits in t[0..n-1].
__device__ __forceinline__ int ray_patch_f64(const double* f, int kind, int first, int cnt, const PatchDev& P,
                                             const RaySet& rs, const double* pa, const double* dir, double ray_dir,
                                             double box_dir, double tri_dir, double* t) {
  if (kind == NS_MESH_TRI) {
    for (int a = 0; a < 2; a++) {
      const int d = a == 0 ? rs.fd : rs.ld;
      if (pa[d] < f[NS_SKIN_LO + d] || pa[d] > f[NS_SKIN_HI + d]) return 0;
    }
    double tdir[3] = {0.0, 0.0, 0.0}, u, v;
    tdir[rs.vc] = tri_dir;
    return ray_triangle_f64(pa, tdir, f, f + 3, f + 6, t, &u, &v) ? 1 : 0;
  }
  if (ns_is_skin(kind)) {
    // the cell's box in the pixel axes, the atom disc for Del0 cells, then the ray-quadric test
    for (int a = 0; a < 2; a++) {
      const int d = a == 0 ? rs.fd : rs.ld;
      if (pa[d] < f[NS_SKIN_LO + d] || pa[d] > f[NS_SKIN_HI + d]) return 0;
    }
    if (kind == NS_SKIN_POINT) {
      const double dx = f[rs.fd] - pa[rs.fd], dy = f[rs.ld] - pa[rs.ld];
      if (dx * dx + dy * dy > f[kR] * f[kR]) return 0;
    }
    double tt[2];
    bool hit = rs.vc == 0 ? ray_quadric_f64<0>(f + NS_SKIN_Q, pa, tt)
                          : (rs.vc == 1 ? ray_quadric_f64<1>(f + NS_SKIN_Q, pa, tt) : ray_quadric_f64<2>(f + NS_SKIN_Q, pa, tt));
    if (!hit) return 0;
    int out = 0;
    for (int i = 0; i < 2; i++) {
      double ip[3] = {pa[0], pa[1], pa[2]};
      ip[rs.vc] += tt[i];
      if (feasible_skin_f64(P.pool, first, cnt, ip)) t[out++] = tt[i] / box_dir;
    }
    return out;
  }
  if (!candidate(f, rs, pa)) return 0;
  return intersect_f64(f, kind, first, cnt, P, rs, pa, dir, ray_dir, t);
}

// Pairs the sorted hits of one ray in place (NEW_INTERSECTION_FILTERING) and turns them into
// interval ends along the ray axis; returns the number of pairs and the interval length sum.
// When vertex_pairs is set, only pairs that clear at least one insideness node are kept.
// With pcol (the hits' patches, gradient mode) the patch column is compacted alongside, and every
// interval end adds its term of d volume / d patch parameters (GradCtx).
struct GradCtx {
  const double* f64;
  const int32_t* i32;
  double probe;
  double w;          // volume weight of an interval length: A / number of ray sets
  double x[3];       // ray origin; x[vc] is replaced by the interval end
  int vc;
  double* gvol;
};

struct SamePid {
  __device__ __forceinline__ int32_t operator()(int32_t p) const { return p; }
};

// pcol holds, per hit, an id that pid_of turns into the hit's patch (the patch itself, or the
// hit's slot in the hit store).
template <class IdT = int32_t, class PidOf = SamePid>
__device__ __forceinline__ int make_pairs(double* col, int stride, int nh, double pa_vc, double dir, double vmin,
                                          double scale, bool vertex_pairs, double* vol, IdT* pcol = nullptr,
                                          GradCtx* gc = nullptr, PidOf pid_of = PidOf()) {
  double v = 0.0;
  int np = 0;
  if (nh > 0 && (nh & 1) == 0) {
    for (int q = 0; q < nh; q += 2) {
      double t1 = col[q * stride], t2 = col[(q + 1) * stride];
      if (fabs(t2 - t1) >= NS_EPS_INT) {
        double lim1 = pa_vc + dir * t1;
        double lim2 = pa_vc + dir * t2;
        v += lim2 - lim1;
        IdT p1 = 0, p2 = 0;
        if (pcol) {
          p1 = pcol[q * stride];
          p2 = pcol[(q + 1) * stride];
          if (gc) {
            double x[3] = {gc->x[0], gc->x[1], gc->x[2]};
            x[gc->vc] = lim1;
            add_hit_grad(gc->f64, gc->i32, gc->probe, pid_of(p1), x, gc->vc, -gc->w, gc->gvol);
            x[gc->vc] = lim2;
            add_hit_grad(gc->f64, gc->i32, gc->probe, pid_of(p2), x, gc->vc, gc->w, gc->gvol);
          }
        }
        if (vertex_pairs) {
          int64_t a = (int64_t)rintp((lim1 - vmin) * scale);
          int64_t b = (int64_t)rintp((lim2 - vmin) * scale);
          if (b <= a) continue;
        }
        col[(2 * np) * stride] = lim1;
        col[(2 * np + 1) * stride] = lim2;
        if (pcol) {
          pcol[(2 * np) * stride] = p1;
          pcol[(2 * np + 1) * stride] = p2;
        }
        np++;
      }
    }
  }
  *vol = v;
  return np;
}

// Nodes of a status row inside one interval: the reference loops over the clamped rintp range
// [i1, i2] and marks the nodes with lim1 <= x <= lim2 (src/Surface.cpp:5427-5552); that set is
// the contiguous range returned here (ia > ib when empty).
__device__ __forceinline__ void status_node_range(const GridDev& g, double lim1, double lim2, int64_t* ia, int64_t* ib) {
  const int64_t NX = g.n[0];
  int64_t i1 = (int64_t)rintp((lim1 - g.mn[0]) * g.scale);
  int64_t i2 = (int64_t)rintp((lim2 - g.mn[0]) * g.scale);
  i1 = i1 < 0 ? 0 : (i1 >= NX ? NX - 1 : i1);
  i2 = i2 < 0 ? 0 : (i2 >= NX ? NX - 1 : i2);
  int64_t a = i1, b = i2;
  while (a <= b && gcoord(g, 0, a) < lim1) a++;
  while (b >= a && gcoord(g, 0, b) > lim2) b--;
  *ia = a;
  *ib = b;
}

// Epsilon-map entries of one interval [lim1, lim2] of a node ray (sets 0, 4, 5): the reference takes
// the clamped rintp node range [c1, c2] of the interval and marks the grid edges that start at a
// node c with coord(c) <= lim2 - hside (src/Surface.cpp:6645-6680 for x, inclusive of c2;
// :6786-6795 for z and :6887-6896 for y, exclusive of c2).  m, n are the ray's pixel indices.
__device__ __forceinline__ void eps_fill(const GridDev& g, const RaySet& rs, int64_t m, int64_t n, double lim1,
                                         double lim2, int32_t* __restrict__ eps, int32_t inside) {
  const int vc = rs.vc;
  const int64_t N = g.n[vc];
  int64_t c1 = (int64_t)rintp((lim1 - g.mn[vc]) * g.scale);
  int64_t c2 = (int64_t)rintp((lim2 - g.mn[vc]) * g.scale);
  c1 = c1 < 0 ? 0 : (c1 >= N ? N - 1 : c1);
  c2 = c2 < 0 ? 0 : (c2 >= N ? N - 1 : c2);
  if (c2 < c1) return;
  int64_t e = vc == 0 ? c2 : c2 - 1;
  const double lim = lim2 - g.hside;
  while (e >= c1 && gcoord(g, vc, e) > lim) e--;
  const int64_t NX = g.n[0], NY = g.n[1];
  // node (i, j, k) of position c along the ray; l = the component of this ray set
  int64_t base, step;
  int l;
  if (vc == 0) { base = (n * NY + m) * NX; step = 1; l = 0; }
  else if (vc == 2) { base = n * NX + m; step = NX * NY; l = 2; }
  else { base = n * NY * NX + m; step = NX; l = 1; }
  for (int64_t c = c1; c <= e; c++) eps[(base + c * step) * 3 + l] = inside;
}

// Warp-aggregated append of this lane's `cnt` records to a shared store; returns the lane's first
// slot, or -1 when the store is full (the error flag is then set to `code`).
__device__ __forceinline__ int64_t warp_append(unsigned long long* cursor, int64_t cap, int cnt, int32_t* error_flag,
                                               int code) {
  const int lane = threadIdx.x & 31;
  int incl = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  int total = __shfl_sync(0xffffffffu, incl, 31);
  unsigned long long base = 0;
  if (lane == 31 && total > 0) base = atomicAdd(cursor, (unsigned long long)total);
  base = __shfl_sync(0xffffffffu, base, 31);
  if ((int64_t)base + total > cap) {
    if (lane == 0 && total > 0) atomicExch(error_flag, code);
    return -1;
  }
  return (int64_t)base + incl - cnt;
}

__device__ __forceinline__ void clear_bits_range(uint32_t* bits, int64_t nwords, int64_t f0, int64_t f1) {
  // clears bits f0..f1 inclusive of the flat bit grid (bit = 0 means inside)
  if (f1 < f0) return;
  if (f0 < 0) f0 = 0;
  int64_t lim = nwords * 32 - 1;
  if (f1 > lim) f1 = lim;
  for (int64_t w = f0 >> 5; w <= (f1 >> 5); w++) {
    int64_t lo = w << 5;
    int s = (int)(f0 > lo ? f0 - lo : 0);
    int e = (int)(f1 < lo + 31 ? f1 - lo : 31);
    uint32_t mask = (e - s == 31) ? 0xffffffffu : (((1u << (e - s + 1)) - 1u) << s);
    atomicAnd(bits + w, ~mask);
  }
}


// Wavefront ray tracing of one ray set, three kernel kinds:
//  * k_cand: one warp per batch of 4 to 32 patches, whose records the lanes load together; then, patch
//    by patch, one lane per pixel row of the patch's pixel window (the reference's CELL_CULLING
//    window, k_windows): each row's rays that pass the bounding-box and equatorial-disc test form
//    an interval, found by moving a predicted end with the exact test.  One atomic per list and batch
//    reserves the slots; the (ray, patch) pairs follow in row-major order, in the sphere list
//    (atoms and probes) or the torus list; a patch's candidates stay contiguous, so the
//    intersection kernels read its record once per warp;
//  * k_isect<torus> (double precision) and k_isect_mixed<torus> (trace_mixed.cu): one thread per
//    candidate pair, sphere and torus pairs in separate launches so that both run converged with
//    their own register budget; hits are filed into the ray's slots of a slot-major hit store
//    through a per-ray atomic counter;
//  * k_fill: one CTA per 32x4 ray tile loads each ray's hits, sorts them and performs the
//    interval fill.
// A k_cand batch of up to 32 patches, staged in shared memory (structure of arrays, one entry per lane
// of the warp that loaded it): the operands of candidate() rounded as there, the pixel window
// and where the patch's rays start.
struct CandBatch {
  double cf[32], cl[32], lo_fd[32], hi_fd[32], lo_ld[32], hi_ld[32], r2[32], mn_fd[32], mn_ld[32], side[32],
      delta[32];
  int64_t nb[32], rbase[32], base[32];
  int m0[32], m1[32], n0[32], ty[32], pid[32], disc[32];
  int64_t gfirst[32], gend[32];
};

// Candidate count of pixel row `row` of batch patch p (its first candidate pixel in *a).  Along a
// row the pixel coordinate pa(m) is non-decreasing in m and dx = cf - pa(m) non-increasing;
// fl(fl(dx*dx) + fl(dy*dy)) is non-decreasing in |dx|.  So
//   Low(m)  = pa(m) >= lo_fd && (dx < 0 || disc(dx))   holds on an upper set of m,
//   High(m) = pa(m) <= hi_fd && (dx > 0 || disc(dx))   holds on a lower set of m,
// and candidate() (box in both axes, then disc) passes exactly when the row's box test holds and
// Low(m) && High(m).  The row's candidates are the interval [first Low, last High] of the window.
// Both ends start at the pixel that an FP32 half chord predicts and are moved with the exact
// double-precision tests until the test flips there, which the monotone tests make the same pixel
// that a search of the whole window finds, in 4 tests instead of 2 log2(window).
__device__ __forceinline__ int cand_row(const CandBatch& q, int p, int row, int* a) {
  *a = 0;
  const double pld = (q.mn_ld[p] + (double)(q.n0[p] + row) * q.side[p]) + q.delta[p];
  if (pld < q.lo_ld[p] || pld > q.hi_ld[p]) return 0;
  const double cl = q.cl[p], cf = q.cf[p], r2 = q.r2[p], mn = q.mn_fd[p], side = q.side[p], delta = q.delta[p];
  const double lo_fd = q.lo_fd[p], hi_fd = q.hi_fd[p];
  const double dy = cl - pld;
  const double dy2 = dy * dy;
  // skin cells other than Del0 have no equatorial-disc test (src/SkinSurface.cpp:3578-3587)
  const bool disc = q.disc[p];
  const int m0 = q.m0[p], m1 = q.m1[p];
  double from = lo_fd, to = hi_fd;
  if (disc) {
    if (dy2 > r2 && cf == cf) return 0;  // no pixel of the row passes the disc test
    const double h = (double)sqrtf((float)(r2 - dy2));
    from = fmax(from, cf - h);
    to = fmin(to, cf + h);
  }
  const double inv = (double)(1.0f / (float)side), org = mn + delta;
  const auto low = [&](int m) {
    const double pa = (mn + (double)m * side) + delta;
    const double dx = cf - pa;
    return !(pa < lo_fd) && (!disc || dx < 0. || !(dx * dx + dy2 > r2));
  };
  const auto high = [&](int m) {
    const double pa = (mn + (double)m * side) + delta;
    const double dx = cf - pa;
    return !(pa > hi_fd) && (!disc || dx > 0. || !(dx * dx + dy2 > r2));
  };
  // the predictions are clamped as doubles: a box far outside the grid does not fit an int
  int lo = (int)fmin(fmax(ceil((from - org) * inv), (double)m0), (double)m1 + 1.);
  while (lo > m0 && low(lo - 1)) lo--;
  while (lo <= m1 && !low(lo)) lo++;
  int hi = (int)fmin(fmax(floor((to - org) * inv) + 1., (double)lo), (double)m1 + 1.);
  while (hi > lo && !high(hi - 1)) hi--;
  while (hi <= m1 && high(hi)) hi++;
  *a = lo;
  return hi - lo;
}

// Rows of a batch whose interval stays in shared memory between the counting and the writing pass
// (first pixel relative to the window and count, 16 bits each); the others are found again.
constexpr int kCandRows = 320;
constexpr uint32_t kCandRowAgain = 0xffffffffu;

// ppw: patches of a warp's batch (launch_trace picks it so that small patch sets fill the GPU).
// Latency-bound (dependent double-precision tests, 5-step shuffles per row group), 12 % of the warps
// resident with 32 patches per warp on a 20,000-atom cast: what counts is warps in flight.  Per
// launch, 32 patches per warp and binary searches in both passes -> as it is here: 26 -> 5.7 us
// (327 atoms, scale 2), 46 -> 8.8 us (2,000, scale 3), 77 -> 25 us (20,000, scale 4), 194 -> 179 us
// (64 conformers, 580,000 patches, whose warps filled the GPU before).
__global__ void __launch_bounds__(256) k_cand(const __grid_constant__ TraceSets T, int ppw) {
  const TraceCtx C{T.P, T.B, T.set[blockIdx.y], T.out[blockIdx.y]};
  const CandOut& co = T.co[blockIdx.y];
  __shared__ CandBatch s_batch[8];
  __shared__ uint32_t s_row[8][kCandRows];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  CandBatch& q = s_batch[wib];
  uint32_t* const rows = s_row[wib];
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t base = (blockIdx.x * (int64_t)(blockDim.x >> 5) + wib) * ppw; base < C.P.n; base += warps * ppw) {
    // 1. the batch's patches, one per lane
    int H = 0;
    {
      const int64_t pid = base + lane;
      q.ty[lane] = 0;
      q.pid[lane] = (int)pid;
      const int32_t* w = C.P.win + 6 * pid;
      if (lane < ppw && pid < C.P.n && w[0] >= 0) {
        const StructDev& S = C.B.s[C.B.patch_struct[pid]];
        const GridDev& g = S.g;
        const RaySet rs = make_ray_set(C.set, g);
        const double* src = C.P.f64 + (int64_t)NS_PATCH_F64 * pid;
        const double cf = __ldg(src + rs.fd), cl = __ldg(src + rs.ld), r = __ldg(src + kR);
        const int kind0 = C.P.i32[NS_PATCH_I32 * pid];
        const bool skin = ns_has_box(kind0);
        q.cf[lane] = cf;
        q.cl[lane] = cl;
        q.lo_fd[lane] = skin ? __ldg(src + NS_SKIN_LO + rs.fd) : cf - r;
        q.hi_fd[lane] = skin ? __ldg(src + NS_SKIN_HI + rs.fd) : cf + r;
        q.lo_ld[lane] = skin ? __ldg(src + NS_SKIN_LO + rs.ld) : cl - r;
        q.hi_ld[lane] = skin ? __ldg(src + NS_SKIN_HI + rs.ld) : cl + r;
        q.disc[lane] = (!skin || kind0 == NS_SKIN_POINT) ? 1 : 0;
        q.r2[lane] = r * r;
        q.mn_fd[lane] = g.mn[rs.fd];
        q.mn_ld[lane] = g.mn[rs.ld];
        q.side[lane] = g.side;
        q.delta[lane] = rs.delta;
        q.nb[lane] = rs.nb;
        q.rbase[lane] = S.ray_base[C.set];
        q.m0[lane] = w[rs.fd];
        q.m1[lane] = w[3 + rs.fd];
        q.n0[lane] = w[rs.ld];
        const int h = w[3 + rs.ld] - w[rs.ld] + 1;
        H = (w[3 + rs.fd] >= w[rs.fd] && h > 0) ? h : 0;
        const int kind = C.P.i32[NS_PATCH_I32 * pid];
        q.ty[lane] = (kind == NS_EDGE_REG || kind == NS_EDGE_SING) ? 1 : 0;  // skin, triangles: sphere list
      }
      q.gfirst[lane] = 0;
      q.gend[lane] = 0;
    }
    // the batch's pixel rows, patch after patch, are processed 32 at a time
    int hincl = H;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, hincl, o);
      if (lane >= o) hincl += v;
    }
    const int hexcl = hincl - H;
    const int R = __shfl_sync(0xffffffffu, hincl, 31);
    __syncwarp();
    if (R == 0) continue;
    // 2. candidate counts: G = running exclusive prefix of the row counts in batch order; the
    //    lanes holding a patch's first and last rows record G there
    int64_t running = 0;
    for (int rb = 0; rb < R; rb += 32) {
      const int k = rb + lane;
      const int kk = k < R ? k : R - 1;
      const int p = owner_lane(hincl, kk);
      const int row = kk - __shfl_sync(0xffffffffu, hexcl, p);
      const int hp = __shfl_sync(0xffffffffu, H, p);
      int a, cnt = 0;
      if (k < R) {
        cnt = cand_row(q, p, row, &a);
        const int rel = a - q.m0[p];
        if (k < kCandRows) rows[k] = (cnt == 0) ? 0u : ((rel | cnt) >> 16 ? kCandRowAgain : (uint32_t)(rel << 16 | cnt));
      }
      int cincl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, cincl, o);
        if (lane >= o) cincl += v;
      }
      if (k < R && row == 0) q.gfirst[p] = running + (cincl - cnt);
      if (k < R && row == hp - 1) q.gend[p] = running + cincl;
      running += __shfl_sync(0xffffffffu, cincl, 31);
    }
    __syncwarp();
    const int my_total = H > 0 ? (int)(q.gend[lane] - q.gfirst[lane]) : 0;
    // 3. one atomic per candidate list for the whole batch
    const int my_ty = q.ty[lane];
    int inc0 = my_ty == 0 ? my_total : 0, inc1 = my_ty == 1 ? my_total : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v0 = __shfl_up_sync(0xffffffffu, inc0, o), v1 = __shfl_up_sync(0xffffffffu, inc1, o);
      if (lane >= o) {
        inc0 += v0;
        inc1 += v1;
      }
    }
    const int sum0 = __shfl_sync(0xffffffffu, inc0, 31), sum1 = __shfl_sync(0xffffffffu, inc1, 31);
    unsigned long long b0 = 0, b1 = 0;
    if (lane == 0 && sum0) b0 = atomicAdd(co.count + 0, (unsigned long long)sum0);
    if (lane == 0 && sum1) b1 = atomicAdd(co.count + 1, (unsigned long long)sum1);
    b0 = __shfl_sync(0xffffffffu, b0, 0);
    b1 = __shfl_sync(0xffffffffu, b1, 0);
    if ((int64_t)(b0 + sum0) > co.cap || (int64_t)(b1 + sum1) > co.tor_cap) {
      if (lane == 0) atomicExch(C.out.error_flag, 6);
      __syncwarp();
      continue;
    }
    // a row's candidate j sits at base[p] + G(row) + j in its patch's list
    const int64_t my_slot = my_ty == 0 ? (int64_t)b0 + (inc0 - my_total) : (int64_t)b1 + (inc1 - my_total);
    q.base[lane] = my_slot - q.gfirst[lane];
    __syncwarp();
    // 4. the candidates, rows in batch order, stores coalesced
    running = 0;
    for (int rb = 0; rb < R; rb += 32) {
      const int k = rb + lane;
      const int kk = k < R ? k : R - 1;
      const int p = owner_lane(hincl, kk);
      const int row = kk - __shfl_sync(0xffffffffu, hexcl, p);
      int a = 0, cnt = 0;
      if (k < R) {
        const uint32_t kept = k < kCandRows ? rows[k] : kCandRowAgain;
        if (kept == kCandRowAgain) {
          cnt = cand_row(q, p, row, &a);
        } else {
          a = q.m0[p] + (int)(kept >> 16);
          cnt = (int)(kept & 0xffffu);
        }
      }
      int cincl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, cincl, o);
        if (lane >= o) cincl += v;
      }
      const int T = __shfl_sync(0xffffffffu, cincl, 31);
      const int cexcl = cincl - cnt;
      for (int kb = 0; kb < T; kb += 32) {
        const int j = kb + lane;
        const int jj = j < T ? j : T - 1;
        const int rr = owner_lane(cincl, jj);
        const int pr = __shfl_sync(0xffffffffu, p, rr), rowr = __shfl_sync(0xffffffffu, row, rr);
        const int ar = __shfl_sync(0xffffffffu, a, rr), er = __shfl_sync(0xffffffffu, cexcl, rr);
        if (j < T) {
          const int m = ar + (j - er);
          const int64_t n = q.n0[pr] + rowr;
          int2* dst = q.ty[pr] ? co.tor : co.sph;
          dst[q.base[pr] + running + j] = make_int2((int)(q.rbase[pr] + n * q.nb[pr] + m), q.pid[pr]);
        }
      }
      running += T;
    }
    __syncwarp();
  }
}

// The torus candidates that may hit (torus_screen.h), in a list of their own, so that the quartic
// solve runs on full warps of them.  A block takes tiles of 1,024 candidates, four per thread, keeps
// their order within the tile (a patch's candidates stay together) and reserves their places with
// one atomic.  Torus stage of a ray set, all candidates -> screen + solve: 64 conformers (11 M
// candidates, mixed) 1,170 -> 135 + 165 us, 20,000 atoms (FP64) 106 -> 15 + 18 us, 2,000 atoms
// 18 -> 4 + 5 us.  Six blocks per SM (40 registers): 540 us for the conformers' four sets, 661 with
// the 64 registers it takes by itself.
constexpr int kScreenThreads = 256, kScreenItems = 4, kScreenTile = kScreenThreads * kScreenItems;
template <int PN>
__device__ __forceinline__ void torus_screen_body(const TraceCtx& C, const CandOut& co) {
  constexpr int fd = Ax<PN>::fd, ld = Ax<PN>::ld, vc = Ax<PN>::vc;
  __shared__ int s_cnt[kScreenItems * (kScreenThreads / 32)];
  __shared__ unsigned long long s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t ncand = co.count[1];
  const int64_t nlim = ncand < co.tor_cap ? ncand : co.tor_cap;
  for (int64_t tile = blockIdx.x * (int64_t)kScreenTile; tile < nlim; tile += (int64_t)gridDim.x * kScreenTile) {
    int2 e[kScreenItems];
    unsigned kept[kScreenItems];
#pragma unroll
    for (int q = 0; q < kScreenItems; q++) {
      const int64_t c = tile + q * kScreenThreads + threadIdx.x;
      e[q] = c < nlim ? co.tor[c] : make_int2(0, -1);
    }
    // the rays' offsets first, so that the loads of the four candidates overlap
    float u[kScreenItems], v[kScreenItems];
#pragma unroll
    for (int q = 0; q < kScreenItems; q++) {
      const int64_t pid = e[q].y >= 0 ? e[q].y : 0;
      const StructDev& S = C.B.s[C.B.n > 1 ? C.B.patch_struct[pid] : 0];
      const GridDev& g = S.g;
      const double delta = ray_set_shifted(C.set) ? NS_DELTA - g.hside : 0.0;
      const unsigned nb = (unsigned)g.n[fd], lr = (unsigned)(e[q].x - S.ray_base[C.set]);
      const unsigned n = lr / nb, m = lr - n * nb;
      const double* f = C.P.f64 + (int64_t)NS_PATCH_F64 * pid;
      u[q] = (float)((gcoord(g, fd, m) + delta) - __ldg(f + fd));
      v[q] = (float)((gcoord(g, ld, n) + delta) - __ldg(f + ld));
    }
#pragma unroll
    for (int q = 0; q < kScreenItems; q++) {
      bool keep = false;
      if (e[q].y >= 0) {
        const int64_t pid = e[q].y;
        float rec[kTorusScreen];
        const float4* src = C.P.screen + (kTorusScreen / 4) * pid;
#pragma unroll
        for (int k = 0; k < kTorusScreen / 4; k++) {
          const float4 x = __ldg(src + k);
          rec[4 * k] = x.x; rec[4 * k + 1] = x.y; rec[4 * k + 2] = x.z; rec[4 * k + 3] = x.w;
        }
        keep = torus_may_hit<fd, ld, vc>(rec, u[q], v[q]);
      }
      kept[q] = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) s_cnt[q * (kScreenThreads / 32) + warp] = __popc(kept[q]);
    }
    __syncthreads();
    if (warp == 0) {
      const int v = s_cnt[lane];  // 4 x 8 counts, in candidate order
      const int incl = warp_incl(v);
      if (lane == 31) s_base = incl ? atomicAdd(co.scr_count, (unsigned long long)incl) : 0;
      s_cnt[lane] = incl - v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kScreenItems; q++)
      if ((kept[q] >> lane) & 1u) {
        const unsigned long long slot = s_base + s_cnt[q * (kScreenThreads / 32) + warp] + __popc(kept[q] & ((1u << lane) - 1u));
        if ((int64_t)slot < co.tor_cap) co.scr[slot] = e[q];
        else atomicExch(C.out.error_flag, 6);
      }
    __syncthreads();
  }
}
static_assert(kScreenItems * (kScreenThreads / 32) == 32, "one warp scans the tile's counts");

__global__ void __launch_bounds__(kScreenThreads, 6) k_torus_screen(const __grid_constant__ TraceSets T) {
  const int y = blockIdx.y;
  if (!T.co[y].scr) return;
  const TraceCtx C{T.P, T.B, T.set[y], T.out[y]};
  per_panel(C.set, [&](auto pn) { torus_screen_body<decltype(pn)::value>(C, T.co[y]); });
}

// Intersection launches of all sets of a group; the grids are sized for `area` candidates a set at
// most, so that a small input does not launch thousands of empty blocks.
void launch_isect(const TraceSets& T, int precision, const TuneParams& tp, int64_t area, cudaStream_t s,
                  int64_t* launches) {
  const bool ses = T.P.kind_mask & kSesKinds, box = T.P.kind_mask & kBoxKinds;
  const auto blocks = [&](int64_t most, int64_t per) {
    const int64_t b = (area + per - 1) / per;
    return dim3((unsigned)(b < 1 ? 1 : (b < most ? b : most)), (unsigned)T.n);
  };
  const int it = tp.isect_threads;
  const dim3 grid = blocks((int64_t)sm_count() * tp.isect_bpsm, it);
  bool screen = false;
  for (int q = 0; q < T.n; q++) screen = screen || T.co[q].scr;
  if (ses && screen) {
    k_torus_screen<<<blocks((int64_t)sm_count() * 8, kScreenTile), kScreenThreads, 0, s>>>(T);
    ++*launches;
  }
  if (precision == 1) {
    // the deferred candidates follow, in double precision (few: a small grid)
    const dim3 few = blocks(sm_count(), 256);
    if (ses) {
      launch_isect_mixed_sphere(T, grid, it, s);
      launch_isect_mixed_torus(T, grid, it, s);
      k_isect<false, true><<<few, 256, 0, s>>>(T);
      k_isect<true, true><<<few, 256, 0, s>>>(T);
      *launches += 4;
    }
    if (box) {
      launch_isect_quad_mixed(T, grid, it, s);
      k_isect_quad<true><<<few, 256, 0, s>>>(T);
      *launches += 2;
    }
  } else {
    if (ses) {
      k_isect<false, false><<<grid, it, 0, s>>>(T);
      k_isect<true, false><<<grid, it, 0, s>>>(T);
      *launches += 2;
    }
    if (box) {
      k_isect_quad<false><<<grid, it, 0, s>>>(T);
      ++*launches;
    }
  }
}

// rintp of a node position as an int (positions outside the range of int saturate, which the clamps
// to the grid and to the bit array make the same): one conversion instead of a 64-bit one.
__device__ __forceinline__ int node_pos(double x) { return __double2int_rd(x + 0.5); }

// Transposes the 32 x 32 bits of a warp: lane l's bit b becomes lane b's bit l (five exchanges of
// half blocks, against 32 ballots).
__device__ __forceinline__ unsigned transpose_bits(unsigned x) {
  const int lane = threadIdx.x & 31;
  unsigned m = 0x0000ffffu;  // positions whose bit j is clear
#pragma unroll
  for (int j = 16; j; j >>= 1) {
    const unsigned y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
    m ^= m << (j >> 1);
  }
  return x;
}

// One CTA per 32x4 ray tile: loads, sorts and pairs the hits of its rays and performs the
// interval fill (status runs, insideness bits, pair store, volume).
// kGrad: the hits carry their patches (sorted along), and every interval end adds its term of
// d volume / d patch parameters; the stored pairs keep their patches for the area adjoint.
template <bool kGrad>
__global__ void __launch_bounds__(kTraceThreads, 6) k_fill(const __grid_constant__ TraceSets T) {
  constexpr int kThreads = kTraceThreads;
  const int64_t tile = blockIdx.x;
  if (tile >= T.ntiles[blockIdx.y]) return;
  const TraceCtx C{T.P, T.B, T.set[blockIdx.y], T.out[blockIdx.y]};
  const HitStore& hs = T.hs[blockIdx.y];
  const int panel = ray_set_panel(C.set);
  const StructDev& S = C.B.s[find_struct(C.B.tile_base[panel], C.B.n, tile)];
  const GridDev g = S.g;
  const RaySet rs = make_ray_set(C.set, g);
  uint32_t* const bits = C.out.bits + S.word_base;
  const int64_t nwords = S.nwords;
  __shared__ double s_hit[kHitCap * kThreads];
  // gradient mode: each hit's slot in the hit store (its patch is read from there when needed),
  // one byte per hit to keep the shared-memory footprint and so the occupancy up
  __shared__ uint8_t s_slot[kGrad ? kHitCap * kThreads : 1];
  const int64_t ntm = (rs.nb + kTileM - 1) / kTileM;
  const int64_t lt = tile - S.tile_base[panel];
  const int64_t tm = lt % ntm, tn = lt / ntm;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t m = tm * kTileM + lane;
  const int64_t n = tn * kTileN + warp;
  const bool valid = (m < rs.nb) && (n < rs.na);
  const int tid = threadIdx.x;
  double* col = s_hit + tid;
  const int64_t lrid = n * rs.nb + m;
  const int64_t rid = S.ray_base[C.set] + lrid;
  int hc = valid ? hs.cnt[rid] : 0;
  const bool mc = ray_set_shifted(rs.set);
  if (!__any_sync(0xffffffffu, hc > 0)) {
    // rays beside the molecule (half of a globule's grid): empty rows
    if (valid) {
      C.out.vol_ray[rid] = 0.0;
      if (mc) C.out.ray_pair_cnt[S.mc_base + rs.ordinal_base + lrid] = 0;
      else if (rs.set == 0) C.out.srun_cnt[rid] = 0;
      if (C.out.hits) {
        C.out.ray_hit_off[rid] = 0;
        C.out.ray_hit_cnt[rid] = 0;
      }
    }
    return;
  }
  bool ovf = hc > kHitCap;
  int nh = ovf ? 0 : hc;
  uint8_t* pcol = kGrad ? s_slot + tid : nullptr;
  for (int i = 0; i < nh; i++) col[i * kThreads] = hs.t[(int64_t)i * hs.nrays + rid];
  if (kGrad)
    for (int i = 0; i < nh; i++) pcol[i * kThreads] = (uint8_t)i;
  for (int i = 1; i < nh; i++) {
    double v = col[i * kThreads];
    uint8_t pv = kGrad ? pcol[i * kThreads] : 0;
    int j = i;
    while (j > 0 && col[(j - 1) * kThreads] > v) {
      col[j * kThreads] = col[(j - 1) * kThreads];
      if (kGrad) pcol[j * kThreads] = pcol[(j - 1) * kThreads];
      j--;
    }
    col[j * kThreads] = v;
    if (kGrad) pcol[j * kThreads] = pv;
  }
  if (valid && ovf) {
    int slot = atomicAdd(C.out.ovf_count, 1);
    if (slot < C.out.ovf_cap) C.out.ovf_rays[slot] = (int32_t)rid;
    else atomicExch(C.out.error_flag, 1);
  }
  if (valid && !ovf && C.out.hits) {
    unsigned long long off = atomicAdd(C.out.hit_cursor, (unsigned long long)nh);
    if ((int64_t)(off + nh) <= C.out.hit_cap) {
      for (int i = 0; i < nh; i++) C.out.hits[off + i] = col[i * kThreads];
      C.out.ray_hit_off[rid] = (int64_t)off;
      C.out.ray_hit_cnt[rid] = nh;
    } else {
      atomicExch(C.out.error_flag, 2);
    }
  }
  // interval ends
  double pa_vc, dirl;
  if (rs.set == 0) {
    pa_vc = gcoord(g, 0, 0);
    dirl = gcoord(g, 0, g.n[0] - 1) - pa_vc;
  } else {
    pa_vc = gcoord(g, rs.vc, 0) + rs.delta;
    double pb = gcoord(g, rs.vc, g.n[rs.vc] - 1) + rs.delta;
    dirl = pb - pa_vc;
  }
  double vol = 0.0;
  int np = 0;
  const auto slot_pid = [&](uint8_t sl) { return hs.pid[(int64_t)sl * hs.nrays + rid]; };
  if (kGrad && C.out.gvol) {
    // d volume / d patch parameters, interval end by interval end (the pairing rule of
    // make_pairs), summed over runs of lanes on the same patch before the atomics
    const double W = S.A * C.out.grad_scale;
    __syncwarp();  // the lanes read each other's sorted hit columns below
    const int nhw = (valid && !ovf && nh > 0 && (nh & 1) == 0) ? nh : 0;
    const int maxn = (int)__reduce_max_sync(0xffffffffu, (unsigned)nhw);
    // The warp's interval ends, 32 at a time: end q of every ray that has one (level q), levels in
    // order, so that neighbouring lanes hold neighbouring rays (which mostly hit the same patch).
    // Lane q keeps the ray mask of level q.
    unsigned lvl_mask = 0;
    for (int q = 0; q < maxn; q++) {
      const unsigned mq = __ballot_sync(0xffffffffu, nhw > q);
      if (lane == q) lvl_mask = mq;
    }
    const int lvl_size = __popc(lvl_mask);
    int lincl = lvl_size;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, lincl, o);
      if (lane >= o) lincl += v;
    }
    const int nends = __shfl_sync(0xffffffffu, lincl, 31);
    for (int kb = 0; kb < nends; kb += 32) {
      const int k = kb + lane;
      const int kk = k < nends ? k : nends - 1;
      int q = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        const int x = __shfl_sync(0xffffffffu, lincl, q + step - 1);
        if (x <= kk) q += step;
      }
      const int idx = kk - __shfl_sync(0xffffffffu, lincl - lvl_size, q);
      unsigned mq = __shfl_sync(0xffffffffu, lvl_mask, q);
      for (int c2 = 0; c2 < idx; c2++) mq &= mq - 1;
      const int r = __ffs(mq) - 1;  // the ray (lane) of this end
      const int64_t rid_r = __shfl_sync(0xffffffffu, rid, r);
      double gk[NS_GRAD_PER_PATCH];
      int32_t pid = -1;
      if (k < nends) {
        const double* cr = s_hit + warp * 32 + r;
        const double t1 = cr[(q & ~1) * kThreads], t2 = cr[(q | 1) * kThreads];
        if (fabs(t2 - t1) >= NS_EPS_INT) {
          const uint8_t sl = s_slot[(q * kThreads) + warp * 32 + r];
          pid = hs.pid[(int64_t)sl * hs.nrays + rid_r];
          double x[3];
          x[rs.fd] = gcoord(g, rs.fd, tm * kTileM + r) + rs.delta;
          x[rs.ld] = gcoord(g, rs.ld, n) + rs.delta;
          x[rs.vc] = pa_vc + dirl * ((q & 1) ? t2 : t1);
          if (hit_grad(C.P.f64 + (int64_t)NS_PATCH_F64 * pid, C.P.i32[NS_PATCH_I32 * pid], C.P.probe, x, rs.vc, gk)) {
            const double w = (q & 1) ? W : -W;
#pragma unroll
            for (int c3 = 0; c3 < NS_GRAD_PER_PATCH; c3++) gk[c3] *= w;
          } else {
            pid = -1;
          }
        }
      }
      if (pid < 0)
#pragma unroll
        for (int c3 = 0; c3 < NS_GRAD_PER_PATCH; c3++) gk[c3] = 0.0;
      warp_add_grad(pid, gk, C.out.gvol);
    }
  }
  if (kGrad) {
    // the hits' patches follow their pairs (gradients, analytic normals)
    if (valid && !ovf)
      np = make_pairs(col, kThreads, nh, pa_vc, dirl, g.mn[rs.vc], g.scale, mc, &vol, pcol, (GradCtx*)nullptr,
                      slot_pid);
  } else {
    if (valid && !ovf) np = make_pairs(col, kThreads, nh, pa_vc, dirl, g.mn[rs.vc], g.scale, mc, &vol);
  }
  if (valid && !ovf) C.out.vol_ray[rid] = vol;
  __syncwarp();
  const int64_t NX = g.n[0], NY = g.n[1];
  if (rs.set >= 4) {
    // epsilon-map node rays of panels 1 and 2
    if (valid && !ovf && C.out.epsmap)
      for (int q = 0; q < np; q++)
        eps_fill(g, rs, m, n, col[(2 * q) * kThreads], col[(2 * q + 1) * kThreads], C.out.epsmap, C.out.eps_inside);
    return;
  }
  if (!mc) {
    // status row (., j = m, k = n): runs of inside nodes
    int nr = 0;
    if (valid && !ovf)
      for (int q = 0; q < np; q++) {
        if (C.out.epsmap)
          eps_fill(g, rs, m, n, col[(2 * q) * kThreads], col[(2 * q + 1) * kThreads], C.out.epsmap, C.out.eps_inside);
        int64_t ia, ib;
        status_node_range(g, col[(2 * q) * kThreads], col[(2 * q + 1) * kThreads], &ia, &ib);
        if (ia > ib) continue;
        col[(2 * nr) * kThreads] = (double)ia;
        col[(2 * nr + 1) * kThreads] = (double)ib;
        nr++;
      }
    int64_t off = warp_append(C.out.srun_cursor, C.out.srun_cap, nr, C.out.error_flag, 5);
    if (valid && !ovf) {
      if (off >= 0) {
        for (int q = 0; q < nr; q++)
          C.out.sruns[off + q] = make_int2((int)col[(2 * q) * kThreads], (int)col[(2 * q + 1) * kThreads]);
        C.out.srun_off[rid] = off;
        C.out.srun_cnt[rid] = nr;
      } else {
        C.out.srun_cnt[rid] = 0;
      }
    }
    return;
  }
  // accurate-triangulation rays: pair store for the vertex assembly; in the ray's column the node
  // positions a < v <= b that a pair covers take the place of its ends
  const double vmin = g.mn[rs.vc];
  const auto set_span = [&](int q, int a, int b) { col[(2 * q) * kThreads] = __hiloint2double(b, a); };
  const auto span = [&](int q) {
    const double w = col[(2 * q) * kThreads];
    return make_int2(__double2loint(w), __double2hiint(w));
  };
  {
    int64_t off = warp_append(C.out.pair_cursor, C.out.pair_cap, np, C.out.error_flag, 3);
    if (valid && !ovf) {
      int64_t ord = S.mc_base + rs.ordinal_base + lrid;
      for (int q = 0; q < np; q++) {
        const double lim1 = col[(2 * q) * kThreads], lim2 = col[(2 * q + 1) * kThreads];
        if (off >= 0) {
          reinterpret_cast<double2*>(C.out.pairs)[off + q] = make_double2(lim1, lim2);
          if (kGrad)
            C.out.pair_pid[off + q] = make_int2(slot_pid(pcol[(2 * q) * kThreads]), slot_pid(pcol[(2 * q + 1) * kThreads]));
        }
        set_span(q, node_pos((lim1 - vmin) * g.scale), node_pos((lim2 - vmin) * g.scale));
      }
      if (off >= 0) {
        C.out.ray_pair_off[ord] = off;
        C.out.ray_pair_cnt[ord] = np;
      } else {
        C.out.ray_pair_cnt[ord] = 0;
      }
    }
  }
  if (rs.panel == 0) {
    // row bits (i, j = m, k = n), i in (a, b]: every lane clears the runs of its own row
    if (valid && !ovf) {
      const int64_t f0 = (n * NY + m) * NX;
      const int64_t maxb = nwords * 32 - 1;
      for (int q = 0; q < np; q++) {
        const int2 ab = span(q);
        int64_t lo = f0 + ab.x + 1, hi = f0 + ab.y;
        if (lo < 0) lo = 0;
        if (hi > maxb) hi = maxb;
        for (int64_t w = lo >> 5; w <= (hi >> 5) && hi >= lo; w++) {
          const int64_t wl = w << 5;
          const int s0 = (int)(lo > wl ? lo - wl : 0);
          const int s1 = (int)(hi < wl + 31 ? hi - wl : 31);
          const uint32_t mask = (s1 - s0 == 31) ? 0xffffffffu : (((1u << (s1 - s0 + 1)) - 1u) << s0);
          atomicAnd(bits + w, ~mask);
        }
      }
    }
    return;
  }
  // panels 1 and 2: lanes are consecutive i; 32 positions along the ray axis at a time
  int vlo = INT_MAX, vhi = INT_MIN;
  if (np > 0) {
    const int a0 = span(0).x;
    vlo = a0 < INT_MAX ? a0 + 1 : a0;
    vhi = span(np - 1).y;
  }
  vlo = __reduce_min_sync(0xffffffffu, vlo);
  vhi = __reduce_max_sync(0xffffffffu, vhi);
  // far outside any grid; keeps the steps below from overflowing
  if (vlo < -(1 << 30)) vlo = -(1 << 30);
  if (vhi > (1 << 30)) vhi = 1 << 30;
  if (vlo > vhi) return;
  // every lane builds the 32-bit membership word of its ray over [v0, v0 + 31] from its intervals;
  // transposed, lane l holds the mask of the 32 rays at position v0 + l, and the lanes clear their
  // rows' bits in parallel
  int q = 0, qa = 0, qb = -1;
  if (np > 0) {
    const int2 ab = span(0);
    qa = ab.x;
    qb = ab.y;
  }
  const int64_t m0 = tm * kTileM;
  for (int v0 = vlo; v0 <= vhi; v0 += 32) {
    const int v1 = v0 + 31;
    unsigned mem = 0;
    while (q < np && qa < v1) {
      // positions qa < v <= qb of the current interval that fall in [v0, v1]
      const int lo = qa + 1 > v0 ? qa + 1 : v0, hi = qb < v1 ? qb : v1;
      if (lo <= hi) {
        const int s0 = lo - v0, s1 = hi - v0;
        mem |= (s1 - s0 == 31) ? 0xffffffffu : (((1u << (s1 - s0 + 1)) - 1u) << s0);
      }
      if (qb > v1) break;  // the interval continues in the next window
      q++;
      if (q < np) {
        const int2 ab = span(q);
        qa = ab.x;
        qb = ab.y;
      }
    }
    const unsigned mask = transpose_bits(mem);
    const int v = v0 + lane;
    if (mask && v <= vhi) {
      const int64_t f0 = (rs.panel == 1) ? (((int64_t)v * NY + n) * NX + m0) : ((n * NY + v) * NX + m0);
      if (f0 >= 0) {
        const int64_t w = f0 >> 5;
        const int sh = (int)(f0 & 31);
        if (w < nwords) atomicAnd(bits + w, ~(mask << sh));
        if (sh && w + 1 < nwords) atomicAnd(bits + w + 1, ~(mask >> (32 - sh)));
      }
    }
  }
}

// One thread per overflow ray: the same candidate tests with the hits kept in a global column.
__global__ void k_trace_overflow(const __grid_constant__ TraceSets T, const int64_t* __restrict__ tile_off,
                                 const int32_t* __restrict__ tile_list, int n_ovf, double* scratch, int32_t* pscratch) {
  const TraceCtx C{T.P, T.B, T.set[0], T.out[0]};
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_ovf) return;
  int64_t rid = C.out.ovf_rays[idx];
  const StructDev& S = C.B.s[find_struct(C.B.ray_base[C.set], C.B.n, rid)];
  const GridDev g = S.g;
  const RaySet rs = make_ray_set(C.set, g);
  uint32_t* const bits = C.out.bits + S.word_base;
  const int64_t nwords = S.nwords;
  const int64_t lrid = rid - S.ray_base[C.set];
  int64_t m = lrid % rs.nb, n = lrid / rs.nb;
  int64_t ntm = (rs.nb + kTileM - 1) / kTileM;
  int64_t tile = S.tile_base[rs.panel] + (n / kTileN) * ntm + m / kTileM;
  double* col = scratch + (int64_t)idx * kOverflowCap;
  int32_t* pcol = pscratch ? pscratch + (int64_t)idx * kOverflowCap : nullptr;
  double pa[3], dir[3] = {0., 0., 0.};
  pa[rs.fd] = gcoord(g, rs.fd, m) + rs.delta;
  pa[rs.ld] = gcoord(g, rs.ld, n) + rs.delta;
  pa[rs.vc] = gcoord(g, rs.vc, 0) + rs.delta;
  const double ray_dir = gcoord(g, rs.vc, g.n[rs.vc] - 1) - gcoord(g, rs.vc, 0);
  dir[rs.vc] = ray_dir;
  int nh = 0;
  for (int64_t e = tile_off[tile]; e < tile_off[tile + 1]; e++) {
    int64_t pid = tile_list[e];
    const int32_t* w = C.P.win + 6 * pid;
    if (m < w[rs.fd] || m > w[3 + rs.fd] || n < w[rs.ld] || n > w[3 + rs.ld]) continue;
    double f[NS_PATCH_F64];
    for (int k = 0; k < NS_PATCH_F64; k++) f[k] = C.P.f64[(int64_t)NS_PATCH_F64 * pid + k];
    const int32_t* ir = C.P.i32 + NS_PATCH_I32 * pid;
    double t[4];
    const double tri_dir = (gcoord(g, rs.vc, g.n[rs.vc] - 1) + rs.delta) - pa[rs.vc];
    int k = ray_patch_f64(f, ir[0], ir[1], ir[2], C.P, rs, pa, dir, ray_dir, S.box_dir[rs.vc], tri_dir, t);
    for (int i = 0; i < k; i++) {
      if (nh >= kOverflowCap) {
        atomicExch(C.out.error_flag, 4);
        return;
      }
      int pos = nh++;
      while (pos > 0 && col[pos - 1] > t[i]) {
        col[pos] = col[pos - 1];
        if (pcol) pcol[pos] = pcol[pos - 1];
        pos--;
      }
      col[pos] = t[i];
      if (pcol) pcol[pos] = (int32_t)pid;
    }
  }
  if (C.out.hits) {
    unsigned long long off = atomicAdd(C.out.hit_cursor, (unsigned long long)nh);
    if ((int64_t)(off + nh) <= C.out.hit_cap) {
      for (int i = 0; i < nh; i++) C.out.hits[off + i] = col[i];
      C.out.ray_hit_off[rid] = (int64_t)off;
      C.out.ray_hit_cnt[rid] = nh;
    } else {
      atomicExch(C.out.error_flag, 2);
    }
  }
  const bool mc = ray_set_shifted(rs.set);
  double pa_vc, dirl;
  if (rs.set == 0) {
    pa_vc = gcoord(g, 0, 0);
    dirl = gcoord(g, 0, g.n[0] - 1) - pa_vc;
  } else {
    pa_vc = gcoord(g, rs.vc, 0) + rs.delta;
    dirl = (gcoord(g, rs.vc, g.n[rs.vc] - 1) + rs.delta) - pa_vc;
  }
  double vol = 0.0;
  GradCtx gc;
  gc.f64 = C.P.f64;
  gc.i32 = C.P.i32;
  gc.probe = C.P.probe;
  gc.w = S.A * C.out.grad_scale;
  gc.x[rs.fd] = pa[rs.fd];
  gc.x[rs.ld] = pa[rs.ld];
  gc.x[rs.vc] = 0.0;
  gc.vc = rs.vc;
  gc.gvol = C.out.gvol;
  int np = make_pairs(col, 1, nh, pa_vc, dirl, g.mn[rs.vc], g.scale, mc, &vol, pcol, (pcol && gc.gvol) ? &gc : nullptr);
  C.out.vol_ray[rid] = vol;
  const int64_t NX = g.n[0], NY = g.n[1];
  if (rs.set >= 4) {
    if (C.out.epsmap)
      for (int q = 0; q < np; q++) eps_fill(g, rs, m, n, col[2 * q], col[2 * q + 1], C.out.epsmap, C.out.eps_inside);
    return;
  }
  if (!mc) {
    int nr = 0;
    for (int q = 0; q < np; q++) {
      if (C.out.epsmap) eps_fill(g, rs, m, n, col[2 * q], col[2 * q + 1], C.out.epsmap, C.out.eps_inside);
      int64_t ia, ib;
      status_node_range(g, col[2 * q], col[2 * q + 1], &ia, &ib);
      if (ia > ib) continue;
      col[2 * nr] = (double)ia;
      col[2 * nr + 1] = (double)ib;
      nr++;
    }
    unsigned long long off = nr ? atomicAdd(C.out.srun_cursor, (unsigned long long)nr) : 0;
    if ((int64_t)off + nr <= C.out.srun_cap) {
      for (int q = 0; q < nr; q++) C.out.sruns[off + q] = make_int2((int)col[2 * q], (int)col[2 * q + 1]);
      C.out.srun_off[rid] = (int64_t)off;
      C.out.srun_cnt[rid] = nr;
    } else {
      C.out.srun_cnt[rid] = 0;
      atomicExch(C.out.error_flag, 5);
    }
    return;
  }
  int64_t ord = S.mc_base + rs.ordinal_base + lrid;
  unsigned long long off = np ? atomicAdd(C.out.pair_cursor, (unsigned long long)np) : 0;
  if ((int64_t)off + np <= C.out.pair_cap) {
    for (int q = 0; q < np; q++) {
      C.out.pairs[2 * (off + q)] = col[2 * q];
      C.out.pairs[2 * (off + q) + 1] = col[2 * q + 1];
      if (pcol) C.out.pair_pid[off + q] = make_int2(pcol[2 * q], pcol[2 * q + 1]);
    }
    C.out.ray_pair_off[ord] = (int64_t)off;
    C.out.ray_pair_cnt[ord] = np;
  } else {
    C.out.ray_pair_cnt[ord] = 0;
    atomicExch(C.out.error_flag, 3);
  }
  const double vmin = g.mn[rs.vc];
  for (int q = 0; q < np; q++) {
    int64_t a = (int64_t)rintp((col[2 * q] - vmin) * g.scale);
    int64_t b = (int64_t)rintp((col[2 * q + 1] - vmin) * g.scale);
    if (rs.panel == 0) {
      int64_t f0 = (n * NY + m) * NX;
      clear_bits_range(bits, nwords, f0 + a + 1, f0 + b);
    } else {
      for (int64_t v = a + 1; v <= b; v++) {
        int64_t f = (rs.panel == 1) ? ((v * NY + n) * NX + m) : ((n * NY + v) * NX + m);
        clear_bits_range(bits, nwords, f, f);
      }
    }
  }
}

}  // namespace

cudaError_t launch_windows(const PatchDev& P, int32_t* win, float4* screen, const BatchDev& B,
                           unsigned long long* out, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  int64_t blocks = (P.n + kWinThreads - 1) / kWinThreads;
  if (blocks > (int64_t)sm_count() * 8) blocks = (int64_t)sm_count() * 8;
  k_windows<<<(unsigned)blocks, kWinThreads, 0, s>>>(P, win, screen, B, out);
  return cudaGetLastError();
}

cudaError_t launch_pool32(const PatchDev& P, float4* pool32, float4* quad32, double4* quadl, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  k_pool32<<<(unsigned)((P.n + 255) / 256), 256, 0, s>>>(P, pool32, quad32, quadl);
  return cudaGetLastError();
}

cudaError_t launch_bin_count(const PatchDev& P, const BatchDev& B, int set, int32_t* tile_cnt, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  k_bin<<<(unsigned)((P.n + 255) / 256), 256, 0, s>>>(P, B, set, tile_cnt, nullptr, nullptr, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_bin_fill(const PatchDev& P, const BatchDev& B, int set, const int64_t* tile_off,
                            int32_t* tile_cursor, int32_t* tile_list, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  k_bin<<<(unsigned)((P.n + 255) / 256), 256, 0, s>>>(P, B, set, nullptr, tile_off, tile_cursor, tile_list);
  return cudaGetLastError();
}

cudaError_t launch_trace(const TraceSets& T, int precision, const TuneParams& tp, int64_t area, cudaStream_t s,
                         int64_t* launches, cudaEvent_t* ev) {
  int64_t ntiles = 0;
  bool pids = false;
  for (int q = 0; q < T.n; q++) {
    ntiles = T.ntiles[q] > ntiles ? T.ntiles[q] : ntiles;
    pids = pids || T.hs[q].pid;
  }
  if (T.n <= 0 || ntiles <= 0) return cudaSuccess;
  if (ev) cudaEventRecord(ev[0], s);
  if (T.P.n > 0) {
    const int wpb = tp.cand_threads / 32;
    // patches per warp: 32 where the set gives 64 warps per SM (a full SM) that way, fewer below,
    // but no fewer than 4, whose rows fill the 32 lanes (skin, 97,000 patches: 238 us with 32, 213
    // with 16 warps per SM as the line, 172 with 64)
    const int64_t per = T.P.n / ((int64_t)sm_count() * 64);
    const int ppw = per < 4 ? 4 : (per > 32 ? 32 : (int)per);
    int64_t blocks = (T.P.n + ppw * wpb - 1) / (ppw * wpb);
    if (blocks > (int64_t)sm_count() * 64) blocks = (int64_t)sm_count() * 64;
    k_cand<<<dim3((unsigned)blocks, (unsigned)T.n), tp.cand_threads, 0, s>>>(T, ppw);
    ++*launches;
  }
  if (ev) cudaEventRecord(ev[1], s);
  launch_isect(T, precision, tp, area, s, launches);
  if (ev) cudaEventRecord(ev[2], s);
  const dim3 grid((unsigned)ntiles, (unsigned)T.n);
  if (pids) k_fill<true><<<grid, kTraceThreads, 0, s>>>(T);
  else k_fill<false><<<grid, kTraceThreads, 0, s>>>(T);
  ++*launches;
  if (ev) cudaEventRecord(ev[3], s);
  return cudaGetLastError();
}

cudaError_t launch_trace_overflow(const TraceSets& T, const int64_t* tile_off, const int32_t* tile_list, int n_ovf,
                                  double* scratch, int32_t* pscratch, cudaStream_t s) {
  if (n_ovf <= 0) return cudaSuccess;
  k_trace_overflow<<<(n_ovf + 63) / 64, 64, 0, s>>>(T, tile_off, tile_list, n_ovf, scratch, pscratch);
  return cudaGetLastError();
}

}  // namespace nsg
