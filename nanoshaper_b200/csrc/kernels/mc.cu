// Vertex assembly and marching cubes of the SES grid ray caster.
//
// Vertices: every vertex-producing pair of an accurate-triangulation ray yields two analytic
// vertices on the grid edges that contain the interval ends; a vertex is dropped when the two
// end nodes of its edge have the same final insideness, and the first vertex of an edge wins
// (assembleVerticesList src/Surface.cpp:7415-7667).  Vertices keep the reference order: panel 0
// rays (z-major), panel 1 rays (y-major), panel 2 rays (z-major), pairs in ray order.
//
// Marching cubes: cubes (i,j,k) in [1, N-2]^3 are classified from the 8 insideness bits; the
// classification writes the active cubes in (k, j, i) order and, per 32 cubes of a row, their
// active bits and the index of the first (the active-cube map, 8 bytes per 32 cubes, from which
// the active index of any active cube follows).  Every active cube has 12 vertex slots (cube_vl).
// The push pass (k_mc_push) writes each vertex that is the first of its grid edge into the slots
// of the (up to four) cubes that share the edge: a ray's vertices are sorted along it, so the
// vertices of an edge have consecutive ids, the first of them is the one whose predecessor has
// another edge key, and a slot is written once, with a plain store (the slots start at -1: they
// are cleared and filled structure chunk by structure chunk, so that a chunk's slots stay in L2
// between the two, or, where all of them fit a tenth of L2, cleared by the classification).  Active cubes add an edge-midpoint vertex to their own edges 5, 6, 10
// that carry no analytic vertex, in (k, j, i, edge) order, appended after the analytic ones
// (getVertices :8002-8327), and write it into the slots in the same way.  The triangle pass emits
// the case-table triangles with reversed winding and sums their areas (the reference sums Heron
// areas; here |cross product| / 2, the same quantity) (triangulationKernel :9075-9318,
// getTriangles :14559-14780).  Triangles with an edge without a vertex are skipped, as the
// reference does.
#include "grad.cuh"
#include "lookback.cuh"
#include "mc.h"
#include "mc_tables.cuh"

namespace nsg {

namespace {

// Node coordinate, and the grid edge a point on a ray along axis d lies on: the nearest node after
// the half-side shift, floor((p - min) * scale + 0.5).  Each operation is rounded on its own (the
// file is built without contraction), so every kernel here that places or finds a vertex gets the
// same doubles.
__device__ __forceinline__ double gcoord(const GridDev& g, int d, int64_t i) { return g.mn[d] + (double)i * g.side; }
__device__ __forceinline__ int64_t edge_index(const GridDev& g, int d, double p) {
  return (int64_t)floor((p - g.mn[d]) * g.scale + 0.5);
}

__device__ __forceinline__ int rbit(const uint32_t* __restrict__ bits, int64_t nwords, int64_t f) {
  if (f < 0 || (f >> 5) >= nwords) return 1;
  return (bits[f >> 5] >> (f & 31)) & 1;
}

struct RayId {
  int panel;
  int64_t m, n;
};

// Local ray ordinal r of a structure; a panel has fewer than 2^31 rays, so its divisions run in
// 32 bits.
__device__ __forceinline__ RayId ray_of(const GridDev& g, int64_t r) {
  const int64_t NX = g.n[0], NY = g.n[1], NZ = g.n[2];
  RayId id;
  const int64_t R0 = NZ * NY, R1 = NY * NX;
  unsigned w = (unsigned)NX, q;
  if (r < R0) { id.panel = 0; q = (unsigned)r; w = (unsigned)NY; }
  else if (r < R0 + R1) { id.panel = 1; q = (unsigned)(r - R0); }
  else { id.panel = 2; q = (unsigned)(r - R0 - R1); }
  const unsigned n = q / w;
  id.n = n;
  id.m = q - n * w;
  return id;
}

// Structure of ascending items of a batch: one search for the warp's first item, then a step per
// structure boundary, so that a pass over several items per lane searches once.
struct StructWalk {
  const int64_t* base;
  int n, b;
  int64_t next;  // first item of the structure after b
  __device__ __forceinline__ StructWalk(const int64_t* __restrict__ base_, int n_, int64_t warp_first)
      : base(base_), n(n_), b(0) {
    if (n > 1) b = find_struct(base, n, warp_first);
    next = base[b + 1];
  }
  __device__ __forceinline__ int at(int64_t x) {
    while (x >= next && b + 1 < n) next = base[++b + 1];
    return b;
  }
};

// Position of set bit k (from the lowest, k < popc(m)) of m.
__device__ __forceinline__ int nth_bit(unsigned m, int k) {
  int pos = 0;
#pragma unroll
  for (int step = 16; step; step >>= 1) {
    const int c = __popc(m & ((1u << step) - 1u));
    if (k >= c) {
      k -= c;
      m >>= step;
      pos += step;
    } else {
      m &= (1u << step) - 1u;
    }
  }
  return pos;
}

// Edge key (ix, iy, iz, dir) of the vertex at ray position index a.
__device__ __forceinline__ int4 edge_key(const RayId& id, int64_t a) {
  if (id.panel == 0) return make_int4((int)a, (int)id.m, (int)id.n, NS_X_DIR);
  if (id.panel == 1) return make_int4((int)id.m, (int)id.n, (int)a, NS_Z_DIR);
  return make_int4((int)id.m, (int)a, (int)id.n, NS_Y_DIR);
}

__device__ __forceinline__ bool keeps(const GridDev& g, const uint32_t* bits, int64_t nwords, int4 e) {
  const int64_t NX = g.n[0], NY = g.n[1];
  int64_t f = ((int64_t)e.z * NY + e.y) * NX + e.x;
  int64_t step = e.w == NS_X_DIR ? 1 : (e.w == NS_Y_DIR ? NX : NX * NY);
  return rbit(bits, nwords, f) != rbit(bits, nwords, f + step);
}

__device__ __forceinline__ int rec_struct(int w) { return (int)((unsigned)w >> 11); }

// vpid of an analytic vertex: its patch, and in bits 29-30 the axis of its ray (the gradient pass
// reads the axis from here rather than from the 16-byte edge key); -1 without a patch.
constexpr int kVpidAxisShift = 29;
constexpr int32_t kVpidPatchMask = (1 << kVpidAxisShift) - 1;
__device__ __forceinline__ int32_t vpid_pack(int32_t pid, int axis) {
  return pid < 0 ? -1 : (pid | (axis << kVpidAxisShift));
}

// Active index of the active cube (i, j, k) of structure S, from the active-cube map (a structure
// has fewer than 2^31 cubes, so the offsets within it fit 32 bits).
__device__ __forceinline__ int32_t active_index(const int2* __restrict__ amap, const StructDev& S, int i, int j,
                                                int k) {
  const int W = ((int)S.g.n[0] - 2 + 31) >> 5;
  const int b = i - 1;
  const int2 w = amap[S.aword_base + ((k - 1) * ((int)S.g.n[1] - 2) + (j - 1)) * W + (b >> 5)];
  return w.y + __popc((unsigned)w.x & ((1u << (b & 31)) - 1u));
}

// Writes vertex v into the slots of the active cubes (up to four, those inside the cube range)
// that share grid edge (axis, x, y, z).  An x edge at (x, y, z) is edge 0 of cube (x, y, z), 2 of
// (x, y-1, z), 4 of (x, y, z-1), 6 of (x, y-1, z-1); a y edge is 3 of (x, y, z), 1 of (x-1, y, z),
// 7 of (x, y, z-1), 5 of (x-1, y, z-1); a z edge 8 of (x, y, z), 9 of (x-1, y, z), 11 of
// (x, y-1, z), 10 of (x-1, y-1, z).  A cut edge's cubes are all active.
__device__ __forceinline__ void push_vertex(const int2* __restrict__ amap, int32_t* cube_vl, const StructDev& S,
                                            int axis, int x, int y, int z, int32_t v) {
  // per axis: the two offset axes of the four cubes and the slots of (0,0), (1,0), (0,1), (1,1)
  const int u = axis == NS_X_DIR ? 1 : 0, w = axis == NS_Z_DIR ? 1 : 2;
  const int s00 = axis == NS_X_DIR ? 0 : (axis == NS_Y_DIR ? 3 : 8);
  const int s10 = axis == NS_X_DIR ? 2 : (axis == NS_Y_DIR ? 1 : 9);
  const int s01 = axis == NS_X_DIR ? 4 : (axis == NS_Y_DIR ? 7 : 11);
  const int s11 = axis == NS_X_DIR ? 6 : (axis == NS_Y_DIR ? 5 : 10);
  const int nx = (int)S.g.n[0] - 2, ny = (int)S.g.n[1] - 2, nz = (int)S.g.n[2] - 2;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    int c[3] = {x, y, z};
    if (q & 1) c[u]--;
    if (q & 2) c[w]--;
    if (c[0] < 1 || c[1] < 1 || c[2] < 1 || c[0] > nx || c[1] > ny || c[2] > nz) continue;
    const int slot = q == 0 ? s00 : (q == 1 ? s10 : (q == 2 ? s01 : s11));
    cube_vl[12 * (int64_t)active_index(amap, S, c[0], c[1], c[2]) + slot] = v;
  }
}

constexpr int kPassThreads = 256;

// Whether the passes before left complete arrays: no look-back wait ran out and their items fit.  The
// passes that look back themselves ask through take_ticket_if.
__device__ __forceinline__ bool cubes_fit(const MCArgs& A) {
  return A.counts[kMcActive] <= A.cap_active && A.counts[kMcAnalytic] <= A.cap_vert;
}
__device__ __forceinline__ bool cubes_ok(const MCArgs& A) { return *A.lb_rows.err == 0 && cubes_fit(A); }

// Items (rays, map words, cubes) per thread of a one-pass kernel.  A block waits for the blocks
// before it about as long as it counts, so a large input wants tickets with more work: 4 items per
// thread where that leaves four blocks per SM, 8 (for the passes that have them) where it leaves 16;
// a small input is spread over more blocks.  Triangles of 64 conformers, 8.4 M cubes: 1,053 us
// with 1 item (and a 32-ticket look-back), 639 with 4, 579 with 8; of one 20,000-atom molecule,
// 1.1 M cubes: 123, 84, 90.  Vertices of the conformers: 520, 381, 462.
int pass_items(int64_t items, int most) {
  const int64_t per_sm = (int64_t)sm_count() * kPassThreads;
  if (most >= 8 && items >= per_sm * 8 * 16) return 8;
  return items >= per_sm * 4 * 4 ? 4 : 1;
}
constexpr int kVertItems = 4, kRowsItems = 8, kMidItems = 4, kTrisItems = 8;

// Vertices in one pass, one thread per ray, a ticket of consecutive rays per block (lookback.cuh): the
// thread keeps a mask of its pair ends whose edge is cut, the block places its vertices behind
// those of the tickets before it, and the warp writes them with a vertex per lane (coalesced; the
// surviving ends of a ray per lane leave half the lanes idle).  Latency-bound (bit and pair
// gathers).  Count pass, scan and write pass before -> this: 64 conformers (4.3 M rays, 8.4 M
// vertices) 466 + 30 -> 381 us; 20,000 atoms, where 1.2 M rays hold few hits, 64 + 8 -> 75 us and no
// host round trip between the passes.
template <int kItems>
__global__ void __launch_bounds__(kPassThreads) k_vert(VertArgs A) {
  __shared__ unsigned int s_ticket;
  const unsigned t = take_ticket(A.lb, &s_ticket);
  const int lane = threadIdx.x & 31;
  const int64_t r0 = (int64_t)t * (kPassThreads * kItems) + (threadIdx.x >> 5) * (32 * kItems) + lane;
  unsigned mask[kItems];  // kept ends among the first 32
  int cnt[kItems], sum = 0;
  const StructWalk start(A.B.mc_base, A.B.n, r0 - lane);
  StructWalk walk = start;
#pragma unroll
  for (int x = 0; x < kItems; x++) {
    const int64_t r = r0 + 32 * x;
    const bool valid = r < A.nrays;
    mask[x] = 0;
    cnt[x] = 0;
    const int b = walk.at(r);
    const int np = valid ? A.ray_pair_cnt[r] : 0;
    if (np > 0) {
      const StructDev& S = A.B.s[b];
      const RayId id = ray_of(S.g, r - S.mc_base);
      const int vc = id.panel == 0 ? 0 : (id.panel == 1 ? 2 : 1);
      const double* pr = A.pairs + 2 * A.ray_pair_off[r];
      for (int q = 0; q < 2 * np; q++)
        if (keeps(S.g, A.bits + S.word_base, S.nwords, edge_key(id, edge_index(S.g, vc, pr[q])))) {
          cnt[x]++;
          if (q < 32) mask[x] |= 1u << q;
        }
    }
    sum += cnt[x];
  }
  int64_t off = warp_offset<kPassThreads>(A.lb, t, warp_total(sum));
  if (off < 0) return;
  walk = start;
  const auto emit = [&](int b, const RayId& id, int64_t po, int q, int64_t o) {
    if (o >= A.cap) return;
    const GridDev& g = A.B.s[b].g;
    const double delta = NS_DELTA - g.hside;
    const int vc = id.panel == 0 ? 0 : (id.panel == 1 ? 2 : 1);
    const double x = A.pairs[2 * po + q];
    const int4 e = edge_key(id, edge_index(g, vc, x));
    double p0, p1, p2;
    if (id.panel == 0) { p0 = x; p1 = gcoord(g, 1, id.m) + delta; p2 = gcoord(g, 2, id.n) + delta; }
    else if (id.panel == 1) { p0 = gcoord(g, 0, id.m) + delta; p1 = gcoord(g, 1, id.n) + delta; p2 = x; }
    else { p0 = gcoord(g, 0, id.m) + delta; p1 = x; p2 = gcoord(g, 2, id.n) + delta; }
    A.vpos[3 * o + 0] = p0;
    A.vpos[3 * o + 1] = p1;
    A.vpos[3 * o + 2] = p2;
    A.vkey[o] = e;
    A.vstruct[o] = b;
    if (A.vpid) {
      const int2 pp = A.pair_pid[po + (q >> 1)];
      A.vpid[o] = vpid_pack((q & 1) ? pp.y : pp.x, e.w);
    }
  };
#pragma unroll 1
  for (int x = 0; x < kItems; x++) {
    const int64_t r = r0 + 32 * x;
    const bool valid = r < A.nrays;
    int c = cnt[0];
    unsigned m = mask[0];
#pragma unroll
    for (int y = 1; y < kItems; y++)
      if (x == y) { c = cnt[y]; m = mask[y]; }
    const int b = walk.at(r);
    const StructDev& S = A.B.s[b];
    const int incl = warp_incl(c);
    const int T = __shfl_sync(0xffffffffu, incl, 31);
    if (valid && r == S.mc_base) A.voff[b] = off + incl - c;
    if (r == A.nrays - 1) A.voff[A.B.n] = A.counts[kMcAnalytic] = off + incl;
    if (T == 0) continue;
    RayId id{0, 0, 0};
    int64_t po = 0;
    if (c > 0) {
      id = ray_of(S.g, r - S.mc_base);
      po = A.ray_pair_off[r];
    }
    if (__any_sync(0xffffffffu, c > 0 && A.ray_pair_cnt[r] > 16)) {
      // a ray of the overflow path (more ends than the mask holds): each lane writes its own
      // vertices
      int64_t o = off + incl - c;
      const int vc = id.panel == 0 ? 0 : (id.panel == 1 ? 2 : 1);
      const int ends = c > 0 ? 2 * A.ray_pair_cnt[r] : 0;
      for (int q = 0; q < ends; q++)
        if (q < 32 ? (m >> q) & 1u
                   : keeps(S.g, A.bits + S.word_base, S.nwords,
                           edge_key(id, edge_index(S.g, vc, A.pairs[2 * po + q]))))
          emit(b, id, po, q, o++);
      off += T;
      continue;
    }
    const int im = (int)id.m, in = (int)id.n;
    for (int j0 = 0; j0 < T; j0 += 32) {
      const int j = j0 + lane;
      const int l = owner_lane(incl, j < T ? j : T - 1);
      const int k = j - __shfl_sync(0xffffffffu, incl - c, l);
      const unsigned ml = __shfl_sync(0xffffffffu, m, l);
      const int64_t pol = __shfl_sync(0xffffffffu, po, l);
      RayId il;
      il.panel = __shfl_sync(0xffffffffu, id.panel, l);
      il.m = __shfl_sync(0xffffffffu, im, l);
      il.n = __shfl_sync(0xffffffffu, in, l);
      const int bl = __shfl_sync(0xffffffffu, b, l);
      if (j < T) emit(bl, il, pol, nth_bit(ml, k), off + j);
    }
    off += T;
  }
}

// The 32 bits of the flat bit grid starting at bit f (missing words read as outside), and in *next
// the 32 bits starting at f + 1, from the same two words.  A structure's grid has fewer than 2^31
// nodes, so its bit indices fit 32 bits.
__device__ __forceinline__ uint32_t bits32_pair(const uint32_t* __restrict__ bits, int32_t nwords, int32_t f,
                                                uint32_t* next) {
  const int32_t w = f >> 5;
  const int s = (int)(f & 31);
  const uint32_t lo = w < nwords ? bits[w] : 0xffffffffu;
  const uint32_t hi = (w + 1) < nwords ? bits[w + 1] : 0xffffffffu;
  const uint32_t x = s ? __funnelshift_r(lo, hi, s) : lo;
  *next = (x >> 1) | (((hi >> s) & 1u) << 31);  // bit f + 32 is bit s of the second word
  return x;
}

// The 32 cubes of a map word: row (j, k), first cube ic, and in c the inside bits of the cubes' 8
// corners (corner inside = bit 0 of the grid), one pair of words per bit row; returns the active
// cubes, those whose corners do not agree.
__device__ __forceinline__ uint32_t word_cubes(const MCArgs& A, const StructDev& S, int64_t idx, int* ic, int* j, int* k,
                                               uint32_t* c) {
  const int NX = (int)S.g.n[0], NY = (int)S.g.n[1];
  const uint32_t* bits = A.bits + S.word_base;
  const int32_t nwords = (int32_t)S.nwords;
  const unsigned W = (unsigned)(NX - 2 + 31) >> 5;
  const unsigned local = (unsigned)(idx - S.aword_base);
  const unsigned lr = local / W;
  *ic = 1 + 32 * (int)(local - lr * W);
  const unsigned kk = lr / (unsigned)(NY - 2);
  *j = 1 + (int)(lr - kk * (unsigned)(NY - 2));
  *k = 1 + (int)kk;
  const int32_t b00 = (*k * NY + *j) * NX, b10 = b00 + NX, b01 = b00 + NX * NY, b11 = b01 + NX;
  const int32_t nvalid = NX - 1 - *ic;
  const uint32_t vm = nvalid >= 32 ? 0xffffffffu : ((1u << nvalid) - 1u);
  uint32_t n0, n1, n2, n3;
  c[0] = ~bits32_pair(bits, nwords, b00 + *ic, &n0);
  c[1] = ~n0;
  c[3] = ~bits32_pair(bits, nwords, b10 + *ic, &n1);
  c[2] = ~n1;
  c[4] = ~bits32_pair(bits, nwords, b01 + *ic, &n2);
  c[5] = ~n2;
  c[7] = ~bits32_pair(bits, nwords, b11 + *ic, &n3);
  c[6] = ~n3;
  uint32_t d = 0;
#pragma unroll
  for (int q = 1; q < 8; q++) d |= c[0] ^ c[q];
  return d & vm;
}

// Cube classification in one pass, one thread per 32 cubes of a cube row (a word of the active-cube
// map), a ticket of consecutive words per block: the block places its active cubes behind those of
// the tickets before it (words in (k, j, i) order), and each warp writes the records, slots and
// triangle counts of its words with a cube per lane.  Consecutive lanes read consecutive words of
// the bit rows; the words that hold active cubes are read a second time, from L1.
// Row per thread in a count and a write pass before -> this: 64 conformers (300 M cubes) 255 + 30 ->
// 289 us; 20,000 atoms (236 M cubes) 156 + 8 -> 149 us; 2,000 atoms 15 + 5 -> 24 us, without the
// host round trip (about 20 us).
template <int kItems>
__global__ void __launch_bounds__(kPassThreads) k_mc_rows(MCArgs A) {
  __shared__ unsigned int s_ticket;
  __shared__ uint32_t s_corner[kPassThreads / 32][8][32];
  const unsigned t = take_ticket(A.lb_rows, &s_ticket);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)t * (kPassThreads * kItems) + w * (32 * kItems) + lane;
  uint32_t act[kItems];
  int sum = 0;
  const StructWalk start(A.B.aword_base, A.B.n, i0 - lane);
  StructWalk walk = start;
#pragma unroll
  for (int x = 0; x < kItems; x++) {
    const int64_t idx = i0 + 32 * x;
    const bool valid = idx < A.nwords_map;
    const int b = walk.at(idx);
    act[x] = 0;
    if (valid) {
      int ic, j, k;
      uint32_t c[8];
      act[x] = word_cubes(A, A.B.s[b], idx, &ic, &j, &k, c);
    }
    sum += __popc(act[x]);
  }
  int64_t off = warp_offset<kPassThreads>(A.lb_rows, t, warp_total(sum));
  if (off < 0) return;
  walk = start;
#pragma unroll 1
  for (int x = 0; x < kItems; x++) {
    const int64_t idx = i0 + 32 * x;
    const bool valid = idx < A.nwords_map;
    const int b = walk.at(idx);
    const StructDev& S = A.B.s[b];
    uint32_t a = act[0];
#pragma unroll
    for (int y = 1; y < kItems; y++)
      if (x == y) a = act[y];
    const int cnt = __popc(a);
    const int incl = warp_incl(cnt);
    const int T = __shfl_sync(0xffffffffu, incl, 31);
    if (valid) {
      const int64_t first = off + incl - cnt;
      A.amap[idx] = make_int2((int)a, (int)first);
      if (idx == S.aword_base) A.aoff[b] = first;
      if (idx == A.nwords_map - 1) A.aoff[A.B.n] = A.counts[kMcActive] = first + cnt;
    }
    if (T == 0) continue;
    int ic = 0, j = 0, k = 0;
    uint32_t c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (a) word_cubes(A, S, idx, &ic, &j, &k, c);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; q++) s_corner[w][q][lane] = c[q];
    __syncwarp();
    for (int j0 = 0; j0 < T; j0 += 32) {
      const int y = j0 + lane;
      const int l = owner_lane(incl, y < T ? y : T - 1);
      const int first = __shfl_sync(0xffffffffu, incl - cnt, l);
      const unsigned al = __shfl_sync(0xffffffffu, a, l);
      const int il = __shfl_sync(0xffffffffu, ic, l), jl = __shfl_sync(0xffffffffu, j, l),
                kl = __shfl_sync(0xffffffffu, k, l), bl = __shfl_sync(0xffffffffu, b, l);
      const int64_t slot = off + y;
      if (y >= T || slot >= A.cap_active) continue;
      const int bit = nth_bit(al, y - first);
      int cs = 0;
#pragma unroll
      for (int q = 0; q < 8; q++) cs |= ((s_corner[w][q][l] >> bit) & 1u) << q;
      const int i = il + bit;
      // every cut edge of a cube with i, j, k >= 2 has a vertex (an analytic one, or the midpoint
      // its owner cube adds), so its triangles are the case table's; a cube on the low faces of the
      // cube range may lack vertices on edges whose owner lies outside the range, and is counted
      // after the midpoint vertices are in place (k_mc_tris_bnd)
      int ntri = d_mc.ntri[cs];
      if (i < 2 || jl < 2 || kl < 2) {
        ntri = 0;
        const unsigned long long q = atomicAdd((unsigned long long*)(A.counts + kMcLowFace), 1ull);
        A.bnd_list[q] = (int32_t)slot;
      }
      A.tri_cnt[slot] = ntri;
      A.act_rec[slot] = make_int4(i, jl, kl, cs | (bl << 11));
      if (A.clear_slots) {
        int4* v = reinterpret_cast<int4*>(A.cube_vl + 12 * slot);
        const int4 none = make_int4(-1, -1, -1, -1);
        v[0] = none;
        v[1] = none;
        v[2] = none;
      }
    }
    off += T;
  }
}

// Vertex slots of the active cubes of structures [b0, b1) to -1.
__global__ void k_mc_clear(MCArgs A, int b0, int b1) {
  if (!cubes_ok(A)) return;
  int4* v = reinterpret_cast<int4*>(A.cube_vl);
  const int4 none = make_int4(-1, -1, -1, -1);
  for (int64_t q = 3 * A.aoff[b0] + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < 3 * A.aoff[b1];
       q += (int64_t)gridDim.x * blockDim.x)
    v[q] = none;
}

// Midpoint vertices in one pass, one thread per active cube, a ticket of consecutive cubes per
// block: which of the cube's own edges 5 (y at (i+1, j, k+1)), 6 (x at (i, j+1, k+1)), 10 (z at
// (i+1, j+1, k)) are cut and carry no analytic vertex (their slots are still empty after the
// analytic push); the vertices follow the analytic ones in (k, j, i, edge) order and go into the
// slots of the cubes that share their edges.  An edge is slot 5, 6 or 10 of its owner alone, so no
// cube's test reads a slot that another cube's midpoint is written to.  Bound by the slot reads.
template <int kItems>
__global__ void __launch_bounds__(kPassThreads) k_mc_mid(MCArgs A) {
  const int64_t n_act = A.counts[kMcActive], n_an = A.counts[kMcAnalytic];
  unsigned t;
  if (!take_ticket_if(A.lb_mid, [&] { return cubes_fit(A); }, &t)) return;
  if ((int64_t)t * (kPassThreads * kItems) >= n_act) return;
  const int lane = threadIdx.x & 31;
  const int64_t a0 = (int64_t)t * (kPassThreads * kItems) + (threadIdx.x >> 5) * (32 * kItems) + lane;
  int mm[kItems], s5[kItems], s6[kItems], s10[kItems], sum = 0;
#pragma unroll
  for (int x = 0; x < kItems; x++) {
    const int64_t a = a0 + 32 * x < n_act ? a0 + 32 * x : n_act - 1;
    mm[x] = A.act_rec[a].w & 255;
    s5[x] = A.cube_vl[12 * a + 5];
    s6[x] = A.cube_vl[12 * a + 6];
    s10[x] = A.cube_vl[12 * a + 10];
  }
#pragma unroll
  for (int x = 0; x < kItems; x++) {
    // edges 5, 6 and 10 join corners 5-6, 6-7 and 2-6
    const int cs = mm[x], c6 = (cs >> 6) & 1;
    mm[x] = 0;
    if (((cs >> 5) & 1) != c6 && s5[x] < 0) mm[x] |= 1;
    if (((cs >> 7) & 1) != c6 && s6[x] < 0) mm[x] |= 2;
    if (((cs >> 2) & 1) != c6 && s10[x] < 0) mm[x] |= 4;
    if (a0 + 32 * x >= n_act) mm[x] = 0;
    sum += __popc(mm[x]);
  }
  int64_t off = warp_offset<kPassThreads>(A.lb_mid, t, warp_total(sum));
  if (off < 0) return;
#pragma unroll
  for (int x = 0; x < kItems; x++) {
    const int64_t a = a0 + 32 * x;
    const int m = mm[x], cnt = __popc(m);
    const int incl = warp_incl(cnt);
    if (a == n_act - 1) A.counts[kMcMidpoint] = off + incl;
    int64_t v = n_an + off + incl - cnt;
    off += __shfl_sync(0xffffffffu, incl, 31);
    if (!m || v + cnt > A.cap_vert) continue;
    const int4 rec = A.act_rec[a];
    const int i = rec.x, j = rec.y, k = rec.z;
    const StructDev& S = A.B.s[rec_struct(rec.w)];
    const GridDev& g = S.g;
    for (int q = 0; q < cnt; q++) A.vstruct[v + q] = rec_struct(rec.w);
    if (m & 1) {
      A.vpos[3 * v] = gcoord(g, 0, i + 1) - g.hside; A.vpos[3 * v + 1] = gcoord(g, 1, j);
      A.vpos[3 * v + 2] = gcoord(g, 2, k + 1) - g.hside;
      A.vkey[v] = make_int4(i + 1, j, k + 1, NS_Y_DIR);
      push_vertex(A.amap, A.cube_vl, S, NS_Y_DIR, i + 1, j, k + 1, (int32_t)v);
      v++;
    }
    if (m & 2) {
      A.vpos[3 * v] = gcoord(g, 0, i); A.vpos[3 * v + 1] = gcoord(g, 1, j + 1) - g.hside;
      A.vpos[3 * v + 2] = gcoord(g, 2, k + 1) - g.hside;
      A.vkey[v] = make_int4(i, j + 1, k + 1, NS_X_DIR);
      push_vertex(A.amap, A.cube_vl, S, NS_X_DIR, i, j + 1, k + 1, (int32_t)v);
      v++;
    }
    if (m & 4) {
      A.vpos[3 * v] = gcoord(g, 0, i + 1) - g.hside; A.vpos[3 * v + 1] = gcoord(g, 1, j + 1) - g.hside;
      A.vpos[3 * v + 2] = gcoord(g, 2, k);
      A.vkey[v] = make_int4(i + 1, j + 1, k, NS_Z_DIR);
      push_vertex(A.amap, A.cube_vl, S, NS_Z_DIR, i + 1, j + 1, k, (int32_t)v);
    }
  }
}

// One thread per analytic vertex: the first vertex of each grid edge goes into the slots of the
// edge's cubes.  A ray's vertices are sorted along it and an edge's vertices all lie on one ray,
// so they have consecutive ids: vertex v is the first of its edge unless vertex v - 1 has the same
// edge key in the same structure.  Each slot is written once, with a plain store.
__global__ void k_mc_push(MCArgs A, int b0, int b1) {
  if (!cubes_ok(A)) return;
  const int64_t v0 = A.voff[b0], v1 = A.voff[b1];
  for (int64_t v = v0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < v1; v += (int64_t)gridDim.x * blockDim.x) {
    const int4 e = A.vkey[v];
    const int32_t sv = A.vstruct[v];
    if (v > v0) {
      const int4 p = A.vkey[v - 1];
      if (p.x == e.x && p.y == e.y && p.z == e.z && p.w == e.w && A.vstruct[v - 1] == sv) continue;
    }
    push_vertex(A.amap, A.cube_vl, A.B.s[sv], e.w, e.x, e.y, e.z, (int32_t)v);
  }
}

// Triangle counts of the active cubes on the low faces of the cube range (listed by k_mc_rows): the
// case-table triangles whose three edges have vertices.
__global__ void k_mc_tris_bnd(MCArgs A) {
  if (!cubes_ok(A)) return;
  const int64_t n = A.counts[kMcLowFace];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int32_t a = A.bnd_list[q];
    const int c = A.act_rec[a].w & 255;
    const int32_t* cv = A.cube_vl + 12 * (int64_t)a;
    int cnt = 0;
    for (int t = 0; t < 16 && d_mc.tri[c][t] >= 0; t += 3)
      if (cv[d_mc.tri[c][t]] >= 0 && cv[d_mc.tri[c][t + 1]] >= 0 && cv[d_mc.tri[c][t + 2]] >= 0) cnt++;
    A.tri_cnt[a] = cnt;
  }
}

constexpr int kTrisThreads = 256;
constexpr int kTrisWarps = kTrisThreads / 32;
constexpr int kMaxCubeTris = 5;  // the most triangles of a case

// Triangles, 32 active cubes per warp at a time, a ticket of consecutive cubes per block: the block
// places its triangles (tri_cnt per cube) behind those of the tickets before it; then the lanes
// load their cubes' 12 vertex slots into shared memory and the warp's triangles are spread over its
// lanes, one per lane, whatever the cubes' cases.  Each writes its triangle with reversed winding
// (coalesced across the warp) and its area (and, in gradient mode, the area's derivatives with
// respect to its analytic vertices); each cube's area is the sum of its triangles' in case-table
// order.  Bound by the vertex gathers.  Scan of the counts, then triangles -> this: 64
// conformers 30 + 582 -> 579 us, 20,000 atoms 8 + 145 -> 83 us (most of it the case table, which
// every block read from the constant bank), 2,000 atoms 5 + 28 -> 22 us.
template <int kMinBlocks, int kItems>
__global__ void __launch_bounds__(kTrisThreads, kMinBlocks) k_mc_tris(MCArgs A) {
  __shared__ alignas(16) int8_t s_tri[256][16];
  __shared__ alignas(16) uint8_t s_ntri[256];
  // per warp: each cube's vertex slots ([slot][lane]) and the areas of the warp's triangles
  __shared__ int32_t s_vid[kTrisWarps][12][32];
  __shared__ double s_area[kTrisWarps][kMaxCubeTris * 32];
  const int64_t n_act = A.counts[kMcActive], n_an = A.counts[kMcAnalytic];
  unsigned ticket;
  if (!take_ticket_if(A.lb_tris, [&] { return cubes_fit(A) && n_an + A.counts[kMcMidpoint] <= A.cap_vert; }, &ticket))
    return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if ((int64_t)ticket * (kTrisThreads * kItems) >= n_act) return;
  const int64_t a0 = (int64_t)ticket * (kTrisThreads * kItems) + w * (32 * kItems) + lane;
  // the 4 KB case table: one 16-byte load per thread
  reinterpret_cast<int4*>(&s_tri[0][0])[threadIdx.x] = reinterpret_cast<const int4*>(&d_mc.tri[0][0])[threadIdx.x];
  if (threadIdx.x < 16)
    reinterpret_cast<int4*>(s_ntri)[threadIdx.x] = reinterpret_cast<const int4*>(d_mc.ntri)[threadIdx.x];
  int sum = 0;
#pragma unroll
  for (int x = 0; x < kItems; x++) sum += a0 + 32 * x < n_act ? A.tri_cnt[a0 + 32 * x] : 0;
  int64_t tbase = warp_offset<kTrisThreads>(A.lb_tris, ticket, warp_total(sum));  // synchronises the block
  if (tbase < 0) return;
#pragma unroll 1
  for (int x = 0; x < kItems; x++) {
    const int64_t a = a0 + 32 * x;
    const bool valid = a < n_act;
    if (!__any_sync(0xffffffffu, valid)) break;
    const int cw = valid ? A.act_rec[a].w : 0;
    const int cnt = valid ? A.tri_cnt[a] : 0;
    if (valid) {
      const int4* cv = reinterpret_cast<const int4*>(A.cube_vl + 12 * a);
      const int4 v0 = cv[0], v1 = cv[1], v2 = cv[2];
      s_vid[w][0][lane] = v0.x; s_vid[w][1][lane] = v0.y; s_vid[w][2][lane] = v0.z; s_vid[w][3][lane] = v0.w;
      s_vid[w][4][lane] = v1.x; s_vid[w][5][lane] = v1.y; s_vid[w][6][lane] = v1.z; s_vid[w][7][lane] = v1.w;
      s_vid[w][8][lane] = v2.x; s_vid[w][9][lane] = v2.y; s_vid[w][10][lane] = v2.z; s_vid[w][11][lane] = v2.w;
    }
    const int incl = warp_incl(cnt);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (a == n_act - 1) A.counts[kMcTriangle] = tbase + incl;
    __syncwarp();
    for (int t0 = 0; t0 < total; t0 += 32) {
      const int t = t0 + lane;
      // the cube of triangle t: the first lane whose inclusive count exceeds t
      int l = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        const int x = __shfl_sync(0xffffffffu, incl, l + step - 1);
        if (x <= t) l += step;
      }
      const int ll = l < 31 ? l : 31;
      const int first = __shfl_sync(0xffffffffu, incl - cnt, ll);
      const int lcnt = __shfl_sync(0xffffffffu, cnt, ll);
      const int lw = __shfl_sync(0xffffffffu, cw, ll);
      if (t >= total) continue;
      const int q = t - first;
      const int c = lw & 255;
      const int32_t* lv = &s_vid[w][0][ll];
      // the q-th case triangle whose three edges have vertices: the q-th of the case when the cube
      // keeps all of them (every cube off the low faces), else found by a scan
      int e0 = s_tri[c][3 * q], e1 = s_tri[c][3 * q + 1], e2 = s_tri[c][3 * q + 2];
      if (lcnt != s_ntri[c]) {
        for (int qq = 0, seen = 0; qq < 15 && s_tri[c][qq] >= 0; qq += 3) {
          e0 = s_tri[c][qq];
          e1 = s_tri[c][qq + 1];
          e2 = s_tri[c][qq + 2];
          if (lv[32 * e0] >= 0 && lv[32 * e1] >= 0 && lv[32 * e2] >= 0) {
            if (seen == q) break;
            seen++;
          }
        }
      }
      const int32_t v0 = lv[32 * e0], v1 = lv[32 * e1], v2 = lv[32 * e2];
      if (tbase + t < A.cap_tri) {
        A.tris[3 * (tbase + t) + 0] = v2;
        A.tris[3 * (tbase + t) + 1] = v1;
        A.tris[3 * (tbase + t) + 2] = v0;
      }
      const double* P0 = A.vpos + 3 * (int64_t)v0;
      const double* P1 = A.vpos + 3 * (int64_t)v1;
      const double* P2 = A.vpos + 3 * (int64_t)v2;
      const double p0[3] = {P0[0], P0[1], P0[2]}, p1[3] = {P1[0], P1[1], P1[2]}, p2[3] = {P2[0], P2[1], P2[2]};
      // area = |n| / 2, n = (P1 - P0) x (P2 - P0): the area the reference computes with Heron's
      // formula (getTriangles, src/Surface.cpp:14559-14780), with one square root instead of four
      const double f1[3] = {p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2]};
      const double f2[3] = {p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2]};
      double nn[3] = {f1[1] * f2[2] - f1[2] * f2[1], f1[2] * f2[0] - f1[0] * f2[2], f1[0] * f2[1] - f1[1] * f2[0]};
      const double nl = sqrt(nn[0] * nn[0] + nn[1] * nn[1] + nn[2] * nn[2]);
      s_area[w][t] = nl > 0 ? 0.5 * nl : 0.0;
      if (nl > 0 && A.vgrad) {
        // d area / d (position of vertex vv along the axis of its cube edge ev, which is the ray
        // an analytic vertex moves on): ((Pa - Pb) x n / (2 |n|)) along that axis
        const double h = 0.5 / nl;
        nn[0] *= h;
        nn[1] *= h;
        nn[2] *= h;
        const auto add = [&](int32_t vv, int ev, double dx, double dy, double dz) {
          if (vv >= n_an) return;
          double comp;
          if (ev >= 8) comp = dx * nn[1] - dy * nn[0];        // z
          else if (ev & 1) comp = dz * nn[0] - dx * nn[2];    // y
          else comp = dy * nn[2] - dz * nn[1];                // x
          if (comp != 0.0) atomicAdd(A.vgrad + vv, comp);
        };
        add(v0, e0, p1[0] - p2[0], p1[1] - p2[1], p1[2] - p2[2]);
        add(v1, e1, p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2]);
        add(v2, e2, p0[0] - p1[0], p0[1] - p1[1], p0[2] - p1[2]);
      }
    }
    __syncwarp();
    if (valid) {
      double area = 0.0;
      for (int q = 0; q < cnt; q++) area += s_area[w][incl - cnt + q];
      A.cube_area[a] = area;
    }
    __syncwarp();
    tbase += total;
  }
}

// One thread per analytic vertex: d area / d patch parameters += (d area / d s) * ds / d theta.
// Consecutive vertices (along a ray, and of neighbouring rays) mostly lie on the same patch, so the
// per-patch sums go through warp_add_grad.
__global__ void k_grad_vert(MCArgs A) {
  const int64_t n_an = A.counts[kMcAnalytic];
  if (!cubes_ok(A) || n_an + A.counts[kMcMidpoint] > A.cap_vert) return;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n_an; base += stride) {
    const int64_t v = base + (threadIdx.x & 31);
    double g[NS_GRAD_PER_PATCH];
    int32_t pid = -1;
    const double gv = v < n_an ? A.vgrad[v] : 0.0;
    if (gv != 0.0) {
      const double x[3] = {A.vpos[3 * v], A.vpos[3 * v + 1], A.vpos[3 * v + 2]};
      const int32_t vp = A.vpid[v];
      pid = vp & kVpidPatchMask;
      if (vp >= 0 &&
          hit_grad(A.f64 + (int64_t)NS_PATCH_F64 * pid, A.i32[NS_PATCH_I32 * pid], A.probe, x, vp >> kVpidAxisShift, g)) {
#pragma unroll
        for (int k = 0; k < NS_GRAD_PER_PATCH; k++) g[k] *= gv;
      } else {
        pid = -1;
      }
    }
    if (pid < 0)
#pragma unroll
      for (int k = 0; k < NS_GRAD_PER_PATCH; k++) g[k] = 0.0;
    warp_add_grad(pid, g, A.garea);
  }
}

// The patch normal at a vertex: ConnollySurface::getNormal (src/ConnollySurface.cpp:5736-5819) for
// atom spheres (y - c) / r, probe spheres (c - y) / probe and tori (getNormalToTorus, with the
// frame's transpose for Rot); for skin cells the quadric's gradient times 2 (-2 for reduced
// tetrahedra), as SkinSurface::getPatchIntersectionData stores it (src/SkinSurface.cpp:3684-3712).
__global__ void k_vertex_normals(const double* __restrict__ vpos, const int32_t* __restrict__ vpid, int64_t n,
                                 const double* __restrict__ f64, const int32_t* __restrict__ i32, double probe,
                                 double* out) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const int32_t vp = vpid[v];
    if (vp < 0) continue;
    const int32_t pid = vp & kVpidPatchMask;
    const double* f = f64 + (int64_t)NS_PATCH_F64 * pid;
    const int kind = i32[NS_PATCH_I32 * pid];
    const double y[3] = {vpos[3 * v], vpos[3 * v + 1], vpos[3 * v + 2]};
    double nrm[3] = {0.0, 0.0, 0.0};
    if (kind == NS_FACE_REG || kind == NS_FACE_SING) {
      for (int d = 0; d < 3; d++) nrm[d] = (f[d] - y[d]) / probe;
    } else if (kind == NS_POINT) {
      for (int d = 0; d < 3; d++) nrm[d] = (y[d] - f[d]) / f[3];
    } else if (kind == NS_EDGE_REG || kind == NS_EDGE_SING) {
      const double* inv = f + 9;
      const double t[3] = {y[0] - f[4], y[1] - f[5], y[2] - f[6]};
      double C[3];
      for (int i = 0; i < 3; i++) C[i] = inv[3 * i] * t[0] + inv[3 * i + 1] * t[1] + inv[3 * i + 2] * t[2];
      double dd = C[0] * C[0] + C[1] * C[1];
      const double rm1 = f[7] / sqrt(dd) - 1.;
      dd = sqrt(dd * rm1 * rm1 + C[2] * C[2]);
      C[0] *= rm1 / dd;
      C[1] *= rm1 / dd;
      C[2] /= -dd;
      for (int i = 0; i < 3; i++) nrm[i] = inv[i] * C[0] + inv[3 + i] * C[1] + inv[6 + i] * C[2];
    } else if (ns_is_skin(kind)) {
      const double* Q = f + NS_SKIN_Q;
      const double sg = kind == NS_SKIN_TETRA ? -2.0 : 2.0;
      nrm[0] = sg * (Q[0] * y[0] + Q[4] * y[1] + Q[7] * y[2] + Q[9]);
      nrm[1] = sg * (Q[4] * y[0] + Q[1] * y[1] + Q[5] * y[2] + Q[8]);
      nrm[2] = sg * (Q[7] * y[0] + Q[5] * y[1] + Q[2] * y[2] + Q[6]);
    }
    for (int d = 0; d < 3; d++) out[3 * v + d] = nrm[d];
  }
}

int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)sm_count() * 32;
  return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

}  // namespace

static unsigned tickets(int64_t items, int most) {
  const int64_t per = (int64_t)kPassThreads * pass_items(items, most);
  return (unsigned)((items + per - 1) / per);
}

McTickets mc_tickets(int64_t rays, int64_t words, int64_t cubes) {
  return McTickets{tickets(rays, kVertItems), tickets(words, kRowsItems), tickets(cubes, kMidItems),
                   tickets(cubes, kTrisItems)};
}

cudaError_t launch_vert(const VertArgs& A, cudaStream_t s) {
  if (A.nrays == 0) return cudaSuccess;
  const unsigned b = tickets(A.nrays, kVertItems);
  if (pass_items(A.nrays, kVertItems) == 4) k_vert<4><<<b, kPassThreads, 0, s>>>(A);
  else k_vert<1><<<b, kPassThreads, 0, s>>>(A);
  return cudaGetLastError();
}

cudaError_t launch_mc_rows(const MCArgs& A, cudaStream_t s) {
  if (A.nwords_map <= 0) return cudaSuccess;
  const unsigned b = tickets(A.nwords_map, kRowsItems);
  const int items = pass_items(A.nwords_map, kRowsItems);
  if (items == 8) k_mc_rows<8><<<b, kPassThreads, 0, s>>>(A);
  else if (items == 4) k_mc_rows<4><<<b, kPassThreads, 0, s>>>(A);
  else k_mc_rows<1><<<b, kPassThreads, 0, s>>>(A);
  return cudaGetLastError();
}

cudaError_t launch_mc_clear(const MCArgs& A, int b0, int b1, int64_t cubes, cudaStream_t s) {
  k_mc_clear<<<grid_for(3 * cubes, 256), 256, 0, s>>>(A, b0, b1);
  return cudaGetLastError();
}

// The midpoint and triangle passes take tickets for the capacity; those past the active cubes return
// at once.
cudaError_t launch_mc_mid(const MCArgs& A, cudaStream_t s) {
  const unsigned b = tickets(A.cap_active, kMidItems);
  if (pass_items(A.cap_active, kMidItems) == 4) k_mc_mid<4><<<b, kPassThreads, 0, s>>>(A);
  else k_mc_mid<1><<<b, kPassThreads, 0, s>>>(A);
  return cudaGetLastError();
}

template <int kMinBlocks>
void launch_tris(const MCArgs& A, cudaStream_t s) {
  const unsigned b = tickets(A.cap_active, kTrisItems);
  const int items = pass_items(A.cap_active, kTrisItems);
  if (items == 8) k_mc_tris<kMinBlocks, 8><<<b, kTrisThreads, 0, s>>>(A);
  else if (items == 4) k_mc_tris<kMinBlocks, 4><<<b, kTrisThreads, 0, s>>>(A);
  else k_mc_tris<kMinBlocks, 1><<<b, kTrisThreads, 0, s>>>(A);
}

cudaError_t launch_mc_tris(const MCArgs& A, int blocks_per_sm, cudaStream_t s) {
  static_assert(kTrisThreads == kPassThreads, "one ticket count for both passes");
  if (blocks_per_sm >= 4) launch_tris<4>(A, s);
  else launch_tris<3>(A, s);
  return cudaGetLastError();
}

cudaError_t launch_vertex_normals(const double* vpos, const int32_t* vpid, int64_t n_analytic, const double* f64,
                                  const int32_t* i32, double probe, double* normals, cudaStream_t s) {
  if (n_analytic <= 0) return cudaSuccess;
  k_vertex_normals<<<grid_for(n_analytic, 256), 256, 0, s>>>(vpos, vpid, n_analytic, f64, i32, probe, normals);
  return cudaGetLastError();
}

cudaError_t launch_mc_push(const MCArgs& A, int b0, int b1, int64_t vertices, cudaStream_t s) {
  k_mc_push<<<grid_for(vertices, 256), 256, 0, s>>>(A, b0, b1);
  return cudaGetLastError();
}

cudaError_t launch_mc_tris_bnd(const MCArgs& A, cudaStream_t s) {
  k_mc_tris_bnd<<<sm_count(), 256, 0, s>>>(A);
  return cudaGetLastError();
}

cudaError_t launch_grad_vert(const MCArgs& A, int64_t vertices, cudaStream_t s) {
  if (!A.vgrad) return cudaSuccess;
  k_grad_vert<<<grid_for(vertices, 256), 256, 0, s>>>(A);
  return cudaGetLastError();
}

}  // namespace nsg
