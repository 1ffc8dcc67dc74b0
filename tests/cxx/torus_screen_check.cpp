// Every torus candidate of a patch set on one panel: the single-precision screen (torus_screen.h)
// against the double-precision path (ray_math.cuh, compiled for the host).  counts: candidates,
// candidates with a hit, candidates the screen keeps, candidates with a hit that it drops.
#define __device__
#define __forceinline__ inline
#define __restrict__
#include <cmath>
#include <cstdint>
#include <algorithm>
using std::floor;
using std::fmax;
using std::fmin;
struct double4 {
  double x, y, z, w;
};
#include "kernels/ray_math.cuh"
#include "torus_screen.h"

using namespace nsg;

template <int fd, int ld, int vc>
static void check(const NsGrid& g, int64_t np, const double* f64, const int32_t* i32, const double4* pool,
                  const int8_t* flag, double probe, double delta, int64_t* counts) {
  const double mn[3] = {g.xmin, g.ymin, g.zmin};
  const int64_t nn[3] = {g.nx, g.ny, g.nz};
  const double len = (double)(nn[vc] - 1) * g.side;
  for (int64_t p = 0; p < np; p++) {
    const int kind = i32[4 * p], first = i32[4 * p + 1], cnt = i32[4 * p + 2];
    if (kind != NS_EDGE_REG && kind != NS_EDGE_SING) continue;
    const double* f = f64 + NS_PATCH_F64 * p;
    float rec[kTorusScreen];
    const bool wedge = cnt == 2 && flag[first] != 0;
    torus_screen_record(f, wedge ? (const double*)(pool + first) : nullptr, wedge, probe, rec);
    int64_t lo[2], hi[2];
    const int ax[2] = {fd, ld};
    for (int q = 0; q < 2; q++) {
      const int d = ax[q];
      lo[q] = std::max<int64_t>(0, (int64_t)((f[d] - f[3] - mn[d] - delta) / g.side) - 1);
      hi[q] = std::min<int64_t>(nn[d] - 1, (int64_t)((f[d] + f[3] - mn[d] - delta) / g.side) + 1);
    }
    for (int64_t n = lo[1]; n <= hi[1]; n++)
      for (int64_t m = lo[0]; m <= hi[0]; m++) {
        double pa[3];
        pa[fd] = (mn[fd] + (double)m * g.side) + delta;
        pa[ld] = (mn[ld] + (double)n * g.side) + delta;
        pa[vc] = mn[vc] + delta;
        const double dx = f[fd] - pa[fd], dy = f[ld] - pa[ld];
        if (dx * dx + dy * dy > f[3] * f[3]) continue;
        counts[0]++;
        double dir[3] = {0, 0, 0}, t[4];
        dir[vc] = len;
        int hits = 0;
        if (ray_sphere_f64(pa, dir, f, f[3], &t[0], &t[1])) {
          const int k = ray_torus_f64(f, probe, vc, pa, len, t);
          for (int i = 0; i < k; i++) {
            double ip[3] = {pa[0], pa[1], pa[2]};
            ip[vc] += t[i] * len;
            hits += feasible_f64(f, kind, first, cnt, pool, flag, ip);
          }
        }
        const bool may = torus_may_hit<fd, ld, vc>(rec, (float)(pa[fd] - f[fd]), (float)(pa[ld] - f[ld]));
        counts[1] += hits > 0;
        counts[2] += may;
        counts[3] += hits > 0 && !may;
      }
  }
}

extern "C" void torus_screen_check(const NsGrid* g, int64_t np, const double* f64, const int32_t* i32,
                                   const double* pool, const int8_t* flag, double probe, int panel, double delta,
                                   int64_t* counts) {
  const double4* p = (const double4*)pool;
  if (panel == 0) check<1, 2, 0>(*g, np, f64, i32, p, flag, probe, delta, counts);
  else if (panel == 1) check<0, 1, 2>(*g, np, f64, i32, p, flag, probe, delta, counts);
  else check<0, 2, 1>(*g, np, f64, i32, p, flag, probe, delta, counts);
}
