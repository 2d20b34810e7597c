// Host-side geometry shared by the solver context (solver.cu) and the
// allocation-free operator (qbq_static.cu): FFT plans of the three axes, the
// plane/pencil layout, the per-k table offsets, the Bloch phases theta and the
// reduced size Nd.  Both translation units build their Geom here, so the layout the
// kernels index is the same in both.
#pragma once
#include <math.h>
#include <string.h>

#include <algorithm>
#include <string>

#include "../../include/fame_b200.h"
#include "op_kernels_decl.h"

namespace fame {

// Radix plan of an axis.  Radix order 0 (the default): the fewest passes out of the
// butterflies 2..13, the smallest radix sum among those, largest radix first; every
// length up to 144 without a prime factor >= 17 takes at most two passes but a few (75, 98, 105, ...),
// where 8, 4, 2, 5, 3 in turn took three or four, each a round trip of the
// whole plane through shared memory.  Order 1: the same radices, smallest first.  Orders
// 2 and 3: the listed radices as often as they divide n, in turn.  Prime factors
// from 17 up come last.  The plan tuner tries all four.
constexpr int kNumRadixOrders = 4;
constexpr int kNumListed = 8;
constexpr int kListedRadices[2][kNumListed] = {
    {8, 4, 2, 5, 3, 7, 11, 13},  // 64 = 8 8, 96 = 8 4 3
    {3, 5, 7, 11, 13, 4, 8, 2},  // odd radices first: 96 = 3 4 4 2
};

// Fewest radices <= hi whose product is m (smallest sum among equals), non-increasing;
// returns their number or kMaxPasses + 1.
inline int fewest_radices(int m, int hi, int* out) {
  if (m == 1) return 0;
  int best = kMaxPasses + 1, best_sum = 0;
  for (int r = std::min(hi, m); r >= 2; r--) {
    if (m % r) continue;
    int rest[kMaxPasses + 1] = {};
    const int c = 1 + fewest_radices(m / r, r, rest);
    if (c > kMaxPasses) continue;
    int sum = r;
    for (int i = 0; i < c - 1; i++) sum += rest[i];
    if (c < best || (c == best && sum < best_sum)) {
      best = c;
      best_sum = sum;
      out[0] = r;
      for (int i = 0; i < c - 1; i++) out[i + 1] = rest[i];
    }
  }
  return best;
}

inline bool factor_axis(int n, AxisPlan& p, int order = 0) {
  p.n = n;
  p.npass = 0;
  int m = n;  // n without its prime factors >= 17
  for (int q = 17; q <= m; q++) {
    int k = m;
    while (k % 2 == 0) k /= 2;
    for (int r : {3, 5, 7, 11, 13})
      while (k % r == 0) k /= r;
    if (k == 1) break;
    while (k % q == 0) {
      k /= q;
      m /= q;
    }
  }
  const int big = n / m;
  if (order <= 1) {
    int rad[kMaxPasses + 1] = {};
    const int c = fewest_radices(m, 13, rad);
    if (c > kMaxPasses) return false;
    for (int i = 0; i < c; i++) p.radix[p.npass++] = rad[order == 0 ? i : c - 1 - i];
  } else {
    for (int r : kListedRadices[order - 2])
      for (; m % r == 0; m /= r) {
        if (p.npass >= kMaxPasses) return false;
        p.radix[p.npass++] = r;
      }
  }
  int rest = big;
  for (int q = 17; rest > 1 && q <= rest; q++)
    for (; rest % q == 0; rest /= q) {
      if (p.npass >= kMaxPasses) return false;
      p.radix[p.npass++] = q;
    }
  return true;
}

// Lengths, plans, table and twiddle offsets of lattice L.  Simple lattices walk
// (slow, mid, fast) = (z, y, x); General lattices (x, y, z) in frequency (the
// reference's z-fastest order, FAME_Main/FAME_Matrix_Lambdas.cu:317).  Returns a
// FAME_* status; err receives the reason.  max_points bounds N.
inline int layout_geom(const fame_lattice& L, Geom& g, long max_points, std::string& err, int radix_order = 0) {
  memset(&g, 0, sizeof(g));
  g.Nx = L.grid[0];
  g.Ny = L.grid[1];
  g.Nz = L.grid[2];
  if (g.Nx < 2 || g.Ny < 2 || g.Nz < 2) {
    err = "grid dimensions must be >= 2";
    return FAME_ERR_BAD_INPUT;
  }
  const long N = (long)g.Nx * g.Ny * g.Nz;
  if (N > max_points) {
    err = "grid too large";
    return FAME_ERR_BAD_INPUT;
  }
  g.N = (int)N;
  g.general = L.simple ? 0 : 1;
  g.hx = L.mesh_len[0];
  g.hy = L.mesh_len[1];
  g.hz = L.mesh_len[2];
  g.ihz = 1.0 / g.hz;
  g.tnz = 2.0 / g.Nz;
  g.Ls = g.general ? g.Nx : g.Nz;
  g.Lm = g.Ny;
  g.Lf = g.general ? g.Nz : g.Nx;
  g.P = g.Lm * g.Lf;
  g.mLf = g.Lf == 1 ? 0u : 0xffffffffu / (unsigned)g.Lf + 1u;
  g.S = g.Lf | 1;  // odd row pitch: bank-conflict-free passes along both plane axes
  if (!factor_axis(g.Lf, g.pf, radix_order) || !factor_axis(g.Lm, g.pm, radix_order) ||
      !factor_axis(g.Ls, g.ps, radix_order)) {
    err = "axis length needs more than 10 FFT passes";
    return FAME_ERR_UNSUPPORTED;
  }
  if (plane_smem_bytes<double>(g.Lf, g.Lm, g.S) > 227 * 1024) {
    err = "plane " + std::to_string(g.Lm) + "x" + std::to_string(g.Lf) + " exceeds one CTA";
    return FAME_ERR_UNSUPPORTED;
  }
  int o = 0;
  if (!g.general) {
    g.oLx = o; o += g.Nx;
    g.oLy = o; o += g.Ny;
    g.oLz = o; o += g.Nz;
    g.oDx = o; o += g.Nx;
    g.oDy = o; o += g.Ny;
    g.oDz = o; o += g.Nz;
  } else {
    g.oLx = o; o += g.Nx;
    g.oLy = o; o += g.Nx * g.Ny;
    g.oExy = o; o += g.Nx * g.Ny;
    g.oWz = o; o += g.Nz;
    g.oDky = o; o += g.Nx * g.Ny;
    g.oPhi = o; o += g.Nx * g.Ny;
    g.oDkx = o; o += g.Nx;
  }
  g.tab_stride = (o + 7) / 8 * 8;
  // forward twiddle tables e^{-2 pi i m / n} of the fast, mid and slow axes, back to back
  g.twf = 0;
  g.twm = g.Lf;
  g.tws = g.Lf + g.Lm;
  return FAME_OK;
}

// Pass level of the three axis plans.
inline int geom_level(const Geom& g) {
  return std::max(plan_level(g.pf), std::max(plan_level(g.pm), plan_level(g.ps)));
}
// ... the plane stages' axes (fast, mid) and the pencil stage's axis (slow) alone: each
// stage kernel carries the prime passes only when its own axes need them (fewer
// registers, no spills from passes it never runs)
inline int plane_level(const Geom& g) { return std::max(plan_level(g.pf), plan_level(g.pm)); }
inline int pencil_level(const Geom& g) { return plan_level(g.ps); }

// Threads a plane CTA of precision R must have (every pass covers whole lines), and may have (the
// kernels' launch bounds, DynGeom::max_plane_threads).
template <typename R> inline int plane_threads_min(const Geom& g) {
  constexpr int mu = PrimeBlock<R, false>::mu;
  return (std::max(plan_threads(g.pf, Emax<R>::v, mu), plan_threads(g.pm, Emax<R>::v, mu)) + 31) / 32 * 32;
}
template <typename R> constexpr int plane_threads_most(int level) { return sizeof(R) == 4 && level < 2 ? 768 : kMaxPassThreads; }

// Threads of a runtime-plan CTA that works on `work` elements, for a launch of `ctas` CTAs with
// `smem` bytes each, from `lo` up to `hi` in steps of 32; `sm_threads` is what the register
// budget leaves resident per SM.  A CTA's time hardly falls with its threads (barriers and
// global latency make up most of it: about 35 + 1.6 work / threads, in microseconds at 3,000
// elements), so what counts is how many run at once: the choice minimises waves times that
// time, a partly filled last wave counted half beyond the first.  The clusters of three fill
// about 0.94 of the CTA places.  Measured on launches of 4 to 6 k-points against about 12 elements per thread
// (FP32 CG plane stage, us per k-point): 45x66x50 23.6 -> 17.8, 50x63x45 23.1 -> 15.9, 36x30x26
// 14.7 -> 14.0, 92x80x75 63.5 -> 57.7.
inline int stage_threads(long work, long ctas, size_t smem, int sm_threads, int lo, int hi) {
  constexpr int kSMs = 148;
  constexpr size_t kSmemSM = 228 * 1024, kSmemCta = 1024;
  lo = std::max(64, (lo + 31) / 32 * 32);
  // At most 24 elements a thread up to 192 threads.  It cuts both ways (us per k-point with and without, FP32
  // CG iteration at 12 k-points): 45x66x50 14.8 and 15.8, 92x80x75 at four 74.5 and 75.8, but 50x63x45 15.2
  // and 13.6, 64^3 21.3 and 19.8: the model has no term for the passes' rounds, which decide here.
  lo = (int)std::max<long>(lo, std::min<long>(std::min(192, hi), (work / 24 + 31) / 32 * 32));
  hi = (int)std::max<long>(lo, std::min<long>(hi, (work / 8 + 31) / 32 * 32));
  int best = lo;
  double best_cost = 1e300;
  for (int t = lo; t <= hi; t += 32) {
    const int per_sm = std::min<int>({sm_threads / t, (int)(kSmemSM / (smem + kSmemCta)), 32});
    if (per_sm < 1) continue;
    const double w = ctas / (0.94 * kSMs * per_sm), up = ceil(w);
    const double cost = (w <= 1.0 ? 1.0 : w + 0.5 * (up - w)) * (35.0 + 1.6 * work / t);
    if (cost < best_cost) {
      best_cost = cost;
      best = t;
    }
  }
  return best;
}

// ... of a plane stage: `planes` planes (3 CTAs each) of precision R.
template <typename R>
inline int plane_threads_rule(const Geom& g, int level, long planes) {
  return stage_threads(g.P, 3 * planes, plane_smem_bytes<R>(g.Lf, g.Lm, g.S), plane_threads_most<R>(level),
                       plane_threads_min<R>(g), 512);
}
// ... and of a pencil stage over `vecs` vectors: with a prime pass, enough that it is one round
// (92 = 4 x 23 in FP64: 51.7 us per k-point with 256 threads, 81.6 with 64).
template <typename R>
inline int pencil_threads_rule(const Geom& g, int level, long vecs) {
  constexpr int TW = PencilTW<R>::v, mu = PrimeBlock<R, true>::mu, ml = PrimeBlock<R, true>::ml;
  int lo = plan_threads(g.ps, Emax<R>::v, mu);
  for (int p = 0; p < g.ps.npass; p++) {
    const int r = g.ps.radix[p];
    if (r > 13) lo = std::max(lo, g.ps.n / r * (((r - 1) / 2 + mu) / mu) * ((TW + ml - 1) / ml));
  }
  return stage_threads((long)g.Ls * TW, 3 * vecs * ((g.P + TW - 1) / TW), pencil_smem_bytes<R>(g.Ls),
                       level < 2 ? 768 : 512, std::min(lo, kPencilThreads), kPencilThreads);
}

// The passes of the plane stage's two axes (a plane of pitch S) and of the pencil stage's, for
// CTAs of `threads` threads.
template <typename R> inline void plane_passes(const Geom& g, int threads, AxisPasses (&ax)[2]) {
  ax[0] = axis_passes(g.pf, g.Lm, g.S, 1, threads, Emax<R>::v);
  ax[1] = axis_passes(g.pm, g.Lf, 1, g.S, threads, Emax<R>::v);
}
template <typename R> inline AxisPasses pencil_passes(const Geom& g, int threads) {
  return axis_passes(g.ps, PencilTW<R>::v, 1, PencilTW<R>::v, threads, Emax<R>::v);
}

// theta_x, theta_y(xy), theta_z(xyz) of wave vector k (FAME_Main/FAME_Matrix_Lambdas.cu:43-70)
inline void lattice_thetas(const fame_lattice& L, const double* k, double th[3]) {
  const double* a = L.lattice_vec_a;
  auto dot = [&](const double* v) { return k[0] * v[0] + k[1] * v[1] + k[2] * v[2]; };
  th[0] = dot(a);
  if (L.simple) {
    th[1] = dot(a + 3);
    th[2] = dot(a + 6);
    return;
  }
  double c1 = 0.0;
  if (a[3] > 0)
    c1 = -(double)L.m[0] / (double)L.grid[0];
  else if (a[3] < 0)
    c1 = 1. - (double)L.m[0] / (double)L.grid[0];
  const double c2 = (double)L.m[2] / (double)L.grid[1];
  const double c3 = (double)L.m[1] / (double)L.grid[0];
  double a2h[3], a3h[3];
  for (int i = 0; i < 3; i++) a2h[i] = c1 * a[i] + a[3 + i];
  for (int i = 0; i < 3; i++) a3h[i] = a[6 + i] - c2 * a2h[i] - c3 * a[i] + L.t1[i];
  th[1] = dot(a2h);
  th[2] = dot(a3h);
}

// Nd of wave vector k: N - 1 at the Gamma point, |k| below 1e-4 for Simple lattices
// (FAME_Main/FAME_Matrix_Lambdas.cu:157) and 1e-3 for General ones (:406), else N.
inline int lattice_reduced_size(const fame_lattice& L, const double* k) {
  const int N = L.grid[0] * L.grid[1] * L.grid[2];
  const double nrm = sqrt(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]);
  return nrm < (L.simple ? 1e-4 : 1e-3) ? N - 1 : N;
}

// The slot of wave vector k.
inline Slot make_slot(const fame_lattice& L, const double* k) {
  Slot sl;
  memset(&sl, 0, sizeof(sl));
  lattice_thetas(L, k, sl.th);
  sl.Nd = lattice_reduced_size(L, k);
  sl.off = L.grid[0] * L.grid[1] * L.grid[2] - sl.Nd;
  sl.active = 1;
  return sl;
}

}  // namespace fame
