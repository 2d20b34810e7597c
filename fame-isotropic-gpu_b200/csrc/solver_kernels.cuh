// CG, invAr and FP64 Lanczos kernels.
#pragma once
#include "state.cuh"

namespace fame {

// ------------------------------------------------------------------ tables
// Per-k tables (FAME_Main/FAME_Matrix_Lambdas.cu:77-244 Simple, :288-489 General)
// computed on the device: one thread per table entry, FP64 sincospi.  General lattices:
// also D_kz (…Lambdas.cu:389-400) of every point in the precisions asked for (dkz64, dkz32; N
// values per slot), which the plane stages read instead of evaluating it six times per CG
// iteration.
// k_tables_of: the one k-point of an operator apply comes as an argument and is stored as
// slot 0 too (a copy of 48 bytes from the host in front of the kernels cost more than they do).  It also
// clears the fault marker, which an earlier call may have left set.
__device__ __forceinline__ void tables_of(const Geom& g, const Slot& sl, int slot, double2* tabs, double m1, double m2,
                                          double m3, double2* dkz64, float2* dkz32) {
  double2* t = tabs + (size_t)slot * g.tab_stride;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int Nx = g.Nx, Ny = g.Ny, Nz = g.Nz;
  if (!g.general) {
    // Lambda_d[n] = (e^{i 2 pi (n + theta_d)/N_d} - 1)/h_d,  D_d[n] = e^{i 2 pi theta_d n / N_d}
    if (i < Nx) {
      double2 e = expipi(2.0 * (i + sl.th[0]) / Nx);
      t[g.oLx + i] = make_double2((e.x - 1.0) / g.hx, e.y / g.hx);
      t[g.oDx + i] = expipi(2.0 * sl.th[0] * i / Nx);
    }
    if (i < Ny) {
      double2 e = expipi(2.0 * (i + sl.th[1]) / Ny);
      t[g.oLy + i] = make_double2((e.x - 1.0) / g.hy, e.y / g.hy);
      t[g.oDy + i] = expipi(2.0 * sl.th[1] * i / Ny);
    }
    if (i < Nz) {
      double2 e = expipi(2.0 * (i + sl.th[2]) / Nz);
      t[g.oLz + i] = make_double2((e.x - 1.0) / g.hz, e.y / g.hz);
      t[g.oDz + i] = expipi(2.0 * sl.th[2] * i / Nz);
    }
  } else {
    const double c1 = (m1 * m3) / ((double)Ny * Nx) - (m2 / Nx);
    const double c2 = -(m3 / Ny);
    if (i < Nx) {
      double2 e = expipi(2.0 * (i + sl.th[0]) / Nx);
      t[g.oLx + i] = make_double2((e.x - 1.0) / g.hx, e.y / g.hx);
      t[g.oDkx + i] = expipi(2.0 * sl.th[0] * i / Nx);
    }
    if (i < Nx * Ny) {
      const int x = i / Ny, y = i - x * Ny;
      // mxy = -m1*x/Nx + y (…Lambdas.cu:333-335), Lambda_y over (x, y)
      const double mxy = (-(m1 / Nx) * x) + y;
      double2 e = expipi(2.0 * (mxy + sl.th[1]) / Ny);
      t[g.oLy + i] = make_double2((e.x - 1.0) / g.hy, e.y / g.hy);
      // D_ky[x, y] = e^{i 2 pi (theta_xy - m1 x / Nx) y / Ny} (…Lambdas.cu:382-388)
      t[g.oDky + i] = expipi(2.0 * (sl.th[1] + x * (-m1 / Nx)) * y / Ny);
      // phase base of Lambda_z and D_kz: phi = (theta_xyz + c1 x + c2 y)
      const double ph = sl.th[2] + c1 * x + c2 * y;
      t[g.oExy + i] = expipi(2.0 * ph / Nz);
      t[g.oPhi + i] = make_double2(ph, 0.0);
    }
    if (i < Nz) t[g.oWz + i] = expipi(2.0 * i / Nz);
    if (dkz64 || dkz32) {
      for (int e = i; e < g.N; e += gridDim.x * blockDim.x) {
        const int xy = (int)((unsigned)e / (unsigned)Nz), z = e - xy * Nz;
        const int x = (int)((unsigned)xy / (unsigned)Ny), y = xy - x * Ny;
        const double2 d = expipi((sl.th[2] + c1 * x + c2 * y) * z * g.tnz);
        if (dkz64) dkz64[(size_t)slot * g.N + e] = d;
        if (dkz32) dkz32[(size_t)slot * g.N + e] = to_f(d);
      }
    }
  }
}
__global__ void k_tables(Geom g, const Slot* slots, double2* tabs, double m1, double m2, double m3, double2* dkz64,
                         float2* dkz32) {
  FAME_COUNT_LAUNCH();
  tables_of(g, slots[blockIdx.y], blockIdx.y, tabs, m1, m2, m3, dkz64, dkz32);
}
__global__ void k_tables_of(Geom g, Slot sl, Slot* slots, double2* tabs, double m1, double m2, double m3, double2* dkz64,
                            float2* dkz32, int* fault) {
  FAME_COUNT_LAUNCH();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    slots[0] = sl;
    *fault = 0;
  }
  tables_of(g, sl, 0, tabs, m1, m2, m3, dkz64, dkz32);
}


// Global index of reduced element i (0 <= i < 2*Nd) to its full frequency index.
__device__ __forceinline__ int full_index(int i, int Nd, int off) { return (i < Nd ? i : i - Nd) + off; }

struct VecArgs {
  Geom g;
  const Slot* slots;
  const double2* tabs;
  long vstride;            // per-slot stride of reduced vectors
  CgState* cg;
  double* partials;
  unsigned* counters;      // [nslots] slot tickets, [nslots] grid ticket
  Cond cond;
  int nslots;
};

// ---------------------------------------------------------------- invAr prologue
// rhs = u / sqrt(Lambda_q) (…invAr.cu:26), CG start x = 0, r = rhs (CG.cu:30-33).
// Plain FP64 (MIXED = false): r64 is the CG's residual (k_plane_cg takes x = 0 at k = 1 as
// read).  Mixed, and FP64 with refinement: b = rhs, y = x64 = 0, r64 = b, and the outer refinement
// loop state is initialised (REFINE).
struct LzArgs {
  double2* U;              // [nslots][nstep + 1][ustride]
  long ustride;            // column stride (elements)
  int nstep, nwant;
  int nkeep;               // Lanczos vectors a restart after the first keeps (keep_vectors, >= nwant)
  double* T0;              // [nslots][nstep]
  double* T1;              // [nslots][nstep]
  double* h;               // [nslots][nstep+2] reorthogonalisation coefficients
  LzState* lz;
  int* prof;               // [nslots][3]: ls_iter, es_iter (reference Profile counters), FP64 refinements
  int* status;             // [nslots] per-k status bits (kStatus*)
};

// Per-k status bits: the tridiagonal QL iteration failed; Lanczos ended at es_maxit
// restarts unconverged (Lanczos_Isotropic.cu:84-85 prints this case); an A_r^-1 solve
// ended at ls_maxit (plain) or at the refinement cap (mixed) above ls_tol (CG.cu:81-84
// prints this case).  The host reports any of them as FAME_ERR_NO_CONVERGENCE.
constexpr int kStatusQL = 1, kStatusLanczos = 2, kStatusCG = 4;

// whether Lanczos step j is one of this slot's
__device__ __forceinline__ bool lz_live(const LzArgs& L, int slot, int j) {
  return !L.lz[slot].converged && j >= L.lz[slot].keep;
}

__device__ __forceinline__ double2* ucol(const LzArgs& L, int slot, int c) {
  return L.U + ((size_t)slot * (L.nstep + 1) + c) * L.ustride;
}

template <bool REFINE>
__global__ void __launch_bounds__(256) k_invar_pro(VecArgs va, LzArgs L, int j, double2* r64,
                                                   double2* x64, double2* b64, LsParams ls, const LsParams* lsp) {
  FAME_COUNT_LAUNCH();
  if (lsp) ls = *lsp;
  const double tol2 = ls.tol2;
  const int maxit = ls.maxit;
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  CgState* st = va.cg + slot;
  const bool live = sl.active && lz_live(L, slot, j);
  if (live) {
    const long b = (long)slot * va.vstride;
    const double2* tab = va.tabs + (size_t)slot * va.g.tab_stride;
    const double2* u = ucol(L, slot, j);
    const int Nd = sl.Nd, n = 2 * Nd;
    double acc[1] = {0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const double s = lq_sqrt_at(va.g, tab, full_index(i, Nd, sl.off));
      const double2 v = make_double2(u[i].x / s, u[i].y / s);
      r64[b + i] = v;
      if (REFINE) {
        x64[b + i] = make_double2(0.0, 0.0);
        b64[b + i] = v;
      }
      acc[0] += cabs2(v);
    }
    __shared__ double sred[32];
    block_reduce<1>(acc, sred);
    double tot[1];
    if (slot_reduce<1>(acc, va.partials + (size_t)slot * gridDim.x, va.counters + slot, blockIdx.x,
                       gridDim.x, tot)) {
      if (threadIdx.x == 0) {
        if (!REFINE) {
          st->r1 = tot[0];
          st->tol2 = tol2;
          st->iter = 1;
          st->maxit = maxit;
          st->active = (tot[0] > tol2) && (1 <= maxit);
        } else {
          st->rr = tot[0];
          st->otol2 = tol2;
          st->scale = 1.0 / sqrt(tot[0] > 0 ? tot[0] : 1.0);
          st->outer = 0;
          st->outer_max = 40;  // refinement steps per solve; each gains ~5 digits
          st->rounded = 0;
          st->total = 0;
          st->outer_total = 0;
          st->outer_active = tot[0] > tol2;
          st->iter = 1;
          st->active = 0;
        }
        __threadfence();
      }
    }
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->active = 0;
    st->outer_active = 0;
  }
  if (grid_last(va.counters + va.nslots, gridDim.x * gridDim.y * gridDim.z)) {
    if (threadIdx.x == 0) {
      int any = 0;
      for (int q = 0; q < va.nslots; q++)
        any |= va.slots[q].active && (REFINE ? va.cg[q].outer_active : va.cg[q].active);
      start_cond(va.cond, any);
    }
  }
}

// Start of one FP32 inner solve: r32 = (float)(r64 * scale) (x32 = 0 is implied); stop when
// ||r32|| <= tau' ||r32_0|| or after `maxit` products, where tau' = max(tau,
// ls_tol / (2 ||r64||)): a refinement step never reduces the residual further than
// the outer tolerance needs (outer_tol2 = ls_tol^2).
__global__ void __launch_bounds__(256) k_cg32_init(VecArgs va, const double2* r64, float2* r32, double tau2, int maxit, double outer_tol2,
                                                   Cond outer_reset) {
  FAME_COUNT_LAUNCH();
  if ((threadIdx.x | blockIdx.x | blockIdx.y | blockIdx.z) == 0) set_cond(outer_reset, 0);
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  CgState* st = va.cg + slot;
  const bool live = sl.active && st->outer_active;
  if (live) {
    const long b = (long)slot * va.vstride;
    const int n = 2 * sl.Nd;
    const double sc = st->scale;
    double acc[1] = {0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const float2 v = make_float2((float)(r64[b + i].x * sc), (float)(r64[b + i].y * sc));
      r32[b + i] = v;
      acc[0] += (double)cabs2(v);
    }
    __shared__ double sred[32];
    block_reduce<1>(acc, sred);
    double tot[1];
    if (slot_reduce<1>(acc, va.partials + (size_t)slot * gridDim.x, va.counters + slot, blockIdx.x,
                       gridDim.x, tot)) {
      if (threadIdx.x == 0) {
        const double need = st->rr > 0 ? 0.25 * outer_tol2 / st->rr : 0.0;
        st->r1 = tot[0];
        st->tol2 = (need > tau2 ? need : tau2) * tot[0];
        st->iter = 1;
        st->maxit = maxit;
        st->active = (tot[0] > st->tol2) && (1 <= maxit);
        __threadfence();
      }
    }
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->active = 0;
  }
  if (grid_last(va.counters + va.nslots, gridDim.x * gridDim.y * gridDim.z)) {
    if (threadIdx.x == 0) {
      int any = 0;
      for (int q = 0; q < va.nslots; q++) any |= va.slots[q].active && va.cg[q].active;
      start_cond(va.cond, any);
    }
  }
}

// FP64 CG with restarts from the true residual, for a permittivity contrast beyond 32
// (refine64_tol): the start of one CG solve, from r64 = b - A y (r64 is the CG's start residual as it
// stands).  It ends at ls_tol or after a reduction by ls.floor2 (squared), where the three-term recurrences stop
// being worth more; ls.maxit bounds the products over all restarts.  A restart that has not halved the true
// residual has reached what rounding leaves: that counts as solved where it is within the
// rounding of the form with search directions, ls.rounding2 ||b||^2, which could not tell either.
__global__ void __launch_bounds__(32) k_cg64_init(VecArgs va, LsParams ls, const LsParams* lsp, Cond outer_reset) {
  FAME_COUNT_LAUNCH();
  if (lsp) ls = *lsp;
  if (threadIdx.x == 0) set_cond(outer_reset, 0);
  int any = 0;
  for (int q = threadIdx.x; q < va.nslots; q += 32) {
    CgState* st = va.cg + q;
    st->active = 0;
    if (!va.slots[q].active || !st->outer_active) continue;
    const double rr = st->rr;
    if (st->outer == 0) st->bb = rr;
    const bool halved = st->outer == 0 || rr <= 0.25 * st->rr_old;
    if (!halved || st->total >= ls.maxit) {
      st->rounded = !halved && rr <= ls.rounding2 * st->bb;
      st->outer_active = 0;
      continue;
    }
    st->rr_old = rr;
    st->r1 = rr;
    st->tol2 = fmax(st->otol2, ls.floor2 * rr);
    st->iter = 1;
    st->maxit = ls.maxit - st->total;
    st->active = 1;
    any = 1;
  }
  any = __any_sync(0xffffffffu, any);
  if (threadIdx.x == 0) start_cond(va.cond, any);
}

// The end of it: y += x, the CG's solution in the buffer of its last iteration's parity.
__global__ void __launch_bounds__(256) k_cg64_add(VecArgs va, double2* y, const double2* x64, const double2* x64b) {
  FAME_COUNT_LAUNCH();
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  const CgState* st = va.cg + slot;
  if (!sl.active || !st->outer_active || st->iter == 1) return;
  const long b = (long)slot * va.vstride;
  const double2* xs = (st->iter & 1) ? x64 : x64b;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * sl.Nd; i += gridDim.x * blockDim.x)
    y[b + i] = cadd(y[b + i], xs[b + i]);
}

// invAr epilogue: w = x / sqrt(Lambda_q) into U[:, j+1] (…invAr.cu:45) and
// alpha_j = Re<w, u_j> (Lanczos_decomp_gpu.cu:64-66); profile counters
// (…invAr.cu:41-43: ls_iter += k, es_iter++).  MODE: plain FP64 CG, FP64 with refinement, mixed.
enum InvMode { INV_PLAIN = 0, INV_REFINE64 = 1, INV_MIXED = 2 };
template <int MODE>
__global__ void __launch_bounds__(256) k_invar_epi(VecArgs va, LzArgs L, int j, const double2* x64,
                                                   const double2* x64b) {
  FAME_COUNT_LAUNCH();
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  if (!sl.active || !lz_live(L, slot, j)) return;
  const long b = (long)slot * va.vstride;
  const double2* tab = va.tabs + (size_t)slot * va.g.tab_stride;
  const double2* u = ucol(L, slot, j);
  double2* w = ucol(L, slot, j + 1);
  const int Nd = sl.Nd, n = 2 * Nd;
  // plain FP64: the solution is in the buffer of the last iteration's parity (x64 odd, x64b
  // even), and zero if the CG did no product; else the refinement's sum, in x64
  constexpr bool kSum = MODE != INV_PLAIN;
  const int iter = va.cg[slot].iter;
  const double2* xs = kSum || (iter & 1) ? x64 : x64b;
  const bool none = !kSum && iter == 1;
  double acc[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double s = lq_sqrt_at(va.g, tab, full_index(i, Nd, sl.off));
    const double2 xx = none ? make_double2(0.0, 0.0) : xs[b + i];
    const double2 v = make_double2(xx.x / s, xx.y / s);
    w[i] = v;
    acc[0] += v.x * u[i].x + v.y * u[i].y;
  }
  __shared__ double sred[32];
  block_reduce<1>(acc, sred);
  double tot[1];
  if (slot_reduce<1>(acc, va.partials + (size_t)slot * gridDim.x, va.counters + slot, blockIdx.x,
                     gridDim.x, tot)) {
    if (threadIdx.x == 0) {
      L.T0[slot * L.nstep + j] = tot[0];
      const CgState* st = va.cg + slot;
      L.prof[slot * 3 + 0] += MODE == INV_MIXED ? st->total : MODE == INV_REFINE64 ? st->total + 1 : st->iter;
      L.prof[slot * 3 + 1] += 1;
      if (kSum) L.prof[slot * 3 + 2] += st->outer_total;
      // (a NaN ends the loops and is no convergence either)
      const bool solved = kSum ? st->rr <= st->otol2 || (MODE == INV_REFINE64 && st->rounded) : st->r1 <= st->tol2;
      if (!solved) L.status[slot] |= kStatusCG;
    }
  }
}

// ---------------------------------------------------------------- Lanczos step
// w' = w - alpha_j u_j - beta_{j-1} u_{j-1}; ||w'||^2 and, for j >= 1, the
// coefficients <u_i, w'> (i <= j) of one classical Gram-Schmidt pass.  The
// reference normalises first and then runs one modified Gram-Schmidt pass
// without renormalising (Lanczos_decomp_gpu.cu:68-87); both leave u_{j+1}
// orthogonal to the basis to rounding level.
constexpr int kLzRows = 2048;  // rows per CTA, staged in shared memory (32 KB)

__global__ void __launch_bounds__(256) k_lz_dots(VecArgs va, LzArgs L, int j) {
  FAME_COUNT_LAUNCH();
  __shared__ double2 wsh[kLzRows];
  __shared__ double red[(2 * 64 + 1) * 8];  // [value][warp]
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  if (!sl.active || !lz_live(L, slot, j)) return;
  const int n = 2 * sl.Nd;
  const int r0 = blockIdx.x * kLzRows;
  const int rows = min(kLzRows, n - r0);
  const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double al = L.T0[slot * L.nstep + j];
  const double be = j > 0 ? L.T1[slot * L.nstep + j - 1] : 0.0;
  const double2* w = ucol(L, slot, j + 1);
  const double2* uj = ucol(L, slot, j);
  const double2* ujm = j > 0 ? ucol(L, slot, j - 1) : uj;
  const int nval = 1 + (j > 0 ? 2 * (j + 1) : 0);
  double nrm = 0.0;
  for (int q = threadIdx.x; q < rows; q += blockDim.x) {
    const int i = r0 + q;
    double2 v = w[i];
    v.x -= al * uj[i].x + be * ujm[i].x;
    v.y -= al * uj[i].y + be * ujm[i].y;
    wsh[q] = v;
    nrm += cabs2(v);
  }
  for (int o = 16; o > 0; o >>= 1) nrm += __shfl_down_sync(0xffffffffu, nrm, o);
  if (lane == 0) red[0 * 8 + wid] = nrm;
  __syncthreads();
  if (j > 0) {
    for (int c = 0; c <= j; c++) {
      const double2* u = ucol(L, slot, c);
      double dr = 0.0, di = 0.0;
      for (int q = threadIdx.x; q < rows; q += blockDim.x) {
        const double2 a = u[r0 + q], b = wsh[q];
        dr += a.x * b.x + a.y * b.y;  // conj(u) w'
        di += a.x * b.y - a.y * b.x;
      }
      for (int o = 16; o > 0; o >>= 1) {
        dr += __shfl_down_sync(0xffffffffu, dr, o);
        di += __shfl_down_sync(0xffffffffu, di, o);
      }
      if (lane == 0) {
        red[(1 + 2 * c) * 8 + wid] = dr;
        red[(2 + 2 * c) * 8 + wid] = di;
      }
    }
  }
  __syncthreads();
  // per-CTA partials in global memory, last CTA of the slot sums them in order
  double* part = va.partials + (size_t)slot * gridDim.x * (2 * 64 + 1);
  for (int v = threadIdx.x; v < nval; v += blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < nw; q++) s += red[v * 8 + q];
    part[(size_t)blockIdx.x * (2 * 64 + 1) + v] = s;
  }
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(va.counters + slot, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // one warp per value, lanes strided over the CTAs' partials (a fixed order)
  __syncthreads();
  for (int v = wid; v < nval; v += nw) {
    const double s = warp_sum_strided_cg(part + v, gridDim.x, 2 * 64 + 1);
    if (lane == 0) red[v] = s;  // reuse (every warp has read its own red entries)
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double beta = sqrt(red[0]);
    L.T1[slot * L.nstep + j] = beta;
    double* h = L.h + (size_t)slot * 2 * (L.nstep + 2);
    for (int v = 1; v < nval; v++) h[v - 1] = red[v];
    va.counters[slot] = 0u;
  }
}

// u_{j+1} = (w' - sum_i <u_i, w'> u_i) / beta_j
__global__ void __launch_bounds__(256) k_lz_update(VecArgs va, LzArgs L, int j) {
  FAME_COUNT_LAUNCH();
  __shared__ double2 hs[64];
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  if (!sl.active || !lz_live(L, slot, j)) return;
  const int n = 2 * sl.Nd;
  const double beta = L.T1[slot * L.nstep + j];
  const double inv = 1.0 / beta;
  const double al = L.T0[slot * L.nstep + j];
  const double be = j > 0 ? L.T1[slot * L.nstep + j - 1] : 0.0;
  const double* h = L.h + (size_t)slot * 2 * (L.nstep + 2);
  if (j > 0)
    for (int c = threadIdx.x; c <= j; c += blockDim.x) hs[c] = make_double2(h[2 * c], h[2 * c + 1]);
  __syncthreads();
  double2* w = ucol(L, slot, j + 1);
  const double2* uj = ucol(L, slot, j);
  const double2* ujm = j > 0 ? ucol(L, slot, j - 1) : uj;
  const double2* u0 = ucol(L, slot, 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double2 v = w[i];
    v.x -= al * uj[i].x + be * ujm[i].x;
    v.y -= al * uj[i].y + be * ujm[i].y;
    if (j > 0) {
      const double2* uc = u0 + i;
      // (one column at a time: with 4 or 8 loads of a thread in flight the 40 steps of a 96^3 k-point take
      // 4.82 and 5.09 ms, with 1 or 2 4.57; the resident warps keep DRAM busy)
#pragma unroll 1
      for (int c = 0; c <= j; c++) {
        const double2 u = uc[c * L.ustride];
        const double2 hc = hs[c];
        v.x -= hc.x * u.x - hc.y * u.y;
        v.y -= hc.x * u.y + hc.y * u.x;
      }
    }
    w[i] = make_double2(v.x * inv, v.y * inv);
  }
}

// A uniform number in [-1, 1) from an index (splitmix64 finaliser).
__device__ __forceinline__ double hash_unit(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  return (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// Start vector e_M (Lanczos_decomp_gpu.cu:93-107) plus a fixed pseudo-random
// perturbation of total norm 1e-12, and the Lanczos state.  When a lattice
// symmetry makes A_r block diagonal (a permittivity independent of z decouples the
// z frequencies), e_M lies in one block and exact Krylov spaces never leave it; the
// reference escapes through cuFFT rounding noise, which the perturbation stands in
// for, so the same lowest bands are found.
// ls_out (an operator apply): where the solve's bounds go, for its graph.
__global__ void k_lz_init(VecArgs va, LzArgs L, LsParams* ls_out, LsParams ls) {
  FAME_COUNT_LAUNCH();
  const int slot = blockIdx.z;
  if (ls_out && (threadIdx.x | blockIdx.x | blockIdx.z) == 0) *ls_out = ls;
  const Slot sl = va.slots[slot];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    L.lz[slot].converged = 0;
    L.lz[slot].restarts = 0;
    L.lz[slot].nconv = 0;
    L.lz[slot].keep = 0;
    L.prof[slot * 3] = 0;
    L.prof[slot * 3 + 1] = 0;
    L.prof[slot * 3 + 2] = 0;
  }
  if (!sl.active) return;
  double2* u = ucol(L, slot, 0);
  const int n = 2 * sl.Nd;
  const double eta = 1e-12 / sqrt((double)n);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    u[i] = make_double2((i == n - 1 ? 1.0 : 0.0) + eta * hash_unit(2ull * i), eta * hash_unit(2ull * i + 1));
}

// ---------------------------------------------------------------- tridiagonal stage
// One warp per slot.  (1) Eigen-decomposition of the symmetric tridiagonal T
// (diag T0, off-diag T1) by the implicit QL method with Wilkinson shifts (Bowdler,
// Martin, Reinsch and Wilkinson, "The QR and QL algorithms for symmetric matrices",
// Numer. Math. 11, 1968), eigenvalues sorted in descending order as zpteqr returns
// them (Lanczos_Isotropic.cu:53).  (2) The convergence test of Lanczos_Isotropic.cu:58-72.
// (3) If not converged: the lock/purge restart of Lanczos_LockPurge_gpu.cu:7-48
// (exact shifts = unwanted Ritz values, GVqrrq_g steps, :95-190), applied to an
// identity matrix G of order nstep+1 instead of to U, so that U is updated later by
// one product U*G[:, 0..keep] (k_restart).
constexpr int kMaxStep = 64;

struct TriArgs {
  LzArgs L;
  const Slot* slots;
  double* theta;   // [nslots][nstep] Ritz values (descending)
  double* Z;       // [nslots][nstep*nstep] eigenvectors, column-major (z[r + c*nstep])
  double* G;       // [nslots][(nstep+1)*(nkeep+1)] restart transform, column-major
  double tol;
  int maxit;
  Cond cond;       // "some slot needs another restart"
  int nslots;
  int* status;     // [nslots] bits: kStatusQL, kStatusLanczos, kStatusCG (0: converged)
  unsigned* ctr;   // grid ticket counter
  int first;       // 1: the call before the restart loop (starts it), 0: end of a loop body
};

// dynamic shared memory of k_tridiag for nstep = n
inline size_t tridiag_smem(int n) {
  return sizeof(double) * ((size_t)n * n + (size_t)(n + 1) * (n + 1) + 8 * (size_t)n) + sizeof(int) * n;
}

__device__ void givens_ref(double a, double b, double& c, double& s, double& r) {
  // given_rotation (Lanczos_LockPurge_gpu.cu:245-265)
  double t, u;
  if (fabs(a) > fabs(b)) {
    t = b / a;
    u = (fabs(a) / a) * sqrt(1 + t * t);
    c = 1.0 / u;
    s = c * t;
    r = a * u;
    s = -s;
  } else {
    t = a / b;
    u = (fabs(b) / b) * sqrt(1 + t * t);
    s = 1.0 / u;
    c = s * t;
    r = b * u;
    s = -s;
  }
}

__global__ void __launch_bounds__(32) k_tridiag(TriArgs a) {
  FAME_COUNT_LAUNCH();
  extern __shared__ __align__(16) double tsm[];
  const LzArgs& L = a.L;
  const int n = L.nstep, nw = L.nwant, lane = threadIdx.x;
  double* Zs = tsm;                       // n*n
  double* Gs = Zs + n * n;                // (n+1)^2
  double* d = Gs + (n + 1) * (n + 1);     // 8 vectors of n
  double* e = d + n;
  double* T0 = e + n;
  double* T1 = T0 + n;
  double* T2 = T1 + n;
  double* T3 = T2 + n;
  double* cc = T3 + n;
  double* ss = cc + n;
  int* order = reinterpret_cast<int*>(ss + n);
  __shared__ int fail;
  const int slot = blockIdx.x;
  LzState* lz = L.lz + slot;
  const bool live = a.slots[slot].active && !lz->converged;
  if (live) {
    for (int i = lane; i < n; i += 32) {
      d[i] = L.T0[slot * n + i];
      e[i] = i < n - 1 ? L.T1[slot * n + i] : 0.0;
      T0[i] = d[i];
      T1[i] = L.T1[slot * n + i];
    }
    for (int i = lane; i < n * n; i += 32) Zs[i] = (i % (n + 1)) == 0 ? 1.0 : 0.0;  // Z[r + c*n]
    if (lane == 0) fail = 0;
    __syncwarp();
    // ---- implicit QL; lane 0 runs the scalar recurrence, all lanes rotate Z rows
    for (int l = 0; l < n; l++) {
      int iter = 0;
      while (true) {
        int m = l;
        for (; m < n - 1; m++) {
          const double dd = fabs(d[m]) + fabs(d[m + 1]);
          if (fabs(e[m]) <= 1e-300 || fabs(e[m]) + dd == dd) break;
        }
        if (m == l) break;
        if (++iter > 60) {
          if (lane == 0) fail = 1;
          break;
        }
        double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
        double r = hypot(g, 1.0);
        g = d[m] - d[l] + e[l] / (g + (g >= 0 ? fabs(r) : -fabs(r)));
        double s = 1.0, c = 1.0, p = 0.0;
        int i = m - 1;
        bool underflow = false;
        for (; i >= l; i--) {
          const double f = s * e[i], b = c * e[i];
          r = hypot(f, g);
          __syncwarp();
          if (lane == 0) e[i + 1] = r;
          if (r == 0.0) {
            __syncwarp();
            if (lane == 0) {
              d[i + 1] -= p;
              e[m] = 0.0;
            }
            underflow = true;
            __syncwarp();
            break;
          }
          s = f / r;
          c = g / r;
          g = d[i + 1] - p;
          r = (d[i] - g) * s + 2.0 * c * b;
          p = s * r;
          __syncwarp();
          if (lane == 0) d[i + 1] = g + p;
          g = c * r - b;
          for (int k = lane; k < n; k += 32) {
            const double fz = Zs[k + (i + 1) * n];
            Zs[k + (i + 1) * n] = s * Zs[k + i * n] + c * fz;
            Zs[k + i * n] = c * Zs[k + i * n] - s * fz;
          }
          __syncwarp();
        }
        if (underflow) continue;
        __syncwarp();
        if (lane == 0) {
          d[l] -= p;
          e[l] = g;
          e[m] = 0.0;
        }
        __syncwarp();
      }
    }
    __syncwarp();
    // ---- sort descending (selection on lane 0; n <= 64)
    if (lane == 0) {
      for (int i = 0; i < n; i++) order[i] = i;
      for (int i = 0; i < n; i++) {
        int best = i;
        for (int k = i + 1; k < n; k++)
          if (d[order[k]] > d[order[best]]) best = k;
        const int t = order[i];
        order[i] = order[best];
        order[best] = t;
      }
    }
    __syncwarp();
    double* th = a.theta + (size_t)slot * n;
    double* Zg = a.Z + (size_t)slot * n * n;
    for (int i = lane; i < n; i += 32) th[i] = d[order[i]];
    for (int q = lane; q < n * n; q += 32) {
      const int r = q % n, c = q / n;
      Zg[q] = Zs[r + order[c] * n];
    }
    __syncwarp();
    // ---- convergence (Lanczos_Isotropic.cu:58-72): |beta_last * z(last, i)| < tol
    int conv = 0;
    if (lane == 0) {
      const double bl = L.T1[slot * n + n - 1];
      for (int i = 0; i < nw; i++) {
        const double res = bl * fabs(Zs[(n - 1) + order[i] * n]);
        if (res < a.tol) conv++;
        else break;
      }
      lz->nconv = conv;
      if (fail) a.status[slot] |= kStatusQL;
    }
    conv = __shfl_sync(0xffffffffu, conv, 0);
    const bool done = conv == nw || fail;
    if (done) {
      if (lane == 0) lz->converged = 1;
    } else if (lz->restarts >= a.maxit) {
      if (lane == 0) {
        lz->converged = 1;
        a.status[slot] |= kStatusLanczos;
      }
    } else {
      // ---- lock & purge on G (order nstep+1)
      const int nk = lz->restarts == 0 ? nw : L.nkeep;
      const int n1 = n + 1;
      for (int q = lane; q < n1 * n1; q += 32) Gs[q] = (q % (n1 + 1)) == 0 ? 1.0 : 0.0;
      __syncwarp();
      for (int jj0 = 0; jj0 < n - nk; jj0++) {
        const int nn = n - jj0;
        const double shift = d[order[nk + jj0]];
        if (lane == 0) {
          // GVqrrq_g(T0, T1, T2, T3, c, s, shift, nn)
          for (int i = 0; i < nn - 1; i++) T3[i] = T1[i];
          for (int i = 0; i < nn; i++) T0[i] -= shift;
          for (int i = 0; i < nn - 1; i++) {
            double ci, si, r;
            givens_ref(T0[i], T1[i], ci, si, r);
            cc[i] = ci;
            ss[i] = si;
            T0[i] = r;
            T1[i] = 0.0;
            const double aa = T3[i], bb = T0[i + 1];
            T3[i] = ci * aa - si * bb;
            T0[i + 1] = si * aa + ci * bb;
            if (i < nn - 2) {
              T2[i] = -si * T3[i + 1];
              T3[i + 1] = ci * T3[i + 1];
            }
          }
          double R0 = T0[0], R1 = T3[0], R2 = T1[0], R3 = T0[1];
          T0[0] = cc[0] * R0 - ss[0] * R1;
          T3[0] = ss[0] * R0 + cc[0] * R1;
          T1[0] = cc[0] * R2 - ss[0] * R3;
          T0[1] = ss[0] * R2 + cc[0] * R3;
          for (int i = 1; i < nn - 1; i++) {
            const double q0 = T3[i - 1], q1 = T2[i - 1], q2 = T0[i], q3 = T3[i], q4 = T1[i], q5 = T0[i + 1];
            T3[i - 1] = cc[i] * q0 - ss[i] * q1;
            T2[i - 1] = ss[i] * q0 + cc[i] * q1;
            T0[i] = cc[i] * q2 - ss[i] * q3;
            T3[i] = ss[i] * q2 + cc[i] * q3;
            T1[i] = cc[i] * q4 - ss[i] * q5;
            T0[i + 1] = ss[i] * q4 + cc[i] * q5;
          }
          for (int i = 0; i < nn - 1; i++) T1[i] = (T1[i] + T3[i]) / 2.0;
          for (int i = 0; i < nn; i++) T0[i] += shift;
          // the final rotation couples column nn-1 with the residual column nn:
          // (c, s) = (T1[nn-2], s[nn-2] * T1[nn-1]) (Lanczos_LockPurge_gpu.cu:30-31)
          ss[nn - 1] = ss[nn - 2] * T1[nn - 1];
          cc[nn - 1] = T1[nn - 2];
        }
        __syncwarp();
        // Zdrot(U[:, jj+1], U[:, jj], c, s) for jj < nn-1, then (c, s) = (T1[nn-2], s[nn-2]*T1[nn-1])
        for (int jj = 0; jj < nn; jj++) {
          const double c = cc[jj];
          const double s = ss[jj];
          for (int r = lane; r < n1; r += 32) {
            const double x = Gs[r + (jj + 1) * n1], y = Gs[r + jj * n1];
            Gs[r + (jj + 1) * n1] = c * x + s * y;
            Gs[r + jj * n1] = -s * x + c * y;
          }
          __syncwarp();
        }
        // normalise column nn-1, purge T0/T1[nn-1] and column nn
        double nrm = 0.0;
        for (int r = lane; r < n1; r += 32) nrm += Gs[r + (nn - 1) * n1] * Gs[r + (nn - 1) * n1];
        for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
        nrm = sqrt(nrm);
        for (int r = lane; r < n1; r += 32) {
          Gs[r + (nn - 1) * n1] /= nrm;
          Gs[r + nn * n1] = 0.0;
        }
        __syncwarp();
        if (lane == 0) {
          T1[nn - 2] = nrm;
          T0[nn - 1] = 0.0;
          T1[nn - 1] = 0.0;
        }
        __syncwarp();
      }
      double* Gg = a.G + (size_t)slot * n1 * (L.nkeep + 1);
      for (int q = lane; q < n1 * (nk + 1); q += 32) Gg[q] = Gs[q];
      for (int i = lane; i < n; i += 32) {
        L.T0[slot * n + i] = T0[i];
        L.T1[slot * n + i] = T1[i];
      }
      __syncwarp();  // every lane has read lz->restarts
      if (lane == 0) {
        lz->restarts++;
        lz->keep = nk;
      }
    }
  }
  __syncwarp();
  // grid-wide "any slot still restarting" (gridDim.x == nslots, one warp each)
  __shared__ bool last;
  __threadfence();
  if (lane == 0) last = atomicAdd(a.ctr, 1u) == (unsigned)gridDim.x - 1;
  __syncwarp();
  if (last && lane == 0) {
    __threadfence();
    *a.ctr = 0u;
    int any = 0;
    for (int q = 0; q < a.nslots; q++) any |= a.slots[q].active && !a.L.lz[q].converged;
    if (a.first)
      start_cond(a.cond, any);
    else
      decide_cond(a.cond, any);
  }
}

// ---------------------------------------------------------------- U * G products
// The restart: U[:, c] = sum_r U[:, r] * G[r, c] for c <= keep, in place (G real, column-major, order
// nstep + 1).  A CTA holds kRestartRows rows of all nstep + 1 columns in shared memory, so U is read once
// and needs no second copy: with the products out of place, a slot's basis took nkeep + 1 columns more (of 70 at nwant 10
// of 40, 28 MB each at 96^3) and U was read once per 8 new columns (two restarts of a 96^3 k-point, to 11 and
// 29 columns: 1.71 ms out of place, 1.38 so).  Eight warps share the new columns, a lane to a row, four
// columns at a time.
constexpr int kRestartRows = 32;
inline size_t restart_smem(int nstep, int nkeep) {
  return sizeof(double2) * kRestartRows * (nstep + 1) + sizeof(double) * (nstep + 1) * (nkeep + 1);
}
__global__ void __launch_bounds__(256) k_restart(VecArgs va, LzArgs L, const double* G) {
  FAME_COUNT_LAUNCH();
  extern __shared__ __align__(16) unsigned char rsm[];
  if ((threadIdx.x | blockIdx.x | blockIdx.y | blockIdx.z) == 0) set_cond(va.cond, 0);
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  if (!sl.active || L.lz[slot].converged) return;
  const int n1 = L.nstep + 1, nc = L.lz[slot].keep + 1;
  double2* us = reinterpret_cast<double2*>(rsm);                    // [n1][kRestartRows]
  double* Gs = reinterpret_cast<double*>(us + kRestartRows * n1);  // [nc][n1]
  const double* Gg = G + (size_t)slot * n1 * (L.nkeep + 1);
  for (int q = threadIdx.x; q < n1 * nc; q += blockDim.x) Gs[q] = Gg[q];
  const int n = 2 * sl.Nd, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2* U = ucol(L, slot, 0);
  for (int i0 = blockIdx.x * kRestartRows; i0 < n; i0 += gridDim.x * kRestartRows) {
    const bool in = i0 + lane < n;
    __syncthreads();  // the last rows are done with
    for (int r = warp; r < n1; r += 8)
      us[r * kRestartRows + lane] = in ? U[(size_t)r * L.ustride + i0 + lane] : make_double2(0.0, 0.0);
    __syncthreads();
    for (int c0 = 4 * warp; c0 < nc; c0 += 32) {
      double2 acc[4];
#pragma unroll
      for (int c = 0; c < 4; c++) acc[c] = make_double2(0.0, 0.0);
      for (int r = 0; r < n1; r++) {
        const double2 u = us[r * kRestartRows + lane];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const double gv = Gs[min(c0 + c, nc - 1) * n1 + r];
          acc[c].x += gv * u.x;
          acc[c].y += gv * u.y;
        }
      }
#pragma unroll
      for (int c = 0; c < 4; c++)
        if (in && c0 + c < nc) U[(size_t)(c0 + c) * L.ustride + i0 + lane] = acc[c];
    }
  }
}

// Ritz vectors: out[:, c] = sum_r U[:, r] * Z[r, c] for c < nwant (Z real, column-major, leading dimension
// nstep), ev = U(:, 0:nstep) z(:, 0:nwant) (Lanczos_Isotropic.cu:93), CH columns from c0 on.
template <int CH>
__global__ void __launch_bounds__(256) k_ugemm(VecArgs va, LzArgs L, const double* Z, double2* out, int c0) {
  FAME_COUNT_LAUNCH();
  const int slot = blockIdx.z;
  const Slot sl = va.slots[slot];
  if (!sl.active) return;
  __shared__ double Zs[kMaxStep * CH];
  const int nrows = L.nstep;
  const double* Zg = Z + (size_t)slot * nrows * nrows;
  const int nc = min(CH, L.nwant - c0);
  for (int q = threadIdx.x; q < nrows * nc; q += blockDim.x) Zs[q] = Zg[q + c0 * nrows];
  __syncthreads();
  const int n = 2 * sl.Nd;
  const double2* U = ucol(L, slot, 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double2 acc[CH];
#pragma unroll
    for (int c = 0; c < CH; c++) acc[c] = make_double2(0.0, 0.0);
    for (int r = 0; r < nrows; r++) {
      const double2 u = U[(size_t)r * L.ustride + i];
#pragma unroll
      for (int c = 0; c < CH; c++) {
        const double gv = Zs[r + c * nrows];
        acc[c].x += gv * u.x;
        acc[c].y += gv * u.y;
      }
    }
#pragma unroll
    for (int c = 0; c < CH; c++)
      if (c < nc) out[((size_t)slot * L.nwant + c0 + c) * L.ustride + i] = acc[c];
  }
}

}  // namespace fame
