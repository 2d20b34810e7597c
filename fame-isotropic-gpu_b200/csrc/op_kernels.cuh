// Operator stage kernels (plane inverse, pencil, plane forward); explicitly
// instantiated per precision, lattice family and geometry policy in ops_*.cu.
//
// GP is the geometry policy (geom_policy.cuh): runtime lengths (DynGeom) or
// compile-time lengths (StatGeom<...>).
#pragma once
#include "geom_policy.cuh"

namespace fame {

// Lambda_x, Lambda_y, Lambda_z at plane element (m, f) of plane s, in precision R.
// Simple lattices read the per-CTA shared tables lx[f], ly[m]; `lp` is what is constant on the
// plane: Lambda_z (Simple) or Lambda_x (General).  (A table of Lambda_z in FP32, 8 bytes a point, was
// slower than the two loads and the FP64 product: FCC 64 CG plane stage 14.8 against 14.4 us per
// k-point.)
template <typename R, bool GEN>
__device__ __forceinline__ void lam_elem(const Geom& g, const double2* tab, const cplx<R>* lx, const cplx<R>* ly, int lys,
                                         cplx<R> lp, int s, int m, int f, cplx<R>& Lx, cplx<R>& Ly, cplx<R>& Lz) {
  if constexpr (!GEN) {
    Lx = lx[f];
    Ly = ly[m * lys];
    Lz = lp;
  } else {
    Lx = lp;
    Ly = cvt<R>(tab[g.oLy + s * g.Ny + m]);
    const double2 e = cmul(tab[g.oExy + s * g.Ny + m], tab[g.oWz + f]);
    Lz = cvt<R>(make_double2((e.x - 1.0) * g.ihz, e.y * g.ihz));
  }
}
template <typename R, bool GEN> __device__ __forceinline__ cplx<R> lam_plane(const Geom& g, const double2* tab, int s) {
  return cvt<R>(tab[(GEN ? g.oLx : g.oLz) + s]);
}

// ------------------------------------------------------------------ L2 prefetch
// The CTAs of a stage kernel run in waves in launch order, and each one spends most of
// its time on shared-memory transforms.  With the option "prefetch" a CTA of the CG's pencil stage
// issues bulk L2 prefetches of the global operands of the CTA pf_dist places later (about one wave
// ahead), so that CTA finds them in L2 instead of waiting on DRAM.  The prefetches only
// cover bytes that CTA will read.

// Linear launch index of this CTA, and the (x, y, z) block of linear index t.
__device__ __forceinline__ long cta_linear() {
  return blockIdx.x + (long)gridDim.x * (blockIdx.y + (long)gridDim.y * blockIdx.z);
}
__device__ __forceinline__ bool cta_of(long t, int& x, int& y, int& z) {
  const long n = (long)gridDim.x * gridDim.y * gridDim.z;
  if (t >= n) return false;
  x = (int)(t % gridDim.x);
  const long r = t / gridDim.x;
  y = (int)(r % gridDim.y);
  z = (int)(r / gridDim.y);
  return true;
}

// The reduced-vector range [e0, e1) of plane s that the component-`comp` CTA of a
// plane cluster mixes, as element offsets (first half; the second starts Nd later).
__device__ __forceinline__ bool plane_vec_range(int P, int s, int comp, const Slot& sl, long& i0, long& i1) {
  const int per = (P + 2) / 3;
  const int e0 = comp * per, e1 = min(P, e0 + per);
  i0 = max(0L, (long)s * P + e0 - sl.off);
  i1 = (long)s * P + e1 - sl.off;
  return i1 > i0;
}

// ------------------------------------------------------------------ plane stages
// One cluster = 3 CTAs = the 3 components of plane s, or 6 where two CTAs share a component
// (GP::kHalves).  grid = (3*kHalves*Ls, vec_per_slot, nslots)
struct PlanePos {
  int s, comp, half, vec, slot;
};
// Read afresh from the special registers at every call (the empty asm hides the value from
// the compiler): a kernel asks again after its transforms, so that nothing but the plane
// lives across them.  Kept in registers instead, the two dozen values of the mixing
// phase were spilled and reloaded around every one of the runtime plans' passes.
template <class GP> __device__ __forceinline__ PlanePos plane_pos() {
  unsigned x = blockIdx.x, y = blockIdx.y, z = blockIdx.z;
  asm volatile("" : "+r"(x), "+r"(y), "+r"(z));
  PlanePos p;
  constexpr int C = 3 * GP::kHalves;
  p.s = (int)(x / C);
  const int rank = (int)x - C * p.s;
  p.half = GP::kHalves == 1 ? 0 : rank / 3;
  p.comp = rank - 3 * p.half;
  p.vec = (int)y;
  p.slot = (int)z;
  return p;
}

// Dynamic shared memory of a plane CTA.  Plane rows have the odd pitch S >= Lf.  lx, ly hold
// the Lambda tables of the plane's axes (Simple lattices) or, in ly, D_ky(s, .) (General);
// element m of ly is ly[m * lys].  Static geometries have one twiddle table (equal axes) and
// keep ly in the column that pads the rows.
template <typename R> struct PlaneSmem {
  cplx<R>*plane, *twf, *twm, *lx, *ly;
  int lys;
};
template <typename R, class GP> __device__ __forceinline__ PlaneSmem<R> plane_smem_of(const Geom& g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PlaneSmem<R> m;
  m.plane = reinterpret_cast<cplx<R>*>(smem_raw);
  m.twf = m.plane + GP::Lm(g) * GP::S(g);
  m.twm = GP::kStatic ? m.twf : m.twf + GP::Lf(g);
  m.lx = GP::kStatic ? m.twf + GP::Lf(g) : m.twm + GP::Lm(g);
  m.ly = GP::kStatic ? m.plane + GP::Lf(g) : m.lx + GP::Lf(g);
  m.lys = GP::kStatic ? GP::S(g) : 1;
  return m;
}

// Lambda_x of the plane's axis: in shared memory, or (half planes, FP64) the k-point's table itself.
template <typename R, class GP>
__device__ __forceinline__ const cplx<R>* plane_lx(const Geom& g, const double2* tab, const PlaneSmem<R>& m) {
  if constexpr (GP::kHalves == 1)
    return m.lx;
  else
    return tab + g.oLx;
}
// Where element e (row r) of the CTA's share lies in the plane.
template <class GP> __device__ __forceinline__ int plane_elem(const Geom& g, int half, int e, int r) {
  return GP::kHalves == 1 ? e : e + (r + half) * GP::Lf(g);
}

// Twiddle and Lambda (or D_ky) tables into shared memory; a barrier must follow.
template <typename R, bool GEN, class GP>
__device__ __forceinline__ void plane_tables(const Geom& g, const cplx<R>* tw, const double2* tab, int s,
                                             int half, const PlaneSmem<R>& m) {
  const int Lf = GP::Lf(g), Lm = GP::Lm(g);
  for (int i = threadIdx.x; i < Lf; i += GP::plane_threads()) {
    m.twf[i] = tw[g.twf + i];
    if constexpr (!GEN && GP::kHalves == 1) m.lx[i] = cvt<R>(tab[g.oLx + i]);
  }
  for (int i = threadIdx.x; i < Lm; i += GP::plane_threads()) {
    if constexpr (!GP::kStatic) m.twm[i] = tw[g.twm + i];
    m.ly[i * m.lys] = cvt<R>(GEN ? tab[g.oDky + s * g.Ny + i] : tab[g.oLy + GP::kHalves * i + half]);
  }
}

// plane *= conj(D_kz), General lattices: from the table of the k-point where there is one
// (coalesced; evaluated in place, the sincospi were a quarter of the plane kernels'
// instructions), else evaluated.  In the inverse direction the values have their parts swapped,
// and multiplying by the conjugate is what multiplies the value by D_kz.
template <typename R, class GP>
__device__ __forceinline__ void plane_times_dkz(const Geom& g, const double2* tabs, const cplx<R>* dkz, cplx<R>* plane) {
  const PlanePos p = plane_pos<GP>();
  const int Lf = GP::Lf(g), S = GP::S(g), P = GP::P(g);
  const cplx<R>* d = dkz ? dkz + (size_t)p.slot * g.N + (size_t)p.s * P : nullptr;
  const double2* tab = tabs + (size_t)p.slot * g.tab_stride;
#pragma unroll 4
  for (int e = threadIdx.x; e < P; e += GP::plane_threads()) {
    const int m = div_magic(e, g.mLf), q = e + m * (S - Lf);
    plane[q] = cmulc(d ? d[e] : dkz_at<R>(g, tab, p.s, m, e - m * Lf), plane[q]);
  }
  __syncthreads();
}

// The plane's part of the D_kz table where the mid axis' passes can multiply by it, else null.
template <typename R, class GP>
__device__ __forceinline__ const cplx<R>* plane_dkz(const Geom& g, const AxisPasses& mid, const cplx<R>* dkz) {
  if (!dkz || !GP::mul_ok(mid)) return nullptr;
  const PlanePos p = plane_pos<GP>();
  return dkz + (size_t)p.slot * g.N + (size_t)p.s * GP::P(g);
}

// Whether the inverse transforms of a plane run as forward ones on values with swapped real and
// imaginary parts, swap(z) = i conj(z): swap(IDFT z) = DFT swap(z).  The mix writes them so and
// plane_store swaps them back.  (Static Simple geometries have the direction at compile time.)
template <bool GEN, class GP> constexpr bool kSwapInv = !(GP::kStatic && !GEN);
template <bool SWAP, typename T> __device__ __forceinline__ T maybe_swap(T z) {
  if constexpr (SWAP) {
    T y;
    y.x = z.y;
    y.y = z.x;
    return y;
  } else {
    return z;
  }
}

// Unnormalised inverse 2-D transform of the CTA's plane: fast axis, (x D_kz), mid axis; x D_ky
// follows in plane_store (General lattices, FAME_FFT_CUDA.cu:104-117).  D_kz multiplies the mid axis'
// inputs (forward: its outputs) in the pass that reads (writes) them, coalesced there; a pass of its own
// (a prime mid axis, or no table) is another round trip of the plane through shared memory.
template <typename R, bool GEN, int RARE, class GP>
__device__ __forceinline__ void plane_inverse(const Geom& g, const AxisPasses* axes, const double2* tabs,
                                              const cplx<R>* dkz) {
  const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
  if constexpr (GP::kStatic && !GEN) {
    GP::template fft_plane_c<R, true, true>(m.plane, m.twf);
    GP::template fft_plane_c<R, false, true>(m.plane, m.twm);
  } else {
    // one FFT call site per axis loop: the runtime plans' passes are long
#pragma unroll 1
    for (int ax = 0; ax < 2; ax++) {
      const cplx<R>* pre = GEN && ax == 1 ? plane_dkz<R, GP>(g, axes[1], dkz) : nullptr;
      if (GEN && ax == 1 && !pre) plane_times_dkz<R, GP>(g, tabs, dkz, m.plane);
      GP::template fft_plane<R, RARE, GEN>(m.plane, axes[ax], ax == 0, ax == 0 ? m.twf : m.twm, pre, nullptr);
    }
  }
}

// Unnormalised forward 2-D transform.  General lattices (T*, FAME_FFT_CUDA.cu:128-150): x conj(D_ky)
// (in plane_load), mid pass, x conj(D_kz), fast pass.  Simple lattices: fast then mid axis.
template <typename R, bool GEN, int RARE, class GP>
__device__ __forceinline__ void plane_forward(const Geom& g, const AxisPasses* axes, const double2* tabs,
                                              const cplx<R>* dkz) {
  const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
  if constexpr (GP::kStatic && !GEN) {
    GP::template fft_plane_c<R, true, false>(m.plane, m.twf);
    GP::template fft_plane_c<R, false, false>(m.plane, m.twm);
  } else {
#pragma unroll 1
    for (int ax = 0; ax < 2; ax++) {
      const bool fast = GEN ? ax == 1 : ax == 0;
      const cplx<R>* post = GEN && !fast ? plane_dkz<R, GP>(g, axes[1], dkz) : nullptr;
      GP::template fft_plane<R, RARE, GEN>(m.plane, axes[fast ? 0 : 1], fast, fast ? m.twf : m.twm, nullptr, post);
      if (GEN && !fast && !post) plane_times_dkz<R, GP>(g, tabs, dkz, m.plane);
    }
  }
}

// This CTA's plane of the field in global memory.
template <typename R, class GP>
__device__ __forceinline__ long plane_base(const Geom& g, const PlanePos& p, int vec_per_slot, long fstride) {
  return (long)(p.slot * vec_per_slot + p.vec) * fstride + (long)p.comp * g.N + (long)p.s * GP::P(g);
}

// The plane into shared memory (x conj(D_ky), General): the tables must be in place for
// General lattices; Simple ones leave cp.async copies in flight (cp_async_wait_all).  A half of a plane
// takes the mid axis' first step here: x_m + x_{m + Lm} or (x_m - x_{m + Lm}) w^m.
template <typename R, bool GEN, class GP>
__device__ __forceinline__ void plane_load(const Geom& g, const cplx<R>* T, const cplx<R>* tw, int half,
                                           const PlaneSmem<R>& m) {
  const int Lf = GP::Lf(g), S = GP::S(g), P = GP::PL(g), NT = GP::plane_threads();
  if constexpr (GP::kHalves == 2) {
    constexpr int U = 6;  // pairs in flight per thread
    static_assert(GP::kLm * GP::kLf % (U * GP::kThreads) == 0, "whole batches");
    for (int eb = threadIdx.x; eb < P; eb += U * NT) {
      cplx<R> v[U], u[U];
#pragma unroll
      for (int k = 0; k < U; k++) {
        v[k] = T[eb + k * NT];
        u[k] = T[P + eb + k * NT];
      }
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int e = eb + k * NT, r = e / Lf;
        m.plane[e + r * (S - Lf)] = half ? cmul(tw[g.twm + r], csub(v[k], u[k])) : cadd(v[k], u[k]);
      }
    }
  } else if constexpr (!GEN) {
    for (int e = threadIdx.x; e < P; e += NT) {
      const int r = GP::kStatic ? e / Lf : div_magic(e, g.mLf);
      cp_async_elem(m.plane + e + r * (S - Lf), T + e);
    }
  } else {
    constexpr int U = 32 / (int)sizeof(R);  // loads in flight per thread
    for (int eb = threadIdx.x; eb < P; eb += U * NT) {
      cplx<R> v[U];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (eb + u * NT < P) v[u] = T[eb + u * NT];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int e = eb + u * NT;
        if (e < P) {
          const int r = div_magic(e, g.mLf);
          m.plane[e + r * (S - Lf)] = cmulc(m.ly[r], v[u]);
        }
      }
    }
  }
}

// The plane out to global memory (x D_ky, General).  Halves: each combines rows of both, x_m = E_m + conj(w^m) O_m,
// x_{m + Lm} = E_m - conj(w^m) O_m; plane_store_end must follow before the CTA exits.
template <typename R, bool GEN, class GP>
__device__ __forceinline__ void plane_store(const Geom& g, cplx<R>* T) {
  const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
  const int Lf = GP::Lf(g), S = GP::S(g), P = GP::PL(g);
  if constexpr (GP::kHalves == 2) {
    cg::cluster_group cl = cg::this_cluster();
    const PlanePos p = plane_pos<GP>();
    const cplx<R>* peer = cl.map_shared_rank(m.plane, p.comp + 3 * (1 - p.half));
    constexpr int U = 6;  // remote reads in flight per thread
    const int NT = GP::plane_threads();
    for (int eb = threadIdx.x; eb < P; eb += U * NT) {
      cplx<R> v[U];
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int e = eb + k * NT;
        v[k] = peer[e + e / Lf * (S - Lf)];
      }
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int e = eb + k * NT, r = e / Lf;
        const cplx<R> own = m.plane[e + r * (S - Lf)], w = m.twf[r];
        T[p.half * P + e] = p.half ? csub(v[k], cmulc(w, own)) : cadd(own, cmulc(w, v[k]));
      }
    }
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
  } else {
#pragma unroll 4
    for (int e = threadIdx.x; e < P; e += GP::plane_threads()) {
      const int r = GP::kStatic ? e / Lf : div_magic(e, g.mLf);
      const cplx<R> v = maybe_swap<kSwapInv<GEN, GP>>(m.plane[e + r * (S - Lf)]);
      T[e] = GEN ? cmul(v, m.ly[r]) : v;
    }
  }
}

// Before it: both halves are transformed.  After it: both have been read.
template <class GP> __device__ __forceinline__ void plane_store_begin() {
  if constexpr (GP::kHalves == 2) cg::this_cluster().sync();
}
template <class GP> __device__ __forceinline__ void plane_store_end() {
  if constexpr (GP::kHalves == 2) asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
}

// Exchange of mixed components between the three CTAs.  Static geometries send them with
// st.async into the owner's plane, counted on the owner's barrier (P values arrive per
// plane); the others store to distributed shared memory and use a cluster barrier.
// SWAP: the values are written with swapped parts (kSwapInv).
template <typename R, bool ASYNC, bool SWAP> struct PlaneExchange {
  cplx<R>* dst[3];
  unsigned rplane[3], rbar[3];
  __device__ __forceinline__ PlaneExchange(cplx<R>* plane, unsigned bar, int rank0) {
    cg::cluster_group cl = cg::this_cluster();
#pragma unroll
    for (int c = 0; c < 3; c++) {
      dst[c] = cl.map_shared_rank(plane, rank0 + c);
      rplane[c] = ASYNC ? mapa_u32(smem_u32(plane), rank0 + c) : 0u;
      rbar[c] = ASYNC ? mapa_u32(bar, rank0 + c) : 0u;
    }
  }
  __device__ __forceinline__ void put(int q, const cplx<R>* v) const {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if constexpr (ASYNC)
        st_async(rplane[c] + (unsigned)(q * sizeof(cplx<R>)), maybe_swap<SWAP>(v[c]), rbar[c]);
      else
        dst[c][q] = maybe_swap<SWAP>(v[c]);
    }
  }
};

// Start of an exchange (thread 0 of each CTA): the barrier, and the fault marker of an earlier
// exchange, after which launches skip their work (rank 0 reads it, all three act on it).
__device__ __forceinline__ void exchange_init(unsigned bar, int* skip, int* fault) {
  mbar_init(bar, 1);
  mbar_init_fence_cluster();
  *skip = fault ? *(volatile int*)fault : 0;
}
// End of it: the CTA's plane is complete once all P values have arrived.  A wait that runs out
// (about 0.1 s; it cannot unless the exchange is broken) records the fault, on the device for later
// launches and in the host's memory for the caller, and goes on.
__device__ __forceinline__ void exchange_wait(unsigned bar, int* fault, int* fault_host) {
  if (!mbar_wait(bar, 0, 200000000LL) && fault) {
    atomicExch(fault, 1);
    *(volatile int*)fault_host = 1;
  }
  __syncthreads();
}

template <typename R, bool GEN, int IN, bool PR, int RARE, class GP>
__global__ void __cluster_dims__(3 * GP::kHalves, 1, 1) __launch_bounds__(GP::template max_plane_threads<R, RARE>(), GP::template plane_min_blocks<R, RARE>())
    k_plane_inv(PlaneInArgs<R> a) {
  FAME_COUNT_LAUNCH();
  pdl_wait();
  const Geom& g = a.g;
  constexpr bool kAsyncMix = GP::kStatic;
  __shared__ __align__(8) unsigned long long xbar;
  __shared__ int skip;
  const unsigned bar = smem_u32(&xbar);
  {
    const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
    const int Lf = GP::Lf(g), S = GP::S(g), P = GP::P(g), PL = GP::PL(g);
    cg::cluster_group cl = cg::this_cluster();
    const PlanePos p = plane_pos<GP>();
    const Slot sl = a.slots[p.slot];
    if (!sl.active) return;  // uniform over the cluster
    const CgState* st = nullptr;
    if constexpr (IN == IN_CG || IN == IN_REFINE) {
      st = a.cg + p.slot;
      if (IN == IN_CG ? !st->active : !st->outer_active) return;
    }
    if (kAsyncMix && threadIdx.x == 0) exchange_init(bar, &skip, a.fault);
    const double2* tab = a.tabs + (size_t)p.slot * g.tab_stride;
    plane_tables<R, GEN, GP>(g, a.tw, tab, p.s, p.half, m);
    const cplx<R> lp = lam_plane<R, GEN>(g, tab, p.s);
    cl.sync();  // every CTA of the cluster is running (and the tables and barriers are in place)
    if constexpr (kAsyncMix) {
      if (*cl.map_shared_rank(&skip, 0)) {
        cl.sync();  // rank 0's marker stays readable until all three have read it
        return;
      }
      if (threadIdx.x == 0) mbar_arrive_expect_tx(bar, (unsigned)(PL * sizeof(cplx<R>)));
    }
    const PlaneExchange<R, kAsyncMix, kSwapInv<GEN, GP>> ex(m.plane, bar, 3 * p.half);
    const long vb = (long)(p.slot * a.vec_per_slot + p.vec) * a.vstride;
    const int Nd = sl.Nd, off = sl.off;
    const int per = (PL + 2) / 3;
    const int e0 = p.comp * per, e1 = min(PL, e0 + per);
    R rscale = 0;
    const float2* x32 = nullptr;
    if constexpr (IN == IN_REFINE) {
      // the FP32 correction (none if the inner solve did no product), and its scale
      rscale = (R)(1.0 / st->scale);
      x32 = st->iter > 1 ? a.x32[st->iter & 1] : nullptr;
    }
    // Input stage and the 2 -> 3 mix.  IN_CG: the start residual r.  IN_REFINE: y += x32 / scale.
    // The operands of KB points per thread are loaded up front, so one global-load latency
    // covers KB points.
    constexpr int KB = !GP::kStatic || IN == IN_REFINE ? 2 : 8 / GP::kHalves;
    const int NT = GP::plane_threads();
    for (int eb = e0 + threadIdx.x; eb < e1; eb += KB * NT) {
      cplx<R> A1[KB], A2[KB];
      float2 F1[KB], F2[KB];
#pragma unroll
      for (int k = 0; k < KB; k++) {
        const int e = eb + k * NT;
        A1[k] = A2[k] = mk<R>(0, 0);
        F1[k] = F2[k] = make_float2(0.f, 0.f);
        const int r = GP::kHalves == 1 ? 0 : e / Lf;
        const int fi = p.s * P + plane_elem<GP>(g, p.half, e, r);
        if (e < e1 && fi >= off) {
          const long i = fi - off;
          if constexpr (IN == IN_REFINE) {
            A1[k] = a.y64[vb + i];
            A2[k] = a.y64[vb + Nd + i];
            F1[k] = x32 ? x32[vb + i] : make_float2(0.f, 0.f);
            F2[k] = x32 ? x32[vb + Nd + i] : make_float2(0.f, 0.f);
          } else {
            A1[k] = a.in[vb + i];
            A2[k] = a.in[vb + Nd + i];
          }
        }
      }
#pragma unroll
      for (int k = 0; k < KB; k++) {
        const int e = eb + k * NT;
        if (e >= e1) break;
        const int r = GP::kStatic ? e / Lf : div_magic(e, g.mLf), f = e - r * Lf;
        const int fi = p.s * P + plane_elem<GP>(g, p.half, e, r);
        cplx<R> v[3] = {mk<R>(0, 0), mk<R>(0, 0), mk<R>(0, 0)};
        if (fi >= off) {
          const long i = fi - off;
          cplx<R> Lx, Ly, Lz;
          lam_elem<R, GEN>(g, tab, plane_lx<R, GP>(g, tab, m), m.ly, m.lys, lp, p.s, r, f, Lx, Ly, Lz);
          cplx<R> x1 = A1[k], x2 = A2[k];
          if constexpr (IN == IN_VEC) {
            if (a.sigma) {
              const R sc = sqrt(cabs2(Lx) + cabs2(Ly) + cabs2(Lz));
              x1 = cscale(x1, sc);
              x2 = cscale(x2, sc);
            }
          } else if constexpr (IN == IN_REFINE) {
            x1.x += (double)F1[k].x * rscale;
            x1.y += (double)F1[k].y * rscale;
            x2.x += (double)F2[k].x * rscale;
            x2.y += (double)F2[k].y * rscale;
            a.y64[vb + i] = x1;
            a.y64[vb + Nd + i] = x2;
          }
          cplx<R> Pc[6];
          pi_from<R>(GEN, PR, Lx, Ly, Lz, Pc);
#pragma unroll
          for (int c = 0; c < 3; c++) v[c] = cadd(cmul(Pc[c], x1), cmul(Pc[3 + c], x2));
        }
        ex.put(r * S + f, v);
      }
    }
    if constexpr (kAsyncMix)
      exchange_wait(bar, a.fault, a.fault_host);
    else
      cl.sync();
  }
  plane_inverse<R, GEN, RARE, GP>(g, a.ax, a.tabs, a.dkz);
  plane_store_begin<GP>();
  pdl_trigger();
  plane_store<R, GEN, GP>(g, a.T + plane_base<R, GP>(g, plane_pos<GP>(), a.vec_per_slot, a.fstride));
  plane_store_end<GP>();
}

// ------------------------------------------------------------------ CG plane stage
// The middle of a CG iteration in one kernel: the forward plane transforms of A r's field,
// the 3 -> 2 unmix (w = A r), the three-term recurrences
//   r' = rho (r - gamma w) + (1 - rho) r_old,   x' = rho (x + gamma r) + (1 - rho) x_old,
//   gamma = ||r||^2 / <r, A r>,   rho = 1 / (1 - gamma ||r||^2 / (gamma_old ||r_old||^2 rho_old))
// (CG in the form without search directions: Hageman and Young, "Applied Iterative Methods",
// 1981, section 7.3; the reference's CG.cu:36-77 takes the same steps through p), the
// 2 -> 3 mix of r' and its inverse plane transforms.  The form with p needs ||r'||^2 of all
// planes before it can mix p' = r' + beta p, so it splits here into two kernels, each of which
// waits for its own loads and evaluates Pi; this one mixes r' itself, reads r, r_old, x and
// x_old once, and evaluates Pi once for both directions.  In exchange the kernel's second half is idle work in
// the last iteration of a solve.  r' and x' overwrite r_old and x_old: the current buffers are
// those of the iteration's parity.
// w and r' pass through the planes in place: element e of all three is read and written by
// its owner alone, between the two exchanges.
template <typename R, bool GEN, int RARE, class GP>
__global__ void __cluster_dims__(3, 1, 1) __launch_bounds__(GP::template max_plane_threads<R, RARE>(), GP::template plane_min_blocks<R, RARE>())
    k_plane_cg(PlaneCgArgs<R> a) {
  static_assert(GP::kHalves == 1, "whole planes");
  FAME_COUNT_LAUNCH();
  const Geom& g = a.g;
  constexpr bool kAsyncMix = GP::kStatic;
  __shared__ __align__(8) unsigned long long xbar;
  __shared__ int skip;
  __shared__ double s_coef[2];
  const unsigned bar = smem_u32(&xbar);
  {
    const PlanePos p = plane_pos<GP>();
    const Slot sl = a.slots[p.slot];
    const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
    // the tables are the solve's, older than the kernel before this one
    if (sl.active) plane_tables<R, GEN, GP>(g, a.tw, a.tabs + (size_t)p.slot * g.tab_stride, p.s, 0, m);
    pdl_wait();
    if ((threadIdx.x | blockIdx.x | blockIdx.y | blockIdx.z) == 0) set_cond(a.reset, 0);
    const CgState* st = a.cg + p.slot;
    if (!sl.active || !st->active) {  // uniform over the cluster
      if (blockIdx.x == 0 && threadIdx.x == 0) a.cg_copy[p.slot].active = 0;
      return;
    }
    const int cur = st->iter & 1;
    if (kAsyncMix && threadIdx.x == 0) exchange_init(bar, &skip, a.fault);
    const cplx<R>* T = a.T + plane_base<R, GP>(g, p, 1, a.fstride);
    if constexpr (GEN) __syncthreads();  // D_ky is in place
    plane_load<R, GEN, GP>(g, T, a.tw, 0, m);
    // gamma and rho from the pencil stage's partial sums of <r, A r>, summed in order by one warp
    // while the plane streams in
    if (threadIdx.x < 32) {
      const double rAr = warp_sum_partials(a.partials + (size_t)p.slot * a.pstride, a.pen_parts) / g.N;
      double gm, rho;
      cg_coefficients(*st, rAr, gm, rho);
      if (threadIdx.x == 0) {
        s_coef[0] = gm;
        s_coef[1] = rho;
        if (blockIdx.x == 0) {
          CgState c = *st;
          c.gm = gm;
          c.rho = rho;
          a.cg_copy[p.slot] = c;
        }
      }
    }
    if constexpr (!GEN) cp_async_wait_all();
    __syncthreads();
    // This CTA's own part of r, r_old, x and x_old: it streams into L2 during the forward
    // transforms.  Asked for before the plane had arrived it only delayed the plane, and the
    // vectors pass through as streams (evicted first), which leaves the L2 to the field that the
    // pencil stage reads next: together 38.7 -> 34.8 us per k-point at 96^3 (20 per launch).
    long i0, i1;
    if (a.self_pf && threadIdx.x < (st->iter == 1 ? 2 : st->iter == 2 ? 6 : 8) &&
        plane_vec_range(GP::P(g), p.s, p.comp, sl, i0, i1)) {
      const int which = threadIdx.x >> 1;
      const cplx<R>* v = which == 0 ? a.r[cur] : which == 1 ? a.r[cur ^ 1] : which == 2 ? a.x[cur] : a.x[cur ^ 1];
      prefetch_l2(v + (long)p.slot * a.vstride + ((threadIdx.x & 1) ? sl.Nd : 0) + i0, (i1 - i0) * sizeof(cplx<R>));
    }
  }
  plane_forward<R, GEN, RARE, GP>(g, a.ax, a.tabs, a.dkz);
  double acc[1] = {0.0};
  {
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();  // all three component planes transformed (and the barriers in place)
    if constexpr (kAsyncMix) {
      if (*cl.map_shared_rank(&skip, 0)) {
        cl.sync();  // rank 0's marker stays readable until all three have read it
        return;
      }
      if (threadIdx.x == 0) mbar_arrive_expect_tx(bar, (unsigned)(GP::P(g) * sizeof(cplx<R>)));
    }
    const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
    const int Lf = GP::Lf(g), S = GP::S(g), P = GP::P(g);
    const PlanePos p = plane_pos<GP>();
    const Slot sl = a.slots[p.slot];
    const double2* tab = a.tabs + (size_t)p.slot * g.tab_stride;
    const cplx<R> lp = lam_plane<R, GEN>(g, tab, p.s);
    const PlaneExchange<R, kAsyncMix, kSwapInv<GEN, GP>> ex(m.plane, bar, 0);
    const int iter = a.cg[p.slot].iter, cur = iter & 1;
    const bool have_r = iter > 1, have_x = iter > 2;  // r_old = 0 at k = 1; x = 0 at k = 1, x_old = 0 at k = 2
    const long vb = (long)p.slot * a.vstride;
    const cplx<R>*rc = a.r[cur] + vb, *xc = a.x[cur] + vb;
    cplx<R>*ro = a.r[cur ^ 1] + vb, *xo = a.x[cur ^ 1] + vb;
    // rho gamma and rho - 1 (rho = 1 at k = 1)
    const R rg = (R)(s_coef[0] * s_coef[1]), rm = (R)(s_coef[1] - 1.0);
    const int Nd = sl.Nd, off = sl.off;
    const int per = (P + 2) / 3;
    const int e0 = p.comp * per, e1 = min(P, e0 + per);
    constexpr int KB = 2;
    const int NT = GP::plane_threads();
    for (int eb = e0 + threadIdx.x; eb < e1; eb += KB * NT) {
      cplx<R> t[KB][3], R1[KB], R2[KB], O1[KB], O2[KB], X1[KB], X2[KB], Y1[KB], Y2[KB];
#pragma unroll
      for (int k = 0; k < KB; k++) {
        const int e = eb + k * NT;
        const int fi = p.s * P + e;
        R1[k] = R2[k] = O1[k] = O2[k] = X1[k] = X2[k] = Y1[k] = Y2[k] = mk<R>(0, 0);
        t[k][0] = t[k][1] = t[k][2] = mk<R>(0, 0);
        if (e < e1 && fi >= off) {
          const long i = fi - off;
          R1[k] = __ldcs(&rc[i]);
          R2[k] = __ldcs(&rc[Nd + i]);
          if (have_r) {
            O1[k] = __ldcs(&ro[i]);
            O2[k] = __ldcs(&ro[Nd + i]);
            X1[k] = __ldcs(&xc[i]);
            X2[k] = __ldcs(&xc[Nd + i]);
          }
          if (have_x) {
            Y1[k] = __ldcs(&xo[i]);
            Y2[k] = __ldcs(&xo[Nd + i]);
          }
          const int r = GP::kStatic ? e / Lf : div_magic(e, g.mLf), q = r * S + (e - r * Lf);
#pragma unroll
          for (int c = 0; c < 3; c++) t[k][c] = ex.dst[c][q];
        }
      }
#pragma unroll
      for (int k = 0; k < KB; k++) {
        const int e = eb + k * NT;
        if (e >= e1) break;
        const int fi = p.s * P + e;
        const int r = GP::kStatic ? e / Lf : div_magic(e, g.mLf), f = e - r * Lf;
        cplx<R> v[3] = {mk<R>(0, 0), mk<R>(0, 0), mk<R>(0, 0)};
        if (fi >= off) {
          const long i = fi - off;
          cplx<R> Lx, Ly, Lz;
          lam_elem<R, GEN>(g, tab, m.lx, m.ly, m.lys, lp, p.s, r, f, Lx, Ly, Lz);
          cplx<R> Pc[6];
          pi_from<R>(GEN, false, Lx, Ly, Lz, Pc);
          const cplx<R> w1 = cadd(cadd(cmulc(Pc[0], t[k][0]), cmulc(Pc[1], t[k][1])), cmulc(Pc[2], t[k][2]));
          const cplx<R> w2 = cadd(cadd(cmulc(Pc[3], t[k][0]), cmulc(Pc[4], t[k][1])), cmulc(Pc[5], t[k][2]));
          // x' = x + rho gamma r + (rho - 1)(x - x_old), r' the same with -w: the corrections added to x and r
          const cplx<R> n1 = cfma_r(csub(R1[k], O1[k]), rm, cfma_r(w1, -rg, R1[k]));
          const cplx<R> n2 = cfma_r(csub(R2[k], O2[k]), rm, cfma_r(w2, -rg, R2[k]));
          __stcs(&ro[i], n1);
          __stcs(&ro[Nd + i], n2);
          __stcs(&xo[i], cfma_r(csub(X1[k], Y1[k]), rm, cfma_r(R1[k], rg, X1[k])));
          __stcs(&xo[Nd + i], cfma_r(csub(X2[k], Y2[k]), rm, cfma_r(R2[k], rg, X2[k])));
          acc[0] += (double)(cabs2(n1) + cabs2(n2));
#pragma unroll
          for (int c = 0; c < 3; c++) v[c] = cadd(cmul(Pc[c], n1), cmul(Pc[3 + c], n2));
        }
        ex.put(r * S + f, v);
      }
    }
    // All P values have arrived: every CTA has read its elements of this plane too, since an
    // owner sends an element after reading it.
    if constexpr (kAsyncMix)
      exchange_wait(bar, a.fault, a.fault_host);
    else
      cl.sync();
  }
  plane_inverse<R, GEN, RARE, GP>(g, a.ax, a.tabs, a.dkz);
  pdl_trigger();
  plane_store<R, GEN, GP>(g, a.T + plane_base<R, GP>(g, plane_pos<GP>(), 1, a.fstride));
  // this CTA's part of ||r'||^2; the pencil stage sums the slot's parts in order
  __shared__ double sred[32];
  block_reduce<1>(acc, sred);
  if (threadIdx.x == 0) a.partials[(size_t)blockIdx.z * a.pstride + a.pen_parts + blockIdx.x] = acc[0];
}

// ------------------------------------------------------------------ end of a CG iteration
// The first CTA of a k-point in the pencil stage ends the CG iteration on the side (a kernel of its
// own took 6 us of the 47 us of an iteration on a small grid): from the plane stage's ||r'||^2
// parts it tells whether the solve goes on (CG.cu:37, :77) and steps the state.  The other CTAs
// do not wait for that: the transforms after a solve's last iteration are work for nothing, but
// a decision in every CTA cost the 96^3 pencil stage 17%.  The state before the step is read from
// cg_in, the copy that the plane stage made (with the coefficients it used: the sums they came
// from are this launch's to overwrite); the new one goes to cg.
// One warp; returns (in all lanes) whether slot q goes on.
template <typename R> __device__ __forceinline__ int cg_advance(const PencilArgs<R>& a, int q, bool write) {
  const CgState* in = a.cg_in + q;
  const double rr = warp_sum_partials<4>(a.partials + (size_t)q * a.pstride + a.pen_parts, a.fwd_parts);
  const int go = rr > in->tol2 && in->iter + 1 <= in->maxit;
  if (write && (threadIdx.x & 31) == 0) {
    CgState* st = a.cg + q;
    st->gm = in->gm;
    st->rho = in->rho;
    st->r1p = in->r1;
    st->r1 = rr;
    st->iter = in->iter + 1;
    st->total = in->total + 1;
    st->active = go;
  }
  return go;
}

// The WHILE condition of the CG loop, by one CTA of `nt` threads: whether any k-point goes on.
template <typename R> __device__ __forceinline__ void cg_loop_decide(const PencilArgs<R>& a, int nt) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int q = threadIdx.x >> 5; q < a.nslots; q += nt / 32)
    if (a.slots[q].active && a.cg_in[q].active && cg_advance(a, q, false) && (threadIdx.x & 31) == 0) any = 1;
  __syncthreads();
  if (threadIdx.x == 0) decide_cond(a.cond, any);
}

// ------------------------------------------------------------------ pencil stage

// Pencil CTAs per SM the register budget is sized for: the prime passes (RARE 2) and the static
// FP64 plans need 128 registers; the static FP32 ones fit 64 (four CTAs: 96^3 CG pencil stage 13.3
// us per k-point at 3, 11.4 at 4).
template <typename R, int RARE, class GP> constexpr int pencil_min_blocks() {
  return RARE >= 2 || (GP::kStatic && sizeof(R) == 8) ? 2 : GP::kStatic ? 4 : 3;
}

// One CTA transforms TW consecutive positions e = m * Lf + f of the plane (a tile may span
// rows, so only the last tile of a plane has idle lines).
// grid = (ceil(P / TW), 3 * vec_per_slot, nslots), GP::pencil_threads() threads
template <typename R, bool GEN, int MODE, int RARE, class GP>
__global__ void __launch_bounds__(kPencilThreads, pencil_min_blocks<R, RARE, GP>())
    k_pencil(PencilArgs<R> a) {
  FAME_COUNT_LAUNCH();
  if constexpr (MODE != PEN_QBQ_CG) pdl_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Geom& g = a.g;
  constexpr int TW = PencilTW<R>::v;
  const int Lf = GP::Lf(g), Ls = GP::Ls(g), P = GP::P(g), NT = GP::pencil_threads();
  // shared memory: tile [Ls][TW] | 1/eps tile [Ls][TW] (PEN_QBQ) | slow-axis twiddles [Ls]
  cplx<R>* tile = reinterpret_cast<cplx<R>*>(smem_raw);
  R* ibt = reinterpret_cast<R*>(tile + Ls * TW);
  cplx<R>* tws = reinterpret_cast<cplx<R>*>(ibt + Ls * TW);
  constexpr bool QBQ = MODE == PEN_QBQ || MODE == PEN_QBQ_CG;
  // The CG walks the k-points backwards here and forwards in its plane stage, so that each
  // stage starts on fields that the other left in L2 (96^3, FP32 CG iteration: 66.8 -> 65.3 us
  // per k-point in a solve of 8).
  const int slot = MODE == PEN_QBQ_CG ? (int)(gridDim.z - 1 - blockIdx.z) : (int)blockIdx.z;
  const Slot sl = a.slots[slot];
  const int comp = blockIdx.y % 3, vec = blockIdx.y / 3;
  const int e0 = blockIdx.x * TW;
  const int tw_n = min(TW, P - e0);
  const bool ib_field = !GEN || a.ib_field;  // 1/eps rows contiguous along the tile's positions
  // twiddles and 1/eps rows: the CG's pencil stage copies them before it waits for the plane stage
  for (int i = threadIdx.x; i < Ls; i += NT) tws[i] = a.tw[g.tws + i];
  constexpr int CH = 16 / sizeof(cplx<R>);  // elements per 16-byte copy
  constexpr int CHB = 16 / sizeof(R);       // 1/eps values per 16-byte copy
  if (QBQ && ib_field && sl.active) {
    const R* ib = a.invB + (long)comp * g.N + e0;
    if (P % CHB == 0 && ((uintptr_t)a.invB & 15) == 0) {
      for (int q = threadIdx.x; q < Ls * (TW / CHB); q += NT) {
        const int s = q / (TW / CHB), c = (q - s * (TW / CHB)) * CHB;
        if (c < tw_n) cp_async16(ibt + s * TW + c, ib + (long)s * P + c);
      }
    } else {
      for (int q = threadIdx.x; q < Ls * TW; q += NT) {
        const int s = q / TW, c = q - s * TW;
        if (c < tw_n) cp_async_real(ibt + q, ib + (long)s * P + c);
      }
    }
  }
  if constexpr (MODE == PEN_QBQ_CG) {
    pdl_wait();
    if (a.cg_in && blockIdx.x == 0 && blockIdx.y == 0 && slot == 0) cg_loop_decide(a, NT);
  }
  if (!sl.active) return;
  const CgState* st = MODE == PEN_QBQ_CG && a.cg_in ? a.cg_in + slot : a.cg + slot;
  if ((a.gate == 1 && !st->active) || (a.gate == 2 && !st->outer_active)) {
    cp_async_wait_all();
    return;
  }
  if constexpr (MODE == PEN_QBQ_CG) {
    // the field rows and 1/eps rows of the tile of the CTA one wave ahead
    int x2, y2, z2;
    if (a.pf_dist > 0 && cta_of(cta_linear() + a.pf_dist, x2, y2, z2)) {
      z2 = gridDim.z - 1 - z2;
      const int f2 = x2 * TW, c2 = y2 % 3, v2 = y2 / 3;
      const int n2 = min(TW, P - f2);
      for (int i = threadIdx.x; i < 2 * Ls; i += NT) {
        const long off = (long)c2 * g.N + (long)(i < Ls ? i : i - Ls) * P + f2;
        if (i < Ls)
          prefetch_l2(a.T + (long)(z2 * a.vec_per_slot + v2) * a.fstride + off, n2 * sizeof(cplx<R>));
        else
          prefetch_l2(a.invB + off, n2 * sizeof(R));
      }
    }
  }
  const double2* tab = a.tabs + (size_t)slot * g.tab_stride;
  const long fb = (long)(slot * a.vec_per_slot + vec) * a.fstride + (long)comp * g.N;
  // spatial index of slow position s at plane position e (QR_OUT, QRS_IN, 1/eps in the
  // spatial layout)
  auto spatial = [&](int s, int e) -> long {
    if (!GEN) return (long)s * P + e;
    const int m = div_magic(e, g.mLf);
    return ((long)(e - m * Lf) * g.Ny + m) * g.Nx + s;
  };
  auto dk_at = [&](int s, int e) -> double2 {  // D_k (Simple) or D_kx
    if (GEN) return tab[g.oDkx + s];
    const int m = div_magic(e, g.mLf);
    return cmul(cmul(tab[g.oDz + s], tab[g.oDy + m]), tab[g.oDx + (e - m * Lf)]);
  };
  // ---- load.  The QBQ streams the field rows (TW contiguous elements at stride P), like the
  // 1/eps rows above, straight into shared memory with cp.async: 16 bytes a copy when every row
  // starts on a 16-byte boundary (P a multiple of the copy's elements, the base aligned), else
  // one element.
  if constexpr (QBQ) {
    const cplx<R>* src = a.T + fb + e0;
    if (CH == 1 || P % CH == 0) {
      for (int q = threadIdx.x; q < Ls * (TW / CH); q += NT) {
        const int s = q / (TW / CH), c = (q - s * (TW / CH)) * CH;
        if (c < tw_n) cp_async16(tile + s * TW + c, src + (long)s * P + c);
      }
    } else {
      for (int q = threadIdx.x; q < Ls * TW; q += NT) {
        const int s = q / TW, c = q - s * TW;
        if (c < tw_n) cp_async_elem(tile + q, src + (long)s * P + c);
      }
    }
    if constexpr (MODE == PEN_QBQ_CG)
      if (a.cg_in && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 32) cg_advance(a, slot, true);
    cp_async_wait_all();
  } else {
    for (int q = threadIdx.x; q < Ls * TW; q += NT) {
      const int s = q / TW, f = q - s * TW;
      cplx<R> v = mk<R>(0, 0);
      if (f < tw_n) {
        if constexpr (MODE == PEN_QRS_IN) {
          // spatial input, x conj(D) before the forward transform
          v = cmul(a.in[(long)(slot * a.vec_per_slot + vec) * a.fstride + (long)comp * g.N + spatial(s, e0 + f)],
                   cvt<R>(cconj(dk_at(s, e0 + f))));
        } else {
          v = a.T[fb + (long)s * P + e0 + f];
        }
      }
      tile[q] = v;
    }
  }
  __syncthreads();
  // QBQ: inverse, x B^{-1}/N, forward.  QR_OUT: inverse, x D/N (and B^{-1}), store.
  // QRS_IN: forward only.  One FFT call site (dir loop) for the register budget, and forward
  // transforms only: DFT(x) holds IDFT(x)[-s] in row s, and the DFT of what is then in rows -s
  // comes out in rows -k, so the rows are counted backwards in between and in the store.
  constexpr int ndir = QBQ ? 2 : 1;
  // PEN_QBQ_CG: sum of |v|^2 / eps over the tile after the inverse transform
  R dot = 0;
  constexpr bool kStatQBQ = GP::kStatic && QBQ;  // whole tiles, 1/eps staged in shared memory
  if constexpr (kStatQBQ) {
    GP::template fft_slow_c<R, true>(tile, tws);
    const R invN = (R)(1.0 / g.N);
#pragma unroll 4
    for (int q = threadIdx.x; q < Ls * TW; q += NT) {
      const R ib = ibt[q];
      const cplx<R> v = tile[q];
      if constexpr (MODE == PEN_QBQ_CG) dot += ib * cabs2(v);
      if constexpr (sizeof(R) == 4)
        tile[q] = pscale(v, ib * invN);
      else
        tile[q] = cscale(v, ib * invN);
    }
    __syncthreads();
    GP::template fft_slow_c<R, false>(tile, tws);
  }
  for (int dir = 0; !kStatQBQ && dir < ndir; dir++) {
    GP::template fft_slow<R, RARE>(tile, a.ax, tws);
    if (MODE != PEN_QRS_IN && dir == 0) {
      const R invN = (R)(1.0 / g.N);
      for (int q = threadIdx.x; q < Ls * TW; q += NT) {
        const int row = q / TW, f = q - row * TW, s = row == 0 ? 0 : Ls - row;
        if (f < tw_n) {
          if constexpr (QBQ) {
            const R ib = ib_field ? ibt[s * TW + f] : a.invB[(long)comp * g.N + spatial(s, e0 + f)];
            if constexpr (MODE == PEN_QBQ_CG) dot += ib * cabs2(tile[q]);
            tile[q] = cscale(tile[q], ib * invN);
          } else {
            const long sp = spatial(s, e0 + f);
            const cplx<R> d = cvt<R>(dk_at(s, e0 + f));
            cplx<R> v = cscale(cmul(tile[q], d), invN);
            if (a.invB) v = cscale(v, a.invB[(long)comp * g.N + sp]);
            a.out[(long)(slot * a.vec_per_slot + vec) * a.fstride + (long)comp * g.N + sp] = v;
          }
        }
      }
      __syncthreads();
    }
  }
  pdl_trigger();
  if constexpr (QBQ || MODE == PEN_QRS_IN) {
    for (int q = threadIdx.x; q < Ls * TW; q += NT) {
      const int row = q / TW, f = q - row * TW;
      const int s = QBQ && !kStatQBQ && row > 0 ? Ls - row : row;
      if (f < tw_n) a.T[fb + (long)s * P + e0 + f] = tile[q];
    }
  }
  if constexpr (MODE == PEN_QBQ_CG) {
    // <v, Av> for A = Q_r^* B^-1 Q_r: Q_r^* is N times the adjoint of Q_r (unnormalised
    // forward DFT against the 1/N-scaled inverse), so <v, Av> = N ||B^-1/2 Q_r v||^2 =
    // (1/N) sum_e |IDFT(Pi v)_e|^2 / eps_e, real and positive (CG.cu:57-63, with Zdotc
    // formed in the field domain).  This CTA writes its partial sum; the CG plane stage
    // sums the slot's partials in order.
    double acc[1] = {(double)dot};
    __shared__ double sred[32];
    block_reduce<1>(acc, sred);
    if (threadIdx.x == 0) a.partials[(size_t)slot * a.pstride + blockIdx.y * gridDim.x + blockIdx.x] = acc[0];
  }
}

// Pipelined Q_r^* B^-1 Q_r pencil stage for the static 96^3 geometry (used in FP64,
// where it takes 26.5 instead of 28.5 us per k-point at batch 20).  Each CTA
// walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ... of all k-points in the
// launch and streams the next tile's field and 1/eps rows into its second buffer
// (16-byte cp.async, one copy group per tile) while it transforms the current one,
// so the memory phase of one tile runs under the transforms of the previous.
// grid = (resident CTAs), kPencilThreads threads.
// Tile t of a pipelined 96^3 pencil launch (t = ((slot * 3 * vec_per_slot + 3 * vec
// + comp) * 96 + m) * nft + fast block): its slot (returned), component, field base
// of that component and offset of its first element in every slow-axis plane.
template <typename R>
__device__ __forceinline__ int pencil_pipe_tile(const PencilArgs<R>& a, int t, long& fb, int& off, int& comp) {
  constexpr int TW = PencilTW<R>::v, nft = 96 / TW, per_vec = 96 * nft;
  const int per_slot = 3 * a.vec_per_slot * per_vec;
  const int slot = t / per_slot;
  const int r = t - slot * per_slot;
  const int y = r / per_vec, x = r - y * per_vec;
  comp = y % 3;
  const int vec = y / 3;
  const int m = x / nft, f0 = (x - m * nft) * TW;
  fb = (long)(slot * a.vec_per_slot + vec) * a.fstride + (long)comp * a.g.N;
  off = m * 96 + f0;
  return slot;
}
template <typename R> __device__ __forceinline__ bool pencil_pipe_live(const PencilArgs<R>& a, int t, const unsigned* on) {
  const int slot = t / (3 * a.vec_per_slot * 96 * (96 / PencilTW<R>::v));
  return (on[slot >> 5] >> (slot & 31)) & 1;
}
// Starts the 16-byte copies of tile t's field rows and 1/eps rows into (tile, ibt).
template <typename R>
__device__ __forceinline__ void pencil_pipe_issue(const PencilArgs<R>& a, int t, int total, const unsigned* on, cplx<R>* tile,
                                                  R* ibt) {
  constexpr int TW = PencilTW<R>::v, P = 96 * 96;
  constexpr int CH = 16 / sizeof(cplx<R>), CHB = 16 / sizeof(R);
  if (t >= total || !pencil_pipe_live(a, t, on)) return;
  long fb;
  int off, comp;
  pencil_pipe_tile<R>(a, t, fb, off, comp);
  const long ib = (long)comp * a.g.N;
  for (int q = threadIdx.x; q < 96 * (TW / CH); q += kPencilThreads) {
    const int s = q / (TW / CH), c = q - s * (TW / CH);
    cp_async16(tile + s * TW + c * CH, a.T + fb + (long)s * P + off + c * CH);
  }
  for (int q = threadIdx.x; q < 96 * (TW / CHB); q += kPencilThreads) {
    const int s = q / (TW / CHB), c = q - s * (TW / CHB);
    cp_async16(ibt + s * TW + c * CHB, a.invB + ib + (long)s * P + off + c * CHB);
  }
}

// DOT: also the partial sum of <v, Av> of every tile (PEN_QBQ_CG).
template <typename R, bool DOT>
__global__ void __launch_bounds__(kPencilThreads, sizeof(R) == 4 ? 3 : 2) k_pencil_pipe(PencilArgs<R> a) {
  FAME_COUNT_LAUNCH();
  pdl_wait();
  using GP = Stat96<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Geom& g = a.g;
  constexpr int TW = PencilTW<R>::v;
  constexpr int Lf = 96, Lm = 96, Ls = 96, P = Lf * Lm;
  constexpr int nft = Lf / TW;
  constexpr int TILE = Ls * TW;
  constexpr int CHB = 16 / sizeof(R);  // 1/eps values per 16-byte copy
  static_assert(Lf % TW == 0 && TW % CHB == 0, "whole tiles of whole 16-byte copies");
  cplx<R>* tiles = reinterpret_cast<cplx<R>*>(smem_raw);     // [2][TILE]
  R* ibts = reinterpret_cast<R*>(tiles + 2 * TILE);            // [2][TILE]
  cplx<R>* tws = reinterpret_cast<cplx<R>*>(ibts + 2 * TILE);  // [Ls]
  __shared__ double sred[32];
  for (int i = threadIdx.x; i < Ls; i += kPencilThreads) tws[i] = a.tw[g.tws + i];
  const int total = a.nslots * 3 * a.vec_per_slot * Lm * nft;
  // the live k-points (a slot of this grid takes over 0.3 GB, so 1024 of them do not fit), and,
  // in the first CTA of a CG's launch, the end of the iteration for each
  __shared__ unsigned on[32];
  __shared__ int goes_on;
  if (threadIdx.x < 32) on[threadIdx.x] = 0;
  if (threadIdx.x == 0) goes_on = 0;
  __syncthreads();
  for (int q = threadIdx.x >> 5; q < a.nslots; q += kPencilThreads / 32) {
    int live = a.slots[q].active;
    if (live && DOT && a.cg_in) {
      live = a.cg_in[q].active;
      if (live && blockIdx.x == 0 && cg_advance(a, q, true) && (threadIdx.x & 31) == 0) goes_on = 1;
    } else if (live && a.gate == 1)
      live = a.cg[q].active;
    else if (live && a.gate == 2)
      live = a.cg[q].outer_active;
    if ((threadIdx.x & 31) == 0 && live) atomicOr(&on[q >> 5], 1u << (q & 31));
  }
  __syncthreads();
  if (DOT && a.cg_in && blockIdx.x == 0 && threadIdx.x == 0) decide_cond(a.cond, goes_on);
  int t = blockIdx.x;
  pencil_pipe_issue<R>(a, t, total, on, tiles, ibts);
  cp_async_commit();
  for (int b = 0; t < total; b ^= 1, t += gridDim.x) {
    // buffer b ^ 1 was released at the end of the last iteration
    pencil_pipe_issue<R>(a, t + gridDim.x, total, on, tiles + (b ^ 1) * TILE, ibts + (b ^ 1) * TILE);
    cp_async_commit();
    cp_async_wait_group<1>();  // this tile's group has landed
    __syncthreads();
    if (pencil_pipe_live(a, t, on)) {  // uniform over the CTA
      cplx<R>* tile = tiles + b * TILE;
      double dot[1] = {0.0};
      // inverse, x B^{-1}/N, forward; one FFT call site for the register budget, both
      // transforms forward with the rows counted backwards in between (see k_pencil)
      for (int dir = 0; dir < 2; dir++) {
        GP::template fft_slow<R, 0>(tile, a.ax, tws);
        if (dir == 0) {
          const R invN = (R)(1.0 / g.N);
          const R* ibt = ibts + b * TILE;
          for (int q = threadIdx.x; q < TILE; q += kPencilThreads) {
            const int row = q / TW;
            const R ib = ibt[row == 0 ? q : q + (Ls - 2 * row) * TW];
            if constexpr (DOT) dot[0] += (double)(ib * cabs2(tile[q]));
            tile[q] = cscale(tile[q], ib * invN);
          }
          __syncthreads();
        }
      }
      long fb;
      int off, comp;
      pencil_pipe_tile<R>(a, t, fb, off, comp);
      for (int q = threadIdx.x; q < TILE; q += kPencilThreads) {
        const int row = q / TW, f = q - row * TW;
        a.T[fb + (long)(row == 0 ? 0 : Ls - row) * P + off + f] = tile[q];
      }
      if constexpr (DOT) {
        const int per_slot = 3 * Lm * nft, slot = t / per_slot;
        block_reduce<1>(dot, sred);
        if (threadIdx.x == 0) a.partials[(size_t)slot * a.pstride + (t - slot * per_slot)] = dot[0];
      }
    }
    __syncthreads();  // every thread is done with buffer b before it is refilled
  }
  cp_async_wait_group<0>();
}

// ------------------------------------------------------------------ plane stage (forward)
// The last CTA of the grid decides whether the refinement loop runs again.  Every CTA, live or
// not, arrives here once.
template <typename R> __device__ __forceinline__ void plane_fwd_decide(const PlaneOutArgs<R>& a) {
  if (grid_last(a.counters + a.nslots, gridDim.x * gridDim.y * gridDim.z)) {
    if (threadIdx.x == 0) {
      int any = 0;
      for (int q = 0; q < a.nslots; q++) any |= a.slots[q].active && a.cg[q].outer_active;
      decide_cond(a.cond, any);
    }
  }
}

template <typename R, bool GEN, int EPI, bool PR, int RARE, class GP>
__global__ void __cluster_dims__(3 * GP::kHalves, 1, 1) __launch_bounds__(GP::template max_plane_threads<R, RARE>(), GP::template plane_min_blocks<R, RARE>())
    k_plane_fwd(PlaneOutArgs<R> a) {
  FAME_COUNT_LAUNCH();
  pdl_wait();
  const Geom& g = a.g;
  {
    const PlanePos p = plane_pos<GP>();
    bool live = a.slots[p.slot].active;
    if constexpr (EPI == EPI_RESID) live = live && a.cg[p.slot].outer_active;
    if (!live) {
      if constexpr (EPI == EPI_RESID) plane_fwd_decide(a);
      return;
    }
    const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
    const cplx<R>* T = a.T + plane_base<R, GP>(g, p, a.vec_per_slot, a.fstride);
    if constexpr (!GEN) plane_load<R, GEN, GP>(g, T, a.tw, p.half, m);
    plane_tables<R, GEN, GP>(g, a.tw, a.tabs + (size_t)p.slot * g.tab_stride, p.s, p.half, m);
    if constexpr (GEN) {
      __syncthreads();  // D_ky is in place
      plane_load<R, GEN, GP>(g, T, a.tw, p.half, m);
    } else {
      cp_async_wait_all();
    }
    __syncthreads();
  }
  plane_forward<R, GEN, RARE, GP>(g, a.ax, a.tabs, a.dkz);
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();  // all three component planes transformed

  const PlaneSmem<R> m = plane_smem_of<R, GP>(g);
  const int Lf = GP::Lf(g), S = GP::S(g), P = GP::P(g), PL = GP::PL(g);
  const PlanePos p = plane_pos<GP>();
  const Slot sl = a.slots[p.slot];
  const double2* tab = a.tabs + (size_t)p.slot * g.tab_stride;
  const cplx<R> lp = lam_plane<R, GEN>(g, tab, p.s);
  const int rank0 = 3 * p.half;
  const cplx<R>* src[3] = {cl.map_shared_rank(m.plane, rank0), cl.map_shared_rank(m.plane, rank0 + 1),
                           cl.map_shared_rank(m.plane, rank0 + 2)};
  const int per = (PL + 2) / 3;
  const int e0 = p.comp * per, e1 = min(PL, e0 + per);
  const int Nd = sl.Nd, off = sl.off;
  const long vb = (long)(p.slot * a.vec_per_slot + p.vec) * a.vstride;
  double acc[1] = {0.0};
  // 3 -> 2 unmix and the epilogue.  The three components (remote shared memory) and
  // the vector operand of KB points per thread are read up front, so one latency of
  // each kind covers KB points.
  constexpr int KB = GP::kStatic ? 4 / GP::kHalves : 2;
  const int NT = GP::plane_threads();
  for (int eb = e0 + threadIdx.x; eb < e1; eb += KB * NT) {
    cplx<R> t[KB][3], va[KB], vb2[KB];
#pragma unroll
    for (int k = 0; k < KB; k++) {
      const int e = eb + k * NT;
      const int r = GP::kStatic ? e / Lf : div_magic(e, g.mLf);
      const int fi = p.s * P + plane_elem<GP>(g, p.half, e, r);
      va[k] = vb2[k] = t[k][0] = t[k][1] = t[k][2] = mk<R>(0, 0);
      if (e < e1 && fi >= off) {
        const long i = fi - off;
        const int q = r * S + (e - r * Lf);
#pragma unroll
        for (int c = 0; c < 3; c++) t[k][c] = src[c][q];
        if constexpr (EPI == EPI_RESID) {
          va[k] = a.b[vb + i];
          vb2[k] = a.b[vb + Nd + i];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < KB; k++) {
      const int e = eb + k * NT;
      const int r = GP::kStatic ? e / Lf : div_magic(e, g.mLf), f = e - r * Lf;
      const int fi = p.s * P + plane_elem<GP>(g, p.half, e, r);
      if (e >= e1 || fi < off) continue;
      const long i = fi - off;
      cplx<R> Lx, Ly, Lz;
      lam_elem<R, GEN>(g, tab, plane_lx<R, GP>(g, tab, m), m.ly, m.lys, lp, p.s, r, f, Lx, Ly, Lz);
      cplx<R> Pc[6];
      pi_from<R>(GEN, PR, Lx, Ly, Lz, Pc);
      const cplx<R> t0 = t[k][0], t1 = t[k][1], t2 = t[k][2];
      const cplx<R> o1 = cadd(cadd(cmulc(Pc[0], t0), cmulc(Pc[1], t1)), cmulc(Pc[2], t2));
      const cplx<R> o2 = cadd(cadd(cmulc(Pc[3], t0), cmulc(Pc[4], t1)), cmulc(Pc[5], t2));
      if constexpr (EPI == EPI_OUT) {
        a.out[vb + i] = o1;
        a.out[vb + Nd + i] = o2;
      } else {  // EPI_RESID
        const cplx<R> r1 = csub(va[k], o1), r2 = csub(vb2[k], o2);
        a.out[vb + i] = r1;
        a.out[vb + Nd + i] = r2;
        acc[0] += (double)(cabs2(r1) + cabs2(r2));
      }
    }
  }
  // This CTA is done reading the other CTAs' planes.  A relaxed arrival (no wait for
  // this CTA's global stores to drain); the matching wait below keeps every plane alive
  // until all three CTAs have read it.
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");

  if constexpr (EPI == EPI_RESID) {
    __shared__ double sred[32];
    block_reduce<1>(acc, sred);
    const int nblk = gridDim.x;  // CTAs of this slot (vec_per_slot == 1 in solves)
    double tot[1];
    if (slot_reduce<1>(acc, a.partials + (size_t)p.slot * nblk, a.counters + p.slot, blockIdx.x, nblk, tot)) {
      if (threadIdx.x == 0) {
        CgState* st = a.cg + p.slot;
        st->rr = tot[0];
        st->outer++;
        st->outer_total++;
        st->outer_active = (tot[0] > st->otol2) && (st->outer < st->outer_max);
        st->scale = 1.0 / sqrt(tot[0] > 0 ? tot[0] : 1.0);
        __threadfence();
      }
    }
    plane_fwd_decide(a);
  }
  asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");  // every CTA has read this plane
}

}  // namespace fame
