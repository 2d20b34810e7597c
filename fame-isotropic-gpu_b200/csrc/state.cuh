// State, loop conditions and kernel argument structs shared by the operator
// kernels (op_kernels.cuh) and the solver kernels (solver_kernels.cuh).
#pragma once
#include "operator.cuh"

namespace fame {

// complex elements a thread stages in registers during one round of a runtime-plan
// pass (per precision; a radix above it stages one butterfly)
template <typename R> struct Emax;
template <> struct Emax<float> { static constexpr int v = 16; };
template <> struct Emax<double> { static constexpr int v = 8; };
// plane positions per pencil CTA: 256-byte rows
template <typename R> struct PencilTW { static constexpr int v = 256 / (int)sizeof(cplx<R>); };

// ------------------------------------------------------------------ state
struct CgState {
  double r1, r1p;            // ||r||^2 now / one iteration before
  double gm, rho;            // the last iteration's gamma and rho (cg_coefficients)
  double tol2;               // stop threshold on ||r||^2
  int iter;                  // the reference's counter k (starts at 1, CG.cu:36)
  int active;
  int maxit;
  int total;                 // CG products accumulated for the profile counter
  // outer iterative refinement (mixed precision; FP64 at a high contrast)
  double rr, scale;          // ||b - A y||^2, 1/||b - A y|| used to scale the FP32 rhs
  double otol2;              // stop threshold of the refinement on ||b - A y||^2 (ls_tol^2)
  int outer, outer_active, outer_max, outer_total;
  double bb, rr_old;         // FP64: ||b||^2, and rr one restart before
  int rounded;               // FP64: the residual has reached what FP64 can hold
};

// gamma = ||r||^2 / <r, A r> and rho of the three-term CG recurrences (k_plane_cg) from the state
// before the iteration and <r, A r>.  <r, A r> <= 0 (a residual of zero, or an FP32 sum that
// underflowed): no step, gamma = 0.  rho = 1 starts the recurrences afresh from the current r and x: in
// the first iteration, after one without a step, and where rounding leaves nothing of the
// denominator (1 / rho is a product of step ratios of CG, far above 1e-12 in exact arithmetic).
__host__ __device__ __forceinline__ void cg_coefficients(const CgState& st, double rAr, double& gm, double& rho) {
  gm = rAr > 0 ? st.r1 / rAr : 0.0;
  if (!(gm <= 1e300)) gm = 0.0;
  rho = 1.0;
  if (st.iter > 1 && gm > 0 && st.gm > 0) {
    const double den = 1.0 - (gm / st.gm) * (st.r1 / st.r1p) / st.rho;
    if (den > 1e-12) rho = 1.0 / den;
  }
}

// What bounds an A_r^-1 solve: by value in a solve's graph, from device memory in the graph of the
// operator apply, which serves every tolerance and product cap.
struct LsParams {
  double tol2;               // ls_tol^2
  double floor2, rounding2;  // FP64 with restarts: k_cg64_init
  int maxit;
};

struct LzState {
  int converged;
  int restarts;
  int nconv;
  int keep;  // Lanczos vectors the last restart kept: steps j < keep are not this slot's (0 before)
};

// Condition of one CUDA-graph WHILE node (in host-driven mode only `flag` is used).
// Every loop is fail-safe: the first kernel of the body clears the condition, the
// deciding kernel sets it again only while work remains and the loop's trip count
// (counted on the device) is below `cap`; hitting the cap records an overflow in
// trips[1] and ends the loop, so no data-dependent loop can run unbounded.
struct Cond {
  cudaGraphConditionalHandle handle;
  int* flag;
  int* trips;  // [0] trips of the current loop, [1] overflow marker
  int cap;
};

__device__ __forceinline__ void set_cond(const Cond& c, int v) {
  if (!c.flag) return;
  *c.flag = v;
  if (c.handle) cudaGraphSetConditional(c.handle, (unsigned)v);
}

// decision at the end of a loop body
__device__ __forceinline__ void decide_cond(const Cond& c, int any) {
  if (c.trips) {
    const int t = ++c.trips[0];
    if (any && t >= c.cap) {
      c.trips[1] = 1;
      any = 0;
    }
  }
  set_cond(c, any);
}

// before the loop: reset the trip counter and set the first decision
__device__ __forceinline__ void start_cond(const Cond& c, int any) {
  if (c.trips) c.trips[0] = 0;
  set_cond(c, any);
}

// Ticket counter over the whole grid: true in exactly one CTA, the last one.
__device__ __forceinline__ bool grid_last(unsigned* ctr, unsigned total) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ctr, 1u) == total - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    *ctr = 0u;
  }
  return last;
}

// D_kz(x, y, z) = e^{i 2 pi phi(x,y) z / Nz} (…Lambdas.cu:389-400)
template <typename R>
__device__ __forceinline__ cplx<R> dkz_at(const Geom& g, const double2* tab, int x, int y, int z) {
  const double ph = tab[g.oPhi + x * g.Ny + y].x;
  const double a = ph * z * g.tnz;  // e^{i pi a}, a = 2 ph z / Nz
  if constexpr (sizeof(R) == 8) {
    return expipi(a);
  } else {
    // FP32: the argument reduced to [-1, 1] in FP64 (a - 2n changes nothing), then a
    // single-precision sincospi
    return expipi((float)(a - 2.0 * rint(0.5 * a)));
  }
}

// ------------------------------------------------------------------ plane stage
// IN_CG: the start residual of a CG solve (gated on the solve being active)
enum InMode { IN_VEC = 0, IN_CG = 1, IN_REFINE = 2 };
enum EpiMode { EPI_OUT = 0, EPI_RESID = 2 };
// PEN_QBQ_CG: PEN_QBQ that also reduces <v, Av> = (1/N) sum_e |(IDFT Pi v)_e|^2 / eps_e
enum PencilMode { PEN_QBQ = 0, PEN_QR_OUT = 1, PEN_QRS_IN = 2, PEN_QBQ_CG = 3 };

template <typename R>
struct PlaneInArgs {
  Geom g;
  AxisPasses ax[2];       // runtime plans: fast and mid axis
  const Slot* slots;
  const double2* tabs;
  const cplx<R>* dkz;     // General: D_kz of every slot (N values each), or NULL
  const cplx<R>* tw;      // forward twiddle tables, R precision
  long vstride;           // per-slot stride of reduced vectors (elements)
  long fstride;           // per-slot stride of 3N fields (elements)
  int vec_per_slot;       // number of vectors per slot (batched Qr over bands)
  const cplx<R>* in;      // IN_VEC, IN_CG: reduced input
  const CgState* cg;      // IN_CG / IN_REFINE
  double2* y64;           // IN_REFINE: FP64 accumulated solution (updated)
  const float2* x32[2];   // IN_REFINE: FP32 correction, the buffer of the last iteration's parity
  int sigma;              // IN_VEC: multiply the input by sqrt(Lambda_q) first (Sigma, …_Isotropic.cu:109)
  cplx<R>* T;             // output field (3 components)
  int* fault;             // set to 1 if a bounded wait of the component exchange ran out (or NULL)
  int* fault_host;        // the same in pinned host memory
};

template <typename R>
struct PlaneCgArgs {
  Geom g;
  AxisPasses ax[2];
  const Slot* slots;
  const double2* tabs;
  const cplx<R>* dkz;
  const cplx<R>* tw;
  long vstride, fstride;
  cplx<R>* r[2];          // residual: buffer iter & 1 is the current one, the other r_old / r'
  cplx<R>* x[2];          // solution, the same way
  const CgState* cg;
  CgState* cg_copy;       // the state with this iteration's gamma and rho, for the pencil stage that ends it
  cplx<R>* T;             // field of A r before the forward plane transforms in, of r' out
  double* partials;       // per slot: the pencil's <r, A r> parts, then this kernel's ||r'||^2 parts
  long pstride;           // per-slot stride of `partials`
  int pen_parts;
  Cond reset;             // loop condition cleared by this kernel, the first of the loop body
  int self_pf;            // L2 prefetch of this CTA's own vectors, once its plane has arrived
  int *fault, *fault_host;
};

template <typename R>
struct PencilArgs {
  Geom g;
  AxisPasses ax;           // runtime plans: slow axis
  const Slot* slots;
  const double2* tabs;
  const cplx<R>* tw;
  long fstride;
  int vec_per_slot;
  cplx<R>* T;              // field in frequency-plane layout (in/out)
  const R* invB;           // PEN_QBQ and PEN_QR_OUT (optional): 1/eps per edge, 3N
  int ib_field;            // invB in the field layout (else the spatial layout; same for Simple lattices)
  cplx<R>* out;            // PEN_QR_OUT: spatial field out (3N per vector)
  const cplx<R>* in;       // PEN_QRS_IN: spatial field in
  CgState* cg;             // optional activity gate; the new state of a CG iteration (cg_in set)
  const CgState* cg_in;    // PEN_QBQ_CG at the end of a CG iteration: the plane stage's copy, else NULL
  int pen_parts, fwd_parts;  // partial sums per slot: <r, A r> (at the slot's start), then ||r'||^2
  Cond cond;               // CG WHILE condition (cg_in set)
  int gate;                // 0 none, 1 CG active, 2 outer refinement active
  double* partials;        // PEN_QBQ_CG: partial sums of <v, Av>, [slot * pstride + CTA (or tile) of the slot]
  long pstride;            // per-slot stride of `partials`
  int TW;                  // plane positions per CTA
  int nslots;              // k-points of the launch (k_pencil_pipe walks all their tiles)
  int pf_dist;             // > 0: L2 prefetch of the tile of the CTA this many places later
};

template <typename R>
struct PlaneOutArgs {
  Geom g;
  AxisPasses ax[2];
  const Slot* slots;
  const double2* tabs;
  const cplx<R>* dkz;
  const cplx<R>* tw;
  long vstride, fstride;
  int vec_per_slot;
  const cplx<R>* T;        // field after the slow-axis forward pass
  cplx<R>* out;            // EPI_OUT: reduced output; EPI_RESID: r (FP64)
  const cplx<R>* b;        // EPI_RESID: right-hand side
  CgState* cg;
  double* partials;        // EPI_RESID: [nslots][blocks per slot]
  unsigned* counters;      // [nslots] ticket counters, plus [nslots] = grid counter
  Cond cond;               // EPI_RESID: outer WHILE condition
  int nslots;
};

// Ordered sum of p[0], p[stride], ..., p[(n - 1) stride] by one warp (lane-strided,
// then a fixed shuffle tree); valid in all lanes.
__device__ __forceinline__ double warp_sum_strided(const double* p, int n, int stride) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int i = lane; i < n; i += 32) s += p[(size_t)i * stride];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// warp_sum_strided over data other CTAs of this grid wrote (loads through L2, not L1).
__device__ __forceinline__ double warp_sum_strided_cg(const double* p, int n, int stride) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int i = lane; i < n; i += 32) s += __ldcg(p + (size_t)i * stride);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Ordered sum of n partial sums by one warp (lane-strided, then a fixed shuffle tree):
// every caller gets the same bits, so CTAs that need the same CG scalar agree exactly.  Valid in
// all lanes.  U independent loads per lane are in flight per round (a few hundred partials take
// one or two L2 round trips, not one per element); they take 2 U registers.
template <int U = 16> __device__ __forceinline__ double warp_sum_partials(const double* p, int n) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int b = 0; b < n; b += 32 * U) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = b + u * 32 + lane;
      v[u] = i < n ? p[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) s += v[u];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

}  // namespace fame
