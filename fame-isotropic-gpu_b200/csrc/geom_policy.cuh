// Geometry policies of the operator kernels.
//
// DynGeom takes every length from the runtime Geom and runs the runtime-planned
// FFT passes (any grid).  StatGeom<LF, LM, LS> fixes the fast, mid and slow line
// lengths at compile time: the FFT passes are fully unrolled and all index
// arithmetic folds to constants.  The solver instantiates StatGeom for the grids
// it runs most (cubic 96^3) and falls back to DynGeom elsewhere.
#pragma once
#include "state.cuh"

namespace fame {

constexpr int kPlaneThreads = 512;      // most threads of a plane CTA that an option can set
constexpr int kPencilThreads = 256;     // threads of a pencil CTA (at most, with runtime plans)

struct DynGeom {
  static constexpr bool kStatic = false;
  // Launch bounds of the plane kernels: registers per thread.  FP32: 80 (768 threads per
  // SM), so 24 warps are resident whether a CTA has 96 threads or 768.  FP64, and the kernels
  // with the prime pass (RARE 2), whose MU x ML accumulator block needs more: 128 (512).
  template <typename R, int RARE> static constexpr int max_plane_threads() {
    return sizeof(R) == 4 && RARE < 2 ? 768 : 512;
  }
  __device__ __forceinline__ static int plane_threads() { return blockDim.x; }
  __device__ __forceinline__ static int pencil_threads() { return blockDim.x; }
  // plane CTAs of that size per SM the register budget is sized for (launch bounds)
  template <typename R, int RARE> static constexpr int plane_min_blocks() { return 1; }
  __device__ __forceinline__ static int Lf(const Geom& g) { return g.Lf; }
  __device__ __forceinline__ static int Lm(const Geom& g) { return g.Lm; }
  __device__ __forceinline__ static int Ls(const Geom& g) { return g.Ls; }
  __device__ __forceinline__ static int S(const Geom& g) { return g.S; }
  __device__ __forceinline__ static int P(const Geom& g) { return g.P; }
  static constexpr int kHalves = 1;  // CTAs that share a component's plane (StatGeom)
  __device__ __forceinline__ static int PL(const Geom& g) { return g.P; }  // points of a CTA's share
  // lines of a plane (pitch S) along its fast axis (fast = true) or mid axis, and
  // the TW lines of a pencil tile.  One FFT call site per kernel keeps the kernel
  // within its register budget, so the plane axis is a runtime argument.  Forward transforms
  // only: the inverse ones run on values with swapped parts (plane stages) or come out in
  // reversed order (pencil stage), which takes the conjugations and sign choices of a runtime
  // direction out of every pass.
  // MUL (General lattices): conj(pre) on the inputs, conj(post) on the outputs of the mid axis
  template <typename R, int RARE, bool MUL>
  __device__ __forceinline__ static void fft_plane(cplx<R>* b, const AxisPasses& A, bool, const cplx<R>* tw,
                                                   const cplx<R>* pre, const cplx<R>* post) {
    fft_lines<R, Emax<R>::v, RARE, false, MUL>(b, A, tw, pre, post);
  }
  // whether the mid axis can take pre and post (its first and last pass are butterflies)
  __device__ __forceinline__ static bool mul_ok(const AxisPasses& A) {
    return A.d[0].radix <= 13 && A.d[A.npass - 1].radix <= 13;
  }
  template <typename R, int RARE>
  __device__ __forceinline__ static void fft_slow(cplx<R>* b, const AxisPasses& A, const cplx<R>* tw) {
    fft_lines<R, Emax<R>::v, RARE, true>(b, A, tw);
  }
};

// elements a thread stages per round in the static passes: plane passes (96 registers at three
// CTAs per SM) and pencil passes
template <typename R> struct SEmax;
template <> struct SEmax<float> { static constexpr int v = 24; };
template <> struct SEmax<double> { static constexpr int v = 12; };
template <typename R> struct SPenEmax;
template <> struct SPenEmax<float> { static constexpr int v = 24; };
template <> struct SPenEmax<double> { static constexpr int v = 12; };
// static plane passes of the runtime-geometry grids (96 to 128 registers, the general-lattice
// Pi mixing in the same kernel): half the 96^3 staging in FP32, a third in FP64, which
// keeps the radix-11 and radix-13 passes of the FCC and BCC planes in registers (measured with two
// 256-thread CTAs per SM; FCC 64x55x52: FP32 CG iteration 37.5 -> 33.9 us per k-point; BCC
// 48x45x39: FP64 plane stages 23.5 -> 20.7 us)
template <typename R> struct PlaneEmax;
template <> struct PlaneEmax<float> { static constexpr int v = 12; };
template <> struct PlaneEmax<double> { static constexpr int v = 4; };
// static slow-axis passes of the runtime-geometry grids (80 registers at three
// pencil CTAs per SM, the general-lattice twiddles in the same kernel): a third of
// the 96^3 pencil staging, which removes the FP32 spills (hexagonal 128-point slow
// axis: FP32 pencil stage 37.6 -> 28.3 us per k-point)
template <typename R> struct SlowEmax;
template <> struct SlowEmax<float> { static constexpr int v = 8; };
template <> struct SlowEmax<double> { static constexpr int v = 4; };

// DynGeom with the slow-axis length fixed at compile time: the pencil stage's
// slow-axis transforms run the static plan (unrolled passes, constant strides and
// twiddle indices); everything else stays runtime.  The solver uses it for the
// pencils of runtime-geometry grids whose slow axis is one of the lengths
// instantiated in ops_slow_static.cu.
template <int LSL>
struct DynGeomSlow : DynGeom {
  __device__ __forceinline__ static constexpr int pencil_threads() { return kPencilThreads; }
  template <typename R, int RARE>
  __device__ __forceinline__ static void fft_slow(cplx<R>* b, const AxisPasses&, const cplx<R>* tw) {
    constexpr int TW = PencilTW<R>::v;
    sfft<R, LSL, TW, kPencilThreads, SlowEmax<R>::v>(b, 1, TW, tw, false);
  }
};

// DynGeom with the two plane axes' lengths fixed at compile time: the plane stages'
// fast- and mid-axis transforms run static plans (spass, and the prime pass with
// constant sizes); T threads per plane CTA, MB CTAs per SM in the register budget.
// Index arithmetic outside the transforms stays runtime.  The solver uses it for the
// plane stages of the runtime-geometry grids instantiated in ops_plane_static.cu.
template <int LF, int LM, int T, int MB>
struct DynGeomPlane : DynGeom {
  static constexpr int kMaxPlaneThreads = T;
  template <typename R, int RARE> static constexpr int max_plane_threads() { return T; }
  __device__ __forceinline__ static constexpr int plane_threads() { return T; }
  template <typename R, int RARE> static constexpr int plane_min_blocks() { return MB; }
  template <typename R, int RARE, bool MUL>
  __device__ __forceinline__ static void fft_plane(cplx<R>* b, const AxisPasses&, bool fast, const cplx<R>* tw,
                                                   const cplx<R>* pre, const cplx<R>* post) {
    if (fast)
      sfft<R, LF, LM, T, PlaneEmax<R>::v>(b, LF | 1, 1, tw, false);
    else
      sfft<R, LM, LF, T, PlaneEmax<R>::v>(b, 1, LF | 1, tw, false, pre, post);
  }
  __device__ __forceinline__ static constexpr bool mul_ok(const AxisPasses&) {
    return splan_radix(LM, 0) <= 13 && splan_radix(LM, splan_count(LM) - 1) <= 13;
  }
};

// H = 2: two CTAs share a component's plane, split by the first radix-2 step of the mid axis
// (decimation in frequency): half h holds the frequencies 2 r + h as row r, so that a
// transform of LM / 2 points on each CTA's own rows is all that is left of that axis.  The forward
// stage takes its step as it loads the plane (rows m and m + LM / 2 are read by both halves, the
// second time from L2), the inverse one as it stores it (through distributed shared memory).
template <int LF, int LM, int LSL, int T, int MB, int H = 1>
struct StatGeom {
  static constexpr bool kStatic = true;
  static constexpr int kHalves = H;
  static constexpr int kS = LF | 1, kLf = LF, kLm = LM / H, kThreads = T;
  template <typename R, int RARE> static constexpr int max_plane_threads() { return T; }
  __device__ __forceinline__ static constexpr int plane_threads() { return T; }
  __device__ __forceinline__ static constexpr int pencil_threads() { return kPencilThreads; }
  template <typename R, int RARE> static constexpr int plane_min_blocks() { return MB; }
  __device__ __forceinline__ static constexpr int Lf(const Geom&) { return LF; }
  __device__ __forceinline__ static constexpr int Lm(const Geom&) { return kLm; }  // rows of a CTA's share
  __device__ __forceinline__ static constexpr int Ls(const Geom&) { return LSL; }
  __device__ __forceinline__ static constexpr int S(const Geom&) { return kS; }
  __device__ __forceinline__ static constexpr int P(const Geom&) { return LF * LM; }
  __device__ __forceinline__ static constexpr int PL(const Geom&) { return LF * kLm; }
  static_assert(LF == LM, "a static plane geometry has equal fast and mid lengths");
  template <typename R, int RARE>
  __device__ __forceinline__ static void fft_slow(cplx<R>* b, const AxisPasses&, const cplx<R>* tw) {
    fft_slow_c<R, false>(b, tw);
  }
  // Passes with the axis and the direction fixed at compile time: every
  // stride, twiddle sign and rotation folds to a constant (one call site each).
  template <typename R, bool FAST, bool INV>
  __device__ __forceinline__ static void fft_plane_c(cplx<R>* b, const cplx<R>* tw) {
    if constexpr (FAST)
      sfft<R, LF, kLm, T, SEmax<R>::v>(b, kS, 1, tw, INV);
    else
      sfft<R, kLm, LF, T, SEmax<R>::v, H>(b, 1, kS, tw, INV);
  }
  template <typename R, bool INV>
  __device__ __forceinline__ static void fft_slow_c(cplx<R>* b, const cplx<R>* tw) {
    constexpr int TW = PencilTW<R>::v;
    sfft<R, LSL, TW, kPencilThreads, SPenEmax<R>::v>(b, 1, TW, tw, INV);
  }
};

// 96^3.  FP32: three plane CTAs of 192 threads per SM.  An FP64 plane is 149 KB, one CTA per SM, and one
// k-point is then three rounds of clusters (45 of 96 at a time); with halves (75 KB) it is
// again three CTAs of 192 threads per SM: FP64 operator 151.9 -> 133.9 us (one k-point), 105.9 -> 94.1
// (ten).  256 threads, at two or three CTAs per SM, 149.5 and 142.5; 128 threads 142.0.
template <typename R> using Stat96 = StatGeom<96, 96, 96, 192, 3, sizeof(R) == 4 ? 1 : 2>;
// The CG plane stage keeps whole planes in FP64: at the 96 registers of three CTAs a thread has one point of the
// recurrences in flight, and what the halves gain in the transforms is lost (plain FP64 solve of
// one k-point: 324 ms whole, 343 halves, 326 halves of 128 threads).
template <typename R>
using Stat96Cg = StatGeom<96, 96, 96, sizeof(R) == 4 ? 192 : 384, sizeof(R) == 4 ? 3 : 1>;
// static plane plans of the general-lattice benchmark grids (fast, mid, threads, CTAs per SM)
template <typename R> using PlaneFcc64 = DynGeomPlane<52, 55, 128, sizeof(R) == 4 ? 5 : 4>;
template <typename R> using PlaneBcc48 = DynGeomPlane<39, 45, 128, sizeof(R) == 4 ? 5 : 4>;
template <typename R>
using PlaneHex128 = DynGeomPlane<92, 107, sizeof(R) == 4 ? 256 : 512, sizeof(R) == 4 ? 2 : 1>;

}  // namespace fame
