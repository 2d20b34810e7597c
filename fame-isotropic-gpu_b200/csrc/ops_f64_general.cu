// Operator stage kernels, FP64, General lattices, radices 2 to 13.
#include "op_kernels.cuh"

namespace fame {
template __global__ void k_plane_inv<double, true, IN_CG, false, 0, DynGeom>(PlaneInArgs<double>);
template __global__ void k_plane_inv<double, true, IN_VEC, false, 0, DynGeom>(PlaneInArgs<double>);
template __global__ void k_plane_inv<double, true, IN_VEC, true, 0, DynGeom>(PlaneInArgs<double>);
template __global__ void k_plane_inv<double, true, IN_REFINE, false, 0, DynGeom>(PlaneInArgs<double>);
template __global__ void k_plane_cg<double, true, 0, DynGeom>(PlaneCgArgs<double>);
template __global__ void k_pencil<double, true, PEN_QBQ, 0, DynGeom>(PencilArgs<double>);
template __global__ void k_pencil<double, true, PEN_QBQ_CG, 0, DynGeom>(PencilArgs<double>);
template __global__ void k_pencil<double, true, PEN_QR_OUT, 0, DynGeom>(PencilArgs<double>);
template __global__ void k_pencil<double, true, PEN_QRS_IN, 0, DynGeom>(PencilArgs<double>);
template __global__ void k_plane_fwd<double, true, EPI_OUT, false, 0, DynGeom>(PlaneOutArgs<double>);
template __global__ void k_plane_fwd<double, true, EPI_OUT, true, 0, DynGeom>(PlaneOutArgs<double>);
template __global__ void k_plane_fwd<double, true, EPI_RESID, false, 0, DynGeom>(PlaneOutArgs<double>);
FAME_DEFINE_LAUNCH_GETTER(launches_ops_f64_general)
}  // namespace fame
