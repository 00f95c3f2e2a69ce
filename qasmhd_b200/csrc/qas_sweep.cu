// qas_sweep.cu -- the face-sweep kernels (a translation unit of its own for the build's sake; without
// QAS_SEPARATE_UNITS qas_api.cu includes it)
#include "qas_kernels.cuh"

namespace qas {

// AX = 7 (2nd order): every axis of a stage in one launch, the short blocks of the x faces filling the gaps
// that the marching blocks leave at their end.  The 4th order launches each axis by itself: together
// the three paths spill more (KH 160^3 1890 -> 1950 us a stage, OT 1024^2 1198 -> 1236 us a step).
template <int ODR, int RMN, int PR, int AX>
__global__ void __launch_bounds__(SWB, QAS_SWEEP_MINB_OF(RMN)) k_sweep(const __grid_constant__ View v,
                                                                       const __grid_constant__ SweepPlan pl)
{
  pdl_begin();
  if (v.ctl->done) return;
  __shared__ double sm[SLOTS * SLP];
  sweep_block<ODR, RMN, PR, AX, (PR < 0)>(v, pl, blockIdx.x, sm);
}

template <int ODR, int PR, int AX>
static SweepFn sweep_of(int rmn)
{
  switch (rmn) {
    case 0: return k_sweep<ODR, 0, PR, AX>;
    case 1: return k_sweep<ODR, 1, PR, AX>;
    case 2: return k_sweep<ODR, 2, PR, AX>;
    default: return k_sweep<ODR, 3, PR, AX>;
  }
}
template <int PR>
static SweepFn sweep_of_axis(int rmn, int ax)
{
  return ax == 1 ? sweep_of<4, PR, 1>(rmn) : (ax == 2 ? sweep_of<4, PR, 2>(rmn) : sweep_of<4, PR, 4>(rmn));
}
SweepFn sweep_kernel(int odr, int rmn, bool any, int ax)
{
  if (odr == 2) return sweep_of<2, 0, 7>(rmn);
  return any ? sweep_of_axis<-1>(rmn, ax) : sweep_of_axis<0>(rmn, ax);
}

}  // namespace qas
