// qas_stage1d.cu -- the 1D stage kernels (a translation unit of its own for the build's sake; without
// QAS_SEPARATE_UNITS qas_api.cu includes it)
#include "qas_stage1d.cuh"

namespace qas {

template <int ODR>
static Stage1Fn stage1_of(int rmn)
{
  switch (rmn) {
    case 0: return k_stage1<ODR, 0>;
    case 1: return k_stage1<ODR, 1>;
    case 2: return k_stage1<ODR, 2>;
    default: return k_stage1<ODR, 3>;
  }
}
Stage1Fn stage1_kernel(int odr, int rmn) { return odr == 2 ? stage1_of<2>(rmn) : stage1_of<4>(rmn); }

}  // namespace qas
