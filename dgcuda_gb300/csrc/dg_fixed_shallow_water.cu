// dg_fixed_shallow_water.cu -- the fixed-point element stage and traces of the ShallowWater
// module, p = 1..4.
#include "dg_fixed_launch.cuh"

namespace dg {
namespace fx {
template void element<ShallowWater>(const Ctx &, const ElemArgs &, int);
template void trace<ShallowWater>(const Ctx &, double *, int);
template void batch_element<ShallowWater>(const BatchLaunch &, cudaStream_t, int, int, int, int, int,
                                  int);
template void batch_limit<ShallowWater>(const BatchLaunch &, int, int, int, int, int);
}  // namespace fx
}  // namespace dg
