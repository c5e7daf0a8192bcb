// dg_fixed_advection.cu -- the fixed-point element stage and traces of the Advection
// module, p = 1..4.
#include "dg_fixed_launch.cuh"

namespace dg {
namespace fx {
template void element<Advection>(const Ctx &, const ElemArgs &, int);
template void trace<Advection>(const Ctx &, double *, int);
template void batch_element<Advection>(const BatchLaunch &, cudaStream_t, int, int, int, int, int,
                                  int);
template void batch_limit<Advection>(const BatchLaunch &, int, int, int, int, int);
}  // namespace fx
}  // namespace dg
