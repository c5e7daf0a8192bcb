// dg_fixed_maxwell.cu -- the fixed-point element stage and traces of the Maxwell
// module, p = 1..4.
#include "dg_fixed_launch.cuh"

namespace dg {
namespace fx {
template void element<Maxwell>(const Ctx &, const ElemArgs &, int);
template void trace<Maxwell>(const Ctx &, double *, int);
template void batch_element<Maxwell>(const BatchLaunch &, cudaStream_t, int, int, int, int, int,
                                  int);
template void batch_limit<Maxwell>(const BatchLaunch &, int, int, int, int, int);
}  // namespace fx
}  // namespace dg
