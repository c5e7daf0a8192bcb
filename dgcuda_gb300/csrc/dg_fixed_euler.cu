// dg_fixed_euler.cu -- the fixed-point element stage and traces of the Euler
// module, p = 1..4.
#include "dg_fixed_launch.cuh"

namespace dg {
namespace fx {
template void element<Euler>(const Ctx &, const ElemArgs &, int);
template void trace<Euler>(const Ctx &, double *, int);
}  // namespace fx
}  // namespace dg
