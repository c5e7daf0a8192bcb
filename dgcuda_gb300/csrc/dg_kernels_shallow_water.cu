// dg_kernels_shallow_water.cu -- kernel instances for the ShallowWater module, p = 0..5.
#include "dg_kernels.cuh"

namespace dg {
const Ops &ops_shallow_water() {
  static const Ops o = [] {
    Ops v = Launch<ShallowWater>::ops();
    v.bed_slopes = Launch<ShallowWater>::bed_slopes;
    return v;
  }();
  return o;
}
const BatchOps &batch_ops_shallow_water() { return Launch<ShallowWater>::batch_ops(); }
}  // namespace dg
