// dg_kernels_euler.cu -- kernel instances for the Euler module, p = 0..5.
#include "dg_kernels.cuh"

namespace dg {
namespace {

using L = Launch<Euler>;

Ops make_ops() {
  Ops o = L::ops();
  o.face_fs = L::face_fs;
  o.means = L::means;
  o.element_lim = L::element_lim;
  return o;
}

}  // namespace

const Ops &ops_euler() {
  static const Ops o = make_ops();
  return o;
}
const BatchOps &batch_ops_euler() {
  static const BatchOps o = [] {
    BatchOps b = Launch<Euler>::batch_ops();
    b.face_fs = Launch<Euler>::b_face_fs;
    b.means = Launch<Euler>::b_means;
    b.element_lim = Launch<Euler>::b_element_lim;
    return b;
  }();
  return o;
}
}  // namespace dg
