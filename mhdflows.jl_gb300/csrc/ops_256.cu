// Pass kernels of the 256^3 grid: the default of each class and autotuner candidates.  The first column
// variant also serves the single-field transforms.  Times per launch (us) of the defaults and of the
// next best: column pairs z_inverse 57 / 61, y_inverse 80 / 87, y_forward 99 / 107 (hydrodynamics 68 /
// 71, with penalty planes 167 / 180), z_forward 77 / 81; x rows in pairs 160 / 170 (hydrodynamics
// 101 / 124).
#include "ops.cuh"

namespace mhdgb {

OpsBase* make_ops_256() {
  auto* o = new Ops<256>();
  o->add_col<Plan<256, 16, 16, 16>, 16, 3>();
  o->add_col<Plan<256, 16, 16, 16>, 8, 6, 3>();
  o->add_col_tma<Plan<256, 16, 16, 16>, 3, 2>();
  o->add_col_tma<Plan<256, 16, 16, 16>, 2, 3>();
  o->add_col_pair<Plan<256, 16, 16, 16>, 2, 3>(kDefaultZinv | kDefaultYinv);
  o->add_col_pair<Plan<256, 16, 16, 16>, 3, 2>(kDefaultYfwd | kDefaultZfwd);
  o->add_x_form<Plan<256, 16, 16, 16>, 1, 1, 1, 8, false, false, true>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 8, 1, 1, 2>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 4, 1, 1, 4>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 4, 3, 1, 3>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 4, 3, 2, 3>();
  o->add_x<Plan<256, 16, 16, 16>, 4, 1, 1, 2>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 2, 1, 1, 8>();
  o->add_x_vp<Plan<256, 32, 8, 8, 4>, 4, 1, 3>();
  o->add_x_hd<Plan<256, 16, 16, 16>, 1, 12, 0, false, true>();
  o->add_x_hd<Plan<256, 32, 8, 8, 4>, 8, 2>();
  o->add_x_hd<Plan<256, 32, 8, 8, 4>, 4, 4>();
  o->add_x_hdvp<Plan<256, 32, 8, 8, 4>, 4, 3>();
  o->add_x_tc<SPLIT_F16, 4, 2>();
  o->add_x_tc<SPLIT_BF16, 4, 2>();
  o->add_x_tc5();
  o->set_rows<Plan<256, 32, 8, 8, 4>, 4>();
  return o;
}

}  // namespace mhdgb
