// Pass kernels of the 512^3 grid: the default of each class and autotuner candidates.  The first column
// variant also serves the single-field transforms.  All column variants run the two-stage plan (one
// exchange; the three-stage 16 x 8 x 4 took 630 to 1150 us per launch).  Times per launch (us) of the
// defaults and of the next best: z_inverse 390 / 422, y_inverse 571 / 629 in column pairs, y_forward 710 /
// 752 and z_forward 549 / 557 TMA-fed (column pairs 763 and 545: four warps per SM are too few for the
// full-length loads); x rows 1557 read directly / 1603, hydrodynamics 1124 / 1161.
#include "ops.cuh"

namespace mhdgb {

OpsBase* make_ops_512() {
  auto* o = new Ops<512>();
  o->add_col<Plan<512, 16, 32, 16>, 16, 1, 3, true>();
  o->add_col_tma<Plan<512, 16, 32, 16>, 1, 2, true>(kDefaultZfwd);
  o->add_col_tma<Plan<512, 16, 32, 16>, 1, 3, true>(kDefaultYfwd);
  o->add_col_pair<Plan<512, 16, 32, 16>, 1, 3>(kDefaultZinv | kDefaultYinv);
  o->add_x_form<Plan<512, 32, 8, 8, 8>, 4, 1, 1, 2, true>();
  o->add_x<Plan<512, 64, 8, 8, 8>, 2, 1, 1, 4>();
  o->add_x<Plan<512, 32, 16, 8, 4>, 4, 1, 1, 2>();
  o->add_x<Plan<512, 32, 8, 8, 8>, 4, 1, 1, 2>();
  o->add_x_vp<Plan<512, 64, 8, 8, 8>, 2, 1, 4>();
  o->add_x_hd<Plan<512, 32, 8, 8, 8>, 4, 2>();
  o->add_x_hd<Plan<512, 64, 8, 8, 8>, 2, 4>();
  o->add_x_hdvp<Plan<512, 64, 8, 8, 8>, 2, 4>();
  o->add_x_tc<SPLIT_F16, 4, 2>();
  o->add_x_tc<SPLIT_BF16, 4, 2>();
  o->set_rows<Plan<512, 64, 8, 8, 8>, 2>();
  return o;
}

}  // namespace mhdgb
