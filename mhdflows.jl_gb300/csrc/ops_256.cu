// Pass kernels of the 256^3 grid: the default of each class and autotuner candidates.  The first column
// variant also serves the single-field transforms.  Defaults from the times per launch (us): y_forward
// 107.1 with 8-column tiles and three buffers against 118.0 for the first variant (70.9 / 75.0 in the
// hydrodynamic form, 181.6 / 208.3 with penalty planes), z_forward 80.9 with TMA against 84.5.
#include "ops.cuh"

namespace mhdgb {

OpsBase* make_ops_256() {
  auto* o = new Ops<256>();
  o->add_col<Plan<256, 16, 16, 16>, 16, 3>(kDefaultZinv | kDefaultYinv);
  o->add_col<Plan<256, 16, 16, 16>, 8, 4>();
  o->add_col<Plan<256, 32, 8, 8, 4>, 8, 3>();
  o->add_col<Plan<256, 32, 8, 8, 4>, 16, 2>();
  o->add_col<Plan<256, 32, 8, 8, 4>, 16, 3>();
  o->add_col<Plan<256, 16, 16, 16>, 16, 4>();
  o->add_col<Plan<256, 16, 16, 16>, 16, 2, 3>();
  o->add_col<Plan<256, 16, 16, 16>, 8, 4, 4>();
  o->add_col<Plan<256, 16, 16, 16>, 8, 6, 3>(kDefaultYfwd);
  o->add_col_tma<Plan<256, 16, 16, 16>, 3, 2>();
  o->add_col_tma<Plan<256, 16, 16, 16>, 2, 3>(kDefaultZfwd);
  o->add_x<Plan<256, 32, 8, 8, 4>, 8, 1, 1, 2>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 4, 1, 1, 4>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 4, 3, 1, 3>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 4, 3, 2, 3>();
  o->add_x<Plan<256, 16, 16, 16>, 4, 1, 1, 2>();
  o->add_x<Plan<256, 32, 8, 8, 4>, 2, 1, 1, 8>();
  o->add_x_vp<Plan<256, 32, 8, 8, 4>, 4, 1, 3>();
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
