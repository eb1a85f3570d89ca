// Pass kernels of the 128^3 grid: default configuration first, then autotuner candidates.  FP32 runs on
// the plane passes, the split-precision forms on the column passes.
#include "ops.cuh"

namespace mhdgb {

OpsBase* make_ops_128() {
  auto* o = new Ops<128>();
  using R = Plan<128, 16, 8, 4, 4>;
  using S = Split2<Plan<64, 8, 8, 8>>;
  o->add_plane<Plan<128, 8, 16, 8>, 352, 2>();    // inverse 20.5 us, forward 22.6 us
  o->add_plane<Plan<128, 8, 16, 8>, 256, 2>(0);   // 21.8, 23.4
  o->add_x_tile<Plan<128, 8, 16, 8>, 1, 2, 0, false, true>();  // 30.6 us
  o->add_x_tile<R, 1, 2>();                                    // 30.8
  o->add_x_form<R, 4, 1, 1, 4, true, true>();
  o->add_x_tile<S, 1, 2, 1>();                                 // 39.3 us (three-stage plan 41.1)
  o->add_x_tile<R, 1, 2, 2>();                                 // with walls 49.3 (two halves 53.7, 16 x 8 84)
  o->add_x_vp<R, 4, 1, 3, true>();
  o->add_x_tile<Plan<128, 8, 16, 8>, 1, 3, 0, true, true>();   // hydrodynamics 18.5 us, one at a time 22.8
  o->add_x_tile<R, 1, 2, 0, true>();
  o->add_x_hd<R, 4, 4, 0, true>();
  o->add_x_tile<R, 1, 2, 1, true>();
  o->add_x_tile<R, 1, 2, 2, true>();
  o->add_x_hdvp<R, 4, 3, true>();
  // column passes of the split-precision forms (their x rows work on contiguous rows)
  o->add_col<Plan<128, 8, 16, 8>, 16, 2>();
  o->add_col<Plan<128, 8, 16, 8>, 8, 4>();
  o->add_col<Plan<128, 16, 8, 4, 4>, 8, 3>();
  o->add_col_tma<Plan<128, 8, 16, 8>, 2, 2>();
  o->add_x_tc<SPLIT_F16, 4, 2>();
  o->add_x_tc<SPLIT_BF16, 4, 2>();
  o->set_rows<Plan<128, 16, 8, 4, 4>, 8>();
  return o;
}

}  // namespace mhdgb
