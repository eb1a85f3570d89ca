// Pass kernels of the small grid sizes (16, 32, 48, 64, 96): plane passes and x rows in plane order.
// The first x-row variant of a form is its default; plane variants name the class and capacity they
// are the default of (PlaneVariant::pref), from the times beside them (us per launch, one problem
// and a batch of 24, 20, 12 and 8 boxes of 32, 48, 64 and 96).
#include "ops.cuh"

namespace mhdgb {

OpsBase* make_ops_16() {
  using R = Plan<16, 4, 4, 4>;
  auto* o = new Ops<16>();
  o->add_plane<R, 64, 8>();
  o->add_x_form<R, 1, 1, 1, 16, true, true>();
  o->add_x_vp<R, 1, 1, 16, true>();
  o->add_x_hd<R, 1, 16, 0, true>();
  o->add_x_hdvp<R, 1, 16, true>();
  o->set_rows<R, 32>();
  return o;
}

OpsBase* make_ops_32() {
  using R = Plan<32, 4, 8, 4>;
  auto* o = new Ops<32>();
  o->add_plane<R, 128, 6>();                     // inverse 7.3, 12.9; forward 6.1, 12.0
  o->add_x_tile<R, 1, 8, 0, false, true>();      // 7.9, 16.5
  o->add_x_form<R, 1, 1, 1, 16, true, true>();   // 8.1, 20.5
  o->add_x_vp<R, 1, 1, 16, true>();
  o->add_x_hd<R, 1, 16, 0, true>();
  o->add_x_hdvp<R, 1, 16, true>();
  o->set_rows<R, 32>();
  return o;
}

OpsBase* make_ops_48() {
  using R = Plan<48, 4, 12, 4>;
  auto* o = new Ops<48>();
  o->add_plane<R, 192, 1>(1 | 2);                // inverse 9.2, 39.7; forward 7.7, 22.4
  o->add_plane<R, 128, 6>(4 | 8);                // inverse 10.5, 28.6; forward 8.0, 20.3
  o->add_x_tile<R, 1, 5, 0, false, true>();      // 9.6, 34.7 (one at a time 10.0, 42.8)
  o->add_x_form<R, 1, 1, 1, 8, true, true>();
  o->add_x_tile<R, 1, 4, 1>();
  o->add_x_tile<R, 1, 4, 2>();
  o->add_x_vp<R, 1, 1, 8, true>();
  o->add_x_tile<R, 1, 5, 0, true>();
  o->add_x_hd<R, 1, 8, 0, true>();
  o->add_x_tile<R, 1, 5, 1, true>();
  o->add_x_tile<R, 1, 5, 2, true>();
  o->add_x_hdvp<R, 1, 8, true>();
  o->set_rows<R, 32>();
  return o;
}

OpsBase* make_ops_64() {
  using R = Plan<64, 8, 8, 8>;
  auto* o = new Ops<64>();
  o->add_plane<R, 512, 1>(1);                    // inverse 9.9, 54.1; forward 9.0, 28.7
  o->add_plane<R, 192, 5>(2 | 4 | 8);            // inverse 13.6, 42.2; forward 8.3, 24.4
  o->add_x_tile<R, 2, 3, 0, false, true>();      // 9.7, 33.8 (one at a time 10.2, 38.3)
  o->add_x_form<R, 1, 1, 1, 16, true, true>();
  o->add_x_tile<R, 1, 3, 1>();
  o->add_x_tile<R, 1, 3, 2>();
  o->add_x_vp<R, 1, 1, 12, true>();
  o->add_x_tile<R, 2, 4, 0, true>();
  o->add_x_hd<R, 1, 16, 0, true>();
  o->add_x_tile<R, 1, 3, 1, true>();
  o->add_x_tile<R, 1, 3, 2, true>();
  o->add_x_hdvp<R, 1, 12, true>();
  o->set_rows<R, 16>();
  return o;
}

OpsBase* make_ops_96() {
  using R = Plan<96, 8, 12, 4, 2>;
  auto* o = new Ops<96>();
  o->add_plane<Plan<96, 4, 8, 12>, 256, 2>();    // inverse 14.4, 66; forward 16.2, 68
  o->add_plane<Plan<96, 4, 8, 12>, 384, 2>(0);   // inverse 14.9, 64; forward 16.3, 72
  using S = Split2<Plan<48, 4, 12, 4>>;
  o->add_x_tile<S, 2, 2, 0, false, true>();      // 16.4, 83 (three-stage plan 16.5, 93; one buffer 17.2, 106)
  o->add_x_form<R, 1, 1, 1, 8, true, true>();
  o->add_x_tile<S, 1, 2, 1>();                   // 22.7 (three-stage plan 24.6; two buffers leave one block per SM: 32.9)
  o->add_x_tile<S, 1, 2, 2>();                   // with walls 26.7 (27.5)
  o->add_x_vp<R, 1, 1, 8, true>();
  o->add_x_tile<S, 2, 2, 0, true, true>();       // hydrodynamics 13.2 (three-stage plan 14.4)
  o->add_x_hd<R, 1, 8, 0, true>();
  o->add_x_tile<R, 1, 2, 1, true>();
  o->add_x_tile<R, 1, 2, 2, true>();
  o->add_x_hdvp<R, 1, 8, true>();
  o->set_rows<R, 16>();
  return o;
}

}  // namespace mhdgb
