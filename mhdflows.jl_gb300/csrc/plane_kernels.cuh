// Plane passes of the small grids (sm_103a): the y and z transforms of one (field, kx) plane in
// one CTA, with the Runge-Kutta stage update folded into the inverse one.
//
// Up to n = kPlaneMax a whole (z, y) plane of one kx mode fits in a CTA's shared memory, so the
// intermediate between the two column transforms never leaves the chip: a right-hand side is three
// launches up to n = 64 (x rows, plane_forward, plane_stage) and four at 96 and 128 (plane_inverse
// and stage_kernel in place of plane_stage), against six with column passes, which at these sizes
// spend most of their 3 to 5 us on launch, drain and the loads of their first tile.  One RK4 step of
// one problem, column passes (with stage_kernel) -> plane passes with the x-row tiles and chained
// graphs of today: 32^3 75 -> 39 us, 64^3 101 -> 63, 96^3 172 -> 153, 128^3 335 -> 290; 24 boxes of
// 32^3 266 -> 148 us per LSRK4 step, 20 of 48^3 536 -> 366, 12 of 64^3 725 -> 466.  Layouts in HBM / L2:
//   state    S[f][kx][kz'][ky']   ky' rows padded to k2p (compact fields of stride fs)
//   planes   R[slot][kx][z][y]    between the plane passes and the x rows (in rowbuf)
//   products P[slot][kx][kz'][ky'] (in colbuf), as the state
// The x rows take tiles of 16 consecutive y of every kx mode and slot by TMA (x_plane_kernel).
#pragma once
#include "stage_math.cuh"

namespace mhdgb {

// Largest grid size with plane passes: at 128 a plane takes 88 KB of shared memory, at 256 it would take 350.
constexpr int kPlaneMax = 128;
// Grid sizes whose stage update is fused with the inverse plane pass (plane_stage_kernel).
__host__ __device__ constexpr bool plane_fused(int n) { return n <= 64; }

// T threads per plane.  Rows (y transforms) take G lanes of a warp each, so they need warp
// barriers only; columns (z transforms) put consecutive ky' on consecutive lanes, free of bank
// conflicts with any row stride, and spread a column's G threads over the block.
// The exchange of a row goes through the row's own words of the plane.  SPLIT (n = 128): real
// parts first, then imaginary parts (row_fft), which takes half the words, so the plane is K2
// columns wide instead of n and more: 88 KB instead of 156 KB, two CTAs per SM instead of one.
// S, the row stride in complex words, is G or 16 - G modulo 16, so that the complex accesses of the
// rows in a half-warp fall on different banks; with SPLIT a row's exchange starts skew() floats
// later in every second half of a warp's rows, so that its 4-byte accesses do, too.
template <class P_, int T_, int MINB_>
struct PlaneCfg {
  using P = P_;
  static_assert(P::STAGES == 2, "plane passes use two-stage plans");
  static constexpr int N = P::N, G = P::G, T = T_, MINB = MINB_;
  static constexpr int KX = kept_kx_of(N), KP = KX, KN = kept_kn_of(N), K2 = KP + KN;
  static constexpr int K2P = (K2 + 3) / 4 * 4;
  static constexpr int RPW = 32 / G;             // rows per warp
  static constexpr int RB = T / 32 * RPW;        // rows per round
  static constexpr int CB = T / G;               // columns per round
  static constexpr int CROUND = (K2 + CB - 1) / CB * CB;  // columns of all rounds (the last may run past K2)
  static constexpr int E1 = P::R1 + 1;           // exchange: floats per stage-1 output label
  static constexpr bool SPLIT = N > 96;
  static constexpr int ROWX = SPLIT ? (P::R0 * E1 + G + 1) / 2 : P::R0 * E1;  // exchange words of a row
  static constexpr int stride() {
    int s = CROUND > ROWX ? CROUND : ROWX;
    if (!SPLIT && s < N) s = N;
    while (s % 16 != G % 16 && s % 16 != 16 - G) ++s;
    return s;
  }
  static constexpr int S = stride();
  static constexpr size_t SMEM = sizeof(float2) * (size_t)N * S;
  static_assert(T % 32 == 0 && T % G == 0 && N % RPW == 0, "whole warps, rows and columns");
  static_assert(K2 % 2 == 0 && S % 2 == 0, "modes go in 16-byte pairs");
  static __device__ __forceinline__ int skew(int rr) { return rr >= RPW / 2 ? G : 0; }
};

// Two-stage transform of one row held as v[V] by G lanes of a warp (fft_run's index conventions),
// exchanging through the row's words of the plane (skewed by the caller when SPLIT).
template <class C, int DIR, bool PK1>
__device__ __forceinline__ void row_fft(float2 (&v)[C::P::V], float2* row, int rr, int g, const float2* __restrict__ tw) {
  using P = typename C::P;
  constexpr int V = P::V, G = P::G, R0 = P::R0, R1 = P::R1;
  dft_groups<R0, DIR, PK1>(v);
  auto twiddle = [&](float2 z, int d, int n1) {
    if (n1 == 0) return z;
    const float2 w = ldtw(tw, n1 * R0 + g + G * d);  // W_N^{n1 k0}
    return cmul_cs<DIR>(z, w.x, w.y);
  };
  if constexpr (C::SPLIT) {
    float* fb = reinterpret_cast<float*>(row) + C::skew(rr);
    float re[V];
#pragma unroll
    for (int d = 0; d < V / R0; ++d)
#pragma unroll
      for (int k0 = 0; k0 < R0; ++k0) fb[k0 * C::E1 + g + G * d] = v[d * R0 + k0].x;
    __syncwarp();
#pragma unroll
    for (int d = 0; d < V / R1; ++d)
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) re[d * R1 + n1] = fb[(g + G * d) * C::E1 + n1];
    __syncwarp();
#pragma unroll
    for (int d = 0; d < V / R0; ++d)
#pragma unroll
      for (int k0 = 0; k0 < R0; ++k0) fb[k0 * C::E1 + g + G * d] = v[d * R0 + k0].y;
    __syncwarp();
#pragma unroll
    for (int d = 0; d < V / R1; ++d)
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1)
        v[d * R1 + n1] = twiddle(make_float2(re[d * R1 + n1], fb[(g + G * d) * C::E1 + n1]), d, n1);
  } else {
#pragma unroll
    for (int d = 0; d < V / R0; ++d)
#pragma unroll
      for (int k0 = 0; k0 < R0; ++k0) row[k0 * C::E1 + g + G * d] = v[d * R0 + k0];
    __syncwarp();
#pragma unroll
    for (int d = 0; d < V / R1; ++d)
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[d * R1 + n1] = twiddle(row[(g + G * d) * C::E1 + n1], d, n1);
  }
  __syncwarp();  // every lane has read the exchange: the row's words are free
  dft_groups<R1, DIR, true>(v);
}

// frequency position of a kept index, and the reverse (-1: alias band), compile-time kept counts
template <class C>
__device__ __forceinline__ int plane_freq(int j) { return j < C::KP ? j : j + C::N - C::K2; }
template <class C>
__device__ __forceinline__ int plane_kept(int r) { return r < C::KP ? r : (r >= C::N - C::KN ? r - (C::N - C::K2) : -1); }
// kept index of position r0 + g (0 <= g < G), r0 compile-time: groups of G positions that lie wholly
// in the kept band take no run-time test
template <class C>
__device__ __forceinline__ int plane_kept_at(int r0, int g) {
  if (r0 + C::G - 1 < C::KP) return r0 + g;
  if (r0 >= C::N - C::KN) return r0 - (C::N - C::K2) + g;
  return plane_kept<C>(r0 + g);
}
template <class C>
__device__ __forceinline__ bool plane_keeps(int r0, int g) {
  return r0 + C::G - 1 < C::KP || r0 >= C::N - C::KN || plane_kept<C>(r0 + g) >= 0;
}
// a group of G consecutive positions from r0 that no lane keeps (compile-time)
template <class C>
__host__ __device__ constexpr bool plane_alias(int r0) { return r0 >= C::KP && r0 + C::G - 1 < C::N - C::KN; }

struct PlaneArgs {
  const float2* src;      // plane_forward: R planes; plane_inverse: compact fields
  float2* dst;            // plane_forward: compact fields; inverse and stage: R planes
  long long sI, dI;       // instance strides
  long long dF;           // compact field stride
  // plane_forward of a right-hand side whose update is a launch of its own (else nullptr): the
  // kx = 0 CTAs of the first hnf planes also write the Hermitian part of the stage state's
  // kx = 0 plane (field stride dF, instance stride hsI) into hout [f][kz'][ky'] (stride hoI)
  const float2* hx;
  float2* hout;
  long long hsI, hoI;
  int hnf;
};

// y then z forward transforms of plane (slot blockIdx.y, kx blockIdx.x) of instance blockIdx.z,
// pruned to the kept modes.
template <class C>
__global__ void __launch_bounds__(C::T, C::MINB) plane_forward_kernel(PlaneArgs a, Geom geo, BatchRef br, const float2* __restrict__ tw) {
  using P = typename C::P;
  constexpr int N = C::N, G = C::G, S = C::S;
  extern __shared__ __align__(16) float2 W[];
  const int active = *br.count, slot = br.slot(blockIdx.z);
  const int x = blockIdx.x, f = blockIdx.y;
  const float2* s = a.src + slot * a.sI + ((long long)f * C::KX + x) * (N * N);
  const int lane = threadIdx.x & 31, g = lane % G;
  float2 u[P::V];
  auto load = [&](int row) {
#pragma unroll
    for (int d = 0; d < P::DI; ++d)
#pragma unroll
      for (int n0 = 0; n0 < P::R0; ++n0) u[d * P::R0 + n0] = s[row * N + g + G * d + P::LI * n0];
  };
  if (!plane_fused(C::N) && slot < 0) return;
  // one round: the loads come before the test of the instance and do not wait for its count
  constexpr bool ONE = C::RB >= N;
  int r0 = (threadIdx.x >> 5) * C::RPW;
  if (ONE && r0 < N) load(r0 + lane / G);
  if ((int)blockIdx.z >= active) return;
  for (; r0 < N; r0 += C::RB) {
    const int row = r0 + lane / G;
    if (!ONE) load(row);
    row_fft<C, -1, true>(u, W + row * S, lane / G, g, tw);
#pragma unroll
    for (int d = 0; d < P::DF; ++d)
#pragma unroll
      for (int e = 0; e < P::RF; ++e) {
        if (plane_alias<C>(G * d + P::LF * e)) continue;
        const int j = plane_kept_at<C>(G * d + P::LF * e, g);
        if (plane_keeps<C>(G * d + P::LF * e, g)) W[row * S + j] = u[d * P::RF + e];
      }
  }
  __syncthreads();
  float2* out = a.dst + slot * a.dI + f * a.dF + (long long)x * (C::K2 * C::K2P);
  const int gc = threadIdx.x / C::CB;
  for (int c = threadIdx.x % C::CB; c < C::CROUND; c += C::CB) {
    float2 v[1][P::V];
#pragma unroll
    for (int d = 0; d < P::DI; ++d)
#pragma unroll
      for (int n0 = 0; n0 < P::R0; ++n0) v[0][d * P::R0 + n0] = W[(gc + G * d + P::LI * n0) * S + c];
    __syncthreads();  // the column is in registers: it becomes the exchange space
    fft_run<Unpadded<P>, -1, 1, 0, S>(v, W, c, gc, tw, BlockSync{});
#pragma unroll
    for (int d = 0; d < P::DF; ++d)
#pragma unroll
      for (int e = 0; e < P::RF; ++e) {
        if (plane_alias<C>(G * d + P::LF * e)) continue;
        const int j = plane_kept_at<C>(G * d + P::LF * e, gc);
        if (c < C::K2 && plane_keeps<C>(G * d + P::LF * e, gc)) out[j * C::K2P + c] = v[0][d * P::RF + e];
      }
  }
  if (a.hx && x == 0 && f < a.hnf) {
    const float2* X = a.hx + slot * a.hsI + f * a.dF;
    float2* H = a.hout + slot * a.hoI + f * (C::K2 * C::K2P);
    for (int m = threadIdx.x; m < C::K2 * C::K2; m += C::T) {
      const int jz = m / C::K2, jy = m % C::K2;
      const int py = kept_of_signed(geo, -signed_of_kept(geo, jy)), pz = kept_of_signed(geo, -signed_of_kept(geo, jz));
      const float2 k = X[jz * C::K2P + jy], q = (py >= 0 && pz >= 0) ? X[pz * C::K2P + py] : make_float2(0.f, 0.f);
      H[jz * C::K2P + jy] = make_float2(0.5f * (k.x + q.x), 0.5f * (k.y - q.y));
    }
  }
}

// z then y inverse transforms of the kept modes in W (kz' rows at their frequency position) into
// the R plane out.
template <class C>
__device__ __forceinline__ void plane_inverse(float2* W, float2* out, const float2* __restrict__ tw) {
  using P = typename C::P;
  constexpr int N = C::N, G = C::G, S = C::S;
  const int gc = threadIdx.x / C::CB;
  for (int c = threadIdx.x % C::CB; c < C::CROUND; c += C::CB) {
    float2 v[1][P::V];
#pragma unroll
    for (int d = 0; d < P::DI; ++d)
#pragma unroll
      for (int n0 = 0; n0 < P::R0; ++n0) {
        const int rmin = G * d + P::LI * n0, r = gc + rmin;
        float2 z = make_float2(0.f, 0.f);
        if (!plane_alias<C>(rmin) && plane_keeps<C>(rmin, gc)) z = W[r * S + c];
        v[0][d * P::R0 + n0] = z;
      }
    __syncthreads();  // the column is in registers: it becomes the exchange space
    fft_run<Unpadded<P>, +1, 1, 0, S, false>(v, W, c, gc, tw, BlockSync{});
    __syncthreads();
#pragma unroll
    for (int d = 0; d < P::DF; ++d)
#pragma unroll
      for (int e = 0; e < P::RF; ++e) W[(gc + G * d + P::LF * e) * S + c] = v[0][d * P::RF + e];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane % G;
  for (int r0 = (threadIdx.x >> 5) * C::RPW; r0 < N; r0 += C::RB) {
    const int row = r0 + lane / G;
    float2 v[P::V];
#pragma unroll
    for (int d = 0; d < P::DI; ++d)
#pragma unroll
      for (int n0 = 0; n0 < P::R0; ++n0) {
        const int rmin = G * d + P::LI * n0;
        float2 z = make_float2(0.f, 0.f);
        if (!plane_alias<C>(rmin)) {
          const int j = plane_kept_at<C>(rmin, g);
          if (plane_keeps<C>(rmin, g)) z = W[row * S + j];
        }
        v[d * P::R0 + n0] = z;
      }
    __syncwarp();  // the row is in registers: it becomes the exchange space
    row_fft<C, +1, false>(v, W + row * S, lane / G, g, tw);
#pragma unroll
    for (int d = 0; d < P::DF; ++d)
#pragma unroll
      for (int e = 0; e < P::RF; ++e) out[row * N + g + G * d + P::LF * e] = v[d * P::RF + e];
  }
}

// Inverse transforms of field blockIdx.y (stride sF, instance stride sI) on the kx plane blockIdx.x
// of instance blockIdx.z into its R plane.
template <class C>
__global__ void __launch_bounds__(C::T, C::MINB) plane_inverse_kernel(PlaneArgs a, BatchRef br, const float2* __restrict__ tw) {
  extern __shared__ __align__(16) float2 W[];
  const int active = *br.count, slot = br.slot(blockIdx.z);
  const int x = blockIdx.x, f = blockIdx.y;
  const float2* X = a.src + slot * a.sI + f * a.dF + (long long)x * (C::K2 * C::K2P);
  if (!plane_fused(C::N) && slot < 0) return;
  for (int m = threadIdx.x; m < C::K2 * C::K2 / 2; m += C::T) {
    const int jz = m / (C::K2 / 2), jy = 2 * (m % (C::K2 / 2));
    *reinterpret_cast<float4*>(W + plane_freq<C>(jz) * C::S + jy) = *reinterpret_cast<const float4*>(X + jz * C::K2P + jy);
  }
  if ((int)blockIdx.z >= active) return;
  __syncthreads();
  plane_inverse<C>(W, a.dst + slot * a.dI + ((long long)f * C::KX + x) * (C::N * C::N), tw);
}

// whether the curl component of induction field f (3, 4, 5) reads product q of Axy Axz Ayz
__device__ __forceinline__ bool plane_reads(int f, int q) { return q != 5 - f; }

// Stage update of field blockIdx.y on the kx plane blockIdx.x of instance blockIdx.z, then (inv)
// the inverse transforms of the updated field: one launch for what stage_kernel and
// plane_inverse_kernel do in two.  Every field's CTA reads all the product planes of its
// right-hand side (five for a velocity component), so this form trades reads that hit L2 for a
// launch: it is used up to n = 64 (plane_fused).  A cluster of the triple's three CTAs, each
// updating a third of the modes and passing the values on through distributed shared memory, read
// every plane once but was slower: 64^3 single step 90 us against 78, 32^3 55 against 47.
// The kx = 0 plane diffuses its Hermitian part (herm_kx0_items): the partner of every mode lies
// in this CTA's own plane, and all reads of X precede all writes.
template <class C, bool GENERAL, bool HD>
__global__ void __launch_bounds__(C::T, C::MINB) plane_stage_kernel(RkArgs a, PlaneArgs pa, Geom geo, BatchRef br, int inv,
                                                           const float2* __restrict__ tw) {
  constexpr int N = C::N, S = C::S, K2 = C::K2, K2P = C::K2P, T = C::T;
  constexpr int PAIRS = K2 * K2 / 2, NP = (PAIRS + T - 1) / T;
  extern __shared__ __align__(16) float2 W[];
  const int active = *br.count, slot = br.slot(blockIdx.z);
  const int x = blockIdx.x, f = blockIdx.y, t = f / 3, op = a.op;
  const long long so = slot * a.stI + f * a.fs + (long long)x * (K2 * K2P);
  const float2* X = a.X + so;
  float4 xv[NP], xd[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int m = threadIdx.x + i * T, jz = m / (K2 / 2), jy = 2 * (m % (K2 / 2));
    if (m < PAIRS) xv[i] = *reinterpret_cast<const float4*>(X + jz * K2P + jy);
    xd[i] = xv[i];
  }
  if ((int)blockIdx.z >= active) return;  // after the first loads, which do not wait for the count
  if (x == 0) {  // X(-k) = 0 when -k lies in the alias band
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int m = threadIdx.x + i * T, jz = m / (K2 / 2), jy = 2 * (m % (K2 / 2));
      if (m < PAIRS) {
        const int pz = kept_of_signed(geo, -signed_of_kept(geo, jz));
        float2 q[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int py = kept_of_signed(geo, -signed_of_kept(geo, jy + h));
          q[h] = (py >= 0 && pz >= 0) ? X[pz * K2P + py] : make_float2(0.f, 0.f);
        }
        xd[i] = make_float4(0.5f * (xv[i].x + q[0].x), 0.5f * (xv[i].y - q[0].y), 0.5f * (xv[i].z + q[1].x),
                            0.5f * (xv[i].w - q[1].y));
      }
    }
    __syncthreads();
  }
  const SlotParams sp = a.sp[slot];
  const RkSlot rs{a.sol + so, a.acc + so, a.xn + so, a.hf * sp.dt, sp.dt, sp.dt / 6.f, a.ca, a.cb};
  const float2* prod = a.prod + slot * a.prodI + (long long)x * (K2 * K2P);
  const float kxv = geo.kscale * (float)x;
  const bool rd_sol = op == OP_RK4_MID || op == OP_RK4_LAST, rd_acc = rd_sol || op == OP_LS;
  const int npl = t ? 3 : 5;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int m = threadIdx.x + i * T, jz = m / (K2 / 2), jy = 2 * (m % (K2 / 2));
    if (m >= PAIRS) continue;
    const int o = jz * K2P + jy;
    float4 pl[5], pn[3], s4 = zero4, q4 = zero4;
#pragma unroll
    for (int q = 0; q < 5; ++q)
      pl[q] = q < npl && (t == 0 || plane_reads(f, q)) ? *reinterpret_cast<const float4*>(prod + (5 * t + q) * a.fs + o) : zero4;
    if constexpr (GENERAL) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int plane = HD ? (q == 0 ? 6 : q == 1 ? 7 : 5) : 8 + 3 * t + q;
        pn[q] = a.vpen ? *reinterpret_cast<const float4*>(prod + plane * a.fs + o) : zero4;
      }
    }
    if (rd_sol) s4 = *reinterpret_cast<const float4*>(rs.sol + o);
    if (rd_acc) q4 = *reinterpret_cast<const float4*>(rs.acc + o);
    float2 nx[2], ac[2];
    const float kzv = geo.kscale * (float)signed_of_kept(geo, jz);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      auto half = [&](const float4& v) { return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y); };
      float2 p[5], pen[3], R[3];
#pragma unroll
      for (int q = 0; q < 5; ++q) p[q] = half(pl[q]);
      if constexpr (GENERAL) {
#pragma unroll
        for (int q = 0; q < 3; ++q) pen[q] = half(pn[q]);
      }
      const float2 d[3] = {half(xd[i]), half(xd[i]), half(xd[i])};  // only this field's component is used
      const float kyv = geo.kscale * (float)signed_of_kept(geo, jy + h);
      triple_rhs<GENERAL, HD>(a, geo, sp, slot, t, x, jy + h, jz, kxv, kyv, kzv, d, p, pen, R);
      const int c = f - 3 * t;
      nx[h] = stage_update(op, rs, half(xv[i]), c == 0 ? R[0] : c == 1 ? R[1] : R[2], half(s4), half(q4), ac[h]);
    }
    const float4 n4 = make_float4(nx[0].x, nx[0].y, nx[1].x, nx[1].y);
    if (op == OP_RK4_LAST) {
      *reinterpret_cast<float4*>(rs.sol + o) = n4;
    } else {
      *reinterpret_cast<float4*>(rs.acc + o) = make_float4(ac[0].x, ac[0].y, ac[1].x, ac[1].y);
      if (op != OP_RHS) *reinterpret_cast<float4*>(rs.xn + o) = n4;
    }
    if (inv) *reinterpret_cast<float4*>(W + plane_freq<C>(jz) * S + jy) = n4;
  }
  if (!inv) return;
  __syncthreads();
  plane_inverse<C>(W, pa.dst + slot * pa.dI + ((long long)f * C::KX + x) * (N * N), tw);
}

// ------------------------------------------------------------------------------------------
// x rows in plane order through tiles of 16 consecutive y (at one z, every kx mode and slot).
// One thread brings a tile in with a TMA copy per slot (128-byte rows, 128-byte swizzle: the
// 16-byte chunk of a row is exclusive-or'ed with the kx mode, so the lanes of a transform, which
// hold consecutive kx, read distinct banks), the rows transform in place in the tile, and the
// products leave with a TMA copy per slot.  Reading and writing the planes directly instead costs
// a 32-byte piece per kx mode and warp at G = 8 (measured: 96^3 x 8 boxes 145 us against 95 us for
// contiguous rows), with tiles every piece is a full 128-byte line.
// ------------------------------------------------------------------------------------------
template <class P, int NBUF, int VPM, bool HDX, bool PAIR>
struct XPlaneCfg {
  static constexpr int N = P::N, G = P::G, ROWS = 16, THREADS = ROWS * G;
  static constexpr int KX = kept_kx_of(N);
  static constexpr int NIN = HDX ? 3 : 6;
  static constexpr int NPAIR = HDX ? (VPM ? 4 : 3) : VPM ? 7 : 4;
  static constexpr int NOUT = (HDX && !VPM) ? 5 : 2 * NPAIR;
  static constexpr int NSLOT = 2 * NPAIR > NIN ? 2 * NPAIR : NIN;
  static constexpr int SLOTB = (KX + 7) / 8 * 1024;    // bytes of a slot: kx rows of 128 bytes, whole swizzle periods
  static constexpr int TILEB = NSLOT * SLOTB;
  static constexpr int TS = XCfg<P, 1, true, PAIR>::TS;
  static constexpr size_t SMEM = 1024 + (size_t)NBUF * TILEB + sizeof(float2) * ROWS * TS + 32;
  static_assert(N % ROWS == 0 && NBUF >= 1 && NBUF <= 2, "whole tiles, one or two buffers");
};

__device__ __forceinline__ void tma_load4(unsigned int dst, const void* map, int c0, int c1, int c2, int c3, unsigned int bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_store4(const void* map, int c0, int c1, int c2, int c3, unsigned int src) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];\n" ::"l"(map), "r"(c0),
               "r"(c1), "r"(c2), "r"(c3), "r"(src)
               : "memory");
}

// PAIR: transforms in pairs as in x_fused_kernel.
template <class P, int NBUF, int MINB, int VPM = 0, bool HDX = false, bool PAIR = false>
__global__ void __launch_bounds__(16 * P::G, MINB)
    x_plane_kernel(const __grid_constant__ CUtensorMap map, int* err, BatchRef br, const float2* __restrict__ tw,
                   const float2* __restrict__ twr, unsigned int* vmax, VpRef vp) {
  using PR = typename Reverse<P>::type;
  using C = XPlaneCfg<P, NBUF, VPM, HDX, PAIR>;
  constexpr int N = P::N, G = P::G, V = P::V, KX = C::KX, TS = C::TS;
  constexpr int NINV = HDX ? 2 : 3;
  extern __shared__ unsigned char xsm[];
  // tiles on 1024-byte boundaries (the swizzle's period)
  unsigned char* tiles = xsm + ((1024u - (smem_u32(xsm) & 1023u)) & 1023u);
  float2* ex = reinterpret_cast<float2*>(tiles + NBUF * C::TILEB);
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(ex + C::ROWS * TS);
  volatile int& abort_flag = *reinterpret_cast<volatile int*>(bars + 2);
  const int yl = threadIdx.x / G, g = threadIdx.x % G;
  float2* sb = ex + yl * TS;
  const RowSync<G> sync{0};
  constexpr int PER = N * (N / C::ROWS);  // tiles of one instance: y blocks fastest, then z
  const int total = *br.count * PER;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int b = 0; b < NBUF; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  // thread 0: tile t into buffer b, once the stores that read the buffer are done with it
  auto issue = [&](int t, int b) {
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    const unsigned int bar = smem_u32(&bars[b]);
    const int inst = t / PER, r = t - inst * PER;
    const int y0 = r % (N / C::ROWS) * C::ROWS, z = r / (N / C::ROWS), slot = br.slot(inst);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((unsigned int)(C::NIN * KX * 128)) : "memory");
#pragma unroll
    for (int f = 0; f < C::NIN; ++f) tma_load4(smem_u32(tiles + b * C::TILEB + f * C::SLOTB), &map, y0, z, f * KX, slot, bar);
  };
  int t = blockIdx.x, issued = 0, it = 0;
  if (NBUF == 2 && threadIdx.x == 0 && t < total) { issue(t, 0); issued = 1; }
  for (; t < total; t += gridDim.x, ++it) {
    const int b = NBUF == 2 ? (it & 1) : 0;
    if (threadIdx.x == 0) {
      const int tn = NBUF == 2 ? t + gridDim.x : t;
      if (tn < total) { issue(tn, NBUF == 2 ? b ^ 1 : 0); ++issued; }
    }
    if (!mbar_wait(smem_u32(&bars[b]), (unsigned int)((it / NBUF) & 1))) {
      atomicExch(err, 1);
      abort_flag = 1;
    }
    if (__syncthreads_or(abort_flag)) break;
    unsigned char* tile = tiles + b * C::TILEB;
    // element (slot f, mode k) of this thread's row
    auto at = [&](int f, int k) {
      return reinterpret_cast<float2*>(tile + f * C::SLOTB + k * 128 + (((yl >> 1) ^ (k & 7)) << 4) + ((yl & 1) << 3));
    };
    float2 v[3][V];
#pragma unroll
    for (int p = 0; p < NINV; ++p) {
      auto f1 = [&](int k) { return *at(2 * p, k); };
      auto f2 = [&](int k) { return *at(2 * p + 1, k); };
      if (HDX && p == 1) load_herm_pair<P, KX, true>(v[p], f1, f2, g);
      else load_herm_pair<P, KX>(v[p], f1, f2, g);
    }
    if constexpr (PAIR) {
      C2 c[V];
#pragma unroll
      for (int i = 0; i < V; ++i) c[i] = C2{make_float2(v[0][i].x, v[1][i].x), make_float2(v[0][i].y, v[1][i].y)};
      row_run_pair<P, +1>(c, reinterpret_cast<float4*>(sb), g, tw, sync);
      sync();
#pragma unroll
      for (int i = 0; i < V; ++i) {
        v[0][i] = make_float2(c[i].re.x, c[i].im.x);
        v[1][i] = make_float2(c[i].re.y, c[i].im.y);
      }
    }
#pragma unroll
    for (int p = PAIR ? 2 : 0; p < NINV; ++p) {
      row_run<P, +1, false>(v[p], sb, g, tw, sync);
      sync();
    }
    if constexpr (HDX) {  // B = 0: the second half of pair 1 is zero up to roundoff, pair 2 unused
#pragma unroll
      for (int i = 0; i < V; ++i) {
        v[1][i].y = 0.f;
        v[2][i] = make_float2(0.f, 0.f);
      }
    }
    const int inst = t / PER, r = t - inst * PER;
    const int y0 = r % (N / C::ROWS) * C::ROWS, z = r / (N / C::ROWS), slot = br.slot(inst);
    if (vmax) x_vmax(v, vmax + 2 * slot);
    float chi[VPM ? V : 1];
    const float* wrow = nullptr;
    if constexpr (VPM > 0) {
      const long long row = (long long)z * N + y0 + yl;
      const float* crow = vp.chi + slot * vp.cs + row * N;
      if constexpr (VPM == 2) wrow = vp.wall + 6 * slot * vp.cs + row * N;
#pragma unroll
      for (int i = 0; i < V; ++i) chi[i] = __ldg(crow + phys_x<P>(g, i));
    }
    // outputs over the row's own elements: its inputs are in registers, other rows' are elsewhere
    auto put_rows = [&](const float2(&w)[V], int p) {
      split_shfl<PR, KX>(w, g, (threadIdx.x & 31) - g, [&](int k, float2 a, float2 c) {
        *at(2 * p, k) = a;
        *at(2 * p + 1, k) = c;
      });
    };
#pragma unroll
    for (int p = 0; p < C::NPAIR; p += PAIR ? 2 : 1) {
      float2 w[2][V];
      x_pair<P, VPM, HDX>(w[0], p, v, chi, wrow, vp.cs, g);
      if (PAIR && p + 1 < C::NPAIR) {
        x_pair<P, VPM, HDX>(w[1], p + 1, v, chi, wrow, vp.cs, g);
        C2 c[V];
#pragma unroll
        for (int i = 0; i < V; ++i) c[i] = C2{make_float2(w[0][i].x, w[1][i].x), make_float2(w[0][i].y, w[1][i].y)};
        row_run_pair<PR, -1>(c, reinterpret_cast<float4*>(sb), g, twr, sync);
#pragma unroll
        for (int i = 0; i < V; ++i) {
          w[0][i] = make_float2(c[i].re.x, c[i].im.x);
          w[1][i] = make_float2(c[i].re.y, c[i].im.y);
        }
        put_rows(w[0], p);
        put_rows(w[1], p + 1);
      } else {
        row_run<PR, -1, true>(w[0], sb, g, twr, sync);
        put_rows(w[0], p);
      }
      sync();  // the next transform's first exchange overwrites sb
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int f = 0; f < C::NOUT; ++f) tma_store4(&map, y0, z, f * KX, slot, smem_u32(tile + f * C::SLOTB));
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (threadIdx.x == 0) {
    // after an abort: let the loads that were issued and not consumed land before exiting
    if (abort_flag)
      for (int k = it; k < issued; ++k) (void)mbar_wait(smem_u32(&bars[k % NBUF]), (unsigned int)((k / NBUF) & 1));
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
}

}  // namespace mhdgb
