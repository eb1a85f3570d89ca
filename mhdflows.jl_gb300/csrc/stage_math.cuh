// Spectral right-hand side of one retained mode and the Runge-Kutta stage update (sm_103a):
// templates and inline functions only (the spectral epilogue kernel is in step_kernels.cuh).
#pragma once
#include "passes.cuh"

namespace mhdgb {

// Runge-Kutta stage operations of the epilogue.
enum StageOp : int {
  OP_RHS = 0,       // out <- R
  OP_RK4_FIRST = 1, // acc <- R ; xn <- sol + h R              (X = sol)
  OP_RK4_MID = 2,   // acc <- acc + 2 R ; xn <- sol + h R
  OP_RK4_LAST = 3,  // sol <- sol + dt/6 (acc + R)
  OP_LS_FIRST = 4,  // du <- dt R ; u <- u + b du              (X = u)
  OP_LS = 5,        // du <- a du + dt R ; u <- u + b du
};

// ------------------------------------------------------------------------------------------
// Streaming right-hand side + Runge-Kutta stage update over the compact retained band.
// prod: compact spectra of the 8 products [p][kz'][ky'][kx] (Dxz Dyz Txy Txz Tyz Axy Axz Ayz).
// Momentum: R_u = i (V - k (k.V)/k^2) - nu k^2 X_u with V = (kx Dxz + ky Txy + kz Txz,
// kx Txy + ky Dyz + kz Tyz, kx Txz + ky Tyz) (the stress tensor minus Tzz*I, whose gradient the
// projection removes).  Induction: R_b = i k x E - eta k^2 X_b with E = (Ayz, -Axz, Axy) = u x B.
// ------------------------------------------------------------------------------------------
struct RkArgs {
  const float2* prod;   // 8 compact product planes, then 6 penalty planes with VP (slot stride prodI)
  const float2* X;      // stage state (6 fields, slot stride stI)
  const float2* H;      // Hermitian part of X on the kx = 0 plane, [f][kz'][ky'] (slot stride hI)
  float2* sol;          // RK4 step-start state
  float2* acc;          // RK4 accumulator / LSRK4 du / OP_RHS output
  float2* xn;           // RK4 next stage state / LSRK4 u
  const SlotParams* sp; // per-slot nu, eta, dt
  long long fs;         // compact field stride (complex elements)
  long long stI, prodI, hI;
  float hf;             // RK4 stage fraction of dt (1/2 or 1)
  float ca, cb;         // LSRK4 coefficients of the stage
  float pscale;         // 1/n^6: the column and row passes are unnormalised in both directions
  int op;
  const long long* step; // per-slot step counters (random forcing: call = 8 * step + stage)
  int stage;             // right-hand-side evaluation within the step (7: outside a step)
  float vscale;          // 1/n^3: the penalty planes are n^3 times the reference's rfft
  int vpen, forced;      // penalty planes present, forcing on for some slot (read by the GENERAL forms)
};

// ------------------------------------------------------------------------------------------
// A99 random solenoidal forcing (src/pgen/A99ForceDriving_GPU.jl:76-130 of MHDFlows.jl), with
// a counter-based generator in place of the device rand(): uniform numbers from the SplitMix64
// finaliser of (seed, call, mode index in the reference's (nkr, n, n) layout, draw).
// ------------------------------------------------------------------------------------------
__host__ __device__ inline unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float a99_uniform(unsigned long long key, unsigned long long index, int draw) {
  const unsigned long long z = mix64(key ^ (index * 4ull + (unsigned long long)draw));
  return (float)(z >> 40) * (1.0f / 16777216.0f);
}
// forcing of the three velocity components at wavenumber (kx, ky, kz)
// A mode whose Gaussian underflows to zero (at sigma = 1 every mode more than 10.2 from the peak: all but
// 1 % of the band at 128^3) gets exactly zero, whatever is drawn: it skips the draws and the functions
// of them (RK4 stage at 128^3 23.3 -> 20.3 us, at 256^3 135 -> 113.5; unforced 15.4 and 104).
__device__ __forceinline__ void a99_force(const SlotParams& sp, unsigned long long key, unsigned long long index,
                                          float kx, float ky, float kz, float2 (&F)[3]) {
  constexpr float kPi = 3.14159265358979f;
  const float k = sqrtf(kx * kx + ky * ky + kz * kz);
  const float dk = k - sp.fkf;
  const float gauss = expf(-dk * dk / sp.fs2);
  if (gauss == 0.f && isfinite(sp.fA) && sp.fb != 0.f) {  // fb = 0 and an infinite fA give NaN at every mode
    F[0] = F[1] = F[2] = make_float2(0.f, 0.f);
    return;
  }
  const float kp = sqrtf(kx * kx + kz * kz);
  const float kinv = k > 0.f ? 1.f / k : 0.f;
  const float pinv = kp > 0.f ? 1.f / kp : 0.f;
  const float Fk = sp.fA * sqrtf(gauss / 2.f / kPi) * kinv;
  const float e1x = kz * pinv, e1z = -kx * pinv;
  const float e2x = kx * ky * pinv * kinv, e2y = -kp * kinv, e2z = kz * ky * pinv * kinv;
  const float th1 = a99_uniform(key, index, 0) * 2.f * kPi;
  const float phi = a99_uniform(key, index, 1) * kPi;
  const float th2 = a99_uniform(key, index, 2) * 2.f * kPi;
  float gi = -tanhf(sp.fb * (phi - kPi / 2)) / tanhf(sp.fb * kPi / 2);
  if (fabsf(gi) >= 1.f) gi = copysignf(1.f, gi);
  const float gj = sqrtf(1.f - gi * gi);
  float s1, c1, s2, c2;
  sincosf(th1, &s1, &c1);
  sincosf(th2, &s2, &c2);
  const float amp = sp.fA * Fk;
  const float a1 = amp * gi, a2 = amp * gj;
  F[0] = make_float2(a1 * e1x * c1 + a2 * e2x * c2, a1 * e1x * s1 + a2 * e2x * s2);
  F[1] = make_float2(a2 * e2y * c2, a2 * e2y * s2);
  F[2] = make_float2(a1 * e1z * c1 + a2 * e2z * c2, a1 * e1z * s1 + a2 * e2z * s2);
}

struct RkSlot {
  float2* sol;
  float2* acc;
  float2* xn;
  float h, dt, dt6, ca, cb;  // dt6 = dt / 6
};

// The right-hand side of one retained mode, a triple (u or B) at a time:
// V = (kx Dxz + ky Txy + kz Txz, kx Txy + ky Dyz + kz Tyz, kx Txz + ky Tyz) and
// W = k x E with E = (Ayz, -Axz, Axy): Wx = ky Axy + kz Axz, Wy = kz Ayz - kx Axy,
// Wz = -(kx Axz + ky Ayz).  The nonlinear terms are i (V - k (k.V)/k^2) and i W.
// Volume penalisation (VP_UᵢUpdate! / VP_BᵢUpdate!, src/Solver/VPSolver.jl:20-58):
// N_a += -(δ_aj - k_a k_j / k^2) F_j with F = rfft(chi / eta (u - U0)) (and chi / eta (B - B0)),
// eta = 13 dt / 7, 1/k^2 = 0 at k = 0.  MHD: the six penalty planes are 8..13 (u x, u y, u z, B x,
// B y, B z), n^3 times the reference's rfft; the hydrodynamic form keeps u in the spare product
// slots 6, 7, 5 (x, y, z) at the products' scale, n^6.
// Forcing (addforcing!): N[u] += F, then the kx = 0 plane keeps its real part.
//
// Right-hand side of field triple t (0: u, 1: B) at one retained mode from its product
// planes (p[0..5) = Dxz Dyz Txy Txz Tyz, or p[0..3) = Axy Axz Ayz), with the formulas above.  GENERAL: penalty planes (a.vpen) and forcing (a.forced).
template <bool GENERAL, bool HD>
__device__ __forceinline__ void triple_rhs(const RkArgs& a, const Geom& geo, const SlotParams& sp, int slot, int t, int x, int jy,
                                           int jz, float kxv, float kyv, float kzv, const float2 (&xd)[3], const float2 (&p)[5],
                                           const float2 (&pen)[3], float2 (&R)[3]) {
  // the products' scale goes with the wavenumbers of the sums (three factors per mode)
  const float sx = a.pscale * kxv, sy = a.pscale * kyv, sz = a.pscale * kzv;
  const float k2 = kxv * kxv + kyv * kyv + kzv * kzv;
  const float ik2 = k2 > 0.f ? 1.0f / k2 : 0.f;
  const float ks[3] = {kxv, kyv, kzv};
  float2 nl[3];
  if (t == 0) {
    const float2 dxz = p[0], dyz = p[1], txy = p[2], txz = p[3], tyz = p[4];
    const float2 V[3] = {make_float2(sx * dxz.x + sy * txy.x + sz * txz.x, sx * dxz.y + sy * txy.y + sz * txz.y),
                         make_float2(sx * txy.x + sy * dyz.x + sz * tyz.x, sx * txy.y + sy * dyz.y + sz * tyz.y),
                         make_float2(sx * txz.x + sy * tyz.x, sx * txz.y + sy * tyz.y)};
    const float kvx = (kxv * V[0].x + kyv * V[1].x + kzv * V[2].x) * ik2;
    const float kvy = (kxv * V[0].y + kyv * V[1].y + kzv * V[2].y) * ik2;
#pragma unroll
    for (int c = 0; c < 3; ++c) nl[c] = make_float2(-(V[c].y - ks[c] * kvy), V[c].x - ks[c] * kvx);
  } else {
    const float2 axy = p[0], axz = p[1], ayz = p[2];
    const float2 Wc[3] = {make_float2(sy * axy.x + sz * axz.x, sy * axy.y + sz * axz.y),
                          make_float2(sz * ayz.x - sx * axy.x, sz * ayz.y - sx * axy.y),
                          make_float2(-(sx * axz.x + sy * ayz.x), -(sx * axz.y + sy * ayz.y))};
#pragma unroll
    for (int c = 0; c < 3; ++c) nl[c] = make_float2(-Wc[c].y, Wc[c].x);
  }
  const float dk = -(t == 0 ? sp.nu : sp.eta) * k2;
#pragma unroll
  for (int c = 0; c < 3; ++c) R[c] = make_float2(nl[c].x + dk * xd[c].x, nl[c].y + dk * xd[c].y);
  if constexpr (GENERAL) {
    if (a.vpen) {  // N_a += -(delta_aj - k_a k_j / k^2) F_j of this triple
      const float sc = -(HD ? a.pscale : a.vscale) * 7.f / (13.f * sp.dt);
      const float2 f[3] = {cscale(pen[0], sc), cscale(pen[1], sc), cscale(pen[2], sc)};
      const float px = (kxv * f[0].x + kyv * f[1].x + kzv * f[2].x) * ik2;
      const float py = (kxv * f[0].y + kyv * f[1].y + kzv * f[2].y) * ik2;
#pragma unroll
      for (int c = 0; c < 3; ++c) R[c] = make_float2(R[c].x + f[c].x - ks[c] * px, R[c].y + f[c].y - ks[c] * py);
    }
    if (!HD && a.forced && t == 0 && sp.fA != 0.f) {
      const unsigned long long call = 8ull * (unsigned long long)a.step[slot] + (unsigned long long)a.stage;
      const unsigned long long key = mix64(sp.fseed ^ mix64(call));
      const int nkr = geo.n / 2 + 1;
      const unsigned long long index =
          (unsigned long long)x + (unsigned long long)nkr * ((unsigned long long)freq_of_kept(geo, jy) +
                                                              (unsigned long long)geo.n * freq_of_kept(geo, jz));
      float2 F[3];
      a99_force(sp, key, index, kxv, kyv, kzv, F);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        R[c] = make_float2(R[c].x + F[c].x, R[c].y + F[c].y);
        if (x == 0) R[c].y = 0.f;
      }
    }
  }
}

// Stage update of one value (RK4 and LSRK4 as in StageOp); returns the next stage state.
__device__ __forceinline__ float2 stage_update(int op, const RkSlot& a, float2 x, float2 R, float2 s, float2 q, float2& acc) {
  switch (op) {
    case OP_RK4_FIRST:
      acc = R;
      return make_float2(fmaf(a.h, R.x, x.x), fmaf(a.h, R.y, x.y));
    case OP_RK4_MID:  // 2 R is exact: one rounding
      acc = make_float2(fmaf(2.f, R.x, q.x), fmaf(2.f, R.y, q.y));
      return make_float2(fmaf(a.h, R.x, s.x), fmaf(a.h, R.y, s.y));
    case OP_RK4_LAST:
      return make_float2(fmaf(a.dt6, q.x + R.x, s.x), fmaf(a.dt6, q.y + R.y, s.y));
    case OP_LS_FIRST:
      acc = make_float2(a.dt * R.x, a.dt * R.y);
      return make_float2(x.x + a.cb * acc.x, x.y + a.cb * acc.y);
    case OP_LS:
      acc = make_float2(a.ca * q.x + a.dt * R.x, a.ca * q.y + a.dt * R.y);
      return make_float2(x.x + a.cb * acc.x, x.y + a.cb * acc.y);
    default:  // OP_RHS
      acc = R;
      return x;
  }
}

}  // namespace mhdgb
