// Spectral epilogue, layout conversion, CFL and diagnostics kernels of the MHD step (sm_103a).
// Included by the library's main translation unit only (the non-template kernels here have one
// definition); the FFT pass kernels are in passes.cuh.
#pragma once
#include "stage_math.cuh"

namespace mhdgb {

// Streaming right-hand side and Runge-Kutta stage update: one thread per pair of neighbouring
// modes of a compact field (16-byte accesses) and field triple (blockIdx.y: u, B), blockIdx.z the
// instance.  Bound by HBM: 33.5 arrays of a field per RK4 launch on average, 105 us at 256^3
// (6.3 TB/s) and 767 us at 512^3.  One thread per mode for all six fields took 131 and 1004 us, bound by
// instruction issue: 76 M warp instructions at 256^3 against 34 M here, most of them the IEEE
// divisions of R/6 and R/3 (now one multiplication by dt/6 in the last stage) and the products' scale
// applied plane by plane.  Triples as separate blocks keep a thread at 8 to 14 loads (80 registers).
// HD: the hydrodynamic form (three fields, five product planes; B is neither read nor written).
constexpr int kStageThreads = 128;
template <int OP, bool GENERAL, bool HD>
__global__ void __launch_bounds__(kStageThreads) stage_kernel(RkArgs a, Geom geo, BatchRef br) {
  const unsigned int i = 2u * (blockIdx.x * kStageThreads + threadIdx.x);
  const int active = *br.count, slot = br.slot(blockIdx.z);
  int x, jy, jz;
  if (i >= field_elems(geo) || !mode_at(geo, i, x, jy, jz)) return;
  if (slot < 0) return;
  const int t = blockIdx.y;
  const long long so = slot * a.stI + 3 * t * a.fs + i;
  const float2* X = a.X + so;
  const float2* prod = a.prod + slot * a.prodI + i;
  const int npl = t ? 3 : 5;
  constexpr bool rd_sol = OP == OP_RK4_MID || OP == OP_RK4_LAST, rd_acc = rd_sol || OP == OP_LS;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 pl[5], pn[3], xv[3], s4[3], q4[3];
#pragma unroll
  for (int q = 0; q < 5; ++q)
    pl[q] = q < npl ? __ldcs(reinterpret_cast<const float4*>(prod + (5 * t + q) * a.fs)) : zero4;
  const RkSlot rs0{a.sol + so, a.acc + so, a.xn + so, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    xv[c] = *reinterpret_cast<const float4*>(X + c * a.fs);
    s4[c] = rd_sol ? *reinterpret_cast<const float4*>(rs0.sol + c * a.fs) : zero4;
    q4[c] = rd_acc ? *reinterpret_cast<const float4*>(rs0.acc + c * a.fs) : zero4;
    if constexpr (GENERAL) {
      const int pp = HD ? (c == 0 ? 6 : c == 1 ? 7 : 5) : 8 + 3 * t + c;
      pn[c] = a.vpen ? __ldcs(reinterpret_cast<const float4*>(prod + pp * a.fs)) : zero4;
    }
  }
  if ((int)blockIdx.z >= active) return;  // after the loads, which do not wait for the count
  const SlotParams sp = a.sp[slot];
  const RkSlot rs{rs0.sol, rs0.acc, rs0.xn, a.hf * sp.dt, sp.dt, sp.dt / 6.f, a.ca, a.cb};
  // the kx = 0 plane diffuses its Hermitian part, H[f][kz'][ky'] (written before X is updated)
  const long long hrow = geo.planar ? geo.k2p : geo.k2, hpl = hrow * geo.k2;
  const float2* H = a.H + slot * a.hI + 3 * t * hpl + jz * hrow + jy;
  float2 nx[3][2], ac[3][2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    auto half = [&](const float4& v) { return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y); };
    const int xh = geo.planar ? x : x + h, yh = geo.planar ? jy + h : jy;
    float2 p[5], pen[3], d[3], R[3];
#pragma unroll
    for (int q = 0; q < 5; ++q) p[q] = half(pl[q]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      d[c] = half(xv[c]);
      if (xh == 0) d[c] = H[c * hpl + (geo.planar ? h : 0)];
      if constexpr (GENERAL) pen[c] = half(pn[c]);
    }
    const float kxv = geo.kscale * (float)xh;
    const float kyv = geo.kscale * (float)signed_of_kept(geo, yh);
    const float kzv = geo.kscale * (float)signed_of_kept(geo, jz);
    triple_rhs<GENERAL, HD>(a, geo, sp, slot, t, xh, yh, jz, kxv, kyv, kzv, d, p, pen, R);
#pragma unroll
    for (int c = 0; c < 3; ++c) nx[c][h] = stage_update(OP, rs, half(xv[c]), R[c], half(s4[c]), half(q4[c]), ac[c][h]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float4 n4 = make_float4(nx[c][0].x, nx[c][0].y, nx[c][1].x, nx[c][1].y);
    if constexpr (OP == OP_RK4_LAST) {
      *reinterpret_cast<float4*>(rs.sol + c * a.fs) = n4;
    } else {
      *reinterpret_cast<float4*>(rs.acc + c * a.fs) = make_float4(ac[c][0].x, ac[c][0].y, ac[c][1].x, ac[c][1].y);
      if constexpr (OP != OP_RHS) *reinterpret_cast<float4*>(rs.xn + c * a.fs) = n4;
    }
  }
}

// On-device getCFL! (src/integrator.jl:158-198 of MHDFlows.jl) after a step of every active
// slot: t += dt of the step just taken; next dt = min(coef * dx / max(|u|max, |B|max), tdiff)
// from the maxima x_fused recorded on the step's last stage; the maxima are cleared for the next
// step.  A slot with no finite positive maximum keeps its dt.
// vmax holds maxima of the unnormalised fields the passes work with (n^3 times the physical
// values); vscale = 1/n^3 converts them.
__global__ void cfl_update_kernel(BatchRef br, SlotParams* sp, unsigned int* vmax, double* t, float coef_dx,
                                  float vscale, int advance) {
  const int n = *br.count;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int s = br.slot(i);
    SlotParams p = sp[s];
    if (advance) t[s] += (double)p.dt;
    const float vm = vscale * fmaxf(__uint_as_float(vmax[2 * s]), __uint_as_float(vmax[2 * s + 1]));
    if (vm > 0.f && isfinite(vm)) {
      float dt = coef_dx / vm;
      if (p.tdiff > 0.f) dt = fminf(dt, p.tdiff);
      p.dt = dt;
      sp[s] = p;
    }
    vmax[2 * s] = 0u;
    vmax[2 * s + 1] = 0u;
  }
}

// one step of every active slot taken: advance the per-slot step counters (random forcing)
__global__ void step_tick_kernel(BatchRef br, long long* steps) {
  const int n = *br.count;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) steps[br.slot(i)] += 1;
}

// ------------------------------------------------------------------------------------------
// Layout conversion between the reference's column-major sol[kx, ky, kz, f] (half spectrum,
// nkr = n/2+1) and the compact retained-band state.
// ------------------------------------------------------------------------------------------
// These kernels take one z-plane of one field per blockIdx.y, so that an element's row needs one
// 32-bit division and no others, and four elements per thread where the accesses are 8 bytes.  With the
// 64-bit divisions of a flat index by four run-time sizes they ran at a third of HBM's rate: push and
// pull of prob.sol 80 + 206 us at 256^3 and 579 + 1570 us at 512^3, now 55 + 100 and 373 + 754 us.
constexpr int kCopyThreads = 256;

// Retained modes of the reference layout -> compact state, in the reference's order (kx fastest), so
// that the reads, which may cross the host link, are contiguous.  blockIdx.y = f k2 + kz'.  Padding
// elements of S are not written here and hold anything: in column order an odd Kx leaves the second
// half of a row's last pair in the padding (256^3: modes 84 and 85 of 85), which stage_kernel updates with
// the rest, and the column pairs transform the padding columns of a tile.  No kernel mixes a column with
// another before the x rows, and those read the kept modes alone.
__global__ void __launch_bounds__(kCopyThreads) gather_state_kernel(const float2* __restrict__ ref, float2* __restrict__ S,
                                                                    Geom geo) {
  const unsigned int kx = geo.kx, total = (unsigned int)geo.k2 * kx;
  const int nkr = geo.n / 2 + 1, f = blockIdx.y / geo.k2, jz = blockIdx.y - f * geo.k2;
  const float2* src = ref + ((long long)f * geo.n + freq_of_kept(geo, jz)) * geo.n * nkr;
  float2* dst = S + f * geo.fs;
#pragma unroll 4
  for (unsigned int i = blockIdx.x * kCopyThreads + threadIdx.x; i < total; i += gridDim.x * kCopyThreads) {
    const int jy = (int)(i / kx), x = (int)(i - (unsigned int)jy * kx);
    dst[mode_off(geo, x, jy, jz)] = src[freq_of_kept(geo, jy) * nkr + x];
  }
}

// Compact state -> reference layout, two elements (one 16-byte store) per thread and step: a plane
// has n nkr elements, an even number, and ref is 16-byte aligned, so every pair is aligned.  The
// output may be mapped host memory, where wide stores use the host link better.  blockIdx.y =
// f n + the plane's frequency index.
__global__ void __launch_bounds__(kCopyThreads) scatter_state_kernel(const float2* __restrict__ S, float2* __restrict__ ref,
                                                                     Geom geo) {
  const unsigned int nkr = geo.n / 2 + 1, pairs = (unsigned int)geo.n * nkr / 2;
  const int f = blockIdx.y / geo.n, jz = kept_of_freq(geo, blockIdx.y - f * geo.n);
  const float2* src = S + f * geo.fs;
  float4* out = reinterpret_cast<float4*>(ref) + (long long)blockIdx.y * pairs;
  for (unsigned int p = blockIdx.x * kCopyThreads + threadIdx.x; p < pairs; p += gridDim.x * kCopyThreads) {
    float2 v[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (jz >= 0) {
      unsigned int fy = 2 * p / nkr, x = 2 * p - fy * nkr;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int jy = kept_of_freq(geo, fy);
        if ((int)x < geo.kx && jy >= 0) v[h] = src[mode_off(geo, x, jy, jz)];
        if (++x == nkr) { x = 0; ++fy; }
      }
    }
    out[p] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
  }
}

// Compact state -> the retained elements of the reference layout (kx < Kx, ky and kz kept),
// 8-byte stores; every other element is zero and the caller fills it.  blockIdx.y = f k2 + kz'.
__global__ void __launch_bounds__(kCopyThreads) scatter_retained_kernel(const float2* __restrict__ S, float2* __restrict__ ref,
                                                                        Geom geo) {
  const unsigned int kx = geo.kx, total = (unsigned int)geo.k2 * kx;
  const int nkr = geo.n / 2 + 1, f = blockIdx.y / geo.k2, jz = blockIdx.y - f * geo.k2;
  float2* dst = ref + ((long long)f * geo.n + freq_of_kept(geo, jz)) * geo.n * nkr;
  const float2* src = S + f * geo.fs;
#pragma unroll 4
  for (unsigned int i = blockIdx.x * kCopyThreads + threadIdx.x; i < total; i += gridDim.x * kCopyThreads) {
    const int jy = (int)(i / kx), x = (int)(i - (unsigned int)jy * kx);
    dst[freq_of_kept(geo, jy) * nkr + x] = src[mode_off(geo, x, jy, jz)];
  }
}

// ------------------------------------------------------------------------------------------
// Diagnostics.
// ------------------------------------------------------------------------------------------
// Per-block partial sums over the compact state (double accumulation, fixed order):
//   [0] sum w|u|^2  [1] sum w|b|^2  [2] sum w Re(u.conj b)  [3] max|k.u|  [4] max|k.b|  [5] non-finite count
// w = 1 on the kx = 0 plane and 2 elsewhere (the half spectrum stands for both +-kx).
constexpr int kDiagSlots = 6;
constexpr int kDiagThreads = 256;
// Blocks per state: one per SM.  A block's reduction of FP64 sums costs as much of the FP64 pipe as half a mode per
// thread, so few threads with many modes each (8 at 128^3) beat many threads with one.
constexpr int kDiagBlocks = 152;

__device__ __forceinline__ void block_reduce_diag(double (&acc)[kDiagSlots], double* out) {
  __shared__ double red[kDiagThreads / 32][kDiagSlots];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int s = 0; s < kDiagSlots; ++s) {
    double x = acc[s];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_down_sync(0xffffffffu, x, o);
      x = (s == 3 || s == 4) ? fmax(x, y) : x + y;
    }
    if (lane == 0) red[wid][s] = x;
  }
  __syncthreads();
  if (threadIdx.x < kDiagSlots) {
    const int s = threadIdx.x;
    double x = red[0][s];
    for (int w = 1; w < kDiagThreads / 32; ++w) x = (s == 3 || s == 4) ? fmax(x, red[w][s]) : x + red[w][s];
    out[s] = x;
  }
}

// One mode into a thread's sums.  The kernels that call this are bound by the FP64 pipe (2 FMA per clock and
// SM): the maxima are taken of the squares and rooted once a thread (the rounded square root is monotone, so
// the maximum is the same to the bit), which left 57 of about 100 FP64 instructions a mode.  Recorded
// diagnostics with kDiagBlocks: 128^3 78 -> 49 us, 256^3 409 -> 315.
struct DiagAcc {
  double v[kDiagSlots] = {0, 0, 0, 0, 0, 0};
  int bad = 0;
  __device__ __forceinline__ void mode(const Geom& geo, const float2 (&u)[3], const float2 (&b)[3], int x, int jy, int jz) {
    const double w = x == 0 ? 1.0 : 2.0;
    const double k[3] = {(double)geo.kscale * x, (double)geo.kscale * signed_of_kept(geo, jy), (double)geo.kscale * signed_of_kept(geo, jz)};
    double2 ku = make_double2(0, 0), kb = make_double2(0, 0);
    double eu = 0, eb = 0, hc = 0;
    bool nf = false;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      nf |= !isfinite(u[c].x) || !isfinite(u[c].y) || !isfinite(b[c].x) || !isfinite(b[c].y);
      eu += (double)u[c].x * u[c].x + (double)u[c].y * u[c].y;
      eb += (double)b[c].x * b[c].x + (double)b[c].y * b[c].y;
      hc += (double)u[c].x * b[c].x + (double)u[c].y * b[c].y;
      ku.x += k[c] * u[c].x; ku.y += k[c] * u[c].y;
      kb.x += k[c] * b[c].x; kb.y += k[c] * b[c].y;
    }
    v[0] += w * eu;
    v[1] += w * eb;
    v[2] += w * hc;
    v[3] = fmax(v[3], ku.x * ku.x + ku.y * ku.y);
    v[4] = fmax(v[4], kb.x * kb.x + kb.y * kb.y);
    bad += nf;
  }
  __device__ __forceinline__ void finish() {
    v[3] = sqrt(v[3]);
    v[4] = sqrt(v[4]);
    v[5] = bad;
  }
};

// Sums of one state, and i k.B as a one-field compact buffer (input of the div B inverse transform).
__global__ void __launch_bounds__(kDiagThreads) diag_partial_kernel(const float2* __restrict__ S, Geom geo, double* partial,
                                                                    float2* __restrict__ divb) {
  const long long plane = field_elems(geo);
  DiagAcc acc;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < plane; i += (long long)gridDim.x * blockDim.x) {
    int x, jy, jz;
    if (!mode_at(geo, i, x, jy, jz)) {
      divb[i] = make_float2(0.f, 0.f);
      continue;
    }
    float2 u[3], b[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      u[c] = S[c * geo.fs + i];
      b[c] = S[(c + 3) * geo.fs + i];
    }
    const float kx = geo.kscale * x, ky = geo.kscale * signed_of_kept(geo, jy), kz = geo.kscale * signed_of_kept(geo, jz);
    divb[i] = make_float2(-(kx * b[0].y + ky * b[1].y + kz * b[2].y), kx * b[0].x + ky * b[1].x + kz * b[2].x);
    acc.mode(geo, u, b, x, jy, jz);
  }
  acc.finish();
  block_reduce_diag(acc.v, partial + (long long)blockIdx.x * kDiagSlots);
}

// Second pass: reduce the block partials in block order (deterministic).
__global__ void __launch_bounds__(kDiagThreads) diag_final_kernel(const double* __restrict__ partial, int nblocks, double* out) {
  double acc[kDiagSlots] = {0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
#pragma unroll
    for (int s = 0; s < kDiagSlots; ++s) {
      const double x = partial[b * kDiagSlots + s];
      acc[s] = (s == 3 || s == 4) ? fmax(acc[s], x) : acc[s] + x;
    }
  }
  block_reduce_diag(acc, out);
  if (threadIdx.x == 0) out[kDiagSlots] = 0.0;  // where max |div B| is gathered next (its bits, maxabs_kernel)
}

// On-device diagnostics history (getCFL! / increment!(diags) without host synchronisation):
// grid (blocks, cap), blockIdx.y = instance; the partial sums of slot s go to
// partial[(s * gridDim.x + block) * kDiagSlots].
__global__ void __launch_bounds__(kDiagThreads) diag_partial_batch_kernel(const float2* __restrict__ pool, long long stI,
                                                                          Geom geo, BatchRef br, double* partial) {
  const int inst = blockIdx.y;
  if (inst >= *br.count) return;
  const int slot = br.slot(inst);
  const float2* S = pool + slot * stI;
  const long long plane = field_elems(geo);
  DiagAcc acc;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < plane; i += (long long)gridDim.x * blockDim.x) {
    int x, jy, jz;
    if (!mode_at(geo, i, x, jy, jz)) continue;
    float2 u[3], b[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      u[c] = S[c * geo.fs + i];
      b[c] = S[(c + 3) * geo.fs + i];
    }
    acc.mode(geo, u, b, x, jy, jz);
  }
  acc.finish();
  block_reduce_diag(acc.v, partial + ((long long)slot * gridDim.x + blockIdx.x) * kDiagSlots);
}

// grid (cap): one block per instance reduces its slot's partials (block order, deterministic)
// into sample *count of the history: hist[(sample * cap + slot) * kHistVals + v] with v =
// E_u, E_B, H_c (times scale = dV / n^3), max|k.u|, max|k.B|, non-finite count, device time
// (dtime[slot], or -1 without the on-device clock).  Samples past `capacity` are counted, not
// stored.  hist_tick_kernel advances the count after every slot has read it.
constexpr int kHistVals = 7;
__global__ void __launch_bounds__(kDiagThreads) diag_record_kernel(const double* __restrict__ partial, int nblocks, BatchRef br,
                                                                   int cap, double* hist, const int* count, int capacity,
                                                                   const double* dtime, double scale) {
  const int inst = blockIdx.x;
  if (inst >= *br.count) return;
  const int slot = br.slot(inst);
  double acc[kDiagSlots] = {0, 0, 0, 0, 0, 0};
  const double* p = partial + (long long)slot * nblocks * kDiagSlots;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
#pragma unroll
    for (int s = 0; s < kDiagSlots; ++s) {
      const double x = p[b * kDiagSlots + s];
      acc[s] = (s == 3 || s == 4) ? fmax(acc[s], x) : acc[s] + x;
    }
  }
  __shared__ double red[kDiagSlots];
  block_reduce_diag(acc, red);
  __syncthreads();
  const int sample = *count;
  if (threadIdx.x == 0 && sample < capacity) {
    double* o = hist + ((long long)sample * cap + slot) * kHistVals;
    o[0] = red[0] * scale;
    o[1] = red[1] * scale;
    o[2] = red[2] * scale;
    o[3] = red[3];
    o[4] = red[4];
    o[5] = red[5];
    o[6] = dtime ? dtime[slot] : -1.0;
  }
}
__global__ void hist_tick_kernel(int* count) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *count += 1;
}

// DivVCorrection! / DivBCorrection! (src/Solver/VPSolver.jl:60-138): u (mask bit 0) and B (bit 1)
// of every active slot lose their gradient part, X -= k (k.X) / k^2 with 1/k^2 = 0 at k = 0.
// grid (ceil(field_elems / blockDim.x), cap): one thread per element of a compact field.
__global__ void div_correct_kernel(float2* __restrict__ pool, Geom geo, long long fs, long long stI, BatchRef br,
                                   int mask) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int inst = blockIdx.y;
  int x, jy, jz;
  if (i >= field_elems(geo) || inst >= *br.count || !mode_at(geo, i, x, jy, jz)) return;
  float2* X = pool + br.slot(inst) * stI + i;
  const float kx = geo.kscale * (float)x;
  const float ky = geo.kscale * (float)signed_of_kept(geo, jy);
  const float kz = geo.kscale * (float)signed_of_kept(geo, jz);
  const float k2 = kx * kx + ky * ky + kz * kz;
  const float ik2 = k2 > 0.f ? 1.0f / k2 : 0.f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!(mask & (1 << h))) continue;
    float2* F = X + 3 * h * fs;
    const float2 a = F[0], b = F[fs], c = F[2 * fs];
    const float pr = (kx * a.x + ky * b.x + kz * c.x) * ik2;
    const float pi = (kx * a.y + ky * b.y + kz * c.y) * ik2;
    F[0] = make_float2(a.x - kx * pr, a.y - kx * pi);
    F[fs] = make_float2(b.x - ky * pr, b.y - ky * pi);
    F[2 * fs] = make_float2(c.x - kz * pr, c.y - kz * pi);
  }
}

// Check of the bounded wait the TMA-fed passes use: one thread waits on an mbarrier that nothing
// arrives on, with a limit of limit_ns, and records in out[0] whether the wait gave up (1) and in
// out[1] the nanoseconds it waited.  The kernel then returns like a pass that timed out.
__global__ void bounded_wait_check_kernel(unsigned long long limit_ns, unsigned long long* out) {
  __shared__ __align__(8) unsigned long long bar;
  if (threadIdx.x != 0) return;
  const unsigned int b = smem_u32(&bar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  const unsigned long long t0 = global_ns();
  const bool done = mbar_wait(b, 0u, limit_ns);
  out[0] = done ? 0ull : 1ull;
  out[1] = global_ns() - t0;
}

// Bytes of a guard band that differ from its fill value, added to *bad.
__global__ void guard_check_kernel(const unsigned char* __restrict__ g, long long n, unsigned char fill,
                                   unsigned long long* bad) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const unsigned int b = (i < n && g[i] != fill) ? 1u : 0u;
  const unsigned int cnt = __popc(__ballot_sync(0xffffffffu, b));
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(bad, (unsigned long long)cnt);
}

// max |x| over a float array via the ordered bit pattern of non-negative floats (NaN wins), into *out, which
// the caller has cleared.  One atomic a block: with one a warp they took longer than the reads up to 128^3.
__global__ void __launch_bounds__(kDiagThreads) maxabs_kernel(const float4* __restrict__ a, long long n4, unsigned int* out) {
  __shared__ unsigned int red[kDiagThreads / 32];
  unsigned int m = 0;
  auto take = [&](float x) { m = max(m, __float_as_uint(fabsf(x))); };
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 q = a[i];
    take(q.x);
    take(q.y);
    take(q.z);
    take(q.w);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = __reduce_max_sync(0xffffffffu, threadIdx.x < kDiagThreads / 32 ? red[threadIdx.x] : 0u);
    if (threadIdx.x == 0) atomicMax(out, m);
  }
}

}  // namespace mhdgb
