// Column pass on pairs of kx columns (sm_103a), TMA in and out.
//
// The column passes of col_pass_kernel are bound by instruction issue and barriers before HBM
// (256^3 z_inverse: 47 warp instructions per 32 values, issue 58 %, DRAM 55 %).  Here a thread
// transforms the same rows of two neighbouring columns as a pair (fft_pair.cuh).  Shared-memory
// accesses are 16 bytes, twiddle loads serve two columns, and tiles leave with one TMA copy (two for
// pruned outputs) in place of a store and its address per value.
#pragma once
#include "passes.cuh"

namespace mhdgb {

__device__ __forceinline__ void tma_store5(const void* map, int c0, int c1, int c2, int c3, int c4, unsigned int src) {
  asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4, %5}], [%6];\n" ::"l"(map),
               "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(src)
               : "memory");
}

// TX columns per tile, TX/2 * G threads.  min / mout: tensor maps of the pass's source and destination
// with their coordinate roles (pruned arrays in boxes of the kept non-negative and of the kept negative
// rows).  NBUF tile buffers; a tile's exchange and its outputs reuse its buffer.  The load of a
// buffer's next tile is issued between the two transform stages of the tile after, when the copy
// that empties the buffer has had half a tile's time (one buffer and five CTAs per SM instead was
// slower: z_inverse 63 us against 57, y_inverse 89 against 80).
template <class P, int TX, int DIR, bool PIN, bool POUT, int MINB, int NBUF>
__global__ void __launch_bounds__(TX / 2 * P::G, MINB)
    col_pair_kernel(ColArgs a, Geom geo, ColWork w, BatchRef br, const float2* __restrict__ tw, const __grid_constant__ CUtensorMap min,
                    TmaCoords ti, const __grid_constant__ CUtensorMap mout, TmaCoords to, int* err) {
  static_assert(P::STAGES == 2 && TX == 16, "two-stage plans, the maps' 16-column boxes");
  static_assert(kept_kx_of(P::N) == kept_kn_of(P::N), "the two boxes of a pruned array have the same height");
  constexpr int G = P::G, V = P::V, N = P::N, R0 = P::R0, R1 = P::R1, LX = TX / 2, NT = LX * G;
  constexpr int KP = kept_kx_of(N), KN = kept_kn_of(N);
  extern __shared__ __align__(128) float2 smem[];
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + NBUF * N * TX);
  volatile int& abort_flag = *reinterpret_cast<volatile int*>(bars + NBUF);
  const int lx = threadIdx.x % LX, g = threadIdx.x / LX;
  const int per = w.tiles_x * w.outer * w.nf;
  const int total = *br.count * per;
  const unsigned int tx_bytes = PIN ? 2u * ti.rb * TX * 8u : (unsigned int)N * TX * 8u;
  if (threadIdx.x == 0) {
    abort_flag = (smem_u32(smem) & 127u) != 0;  // TMA copies want 128-byte aligned tiles
    if (abort_flag) atomicExch(err, 2);
    for (int b = 0; b < NBUF; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (abort_flag) return;
  struct Cur { int tx, o, f, inst; };
  auto decompose = [&](int t) {
    Cur c;
    c.tx = t % w.tiles_x;
    int r = t / w.tiles_x;
    c.f = r % w.nf;
    r /= w.nf;
    c.o = r % w.outer;
    c.inst = r / w.outer;
    return c;
  };
  auto coords = [&](const Cur& c, const TmaCoords& tc, int (&cc)[5]) {
    cc[0] = c.tx * TX;
    cc[tc.odim] = c.o;
    cc[tc.fdim] = c.f;
    cc[tc.idim] = br.slot(c.inst);
  };
  // thread 0 only
  auto issue = [&](int t, int b) {
    const unsigned int bar = smem_u32(&bars[b]);
    float2* buf = smem + b * (N * TX);
    int cc[5] = {0, 0, 0, 0, 0};
    coords(decompose(t), ti, cc);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(tx_bytes) : "memory");
    if (PIN) {
      cc[ti.rowdim] = 0;
      tma_load5(smem_u32(buf), &min, cc[0], cc[1], cc[2], cc[3], cc[4], bar);
      cc[ti.rowdim] = KP;
      tma_load5(smem_u32(buf + (N - KN) * TX), &min, cc[0], cc[1], cc[2], cc[3], cc[4], bar);
    } else {
      for (int r0 = 0; r0 < N; r0 += ti.rb) {
        cc[ti.rowdim] = r0;
        tma_load5(smem_u32(buf + r0 * TX), &min, cc[0], cc[1], cc[2], cc[3], cc[4], bar);
      }
    }
  };
  int issued = 0, it = 0, t = blockIdx.x;
  if (threadIdx.x == 0)
    for (int j = 0; j < NBUF - 1; ++j)
      if (t + j * (int)gridDim.x < total) { issue(t + j * gridDim.x, j); ++issued; }
  for (; t < total; t += gridDim.x, ++it) {
    const int b = it % NBUF;
    if (!mbar_wait(smem_u32(&bars[b]), (unsigned int)((it / NBUF) & 1))) {
      atomicExch(err, 1);
      abort_flag = 1;
    }
    if (__syncthreads_or(abort_flag)) break;
    float4* cur = reinterpret_cast<float4*>(smem + b * (N * TX));  // [row][LX] column pairs
    C2 v[V];
#pragma unroll
    for (int d = 0; d < P::DI; ++d)
#pragma unroll
      for (int n0 = 0; n0 < R0; ++n0) {
        const int rmin = G * d + P::LI * n0, r = g + rmin;
        C2& z = v[d * R0 + n0];
        const bool all = !PIN || rmin + G - 1 < KP || rmin >= N - KN, none = PIN && rmin >= KP && rmin + G - 1 < N - KN;
        if (!none && (all || r < KP || r >= N - KN)) {  // alias rows are zero, their buffer rows stale
          const float4 q = cur[r * LX + lx];
          z = C2{make_float2(q.x, q.z), make_float2(q.y, q.w)};
        } else {
          z = C2{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        }
      }
    __syncthreads();  // the tile is in registers: its buffer becomes the exchange space
    dft2_groups<R0, DIR>(v);
#pragma unroll
    for (int d = 0; d < V / R0; ++d)
#pragma unroll
      for (int k0 = 0; k0 < R0; ++k0) {
        const C2& z = v[d * R0 + k0];
        cur[(k0 * R1 + g + G * d) * LX + lx] = make_float4(z.re.x, z.re.y, z.im.x, z.im.y);
      }
    __syncthreads();
    if (threadIdx.x == 0) {
      const int tn = t + (NBUF - 1) * (int)gridDim.x;
      if (tn < total) {
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the buffer's outputs have left
        issue(tn, (it + NBUF - 1) % NBUF);
        ++issued;
      }
    }
#pragma unroll
    for (int d = 0; d < V / R1; ++d)
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) {
        const float4 q = cur[((g + G * d) * R1 + n1) * LX + lx];
        C2 z{make_float2(q.x, q.y), make_float2(q.z, q.w)};
        if (n1 != 0) {
          const float2 wv = ldtw(tw, n1 * R0 + g + G * d);
          z = c2mul<DIR>(z, wv.x, wv.y);
        }
        v[d * R1 + n1] = z;
      }
    dft2_groups<R1, DIR>(v);
    __syncthreads();  // every exchange read is done: the buffer takes the outputs
#pragma unroll
    for (int d = 0; d < P::DF; ++d)
#pragma unroll
      for (int e = 0; e < P::RF; ++e) {
        const int kmin = G * d + P::LF * e;
        if (POUT && kmin >= KP && kmin + G - 1 < N - KN) continue;  // no lane keeps this group
        const C2& z = v[d * P::RF + e];
        cur[(g + kmin) * LX + lx] = make_float4(z.re.x, z.im.x, z.re.y, z.im.y);
      }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned int src = smem_u32(cur);
      int cc[5] = {0, 0, 0, 0, 0};
      coords(decompose(t), to, cc);
      if (POUT) {
        cc[to.rowdim] = 0;
        tma_store5(&mout, cc[0], cc[1], cc[2], cc[3], cc[4], src);
        cc[to.rowdim] = KP;
        tma_store5(&mout, cc[0], cc[1], cc[2], cc[3], cc[4], src + (N - KN) * TX * 8);
      } else {
        for (int r0 = 0; r0 < N; r0 += to.rb) {
          cc[to.rowdim] = r0;
          tma_store5(&mout, cc[0], cc[1], cc[2], cc[3], cc[4], src + r0 * TX * 8);
        }
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (threadIdx.x == 0) {
    // after an abort: let the loads that were issued and not consumed land before exiting
    if (abort_flag)
      for (int k = it; k < issued; ++k) (void)mbar_wait(smem_u32(&bars[k % NBUF]), (unsigned int)((k / NBUF) & 1));
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  if (a.hx) herm_kx0_items(a.hx, a.hout, geo, a.hfs, a.hsI, a.hoI, br, (long long)blockIdx.x * NT + threadIdx.x,
                           (long long)gridDim.x * NT);
}

}  // namespace mhdgb
