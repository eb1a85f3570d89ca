// Pairs of transforms in paired FP32 instructions (sm_103a).
//
// Two transforms of the same length run together, held by component (re of both, im of both): every
// paired instruction then works on two values without exchanging components, a twiddle costs two
// instructions per value instead of four, a rotation by i none, and twiddle loads and shared-memory
// accesses (16 bytes) serve both.
#pragma once
#include "fft_core.cuh"

namespace mhdgb {

// One complex value of each of two transforms.
struct C2 {
  float2 re, im;
};
__device__ __forceinline__ C2 c2add(const C2& a, const C2& b) { return C2{padd(a.re, b.re), padd(a.im, b.im)}; }
__device__ __forceinline__ C2 c2sub(const C2& a, const C2& b) { return C2{psub(a.re, b.re), psub(a.im, b.im)}; }
// a + DIR i b and a - DIR i b
template <int DIR>
__device__ __forceinline__ C2 c2add_i(const C2& a, const C2& b) {
  return DIR > 0 ? C2{psub(a.re, b.im), padd(a.im, b.re)} : C2{padd(a.re, b.im), psub(a.im, b.re)};
}
template <int DIR>
__device__ __forceinline__ C2 c2sub_i(const C2& a, const C2& b) {
  return c2add_i<-DIR>(a, b);
}
// a * (c + DIR i s)
template <int DIR>
__device__ __forceinline__ C2 c2mul(const C2& a, float c, float s) {
  const float ds = DIR * s;
  const float2 cc = make_float2(c, c), ss = make_float2(ds, ds), ns = make_float2(-ds, -ds);
  return C2{__ffma2_rn(a.re, cc, __fmul2_rn(a.im, ns)), __ffma2_rn(a.re, ss, __fmul2_rn(a.im, cc))};
}

// In-register DFTs on pairs, x[O + S i], natural order (the factorisation of Dft).
template <int R, int DIR>
struct Dft2;
template <int DIR>
struct Dft2<2, DIR> {
  template <int S, int O, int A>
  __device__ __forceinline__ static void run(C2 (&x)[A]) {
    const C2 a = x[O], b = x[O + S];
    x[O] = c2add(a, b);
    x[O + S] = c2sub(a, b);
  }
};
template <int DIR>
struct Dft2<3, DIR> {
  template <int S, int O, int A>
  __device__ __forceinline__ static void run(C2 (&x)[A]) {
    constexpr float h = 0.86602540378443864676f;  // sqrt(3)/2
    const C2 t1 = c2add(x[O + S], x[O + 2 * S]), d = c2sub(x[O + S], x[O + 2 * S]);
    const float2 mh = make_float2(-0.5f, -0.5f), p = make_float2(DIR * h, DIR * h), m = make_float2(-DIR * h, -DIR * h);
    const C2 t2{paxpy(t1.re, mh, x[O].re), paxpy(t1.im, mh, x[O].im)};
    x[O] = c2add(x[O], t1);
    x[O + S] = C2{paxpy(d.im, m, t2.re), paxpy(d.re, p, t2.im)};  // t2 +- DIR i h (x1 - x2)
    x[O + 2 * S] = C2{paxpy(d.im, p, t2.re), paxpy(d.re, m, t2.im)};
  }
};
template <int DIR>
struct Dft2<4, DIR> {
  template <int S, int O, int A>
  __device__ __forceinline__ static void run(C2 (&x)[A]) {
    const C2 a = c2add(x[O], x[O + 2 * S]), b = c2sub(x[O], x[O + 2 * S]);
    const C2 c = c2add(x[O + S], x[O + 3 * S]), e = c2sub(x[O + S], x[O + 3 * S]);
    x[O] = c2add(a, c);
    x[O + 2 * S] = c2sub(a, c);
    x[O + S] = c2add_i<DIR>(b, e);
    x[O + 3 * S] = c2sub_i<DIR>(b, e);
  }
};
template <int R, int DIR>
struct Dft2 {
  static constexpr int P = FirstFactor<R>::value;
  static constexpr int Q = R / P;
  static_assert(P * Q == R && P > 1 && Q > 1, "unsupported radix");
  template <int S, int O, int A>
  __device__ __forceinline__ static void run(C2 (&x)[A]) {
    constexpr TwTab<R> tw{};
#pragma unroll
    for (int b = 0; b < Q; ++b) {
      C2 t[P];
#pragma unroll
      for (int a = 0; a < P; ++a) t[a] = x[O + S * (Q * a + b)];
      Dft2<P, DIR>::template run<1, 0>(t);
#pragma unroll
      for (int ka = 0; ka < P; ++ka) {
        const int e = (b * ka) % R;
        if (e != 0) {
          if (4 * e == R || 4 * e == 3 * R) {  // +-i: an exchange and one sign
            const float2 m = make_float2(-1.f, -1.f);
            const bool plus = (4 * e == R) == (DIR > 0);
            t[ka] = plus ? C2{__fmul2_rn(t[ka].im, m), t[ka].re} : C2{t[ka].im, __fmul2_rn(t[ka].re, m)};
          } else {
            t[ka] = c2mul<DIR>(t[ka], tw.c[e], tw.s[e]);
          }
        }
        x[O + S * (Q * ka + b)] = t[ka];
      }
    }
    C2 out[R];
#pragma unroll
    for (int ka = 0; ka < P; ++ka) {
      C2 t[Q];
#pragma unroll
      for (int b = 0; b < Q; ++b) t[b] = x[O + S * (Q * ka + b)];
      Dft2<Q, DIR>::template run<1, 0>(t);
#pragma unroll
      for (int kb = 0; kb < Q; ++kb) out[ka + P * kb] = t[kb];
    }
#pragma unroll
    for (int k = 0; k < R; ++k) x[O + S * k] = out[k];
  }
};
template <int R, int DIR, int A>
__device__ __forceinline__ void dft2_groups(C2 (&x)[A]) {
#pragma unroll
  for (int d = 0; d < A / R; ++d) {
    C2 t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) t[r] = x[d * R + r];
    Dft2<R, DIR>::template run<1, 0>(t);
#pragma unroll
    for (int r = 0; r < R; ++r) x[d * R + r] = t[r];
  }
}


// Exchange strides of a plan for 16-byte words (row layouts): the eight lanes of a quarter-warp hold
// consecutive labels, so a stride that spreads them over the eight 16-byte bank groups is odd where
// they differ in k0 alone (R0 >= 8), 2 (mod 8) where they are four k0 of two n2 (R0 = 4); the second
// exchange's is 4 (mod 8) for R0 = 4 and free otherwise.
template <class P>
struct PairRow {
  static constexpr int pad(int s, int r, int m) {
    while (s % m != r) ++s;
    return s;
  }
  static constexpr int E1S = P::R0 == 4 ? pad(P::R1 * P::R2, 2, 8) : pad(P::R1 * P::R2, 1, 2);
  static constexpr int E2S = P::R0 == 4 ? pad(P::R0 * P::R1, 4, 8) : P::R0 * P::R1;
  static constexpr int S1 = P::R0 * E1S, S2 = P::R2 > 1 ? P::R2 * E2S : 0;
  static constexpr int WORDS = S1 > S2 ? S1 : S2;
};

template <class H>
struct PairRow<Split2<H>> {
  static constexpr int WORDS = 2 * SplitCfg<Split2<H>>::OFFP;
};
// exchange strides of a half of a Split2
template <class H>
struct PairRow<SplitHalf<H>> {
  static constexpr int E1S = SplitHalf<H>::E1S, E2S = 0, WORDS = SplitHalf<H>::WORDS;
};

// fft_run of two transforms held as v[V], exchanging through buf (PairRow<P>::WORDS 16-byte words).
template <class P, int DIR, class SyncF>
__device__ __forceinline__ void fft_run_pair(C2 (&v)[P::V], float4* buf, int g, const float2* __restrict__ tw, SyncF SYNC) {
  using X = PairRow<P>;
  constexpr int V = P::V, G = P::G, R0 = P::R0, R1 = P::R1, R2 = P::R2;
  auto put = [&](int i, const C2& z) { buf[i] = make_float4(z.re.x, z.re.y, z.im.x, z.im.y); };
  auto get = [&](int i) {
    const float4 q = buf[i];
    return C2{make_float2(q.x, q.y), make_float2(q.z, q.w)};
  };
  dft2_groups<R0, DIR>(v);
#pragma unroll
  for (int d = 0; d < V / R0; ++d)
#pragma unroll
    for (int k0 = 0; k0 < R0; ++k0) put(k0 * X::E1S + g + G * d, v[d * R0 + k0]);
  SYNC();
#pragma unroll
  for (int d = 0; d < V / R1; ++d) {
    const int l2 = g + G * d, k0 = l2 % R0, n2 = l2 / R0;
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      C2 z = get(k0 * X::E1S + n1 * R2 + n2);
      if (n1 != 0) {
        const float2 w = ldtw(tw, n1 * R0 + k0);  // W_{R0R1}^{n1 k0}
        z = c2mul<DIR>(z, w.x, w.y);
      }
      v[d * R1 + n1] = z;
    }
  }
  dft2_groups<R1, DIR>(v);
  if constexpr (P::STAGES == 3) {
    SYNC();
#pragma unroll
    for (int d = 0; d < V / R1; ++d) {
      const int l2 = g + G * d, k0 = l2 % R0, n2 = l2 / R0;
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        const float2 w = ldtw(tw, PlanTw<P>::T2 + k1 * (R0 * R2) + l2);  // W_N^{n2 (k0 + R0 k1)}
        put(n2 * X::E2S + k0 + R0 * k1, c2mul<DIR>(v[d * R1 + k1], w.x, w.y));
      }
    }
    SYNC();
#pragma unroll
    for (int d = 0; d < V / R2; ++d)
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) v[d * R2 + n2] = get(n2 * X::E2S + g + G * d);
    dft2_groups<R2, DIR>(v);
  }
}

// row_run of two transforms.
template <class P, int DIR, class SyncF>
__device__ __forceinline__ void row_run_pair(C2 (&v)[P::V], float4* buf, int g, const float2* __restrict__ tw, SyncF SYNC) {
  if constexpr (IsSplit<P>::value) {
    using H = SplitHalf<typename P::H>;
    const int h = g & 1;
    const float s = h ? -1.f : 1.f;
    const float2 ss = make_float2(s, s);
    const float2* jt = tw + PlanTw<P>::JOIN + (DIR > 0 ? 0 : PlanTw<P>::VG) + g;
    auto other = [](float2 a) { return make_float2(__shfl_xor_sync(0xffffffffu, a.x, 1), __shfl_xor_sync(0xffffffffu, a.y, 1)); };
    if constexpr (DIR > 0) {
      fft_run_pair<H, DIR>(v, buf + h * SplitCfg<P>::OFFP, g >> 1, tw, SYNC);
#pragma unroll
      for (int i = 0; i < P::V; ++i) {
        const float2 w = __ldg(jt + i * P::G);
        const C2 t = c2mul<DIR>(v[i], w.x, w.y);
        v[i] = C2{paxpy(t.re, ss, other(t.re)), paxpy(t.im, ss, other(t.im))};
      }
    } else {
#pragma unroll
      for (int i = 0; i < P::V; ++i) {
        const float2 w = __ldg(jt + i * P::G);
        v[i] = c2mul<DIR>(C2{paxpy(v[i].re, ss, other(v[i].re)), paxpy(v[i].im, ss, other(v[i].im))}, w.x, w.y);
      }
      fft_run_pair<H, DIR>(v, buf + h * SplitCfg<P>::OFFP, g >> 1, tw, SYNC);
    }
  } else {
    fft_run_pair<P, DIR>(v, buf, g, tw, SYNC);
  }
}

}  // namespace mhdgb
