// sqg_fft.cuh -- complex helpers and the block-level FFT used by every pass.
//
// The FFT is a Stockham auto-sort transform executed by a group of G = N/8
// threads.  Thread j of the group holds the eight values x[j + m*G],
// m = 0..7, in registers ("strided layout") before and after the transform,
// so a pass can read its input straight from coalesced global loads and
// write its output with coalesced stores.  Between radix passes the data is
// exchanged through a shared-memory buffer of N complex values owned by the
// group.  Radix-8 passes; when log2(N) is not a multiple of three the first
// pass has radix 2 or 4 (each thread then runs 4 or 2 butterflies).
// Twiddles come from a table tw[k] = exp(-2 pi i k / N) computed on the host
// in float64 from cos/sin (rounded to float for the float path).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sqg {

template <typename T> struct Cplx;
template <> struct Cplx<float> { using type = float2; };
template <> struct Cplx<double> { using type = double2; };

// Slots of one exchange buffer of an n-element radix-R transform: the padding
// of every exchange (struct Xchg) fits in n + n / R.
template <int R> __host__ __device__ constexpr int spad_size(int n) { return n + n / R; }

template <typename C> __device__ __forceinline__ C mkc(double x, double y) {
  C r; r.x = x; r.y = y; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
// a * conj(b) when CONJ, else a * b
template <bool CONJ, typename C> __device__ __forceinline__ C cmul_tw(C a, C b) {
  C r;
  if (CONJ) { r.x = a.x * b.x + a.y * b.y; r.y = a.y * b.x - a.x * b.y; }
  else      { r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; }
  return r;
}
template <typename C> __device__ __forceinline__ C cconj(C a) { a.y = -a.y; return a; }
template <typename C, typename S> __device__ __forceinline__ C cscale(C a, S s) { a.x *= s; a.y *= s; return a; }
// multiply by DIR * i   (DIR = +1 inverse sign, -1 forward sign)
template <int DIR, typename C> __device__ __forceinline__ C mul_i(C a) {
  C r;
  if (DIR > 0) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; }
  return r;
}

// Single precision: the same operations on packed pairs (sm_100's two-lane
// FP32 add, multiply and fused multiply-add issue one instruction for both
// components; each lane rounds as the scalar operation does).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
// a * b = a.x (b.x, b.y) + a.y (-b.y, b.x)
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return __ffma2_rn(make_float2(a.y, a.y), make_float2(-b.y, b.x), __fmul2_rn(make_float2(a.x, a.x), b));
}
// a * conj(b) = a.x (b.x, -b.y) + a.y (b.y, b.x)
template <bool CONJ> __device__ __forceinline__ float2 cmul_tw(float2 a, float2 b) {
  if (CONJ)
    return __ffma2_rn(make_float2(a.y, a.y), make_float2(b.y, b.x), __fmul2_rn(make_float2(a.x, a.x), make_float2(b.x, -b.y)));
  return cmul(a, b);
}

template <int DIR, typename C>
__device__ __forceinline__ void dft2(C& a0, C& a1) {
  C t = a0; a0 = cadd(t, a1); a1 = csub(t, a1);
}

template <int DIR, typename C>
__device__ __forceinline__ void dft4(C& a0, C& a1, C& a2, C& a3) {
  C s02 = cadd(a0, a2), d02 = csub(a0, a2);
  C s13 = cadd(a1, a3), d13 = mul_i<DIR>(csub(a1, a3));
  a0 = cadd(s02, s13); a2 = csub(s02, s13);
  a1 = cadd(d02, d13); a3 = csub(d02, d13);
}

// In-place DFTs with sign DIR of v[o + s*r], r = 0..n-1 (natural order).
template <int DIR, typename T, typename C>
__device__ __forceinline__ void dft8s(C* v, int o, int st) {
  C e0 = v[o], e1 = v[o + 2 * st], e2 = v[o + 4 * st], e3 = v[o + 6 * st];
  C o0 = v[o + st], o1 = v[o + 3 * st], o2 = v[o + 5 * st], o3 = v[o + 7 * st];
  dft4<DIR>(e0, e1, e2, e3);
  dft4<DIR>(o0, o1, o2, o3);
  const T r = (T)0.70710678118654752440;  // 1/sqrt(2)
  // t1 = o1 (1 + DIR i)/sqrt2 = (o1 + DIR i o1) r;  t3 = o3 (-1 + DIR i)/sqrt2
  const C t1 = cscale(cadd(o1, mul_i<DIR>(o1)), r);
  C t2 = mul_i<DIR>(o2);
  const C t3 = cscale(csub(mul_i<DIR>(o3), o3), r);
  v[o] = cadd(e0, o0); v[o + 4 * st] = csub(e0, o0);
  v[o + st] = cadd(e1, t1); v[o + 5 * st] = csub(e1, t1);
  v[o + 2 * st] = cadd(e2, t2); v[o + 6 * st] = csub(e2, t2);
  v[o + 3 * st] = cadd(e3, t3); v[o + 7 * st] = csub(e3, t3);
}

// 16-point DFT as 4 x 4: DFT4 over the stride-4 subsequences, twiddles
// exp(DIR 2 pi i k m / 16), DFT4 across, transposed write-back.
template <int DIR, typename T, typename C>
__device__ __forceinline__ void dft16(C (&v)[16]) {
  const T c1 = (T)0.92387953251128675613;  // cos(pi/8)
  const T s1 = (T)0.38268343236508977173;  // sin(pi/8)
  const T h = (T)0.70710678118654752440;   // cos(pi/4)
#pragma unroll
  for (int k = 0; k < 4; ++k) dft4<DIR>(v[k], v[k + 4], v[k + 8], v[k + 12]);
  // v[k + 4 m] now holds X_k[m]; multiply by w16^(k m), w16 = exp(DIR 2 pi i / 16)
  auto rot = [&](C a, T c, T s) {  // a * (c + DIR i s) = a c + (DIR i a) s
    if constexpr (sizeof(T) == 4) {
      return __ffma2_rn(mul_i<DIR>(a), make_float2(s, s), __fmul2_rn(a, make_float2(c, c)));
    } else {
      C r;
      r.x = a.x * c - (T)DIR * a.y * s;
      r.y = a.y * c + (T)DIR * a.x * s;
      return r;
    }
  };
  v[5] = rot(v[5], c1, s1);    // k=1 m=1: w^1
  v[9] = rot(v[9], h, h);      // k=1 m=2: w^2
  v[13] = rot(v[13], s1, c1);  // k=1 m=3: w^3
  v[6] = rot(v[6], h, h);      // k=2 m=1: w^2
  v[10] = mul_i<DIR>(v[10]);   // k=2 m=2: w^4
  v[14] = rot(v[14], -h, h);   // k=2 m=3: w^6
  v[7] = rot(v[7], s1, c1);    // k=3 m=1: w^3
  v[11] = rot(v[11], -h, h);   // k=3 m=2: w^6
  v[15] = rot(v[15], -c1, -s1);  // k=3 m=3: w^9
#pragma unroll
  for (int m = 0; m < 4; ++m) dft4<DIR>(v[4 * m], v[4 * m + 1], v[4 * m + 2], v[4 * m + 3]);
  // v[4 m + n] holds X[m + 4 n]; transpose to natural order
  C t[16];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) t[m + 4 * n] = v[4 * m + n];
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = t[i];
}

// Two independent single-precision transforms carried in the two lanes of
// sm_100's packed FP32 operations: re and im hold the real and imaginary parts
// of (transform 0, transform 1).  Every operation of the pair is one packed
// instruction per component with no register shuffles (a multiplication by i
// is a renaming), twiddles are broadcast pairs, and an element of both
// transforms moves through shared memory as one 16-byte access.
struct __align__(16) Dual {
  float2 re, im;
};
__device__ __forceinline__ Dual dadd(const Dual& a, const Dual& b) {
  return {__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)};
}
__device__ __forceinline__ float2 fneg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ Dual dsub(const Dual& a, const Dual& b) {
  return {__fadd2_rn(a.re, fneg2(b.re)), __fadd2_rn(a.im, fneg2(b.im))};
}
// a + DIR i b and a - DIR i b
template <int DIR> __device__ __forceinline__ Dual dadd_i(const Dual& a, const Dual& b) {
  if (DIR > 0) return {__fadd2_rn(a.re, fneg2(b.im)), __fadd2_rn(a.im, b.re)};
  return {__fadd2_rn(a.re, b.im), __fadd2_rn(a.im, fneg2(b.re))};
}
template <int DIR> __device__ __forceinline__ Dual dsub_i(const Dual& a, const Dual& b) {
  return dadd_i<-DIR>(a, b);
}
__device__ __forceinline__ Dual dscale(const Dual& a, float r) {
  const float2 rr = make_float2(r, r);
  return {__fmul2_rn(a.re, rr), __fmul2_rn(a.im, rr)};
}
// a * (c + i s), the same factor for both transforms
__device__ __forceinline__ Dual dmul(const Dual& a, float c, float s) {
  const float2 cc = make_float2(c, c), ss = make_float2(s, s);
  return {__ffma2_rn(fneg2(a.im), ss, __fmul2_rn(a.re, cc)), __ffma2_rn(a.im, cc, __fmul2_rn(a.re, ss))};
}

template <int DIR> __device__ __forceinline__ void dft2(Dual& a0, Dual& a1) {
  const Dual t = a0;
  a0 = dadd(t, a1);
  a1 = dsub(t, a1);
}
template <int DIR> __device__ __forceinline__ void dft4(Dual& a0, Dual& a1, Dual& a2, Dual& a3) {
  const Dual s02 = dadd(a0, a2), d02 = dsub(a0, a2);
  const Dual s13 = dadd(a1, a3), d13 = dsub(a1, a3);
  a0 = dadd(s02, s13);
  a2 = dsub(s02, s13);
  a1 = dadd_i<DIR>(d02, d13);
  a3 = dsub_i<DIR>(d02, d13);
}
template <int DIR> __device__ __forceinline__ void dft8s(Dual* v, int o, int st) {
  Dual e0 = v[o], e1 = v[o + 2 * st], e2 = v[o + 4 * st], e3 = v[o + 6 * st];
  Dual o0 = v[o + st], o1 = v[o + 3 * st], o2 = v[o + 5 * st], o3 = v[o + 7 * st];
  dft4<DIR>(e0, e1, e2, e3);
  dft4<DIR>(o0, o1, o2, o3);
  const float r = 0.70710678118654752440f;  // 1/sqrt(2)
  // t1 = o1 (1 + DIR i)/sqrt2, t3 = o3 (1 - DIR i)/sqrt2 (rounded as the one-transform form does)
  const Dual t1 = dscale(dadd_i<DIR>(o1, o1), r), t3 = dscale(dsub_i<DIR>(o3, o3), r);
  v[o] = dadd(e0, o0); v[o + 4 * st] = dsub(e0, o0);
  v[o + st] = dadd(e1, t1); v[o + 5 * st] = dsub(e1, t1);
  v[o + 2 * st] = dadd_i<DIR>(e2, o2); v[o + 6 * st] = dsub_i<DIR>(e2, o2);
  v[o + 3 * st] = dsub(e3, t3); v[o + 7 * st] = dadd(e3, t3);
}
template <int DIR> __device__ __forceinline__ void dft16(Dual (&v)[16]) {
  const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
  const float D = (float)DIR;
#pragma unroll
  for (int k = 0; k < 4; ++k) dft4<DIR>(v[k], v[k + 4], v[k + 8], v[k + 12]);
  v[5] = dmul(v[5], c1, D * s1);     // k=1 m=1: w^1
  v[9] = dmul(v[9], h, D * h);       // k=1 m=2: w^2
  v[13] = dmul(v[13], s1, D * c1);   // k=1 m=3: w^3
  v[6] = dmul(v[6], h, D * h);       // k=2 m=1: w^2
  v[14] = dmul(v[14], -h, D * h);    // k=2 m=3: w^6
  v[7] = dmul(v[7], s1, D * c1);     // k=3 m=1: w^3
  v[11] = dmul(v[11], -h, D * h);    // k=3 m=2: w^6
  v[15] = dmul(v[15], -c1, -D * s1); // k=3 m=3: w^9
  // k=2 m=2 is a multiplication by DIR i: renamed
  v[10] = DIR > 0 ? Dual{fneg2(v[10].im), v[10].re} : Dual{v[10].im, fneg2(v[10].re)};
#pragma unroll
  for (int m = 0; m < 4; ++m) dft4<DIR>(v[4 * m], v[4 * m + 1], v[4 * m + 2], v[4 * m + 3]);
  Dual t[16];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) t[m + 4 * n] = v[4 * m + n];
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = t[i];
}

// Shared-memory addresses of the exchange after a pass of stride p = 2^lp and
// radix 2^lr: element i sits at i + mul (i >> sh), which puts the accesses a
// bank cycle serves (BK = 128 bytes / element) in different banks for both
// patterns.  The stores, thread j = a p + k writing elements a p 2^lr + k + r p,
// need the blocks of different a moved apart while p < BK (mul = p slots per
// 2^sh = max(BK, p 2^lr) elements); the loads, elements j + m G, are BK
// consecutive elements of one such block.  i >> sh is the same for all r of a
// thread, and for G >= BK linear in m, so every address is a base plus r p or
// m ls: one add, where the earlier XOR swizzle took six integer operations per
// store (a third of the row pass's instructions were integer).
template <int BK, int G>
struct Xchg {
  int sh, mul, p;
  __device__ __forceinline__ Xchg(int p_, int lp, int lr) : p(p_) {
    constexpr int LB = BK == 16 ? 4 : 3;
    sh = lp + lr > LB ? lp + lr : LB;
    mul = p_ < BK ? p_ : 0;
  }
  __device__ __forceinline__ int at(int i) const { return i + mul * (i >> sh); }
  // first of the addresses base + r p of the stores from element b
  __device__ __forceinline__ int store(int b) const { return at(b); }
  // address of element j + m G
  __device__ __forceinline__ int load(int j, int m) const {
    if constexpr (G >= BK) return at(j) + m * (G + mul * (G >> sh));
    else return at(j + m * G);
  }
};

// NF independent group FFTs executed together.  v[f]: this thread's R
// values of transform f in strided layout, v[f][m] = x_f[j + m G] with
// G = N/R (in and out).  sbuf + f * bstride: spad_size<R>(N) complex slots of
// shared memory for transform f.  The NF transforms share every barrier and
// every twiddle load, which gives each thread NF times the independent work
// per pass.  All threads of the block must call it together (it uses
// __syncthreads).  The routine begins with a barrier before its first write to
// sbuf; on exit other threads may still be reading sbuf, so callers
// synchronise before writing to it again.  Passes: one pass of radix
// 2^(log2 N mod log2 R) first when log2 N is not a multiple of log2 R (each
// thread then runs R / that radix butterflies), then radix-R passes.  Single
// precision runs an even NF in pairs (Dual, fft_dual): the buffers
// of transforms f and f + 1 are then one buffer of 16-byte slots, so bstride
// must be the distance of adjacent buffers and sbuf 16-byte aligned.
//
// Element type of the passes: E = Dual (two transforms) or the complex type.
template <typename E> struct FftElem {  // one complex transform
  template <bool INV> static __device__ __forceinline__ E twiddle(const E& a, const E& w) { return cmul_tw<INV>(a, w); }
};
template <> struct FftElem<Dual> {
  template <bool INV> static __device__ __forceinline__ Dual twiddle(const Dual& a, const float2& w) {
    return dmul(a, w.x, INV ? -w.y : w.y);
  }
};

template <typename T, int LOG2N, int R>
__host__ __device__ constexpr bool fft_tw2() { return R == 8 && LOG2N == 11; }

template <typename T, int LOG2N, int R, int DIR, int NE, typename E>
__device__ __forceinline__ void fft_elems(E (&v)[NE][R], E* sbuf, int bstride, int j,
                                          const typename Cplx<T>::type* __restrict__ tw) {
  using C = typename Cplx<T>::type;
  constexpr int LR = R == 16 ? 4 : (R == 8 ? 3 : 2);
  constexpr int N = 1 << LOG2N;
  constexpr int G = N / R;
  constexpr int REM = LOG2N % LR;
  constexpr int NPR = LOG2N / LR;
  constexpr bool INV = DIR > 0;
  constexpr int BK = 128 / (int)sizeof(E);
  constexpr bool dual = sizeof(E) == 2 * sizeof(C);
  static_assert(R == 4 || R == 8 || R == 16, "radix 4, 8 or 16");
  static_assert(LOG2N >= LR, "N >= R");
  auto bf4 = [](E& a0, E& a1, E& a2, E& a3) { dft4<DIR>(a0, a1, a2, a3); };
  auto bf8 = [](E* x, int o, int st) {
    if constexpr (dual) dft8s<DIR>(x, o, st);
    else dft8s<DIR, T>(x, o, st);
  };
  // Twiddle root of the first radix pass, requested before any work: each
  // pass's root is loaded one pass ahead so the load's latency (the table is
  // often not L1-resident next to large shared-memory buffers) overlaps the
  // butterflies and exchange of the pass before.
  // (TW2, every radix-8 transform of N = 2048 -- the row pass of both precisions
  // and the column pass in double: w and w^3 from the table instead of w alone.
  // Powers of w carry its rounding r-fold, and the row pass there, radix 8 instead
  // of radix 4, is to be no further from exact: at w, w^3 the squared errors of
  // its twiddles sum to 12 units over its passes, to 17.5 in radix 4, to 52 from
  // w alone.)
  constexpr bool TW2 = fft_tw2<T, LOG2N, R>();
  auto root = [&](int pp, int lpp, int e) -> C {
    return tw[((e * (j & (pp - 1))) << (LOG2N - lpp - LR)) & (N - 1)];
  };
  C w_next = REM != 0 ? root(1 << REM, REM, 1) : C{};
  C w3_next = REM != 0 && TW2 ? root(1 << REM, REM, 3) : C{};
  int p = 1;
  if (REM != 0) {
    constexpr int RP = 1 << REM;
    constexpr int NB = R / RP;
#pragma unroll
    for (int f = 0; f < NE; ++f)
#pragma unroll
      for (int q = 0; q < NB; ++q) {
        if constexpr (RP == 2) {
          dft2<DIR>(v[f][q], v[f][q + NB]);
        } else if constexpr (RP == 4) {
          bf4(v[f][q], v[f][q + NB], v[f][q + 2 * NB], v[f][q + 3 * NB]);
        } else {
          bf8(v[f], q, NB);
        }
      }
    __syncthreads();
    const Xchg<BK, G> x(1, 0, REM);
#pragma unroll
    for (int f = 0; f < NE; ++f)
#pragma unroll
      for (int q = 0; q < NB; ++q) {
        const int a = x.store((j + q * G) * RP);  // butterfly j + q G, p = 1 so k = 0
#pragma unroll
        for (int r = 0; r < RP; ++r) sbuf[f * bstride + a + r] = v[f][q + r * NB];
      }
    __syncthreads();
#pragma unroll
    for (int f = 0; f < NE; ++f)
#pragma unroll
      for (int m = 0; m < R; ++m) v[f][m] = sbuf[f * bstride + x.load(j, m)];
    p = RP;
  }
  // Radix-R passes.  The pass loop is kept rolled so that its code is shared
  // by all passes (the unrolled form overflows the instruction cache).
  int lp = REM;  // log2(p)
#pragma unroll 1
  for (int pass = 0; pass < NPR; ++pass) {
    const int k = j & (p - 1);
    const C w_cur = w_next, w3_cur = w3_next;
    if (pass + 1 < NPR) {
      w_next = root(p * R, lp + LR, 1);
      if (TW2) w3_next = root(p * R, lp + LR, 3);
    }
    if (p > 1) {
      // w^r for r = 1..R-1 from one table load w = exp(-+2 pi i k / (p R)):
      // powers by complex products (at most three chained roundings)
      const C w1 = w_cur;
      C wp[R];
      wp[1] = w1;
      wp[2] = cmul(w1, w1);
      wp[3] = TW2 ? w3_cur : cmul(wp[2], w1);
      if constexpr (R >= 8) {
        wp[4] = TW2 ? cmul(wp[3], w1) : cmul(wp[2], wp[2]);
        wp[5] = TW2 ? cmul(wp[3], wp[2]) : cmul(wp[4], w1);
        wp[6] = cmul(wp[3], wp[3]);
        wp[7] = cmul(wp[4], wp[3]);
      }
      if constexpr (R == 16) {
        wp[8] = cmul(wp[4], wp[4]);
#pragma unroll
        for (int r = 9; r < 16; ++r) wp[r] = cmul(wp[8], wp[r - 8]);
      }
#pragma unroll
      for (int r = 1; r < R; ++r)
#pragma unroll
        for (int f = 0; f < NE; ++f) v[f][r] = FftElem<E>::template twiddle<INV>(v[f][r], wp[r]);
    }
#pragma unroll
    for (int f = 0; f < NE; ++f) {
      if constexpr (R == 16) {
        if constexpr (dual) dft16<DIR>(v[f]);
        else dft16<DIR, T>(v[f]);
      } else if constexpr (R == 8) {
        bf8(v[f], 0, 1);
      } else {
        bf4(v[f][0], v[f][1], v[f][2], v[f][3]);
      }
    }
    if (pass != NPR - 1) {
      __syncthreads();
      const Xchg<BK, G> x(p, lp, LR);
      const int a = x.store((j - k) * R + k);
#pragma unroll
      for (int f = 0; f < NE; ++f)
#pragma unroll
        for (int r = 0; r < R; ++r) sbuf[f * bstride + a + r * p] = v[f][r];
      __syncthreads();
#pragma unroll
      for (int f = 0; f < NE; ++f)
#pragma unroll
        for (int m = 0; m < R; ++m) v[f][m] = sbuf[f * bstride + x.load(j, m)];
    }
    p *= R;
    lp += LR;
  }
}

// Whether NF transforms run in pairs.  Not in radix 16 with a shorter first
// pass (N = 2048): its 8-byte exchange is conflict-free in n + n / 16 slots, the
// 16-byte one needs n + n / 8, and the pairs were slower (theta column pass
// 40.1 -> 43.6 us; at N = 4096, 190 -> 181 us, row stage pass 277 -> 264 us).
template <typename T, int LOG2N, int R>
__host__ __device__ constexpr bool fft_dual(int nf) {
  return sizeof(T) == 4 && nf % 2 == 0 && (R != 16 || LOG2N % 4 == 0);
}

template <typename T, int LOG2N, int R, int DIR, int NF>
__device__ __forceinline__ void fft_multi(typename Cplx<T>::type (&v)[NF][R], typename Cplx<T>::type* sbuf,
                                          int bstride, int j, const typename Cplx<T>::type* __restrict__ tw) {
  if constexpr (fft_dual<T, LOG2N, R>(NF)) {
    Dual d[NF / 2][R];
#pragma unroll
    for (int f = 0; f < NF / 2; ++f)
#pragma unroll
      for (int m = 0; m < R; ++m) {
        d[f][m].re = make_float2(v[2 * f][m].x, v[2 * f + 1][m].x);
        d[f][m].im = make_float2(v[2 * f][m].y, v[2 * f + 1][m].y);
      }
    fft_elems<T, LOG2N, R, DIR, NF / 2, Dual>(d, reinterpret_cast<Dual*>(sbuf), bstride, j, tw);
#pragma unroll
    for (int f = 0; f < NF / 2; ++f)
#pragma unroll
      for (int m = 0; m < R; ++m) {
        v[2 * f][m] = make_float2(d[f][m].re.x, d[f][m].im.x);
        v[2 * f + 1][m] = make_float2(d[f][m].re.y, d[f][m].im.y);
      }
  } else {
    fft_elems<T, LOG2N, R, DIR, NF, typename Cplx<T>::type>(v, sbuf, bstride, j, tw);
  }
}

// One group FFT (see fft_multi).
template <typename T, int LOG2N, int R, int DIR>
__device__ __forceinline__ void fft_group(typename Cplx<T>::type (&v)[R], typename Cplx<T>::type* sbuf, int j,
                                          const typename Cplx<T>::type* __restrict__ tw) {
  using C = typename Cplx<T>::type;
  fft_multi<T, LOG2N, R, DIR, 1>(*reinterpret_cast<C(*)[1][R]>(&v), sbuf, 0, j, tw);
}

}  // namespace sqg
