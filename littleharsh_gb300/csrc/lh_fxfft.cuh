// lh_fxfft.cuh -- FP64-grade FFTs in 64-bit fixed point.
//
// GB300 issues 2 FP64 instructions per clock and SM (1.25 TFLOP/s), but 128
// 32-bit integer additions and 32 wide or high 32-bit products.  A 64-bit
// integer addition (two instructions) therefore costs 1/30 of an FP64 one and
// a 64-bit product with a constant (two high products, one wide one) about
// 1/4, measured 57 and 7-11 lanes per clock and SM against 1.93.  FP64
// transforms keep the FP64 pipe 85-89 % busy; the conditional statistics'
// z-inverse runs here instead: every line is scaled by a power of two of its
// own into 64-bit integers (block floating point), transformed exactly except
// for one rounding per product (at 2^-60 of the line's bound), and scaled back
// to FP64.  The step's transforms stay in FP64: a line has one exponent here
// where FP64 has one per value, and the step's last bits are part of
// established runs.
//
// Error.  FP64 rounds every intermediate value to 2^-53 of itself.  Here a
// line's largest value is scaled to just below 2^59, and each pass but the
// first shifts its input right, rounding to nearest, by as much as it can have
// grown:
//  * a forward transform (physical to spectrum) by the plan's shifts, which
//    hold for any line;
//  * an inverse transform by no more than its line's sum of moduli asks for,
//    since no partial sum exceeds it: a spectrum with a few large modes is
//    hardly shifted, and its modes' rounding stays at 2^-59 of the largest.
// Both come out below the FP64 transforms' error, in the 2-norm and at the
// worst point (measured against extended precision over the lengths in use,
// see the tests).
//
// Algorithm.  n = P Q with P = 2^a, Q = 3^b: the prime-factor map
// (sample n = Q n1 + P n2 mod N, frequency k by the Chinese remainder) leaves
// no twiddles between the two parts; within a part, decimation-in-time passes
// of radix 8, 4, 2 and 9, 3.  576 = 8 x 8 x 9 takes three passes and 6 real
// products a point, where the FP64 radix-4/3 transform takes five passes.
// An inverse transform is the forward one with real and imaginary parts
// exchanged.  Twiddles are integers of 62 fractional bits from extended
// precision; w z takes three real products with w_r, w_r + w_i, w_r - w_i, the
// last two subtracted from the first, so that what a product's rounding has of
// a mean cancels in both parts (added to one of them it came out at the first
// output, 9e-16 of the line's rms at n = 576).
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

namespace lh {

typedef long long i64;
typedef longlong2 fx2;  // complex fixed-point value (re, im)

#define FX_HD __host__ __device__ __forceinline__

constexpr int kFxMaxPass = 9;
constexpr int kFxBits = 59;  // a line's real and imaginary parts are below 2^kFxBits before its first pass

// One pass: rad elements at distance mI per item; item t of a vector works at element
// (t / mI) * rad * mI + t % mI and its twiddles are those of k = (t % mI) / inner.
struct FxPass {
  unsigned mI_m, inner_m;           // fdiv multipliers of mI and inner
  short mI, inner, tw;              // tw: first twiddle (-1: none)
  unsigned char rad, shift, before; // shift: bits the input may have to be shifted by; before: of earlier passes
};

// One transform length.  Passed by value to kernels.
struct FxPlan {
  int n, npass;
  int last_step;         // distance of an item's frequencies in the last pass, modulo n
  int shift;             // bits a forward line, and at most an inverse line, is shifted by in all
  FxPass ps[kFxMaxPass];
  const short* pos_sample;   // position of sample s
  const short* freq_pos;     // frequency at a position
  const int4* tw;            // two int4 per twiddle: (w_r, w_r + w_i), (w_r - w_i, -), each high and low word
};

// ---------------------------------------------------------------------------
// arithmetic
// ---------------------------------------------------------------------------

// high 32 bits of a * b
FX_HD int fx_mhi(int a, int b) {
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int)(((i64)a * b) >> 32);
#endif
}

FX_HD i64 fx_shl(i64 a, int s) { return (i64)((unsigned long long)a << s); }

FX_HD i64 fx_pack(int h, int l) { return (i64)(((unsigned long long)(unsigned)h << 32) | (unsigned)l); }
// a >> s with 0 <= s < 32
FX_HD i64 fx_sar(i64 a, int s) {
#ifdef __CUDA_ARCH__
  return fx_pack((int)(a >> 32) >> s, (int)__funnelshift_r((unsigned)a, (unsigned)(a >> 32), s));
#else
  return a >> s;
#endif
}
// high word of a for a signed low word: a = h 2^32 + (int)a.  Written with the sign of the low word: 17 issue slots
// a product against 22 with a 64-bit addition of 2^31.
FX_HD int fx_high(i64 a) { return (int)(a >> 32) - ((int)a >> 31); }

// a * b / 2^64 for b = bh 2^32 + bl with bl signed, after shifting a left by PRE and before shifting the result
// left by POST.  The product of the two low words is left out (below one unit of the result); |a| 2^PRE < 2^63 - 2^31.
// The two truncations are centred by a unit, but where the low word is zero: zeros stay zeros.
template <int PRE, int POST>
FX_HD i64 fx_mul(i64 a, int bh, int bl) {
  const i64 s = fx_shl(a, PRE);
  const int l = (int)s, h = fx_high(s);
  const int t = fx_mhi(h, bl) + fx_mhi(l, bh) + (l != 0);
  return fx_shl((i64)h * bh + t, POST);
}

FX_HD fx2 fx_add(fx2 a, fx2 b) { return fx2{a.x + b.x, a.y + b.y}; }
FX_HD fx2 fx_sub(fx2 a, fx2 b) { return fx2{a.x - b.x, a.y - b.y}; }

// z w for a twiddle with 62 fractional bits (|z| < 2^60.5 in modulus)
FX_HD fx2 fx_cmul(fx2 z, int4 w0, int4 w1) {
  const i64 k = fx_mul<2, 0>(z.x + z.y, w0.x, w0.y);
  return fx2{k - fx_mul<2, 0>(z.y, w0.z, w0.w), k - fx_mul<2, 0>(z.x, w1.x, w1.y)};
}

// radix-3 butterfly; LATE: |b - c| may reach 2^62.1, else 2^61.9 / 2
template <bool LATE>
FX_HD void fx_bfly3(fx2& a, fx2& b, fx2& c) {
  constexpr i64 s3 = 0x6ed9eba16132a9cfll;  // sqrt(3)/2 * 2^63
  constexpr int sh = (int)((s3 + 0x80000000ll) >> 32), sl = (int)(s3 & 0xffffffffll);
  const fx2 t = fx_add(b, c), e = fx_sub(b, c);
  const fx2 d = LATE ? fx2{fx_mul<0, 1>(e.x, sh, sl), fx_mul<0, 1>(e.y, sh, sl)}
                     : fx2{fx_mul<1, 0>(e.x, sh, sl), fx_mul<1, 0>(e.y, sh, sl)};
  const fx2 m = fx2{a.x - (t.x >> 1), a.y - (t.y >> 1)};
  a = fx_add(a, t);
  b = fx2{m.x + d.y, m.y - d.x};
  c = fx2{m.x - d.y, m.y + d.x};
}

FX_HD void fx_bfly4(fx2& a, fx2& b, fx2& c, fx2& d) {
  const fx2 t0 = fx_add(a, c), t1 = fx_sub(a, c), t2 = fx_add(b, d), t3 = fx_sub(b, d);
  a = fx_add(t0, t2);
  c = fx_sub(t0, t2);
  b = fx2{t1.x + t3.y, t1.y - t3.x};
  d = fx2{t1.x - t3.y, t1.y + t3.x};
}

// z exp(-i a), |z| < 2^61.6: c = cos a, s = sin a given as round(2^62 .) of (c, c - s, c + s): three products
template <i64 R, i64 S, i64 D>
FX_HD fx2 fx_cmulc(fx2 z) {
  constexpr int rh = (int)((R + 0x80000000ll) >> 32), rl = (int)(R & 0xffffffffll);
  constexpr int sh = (int)((S + 0x80000000ll) >> 32), sl = (int)(S & 0xffffffffll);
  constexpr int dh = (int)((D + 0x80000000ll) >> 32), dl = (int)(D & 0xffffffffll);
  const i64 k = fx_mul<1, 1>(z.x + z.y, rh, rl);
  return fx2{k - fx_mul<1, 1>(z.y, sh, sl), k - fx_mul<1, 1>(z.x, dh, dl)};
}

// RAD-point DFT of v in place (natural order), exp(-2 pi i k p / RAD)
template <int RAD>
FX_HD void fx_dft(fx2* v) {
  if constexpr (RAD == 2) {
    const fx2 a = v[0], b = v[1];
    v[0] = fx_add(a, b);
    v[1] = fx_sub(a, b);
  } else if constexpr (RAD == 3) {
    fx_bfly3<false>(v[0], v[1], v[2]);
  } else if constexpr (RAD == 4) {
    fx_bfly4(v[0], v[1], v[2], v[3]);
  } else if constexpr (RAD == 8) {
    constexpr i64 c8 = 0x5a827999fcef3242ll;  // sqrt(1/2) * 2^63
    constexpr int ch = (int)((c8 + 0x80000000ll) >> 32), cl = (int)(c8 & 0xffffffffll);
    fx_bfly4(v[0], v[2], v[4], v[6]);
    fx_bfly4(v[1], v[3], v[5], v[7]);
    // odd outputs times exp(-i pi j / 4): (x + y, y - x) c, -i, (y - x, -(x + y)) c
    const fx2 o1 = fx2{fx_mul<0, 1>(v[3].x + v[3].y, ch, cl), fx_mul<0, 1>(v[3].y - v[3].x, ch, cl)};
    const fx2 o2 = fx2{v[5].y, -v[5].x};
    const fx2 o3 = fx2{fx_mul<0, 1>(v[7].y - v[7].x, ch, cl), -fx_mul<0, 1>(v[7].x + v[7].y, ch, cl)};
    const fx2 o0 = v[1], e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = fx_add(e0, o0); v[4] = fx_sub(e0, o0);
    v[1] = fx_add(e1, o1); v[5] = fx_sub(e1, o1);
    v[2] = fx_add(e2, o2); v[6] = fx_sub(e2, o2);
    v[3] = fx_add(e3, o3); v[7] = fx_sub(e3, o3);
  } else {  // 9 = 3 x 3
    fx_bfly3<false>(v[0], v[3], v[6]);
    fx_bfly3<false>(v[1], v[4], v[7]);
    fx_bfly3<false>(v[2], v[5], v[8]);
    // exp(-2 pi i m / 9), m = 1, 2, 2, 4: (cos, cos - sin, cos + sin) * 2^62 as (w_r, w_r + w_i, w_r - w_i)
    v[4] = fx_cmulc<3532756447825785444ll, 568421815416011021ll, 6497091080235559868ll>(v[4]);
    v[7] = fx_cmulc<800810873071977681ll, -3740813272333314531ll, 5342435018477269894ll>(v[7]);
    v[5] = fx_cmulc<800810873071977681ll, -3740813272333314531ll, 5342435018477269894ll>(v[5]);
    v[8] = fx_cmulc<-4333567320897763126ll, -5910856833893280915ll, -2756277807902245337ll>(v[8]);
    fx_bfly3<true>(v[0], v[1], v[2]);
    fx_bfly3<true>(v[3], v[4], v[5]);
    fx_bfly3<true>(v[6], v[7], v[8]);
    // output k1 + 3 k2 sits at 3 k1 + k2
    fx2 t;
    t = v[1]; v[1] = v[3]; v[3] = t;
    t = v[2]; v[2] = v[6]; v[6] = t;
    t = v[5]; v[5] = v[7]; v[7] = t;
  }
}

// Bits by which a pass shifts the input of a line that may be shifted by g in all.
FX_HD int fx_pass_shift(const FxPass& ps, int g) {
  const int left = g - ps.before;
  return left <= 0 ? 0 : (left < ps.shift ? left : ps.shift);
}

// One pass item: rad elements in registers, shifted right with rounding, twiddled and transformed.
template <int RAD>
FX_HD void fx_item(fx2* v, const int4* tw, int shift) {
  if (shift) {
    const i64 half = (i64)(1u << (shift - 1));
#pragma unroll
    for (int p = 0; p < RAD; ++p) v[p] = fx2{fx_sar(v[p].x + half, shift), fx_sar(v[p].y + half, shift)};
  }
  if (tw) {
#pragma unroll
    for (int p = 1; p < RAD; ++p) {
#ifdef __CUDA_ARCH__
      const int4 w0 = __ldg(tw + 2 * (p - 1)), w1 = __ldg(tw + 2 * (p - 1) + 1);
#else
      const int4 w0 = tw[2 * (p - 1)], w1 = tw[2 * (p - 1) + 1];
#endif
      v[p] = fx_cmul(v[p], w0, w1);
    }
  }
  fx_dft<RAD>(v);
}

// ---------------------------------------------------------------------------
// FP64 <-> fixed point
// ---------------------------------------------------------------------------

// biased exponent of |x| from its high word (0 for zeros and subnormals, 2047 for infinities and NaN)
FX_HD int fx_exp(unsigned hi) { return (int)((hi >> 20) & 2047u); }

// Scale exponent of a line whose largest biased exponent is e: its real and imaginary parts times 2^S are below
// 2^kFxBits, so their moduli are below 2^(kFxBits + 1/2).
FX_HD int fx_scale(int e) { return kFxBits - ((e ? e : 1) - 1022); }

// An upper bound of |x| for a scaled value, in units of 2^42: 2^15 of them (two parts of the longest line) fit 32 bits.
FX_HD unsigned fx_mag(i64 x) {
  const int h = (int)(x >> 32);
  return ((unsigned)(h ^ (h >> 31)) >> 10) + 1u;
}

// Bits that an inverse line is shifted right by over its passes: its sum of moduli, at most sum * 2^42 for the sum of
// fx_mag, comes down to 2^(kFxBits + 1), which no partial sum can exceed; never more than the plan's own shifts,
// which hold for every line.
FX_HD int fx_inv_shift(unsigned sum, int most) {
  int bits = 0;  // sum < 2^bits
#ifdef __CUDA_ARCH__
  bits = 32 - __clz((int)sum);
#else
  while (bits < 32 && (sum >> bits)) ++bits;
#endif
  const int g = bits - (kFxBits + 1 - 42);
  return g < 0 ? 0 : (g < most ? g : most);
}

// x 2^S, S = fx_scale(e) of its line's largest biased exponent e, truncated to an integer below 2^kFxBits
FX_HD i64 fx_from(double x, int e) {
#ifdef __CUDA_ARCH__
  const int hi = __double2hiint(x), lo = __double2loint(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  const int hi = (int)(b >> 32), lo = (int)b;
#endif
  const int ex = fx_exp((unsigned)hi);
  const int d = (e ? e : 1) - (ex ? ex : 1);  // >= 0
  const unsigned long long m =
      ((((unsigned long long)(((unsigned)hi & 0xfffffu) | (ex ? 0x100000u : 0u)) << 32) | (unsigned)lo) << 6) >> (d < 63 ? d : 63);
  const i64 sg = (i64)(hi >> 31);
  return ((i64)m ^ sg) - sg;
}

// x 2^-S as a double (any S)
FX_HD double fx_to(i64 x, int S) {
#ifdef __CUDA_ARCH__
  const double d = __ll2double_rn(x);
  return scalbn(scalbn(d, -S / 2), -S + S / 2);
#else
  return std::ldexp((double)x, -S);
#endif
}

// ---------------------------------------------------------------------------
// passes over shared memory
// ---------------------------------------------------------------------------
#ifdef __CUDACC__

__device__ __forceinline__ int fx_div(int t, int d, unsigned mult) { return d > 1 ? (int)__umulhi((unsigned)t, mult) : t; }

// Where item t of a pass works: first element and twiddles.
struct FxItem {
  int e0;
  const int4* tw;
};
template <int RAD>
__device__ __forceinline__ FxItem fx_at(const FxPlan& P, const FxPass& ps, int t) {
  const int blk = fx_div(t, ps.mI, ps.mI_m), r0 = t - blk * ps.mI;
  FxItem it{blk * RAD * ps.mI + r0, nullptr};
  if (ps.tw >= 0) it.tw = P.tw + 2 * (ps.tw + fx_div(r0, ps.inner, ps.inner_m) * (RAD - 1));
  return it;
}

#define FX_RADIX(r, CALL)                           \
  switch (r) {                                      \
    case 2: { constexpr int RAD = 2; CALL; break; } \
    case 3: { constexpr int RAD = 3; CALL; break; } \
    case 4: { constexpr int RAD = 4; CALL; break; } \
    case 8: { constexpr int RAD = 8; CALL; break; } \
    default: { constexpr int RAD = 9; CALL; break; } \
  }

// 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void fx_copy(fx2* dst, const double2* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void fx_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A column of a tile of 2^ltx columns: element e of column c at buf[e << ltx | c].  A thread works on column
// threadIdx.x % 2^ltx throughout, so that what a column's scale decides is decided once per thread.
struct FxCol {
  fx2* buf;     // of the thread's column
  int ltx;      // log2 of the tile's width
  int t0, dt;   // the thread's first item and its stride
};

// First pass: the column's FP64 values, staged in the places of its integers, scaled by in(value).
template <int RAD, typename In>
__device__ __forceinline__ void fx_first(const FxCol& C, const FxPlan& P, const FxPass& ps, In in) {
  const int items = P.n / RAD;
  for (int t = C.t0; t < items; t += C.dt) {
    const FxItem it = fx_at<RAD>(P, ps, t);
    fx2 v[RAD];
#pragma unroll
    for (int p = 0; p < RAD; ++p) v[p] = in(reinterpret_cast<const double2*>(C.buf)[(it.e0 + p * ps.mI) << C.ltx]);
    fx_dft<RAD>(v);
#pragma unroll
    for (int p = 0; p < RAD; ++p) C.buf[(it.e0 + p * ps.mI) << C.ltx] = v[p];
  }
}

template <int RAD>
__device__ __forceinline__ void fx_middle(const FxCol& C, const FxPlan& P, const FxPass& ps, int shift) {
  const int items = P.n / RAD;
  for (int t = C.t0; t < items; t += C.dt) {
    const FxItem it = fx_at<RAD>(P, ps, t);
    fx2 v[RAD];
#pragma unroll
    for (int p = 0; p < RAD; ++p) v[p] = C.buf[(it.e0 + p * ps.mI) << C.ltx];
    fx_item<RAD>(v, it.tw, shift);
#pragma unroll
    for (int p = 0; p < RAD; ++p) C.buf[(it.e0 + p * ps.mI) << C.ltx] = v[p];
  }
}

// Last pass: outputs to store(frequency, value), the frequencies of an item last_step apart modulo n.
template <int RAD, typename Store>
__device__ __forceinline__ void fx_last(const FxCol& C, const FxPlan& P, const FxPass& ps, int shift, Store store) {
  const int items = P.n / RAD;
  for (int t = C.t0; t < items; t += C.dt) {
    const FxItem it = fx_at<RAD>(P, ps, t);
    fx2 v[RAD];
#pragma unroll
    for (int p = 0; p < RAD; ++p) v[p] = C.buf[(it.e0 + p * ps.mI) << C.ltx];
    fx_item<RAD>(v, it.tw, shift);
    int k = P.freq_pos[it.e0];
#pragma unroll
    for (int p = 0; p < RAD; ++p) {
      store(k, v[p]);
      k += P.last_step;
      if (k >= P.n) k -= P.n;
    }
  }
}

// A tile from its staged FP64 values to store.  total() gives the bits the thread's column is shifted by in all; it is
// called after the first pass (which shifts nothing) and holds a barrier.
template <typename In, typename Total, typename Store>
__device__ __forceinline__ void fx_tile(const FxCol& C, const FxPlan& P, In in, Total total, Store store) {
  FX_RADIX(P.ps[0].rad, (fx_first<RAD>(C, P, P.ps[0], in)));
  const int g = total();
  for (int i = 1; i + 1 < P.npass; ++i) {
    const FxPass& ps = P.ps[i];
    FX_RADIX(ps.rad, (fx_middle<RAD>(C, P, ps, fx_pass_shift(ps, g))));
    __syncthreads();
  }
  if (P.npass > 1) {
    const FxPass& ps = P.ps[P.npass - 1];
    FX_RADIX(ps.rad, (fx_last<RAD>(C, P, ps, fx_pass_shift(ps, g), store)));
  } else {
    for (int pos = C.t0; pos < P.n; pos += C.dt) store(P.freq_pos[pos], C.buf[pos << C.ltx]);
  }
}

// x 2^S for the thread's line (S = fx_scale(e)), on the FP64 pipe: an addition to the exponent and a conversion.
struct FxIn {
  int e, add, least;  // add: S << 20; least: high words up to this one scale to nothing
  bool far;           // exponents beyond the conversion's range: by integer shifts
  __device__ __forceinline__ FxIn() {}
  __device__ __forceinline__ explicit FxIn(int e_) : e(e_) {
    const int S = fx_scale(e);
    add = (int)((unsigned)S << 20);
    least = (int)((unsigned)max(1 - S, 1) << 20) - 1;
    far = S > 900 || S < -900;
  }
  __device__ __forceinline__ i64 operator()(double x) const {
    if (far) return fx_from(x, e);
    const int hi = __double2hiint(x);
    const i64 v = __double2ll_rn(__hiloint2double(hi + add, __double2loint(x)));
    return (hi & 0x7fffffff) > least ? v : 0;
  }
};
// x 2^-S for the thread's line: a conversion and an addition to the exponent.  NaN for a line that held one or an infinity.
struct FxOut {
  int S, sub;
  bool far, bad;
  __device__ __forceinline__ FxOut(int e, int S_) : S(S_), bad(e == 2047) {
    sub = (int)((unsigned)S << 20);
    far = S > 900 || S < -900;
  }
  __device__ __forceinline__ double operator()(i64 x) const {
    if (far) return bad ? __longlong_as_double(0x7ff8000000000000ll) : fx_to(x, S);
    const double d = __ll2double_rn(x);
    const int hi = __double2hiint(d);
    return __hiloint2double(hi ? hi - sub : 0, __double2loint(d));
  }
};

// larger biased exponent word of a complex value (sign removed)
__device__ __forceinline__ unsigned fx_hi(double2 v) {
  return max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
}
#endif

// ---------------------------------------------------------------------------
// plan tables (host)
// ---------------------------------------------------------------------------

struct FxTables {
  std::vector<short> pos_sample, pos_freq, freq_pos;
  std::vector<int4> tw;
};

// high and signed low word of round(v 2^62)
inline void fx_word(long double v, int* h, int* l) {
  v *= 4611686018427387904.0L;
  const i64 q = (i64)(v < 0 ? v - 0.5L : v + 0.5L);
  *h = (int)((q + 0x80000000ll) >> 32);
  *l = (int)q;
}

inline unsigned fx_div_mult(unsigned d) { return d > 1 ? 0xFFFFFFFFu / d + 1u : 0u; }

// Fills the plan and its tables for a length of factors 2 and 3; false for another one.
inline bool fx_build(int n, FxPlan* plan, FxTables* tab) {
  int P = 1, Q = 1, m = n, a = 0, b = 0;
  while (m % 2 == 0) { m /= 2; P *= 2; ++a; }
  while (m % 3 == 0) { m /= 3; Q *= 3; ++b; }
  if (m != 1 || n > 16384) return false;
  int rad[2][kFxMaxPass], np[2] = {0, 0};
  if (a == 1) rad[0][np[0]++] = 2;
  else {
    int r8 = a / 3, r4 = 0;
    if (a % 3 == 2) r4 = 1;
    if (a % 3 == 1) { --r8; r4 = 2; }
    for (int i = 0; i < r8; ++i) rad[0][np[0]++] = 8;
    for (int i = 0; i < r4; ++i) rad[0][np[0]++] = 4;
  }
  if (b % 2) rad[1][np[1]++] = 3;
  for (int i = 0; i < b / 2; ++i) rad[1][np[1]++] = 9;
  if (np[0] + np[1] > kFxMaxPass) return false;
  std::memset(plan, 0, sizeof *plan);
  plan->n = n;
  // digit-reversed place of index x in a part of length len
  auto place = [&](int part, int x, int len) {
    int pos = 0;
    for (int i = np[part] - 1; i >= 0; --i) {
      const int r = rad[part][i];
      len /= r;
      pos += (x % r) * len;
      x /= r;
    }
    return pos;
  };
  auto inverse = [](int v, int mod) {  // v^-1 modulo mod
    for (int i = 0; i < mod; ++i)
      if ((long long)v * i % mod == 1 % mod) return i;
    return 0;
  };
  const int qi = inverse(Q % P, P), pi = inverse(P % Q, Q);
  tab->pos_sample.resize(n); tab->pos_freq.resize(n); tab->freq_pos.resize(n);
  for (int s = 0; s < n; ++s) {
    const int n1 = (int)((long long)s * qi % P), n2 = (int)((long long)s * pi % Q);
    const int ps = place(0, n1, P) * Q + place(1, n2, Q), pf = (s % P) * Q + s % Q;
    tab->pos_sample[s] = (short)ps;
    tab->pos_freq[s] = (short)pf;
    tab->freq_pos[pf] = (short)s;
  }
  tab->tw.clear();
  const long double two_pi = 6.283185307179586476925286766559005768L;
  double bits = kFxBits + 0.5;  // log2 bound of a forward line's moduli
  int ip = 0;
  for (int part = 0; part < 2; ++part) {
    const int inner = part == 0 ? Q : 1;
    int mm = 1;
    for (int i = 0; i < np[part]; ++i, ++ip) {
      const int r = rad[part][i];
      FxPass& ps = plan->ps[ip];
      ps.rad = (unsigned char)r;
      ps.mI = (short)(mm * inner);
      ps.inner = (short)inner;
      ps.tw = -1;
      ps.mI_m = fx_div_mult((unsigned)(mm * inner));
      ps.inner_m = fx_div_mult((unsigned)inner);
      if (mm > 1) {
        ps.tw = (short)(tab->tw.size() / 2);
        for (int k = 0; k < mm; ++k)
          for (int p = 1; p < r; ++p) {
            const long double t = two_pi * (long double)(k * p) / (long double)(mm * r);
            const long double c = cosl(t), s = -sinl(t);
            int4 w0{}, w1{};
            fx_word(c, &w0.x, &w0.y);
            fx_word(c + s, &w0.z, &w0.w);
            fx_word(c - s, &w1.x, &w1.y);
            tab->tw.push_back(w0);
            tab->tw.push_back(w1);
          }
      }
      ps.before = (unsigned char)plan->shift;
      for (; bits > kFxBits + 0.5 + 1e-9; bits -= 1.0) {
        ++ps.shift;
        ++plan->shift;
      }
      bits += std::log2((double)r);  // below 2^62.7 after the last pass
      mm *= r;
    }
  }
  plan->npass = np[0] + np[1];
  if (plan->npass) {
    const FxPass& l = plan->ps[plan->npass - 1];
    plan->last_step = n > 1 ? (tab->freq_pos[l.mI] - tab->freq_pos[0] + n) % n : 0;
  }
  return true;
}

}  // namespace lh
