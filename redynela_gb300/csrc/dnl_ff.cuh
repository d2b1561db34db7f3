// Pairs of FP32 numbers ("ff": the unevaluated sum h + l, ~46-47 bits) for the element pass.
//
// Why: on GB300 every FP64 instruction (add, multiply, fma, compare, conversion to or from FP32)
// holds its scheduler partition's FP64 pipe for 64 cycles per warp (measured: 0.5 lanes per cycle
// and partition, the same as its latency), where an FP32 fma takes one.  A multiply-add on pairs is
// 6 FP32 instructions in the form below, ten times less, and the FP64 pipe stays free for what
// needs it: coordinate differences and the sums into the stored FP64 state.
//
// Why it is precise enough: in an explicit step the strain increment is small (|F - I| <= kFastMax, 0.5 %;
// larger increments take the FP64 path), and the pairs carry F - I, C - I, ln U and R - I themselves, not 1 +
// them.  FP64 rounds 1 + x at 2^-53 absolute; a pair rounds x at 2^-47 relative.  Root mean square errors
// of a force pass against 80-bit arithmetic, separate distorted elements at 5 to 60 edges from the origin,
// six kinds of increments, hexahedra, pairs | FP64, stresses and forces relative:
//   |G|      ln U               R                  S                  evp                forces
//   2^-8     1.9e-17 | 5.5e-17  2.4e-17 | 2.0e-16  1.5e-14 | 4.0e-14  1.4e-16 | 1.9e-16  1.3e-14 | 4.6e-14
//   2^-10    9e-18   | 5.5e-17  2.1e-17 | 2.0e-16  1.2e-14 | 6.0e-14  4.1e-17 | 1.2e-16  1.2e-14 | 6.9e-14
//   2^-14.5  7e-18   | 5.7e-17  2.3e-17 | 1.8e-16  9e-15   | 7.1e-14  1.8e-17 | 4.8e-17  1.3e-14 | 1.0e-13
// The other element types are alike.  Above the limit the stress, which the return maps back from a trial
// value several times as large, and the plastic multiplier would carry more than FP64 (uniaxial increments
// of 2^-7 in the quads: S 2.1 to 2.3 times FP64's error; evp of hexahedra 3.0e-16 | 2.0e-16).
//
// Error-free steps used: Knuth's two-sum, Dekker's fast two-sum, the product error by fma.  Dot
// products accumulate on a fixed grid (Acc): the running sum starts at C = 1.5 2^k with 2^(k-1) an
// upper bound of the result, so every partial sum lies in one binade, rounds to multiples of
// u = 2^(k-23), and both s1 - s0 and the term's remainder are exact: 6 instructions per term
// instead of 12 with two-sums.  The error is absolute, ~2^-48 of 2^k.
//
// All functions are host and device: the host build is the CPU test of this arithmetic.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

namespace dnl {

#define FFD __host__ __device__ __forceinline__

struct ff {
  float h, l;
};

FFD uint32_t f_bits(float a)
{
#ifdef __CUDA_ARCH__
  return __float_as_uint(a);
#else
  uint32_t u;
  memcpy(&u, &a, 4);
  return u;
#endif
}
FFD float bits_f(uint32_t u)
{
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float a;
  memcpy(&a, &u, 4);
  return a;
#endif
}
FFD uint64_t d_bits(double a)
{
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(a);
#else
  uint64_t u;
  memcpy(&u, &a, 8);
  return u;
#endif
}
FFD double bits_d(uint64_t u)
{
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double a;
  memcpy(&a, &u, 8);
  return a;
#endif
}
FFD float f_fma(float a, float b, float c)
{
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return fmaf(a, b, c);
#endif
}
FFD float f_rsqrt(float a)  // hardware seed (2 ulps), refined by the callers
{
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
#else
  return 1.0f / sqrtf(a);
#endif
}
FFD float f_rcp(float a)  // hardware seed (1 ulp), refined by the callers
{
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
#else
  return 1.0f / a;
#endif
}
FFD float f_abs(float a) { return bits_f(f_bits(a) & 0x7fffffffu); }
FFD float f_max(float a, float b)  // NaN in either argument is kept
{
#ifdef __CUDA_ARCH__
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
#else
  return a != a || a > b ? a : b;
#endif
}

FFD ff ff_norm(float h, float l)  // |h| >= |l| or h = 0
{
  ff r;
  r.h = h + l;
  r.l = l - (r.h - h);
  return r;
}
FFD ff two_sum(float a, float b)
{
  ff r;
  r.h = a + b;
  const float bb = r.h - a;
  r.l = (a - (r.h - bb)) + (b - bb);
  return r;
}
FFD ff ff_neg(ff a) { return ff{-a.h, -a.l}; }
FFD ff ff_add(ff a, ff b)
{
  ff s = two_sum(a.h, b.h);
  return ff_norm(s.h, s.l + (a.l + b.l));
}
FFD ff ff_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }
FFD ff ff_mul(ff a, ff b)
{
  const float p = a.h * b.h;
  float e = f_fma(a.h, b.h, -p);
  e = f_fma(a.h, b.l, e);
  e = f_fma(a.l, b.h, e);
  return ff_norm(p, e);
}
FFD ff ff_mulf(ff a, float b)
{
  const float p = a.h * b;
  return ff_norm(p, f_fma(a.l, b, f_fma(a.h, b, -p)));
}
FFD ff ff_scale(ff a, float p2) { return ff{a.h * p2, a.l * p2}; }  // p2 a power of two: exact
// 1/a: the seed and one Newton step with the squared residual (relative error ~2^-45)
FFD ff ff_rcp(ff a)
{
  const float r = f_rcp(a.h);
  const float e = f_fma(-a.l, r, f_fma(-a.h, r, 1.0f));
  return ff_norm(r, r * f_fma(e, e, e));
}
// 1/sqrt(a): the seed w, the residual 1 - a w^2 exact to 2^-46, w (1 + r/2 + 3 r^2/8)
FFD ff ff_rsqrt(ff a)
{
  const float w = f_rsqrt(a.h);
  const float y = a.h * w;
  const float ye = f_fma(a.l, w, f_fma(a.h, w, -y));
  const float r = f_fma(-ye, w, f_fma(-y, w, 1.0f));
  return ff_norm(w, w * (r * f_fma(0.375f, r, 0.5f)));
}
// sqrt(a) from w = 1/sqrt(a) in single precision: n = a w, n + (a - n^2) w / 2
FFD ff ff_sqrt(ff a, float w)
{
  const float n = a.h * w;
  return ff_norm(n, (f_fma(-n, n, a.h) + a.l) * (0.5f * w));
}
// |a| < |b| / a > b: the high parts' difference is exact where the low ones decide
FFD bool ff_abs_lt(ff a, ff b)
{
  const float sa = a.h < 0.f || (a.h == 0.f && a.l < 0.f) ? -1.f : 1.f;
  const float sb = b.h < 0.f || (b.h == 0.f && b.l < 0.f) ? -1.f : 1.f;
  return (sa * a.h - sb * b.h) + (sa * a.l - sb * b.l) < 0.f;
}
FFD bool ff_gt(ff a, ff b) { return (a.h - b.h) + (a.l - b.l) > 0.f; }

// ------------------------------------------------------------------------ FP64 <-> pairs
// x 2^k as a pair by moving bits (a conversion instruction would cost as much as an FP64 add): the
// high part is x cut to 24 bits, the low part the other 29 bits rounded to 24 (2^-49 of x).
// |x 2^k| below 2^-70 gives 0; the caller keeps |x 2^k| below 2^100.  k20 = k << 20.
FFD ff ff_of(double x, int k20 = 0)
{
  const uint64_t b = d_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
  const uint32_t mag = (hi & 0x7fffffffu) + (uint32_t)k20;  // exponent field moved
  const uint32_t f = (mag << 3) | (lo >> 29);               // its low 8 bits | 23 bits of mantissa
  const bool ok = (int32_t)mag >= ((1023 - 70) << 20);
  // field - 896 = field + 128 modulo 256
  const uint32_t h = ok ? (((f ^ 0x40000000u) & 0x7fffffffu) | (hi & 0x80000000u)) : 0u;
  const float ulp52 = bits_f((h & 0xff800000u) - (52u << 23));  // sign x 2^(exponent - 52)
  ff r;
  r.h = bits_f(h);
#ifdef __CUDA_ARCH__
  const float m = __uint2float_rn(lo & 0x1fffffffu);
#else
  const float m = (float)(lo & 0x1fffffffu);
#endif
  r.l = ok ? m * ulp52 : 0.f;
  return r;
}
// (h + l) 2^k as a double for a normalised pair, rounded to nearest, without an FP64 instruction: the
// high part's bits, and the low part as a whole number of the high part's FP64 ulps added to them as
// a 64-bit integer.  Where h is a power of two and l takes the sum below it an ulp is half as large.
// |h| below 2^-75 is converted without l, 0 and subnormal h give 0.  For finite pairs: an infinite or
// NaN h would come out as a number near 2^128, so the element pass looks at its inputs' ranges first.
FFD double f64_of(ff a, int k20 = 0)
{
  const uint32_t b = f_bits(a.h), sign = b & 0x80000000u;
  const uint32_t ex = (b >> 23) & 255u;
  const uint32_t hi = (uint32_t)((((int32_t)b >> 3) & (int32_t)0x8fffffff) + (896 << 20) + k20);
  const bool below = (b & 0x7fffffu) == 0u && ((f_bits(a.l) ^ b) & 0x80000000u);
  const uint32_t f = (306u + (below ? 1u : 0u)) - ex;  // field of 2^(52 - exponent)
  const float t = ex < 53u ? 0.f : a.l * bits_f((f << 23) | sign);
#ifdef __CUDA_ARCH__
  const int n = __float2int_rn(t);
#else
  const int n = (int)rintf(t);
#endif
  const uint64_t m = (((uint64_t)hi << 32) | (uint64_t)(b << 29)) + (uint64_t)(int64_t)n;
  return bits_d(ex != 0u ? m : 0ull);
}
// x + a 2^k with x FP64: the pass's sums into stored state, one FP64 addition each
FFD double f64_add(double x, ff a, int k20 = 0) { return x + f64_of(a, k20); }
// high word of |x| (orders like |x|): for range checks without FP64 compares
FFD uint32_t f64_mag(double x) { return (uint32_t)(d_bits(x) >> 32) & 0x7fffffffu; }
FFD uint32_t f64_mag_at(const double *x) { return reinterpret_cast<const uint32_t *>(x)[1] & 0x7fffffffu; }  // that word alone

// ------------------------------------------------------------------------ grid accumulation
// C = 1.5 2^k with 2^(k-1) the power of two at or above bound (finite, >= 0)
FFD float grid_of(float bound)
{
  return bits_f(((f_bits(bound) + 0x7fffffu) & 0x7f800000u) + 0x00c00000u);
}
struct Acc {
  float s, e;
  FFD explicit Acc(float C) : s(C), e(0.f) {}
  FFD void mac(ff a, ff b)
  {
    const float s1 = f_fma(a.h, b.h, s);
    const float t = s1 - s;
    const float r = f_fma(a.h, b.h, -t);
    e = f_fma(a.l, b.h, f_fma(a.h, b.l, e + r));
    s = s1;
  }
  FFD void macf(ff a, float b)
  {
    const float s1 = f_fma(a.h, b, s);
    const float t = s1 - s;
    const float r = f_fma(a.h, b, -t);
    e = f_fma(a.l, b, e + r);
    s = s1;
  }
  FFD void add(ff a)
  {
    const float s1 = s + a.h;
    const float r = a.h - (s1 - s);
    e = (e + r) + a.l;
    s = s1;
  }
  FFD void addf(float a) { e += a; }  // |a| of the grid's order or below it
  FFD ff raw(float C) const { return ff{s - C, e}; }
  FFD ff get(float C) const { return ff_norm(s - C, e); }
};

// The same without a bound: product errors by fma, Knuth's sums (the Dot2 of Ogita, Rump and Oishi,
// with the cross terms of the pairs): 12 instructions per term, error 2^-48 of the largest partial sum.
// For the terms whose relative precision the nodal forces, sums that cancel, depend on.
struct Dot {
  float s, e;
  FFD Dot(ff a, ff b)
  {
    s = a.h * b.h;
    e = f_fma(a.l, b.h, f_fma(a.h, b.l, f_fma(a.h, b.h, -s)));
  }
  FFD void mac(ff a, ff b)
  {
    const float p = a.h * b.h;
    const float pe = f_fma(a.h, b.h, -p);
    const ff t = two_sum(s, p);
    s = t.h;
    e = f_fma(a.l, b.h, f_fma(a.h, b.l, (e + t.l) + pe));
  }
  FFD ff get() const { return ff_norm(s, e); }
};
// a + b without the final normalisation: for a few sums in a row
FFD ff ff_add_raw(ff a, ff b)
{
  const ff t = two_sum(a.h, b.h);
  return ff{t.h, t.l + (a.l + b.l)};
}

// a constant as a pair
FFD constexpr ff ff_host(double x)
{
  return ff{(float)x, (float)(x - (double)(float)x)};
}

// 1 + s^2/3 + s^4/5 + ... to s^18 for |s| <= 0.18: atanh(s) / s.  Leading terms as pairs.
FFD ff atanh_series_ff(ff s)
{
  const ff one = {1.f, 0.f};
  const ff u = ff_mul(s, s);
  const float v = u.h;
  const float f = f_fma(v, f_fma(v, f_fma(v, f_fma(v, f_fma(v, 1.f / 19.f, 1.f / 17.f), 1.f / 15.f), 1.f / 13.f), 1.f / 11.f), 1.f / 9.f);
  ff p = ff_add(ff_host(1. / 7.), ff_mulf(u, f));
  p = ff_add(ff_host(1. / 5.), ff_mul(u, p));
  p = ff_add(ff_host(1. / 3.), ff_mul(u, p));
  return ff_add(one, ff_mul(u, p));
}
// ln(1 + x)/2 for -1/2 <= x <= 1, to 2^-45 of itself: ln r with r = sqrt(1 + x) from 1/sqrt 2 to sqrt 2, which is
// 2 atanh(s), s = (r - 1)/(r + 1) = x / (1 + r)^2 within 0.172 (without the root s reaches 1/3, past the series)
FFD ff half_log1p_ff(ff x)
{
  const ff y = ff_add(ff{1.f, 0.f}, x);
  const ff d = ff_add(ff{1.f, 0.f}, ff_sqrt(y, f_rsqrt(y.h)));
  const ff s = ff_mul(x, ff_rcp(ff_mul(d, d)));
  return ff_scale(ff_mul(s, atanh_series_ff(s)), 2.f);
}
// (ln(1 + a) - ln(1 + b)) / (2 (a - b)), 1 / (2 (1 + a)) in the limit, |a|, |b| <= 0.4: with w = 2 + a + b and
// u = (a - b) / w it is atanh(u) / (u w), no difference of logarithms; where u is beyond the series the
// logarithms are apart enough to be subtracted
FFD ff half_log_slope_ff(ff a, ff b)
{
  const ff d = ff_sub(a, b), rw = ff_rcp(ff_add(ff{2.f, 0.f}, ff_add(a, b)));
  const ff u = ff_mul(d, rw);
  if (f_abs(u.h) <= 0.17f) return ff_mul(atanh_series_ff(u), rw);
  return ff_mul(ff_sub(half_log1p_ff(a), half_log1p_ff(b)), ff_rcp(d));
}
// (1 + x)^(-1/2) - 1 for -1/2 <= x <= 1, to 2^-45 of itself
FFD ff rsqrt1p_ff(ff x)
{
  const ff y = ff_add(ff{1.f, 0.f}, x);
  return ff_neg(ff_mul(x, ff_rcp(ff_add(y, ff_sqrt(y, f_rsqrt(y.h))))));
}

// ------------------------------------------------------------------------ kinematics
// G = G_u J^-1 by the adjugate: adj(J) and det(J) too; mJ: largest entry of each column of J, cols: their
// product, against which a badly shaped element's |det J| is small: its differences of products cancel.
template <int DIM>
FFD void deform_ff(const ff (&J)[DIM][DIM], const ff (&GU)[DIM][DIM], const float (&mJ)[DIM],
                   ff (&adj)[DIM][DIM], ff &det, ff &rdet, ff (&G)[3][3], float &cols)
{
  if constexpr (DIM == 2) {
    adj[0][0] = J[1][1];
    adj[0][1] = ff_neg(J[0][1]);
    adj[1][0] = ff_neg(J[1][0]);
    adj[1][1] = J[0][0];
    det = ff_sub(ff_mul(J[0][0], J[1][1]), ff_mul(J[0][1], J[1][0]));
    cols = mJ[0] * mJ[1];
  } else {
#pragma unroll
    for (int l = 0; l < 3; l++) {
      const int p = (l + 1) % 3, q = (l + 2) % 3;  // row l of the adjugate: columns p x q
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int u = (c + 1) % 3, v = (c + 2) % 3;
        adj[l][c] = ff_sub(ff_mul(J[u][p], J[v][q]), ff_mul(J[v][p], J[u][q]));
      }
    }
    Dot s(J[0][0], adj[0][0]);
#pragma unroll
    for (int r = 1; r < 3; r++) s.mac(J[r][0], adj[0][r]);
    det = s.get();
    cols = mJ[0] * mJ[1] * mJ[2];
  }
  rdet = ff_rcp(det);
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (r >= DIM || c >= DIM) {
        G[r][c] = ff{0.f, 0.f};
        continue;
      }
      Dot s(GU[r][0], adj[0][c]);
#pragma unroll
      for (int l = 1; l < DIM; l++) s.mac(GU[r][l], adj[l][c]);
      G[r][c] = ff_mul(s.get(), rdet);
    }
}

// ------------------------------------------------------------------------ polar decomposition
// Limit of |F - I|'s entries for the pair arithmetic (2^-7.75): the errors of S and evp, the first to cross
// FP64's, are the same there (uniaxial increments, pairs over FP64: S 0.8 (solids) to 1.4 (plane) at 2^-7.5,
// 1.3 to 2.3 at 2^-7; evp of all kinds of increments 0.7 to 0.9 at 2^-8, 1.0 to 1.2 at 2^-7.5).  For distorted elements
// G = G_u J^-1 carries the pairs' error times the products' cancellation, so the limit falls with the ratio
// of the product of J's columns to det J: from kShapeMax on, a hexahedron with columns sheared by 2 crosses
// FP64 at 2^-8.2, by 3 at 2^-9.0, by 4 at 2^-9.7, its ratio being 1.2, 2.3 and 3.9 times kShapeMax.
constexpr float kFastMax = 0x1.3p-8f;
constexpr float kShapeMax = 1.8f;

// symmetric component order of the six-entry arrays: xx yy zz xy xz yz
FFD constexpr int sym_i(int k) { return k < 3 ? k : (k == 5 ? 1 : 0); }
FFD constexpr int sym_j(int k) { return k < 3 ? k : (k == 3 ? 1 : 2); }
FFD constexpr int sym_of(int i, int j) { return i == j ? i : (i + j == 1 ? 3 : (i + j == 2 ? 4 : 5)); }

template <bool TWO_D>
FFD float max_sym(const ff (&A)[6])
{
  float m = f_max(f_abs(A[0].h), f_max(f_abs(A[1].h), f_abs(A[2].h)));
  m = f_max(m, f_abs(A[3].h));
  if (!TWO_D) m = f_max(m, f_max(f_abs(A[4].h), f_abs(A[5].h)));
  return m;
}
// out = A B of commuting symmetric matrices
template <bool TWO_D>
FFD void mul_sym(const ff (&A)[6], const ff (&B)[6], float C, ff (&out)[6])
{
#pragma unroll
  for (int k = 0; k < (TWO_D ? 4 : 6); k++) {
    const int i = sym_i(k), j = sym_j(k);
    Acc s(C);
#pragma unroll
    for (int m = 0; m < 3; m++) {
      if (TWO_D && ((m == 2) != (i == 2))) continue;  // 2 + 1 blocks
      s.mac(A[sym_of(i, m)], B[sym_of(m, j)]);
    }
    out[k] = s.get(C);
  }
  if (TWO_D) out[4] = out[5] = ff{0.f, 0.f};
}

// E = C - I = G + G^T + G^T G and mg = max |G|
template <bool TWO_D>
FFD float green_ff(const ff (&G)[3][3], ff (&E)[6])
{
  float mg = 0.f;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (!TWO_D || (i == 2) == (j == 2)) mg = f_max(mg, f_abs(G[i][j].h));
  const float C = grid_of(3.f * mg * mg);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int i = sym_i(k), j = sym_j(k);
    if (TWO_D && k > 3) {
      E[k] = ff{0.f, 0.f};
      continue;
    }
    Acc s(C);
#pragma unroll
    for (int m = 0; m < 3; m++) {
      if (TWO_D && ((m == 2) != (i == 2))) continue;
      s.mac(G[m][i], G[m][j]);
    }
    E[k] = ff_add(i == j ? ff_scale(G[i][i], 2.f) : ff_add(G[i][j], G[j][i]), s.get(C));
  }
  return mg;
}

// Whether the two largest off-diagonal entries of E, above tol, are within 2^-36 of its scale of
// each other: the pairs' own error could then choose the first pivot.
FFD bool pivot_tie(const ff (&E)[6], float mg, float tol)
{
  auto mag = [](ff a) { return a.h < 0.f ? ff_neg(a) : a; };
  const ff a = mag(E[3]), b = mag(E[4]), c = mag(E[5]);
  const float top = f_max(a.h, f_max(b.h, c.h)), eps = 0x1p-36f * mg;
  auto near = [top, eps](ff x, ff y) {
    return f_abs((x.h - y.h) + (x.l - y.l)) <= eps && top - f_max(x.h, y.h) <= 2.f * eps;
  };
  return top >= 0.5f * tol && (near(a, b) || near(a, c) || near(b, c));
}

// From G = F - I (|G| <= kFastMax): L = ln U and Q = R - I with the eigen-iteration of
// Tensor2::polarDecomposeLnU (Tensor2.C:1154-1259): its pivots, its stop at |C_pq| < tol and its
// rotations, on E = C - I = G + G^T + G^T G.
//
// The reference forms ln U from the rotated diagonal and the rotations alone, dropping what is left
// off the diagonal (below tol): with C = V (Lambda + r) V^T its result is the logarithm of
// V Lambda V^T = I + E', E' = E - V r V^T.  Here E' is formed from E directly -- r is below 1e-9, so
// V r V^T needs V in single precision only, and a rotation of V is 12 FP32 instructions -- and
// ln U = ln(I + E')/2, U^-1 = (I + E')^(-1/2) are the power series in E': E' and E'^2 as pairs, the
// next powers where |E'| needs them, and the remainder, below 2^-30 of 1, through the single-precision
// eigenpairs.
// KEEP: V as pairs, the rotated diagonal and U^-1 - I too (the sensitivities' record).
// E, mg: from green_ff (E is changed); first: the first rotation's pivot where the caller decided it
// (pivot_tie), else -1.  Returns false when the iteration reaches cap rotations without meeting tol.
template <bool TWO_D, bool KEEP>
FFD bool strain_ff(const ff (&G)[3][3], ff (&E)[6], float mg, ff tol, int cap, int first, ff (&L)[6],
                   ff (&Q)[3][3], ff (*Vk)[3] = nullptr, ff *lam = nullptr, ff *Hk = nullptr)
{
  // the rotated entries stay below E's Frobenius norm: high parts on the grid of that bound, so
  // such pairs add and subtract term by term
  float C;
  {
    const float off = f_fma(E[3].h, E[3].h, f_fma(E[4].h, E[4].h, E[5].h * E[5].h));
    const float n2 = f_fma(E[0].h, E[0].h, f_fma(E[1].h, E[1].h, f_fma(E[2].h, E[2].h, 2.f * off)));
    C = grid_of(n2 * f_rsqrt(f_max(n2, 0x1p-120f)) * 1.0001f);
  }
  auto on_grid = [C](ff a) {
    Acc s(C);
    s.add(a);
    return s.raw(C);
  };
  ff f00 = on_grid(E[0]), f11 = on_grid(E[1]), f22 = on_grid(E[2]), f01 = on_grid(E[3]);
  ff f02 = TWO_D ? E[4] : on_grid(E[4]), f12 = TWO_D ? E[5] : on_grid(E[5]);
  float V[3][3] = {{1.f, 0.f, 0.f}, {0.f, 1.f, 0.f}, {0.f, 0.f, 1.f}};
  if (KEEP) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) Vk[i][j] = ff{i == j ? 1.f : 0.f, 0.f};
  }
  bool conv = false, rotated = false;
  for (int it = 1; it <= cap; it++) {
    // pivot of Tensor2.C:1173-1178: q = |C01| > |C02| ? 1 : 2, p = |C0q| > |C12| ? 0 : 1
    int k = 0;
    ff x = f01;
    if (!TWO_D) {
      const bool q1 = ff_abs_lt(f02, f01);
      const ff f0q = q1 ? f01 : f02;
      const bool p0 = ff_abs_lt(f12, f0q);
      k = it == 1 && first >= 0 ? first : (p0 ? (q1 ? 0 : 1) : 2);
      x = k == 0 ? f01 : (k == 1 ? f02 : f12);
    }
    if (ff_abs_lt(x, tol)) {
      conv = true;
      break;
    }
    rotated = true;
    const ff a = k == 2 ? f11 : f00, b = k == 0 ? f11 : f22;
    // the rotation angle by half-angle identities: w = 1 / sqrt(d^2 + (2x)^2), c^2 = (1 + |d| w) / 2,
    // s = |x| w / c, t = s / c, their sign that of d x (positive when d = 0)
    const ff d = ff_norm(b.h - a.h, b.l - a.l), xn = ff_norm(x.h, x.l), x2 = ff_scale(xn, 2.f);
    const ff dd = ff_mul(d, d), xx = ff_mul(x2, x2);
    const ff q = ff_add(dd, xx);
    const ff w = ff_rsqrt(q);
    const ff dw = ff_mul(d, w);
    const float hw = 0.5f * f_abs(dw.h), lw = d.h < 0.f ? -0.5f * dw.l : 0.5f * dw.l;
    const ff h = ff_norm(0.5f, hw);
    const ff c2 = ff_norm(h.h, h.l + lw);
    const ff rc = ff_rsqrt(c2);
    const ff c = ff_mul(c2, rc);
    const ff wr = ff_mul(w, rc);
    ff s = ff_mul(xn, wr);  // signed by x
    const bool flip = d.h < 0.f;  // sign(d x); d = 0: |s|
    if (flip || (d.h == 0.f && s.h < 0.f)) s = ff_neg(s);
    const ff t = ff_mul(s, rc);
    // a' = a - t x, b' = b + t x, y' = c y - s z, z' = s y + c z on the grid of C
    {
      const float p1 = f_fma(t.h, xn.h, C), p = p1 - C;
      const float r = f_fma(t.l, xn.h, f_fma(t.h, xn.l, f_fma(t.h, xn.h, -p)));
      const ff a2 = ff{a.h - p, a.l - r}, b2 = ff{b.h + p, b.l + r}, zero = ff{0.f, 0.f};
      if (TWO_D) {
        f00 = a2;
        f11 = b2;
        f01 = zero;
      } else {
        const ff y = k == 0 ? f02 : f01, z = k == 2 ? f02 : f12;
        Acc u(C), v(C);
        u.mac(c, y);
        u.mac(ff_neg(s), z);
        v.mac(s, y);
        v.mac(c, z);
        const ff y2 = u.raw(C), z2 = v.raw(C);
        f00 = k == 2 ? f00 : a2;
        f11 = k == 0 ? b2 : (k == 2 ? a2 : f11);
        f22 = k == 0 ? f22 : b2;
        f01 = k == 0 ? zero : y2;
        f02 = k == 0 ? y2 : (k == 1 ? zero : z2);
        f12 = k == 2 ? zero : z2;
      }
    }
#pragma unroll
    for (int i = 0; i < (TWO_D ? 2 : 3); i++) {
      const float rp = k == 2 ? V[i][1] : V[i][0], rq = k == 0 ? V[i][1] : V[i][2];
      const float np = f_fma(rp, c.h, -(rq * s.h)), nq = f_fma(rp, s.h, rq * c.h);
      V[i][0] = k == 2 ? V[i][0] : np;
      V[i][1] = k == 0 ? nq : (k == 2 ? np : V[i][1]);
      V[i][2] = k == 0 ? V[i][2] : nq;
      if (KEEP) {
        const ff kp = k == 2 ? Vk[i][1] : Vk[i][0], kq = k == 0 ? Vk[i][1] : Vk[i][2];
        Acc u(3.f), v(3.f);
        u.mac(kp, c);
        u.mac(ff_neg(kq), s);
        v.mac(kp, s);
        v.mac(kq, c);
        const ff kp2 = u.get(3.f), kq2 = v.get(3.f);
        Vk[i][0] = k == 2 ? Vk[i][0] : kp2;
        Vk[i][1] = k == 0 ? kq2 : (k == 2 ? kp2 : Vk[i][1]);
        Vk[i][2] = k == 0 ? Vk[i][2] : kq2;
      }
    }
  }
  if (KEEP) {
    lam[0] = ff_norm(f00.h, f00.l);
    lam[1] = ff_norm(f11.h, f11.l);
    lam[2] = ff_norm(f22.h, f22.l);
  }
  ff H[6];
  // E' = E - V r V^T; without a rotation V = I and E' is E's diagonal
  {
    const float r01 = f01.h + f01.l, r02 = f02.h + f02.l, r12 = f12.h + f12.l;
#pragma unroll
    for (int k = 0; k < (TWO_D ? 4 : 6); k++) {
      const int i = sym_i(k), j = sym_j(k);
      float K = 0.f;
      if (!TWO_D || k != 2) {
        K = r01 * f_fma(V[i][0], V[j][1], V[i][1] * V[j][0]);
        if (!TWO_D) {
          K = f_fma(r02, f_fma(V[i][0], V[j][2], V[i][2] * V[j][0]), K);
          K = f_fma(r12, f_fma(V[i][1], V[j][2], V[i][2] * V[j][1]), K);
        }
      }
      const ff e = ff_norm(E[k].h, E[k].l - K);
      E[k] = rotated || i == j ? e : ff{0.f, 0.f};
    }
  }
  const float me = max_sym<TWO_D>(E);
  constexpr int DN = TWO_D ? 2 : 3;
  const float C2 = grid_of(DN * me * me);
  ff S2[6];
  mul_sym<TWO_D>(E, E, C2, S2);
  // remainders of ln(1 + x)/2 and (1 + x)^(-1/2) per eigenvalue, to matrices through V: from x^3 on
  // (level 0, |x| <= 2^-10), x^5 (level 1, 2^-6) or x^8 (level 2).  The lines lie where the remainder's
  // rounding in single precision (2^-24 of x^3/6, x^5/10) is 2^-56 at most.  By the eigenvalues: they reach
  // three times the entries, and with the entries' size the error was 9e-17 at |G| = 2^-11 and 6e-16
  // at 2^-7 (root mean square of ln U, FP64 6e-17), now 8e-18 and 5e-17.
  const float ev[3] = {f00.h + f00.l, f11.h + f11.l, f22.h + f22.l};
  const float mv = f_max(f_abs(ev[0]), f_max(f_abs(ev[1]), f_abs(ev[2])));
  const int level = mv <= 0x1p-10f ? 0 : (mv <= 0x1p-6f ? 1 : 2);
  float gl[3], gh[3];
#pragma unroll
  for (int m = 0; m < 3; m++) {
    const float x = ev[m], x3 = x * x * x;
    float l, h;
    if (level == 2) {  // to x^15; the next is below 2^-60
      l = f_fma(x, f_fma(x, f_fma(x, 1.f / 30.f, -1.f / 28.f), 1.f / 26.f), -1.f / 24.f);
      l = f_fma(x, f_fma(x, f_fma(x, f_fma(x, l, 1.f / 22.f), -1.f / 20.f), 1.f / 18.f), -1.f / 16.f);
      h = f_fma(x, f_fma(x, f_fma(x, -0.14446444809436798f, 0.14944598078727722f), -0.15498101711273193f), 0.16118025779724121f);
      h = f_fma(x, f_fma(x, f_fma(x, f_fma(x, h, -88179.f / 524288.f), 46189.f / 262144.f), -12155.f / 65536.f), 6435.f / 32768.f);
      const float x8 = x3 * x3 * x * x;
      gl[m] = x8 * l;
      gh[m] = x8 * h;
    } else {
      l = f_fma(x, f_fma(x, f_fma(x, 1.f / 18.f, -1.f / 16.f), 1.f / 14.f), -1.f / 12.f);
      h = f_fma(x, f_fma(x, f_fma(x, -12155.f / 65536.f, 6435.f / 32768.f), -429.f / 2048.f), 231.f / 1024.f);
      l = f_fma(x, l, 0.1f);
      h = f_fma(x, h, -63.f / 256.f);
      gl[m] = x3 * (level == 0 ? f_fma(x, f_fma(x, l, -0.125f), 1.f / 6.f) : x * x * l);
      gh[m] = x3 * (level == 0 ? f_fma(x, f_fma(x, h, 35.f / 128.f), -5.f / 16.f) : x * x * h);
    }
  }
  // P, R: the parts of fourth and higher order (ln and inverse root) that are formed as pairs
  ff S3[6], P[6], R[6];
  if (level > 0) {
    ff S4[6];
    const float m4 = DN * DN * DN * me * me * me * me;
    mul_sym<TWO_D>(E, S2, grid_of(DN * DN * me * me * me), S3);
    mul_sym<TWO_D>(S2, S2, grid_of(m4), S4);
    if (level == 1) {
#pragma unroll
      for (int k = 0; k < 6; k++) {
        P[k] = ff_scale(S4[k], -0.125f);
        R[k] = ff_mulf(S4[k], 35.f / 128.f);
      }
    } else {  // E'^4 (c4 + c5 E' + c6 E'^2 + c7 E'^3)
      ff A[6], B[6];
#pragma unroll
      for (int k = 0; k < 6; k++) {
        if (TWO_D && k > 3) {
          A[k] = B[k] = ff{0.f, 0.f};
          continue;
        }
        Acc a(1.5f), b(1.5f);
        a.macf(E[k], 0.1f);
        a.macf(S2[k], -1.f / 12.f);
        a.macf(S3[k], 1.f / 14.f);
        b.macf(E[k], -63.f / 256.f);
        b.macf(S2[k], 231.f / 1024.f);
        b.macf(S3[k], -429.f / 2048.f);
        if (k < 3) {
          a.add(ff{-0.125f, 0.f});
          b.add(ff{35.f / 128.f, 0.f});
        }
        A[k] = a.get(1.5f);
        B[k] = b.get(1.5f);
      }
      mul_sym<TWO_D>(S4, A, grid_of(0.5f * m4), P);
      mul_sym<TWO_D>(S4, B, grid_of(m4), R);
    }
  }
  // the first-order parts by sums of pairs, the rest on the grid of its own size
  const float CL = grid_of(0.625f * DN * me * me);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int i = sym_i(k), j = sym_j(k);
    if (TWO_D && k > 3) {
      L[k] = H[k] = ff{0.f, 0.f};
      continue;
    }
    float rl = 0.f, rh = 0.f;
#pragma unroll
    for (int m = 0; m < 3; m++) {
      if (TWO_D && ((m == 2) != (i == 2))) continue;
      const float vv = V[i][m] * V[j][m];
      rl = f_fma(vv, gl[m], rl);
      rh = f_fma(vv, gh[m], rh);
    }
    Acc sl(CL), sh(CL);
    sl.add(ff_scale(S2[k], -0.25f));
    sh.macf(S2[k], 0.375f);
    if (level > 0) {
      sl.mac(S3[k], ff{1.f / 6.f, (float)(1. / 6. - (double)(1.f / 6.f))});
      sl.add(P[k]);
      sh.macf(S3[k], -0.3125f);
      sh.add(R[k]);
    }
    sl.addf(rl);
    sh.addf(rh);
    const ff e2 = ff_scale(E[k], 0.5f);
    L[k] = ff_add(e2, sl.get(CL));
    H[k] = ff_sub(sh.get(CL), e2);
  }
  if (KEEP) {
#pragma unroll
    for (int k = 0; k < 6; k++) Hk[k] = H[k];
  }
  // Q = R - I = (I + G)(I + H) - I
  const float CQ = grid_of(0.75f * (TWO_D ? 2 : 3) * mg * me);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      if (TWO_D && (i == 2) != (j == 2)) {
        Q[i][j] = ff{0.f, 0.f};
        continue;
      }
      Acc s(CQ);
#pragma unroll
      for (int m = 0; m < 3; m++) {
        if (TWO_D && ((m == 2) != (i == 2))) continue;
        s.mac(G[i][m], H[sym_of(m, j)]);
      }
      Q[i][j] = ff_add(ff_add(G[i][j], H[sym_of(i, j)]), s.get(CQ));
    }
  return conv;
}

// R X R^T - X for symmetric X with Q = R - I: Y + Y^T + Y Q^T, Y = Q X
template <bool TWO_D>
FFD void rfi_ff(const ff (&Q)[3][3], float mq, const ff (&X)[6], ff (&D)[6])
{
  const float mx = max_sym<TWO_D>(X);
  constexpr float DN = TWO_D ? 2.f : 3.f;
  const float CY = grid_of(DN * mq * mx), CD = grid_of(2.f * DN * mq * mx * (1.f + DN * mq));
  ff Y[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      if (TWO_D && (i == 2) != (j == 2)) continue;
      Acc s(CY);
#pragma unroll
      for (int m = 0; m < 3; m++) {
        if (TWO_D && ((m == 2) != (i == 2))) continue;
        s.mac(Q[i][m], X[sym_of(m, j)]);
      }
      Y[i][j] = s.get(CY);
    }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int i = sym_i(k), j = sym_j(k);
    if (TWO_D && k > 3) {
      D[k] = ff{0.f, 0.f};
      continue;
    }
    Acc s(CD);
    if (i == j) {
      s.add(ff_scale(Y[i][i], 2.f));
    } else {
      s.add(Y[i][j]);
      s.add(Y[j][i]);
    }
#pragma unroll
    for (int m = 0; m < 3; m++) {
      if (TWO_D && ((m == 2) != (i == 2))) continue;
      s.mac(Y[i][m], Q[j][m]);
    }
    D[k] = s.get(CD);
  }
}

// ------------------------------------------------------------------------ radial return
// A material's constants for the pair arithmetic.  Stresses are carried as multiples of 2^k, the
// power of two at or below 2 G (k20 = k << 20).
struct MatFF {
  int k20;
  int ok;                        // constants finite and within the pairs' range (else FP64 only)
  ff g2, A, B, K, rG3, dfun0;    // 2 G, A, B, K, sqrt(3/2) 2 G over 2^k; 2^k / (3 G)
  ff n, c2, c3;                  // n; (n - 1)/2, (n - 2)/3: ratios of the binomial series' terms
  float c4, c5, c6, c7, c8;
  float n3;                      // what the pair n leaves of the exponent
  ff rhoCs4;                     // rho c / 4 over 2^k (the one-point hexahedron's hourglass viscosity)
  int okHg;                      // rho c is 0 or within 2^-40 .. 2^40 of 2^k
};

inline MatFF make_mat_ff(double G2, double G3, double K, double A, double B, double n, double dfun0,
                         double rhoCs)
{
  MatFF m;
  // with evp^n below 2^30 and its growth below 2^58 the products stay below 2^120
  auto in_range = [G2](double x) { return x == 0. || (fabs(x) < 0x1p30 * G2 && fabs(x) > 0x1p-60 * G2); };
  m.ok = G2 > 0x1p-400 && G2 < 0x1p400 && in_range(G3) && in_range(K) && in_range(A) && in_range(B) && fabs(n) < 64.;
  int k = 0;
  frexp(m.ok ? G2 : 1., &k);
  k -= 1;  // 2^k <= G2 < 2^(k+1)
  const double s = ldexp(1.0, -k);
  m.k20 = k * (1 << 20);
  m.g2 = ff_host(G2 * s);
  m.A = ff_host(A * s);
  m.B = ff_host(B * s);
  m.K = ff_host(K * s);
  m.rG3 = ff_host(1.0 / (G3 * s));
  m.dfun0 = ff_host(dfun0 * s);
  m.n = ff_host(n);
  m.n3 = (float)(n - (double)m.n.h - (double)m.n.l);
  m.c2 = ff_host((n - 1.) / 2.);
  m.c3 = ff_host((n - 2.) / 3.);
  m.c4 = (float)((n - 3.) / 4.);
  m.c5 = (float)((n - 4.) / 5.);
  m.c6 = (float)((n - 5.) / 6.);
  m.c7 = (float)((n - 6.) / 7.);
  m.c8 = (float)((n - 7.) / 8.);
  m.rhoCs4 = ff_host(0.25 * rhoCs * s);
  m.okHg = rhoCs == 0. || (rhoCs * s >= 0x1p-40 && rhoCs * s <= 0x1p40);
  return m;
}

// (1 + q)^n - 1, n = n + n3, for q >= 0 with n log2(1 + q) below 60: 1 + q = 2^e z, z in [1/sqrt 2, sqrt 2];
// log2 z from s = (z - 1)/(z + 1) by the area tangent's series, 2 s (1 + s^2/3 + ...) / ln 2 to s^19;
// the power's integer part to the exponent, the rest by the exponential's series on an eighth of it
// and three squarings of 1 + t.  The leading terms as pairs, what is below 2^-24 of them in single
// precision.
FFD ff powq_ff(ff n, float n3, ff q)
{
  const ff one = {1.f, 0.f};
  const ff x = ff_add(one, q);
  const int e = (int)((f_bits(x.h) + 0x004afb0du) >> 23) - 127;  // 0x1.6a09e6p0 and above: one more
  const ff z = ff_scale(x, bits_f((uint32_t)(127 - e) << 23));
  const ff s = ff_mul(ff_sub(z, one), ff_rcp(ff_add(z, one)));
  const ff p = atanh_series_ff(s);
  const ff lg = ff_mul(ff_mul(s, p), ff_host(2.8853900817779268147));  // 2 / ln 2
  // n (e + lg) minus its nearest integer k, n e exactly (n to 72 bits)
  const float E = (float)e, ne = n.h * E;
  const float k = rintf(f_fma(n.h, lg.h, ne));
  const ff fe = two_sum(ne, -k);
  const float nl = n.l * E;
  const ff fl = two_sum(f_fma(n.h, E, -ne), nl);
  const ff fs = two_sum(fe.h, fl.h);
  const ff y = ff_add(ff_mul(n, lg), ff_norm(fs.h, fs.l + (fe.l + (fl.l + f_fma(n3, E, f_fma(n.l, E, -nl))))));
  const ff r = ff_mul(y, ff_host(0.6931471805599453094 / 8.));
  const float w = r.h;
  const float g = f_fma(w, f_fma(w, f_fma(w, f_fma(w, 1.f / 362880.f, 1.f / 40320.f), 1.f / 5040.f), 1.f / 720.f), 1.f / 120.f);
  ff t = ff_add(ff_host(1. / 24.), ff_mulf(r, g));
  t = ff_add(ff_host(1. / 6.), ff_mul(r, t));
  t = ff_add(ff{0.5f, 0.f}, ff_mul(r, t));
  t = ff_add(r, ff_mul(ff_mul(r, r), t));
#pragma unroll
  for (int i = 0; i < 3; i++) t = ff_add(ff_scale(t, 2.f), ff_mul(t, t));
  const float p2 = bits_f((uint32_t)((int)k + 127) << 23);
  return ff_add(ff_add(ff_scale(t, p2), ff{p2, 0.f}), ff{-1.f, 0.f});
}

// (1 + q)^n - 1 for 0 <= q <= 2^-6, |n| <= 2: the binomial series to q^8, its terms' factors from the
// fourth on in single precision (below 2^-24 of the result's scale)
FFD ff pow1p_ff(const MatFF &m, ff q)
{
  const float x = q.h;
  const float f = m.c4 * x * f_fma(m.c5 * x, f_fma(m.c6 * x, f_fma(m.c7 * x, f_fma(m.c8, x, 1.f), 1.f), 1.f), 1.f);
  ff u = ff_mul(ff_mul(m.c3, q), ff_norm(1.f, f));
  u = ff_add(ff{1.f, 0.f}, u);
  u = ff_mul(ff_mul(m.c2, q), u);
  u = ff_add(ff{1.f, 0.f}, u);
  return ff_mul(ff_mul(m.n, q), u);
}

}  // namespace dnl
