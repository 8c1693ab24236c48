// sw_f64.cuh -- the regularized-BGK collision of float64 storage in 64-bit fixed point.
//
// GB300 retires 2 double-precision operations per clock and SM (measured, add,
// multiply, fused multiply-add and the conversions from and to 64-bit integers
// alike) against 64 integer ones: the collision's 206 double operations take
// 3300 clocks per warp, seven times what its 304 bytes per cell take at the
// measured HBM rate.  So the cell's tensors are held as 64-bit integers in
// units of 2^-62 and only the scalar functions stay in double: 1 / rho and
// 1 / tau (three operations each), the two square roots of the Smagorinsky time
// scale (five each), three products and sums and the sponge's four, 23 per cell
// beside about 500 integer ones, which run on other pipes.
//
//  * A population in [2^-10, its limit below 1/2) is a whole number of units, so
//    the conversion is exact, and so are rho, m and Pi: sums of 19 exact terms,
//    below 2 in magnitude.  (In double each partial sum rounds at 2^-53.)
//  * Products take the upper 64 bits of the 128-bit product without the term of
//    the two lower halves: within 3 units.
//  * With T = tr B the regularized write (see collide in sw_step.cuh) is
//      f_0 = 12 A,  f_axis = 2 A + B_aa / 4 +- m_a / 6,
//      f_edge = A + (B_aa + B_bb) / 8 +- B_ab / 4 +- (m_a +- m_b) / 12,
//      A = rho / 36 - T / 24,
//    additions, shifts and four multiplications by constants.
//  * The results are rounded to double once, at the end.
// Cells with a population outside its range (also negative ones, infinities and
// NaN), rho outside (1/2, 2), 1 / tau outside [1/4, 2] or a result outside
// [2^-10, 1) report so and the caller collides them in double.
//
// Error of one collision against 128-bit floats on the same inputs (25 kinds of
// 20 000 cells, |u_a| up to 0.25, |Pi_neq| up to 3e-2): 4.6e-17 to 5.5e-17 of the
// populations' norm, the rounding of the results included, against 1.4e-16 to
// 1.6e-16 in double.
//
// The functions also compile for the host, where the tests compare them with
// long double.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace sw {
namespace fx {

typedef long long i64;
typedef unsigned long long u64;

__host__ __device__ __forceinline__ uint32_t hi32(u64 v) { return (uint32_t)(v >> 32); }
__host__ __device__ __forceinline__ uint32_t lo32(u64 v) { return (uint32_t)v; }
__host__ __device__ __forceinline__ u64 join(uint32_t hi, uint32_t lo) { return ((u64)hi << 32) | lo; }

// double bits, arithmetic and seeds; explicit roundings on the device, so that
// every kernel computes the same bits
#ifdef __CUDA_ARCH__
__device__ __forceinline__ u64 bits_of(double v) { return (u64)__double_as_longlong(v); }
__device__ __forceinline__ double of_bits(u64 v) { return __longlong_as_double((i64)v); }
__device__ __forceinline__ uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t n) { return __funnelshift_l(lo, hi, n); }
__device__ __forceinline__ int clz(uint32_t v) { return __clz((int)v); }
__device__ __forceinline__ double dfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double of_int(i64 v) { return __ll2double_rn(v); }
__device__ __forceinline__ double rcp_seed(double v) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
  return r;
}
__device__ __forceinline__ double rsqrt_seed(double v) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
  return r;
}
#else
inline u64 bits_of(double v) { u64 b; std::memcpy(&b, &v, 8); return b; }
inline double of_bits(u64 b) { double v; std::memcpy(&v, &b, 8); return v; }
inline uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t n) { return (n & 31u) ? (hi << (n & 31u)) | (lo >> (32u - (n & 31u))) : hi; }
inline int clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }
inline double dfma(double a, double b, double c) { return std::fma(a, b, c); }
inline double dmul(double a, double b) { return a * b; }
inline double dadd(double a, double b) { return a + b; }
inline double of_int(i64 v) { return (double)v; }
// the device's seeds are within 2^-22 of the value; here that error is planted
inline double rcp_seed(double v) { return (1.0 / v) * (1.0 + 2e-7); }
inline double rsqrt_seed(double v) { return (1.0 / std::sqrt(v)) * (1.0 - 2e-7); }
#endif

// v * 2^n by the exponent (v normal, the result too)
__host__ __device__ __forceinline__ double scaled(double v, int n) {
  const u64 b = bits_of(v);
  return of_bits(join(hi32(b) + ((uint32_t)n << 20), lo32(b)));
}

constexpr uint32_t kExpMin = 1013;                  // biased exponent of 2^-10: one unit is 2^-52 of it
// largest biased exponents of the rest, axis and edge populations: below 1/2, 1/4
// and 1/8, so that all 19 add up to less than 4 (2^64 units) and |m| < 3/4
constexpr uint32_t kExpRest = 1021, kExpAxis = 1020, kExpEdge = 1019;

// v in units of 2^-62, exact; sets bad when v is outside [2^-10, 2^(emax - 1022)) (then the value is void)
__host__ __device__ __forceinline__ i64 to_units(double v, uint32_t emax, bool &bad) {
  const u64 b = bits_of(v);
  const uint32_t hi = hi32(b), lo = lo32(b);
  const uint32_t t = (hi >> 20) - kExpMin;          // (a set sign bit makes it large)
  bad = bad || t > emax - kExpMin;
  const uint32_t m = (hi & 0xfffffu) | 0x100000u;
  return (i64)join(shl_hi(lo, m, t), lo << (t & 31u));
}

// v units (2^40 <= v < 2^63) as a double, rounded to nearest (ties up)
__host__ __device__ __forceinline__ double of_units(u64 v) {
  const uint32_t hi = hi32(v), lo = lo32(v);
  const uint32_t s = (uint32_t)clz(hi);             // hi has a bit: s < 32
  const uint32_t nh = shl_hi(lo, hi, s), nl = lo << (s & 31u);
  // 53 bits with the leading one, which adds 1 to the exponent below; a carry out of them does so too
  const u64 r = (join(nh, nl) >> 11) + ((nl >> 10) & 1u);
  return of_bits(join(hi32(r) + ((1023u - s) << 20), lo32(r)));   // v = 2^(63 - s) 1.f units: exponent 1 - s
}

// A double in [1/4, 4) as a whole number of units, exact (2^-62 divides its last place); from 2 on the bits are
// those of an unsigned number.
__host__ __device__ __forceinline__ i64 to_units_large(double v) {
  const u64 b = bits_of(v);
  const uint32_t t = (hi32(b) >> 20) - kExpMin, m = (hi32(b) & 0xfffffu) | 0x100000u;
  return (i64)join(shl_hi(lo32(b), m, t), lo32(b) << (t & 31u));
}

// a b / 2^64, within 3 below
__host__ __device__ __forceinline__ i64 mulhi(i64 a, i64 b) {
  const int ah = (int)(a >> 32), bh = (int)(b >> 32);
  const int al = (int)(lo32((u64)a) >> 1), bl = (int)(lo32((u64)b) >> 1);
  const i64 cross = (i64)ah * bl + (i64)bh * al;
  return (i64)ah * bh + (cross >> 31);
}

// Newton's iteration for the reciprocal in its third-order form: y (1 + e + e^2), e = 1 - v y
__host__ __device__ __forceinline__ double reciprocal(double v) {
  const double y = rcp_seed(v);
  const double e = dfma(-v, y, 1.0);
  return dfma(y, dfma(e, e, e), y);
}
// square root by Goldschmidt's coupled iteration g ~ sqrt(v), h ~ 1 / (2 sqrt(v)), then one residual correction
__host__ __device__ __forceinline__ double square_root(double v) {
  const double y = rsqrt_seed(v);
  const double g = dmul(v, y), h = scaled(y, -1);
  const double g1 = dfma(g, dfma(-h, g, 0.5), g);
  return dfma(dfma(-g1, g1, v), h, g1);
}

// The collision of one cell.  tau0 = 3 nu + 1/2, tau0sq its square, c18 = 18 sqrt(2) Cs^2.  out[i] receives the
// new populations and mom rho and u (those are formed where they are used: from the exact m, so that velocities
// near rest keep their relative precision, which the collision's own u in units of 2^-61 has not); false: the
// cell is out of range and nothing of it is valid.
struct Moments {
  double rho, inv;                                  // inv: 2^-62 / rho
  i64 m[3];                                         // m in units of 2^-62
  __host__ __device__ __forceinline__ double vel(int k) const { return dmul(of_int(m[k]), inv); }
};
__host__ __device__ __forceinline__ bool collide(const double (&f)[19], double tau0, double tau0sq, double c18,
                                                 double (&out)[19], Moments &mom) {
  bool bad = false;
  i64 s[9], d[9];
  const i64 f0 = to_units(f[0], kExpRest, bad);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const uint32_t emax = k < 3 ? kExpAxis : kExpEdge;
    const i64 a = to_units(f[2 * k + 1], emax, bad), b = to_units(f[2 * k + 2], emax, bad);
    s[k] = a + b;
    d[k] = a - b;
  }
  if (bad) return false;
  // pairs: 0 (1,0,0) 1 (0,1,0) 2 (0,0,1) 3 (1,1,0) 4 (1,-1,0) 5 (1,0,1) 6 (1,0,-1) 7 (0,1,1) 8 (0,1,-1)
  const i64 sxy = s[3] + s[4], sxz = s[5] + s[6], syz = s[7] + s[8];
  const i64 rho = f0 + (s[0] + s[1] + s[2]) + (sxy + sxz + syz);
  if (rho < (1ll << 61)) return false;              // rho below 1/2, or (as a negative number) 2 and above
  const i64 mx = d[0] + (d[3] + d[4]) + (d[5] + d[6]);
  const i64 my = d[1] + (d[3] - d[4]) + (d[7] + d[8]);
  const i64 mz = d[2] + (d[5] - d[6]) + (d[7] - d[8]);
  mom.rho = of_units((u64)rho);
  const double y = reciprocal(mom.rho);
  mom.inv = scaled(y, -62);
  mom.m[0] = mx, mom.m[1] = my, mom.m[2] = mz;
  const i64 inv = to_units_large(y);                // 1 / rho in (1/2, 2)
  if (inv < 0) return false;                        // a density that rounds to 1/2: its reciprocal 2 has no sign bit left
  // |m| < 3/4, |u| < 3/2: u and m u in units of 2^-61
  const i64 ux = mulhi(mx << 1, inv), uy = mulhi(my << 1, inv), uz = mulhi(mz << 1, inv);
  const i64 mx2 = mx << 1, my2 = my << 1, mz2 = mz << 1, ux2 = ux << 1, uy2 = uy << 1, uz2 = uz << 1;
  const i64 bxx = mulhi(mx2, ux2), byy = mulhi(my2, uy2), bzz = mulhi(mz2, uz2);
  const i64 bxy = mulhi(mx2, uy2), bxz = mulhi(mx2, uz2), byz = mulhi(my2, uz2);
  const i64 third = mulhi(rho, 0x5555555555555556ll);
  const i64 nxx = (s[0] + sxy + sxz) - third - (bxx << 1);
  const i64 nyy = (s[1] + sxy + syz) - third - (byy << 1);
  const i64 nzz = (s[2] + sxz + syz) - third - (bzz << 1);
  const i64 nxy = (s[3] - s[4]) - (bxy << 1);
  const i64 nxz = (s[5] - s[6]) - (bxz << 1);
  const i64 nyz = (s[7] - s[8]) - (byz << 1);
  // |Pi_neq|^2 with the six entries shifted to the largest one's leading bit, below 2^61
  auto mag = [](i64 v) { const int h = (int)(v >> 32); return (uint32_t)(h ^ (h >> 31)); };
  const int lead = clz(mag(nxx) | mag(nyy) | mag(nzz) | mag(nxy) | mag(nxz) | mag(nyz)) - 3;
  if (lead < 0) return false;                       // an entry of 1/2 or more
  auto square = [lead](i64 v) {
    const uint32_t vh = shl_hi(lo32((u64)v), hi32((u64)v), (uint32_t)lead), vl = lo32((u64)v) << lead;
    return (i64)(int)vh * (int)vh + (((i64)(int)vh * (int)(vl >> 1)) >> 30);
  };
  const i64 q = (square(nxx) + square(nyy) + square(nzz)) + ((square(nxy) + square(nxz) + square(nyz)) << 1);
  // below 2^40 only where every entry is below 2^-39: |Pi_neq| then counts as 2^-39, which moves tau by about 2^-40
  // and what it multiplies, those entries, by 2^-79
  const uint32_t qh = hi32((u64)q) < 256u ? 256u : hi32((u64)q);
  const double qn = scaled(square_root(of_units(join(qh, lo32((u64)q)))), 1 - lead);
  const double root = square_root(dfma(dmul(c18, y), qn, tau0sq));
  // keep = 1 - 1 / tau, tau = (tau0 + root) / 2; a 1 / tau outside [1/4, 2 + 2^-19), negative, infinite or NaN (one
  // unsigned range of the upper word) is left to double
  const double rt = scaled(reciprocal(dadd(tau0, root)), 1);
  if (hi32(bits_of(rt)) - (1021u << 20) > (3u << 20)) return false;
  const i64 keep = (i64)((1ull << 62) - (u64)to_units_large(rt));
  const i64 Bxx = bxx + mulhi(nxx << 1, keep), Byy = byy + mulhi(nyy << 1, keep), Bzz = bzz + mulhi(nzz << 1, keep);
  const i64 Bxy = bxy + mulhi(nxy << 1, keep), Bxz = bxz + mulhi(nxz << 1, keep), Byz = byz + mulhi(nyz << 1, keep);
  const i64 t = Bxx + Byy + Bzz;                    // B in units of 2^-61
  if ((u64)(t + (1ll << 61)) >= (1ull << 62)) return false;   // |T| of 1 or more
  const i64 A = mulhi(rho - (t + (t << 1)), 0x071c71c71c71c71cll);                 // (rho - 6 T / 2) / 36
  const i64 wx = mulhi(mx2, 0x0aaaaaaaaaaaaaabll), wy = mulhi(my2, 0x0aaaaaaaaaaaaaabll);   // m / 12
  const i64 wz = mulhi(mz2, 0x0aaaaaaaaaaaaaabll);
  i64 v[19];
  v[0] = (A << 3) + (A << 2);
  const i64 A2 = A << 1;
  const i64 ax = A2 + (Bxx >> 1), ay = A2 + (Byy >> 1), az = A2 + (Bzz >> 1);
  v[1] = ax + (wx << 1);
  v[2] = ax - (wx << 1);
  v[3] = ay + (wy << 1);
  v[4] = ay - (wy << 1);
  v[5] = az + (wz << 1);
  v[6] = az - (wz << 1);
  const i64 exy = A + ((Bxx + Byy) >> 2), exz = A + ((Bxx + Bzz) >> 2), eyz = A + ((Byy + Bzz) >> 2);
  const i64 cxy = Bxy >> 1, cxz = Bxz >> 1, cyz = Byz >> 1;
  v[7] = (exy + cxy) + (wx + wy);
  v[8] = (exy + cxy) - (wx + wy);
  v[9] = (exy - cxy) + (wx - wy);
  v[10] = (exy - cxy) - (wx - wy);
  v[11] = (exz + cxz) + (wx + wz);
  v[12] = (exz + cxz) - (wx + wz);
  v[13] = (exz - cxz) + (wx - wz);
  v[14] = (exz - cxz) - (wx - wz);
  v[15] = (eyz + cyz) + (wy + wz);
  v[16] = (eyz + cyz) - (wy + wz);
  v[17] = (eyz - cyz) + (wy - wz);
  v[18] = (eyz - cyz) - (wy - wz);
  uint32_t any = 0u, least = 0xffffffffu;           // every result in [2^52, 2^62) units
#pragma unroll
  for (int i = 0; i < 19; ++i) {
    const uint32_t h = hi32((u64)v[i]);
    any |= h;
    least = h < least ? h : least;
  }
  if (any >= (1u << 30) || least < (1u << 20)) return false;
#pragma unroll
  for (int i = 0; i < 19; ++i) out[i] = of_units((u64)v[i]);
  return true;
}

}  // namespace fx
}  // namespace sw
