// Device helpers shared by the assembly translation units.
#pragma once
#include "common.cuh"
#include "complex.cuh"

namespace bem {

constexpr int TILE = 64;
constexpr int ASM_THREADS = 256;
constexpr double PI_D = 3.14159265358979323846;

// influence_matrix.rs:42-50: static flat-disc self term (k independent), scaled
// by wt*area, plus the hdiag / gdiag diagonal of preprocess.rs:60-74.
__device__ __forceinline__ void self_term64(double area, double wt, int bm, double beta_im, double hdiag,
                                            double gdiag_im, z2& g, z2& h) {
    double b = sqrt(area / PI_D);
    double g0 = 1.0 / (2.0 * PI_D * b);
    double h0im = bm ? beta_im * (-1.0 / (2.0 * PI_D * (b * b * b))) : 0.0;
    g = make_double2(g0 * wt * area, 0.0);
    h = make_double2(0.0, h0im * wt * area);
    h.x += hdiag;
    g.y += gdiag_im;
}

// ---------------------------------------------------------------------------
// FP64 arithmetic of the kernel functions.  GB300 issues an FP64 instruction of
// a warp every 65 clocks per SM quarter, against 2 for an FP32 or integer one,
// so the count of FP64 instructions is the run time: seeds come from FP32, tails
// of series below 2^-29 of the result are summed in FP32, operands are built
// from bits.

// v 2^-e as a float, truncated to 24 bits (0 far below its range).
__device__ __forceinline__ float near_float(double v, int e) {
    const int hi = __double2hiint(v), lo = __double2loint(v), ex = ((hi >> 20) & 0x7ff) - 1023 - e;
    if (ex < -120) return 0.0f;
    return __int_as_float((hi & 0x80000000) | ((min(ex, 120) + 127) << 23) | ((hi & 0xfffff) << 3) |
                          ((unsigned)lo >> 29));
}
// A float of moderate exponent as a double, without the conversion instruction.
__device__ __forceinline__ double wide(float f) {
    const int b = __float_as_int(f);
    return __hiloint2double((b & 0x80000000) | (((b & 0x7fffffff) >> 3) + ((1023 - 127) << 20)), b << 29);
}
// Any float: by the conversion where the exponent is that of zero, a subnormal, an
// infinity or a NaN.
__device__ __forceinline__ double wide_any(float f) {
    const unsigned e = (__float_as_uint(f) >> 23) & 0xff;
    return e == 0 || e == 0xff ? (double)f : wide(f);
}

// inv = 1 / sqrt(v) and root = sqrt(v): the FP32 seed and one third-order
// correction shared by both, seven FP64 instructions (a square root and a
// division take about 25), each within 0.75 ulp.  v = 0 gives inv = infinity,
// root = 0; a NaN stays one.
__device__ __forceinline__ void root64(double v, double& inv, double& root) {
    const int e = (((__double2hiint(v) >> 20) & 0x7ff) - 1023) & ~1;  // even
    if (e < -960 || e > 960) {
        root = sqrt(v);
        inv = 1.0 / root;
        return;
    }
    const double s = wide(rsqrtf(near_float(v, e))) * __hiloint2double((1023 - e / 2) << 20, 0);
    const double h = v * s;
    const double c = fma(-h, s, 1.0);
    const double p = c * fma(0.375, c, 0.5);
    inv = fma(s, p, s);
    root = fma(h, p, h);
}

// e^{i k r} for |k r| < 10^5 (sincos beyond): t = k r with its rounding error,
// reduced by multiples of pi/2 (two parts of pi/2, the products exact through
// FMA), then the Taylor series, the terms below 2^-36 of the result in FP32.
__device__ __forceinline__ void phase64(double kk, double r, double& c, double& s) {
    const double t = kk * r, tl = fma(kk, r, -t);
    if (!(fabs(t) < 1e5)) {
        sincos(t, &s, &c);
        return;
    }
    const double shift = 6755399441055744.0;  // 1.5 2^52: the sum's low bits hold the nearest integer
    const double k = fma(t, 0.63661977236758134308, shift);
    const int quad = __double2loint(k);
    const double n = k - shift;
    double x = fma(-n, 1.57079632679489661923, t);
    x += fma(-n, 6.12323399573676588613e-17, tl);
    const double z = x * x;
    const float zf = near_float(z, 0);
    // sin x = x + x z (S1 + z (S2 + z (S3 + z (S4 + z (S5 + z tail))))), S_n = (-1)^n / (2n+1)!
    const float ts = fmaf(zf, fmaf(zf, 2.8114573e-15f, -7.6471637e-13f), 1.6059044e-10f);
    double ps = fma(z, wide(ts), -2.50521083854417187751e-8);
    ps = fma(z, ps, 2.75573192239858906526e-6);
    ps = fma(z, ps, -1.98412698412698412698e-4);
    ps = fma(z, ps, 8.33333333333333333333e-3);
    ps = fma(z, ps, -1.66666666666666666667e-1);
    const double sn = fma(x * z, ps, x);
    // cos x = 1 - z / 2 + z^2 (C2 + z (C3 + z (C4 + z (C5 + z tail)))), C_n = (-1)^n / (2n)!
    const float tc = fmaf(zf, fmaf(zf, 4.7794773e-14f, -1.1470746e-11f), 2.0876757e-9f);
    double pc = fma(z, wide(tc), -2.75573192239858906526e-7);
    pc = fma(z, pc, 2.48015873015873015873e-5);
    pc = fma(z, pc, -1.38888888888888888889e-3);
    pc = fma(z, pc, 4.16666666666666666667e-2);
    pc = fma(z, pc, -0.5);
    const double cs = fma(z, pc, 1.0);
    const bool odd = quad & 1;
    const double a = odd ? sn : cs, b = odd ? cs : sn;
    // quadrants: (c, s) = (cs, sn), (-sn, cs), (-cs, -sn), (sn, -cs)
    c = __hiloint2double(__double2hiint(a) ^ (int)(((unsigned)(quad + 1) & 2u) << 30), __double2loint(a));
    s = __hiloint2double(__double2hiint(b) ^ (int)(((unsigned)quad & 2u) << 30), __double2loint(b));
}

// The same functions in 64-bit integers.  An integer instruction costs a
// thirtieth of an FP64 one here, a 64 x 64 -> 64 product about a third, and
// fixed point keeps 60 bits where FP64 keeps 53: the pair's root, its phase
// (k r / 2 pi modulo one turn, exact to the product's bits) and sine and cosine
// leave the FP64 pipe altogether.

// m 2^q for a normalised 53-bit integer m in [2^52, 2^53].
__device__ __forceinline__ double from_mantissa(uint64_t m, int q) {
    return __longlong_as_double((long long)(((uint64_t)(unsigned)(q + 1074) << 52) + m));
}
// u 2^q rounded to nearest (u = 0: 0).
__device__ __forceinline__ double from_integer(uint64_t u, int q) {
    const int lz = __clzll((long long)(u | 1ull));
    const uint64_t n = u << lz;
    return u ? from_mantissa((n >> 11) + ((n >> 10) & 1ull), q + 11 - lz) : 0.0;
}

// 1 / sqrt(v), sqrt(v) and e^{i k sqrt(v)} for v whose phase lies between 2^-10
// and 2^40 turns (false otherwise: nothing is written).  turn 2^(turn_exp - 64)
// is k / 2 pi, turn's top bit set.
__device__ __forceinline__ bool wave_int(double v, unsigned long long turn, int turn_exp, double& inv, double& root,
                                         double& c, double& s) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    const int ev = (int)(b >> 52) - 1023, h = ev >> 1;  // v = w 2^(2 h), 1 <= w < 4
    const int E = h + turn_exp;
    if ((unsigned)(ev + 900) > 1800u || (unsigned)(E + 9) > 49u) return false;
    const uint64_t W = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << (10 + (ev & 1));  // Q62
    // y = the FP32 root's reciprocal as Q24, c = 1 - w y^2 as Q61 (below 2^-21)
    const unsigned Y = __float2uint_rn(rsqrtf(__uint2float_rn((unsigned)(W >> 32)) * 9.31322574615478516e-10f) *
                                       16777216.0f);
    const int64_t d = (int64_t)((1ull << 61) - __umul64hi(W, ((uint64_t)Y * Y) << 15));
    const int64_t dh = d >> 9;
    const int64_t p = (d >> 1) + ((3 * ((dh * dh) >> 43)) >> 3);
    const uint64_t I = ((uint64_t)Y << 37) + (uint64_t)(((int64_t)Y * (p >> 2)) >> 22);  // 1 / sqrt(w), Q61
    const uint64_t R = __umul64hi(W, I << 2);                                      // sqrt(w), Q61
    inv = from_mantissa((I + 128) >> 8, -53 - h);
    root = from_mantissa((R + 256) >> 9, -52 + h);
    // the phase in turns, Q64: (R 2^2)(turn) 2^(E - 63) modulo 2^64
    const uint64_t hi = __umul64hi(R << 2, turn), lo = (R << 2) * turn;
    const int sh = 63 - E;  // 23 .. 72
    const uint64_t F = sh < 64 ? (lo >> sh) | (hi << (64 - sh)) : hi >> (sh - 64);
    const unsigned quad = (unsigned)((F + (1ull << 61)) >> 62);
    const int64_t y = (int64_t)(F - ((uint64_t)quad << 62));  // from the nearest quarter turn
    const bool neg = y < 0;
    const uint64_t X = __umul64hi((uint64_t)(neg ? -y : y) << 2, 0xc90fdaa22168c235ull);  // |x| in radians, Q63
    const uint64_t Z = __umul64hi(X << 1, X << 1);                                       // x^2, Q64
    const unsigned zh = (unsigned)(Z >> 32);
    // 1/3! - z (1/5! - z (1/7! - ...)) and 1/2! - z (1/4! - z (1/6! - ...)), Q64
    unsigned t = 0xd73f9fu - __umulhi(zh, 0xca96u);
    t = 0xb092309du - __umulhi(zh, t);
    uint64_t S = 0x6b99159fd5ull - __umulhi(zh, t);
    S = 0x2e3bc74aad8eull - __umul64hi(Z, S);
    S = 0xd00d00d00d00dull - __umul64hi(Z, S);
    S = 0x222222222222222ull - __umul64hi(Z, S);
    S = 0x2aaaaaaaaaaaaaabull - __umul64hi(Z, S);
    const uint64_t sn = X - __umul64hi(X, __umul64hi(Z, S));  // Q63
    t = 0xc9cba54u - __umulhi(zh, 0xd73fau);
    uint64_t C = 0x8f76c77fcull - __umulhi(zh, t);
    C = 0x49f93edde28ull - __umul64hi(Z, C);
    C = 0x1a01a01a01a02ull - __umul64hi(Z, C);
    C = 0x5b05b05b05b05bull - __umul64hi(Z, C);
    C = 0xaaaaaaaaaaaaaabull - __umul64hi(Z, C);
    C = 0x8000000000000000ull - __umul64hi(Z, C);
    const uint64_t cn = (1ull << 63) - (__umul64hi(Z, C) >> 1);  // Q63, at least 0.7
    const double cs = from_mantissa((cn + 512) >> 10, -53), sv = from_integer(sn, -63);
    // quadrants: (c, s) = (cs, sn), (-sn, cs), (-cs, -sn), (sn, -cs)
    const bool odd = quad & 1u;
    const unsigned flip = neg ? 0x80000000u : 0u;
    const double a = odd ? sv : cs, e = odd ? cs : sv;
    c = __hiloint2double(__double2hiint(a) ^ (int)((((quad + 1u) & 2u) << 30) ^ (odd ? flip : 0u)), __double2loint(a));
    s = __hiloint2double(__double2hiint(e) ^ (int)(((quad & 2u) << 30) ^ (odd ? 0u : flip)), __double2loint(e));
    return true;
}

// influence_matrix.rs:12-37 for one pair, scaled by w = wt area / (4 pi):
// d = source minus observation, ey the observation's normal, ex the source's
// (Burton-Miller, coupling i b with b = 1 / k).  With u = g / r and
// v = u - i k g: G = g, H = (d . ey / r) v and the Burton-Miller terms
//   G += i b dG,  dG = -(d . ex / r) v
//   H += i b dH,  b dH = u ((b m / r - k r p) - i m)
// p the product of the two direction cosines, m = ex . ey + 3 p.
// 19 FP64 instructions, 39 with the Burton-Miller terms (about 85 and 115 as
// the reference writes them).
template <bool BM>
__device__ __forceinline__ void pair64(const KParams& kp, double w, double dx, double dy, double dz, double eyx,
                                       double eyy, double eyz, double exx, double exy, double exz, z2& g, z2& h) {
    double inv, r, c, s;
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    if (!wave_int(r2, kp.turn, kp.turn_exp, inv, r, c, s)) {
        root64(r2, inv, r);
        phase64(kp.k, r, c, s);
    }
    const double q = inv * w;
    g = make_double2(c * q, s * q);
    const z2 u = make_double2(g.x * inv, g.y * inv);
    const z2 v = make_double2(fma(kp.k, g.y, u.x), fma(-kp.k, g.x, u.y));
    const double cy = fma(dx, eyx, fma(dy, eyy, dz * eyz)) * inv;
    h = make_double2(cy * v.x, cy * v.y);
    if (BM) {
        const double b = kp.beta_im;
        const double cx = fma(dx, exx, fma(dy, exy, dz * exz)) * inv;
        const double p = cx * cy, m = fma(3.0, p, fma(eyx, exx, fma(eyy, exy, eyz * exz)));
        const double t = fma(-(kp.k * r), p, (inv * b) * m), bc = b * cx;
        g = make_double2(fma(bc, v.y, g.x), fma(-bc, v.x, g.y));
        h.x = fma(-u.y, t, fma(u.x, m, h.x));
        h.y = fma(u.x, t, fma(u.y, m, h.y));
    }
}

// Entry (observation i, source j) of G and H from the device geometry.
__device__ __forceinline__ void pair64_at(const KParams& kp, int64_t np, const double* __restrict__ geo, int64_t i,
                                          int64_t j, z2& g, z2& h) {
    const double w = geo[GWA * np + j] * (1.0 / (4.0 * PI_D));
    const double dx = geo[GX * np + j] - geo[GX * np + i], dy = geo[GY * np + j] - geo[GY * np + i],
                 dz = geo[GZ * np + j] - geo[GZ * np + i];
    const double eyx = geo[GEX * np + i], eyy = geo[GEY * np + i], eyz = geo[GEZ * np + i];
    if (kp.bm)
        pair64<true>(kp, w, dx, dy, dz, eyx, eyy, eyz, geo[GEX * np + j], geo[GEY * np + j],
                     geo[GEZ * np + j], g, h);
    else
        pair64<false>(kp, w, dx, dy, dz, eyx, eyy, eyz, 0, 0, 0, g, h);
}

int* device_err(Context& ctx);
void finish_norms(Context& ctx, const double* part, int64_t nparts, int nsys, double* out);
void check_device_err(Context& ctx);
void launch_reduce_parts(Context& ctx, int64_t n, int64_t npad, int ntiles, const double2* part, double2* out);

}  // namespace bem
