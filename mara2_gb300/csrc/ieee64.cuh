// ieee64.cuh -- correctly rounded FP64 division, square root and product from
// integer instructions.
//
// The FP64 pipe of this GPU executes half a lane per clock per scheduler (a
// warp's instruction every 64 clocks; measured 1.65 operations per clock per
// SM), so one FP64 operation costs as much as 64 integer instructions, and a
// division or square root is eight to ten FP64 operations.  The functions
// here give the IEEE round-to-nearest-even result bit for bit from about 60
// integer instructions and one hardware reciprocal (or reciprocal square
// root) approximation, a product from about 40 instructions.  Operations per
// clock per SM, measured (the hardware's in brackets): division 1.08 (0.24),
// square root 1.12 (0.23), product 1.85 (1.65).  The product gains because
// the two pipes run side by side: an addition and such a product take the
// time of the addition alone.
//
// Division and square root: schoolbook long division (square root) in two digits of about 28
// bits on the 53-bit significands, each digit from a 32-bit reciprocal that
// one Newton step in integers brings from the hardware's 22 bits to 30, then
// the rounded candidate is checked against the exact remainder, which decides
// the last unit.  A quotient or square root of FP64 numbers is never halfway
// between two FP64 numbers, so round to nearest needs no rule for ties.
// Remainders are formed modulo 2^64; their true magnitudes are below 2^63.
//
// The functions are branch-free and valid for normal operands with a normal
// result, and zero numerators and factors; anything else clears `ok`, and the
// caller repeats its work with the ordinary operators.  They compile for the host
// too, where the tests compare them with the host's own division and square
// root.
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define IEEE64_FN __host__ __device__ __forceinline__
#else
#define IEEE64_FN static inline
#endif

namespace ieee64 {

typedef uint32_t u32;
typedef uint64_t u64;
typedef int64_t i64;

// (an asm move on the device: the compiler turns integer tests of a double's
// bits that it can see through into FP64 compares)
IEEE64_FN u64 bits(double x)
{
#if defined(__CUDA_ARCH__)
    u64 b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
#else
    u64 b;
    memcpy(&b, &x, 8);
    return b;
#endif
}
IEEE64_FN double from_bits(u64 b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long) b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}
IEEE64_FN u32 mulhi(u32 a, u32 b) { return (u32) (((u64) a * b) >> 32); }

// The hardware's approximations of 1/f for f in [1, 2) and 1/sqrt(f) for f in
// [1, 4), times 2^32: 24 bits, in [2^31, 2^32).  The methods below hold for
// any result within 2^-22 (relative); on the host IEEE64_SEED_ULPS shifts the
// result so that the tests cover both ends.
#ifndef IEEE64_SEED_ULPS
#define IEEE64_SEED_ULPS 0
#endif
IEEE64_FN u32 seed_word(u32 r)
{
    r = r < 0x3f000000u ? 0x3f000000u : r > 0x3f7fffffu ? 0x3f7fffffu : r;   // into [1/2, 1)
    return (r << 8) | 0x80000000u;
}
IEEE64_FN u32 seed_rcp(u32 fbits)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
    return seed_word(__float_as_uint(r));
#else
    float f;
    memcpy(&f, &fbits, 4);
    f = 1.0f / f;
    memcpy(&fbits, &f, 4);
    return seed_word(fbits + IEEE64_SEED_ULPS);
#endif
}
IEEE64_FN u32 seed_rsqrt(u32 fbits)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
    return seed_word(__float_as_uint(r));
#else
    float f;
    memcpy(&f, &fbits, 4);
    f = (float) (1.0 / __builtin_sqrt((double) f));
    memcpy(&fbits, &f, 4);
    return seed_word(fbits + IEEE64_SEED_ULPS);
#endif
}

// RN(a b) for factors that are normal or zero, with a normal product
IEEE64_FN double mul(double a, double b)
{
    const u64 x = bits(a), y = bits(b);
    const u32 xh = (u32) (x >> 32), yh = (u32) (y >> 32);
    // significands in [2^63, 2^64)
    const u64 X = (x << 11) | 0x8000000000000000ull, Y = (y << 11) | 0x8000000000000000ull;
    const u32 x0 = (u32) X, x1 = (u32) (X >> 32), y0 = (u32) Y, y1 = (u32) (Y >> 32);
    const u64 t0 = (u64) x0 * y0;
    const u64 t1 = (u64) x1 * y0 + (t0 >> 32);
    const u64 t2 = (u64) x0 * y1 + (u32) t1;
    u64 hi = (u64) x1 * y1 + (t1 >> 32) + (t2 >> 32);     // upper 64 bits, in [2^62, 2^64)
    hi |= ((u32) t2 | (u32) t0) != 0 ? 1 : 0;             // whether the lower 64 are not zero
    const u32 n = (u32) (hi >> 63), s = 10 + n;           // bits below the significand: 10 or 11
    hi += ((1u << (s - 1)) - 1) + ((u32) (hi >> s) & 1);  // half to even; stays below 2^64
    const u32 e = ((xh >> 20) & 0x7ffu) + ((yh >> 20) & 0x7ffu) - 1024 + n;
    const bool zero = (x << 1) == 0 || (y << 1) == 0;
    const u64 r = zero ? 0ull : ((u64) e << 52) + (hi >> s);
    return from_bits(r | ((u64) ((xh ^ yh) & 0x80000000u) << 32));
}
IEEE64_FN double mul(double a, double b, bool& ok)
{
    const u32 ea = (u32) (bits(a) >> 52) & 0x7ffu, eb = (u32) (bits(b) >> 52) & 0x7ffu;
    const bool zero = (bits(a) << 1) == 0 || (bits(b) << 1) == 0;
    ok = ok && ea < 2047u && eb < 2047u && (zero || (ea != 0 && eb != 0 && ea + eb - 1024u < 2044u));
    return mul(a, b);
}

// A divisor's significand, exponent and 32-bit reciprocal, shared by all
// divisions by it.
struct Divisor {
    u64 D;      // significand in [2^52, 2^53)
    u32 R;      // 2^84 / D less 3 to 7 units (R is below 2^32)
    u32 hi;     // upper word (sign, exponent)
};

IEEE64_FN Divisor divisor(double d, bool& ok)
{
    const u64 b = bits(d);
    Divisor v;
    v.hi = (u32) (b >> 32);
    ok = ok && ((v.hi >> 20) & 0x7ffu) - 1u < 2046u;
    v.D = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const u32 d32 = (u32) (v.D >> 21);  // [2^31, 2^32)
    const u32 r0 = seed_rcp(0x3f800000u | ((d32 >> 8) & 0x7fffffu));   // 2^63 / d32 to within 2^-21
    // Newton: r0 (1 + e), e = 1 - r0 d32 / 2^63.  The truncations below take
    // less than 1.1 units off and that of d32 adds less than 2, so the bias
    // of 5 keeps R below 2^84 / D
    const i64 e = (i64) (0x8000000000000000ull - (u64) r0 * d32);
    const int32_t e32 = (int32_t) (e >> 12);               // e 2^51, at most 2^30
    v.R = r0 + (u32) (int32_t) (((i64) e32 * (i64) (r0 >> 1)) >> 50) - 5u;
    return v;
}

// RN(x / d).  LOW: a quotient below 2^(LOW - 1023) clears ok.
template <int LOW = 1> IEEE64_FN double div(double x, const Divisor& v, bool& ok)
{
    const u64 b = bits(x);
    const u32 xhi = (u32) (b >> 32);
    const u32 sign = (xhi ^ v.hi) & 0x80000000u;
    const u32 ex = (xhi >> 20) & 0x7ffu, ed = (v.hi >> 20) & 0x7ffu;
    const bool zero = (b << 1) == 0;
    u64 X = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const bool less = X < v.D;
    X <<= less ? 1 : 0;                                    // X / D in [1, 2)
    const int e = (int) ex - (int) ed + 1023 - (less ? 1 : 0);
    ok = ok && (zero || (ex - 1u < 2046u && (u32) (e - LOW) < 2047u - LOW));
    const u32 q1 = mulhi((u32) (X >> 22), v.R);            // X / D 2^30, at most 9 units low
    const u64 rem = (X << 30) - (u64) q1 * v.D;            // in [0, 9 D), below 2^57
    const u32 q2 = mulhi((u32) (rem >> 25), v.R);          // rem / D 2^27, at most 6 units low
    const u64 Q = ((u64) q1 << 27) + q2;                   // X / D 2^57, as low as q2
    u64 M = (Q + 19u) >> 5;                                // rounded to 53 bits, at most one unit off
    const i64 rr = (i64) (((X << 52) - M * v.D) << 1);     // twice the remainder
    const i64 D = (i64) v.D;
    M += rr > D ? 1 : 0;
    M -= rr < -D ? 1 : 0;
    const u64 q = zero ? 0ull : ((u64) (u32) (e - 1) << 52) + M;
    return from_bits(q | ((u64) sign << 32));
}

template <int LOW = 1> IEEE64_FN double div(double x, double d, bool& ok) { return div<LOW>(x, divisor(d, ok), ok); }

// RN(sqrt(a)) for a >= 0 (zero or normal)
IEEE64_FN double sqrt_rn(double a, bool& ok)
{
    const u64 b = bits(a);
    const u32 hi = (u32) (b >> 32);
    const u32 ea = hi >> 20;                               // sign and exponent field
    const bool zero = b == 0;
    ok = ok && (zero || ea - 1u < 2046u);
    const u32 odd = (ea & 1u) ^ 1u;                        // the bias is odd: an even field is an odd exponent
    const u64 A = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << odd;   // a' 2^52, a' in [1, 4)
    const u32 a32 = (u32) (A >> 22);                       // a' 2^30
    const u32 r0 = seed_rsqrt((0x3f800000u + (odd << 23)) | ((u32) (b >> 29) & 0x7fffffu));   // 2^32 / sqrt(a')
    // Newton: r0 (1 + e / 2), e = 1 - a' r0^2 / 2^64.  The truncations take
    // less than 1.1 units off and add less than 4.1, so the bias of 6 keeps R
    // below 2^32 / sqrt(a'), by at most 7.1 units
    const i64 e = (i64) (0x4000000000000000ull - (u64) mulhi(r0, r0) * a32);   // e 2^62
    const int32_t e32 = (int32_t) (e >> 12);               // e 2^50, below 2^30
    const u32 R = r0 + (u32) (int32_t) (((i64) e32 * (i64) (r0 >> 1)) >> 50) - 6u;
    const u32 s1 = mulhi(a32, R);                          // sqrt(a') 2^30, 0 to 9.1 units low
    const u64 rem = (A << 8) - (u64) s1 * s1;              // a' 2^60 - s1^2 in [0, 2^37)
    const u32 q2 = (u32) (((rem >> 5) * (u64) R) >> 31);   // rem / (2 s1) 2^27, at most 13 units low
    const u64 S = ((u64) s1 << 27) + q2;                   // sqrt(a') 2^57, as low as q2
    u64 M = (S + 22u) >> 5;                                // rounded to 53 bits, at most one unit off
    const i64 rr = (i64) ((A << 52) - M * M);              // (M +- 1/2)^2 = M^2 +- M + 1/4
    const i64 m = (i64) M;
    M += rr > m ? 1 : 0;
    M -= rr <= -m ? 1 : 0;
    const u32 e2 = (ea + 1023u) >> 1;
    return from_bits(zero ? b : ((u64) (e2 - 1u) << 52) + M);
}

} // namespace ieee64
