// f3d_f64.cuh — FP64 arithmetic in the form this GPU's FP64 pipe runs fastest.
//
// Measured with chains over all SMs (cycles per warp instruction and sub-core): an FMA of three
// registers 64; an add, a multiply, or an FMA with an operand from the constant bank, an immediate
// or a uniform register 76; a division 548, a square root 572, a reciprocal square root 368. The
// FP64 kernels keep the pipe busy, so the form of an instruction is 16% of its time. F64 is a
// double whose operators issue only three-register FMAs:
//   a + b = fma(a, 1, b),  a b = fma(a, b, -0),  a b + c = fma(a, b, c)
// with 1, -0 and every constant held in vector registers. Both forms are exact identities of the
// rounded sum and product (signed zeros, infinities and NaN included), so results are those of
// double arithmetic with the same contraction. A constant becomes a vector register by an exclusive
// or with a word that is zero but unknown, and not uniform over the warp, to the compiler.
#pragma once
#include <cuda_runtime.h>

namespace f3d {

static __constant__ unsigned f64_zero_word = 0u;
__device__ __forceinline__ unsigned f64_zero() {
    unsigned lane;
    asm("mov.u32 %0, %%laneid;" : "=r"(lane));
    return f64_zero_word & lane;
}
__device__ __forceinline__ double in_register(double c) {
    const unsigned z = f64_zero();
    return __hiloint2double(__double2hiint(c) ^ (int)z, __double2loint(c) ^ (int)z);
}

// Volatile: made where it is used (two integer instructions), not hoisted out of loops into
// registers that the WENO sums do not have; 1 and -0 stay.
__device__ __forceinline__ double constant_here(double c) {
    const unsigned z = f64_zero();
    int h, l;
    asm volatile("xor.b32 %0, %2, %4;\n\txor.b32 %1, %3, %4;"
                 : "=r"(h), "=r"(l) : "r"(__double2hiint(c)), "r"(__double2loint(c)), "r"(z));
    return __hiloint2double(h, l);
}

struct F64 {
    double v;
    F64() = default;
    __device__ __forceinline__ F64(double c) : v(constant_here(c)) {}  // a constant or a kernel argument
};
__device__ __forceinline__ F64 f64(double v) {  // a value that is in a register already
    F64 r;
    r.v = v;
    return r;
}
// a product not yet rounded: the first operand of an FMA, or a multiplication
struct F64Mul {
    double a, b;
    __device__ __forceinline__ operator F64() const { return f64(__fma_rn(a, b, in_register(-0.0))); }
};

__device__ __forceinline__ F64Mul operator*(F64 a, F64 b) { return F64Mul{a.v, b.v}; }
__device__ __forceinline__ F64 operator-(F64 a) { return f64(-a.v); }
__device__ __forceinline__ F64Mul operator-(F64Mul m) { return F64Mul{-m.a, m.b}; }
__device__ __forceinline__ F64 operator+(F64 a, F64 b) { return f64(__fma_rn(a.v, in_register(1.0), b.v)); }
__device__ __forceinline__ F64 operator-(F64 a, F64 b) { return f64(__fma_rn(a.v, in_register(1.0), -b.v)); }
__device__ __forceinline__ F64 operator+(F64Mul m, F64 c) { return f64(__fma_rn(m.a, m.b, c.v)); }
__device__ __forceinline__ F64 operator+(F64 c, F64Mul m) { return m + c; }
__device__ __forceinline__ F64 operator-(F64Mul m, F64 c) { return f64(__fma_rn(m.a, m.b, -c.v)); }
__device__ __forceinline__ F64 operator-(F64 c, F64Mul m) { return f64(__fma_rn(-m.a, m.b, c.v)); }
__device__ __forceinline__ F64 operator+(F64Mul m, F64Mul n) { return m + F64(n); }
__device__ __forceinline__ F64 operator-(F64Mul m, F64Mul n) { return F64(m) - n; }
__device__ __forceinline__ F64& operator+=(F64& a, F64 b) { return a = a + b; }
__device__ __forceinline__ F64& operator+=(F64& a, F64Mul m) { return a = m + a; }
__device__ __forceinline__ F64& operator-=(F64& a, F64 b) { return a = a - b; }
__device__ __forceinline__ F64& operator-=(F64& a, F64Mul m) { return a = a - m; }
__device__ __forceinline__ bool operator<(F64 a, F64 b) { return a.v < b.v; }
__device__ __forceinline__ bool operator>(F64 a, F64 b) { return a.v > b.v; }
__device__ __forceinline__ bool operator<=(F64 a, F64 b) { return a.v <= b.v; }
__device__ __forceinline__ bool operator>=(F64 a, F64 b) { return a.v >= b.v; }
__device__ __forceinline__ bool operator!=(F64 a, F64 b) { return a.v != b.v; }

// 1/b for any normal b whose reciprocal is normal: an FP32 reciprocal of its mantissa (integer
// operations and the special-function unit), its exponent set by integer arithmetic, and one
// third-order Newton step y (1 + e + e^2), e = 1 - b y (|e| < 2^-21, so the step leaves 2^-63
// before rounding): three FMAs, within an ulp. The IEEE quotient elsewhere.
__device__ __forceinline__ bool recip_range(double b) {
    const unsigned e = ((unsigned)__double2hiint(b) >> 20) & 0x7ffu;
    return e - 2u <= 2040u;
}
__device__ __forceinline__ F64 recip_step(double b) {
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29))));
    const unsigned f = __float_as_uint(y);  // in (1/2, 1]
    // binary64 bits of y 2^-(exponent of b), with b's sign
    const unsigned yh = (f >> 3) + (896u << 20) - ((hi & 0x7ff00000u) - (1023u << 20));
    const F64 y0 = f64(__hiloint2double((int)(yh | (hi & 0x80000000u)), (int)(f << 29)));
    const F64 e = f64(in_register(1.0)) - f64(b) * y0;
    return y0 + y0 * (e + e * e);
}
__device__ __forceinline__ F64 recip(F64 b) {
    if (!recip_range(b.v)) return f64(1.0 / b.v);
    return recip_step(b.v);
}
// 1/b with one residual correction (five FMAs): before its last rounding within 2^-105 of the
// reciprocal, so it is the IEEE reciprocal unless that lies as near to a rounding boundary
__device__ __forceinline__ F64 recip_ieee(F64 b) {
    if (!recip_range(b.v)) return f64(1.0 / b.v);
    const F64 r = recip_step(b.v);
    return r + (f64(in_register(1.0)) - b * r) * r;
}
// a/b: a times the reciprocal and one residual correction (Markstein's; six FMAs; as near to the IEEE
// quotient as recip_ieee) where the quotient and the residual are normal; the IEEE division elsewhere
__device__ __forceinline__ F64 operator/(F64 a, F64 b) {
    const unsigned ha = (unsigned)__double2hiint(a.v) & 0x7fffffffu, ea = ha >> 20;
    const unsigned eb = ((unsigned)__double2hiint(b.v) >> 20) & 0x7ffu;
    // both factors, the quotient and the residual well inside the normal range, or a zero dividend
    const bool zero = (ha | (unsigned)__double2loint(a.v)) == 0u;
    const bool plain = eb - 2u <= 2040u && ((ea - 110u <= 1900u && ea - eb + 900u <= 1800u) || zero);
    if (!plain) return f64(a.v / b.v);
    const F64 r = recip_step(b.v);
    const F64 q = a * r;
    const F64 c = q + (a - b * q) * r;  // (a zero's sign would be lost here)
    return f64(zero ? q.v : c.v);
}
using ::fabs;  // the overloads below stand beside the library's
using ::sqrt;
__device__ __forceinline__ F64 fabs(F64 a) { return f64(::fabs(a.v)); }
__device__ __forceinline__ F64 sqrt(F64 a) { return f64(::sqrt(a.v)); }
__device__ __forceinline__ F64 rsq(F64 a) { return f64(::rsqrt(a.v)); }

// The square root of a normal x: an FP32 reciprocal root of x scaled by an even power of two, one
// step of Goldschmidt's coupled iteration for g = x^(1/2), h = x^(-1/2) / 2 (relative error 2^-22 to
// 2^-43) and the residual correction g + h (x - g^2): seven FMAs (448 cycles against 572), before
// its last rounding within 2^-85 of the root. The library's root elsewhere.
__device__ __forceinline__ F64 root(F64 x) {
    const unsigned hi = (unsigned)__double2hiint(x.v), e = hi >> 20;  // sign and exponent
    if (e - 64u > 1900u) return sqrt(x);
    const unsigned lo = (unsigned)__double2loint(x.v);
    // mantissa times 1 (odd biased exponent) or 2, as binary32 in [1, 4)
    const unsigned odd = (e & 1u) ^ 1u;
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;"
        : "=f"(y) : "f"(__uint_as_float(((127u + odd) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29))));
    const unsigned f = __float_as_uint(y);  // in (1/2, 1]
    // times 2^-((e - odd - 1023) / 2)
    const unsigned yh = (f >> 3) + (896u << 20) - ((((e - odd) - 1023u) << 19) & 0xfff00000u);
    const F64 y0 = f64(__hiloint2double((int)yh, (int)(f << 29)));
    const F64 half = f64(in_register(0.5));
    F64 g = x * y0, h = y0 * half;
    const F64 r = half - g * h;
    g = g + g * r;
    h = h + h * r;
    return g + (x - g * g) * h;
}

// The arithmetic type of a kernel's element type, and values between the two
template <class R> struct Arith { using type = R; };
template <> struct Arith<double> { using type = F64; };
__device__ __forceinline__ F64 arith(double x) { return f64(x); }
__device__ __forceinline__ float arith(float x) { return x; }
__device__ __forceinline__ double plain(F64 x) { return x.v; }
__device__ __forceinline__ float plain(float x) { return x; }

}  // namespace f3d
