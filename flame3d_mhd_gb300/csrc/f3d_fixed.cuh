// f3d_fixed.cuh — the linear reconstruction (UP7 / CD6 blend, schemes.jl:119-142) of FP64 split
// fluxes as exact integer sums.
//
// What bounds it: an FP64 instruction holds an SM sub-core's FP64 pipe for 64 cycles (FMA of
// three registers) or 76 (add, multiply, or an FMA with a constant operand; measured with
// dependent chains), an integer multiply-add of 32 x 32 + 64 bits for 2. The linear face flux is
// 14 products with fixed coefficients per component, 70 FP64 instructions a face and 40% of the
// FP64 work of a sweep. Its coefficients are rationals with a small common denominator D
// (420 for UP7: -3, 25, -101, 319, 214, -38, 4), so D times the flux is an integer combination of
// the fluxes' mantissas. A strip of five faces of one line and one component aligns the eleven Fp
// and eleven Fm it reads to the largest of them as 62-bit integers, sums the 5 x 14 products in
// integers without rounding, and rounds each sum to FP64 once before the product with 1/D: one
// FP64 instruction a face and component instead of 14. On the 256x64x64 shock tube the three
// sweeps' FP64 thread instructions go from 181-189 / 160-167 / 166-184 million a launch to
// 112 / 90 / 107, the sweeps from 517 / 434 / 453 to 366 / 324 / 373 us and the RK3 step from 4.68
// to 3.67 ms; the viscous ramp's step at 512x256x128 from 75.4 to 61.0 ms (all measured before the
// WENO faces left the tiles). Five faces a strip: 22 conversions serve five faces, and 13 strips
// cover a tile's 65 faces exactly.
//
// Accuracy: a value whose exponent lies within 9 of the strip's largest is exact; smaller ones are
// truncated to a multiple of 2^-61 of it (in units of the largest's power of two). The largest need not
// be a value that a sum reads, or reads under a coefficient that matters (they go down to 3/420), so each
// sum is looked at by itself (beyond_spread): it is formed from integers if one of the values under
// its central coefficients (214/420 and above) is within 2^5 of the largest, or if every value (of the
// strip; one-sided sums: that it reads) enters exactly. What is truncated is then at most 2.9 units for a
// face (1.2 for a one-sided sum), the central term alone at least 2^-6 of the largest, so the error is
// below 0.7 x 2^-53 (0.3) of the sum of the magnitudes of the sum's own terms, less than an FP64
// evaluation rounds. A one-sided sum is also formed from integers if a value beside its centre is within
// 2^3 of the largest, or the largest itself beyond that: under coefficients of 38/420 and 4/420 and above
// such a term is at least 2^-6.7 of the largest, and the error again below 0.7 x 2^-53 of the terms (the
// cotangents of a line's first faces, whose outermost is a hundred times the others'). Then one rounding
// to FP64 and one in the product with 1/D. Other sums, infinities, NaN and strips whose magnitudes lie near
// the ends of the FP64 range are formed in FP64. Against extended precision the right-hand side of a coarse
// tube is off by 0.95 / 0.85 / 0.91 (Steger-Warming / Lax-Friedrichs / AUSM) and of a finite-volume
// vortex by 0.97 of what FP64 sums leave.
#pragma once
#include "f3d_kernels.cuh"

namespace f3d {

constexpr int LIN_STRIP = 5;    // faces a strip
constexpr int LIN_SPREAD = 5;   // largest exponent minus that of a sum's centre

// x 2^(1084 - E) as an integer (E: the strip's largest biased exponent), truncated towards zero;
// below: how many exponents x lies below the largest (a zero: E)
__device__ __forceinline__ long long fixed_of(double x, int E, int& below) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int e = (int)((hi >> 20) & 0x7ffu);
    // mantissa with its leading one at bit 63, then right to bit 61 and by the exponent's distance
    // (zeros and subnormals: E >= 200 makes the distance more than 63, which gives 0)
    const unsigned long long m =
        ((unsigned long long)(__funnelshift_l(lo, hi, 11) | 0x80000000u) << 32) | (unsigned long long)(lo << 11);
    unsigned long long v;
    below = E - e;
    asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(below + 2));  // shifts past 63 give 0
    const long long s = (long long)((int)hi >> 31);
    return ((long long)v ^ s) - s;
}
__device__ __forceinline__ long long fixed_of(double x, int E) {
    int below;
    return fixed_of(x, E, below);
}

// The FP64 number nearest to (T 2^32 + r) 2^(E - 1084)
__device__ __forceinline__ double fixed_to_f64(long long T, unsigned r, int E) {
    const bool neg = T < 0;
    if (neg) {
        r = 0u - r;
        T = ~T + (r == 0u ? 1 : 0);
    }
    unsigned w2 = (unsigned)((unsigned long long)T >> 32), w1 = (unsigned)T, w0 = r;
    int lead = 95;
    if (w2 == 0u) {
        w2 = w1; w1 = w0; w0 = 0u; lead -= 32;
        if (w2 == 0u) { w2 = w1; w1 = 0u; lead -= 32; }
    }
    const int lz = __clz((int)w2);
    lead -= lz;
    const unsigned h = __funnelshift_l(w1, w2, lz), l = __funnelshift_l(w0, w1, lz);
    const unsigned long long m = ((unsigned long long)h << 32) | l;
    unsigned long long b = (m >> 11) + ((m >> 10) & 1ull);       // 53 bits, rounded
    b += (unsigned long long)(unsigned)(E + lead - 62) << 52;    // the leading bit adds 1 to the exponent
    if (w2 == 0u) b = 0ull;
    return __longlong_as_double((long long)(b | (neg ? 0x8000000000000000ull : 0ull)));
}

// 12 times the fourth-order central difference, (a - d) - 8 (b - c) for a, b, c, d = f[-2], f[-1], f[1],
// f[2] (viscous.jl:29-42), rounded once: no FP64 instruction instead of four (the 1/12 goes into a
// metric factor). Values within 2^9 of the largest enter exactly. Smaller ones are truncated: at most 17
// units of 2^-61 of the largest's power of two, about half a unit in the last place of a result of 2^-4 of
// it. `plain` is cleared where something was truncated (a zero beside other values is counted in) and
// the result is smaller than that, the large values having cancelled, and for values outside 2^-823 ..
// 2^877 (infinities and NaN among them): the caller then takes difference12_fp64 for all of its
// differences, in a block of its own (a fallback beside each call is turned into predicated FP64
// instructions, which hold the pipe although no lane runs them). 0.4% of the warps take it on the ramp
// and the plate.
__device__ __forceinline__ F64 difference12(double a, double b, double c, double d, bool& plain) {
    const unsigned top = max(max((unsigned)__double2hiint(a) & 0x7fffffffu, (unsigned)__double2hiint(b) & 0x7fffffffu),
                             max((unsigned)__double2hiint(c) & 0x7fffffffu, (unsigned)__double2hiint(d) & 0x7fffffffu));
    const int E = (int)(top >> 20);
    int da, db, dc, dd;
    const long long x = fixed_of(a, E, da) - fixed_of(d, E, dd), y = fixed_of(b, E, db) - fixed_of(c, E, dc);  // below 2^63
    const long long l = (long long)(unsigned)x - 8ll * (long long)(unsigned)y;
    const double r = fixed_to_f64((x >> 32) - 8ll * (y >> 32) + (l >> 32), (unsigned)l, E);
    const bool cut = max(max(da, db), max(dc, dd)) > 9;
    const bool small = ((unsigned)__double2hiint(r) & 0x7fffffffu) < (top & 0x7ff00000u) - (4u << 20);
    // no branches: twelve of these run side by side
    plain &= (top == 0u) | (((unsigned)(E - 200) <= 1700u) & !(cut & small));
    return f64(top == 0u ? 0.0 : r);
}
__device__ __forceinline__ F64 difference12_fp64(double a, double b, double c, double d) {
    return (f64(a) - f64(d)) - F64(8.0) * (f64(b) - f64(c));
}

// The sums of a strip that may not be formed from values truncated at 2^-62 of its largest, of those
// in `want`: sum f is safe when one of its two central values (coefficients of 214/420 and above)
// lies within 2^LIN_SPREAD of the largest. near(f): bit pattern of the larger of them, without sign.
template <class NEAR> __device__ __forceinline__ unsigned beyond_spread(int E, unsigned want, NEAR near) {
    const unsigned least = (unsigned)(E - LIN_SPREAD) << 20;
    unsigned far = 0u;
#pragma unroll
    for (int f = 0; f < LIN_STRIP; f++)
        if (near(f) < least) far |= 1u << f;
    return far & want;
}

// The sums f whose values f .. f + 7 all have their bit in `exact`
__device__ __forceinline__ unsigned whole_windows(unsigned exact) {
    unsigned whole = exact;
#pragma unroll
    for (int k = 1; k < 8; k++) whole &= exact >> k;
    return whole;
}
// Whether a value enters a strip of exponent E without loss: 2^-9 of the largest or more, or zero
__device__ __forceinline__ bool enters_exactly(double x, int E) {
    const unsigned a = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return (a | (unsigned)__double2loint(x)) == 0u || (int)(a >> 20) >= E - 9;
}

// The two one-sided linear combinations of one array on a strip: up[f] = sum_k lin[k] V(t0 + f + k) and
// down[f] = sum_k lin[k] V(t0 + f + 7 - k), f = 0..4 (the left and right states of finite-volume faces;
// the transpose of the linear faces in the reverse sweeps). V(p) is read at p = t0 .. t0 + 11; both
// sums of f have V(t0 + f + 3) and V(t0 + f + 4) at their centre. put(f, up, down) takes those of the f in
// `want`.
template <class VF, class PUT>
__device__ __forceinline__ void linear_strip_both(const DevParams& P, int t0, unsigned want, VF V, PUT put) {
    constexpr int NV = LIN_STRIP + 7;
    unsigned top = 0u, low = 0u, mid[LIN_STRIP + 1];  // mid[i]: magnitude at t0 + 3 + i
#pragma unroll
    for (int p = 0; p < NV; p++) {
        const double v = V(t0 + p);
        const unsigned a = (unsigned)__double2hiint(v) & 0x7fffffffu;
        low |= (unsigned)__double2loint(v);
        top = max(top, a);
        if (p >= 3 && p <= LIN_STRIP + 3) mid[p - 3] = a;
    }
    if ((top | low) == 0u) {
#pragma unroll
        for (int f = 0; f < LIN_STRIP; f++)
            if (want >> f & 1u) put(f, 0.0, 0.0);
        return;
    }
    const int E = (int)(top >> 20);
    unsigned far = want;  // the sums to form in FP64
    if (E >= 200 && E <= 1900) {
        far = beyond_spread(E, want, [&](int f) { return max(mid[f], mid[f + 1]); });
        if (far) {
            unsigned exact = 0u;
            int m[NV];  // magnitudes
#pragma unroll
            for (int p = 0; p < NV; p++) {
                const double v = V(t0 + p);
                m[p] = __double2hiint(v) & 0x7fffffff;
                exact |= (unsigned)enters_exactly(v, E) << p;
            }
            far &= ~whole_windows(exact);
            // values away from the centre count as much less as their coefficients: 38/420 and above
            // beside it, 4/420 and above beyond (both sums; for any blend)
#pragma unroll
            for (int f = 0; f < LIN_STRIP; f++)
                if (max(max(m[f + 2], m[f + 5]) - (3 << 20), max(m[f + 1], m[f + 6]) - (6 << 20)) >= (E - 6) << 20)
                    far &= ~(1u << f);
        }
    }
    if (far != want) {
        long long x[NV];
#pragma unroll
        for (int p = 0; p < NV; p++) x[p] = fixed_of(V(t0 + p), E);
#pragma unroll
        for (int f = 0; f < LIN_STRIP; f++) {
            double both[2];
#pragma unroll
            for (int side = 0; side < 2; side++) {
                long long h = 0;
                unsigned long long lp = 0ull, ln = 0ull;
#pragma unroll
                for (int k = 0; k < 7; k++) {
                    const long long v = x[side == 0 ? f + k : f + 7 - k];
                    h += (long long)(int)(v >> 32) * P.lin_c[k];
                    if (k == 0 || k == 2 || k == 5) ln += (unsigned long long)(unsigned)v * (unsigned)(-P.lin_c[k]);
                    else lp += (unsigned long long)(unsigned)v * (unsigned)P.lin_c[k];
                }
                const long long l = (long long)(lp - ln);
                both[side] = F64(f64(fixed_to_f64(h + (l >> 32), (unsigned)l, E)) * F64(P.lin_s)).v;
            }
            if ((want & ~far) >> f & 1u) put(f, both[0], both[1]);
        }
    }
    for (; far; far &= far - 1u) {
        const int f = __ffs((int)far) - 1;
        double a = 0.0, b = 0.0;
#pragma unroll
        for (int k = 0; k < 7; k++) {
            a += P.cd.lin[k] * V(t0 + f + k);
            b += P.cd.lin[k] * V(t0 + f + 7 - k);
        }
        put(f, a, b);
    }
}

// Of the five faces t0 .. t0+4 of one line and component those in `want`: put(f, sum_k lin[k]
// (Fp(t+k) + Fm(t+7-k))), t = t0 + f. FP / FM(p) read the split fluxes at position p; positions past
// `last` were not filled and count as zero (no face in `want` reads them).
template <class FPA, class FMA, class PUT>
__device__ __forceinline__ void linear_strip(const DevParams& P, int t0, int last, unsigned want, FPA FP, FMA FM, PUT put) {
    constexpr int NV = LIN_STRIP + 6;
    // the strip's values V(q), q = 0..NV-1: Fp at t0 + q, Fm at t0 + 1 + q
    auto P_ = [&](int q) { return t0 + q <= last ? FP(t0 + q) : 0.0; };
    auto M_ = [&](int q) { return t0 + 1 + q <= last ? FM(t0 + 1 + q) : 0.0; };
    // FP64 bit patterns without their sign order like the magnitudes; mid[i]: at position t0 + 3 + i
    unsigned top = 0u, low = 0u, mid[LIN_STRIP + 1];
#pragma unroll
    for (int i = 0; i <= LIN_STRIP; i++) mid[i] = 0u;
#pragma unroll
    for (int q = 0; q < NV; q++) {
        const double v = P_(q), w = M_(q);
        const unsigned a = (unsigned)__double2hiint(v) & 0x7fffffffu, b = (unsigned)__double2hiint(w) & 0x7fffffffu;
        low |= (unsigned)__double2loint(v) | (unsigned)__double2loint(w);
        top = max(top, max(a, b));
        if (q >= 3 && q <= LIN_STRIP + 3) mid[q - 3] = max(mid[q - 3], a);
        if (q >= 2 && q <= LIN_STRIP + 2) mid[q - 2] = max(mid[q - 2], b);
    }
    if ((top | low) == 0u) {
#pragma unroll
        for (int f = 0; f < LIN_STRIP; f++)
            if (want >> f & 1u) put(f, 0.0);
        return;
    }
    const int E = (int)(top >> 20);
    unsigned far = want;  // the faces to sum in FP64
    if (E >= 200 && E <= 1900) {
        far = beyond_spread(E, want, [&](int f) { return max(mid[f], mid[f + 1]); });
        if (far) {
            bool exact = true;
#pragma unroll
            for (int q = 0; q < NV; q++) exact = exact && enters_exactly(P_(q), E) && enters_exactly(M_(q), E);
            if (exact) far = 0u;
        }
    }
    if (far != want) {
        // sums of the upper words (signed), and of the lower words under the positive and the
        // negative coefficients (0, 2 and 5)
        long long hs[LIN_STRIP];
        unsigned long long lp[LIN_STRIP], ln[LIN_STRIP];
#pragma unroll
        for (int f = 0; f < LIN_STRIP; f++) { hs[f] = 0; lp[f] = ln[f] = 0ull; }
        auto add = [&](int f, int k, int vh, unsigned vl) {
            hs[f] += (long long)vh * P.lin_c[k];
            if (k == 0 || k == 2 || k == 5) ln[f] += (unsigned long long)vl * (unsigned)(-P.lin_c[k]);
            else lp[f] += (unsigned long long)vl * (unsigned)P.lin_c[k];
        };
#pragma unroll
        for (int q = 0; q < NV; q++) {
            const long long v = fixed_of(P_(q), E), w = fixed_of(M_(q), E);
#pragma unroll
            for (int f = 0; f < LIN_STRIP; f++) {
                const int kp = q - f, km = 6 + f - q;  // Fp(t + kp), Fm(t + 7 - km)
                if (kp >= 0 && kp < 7) add(f, kp, (int)(v >> 32), (unsigned)v);
                if (km >= 0 && km < 7) add(f, km, (int)(w >> 32), (unsigned)w);
            }
        }
#pragma unroll
        for (int f = 0; f < LIN_STRIP; f++) {
            const long long l = (long long)(lp[f] - ln[f]);
            const double r = F64(f64(fixed_to_f64(hs[f] + (l >> 32), (unsigned)l, E)) * F64(P.lin_s)).v;
            if ((want & ~far) >> f & 1u) put(f, r);
        }
    }
    for (; far; far &= far - 1u) {
        const int f = __ffs((int)far) - 1, t = t0 + f;
        put(f, P.cd.lin[0] * (FP(t) + FM(t + 7)) + P.cd.lin[1] * (FP(t + 1) + FM(t + 6)) +
                   P.cd.lin[2] * (FP(t + 2) + FM(t + 5)) + P.cd.lin[3] * (FP(t + 3) + FM(t + 4)) +
                   P.cd.lin[4] * (FP(t + 4) + FM(t + 3)) + P.cd.lin[5] * (FP(t + 5) + FM(t + 2)) +
                   P.cd.lin[6] * (FP(t + 6) + FM(t + 1)));
    }
}

}  // namespace f3d
