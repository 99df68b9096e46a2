// k_weno_vjp.cu — reverse of the listed WENO7 / WENO5 faces (k_weno.cu's lists).
//
// What bounds it: the FP64 pipe, as in the forward faces, and the same imbalance: reversed within the
// tiles of k_sweep_vjp, the WENO faces (~3000 FP64 instructions and 70 shared-memory atomics each)
// filled one or two of a tile's warps while the others waited, and 234 registers a thread left six
// warps an SM (characteristic xi sweep of the 256x64x64 shock tube: 1.45 ms, eta and zeta 1.10). Here
// blocks of five warps take 32 faces of one kind at a time:
//   1  the split fluxes of the eight stencil cells (one cell of 32 faces a warp), the face basis and
//      the face's flux cotangents;
//   2  one characteristic field (component) a warp: its projections, the reverse of both sides' WENO,
//      the cotangents of its row of L;
//   3  one flux component a warp: the split-flux cotangents L^T of the fields' stencil cotangents, added
//      to ten planes in global memory, which k_sweep_vjp reverses through the split with its own;
//      one warp takes the fields' and rows' cotangents back to the face state (char_state_vjp).
#include "f3d_adjoint.cuh"
#include "f3d_face.cuh"

namespace f3d {

// Reverse of one side of WENO7 in the forms of weno7_sums (f3d_flux.cuh): V(k) the stencil, g the
// cotangent of 12 times its value; returns 12 times the value, Vb the stencil's cotangents.
// With w_k = alpha_k / D the value's cotangents are q_k: g w_k, and through the bases b_k = t_k^2,
// t_k = e_k + sigma_k I_k: I_k-bar = -2 sigma_k g w_k (q_k - N/D) / t_k. The weights and 1 / t_k come from
// products of the b_k and one reciprocal of them all; where that product leaves the range (t above ~1e38,
// fluxes above ~1e18) from four quotients instead, which hold to t ~ 1e154.
__device__ __forceinline__ F64 weno7_reverse(const F64 v[7], F64 s0, F64 g, F64 Vb[7]) {
    using C = W7Ldl<double>;
    const double rw[4] = {1.0, 0.28867513459481287, 0.23570226039551584, 0.5};  // 1 / sqrt(1, 12, 18, 4)
    F64 d[6], y1[4], z2[4], z3[4], sg[4], t[4], b[4];
#pragma unroll
    for (int k = 0; k < 6; k++) d[k] = v[k + 1] - v[k];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        y1[k] = d[k] + F64(C::a(k)) * d[k + 1] + F64(C::b(k)) * d[k + 2];
        const F64 y2 = d[k + 1] + F64(C::c(k)) * d[k + 2];
        z2[k] = F64(C::D2(k) / C::D1(k)) * y2;
        z3[k] = F64(C::D3(k) / C::D1(k)) * d[k + 2];
        const F64 I = y1[k] * y1[k] + z2[k] * y2 + z3[k] * d[k + 2];
        sg[k] = F64(C::D1(k) * rw[k]) * s0;
        t[k] = F64(1e-20 * rw[k]) + sg[k] * I;
        b[k] = t[k] * t[k];
    }
    const F64 q[4] = {F64(13.0) * d[2] + F64(-10.0) * d[1] + F64(3.0) * d[0], (F64(4.0) * d[2] - d[1]) + F64(3.0) * d[3],
                      (F64(6.0) * d[3] + d[2]) - d[4], (F64(-4.0) * d[4] + d[5]) + F64(9.0) * d[3]};
    const F64 p01 = b[0] * b[1], p23 = b[2] * b[3], all = p01 * p23;
    F64 al[4] = {p23 * b[1], p23 * b[0], p01 * b[3], p01 * b[2]}, it[4];  // alpha_k and 1 / t_k
    if (recip_range(all.v)) {
        const F64 rP = recip_step(all.v);
#pragma unroll
        for (int k = 0; k < 4; k++) it[k] = t[k] * (al[k] * rP);  // t_k / b_k
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            it[k] = f64(1.0 / t[k].v);
            al[k] = it[k] * it[k];
        }
    }
    const F64 rD = recip(al[0] + al[1] + al[2] + al[3]);
    const F64 Q = (al[0] * q[0] + al[1] * q[1] + al[2] * q[2] + al[3] * q[3]) * rD;
    const F64 gm = F64(-2.0) * g;
    F64 qb[4], db[6];
#pragma unroll
    for (int k = 0; k < 6; k++) db[k] = f64(0.0);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const F64 w = al[k] * rD;
        qb[k] = g * w;
        const F64 Ib = ((gm * sg[k]) * (w * (q[k] - Q))) * it[k];
        const F64 h = Ib + Ib, y1b = y1[k] * h, y2b = z2[k] * h;
        db[k] += y1b;
        db[k + 1] = (db[k + 1] + y2b) + F64(C::a(k)) * y1b;
        db[k + 2] = ((db[k + 2] + z3[k] * h) + F64(C::b(k)) * y1b) + F64(C::c(k)) * y2b;
    }
    db[0] += F64(3.0) * qb[0];
    db[1] = (db[1] - qb[1]) + F64(-10.0) * qb[0];
    db[2] = ((db[2] + qb[2]) + F64(13.0) * qb[0]) + F64(4.0) * qb[1];
    db[3] = ((db[3] + F64(3.0) * qb[1]) + F64(6.0) * qb[2]) + F64(9.0) * qb[3];
    db[4] = (db[4] - qb[2]) + F64(-4.0) * qb[3];
    db[5] += qb[3];
    Vb[0] = -db[0];
#pragma unroll
    for (int k = 1; k < 6; k++) Vb[k] = db[k - 1] - db[k];
    Vb[6] = db[5];
    Vb[3] += F64(12.0) * g;
    return Q + F64(12.0) * v[3];
}

// The same of WENO5 (weno5_sums): v the five points, g the cotangent of 6 times the value
__device__ __forceinline__ F64 weno5_reverse(const F64 v[5], F64 s0, F64 g, F64 Vb[5]) {
    const double rw[3] = {1.0, 0.40824829046386302, 0.57735026918962576};  // 1 / sqrt(1, 6, 3)
    F64 d[4], t[3], b[3], sg[3];
#pragma unroll
    for (int k = 0; k < 4; k++) d[k] = v[k + 1] - v[k];
    const F64 s[3] = {d[1] - d[0], d[2] - d[1], d[3] - d[2]};
    const F64 f[3] = {F64(3.0) * d[1] - d[0], d[2] + d[1], d[3] + F64(-3.0) * d[2]};
    const F64 k13 = 13.0 / 3.0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        sg[k] = F64(3.0 * rw[k]) * s0;
        t[k] = F64(1e-16 * rw[k]) + sg[k] * ((k13 * s[k]) * s[k] + f[k] * f[k]);
        b[k] = t[k] * t[k];
    }
    const F64 q[3] = {F64(5.0) * d[1] + F64(-2.0) * d[0], d[1] + F64(2.0) * d[2], F64(4.0) * d[2] - d[3]};
    const F64 all = b[0] * b[1] * b[2];
    F64 al[3] = {b[1] * b[2], b[0] * b[2], b[0] * b[1]}, it[3];
    if (recip_range(all.v)) {
        const F64 rP = recip_step(all.v);
#pragma unroll
        for (int k = 0; k < 3; k++) it[k] = t[k] * (al[k] * rP);
    } else {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            it[k] = f64(1.0 / t[k].v);
            al[k] = it[k] * it[k];
        }
    }
    const F64 rD = recip(al[0] + al[1] + al[2]);
    const F64 Q = (al[0] * q[0] + al[1] * q[1] + al[2] * q[2]) * rD;
    const F64 gm = F64(-2.0) * g;
    F64 qb[3], sb[3], fb[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const F64 w = al[k] * rD;
        qb[k] = g * w;
        const F64 Ib = ((gm * sg[k]) * (w * (q[k] - Q))) * it[k];
        const F64 h = Ib + Ib;
        sb[k] = (k13 * s[k]) * h;
        fb[k] = f[k] * h;
    }
    F64 db[4];
    db[0] = ((F64(-2.0) * qb[0]) - sb[0]) - fb[0];
    db[1] = (((F64(5.0) * qb[0] + qb[1]) + sb[0]) - sb[1]) + F64(3.0) * fb[0] + fb[1];
    db[2] = (((F64(2.0) * qb[1] + sb[1]) - sb[2]) + fb[1]) + F64(-3.0) * fb[2] + F64(4.0) * qb[2];
    db[3] = (sb[2] - qb[2]) + fb[2];
    Vb[0] = -db[0];
#pragma unroll
    for (int k = 1; k < 4; k++) Vb[k] = db[k - 1] - db[k];
    Vb[4] = db[3];
    Vb[2] += F64(6.0) * g;
    return Q + F64(6.0) * v[2];
}

// Entry e of right eigenvector k in the order of char_right_row
__device__ __forceinline__ F64 right_entry(const CharBasis<F64>& b, int k, int e) {
    const F64 ae = e == 0 ? f64(1.0) : e == 1 ? b.u : e == 2 ? b.v : e == 3 ? b.w : b.H;
    const F64 ne = e == 0 ? f64(0.0) : e == 1 ? b.nx : e == 2 ? b.ny : e == 3 ? b.nz : b.qn;
    if (k == 0) return ae - b.c * ne;
    if (k == 2) return ae + b.c * ne;
    if (k == 1) return e == 4 ? b.q2 : ae;
    if (k == 3) return e == 0 ? f64(0.0) : e == 1 ? b.lx : e == 2 ? b.ly : e == 3 ? b.lz : b.ql;
    return e == 0 ? f64(0.0) : e == 1 ? b.mx : e == 2 ? b.my : e == 3 ? b.mz : b.qm;
}

// Cotangents (u, v, w, T) of the face state from those of the right-eigenvector products (flux
// cotangent Fb, characteristic fluxes f) and of the rows of L: the reverse of char_basis with the
// metric row held (the tangent basis depends on it alone).
template <class LB>
__device__ __forceinline__ void char_state_vjp(const Cst<double>& K, const CharBasis<F64>& b, const F64 Fb[5],
                                               const F64 f[5], LB lb, F64 out[4]) {
    const F64 K2 = b.K2, Kc = b.Kc, c2 = b.c2;
    const F64 rc = c2 + c2, gT = b.c * b.c;
    // rows 0, 2 (acoustic), 1 (entropy), 3, 4 (shear) of L
    F64 K2b = lb(0, 4) + lb(2, 4), q2b, qnb, c2b, ub, vb, wb, Kcb;
    const F64 a0 = lb(0, 0) + lb(2, 0), a1 = lb(0, 1) + lb(2, 1), a2 = lb(0, 2) + lb(2, 2), a3 = lb(0, 3) + lb(2, 3);
    const F64 s0 = lb(0, 0) - lb(2, 0), s1 = lb(0, 1) - lb(2, 1), s2 = lb(0, 2) - lb(2, 2), s3 = lb(0, 3) - lb(2, 3);
    K2b = K2b + a0 * b.q2 - a1 * b.u - a2 * b.v - a3 * b.w;
    c2b = b.qn * s0 - b.nx * s1 - b.ny * s2 - b.nz * s3;
    q2b = K2 * a0 - Kc * lb(1, 0);
    qnb = c2 * s0;
    ub = Kc * lb(1, 1) - K2 * a1;
    vb = Kc * lb(1, 2) - K2 * a2;
    wb = Kc * lb(1, 3) - K2 * a3;
    Kcb = (b.u * lb(1, 1) - lb(1, 4)) + b.v * lb(1, 2) + b.w * lb(1, 3) - b.q2 * lb(1, 0);
    F64 qlb = -lb(3, 0), qmb = -lb(4, 0);
    // out = R f
    const F64 s012 = f[0] + f[1] + f[2], d20 = f[2] - f[0];
    ub += s012 * Fb[1];
    vb += s012 * Fb[2];
    wb += s012 * Fb[3];
    const F64 cb = d20 * (b.nx * Fb[1] + b.ny * Fb[2] + b.nz * Fb[3] + b.qn * Fb[4]);
    qnb += (b.c * d20) * Fb[4];
    const F64 Hb = (f[0] + f[2]) * Fb[4];
    q2b += f[1] * Fb[4];
    qlb += f[3] * Fb[4];
    qmb += f[4] * Fb[4];
    // K2 = Kc/2, Kc = (g-1) rc^2, c2 = rc/2, c = gT rc, H = gT/(g-1) + q2, rc = gT^(-1/2), gT = g Rg T
    Kcb += F64(0.5) * K2b;
    const F64 rcb = (Kcb * F64(2.0 * K.gm1)) * rc + F64(0.5) * c2b + cb * gT;
    const F64 gTb = cb * rc + Hb * F64(K.inv_gm1) - (rcb * F64(0.5)) * ((rc * rc) * rc);
    q2b += Hb;
    out[0] = ub + q2b * b.u + qnb * b.nx + qlb * b.lx + qmb * b.mx;
    out[1] = vb + q2b * b.v + qnb * b.ny + qlb * b.ly + qmb * b.my;
    out[2] = wb + q2b * b.w + qnb * b.nz + qlb * b.lz + qmb * b.mz;
    out[3] = gTb * F64(K.grg);
}

constexpr int WV_WARPS = 5, WV_FACES = 32;
struct WenoVjpSmem {
    double f[10 * 8 * WV_FACES];          // Fp (5) and Fm (5) of the eight stencil cells
    CharBasis<F64> basis[WV_FACES];
    F64 s0[WV_FACES];
    F64 Fb[5 * WV_FACES];                 // cotangents of the face flux
    F64 flux[5 * WV_FACES];               // characteristic fluxes
    F64 L[25 * WV_FACES];                 // rows of L
    F64 lb[25 * WV_FACES];                // their cotangents
    F64 Vb[5 * 14 * WV_FACES];            // stencil cotangents of the fields, plus and minus side
};

template <bool CHAR>
__global__ void __launch_bounds__(WV_WARPS * 32, 3) k_weno_vjp(const WenoVjpArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WenoVjpSmem& sm = *reinterpret_cast<WenoVjpSmem*>(smem_raw);
    const DevParams& P = a.P;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const long long pl = P.plane;
    int nf[6], nchunk = 0;  // WENO7 and WENO5 faces of the directions taken here
#pragma unroll
    for (int li = 0; li < 6; li++) {
        nf[li] = li % 3 >= a.d0 && li % 3 < a.d1 ? (int)a.w.count[li] : 0;
        nchunk += (nf[li] + WV_FACES - 1) / WV_FACES;
    }
    if (blockIdx.x == 0 && (int)threadIdx.x < 3 && (int)threadIdx.x >= a.d0 && (int)threadIdx.x < a.d1)
        a.any[threadIdx.x] = a.w.count[threadIdx.x] + a.w.count[threadIdx.x + 3];
    for (int ch = blockIdx.x; ch < nchunk; ch += gridDim.x) {
        int li = 0, first = 0;
        {
            int left = ch;
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const int n = (nf[q] + WV_FACES - 1) / WV_FACES;
                if (left >= 0 && left < n) { li = q; first = left * WV_FACES; }
                left -= n;
            }
        }
        const int d = li % 3, k0 = first + lane;
        const bool w7 = li < 3, on = k0 < (int)a.w.count[li];
        const long long stride = d == 0 ? 1 : (d == 1 ? (long long)P.nxt : (long long)P.nxt * P.nyt);
        const long long cl = on ? (long long)a.w.list[d * pl + (w7 ? (long long)k0 : pl - 1 - k0)] : 0ll, cr = cl + stride;
        const double *A0 = a.A[3 * d], *A1 = a.A[3 * d + 1], *A2 = a.A[3 * d + 2], *S = a.S[d];
        const double *H0 = a.H[3 * d], *H1 = a.H[3 * d + 1], *H2 = a.H[3 * d + 2];
        if (on) {
            for (int p = wp; p < 8; p += WV_WARPS) {
                if (!w7 && (p == 0 || p == 7)) continue;  // WENO5 reads positions 1 .. 6
                const long long c = cl + (p - 3) * stride;
                F64 q[6], fp[5], fm[5];
#pragma unroll
                for (int n = 0; n < 6; n++) q[n] = f64(a.Q[c + n * pl]);
                split_cell<F64>(P.split, P.cd, q, f64(a.csnd[c]), f64(A0[c]), f64(A1[c]), f64(A2[c]), f64(H0[c]),
                                f64(H1[c]), f64(H2[c]), f64(S[c]), fp, fm);
#pragma unroll
                for (int n = 0; n < 5; n++) {
                    sm.f[(n * 8 + p) * WV_FACES + lane] = fp[n].v;
                    sm.f[((n + 5) * 8 + p) * WV_FACES + lane] = fm[n].v;
                }
            }
            if (wp == 3) {
                const F64 s0 = F64(2.0) / (f64(S[cl]) + f64(S[cr]));
                sm.s0[lane] = s0;
                auto as = [](const double* p) { return reinterpret_cast<const F64*>(p); };
                if (CHAR) char_basis<F64>(P, as(a.Q), as(A0), as(A1), as(A2), s0, cl, cr, sm.basis[lane]);
            }
            if (wp == 4) {  // face f is the left face of interior cell f and the right face of f - 1
                int g[3];
                split3(cl, P.dnxt, P.dnyt, g[0], g[1], g[2]);
                const int N = d == 0 ? P.nx : (d == 1 ? P.ny : P.nz);
                const bool has_l = g[d] >= NG, has_r = g[d] + 1 < N + NG;
                const F64 jr = f64(has_r ? a.J[cr] : 0.0), jl = f64(has_l ? a.J[cl] : 0.0);
                for (int n = 0; n < 5; n++)
                    sm.Fb[n * WV_FACES + lane] = jr * f64(has_r ? a.Lb[cr + n * pl] : 0.0) -
                                                 jl * f64(has_l ? a.Lb[cl + n * pl] : 0.0);
            }
        }
        __syncthreads();
        const F64 unit = w7 ? F64(1.0 / 12.0) : F64(1.0 / 6.0);
        if (on) {
            const F64 s0 = sm.s0[lane];
            F64 l[5], fb;
            if (CHAR) {
                char_left_row<F64>(sm.basis[lane], wp, l);
                fb = sm.Fb[lane] * right_entry(sm.basis[lane], wp, 0);
#pragma unroll
                for (int e = 1; e < 5; e++) fb += sm.Fb[e * WV_FACES + lane] * right_entry(sm.basis[lane], wp, e);
            } else {
                fb = sm.Fb[wp * WV_FACES + lane];
            }
            const F64 g = fb * unit;
            // a component without a cotangent has none to pass on, whatever its stencil holds
            const bool none = !CHAR && (__double_as_longlong(fb.v) << 1) == 0;
            if (none)
#pragma unroll
                for (int k = 0; k < 14; k++) sm.Vb[(wp * 14 + k) * WV_FACES + lane] = f64(0.0);
            F64 lb[5], both = f64(0.0);
#pragma unroll
            for (int e = 0; e < 5; e++) lb[e] = f64(0.0);
#pragma unroll 1
            for (int side = none ? 2 : 0; side < 2; side++) {
                const double* f = sm.f + (side == 0 ? 0 : 40 * WV_FACES) + lane;
                // upwind order: position k of the plus side, 7 - k of the minus side
                auto at = [&](int k) { return (side == 0 ? k : 7 - k) * WV_FACES; };
                auto value = [&](int k) {
                    const int o = at(k);
                    if (!CHAR) return f64(f[wp * 8 * WV_FACES + o]);
                    F64 r = l[0] * f64(f[o]);
#pragma unroll
                    for (int e = 1; e < 5; e++) r += l[e] * f64(f[e * 8 * WV_FACES + o]);
                    return r;
                };
                F64* out = sm.Vb + ((wp * 14 + side * 7) * WV_FACES + lane);
                auto finish = [&](int k, F64 vb) {
                    out[k * WV_FACES] = vb;
                    if (CHAR) {
                        const int o = at(k);
#pragma unroll
                        for (int e = 0; e < 5; e++) lb[e] += f64(f[e * 8 * WV_FACES + o]) * vb;
                    }
                };
                if (w7) {
                    F64 V[7], Vb[7];
#pragma unroll
                    for (int k = 0; k < 7; k++) V[k] = value(k);
                    both += weno7_reverse(V, s0, g, Vb);
#pragma unroll
                    for (int k = 0; k < 7; k++) finish(k, Vb[k]);
                } else {
                    F64 V[5], Vb[5];
#pragma unroll
                    for (int k = 0; k < 5; k++) V[k] = value(k + 1);
                    both += weno5_reverse(V, s0, g, Vb);
#pragma unroll
                    for (int k = 0; k < 5; k++) finish(k + 1, Vb[k]);
                }
            }
            if (CHAR) {
                sm.flux[wp * WV_FACES + lane] = both * unit;
#pragma unroll
                for (int e = 0; e < 5; e++) {
                    sm.L[(wp * 5 + e) * WV_FACES + lane] = l[e];
                    sm.lb[(wp * 5 + e) * WV_FACES + lane] = lb[e];
                }
            }
        }
        __syncthreads();
        if (on) {
            const int kb = w7 ? 0 : 1, ke = w7 ? 7 : 6;
#pragma unroll 1
            for (int side = 0; side < 2; side++) {
                double* Sb = a.Sb + ((d - a.d0) * 10 + side * 5 + wp) * pl + cl;
                for (int k = kb; k < ke; k++) {
                    F64 v;
                    if (CHAR) {
                        v = sm.L[wp * WV_FACES + lane] * sm.Vb[(side * 7 + k) * WV_FACES + lane];
#pragma unroll
                        for (int n = 1; n < 5; n++)
                            v += sm.L[(n * 5 + wp) * WV_FACES + lane] * sm.Vb[(n * 14 + side * 7 + k) * WV_FACES + lane];
                    } else {
                        v = sm.Vb[(wp * 14 + side * 7 + k) * WV_FACES + lane];
                    }
                    if (__double_as_longlong(v.v) << 1) atomicAdd(Sb + ((side == 0 ? k : 7 - k) - 3) * stride, v.v);
                }
            }
            if (CHAR && wp == ch % WV_WARPS) {
                F64 Fb[5], f[5], out[4];
#pragma unroll
                for (int n = 0; n < 5; n++) {
                    Fb[n] = sm.Fb[n * WV_FACES + lane];
                    f[n] = sm.flux[n * WV_FACES + lane];
                }
                char_state_vjp(P.cd, sm.basis[lane], Fb, f, [&](int k, int e) { return sm.lb[(k * 5 + e) * WV_FACES + lane]; },
                               out);
                const int qv[4] = {1, 2, 3, 5};  // the face state is the mean of the two cells'
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const double h = F64(F64(0.5) * out[k]).v;
                    atomicAdd(&a.Qb[cl + qv[k] * pl], h);
                    atomicAdd(&a.Qb[cr + qv[k] * pl], h);
                }
            }
        }
        __syncthreads();
    }
}

cudaError_t weno_vjp_configure() {
    cudaError_t e = cudaFuncSetAttribute(k_weno_vjp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WenoVjpSmem));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_weno_vjp<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WenoVjpSmem));
}

cudaError_t launch_weno_vjp(const WenoVjpArgs& a, int sms, cudaStream_t st) {
    const DevParams& P = a.P;
    const long long most = (long long)P.nx * P.ny * P.nz / WV_FACES + 1;
    const int blocks = most < 3 * sms ? (int)most : 3 * sms;
    if (P.character) k_weno_vjp<true><<<blocks, WV_WARPS * 32, sizeof(WenoVjpSmem), st>>>(a);
    else k_weno_vjp<false><<<blocks, WV_WARPS * 32, sizeof(WenoVjpSmem), st>>>(a);
    return cudaGetLastError();
}

}  // namespace f3d
