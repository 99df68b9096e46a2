// k_viscous.cu — viscous and heat fluxes (viscous.jl:1-133, the LES closures included).
//
// One thread per cell of the box 2..Nt-3 (0-based full index), which is cells 3..Nt-2 of
// the reference. Fourth-order central differences of u, v, w, T in xi, eta, zeta, the
// chain rule with the J^-1-scaled metrics and J, Sutherland viscosity, Stokes stress and
// Fourier heat flux, projected on the three metric rows. Output arrays have the
// reference's Fv_x/Fv_y/Fv_z shape ((Nt-4)^3 x 4) with Fv index = cell index - 2.
//
// What bounds it: in FP64 the FP64 pipe (89% busy; 224 bytes a cell would take 0.6 ms on the
// 512x256x128 ramp). Differences as integers, the metrics times J/12 once and the viscosity through
// one reciprocal root: 5.8 -> 3.7 ms a stage there, 118 -> 81 us on the plate 125x61x37. 128 threads, five
// blocks per SM (96 registers): the ramp's step 45.1 ms, 45.3 at four blocks (128 registers), 46.6 with the
// compiler's 138, which the look at cancelled differences asks for (difference12).
#include "f3d_fixed.cuh"

namespace f3d {

__device__ __forceinline__ F64 cube_root(F64 x) { return f64(cbrt(x.v)); }
__device__ __forceinline__ float cube_root(float x) { return cbrtf(x); }

template <class R>
__global__ void __launch_bounds__(128, 5) k_viscous(const DevParams P, const R* __restrict__ Q, const R* m0,
                                                 const R* m1, const R* m2, const R* m3, const R* m4, const R* m5,
                                                 const R* m6, const R* m7, const R* m8, const R* __restrict__ J,
                                                 R* Fvx, R* Fvy, R* Fvz) {
    const int vxt = P.nxt - 4, vyt = P.nyt - 4, vzt = P.nzt - 4;
    const long long vpl = (long long)vxt * vyt * vzt;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= vpl) return;
    int vi, vj, vk;
    split3(t, P.dvxt, P.dvyt, vi, vj, vk);
    const long long c = lin3(P, vi + 2, vj + 2, vk + 2);
    const long long pl = P.plane, sy = P.nxt, sz = (long long)P.nxt * P.nyt;
    const auto& K = cst<R>(P);
    using A = typename Arith<R>::type;
    const A xx = arith(m0[c]), xy = arith(m1[c]), xz = arith(m2[c]);
    const A ex = arith(m3[c]), ey = arith(m4[c]), ez = arith(m5[c]);
    const A zx = arith(m6[c]), zy = arith(m7[c]), zz = arith(m8[c]);
    const A Jac = arith(J[c]);
    const A T = arith(Q[c + 5 * pl]);
    A mu;
    if constexpr (sizeof(R) == 8) {
        // C_s T^(3/2) / (T + T_s) = C_s T^2 (T (T + T_s)^2)^(-1/2): one reciprocal root instead of a
        // root and a quotient (five multiplications and 368 cycles of
        // the FP64 pipe against three and 1120). Where T (T + T_s)^2 is not a positive normal number
        // (T zero, negative or not finite, or beyond 1e102) the quotient itself
        const A a = T + A(K.t_s), b = (T * a) * a;
        const unsigned e = (unsigned)__double2hiint(b.v) >> 20;  // sign and exponent
        if (e - 1u <= 2045u) mu = (A(K.c_s) * T) * (T * rsq(b));
        else mu = f64(K.c_s * T.v * ::sqrt(T.v) / (T.v + K.t_s));
    } else {
        mu = K.c_s * T * sqrt(T) / (T + K.t_s);
    }
    A lam = mu * A(K.cp_pr);
    const A c23 = A(2.0 / 3.0);
    // viscous.jl:29-42: the CD4 coefficients give +d/dxi. FP64: 12 times the differences as integer
    // sums, and the metrics times J/12 once instead of J on each physical gradient (120 FP64
    // instructions a cell instead of 190, which kept the FP64 pipe 98% busy)
    const A c1 = A(1.0 / 12.0), c2 = A(-2.0 / 3.0);
    const int vars[4] = {1, 2, 3, 5};
    const long long st[3] = {1, sy, sz};
    A g[4][3];  // u, v, w, T in xi, eta, zeta
    if constexpr (sizeof(R) == 8) {
        bool plain_values = true;
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const R* f = Q + vars[n] * pl + c;
                g[n][d] = difference12(f[-2 * st[d]], f[-st[d]], f[st[d]], f[2 * st[d]], plain_values);
            }
        if (!plain_values) {
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    const volatile double* f = Q + vars[n] * pl + c;  // read again: not held meanwhile
                    g[n][d] = difference12_fp64(f[-2 * st[d]], f[-st[d]], f[st[d]], f[2 * st[d]]);
                }
        }
    } else {
        auto d4 = [&](int n, long long s) {
            const R* f = Q + n * pl + c;
            return c1 * (f[-2 * s] - f[2 * s]) + c2 * (f[-s] - f[s]);
        };
        g[0][0] = d4(1, 1); g[1][0] = d4(2, 1); g[2][0] = d4(3, 1); g[3][0] = d4(5, 1);
        g[0][1] = d4(1, sy); g[1][1] = d4(2, sy); g[2][1] = d4(3, sy); g[3][1] = d4(5, sy);
        g[0][2] = d4(1, sz); g[1][2] = d4(2, sz); g[2][2] = d4(3, sz); g[3][2] = d4(5, sz);
    }
    const A uxi = g[0][0], vxi = g[1][0], wxi = g[2][0], Txi = g[3][0];
    const A uet = g[0][1], vet = g[1][1], wet = g[2][1], Tet = g[3][1];
    const A uze = g[0][2], vze = g[1][2], wze = g[2][2], Tze = g[3][2];
    const A u = arith(Q[c + pl]), v = arith(Q[c + 2 * pl]), w = arith(Q[c + 3 * pl]);
    A dudx, dudy, dudz, dvdx, dvdy, dvdz, dwdx, dwdy, dwdz, dTdx, dTdy, dTdz;
    if constexpr (sizeof(R) == 8) {
        const A j = Jac * c1;
        const A ax = xx * j, ay = xy * j, az = xz * j, bx = ex * j, by = ey * j, bz = ez * j, gx = zx * j, gy = zy * j,
                gz = zz * j;
        dudx = uxi * ax + uet * bx + uze * gx; dudy = uxi * ay + uet * by + uze * gy; dudz = uxi * az + uet * bz + uze * gz;
        dvdx = vxi * ax + vet * bx + vze * gx; dvdy = vxi * ay + vet * by + vze * gy; dvdz = vxi * az + vet * bz + vze * gz;
        dwdx = wxi * ax + wet * bx + wze * gx; dwdy = wxi * ay + wet * by + wze * gy; dwdz = wxi * az + wet * bz + wze * gz;
        dTdx = Txi * ax + Tet * bx + Tze * gx; dTdy = Txi * ay + Tet * by + Tze * gy; dTdz = Txi * az + Tet * bz + Tze * gz;
    } else {
        dudx = (uxi * xx + uet * ex + uze * zx) * Jac;
        dudy = (uxi * xy + uet * ey + uze * zy) * Jac;
        dudz = (uxi * xz + uet * ez + uze * zz) * Jac;
        dvdx = (vxi * xx + vet * ex + vze * zx) * Jac;
        dvdy = (vxi * xy + vet * ey + vze * zy) * Jac;
        dvdz = (vxi * xz + vet * ez + vze * zz) * Jac;
        dwdx = (wxi * xx + wet * ex + wze * zx) * Jac;
        dwdy = (wxi * xy + wet * ey + wze * zy) * Jac;
        dwdz = (wxi * xz + wet * ez + wze * zz) * Jac;
        dTdx = (Txi * xx + Tet * ex + Tze * zx) * Jac;
        dTdy = (Txi * xy + Tet * ey + Tze * zy) * Jac;
        dTdz = (Txi * xz + Tet * ez + Tze * zz) * Jac;
    }
    const A dv = dudx + dvdy + dwdz;
    if (P.les) {  // viscous.jl:66-106: eddy viscosity and conductivity, Pr_t = 0.9
        const A rho = arith(Q[c]);
        const A s12 = A(0.5) * (dudy + dvdx), s13 = A(0.5) * (dudz + dwdx), s23 = A(0.5) * (dvdz + dwdy);
        const A sii = dudx * dudx + dvdy * dvdy + dwdz * dwdz;
        const A sij = s12 * s12 + s13 * s13 + s23 * s23;
        const A inv_d = A(1) / cube_root(Jac);  // 1 / Delta with Delta = J^(1/3) (cell size, J^-1 = volume)
        A mut;
        if (P.les == F3D_LES_SMAGORINSKY) {
            const A Smag = sqrt(A(2) * (sii + A(2) * sij));  // sqrt(2) |S_ij|
            const A cd = A(0.1) * inv_d;
            mut = rho * cd * cd * Smag;
        } else {  // WALE
            const A S = sqrt(sii + A(2) * sij);
            A d11 = dudx * dudx + dudy * dvdx + dudz * dwdx;
            A d22 = dvdx * dudy + dvdy * dvdy + dvdz * dwdy;
            A d33 = dwdx * dudz + dwdy * dvdz + dwdz * dwdz;
            const A tr = A(1.0 / 3.0) * (d11 + d22 + d33);
            d11 -= tr;
            d22 -= tr;
            d33 -= tr;
            const A d12 = A(0.5) * (dudx * dvdx + dvdx * dvdy + dwdx * dvdz + dudy * dudx + dvdy * dudy + dwdy * dudz);
            const A d13 = A(0.5) * (dudx * dwdx + dvdx * dwdy + dwdx * dwdz + dudz * dudx + dvdz * dudy + dwdz * dudz);
            const A d23 = A(0.5) * (dudy * dwdx + dvdy * dwdy + dwdy * dwdz + dudz * dvdx + dvdz * dvdy + dwdz * dvdz);
            const A Sd = sqrt(d11 * d11 + d22 * d22 + d33 * d33 + A(2) * (d12 * d12 + d13 * d13 + d23 * d23));
            const A S2 = S * S;
            const A D = Sd * Sd * Sd / (S2 * S2 * S + Sd * Sd * sqrt(Sd));
            const A cd = A(0.325) * inv_d;
            mut = rho * cd * cd * D;
        }
        // min(mu_t, 2 mu) returning NaN when either is NaN, as Julia's min does (D = 0/0 where
        // the velocity gradient vanishes)
        const A lim = A(2) * mu;
        mut = (mut != mut) ? mut : (lim < mut ? lim : mut);
        mu += mut;
        lam += A(K.cp) * mut / A(0.9);
    }
    const A t11 = mu * (A(2) * dudx - c23 * dv);
    const A t12 = mu * (dudy + dvdx);
    const A t13 = mu * (dudz + dwdx);
    const A t22 = mu * (A(2) * dvdy - c23 * dv);
    const A t23 = mu * (dwdy + dvdz);
    const A t33 = mu * (A(2) * dwdz - c23 * dv);
    const A E1 = u * t11 + v * t12 + w * t13 + lam * dTdx;
    const A E2 = u * t12 + v * t22 + w * t23 + lam * dTdy;
    const A E3 = u * t13 + v * t23 + w * t33 + lam * dTdz;
    Fvx[t] = plain(A(xx * t11 + xy * t12 + xz * t13));
    Fvx[t + vpl] = plain(A(xx * t12 + xy * t22 + xz * t23));
    Fvx[t + 2 * vpl] = plain(A(xx * t13 + xy * t23 + xz * t33));
    Fvx[t + 3 * vpl] = plain(A(xx * E1 + xy * E2 + xz * E3));
    Fvy[t] = plain(A(ex * t11 + ey * t12 + ez * t13));
    Fvy[t + vpl] = plain(A(ex * t12 + ey * t22 + ez * t23));
    Fvy[t + 2 * vpl] = plain(A(ex * t13 + ey * t23 + ez * t33));
    Fvy[t + 3 * vpl] = plain(A(ex * E1 + ey * E2 + ez * E3));
    Fvz[t] = plain(A(zx * t11 + zy * t12 + zz * t13));
    Fvz[t + vpl] = plain(A(zx * t12 + zy * t22 + zz * t23));
    Fvz[t + 2 * vpl] = plain(A(zx * t13 + zy * t23 + zz * t33));
    Fvz[t + 3 * vpl] = plain(A(zx * E1 + zy * E2 + zz * E3));
}

template <class R>
static cudaError_t launch_visc(const DevParams& P, const R* Q, const R* const m[9], const R* J, R* Fvx, R* Fvy,
                               R* Fvz, cudaStream_t st) {
    const long long n = (long long)(P.nxt - 4) * (P.nyt - 4) * (P.nzt - 4);
    k_viscous<R><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(P, Q, m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7],
                                                              m[8], J, Fvx, Fvy, Fvz);
    return cudaGetLastError();
}
cudaError_t launch_viscous(const DevParams& P, const double* Q, const double* const m[9], const double* J,
                           double* Fvx, double* Fvy, double* Fvz, cudaStream_t st) {
    return launch_visc<double>(P, Q, m, J, Fvx, Fvy, Fvz, st);
}
cudaError_t launch_viscous32(const DevParams& P, const float* Q, const float* const m[9], const float* J,
                             float* Fvx, float* Fvy, float* Fvz, cudaStream_t st) {
    return launch_visc<float>(P, Q, m, J, Fvx, Fvy, Fvz, st);
}

}  // namespace f3d
