// k_fvm.cu — the finite-volume RHS of FVM.jl (the reference's default, run.jl:64-65):
// face geometry from cell-centre coordinates, the hybrid switch on the shock sensor,
// linear / WENO7 / WENO5 / minmod reconstruction of the conserved variables U (component-
// wise, Conser_reconstruct_*, or in Roe-averaged characteristic fields, Eigen_reconstruct_*)
// and the HLLC flux (FVM.jl:1224-1357), differenced into the cells by the sweep epilogue
// shared with the finite-difference sweeps.
//
// k_face_geometry<d>: unit normal and area of every face of direction d, computed once per
//   grid (f3d_set_coordinates) and stored at the face's left cell. The operation order is
//   the oracle's and nothing is contracted into FMA, so the normals are bitwise those of
//   the restatement (the tangent basis of the characteristic fields switches on
//   |nz| <= |ny|, which must agree exactly).
// k_fvm_sweep<d, eigen>: tile of TL lines x TC cells. Phase A stages U and phi of the
//   TC+8 cells a line's faces reach; Phase B computes each face (linear faces at once, the
//   non-linear ones queued and then processed by consecutive threads); Phase C is the
//   shared epilogue (differences, viscous CD4, accumulation).
// k_stage_update: the RK update U = ca (U + dt J acc) + cb Un at interior cells. The
//   finite-volume sweeps read U, so the stage cannot update it inside the last sweep.
#include "f3d_fixed.cuh"
#include "f3d_sweep_epilogue.cuh"

namespace f3d {

// ------------------------------------------------------------------------------------
// geometry
template <int DIR>
__global__ void k_face_geometry(const DevParams P, const double* __restrict__ X, const double* __restrict__ Y,
                                const double* __restrict__ Z, double* gnx, double* gny, double* gnz, double* gar) {
    // faces f = 0..N_d of interior transverse lines; left cell full index f + NG - 1
    const int Nd = DIR == 0 ? P.nx : (DIR == 1 ? P.ny : P.nz);
    const int fa = DIR == 0 ? P.nx + 1 : P.nx, fb = DIR == 1 ? P.ny + 1 : P.ny;
    const long long nfaces = (long long)fa * fb * (DIR == 2 ? P.nz + 1 : P.nz);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nfaces) return;
    (void)Nd;
    const int f0 = (int)(t % fa), f1 = (int)((t / fa) % fb), f2 = (int)(t / ((long long)fa * fb));
    int i = f0 + NG, j = f1 + NG, k = f2 + NG;
    if (DIR == 0) i -= 1;
    if (DIR == 1) j -= 1;
    if (DIR == 2) k -= 1;
    const long long sy = P.nxt, sz = (long long)P.nxt * P.nyt;
    const long long sd = DIR == 0 ? 1 : (DIR == 1 ? sy : sz);
    const long long sa = DIR == 0 ? sy : 1;             // transverse a: y for x faces, else x
    const long long sb = DIR == 2 ? sy : sz;            // transverse b: z, except y for z faces
    const long long c = lin3(P, i, j, k);
    // the cell at pa a + pb b from the face's left (side 0) or right (side 1) cell
    auto at = [&](const double* A, int pa, int pb, int side) { return A[c + side * sd + pa * sa + pb * sb]; };
    // 0.125 x the twelve centres summed left to right in the order of FVM.jl:16-21 (and the
    // j, k kernels): (pa,0), (0,pb), (pa,pb), each on both sides, then (-pa,0), (0,-pb),
    // (-pa,-pb) subtracted
    auto diag = [&](const double* A, int pa, int pb) {
        double s = __dadd_rn(at(A, pa, 0, 0), at(A, pa, 0, 1));
        s = __dadd_rn(s, at(A, 0, pb, 0));
        s = __dadd_rn(s, at(A, 0, pb, 1));
        s = __dadd_rn(s, at(A, pa, pb, 0));
        s = __dadd_rn(s, at(A, pa, pb, 1));
        s = __dsub_rn(s, at(A, -pa, 0, 0));
        s = __dsub_rn(s, at(A, -pa, 0, 1));
        s = __dsub_rn(s, at(A, 0, -pb, 0));
        s = __dsub_rn(s, at(A, 0, -pb, 1));
        s = __dsub_rn(s, at(A, -pa, -pb, 0));
        s = __dsub_rn(s, at(A, -pa, -pb, 1));
        return __dmul_rn(0.125, s);
    };
    const double dx1 = diag(X, 1, 1), dy1 = diag(Y, 1, 1), dz1 = diag(Z, 1, 1);
    const double dx2 = diag(X, -1, 1), dy2 = diag(Y, -1, 1), dz2 = diag(Z, -1, 1);
    const double sg = DIR == 1 ? -1.0 : 1.0;  // (a, b) = (x, z) on j faces: x cross z = -y
    double nx = __dmul_rn(__dmul_rn(sg, 0.5), __dadd_rn(__dmul_rn(dy1, dz2), -__dmul_rn(dz1, dy2)));
    double ny = __dmul_rn(__dmul_rn(sg, 0.5), __dadd_rn(__dmul_rn(dz1, dx2), -__dmul_rn(dx1, dz2)));
    double nz = __dmul_rn(__dmul_rn(sg, 0.5), __dadd_rn(__dmul_rn(dx1, dy2), -__dmul_rn(dy1, dx2)));
    const double area =
        __dsqrt_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(nx, nx), __dmul_rn(ny, ny)), __dmul_rn(nz, nz)), 1e-20));
    gnx[c] = __ddiv_rn(nx, area);
    gny[c] = __ddiv_rn(ny, area);
    gnz[c] = __ddiv_rn(nz, area);
    gar[c] = area;
}

cudaError_t launch_face_geometry(const DevParams& P, const double* x, const double* y, const double* z,
                                 double* const geo[12], cudaStream_t st) {
    const long long n0 = (long long)(P.nx + 1) * P.ny * P.nz, n1 = (long long)P.nx * (P.ny + 1) * P.nz,
                    n2 = (long long)P.nx * P.ny * (P.nz + 1);
    k_face_geometry<0><<<cdiv(n0, 128), 128, 0, st>>>(P, x, y, z, geo[0], geo[1], geo[2], geo[3]);
    k_face_geometry<1><<<cdiv(n1, 128), 128, 0, st>>>(P, x, y, z, geo[4], geo[5], geo[6], geo[7]);
    k_face_geometry<2><<<cdiv(n2, 128), 128, 0, st>>>(P, x, y, z, geo[8], geo[9], geo[10], geo[11]);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// face flux pieces (FVM.jl), double precision

// min / max that return NaN when either argument is NaN, as Julia's min and max do (the
// reference's wave-speed estimates): fmin/fmax would drop a NaN Roe speed and hide a
// negative reconstructed density from the non-finite check.
// Comparisons on the bit patterns with integer instructions (an FP64 comparison takes the FP64 pipe
// as long as an addition): two's complement order for the signs, the NaN patterns lie beyond both
// infinities.
__device__ __forceinline__ long long order_of(F64 a) {
    const long long b = __double_as_longlong(a.v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ bool is_nan(F64 a) {
    return (__double_as_longlong(a.v) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
__device__ __forceinline__ F64 nan_min(F64 a, F64 b) {
    return is_nan(a) ? a : (is_nan(b) ? b : (order_of(b) < order_of(a) ? b : a));
}
__device__ __forceinline__ F64 nan_max(F64 a, F64 b) {
    return is_nan(a) ? a : (is_nan(b) ? b : (order_of(a) < order_of(b) ? b : a));
}
// a >= 0 and a <= 0, either zero included, false for NaN
__device__ __forceinline__ bool not_below_zero(F64 a) {
    return !is_nan(a) && (__double2hiint(a.v) >= 0 || (__double_as_longlong(a.v) << 1) == 0);
}
__device__ __forceinline__ bool not_above_zero(F64 a) { return not_below_zero(-a); }

// HLLC flux along the unit normal n of the conserved states UL, UR (FVM.jl:1224-1357)
__device__ __forceinline__ void hllc(const DevParams& P, const F64 UL[5], const F64 UR[5], F64 nx, F64 ny, F64 nz,
                                     F64 F[5]) {
    const F64 g = P.gamma, gm = P.gm1, half = 0.5;
    const F64 rL = UL[0], irL = recip(rL);
    const F64 uL = UL[1] * irL, vL = UL[2] * irL, wL = UL[3] * irL, EL = UL[4];
    const F64 pL = gm * (EL - (half * rL) * (uL * uL + vL * vL + wL * wL));
    const F64 cL = root(fabs((g * pL) * irL));
    const F64 qL = uL * nx + vL * ny + wL * nz;
    const F64 rR = UR[0], irR = recip(rR);
    const F64 uR = UR[1] * irR, vR = UR[2] * irR, wR = UR[3] * irR, ER = UR[4];
    const F64 pR = gm * (ER - (half * rR) * (uR * uR + vR * vR + wR * wR));
    const F64 cR = root(fabs((g * pR) * irR));
    const F64 qR = uR * nx + vR * ny + wR * nz;
    // Roe averages (sqrt(rL) a + sqrt(rR) b) / (sqrt(rL) + sqrt(rR)) = b + k (a - b) with
    // k = 1 / (1 + sqrt(rR / rL)): one root and one reciprocal; two negative densities, whose roots
    // are NaN in the reference, give NaN too
    F64 ratio = rR * irL;
    if ((__double2hiint(rL.v) | __double2hiint(rR.v)) < 0 && rL.v != 0.0 && rR.v != 0.0)
        ratio = f64(__longlong_as_double(0x7ff8000000000000ll));
    const F64 k = recip(F64(1.0) + root(ratio));
    const F64 ur = uR + k * (uL - uR), vr = vR + k * (vL - vR), wr = wR + k * (wL - wR);
    const F64 qr = ur * nx + vr * ny + wr * nz;
    const F64 HL = (EL + pL) * irL, HR = (ER + pR) * irR;
    const F64 Hr = HR + k * (HL - HR);
    const F64 cr = root(fabs(gm * (Hr - half * (ur * ur + vr * vr + wr * wr))));
    const F64 SL = nan_min(qL - cL, qr - cr);
    const F64 SR = nan_max(qR + cR, qr + cr);
    const F64 mL = rL * (SL - qL), mR = rR * (SR - qR);
    const F64 Ss = (pR - pL + mL * qL - mR * qR) / (mL - mR + F64(1e-12));
    const bool SLp = not_below_zero(SL), SRm = not_above_zero(SR);
    const bool left = SLp || (!SRm && !is_nan(SR) && not_below_zero(Ss));
    const F64 r = left ? rL : rR, u = left ? uL : uR, v = left ? vL : vR, w = left ? wL : wR;
    const F64 E = left ? EL : ER, p = left ? pL : pR, q = left ? qL : qR;
    const F64 rq = r * q;
    F[0] = rq;
    F[1] = rq * u + p * nx;
    F[2] = rq * v + p * ny;
    F[3] = rq * w + p * nz;
    F[4] = (E + p) * q;
    if (SLp || SRm) return;  // supersonic: the upwind state's physical flux
    // star state of the side: F* = F + S (U* - U)
    const F64 S = left ? SL : SR, ir = left ? irL : irR, m = left ? mL : mR;  // m = r (S - q)
    const F64* Us = left ? UL : UR;
    const F64 f = m / (S - Ss), dS = Ss - q;
    const F64 fd = f * dS;
    const F64 st[5] = {f, f * u + fd * nx, f * v + fd * ny, f * w + fd * nz, f * (E * ir) + fd * (Ss + p / m)};
#pragma unroll
    for (int n = 0; n < 5; n++) F[n] += S * (st[n] - Us[n]);
}

// The two sides of a face on seven-point stencils in upwind order (FVM.jl): br 1 = WENO7 (its own
// eps 1e-10), 2 = WENO5 (1e-8), 3 = minmod in the two sides' forms of FVM.jl:204-205. The nonlinear
// sums are those of the finite-difference faces (f3d_flux.cuh); the two values share one reciprocal.
__device__ __forceinline__ void fvm_sides(int br, const F64 L[7], const F64 R[7], F64 ss, F64& l, F64& r) {
    if (br == 3) {
        l = L[3] + F64(0.5) * minmod(F64(L[3] - L[2]), F64(L[4] - L[3]));
        r = R[3] - F64(0.5) * minmod(F64(R[3] - R[2]), F64(R[3] - R[4]));
        return;
    }
    auto VL = [&](int k) { return L[k]; };
    auto VR = [&](int k) { return R[k]; };
    const WenoSums a = br == 1 ? weno7_sums(VL, ss, 1e-10) : weno5_sums(VL, ss, 1e-8);
    const WenoSums b = br == 1 ? weno7_sums(VR, ss, 1e-10) : weno5_sums(VR, ss, 1e-8);
    const F64 unit = br == 1 ? F64(1.0 / 12.0) : F64(1.0 / 6.0);
    const F64 D = a.D * b.D;
    const unsigned e = ((unsigned)__double2hiint(D.v) >> 20) & 0x7ffu;
    if (e - 23u > 1800u) {
        l = a.base + unit * (a.N / a.D);
        r = b.base + unit * (b.N / b.D);
        return;
    }
    const F64 i = unit * recip_step(D.v);
    l = a.base + (a.N * b.D) * i;
    r = b.base + (b.N * a.D) * i;
}

// ------------------------------------------------------------------------------------
// the sweep
template <int DIR> struct FTile;
template <> struct FTile<0> { static constexpr int TL = 8, TC = 32; };
template <> struct FTile<1> { static constexpr int TL = 16, TC = 16; };
template <> struct FTile<2> { static constexpr int TL = 16, TC = 16; };
// Threads and resident blocks per SM of a sweep: the characteristic form is held to 160 registers
// a thread, the component-wise one needs ~125. Small blocks let several blocks share an SM, so one
// block's barrier waits overlap another's face work. RK3 step of the shock tube 256x64x64,
// characteristic: 96 x 4 5.62 ms, 160 x 3 5.65, 144 x 3 5.73, 288 x 2 5.82, 160 x 2 6.15, 288 x 1 7.8
// (64 x 4 at ~255 registers, before the linear states were integer sums, 8.14).
#ifndef FVM_E_THREADS
#define FVM_E_THREADS 96
#define FVM_E_BLOCKS 4
#define FVM_C_THREADS 128
#define FVM_C_BLOCKS 2
#endif
template <bool EIGEN> struct FvmLaunch;
template <> struct FvmLaunch<true> { static constexpr int NT = FVM_E_THREADS, MINB = FVM_E_BLOCKS; };
template <> struct FvmLaunch<false> { static constexpr int NT = FVM_C_THREADS, MINB = FVM_C_BLOCKS; };

template <int DIR> constexpr size_t fvm_smem_bytes() {
    constexpr int TL = FTile<DIR>::TL, TC = FTile<DIR>::TC, NP = TC + 8, NF = TC + 1;
    return sizeof(double) * ((size_t)TL * NP * 6 + (size_t)TL * NF * 15) + sizeof(int) * ((size_t)TL * NF + 2);
}

template <int DIR, bool EIGEN>
__global__ void __launch_bounds__(FvmLaunch<EIGEN>::NT, FvmLaunch<EIGEN>::MINB) k_fvm_sweep(const SweepArgs a, const double* __restrict__ Ur,
                                                           const double* __restrict__ gnx, const double* __restrict__ gny,
                                                           const double* __restrict__ gnz, const double* __restrict__ gar) {
    constexpr int TL = FTile<DIR>::TL, TC = FTile<DIR>::TC, NP = TC + 8, NF = TC + 1;
    constexpr int FVM_THREADS = FvmLaunch<EIGEN>::NT;
    const DevParams& P = a.P;
    const bool hybrid = P.fixed_branch < 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sU = reinterpret_cast<double*>(smem_raw);  // [5][TL*NP]
    double* sPhi = sU + 5 * TL * NP;                    // [TL*NP]
    double* sF = sPhi + TL * NP;                        // [5][TL*NF]
    double* sL = sF + 5 * TL * NF;                      // [10][TL*NF] left and right linear states
    int* list = reinterpret_cast<int*>(sL + 10 * TL * NF);
    int* count = list + TL * NF;
    const double* Q = static_cast<const double*>(a.Q);
    const double* S = static_cast<const double*>(a.S);
    const double* Ph = static_cast<const double*>(a.phi);

    const int Nd = DIR == 0 ? P.nx : (DIR == 1 ? P.ny : P.nz);
    const int Nl = DIR == 0 ? P.ny : P.nx;
    int c0, l0, other;
    if (DIR == 0) { c0 = blockIdx.x * TC; l0 = blockIdx.y * TL; other = blockIdx.z; }
    else { l0 = blockIdx.x * TL; c0 = blockIdx.y * TC; other = blockIdx.z; }
    const int nc = min(TC, Nd - c0);
    const int nl = min(TL, Nl - l0);
    const long long stride = DIR == 0 ? 1 : (DIR == 1 ? (long long)P.nxt : (long long)P.nxt * P.nyt);
    auto cell = [&](int l, int g) -> long long {
        if (DIR == 0) return lin3(P, g, l0 + l + NG, other + NG);
        if (DIR == 1) return lin3(P, l0 + l + NG, g, other + NG);
        return lin3(P, l0 + l + NG, other + NG, g);
    };
    auto sidx = [&](int l, int p) { return DIR == 0 ? l * NP + p : p * TL + l; };
    auto fidx = [&](int l, int t) { return DIR == 0 ? l * NF + t : t * TL + l; };
    const long long pl = P.plane;

    if (threadIdx.x == 0) *count = 0;
    // Phase A: U and phi at positions 0..nc+7 (full index c0 + p along d)
    for (int it = threadIdx.x; it < TL * NP; it += FVM_THREADS) {
        int l, p;
        if (DIR == 0) { l = it / NP; p = it - l * NP; } else { p = it / TL; l = it - p * TL; }
        if (l >= nl || p >= nc + 8) continue;
        const long long c = cell(l, c0 + p);
        const int s = sidx(l, p);
#pragma unroll
        for (int n = 0; n < 5; n++) sU[n * TL * NP + s] = Ur[c + n * pl];
        if (hybrid) sPhi[s] = Ph[c];
    }
    __syncthreads();

    // The linear scheme's left and right states of every face as integer sums over strips of five
    // faces and one component (f3d_fixed.cuh): 10 FP64 instructions a face instead of 70
    if (P.lin_int && P.fixed_branch <= 0) {
        const int ns = (nc + LIN_STRIP) / LIN_STRIP, per = ns * (DIR == 0 ? nl : TL), last = nc + 7;
        for (int k = threadIdx.x; k < 5 * per; k += FVM_THREADS) {
            const int n = k / per, r = k - n * per;
            int l, st;
            if (DIR == 0) { l = r / ns; st = r - l * ns; } else { st = r / TL; l = r - st * TL; }
            if (l >= nl) continue;
            const int t0 = st * LIN_STRIP;
            const double* u = sU + n * TL * NP;
            const unsigned want = (1u << min(LIN_STRIP, nc + 1 - t0)) - 1u;
            linear_strip_both(P, t0, want, [&](int p) { return p <= last ? u[sidx(l, p)] : 0.0; },
                              [&](int f, double up, double down) {
                                  sL[n * TL * NF + fidx(l, t0 + f)] = up;
                                  sL[(n + 5) * TL * NF + fidx(l, t0 + f)] = down;
                              });
        }
        __syncthreads();
    }

    // Phase B: face t between positions t+3 (left cell, the kernels' i) and t+4
    auto face = [&](int l, int t, int br) {
        const long long cl = cell(l, c0 + t + 3);
        auto Uv = [&](int n, int p) { return f64(sU[n * TL * NP + sidx(l, p)]); };
        const F64 nx = f64(gnx[cl]), ny = f64(gny[cl]), nz = f64(gnz[cl]);
        F64 UL[5], UR[5];
        if (br == 0 && P.lin_int) {  // linear scheme on U, FVM.jl:42-60, summed by the strips
            const int f = fidx(l, t);
#pragma unroll
            for (int n = 0; n < 5; n++) {
                UL[n] = f64(sL[n * TL * NF + f]);
                UR[n] = f64(sL[(n + 5) * TL * NF + f]);
            }
        } else if (br == 0) {
#pragma unroll
            for (int n = 0; n < 5; n++) {
                F64 vl = P.cd.lin[0] * Uv(n, t), vr = P.cd.lin[0] * Uv(n, t + 7);
#pragma unroll
                for (int m = 1; m < 7; m++) {
                    vl += P.cd.lin[m] * Uv(n, t + m);
                    vr += P.cd.lin[m] * Uv(n, t + 7 - m);
                }
                UL[n] = vl;
                UR[n] = vr;
            }
        } else {
            const F64 ss = F64(2.0) / (f64(S[cl + stride]) + f64(S[cl]));
            if (!EIGEN) {  // Conser_reconstruct, FVM.jl:739-855
#pragma unroll
                for (int n = 0; n < 5; n++) {
                    F64 VL[7], VR[7];
#pragma unroll
                    for (int m = 0; m < 7; m++) {
                        VL[m] = Uv(n, t + m);
                        VR[m] = Uv(n, t + 7 - m);
                    }
                    fvm_sides(br, VL, VR, ss, UL[n], UR[n]);
                }
            } else {  // Eigen_reconstruct, FVM.jl:65-228
                auto Qv = [&](int n, long long c) { return f64(Q[c + n * pl]); };
                const long long cr = cl + stride;
                const F64 srl = root(Qv(0, cl)), srr = root(Qv(0, cr)), isr = recip(srl + srr);
                const F64 half = 0.5;
                auto roe = [&](F64 a, F64 b) { return F64((srl * a + srr * b) * isr); };
                const F64 u = roe(Qv(1, cl), Qv(1, cr)), v = roe(Qv(2, cl), Qv(2, cr)), w = roe(Qv(3, cl), Qv(3, cr));
                const F64 gg = P.gamma / P.gm1;
                auto Hof = [&](long long c) {
                    const F64 uu = Qv(1, c), vv = Qv(2, c), ww = Qv(3, c);
                    return gg * Qv(4, c) / Qv(0, c) + half * (uu * uu + vv * vv + ww * ww);
                };
                const F64 H = roe(Hof(cl), Hof(cr));
                const F64 v2 = half * (u * u + v * v + w * w);
                const F64 c = root(P.gm1 * (H - v2));
                F64 lx, ly, lz;
                if (fabs(nz) <= fabs(ny)) {
                    const F64 id = rsq(nx * nx + ny * ny + F64(1e-12));
                    lx = -ny * id; ly = nx * id; lz = F64(0.0);
                } else {
                    const F64 id = rsq(nx * nx + nz * nz + F64(1e-12));
                    lx = -nz * id; ly = F64(0.0); lz = nx * id;
                }
                const F64 mx = ny * lz - nz * ly, my = nz * lx - nx * lz, mz = nx * ly - ny * lx;
                const F64 invc = recip(c), invc2 = invc * invc, K = P.gm1;
                const F64 Kc2 = K * invc2, Ku = Kc2 * u, Kv = Kc2 * v, Kw = Kc2 * w, Kv2 = Kc2 * v2;
                const F64 un = u * nx + v * ny + w * nz, ul = u * lx + v * ly + w * lz, um = u * mx + v * my + w * mz;
                const F64 uni = un * invc, nxi = nx * invc, nyi = ny * invc, nzi = nz * invc;
#pragma unroll
                for (int q = 0; q < 5; q++) { UL[q] = F64(0.0); UR[q] = F64(0.0); }
#pragma unroll 1
                for (int n = 0; n < 5; n++) {
                    F64 ln[5], rn[5];
                    if (n == 0 || n == 2) {
                        const F64 sg = n == 0 ? F64(1.0) : F64(-1.0), sc = sg * c;
                        ln[0] = half * (Kv2 + sg * uni); ln[1] = -half * (Ku + sg * nxi); ln[2] = -half * (Kv + sg * nyi);
                        ln[3] = -half * (Kw + sg * nzi); ln[4] = half * Kc2;
                        rn[0] = F64(1.0); rn[1] = u - nx * sc; rn[2] = v - ny * sc; rn[3] = w - nz * sc; rn[4] = H - un * sc;
                    } else if (n == 1) {
                        ln[0] = F64(1.0) - Kv2; ln[1] = Ku; ln[2] = Kv; ln[3] = Kw; ln[4] = -Kc2;
                        rn[0] = F64(1.0); rn[1] = u; rn[2] = v; rn[3] = w; rn[4] = v2;
                    } else if (n == 3) {
                        ln[0] = -ul; ln[1] = lx; ln[2] = ly; ln[3] = lz; ln[4] = F64(0.0);
                        rn[0] = F64(0.0); rn[1] = lx; rn[2] = ly; rn[3] = lz; rn[4] = ul;
                    } else {
                        ln[0] = -um; ln[1] = mx; ln[2] = my; ln[3] = mz; ln[4] = F64(0.0);
                        rn[0] = F64(0.0); rn[1] = mx; rn[2] = my; rn[3] = mz; rn[4] = um;
                    }
                    F64 VL[7], VR[7];
#pragma unroll
                    for (int m = 0; m < 7; m++) {
                        F64 sl = ln[0] * Uv(0, t + m), sr = ln[0] * Uv(0, t + 7 - m);
#pragma unroll
                        for (int q = 1; q < 5; q++) {
                            sl += ln[q] * Uv(q, t + m);
                            sr += ln[q] * Uv(q, t + 7 - m);
                        }
                        VL[m] = sl;
                        VR[m] = sr;
                    }
                    F64 vl, vr;
                    fvm_sides(br, VL, VR, ss, vl, vr);
#pragma unroll
                    for (int q = 0; q < 5; q++) {
                        UL[q] += rn[q] * vl;
                        UR[q] += rn[q] * vr;
                    }
                }
            }
        }
        const F64 ar = f64(gar[cl]);
        F64 Ff[5];
        hllc(P, UL, UR, nx, ny, nz, Ff);
        const int f = fidx(l, t);
#pragma unroll
        for (int n = 0; n < 5; n++) sF[n * TL * NF + f] = F64(Ff[n] * ar).v;
        if (a.faces) {  // face-flux output in the reference's Fx/Fy/Fz shape
            const long long fx = P.nx + (DIR == 0), fy = P.ny + (DIR == 1), fz = P.nz + (DIR == 2);
            long long fi, fj, fk;
            if (DIR == 0) { fi = c0 + t; fj = l0 + l; fk = other; }
            else if (DIR == 1) { fi = l0 + l; fj = c0 + t; fk = other; }
            else { fi = l0 + l; fj = other; fk = c0 + t; }
            const long long fo = fi + fx * (fj + fy * fk), nf = fx * fy * fz;
#pragma unroll
            for (int n = 0; n < 5; n++) a.faces[fo + n * nf] = F64(Ff[n] * ar).v;
        }
    };
    for (int it = threadIdx.x; it < TL * NF; it += FVM_THREADS) {
        int l, t;
        if (DIR == 0) { l = it / NF; t = it - l * NF; } else { t = it / TL; l = it - t * TL; }
        if (l >= nl || t > nc) continue;
        int br = P.fixed_branch;
        if (hybrid) {  // max of phi over cells i-2..i+3 (FVM.jl:33)
            double ph[6];
#pragma unroll
            for (int o = 0; o < 6; o++) ph[o] = sPhi[sidx(l, t + 1 + o)];
            br = branch_of(P, ph);
        }
        if (br != 0) {
            list[atomicAdd(count, 1)] = it * 4 + br;
            continue;
        }
        face(l, t, 0);
    }
    __syncthreads();
    const int nq = *count;
    for (int k = threadIdx.x; k < nq; k += FVM_THREADS) {
        const int e = list[k], it = e >> 2;
        int l, t;
        if (DIR == 0) { l = it / NF; t = it - l * NF; } else { t = it / TL; l = it - t * TL; }
        face(l, t, e & 3);
    }
    if (a.out_mode == OUT_FACES) return;
    __syncthreads();
    // Phase C
    sweep_epilogue<DIR, TL, TC, FVM_THREADS, double>(a, sF, c0, l0, other, nc, nl, cell, fidx);
}

template <int DIR, bool EIGEN> static cudaError_t fvm_configure_one() {
    return cudaFuncSetAttribute(k_fvm_sweep<DIR, EIGEN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)fvm_smem_bytes<DIR>());
}

cudaError_t fvm_configure() {
    cudaError_t e;
    if ((e = fvm_configure_one<0, true>()) != cudaSuccess) return e;
    if ((e = fvm_configure_one<0, false>()) != cudaSuccess) return e;
    if ((e = fvm_configure_one<1, true>()) != cudaSuccess) return e;
    if ((e = fvm_configure_one<1, false>()) != cudaSuccess) return e;
    if ((e = fvm_configure_one<2, true>()) != cudaSuccess) return e;
    return fvm_configure_one<2, false>();
}

template <int DIR, bool EIGEN>
static cudaError_t fvm_launch_dir(const SweepArgs& a, const double* U, const double* const geo[12], cudaStream_t st) {
    constexpr int TL = FTile<DIR>::TL, TC = FTile<DIR>::TC;
    const DevParams& P = a.P;
    dim3 grid;
    if (DIR == 0) grid = dim3(cdiv(P.nx, TC), cdiv(P.ny, TL), P.nz);
    else if (DIR == 1) grid = dim3(cdiv(P.nx, TL), cdiv(P.ny, TC), P.nz);
    else grid = dim3(cdiv(P.nx, TL), cdiv(P.nz, TC), P.ny);
    const double* const* g = geo + 4 * DIR;
    k_fvm_sweep<DIR, EIGEN><<<grid, FvmLaunch<EIGEN>::NT, fvm_smem_bytes<DIR>(), st>>>(a, U, g[0], g[1], g[2], g[3]);
    return cudaGetLastError();
}

cudaError_t launch_fvm_sweep(int dir, bool eigen, const SweepArgs& a, const double* U, const double* const geo[12],
                             cudaStream_t st) {
    if (dir == 0) return eigen ? fvm_launch_dir<0, true>(a, U, geo, st) : fvm_launch_dir<0, false>(a, U, geo, st);
    if (dir == 1) return eigen ? fvm_launch_dir<1, true>(a, U, geo, st) : fvm_launch_dir<1, false>(a, U, geo, st);
    return eigen ? fvm_launch_dir<2, true>(a, U, geo, st) : fvm_launch_dir<2, false>(a, U, geo, st);
}

// ------------------------------------------------------------------------------------
// RK update from the accumulated RHS (div.jl:1-50 fused with linComb, utils.jl:57-70)
__global__ void k_stage_update(const DevParams P, const double* __restrict__ acc, const double* __restrict__ J,
                               double dt, double* U, double* Un, int stage1_copy, int combine, double ca, double cb,
                               const double* __restrict__ dtl) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = (long long)P.nx * P.ny * P.nz;
    if (t >= n) return;
    int i, j, k;
    split3(t, P.dnx, P.dny, i, j, k);
    const long long c = lin3(P, i + NG, j + NG, k + NG), pl = P.plane;
    const double Jact = J[c] * (dtl ? dtl[c] : dt);
#pragma unroll
    for (int v = 0; v < 5; v++) {
        const double u = U[c + v * pl];
        if (stage1_copy) Un[c + v * pl] = u;
        double un = u + acc[c + v * pl] * Jact;
        if (combine) un = un * ca + Un[c + v * pl] * cb;
        U[c + v * pl] = un;
    }
}

cudaError_t launch_stage_update(const DevParams& P, const double* acc, const double* J, double dt, double* U,
                                double* Un, int stage1_copy, int combine, double ca, double cb, cudaStream_t st,
                                const double* dtl) {
    const long long n = (long long)P.nx * P.ny * P.nz;
    k_stage_update<<<cdiv(n, 256), 256, 0, st>>>(P, acc, J, dt, U, Un, stage1_copy, combine, ca, cb, dtl);
    return cudaGetLastError();
}

}  // namespace f3d
