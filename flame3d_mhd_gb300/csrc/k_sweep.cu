// k_sweep.cu — one direction of the inviscid RHS (plus that direction's viscous
// divergence) as a tiled sweep.
//
// A block owns TL grid lines along the sweep direction d and TC consecutive interior
// cells of each. Phase A splits the TC+8 cells the tile's stencils touch into Fp/Fm in
// shared memory (fluxSplit_*, split.jl), once per cell. Phase B reconstructs the TC+1
// faces of the tile, one thread per face, choosing UP7 / WENO7 / WENO5 / NND2 per face
// from the shock sensor (advect_x/xc and their y, z permutations, schemes.jl:86-1643).
// Phase C differences the face fluxes into the cells, adds the 4th-order central
// divergence of the viscous flux of direction d (div.jl:14-39), and accumulates into the
// RHS, or (last sweep) applies the Euler update and SSP-RK3 combination
// (div.jl:40-48, utils.jl:57-70) in place.
//
// Shared-memory layout is [var][line][pos] for d = x (threads run along the line) and
// [var][pos][line] for d = y, z (threads run across x-adjacent lines), so global loads
// coalesce along i and shared loads are conflict-free in both cases.
#include "f3d_face.cuh"
#include "f3d_fixed.cuh"
#include "f3d_sweep_epilogue.cuh"

namespace f3d {

// Tile (lines TL x cells TC), threads and resident blocks per SM of a sweep, by type.
// FP64: 4 x 64 in every direction on 288 threads (~38 KB of shared memory a block): Phase B's
// 260 faces and Phase A's 288 split cells are one pass of the block, so that no warp waits for
// others' second pass. Four blocks per SM where the tiles hold no WENO code (WENO_LISTED, 56
// registers, 36 warps an SM hide the loads, barriers and FP64 latencies), three where they do
// (72 registers). Measured on one box (RK3 step; 160 threads x 4 blocks with WENO code -> 288 x 4
// without): shock tube 256x64x64 5.38 -> 4.56 ms, ramp 512x256x128 49.8 -> 45.5 ms, plate
// 125x61x37 1.29 -> 1.18 ms, RHS of a 16^3 vortex 50.9 -> 43.7 us; with the strips' faces handed over one
// at a time (4-8 bytes spilled instead of 48-60) 4.41 / 45.3 / 1.165 ms and 41.0 us. Without WENO code 288 x 3 takes
// 4.82 / 47.5 / 1.23 ms, 288 x 2 5.69 / 54.5 / 1.37, 288 x 5 (45 registers) 5.07 / 48.7 / 1.27,
// 320 x 4 4.77 / 46.9 / 1.22, 192 x 6 5.19 / 48.7 / 1.23, 160 x 5 4.87 / 46.5 / 1.21. With it (the WENO5 vortex 64^3):
// 160 x 4 4.74 -> 288 x 3 4.64 ms, 320 x 3 4.67, 192 x 5 4.82. Characteristic faces in the tiles (fixed
// branches, no room for the lists, f3d_rhs_noalloc) spill ~380 bytes at 72 registers, and still gain on tiles of
// 8 x 64 with two blocks of 96 registers, before the strips and the WENO sums' rewriting: RHS of the tube
// with every face WENO7 9.24 -> 7.51 ms, WENO5 6.70 -> 5.22, f3d_rhs_noalloc on 32x16x16 298 -> 181 us. Tiles of
// eight lines or of 32 cells lose more on the smaller grids than the ramp gains.
// FP32: the same tile sizes (~20 KB). The Float32 form (FP64 WENO7 weights) on 320 threads, five
// blocks per SM (32 registers, the characteristic form spills ~310 bytes, component-wise ~95): one pass per phase and 50
// warps an SM for the latencies of the weights. RK3 step of its shock tube 256x64x64, 128 threads x
// 6 -> 320 x 5: 4.80 -> 4.07 ms (288 x 6 4.12, 288 x 5 4.19, 160 x 7 4.40, 224 x 6 4.47, 288 x 3 5.06).
// The mixed form (grids without TMA rows) keeps 128 x 6, 80 registers: on small grids the spills
// would lengthen its faces' chains (RHS of 30x10x9: 53 us, 59 us at 320 x 5).
#ifndef SW_D_THREADS
#define SW_D_THREADS 288
#define SW_D_BLOCKS 3
#define SW_D_LISTED_BLOCKS 4
#define SW_D_TL0 4
#define SW_D_TL12 4
#endif
#ifndef SW_D_TC0
#define SW_D_TC0 64
#define SW_D_TC12 64
#endif
// WENO faces: component-, characteristic-wise, from k_weno.cu, the first two with the FP64 WENO7 weights of the Float32 form
enum { WENO_COMP, WENO_CHAR, WENO_LISTED, WENO_COMP_REF32, WENO_CHAR_REF32 };
template <int DIR, class R, int FACES = WENO_COMP> struct Tile;
#ifndef SW_F_THREADS
#define SW_F_THREADS 128
#define SW_F_BLOCKS 6
#define SW_R_THREADS 320
#define SW_R_BLOCKS 5
#define SW_F_TL0 4
#define SW_F_TL12 8
#endif
template <int FACES> struct FloatTile {
    static constexpr bool REF32 = FACES == WENO_COMP_REF32 || FACES == WENO_CHAR_REF32;
    static constexpr int NT = REF32 ? SW_R_THREADS : SW_F_THREADS, MINB = REF32 ? SW_R_BLOCKS : SW_F_BLOCKS;
};
template <int FACES> struct Tile<0, float, FACES> { static constexpr int TL = SW_F_TL0, TC = 64, NT = FloatTile<FACES>::NT, MINB = FloatTile<FACES>::MINB; };
template <int FACES> struct Tile<1, float, FACES> { static constexpr int TL = SW_F_TL12, TC = 32, NT = FloatTile<FACES>::NT, MINB = FloatTile<FACES>::MINB; };
template <int FACES> struct Tile<2, float, FACES> { static constexpr int TL = SW_F_TL12, TC = 32, NT = FloatTile<FACES>::NT, MINB = FloatTile<FACES>::MINB; };
template <int FACES> struct Tile<0, double, FACES> {
    static constexpr int TL = SW_D_TL0, TC = SW_D_TC0, NT = SW_D_THREADS,
                         MINB = FACES == WENO_LISTED ? SW_D_LISTED_BLOCKS : SW_D_BLOCKS;
};
template <int FACES> struct Tile<1, double, FACES> {
    static constexpr int TL = SW_D_TL12, TC = SW_D_TC12, NT = SW_D_THREADS,
                         MINB = FACES == WENO_LISTED ? SW_D_LISTED_BLOCKS : SW_D_BLOCKS;
};
template <int FACES> struct Tile<2, double, FACES> {
    static constexpr int TL = SW_D_TL12, TC = SW_D_TC12, NT = SW_D_THREADS,
                         MINB = FACES == WENO_LISTED ? SW_D_LISTED_BLOCKS : SW_D_BLOCKS;
};

template <int DIR, class R> constexpr size_t sweep_smem_bytes(bool hybrid) {
    using T = Tile<DIR, R>;
    return sizeof(R) * ((size_t)T::TL * (T::TC + 8) * (10 + (hybrid ? 1 : 0)) + (size_t)T::TL * (T::TC + 1) * 5) +
           sizeof(int) * (2 * (size_t)T::TL * (T::TC + 1) + 4) +
           (sizeof(R) == 8 ? (((size_t)T::TL * (T::TC + 1) + 7) & ~(size_t)7) : 0);  // faces of the linear strips
}

template <int DIR, int FACES, class R>
__global__ void __launch_bounds__(Tile<DIR, R, FACES>::NT, Tile<DIR, R, FACES>::MINB) k_sweep(const SweepArgs a) {
    constexpr int TL = Tile<DIR, R>::TL, TC = Tile<DIR, R>::TC, NP = TC + 8, NF = TC + 1;
    constexpr int SWEEP_THREADS = Tile<DIR, R, FACES>::NT;
    using A = typename Arith<R>::type;
    const DevParams& P = a.P;
    const bool hybrid = P.fixed_branch < 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sFp = reinterpret_cast<R*>(smem_raw);
    R* sFm = sFp + 5 * TL * NP;
    R* sF = sFm + 5 * TL * NP;
    R* sPhi = sF + 5 * TL * NF;
    const R* Qr = static_cast<const R*>(a.Q);
    const R* Ar[3] = {static_cast<const R*>(a.A[0]), static_cast<const R*>(a.A[1]), static_cast<const R*>(a.A[2])};
    const R* Hr[3] = {static_cast<const R*>(a.Ah[0]), static_cast<const R*>(a.Ah[1]),
                      static_cast<const R*>(a.Ah[2])};
    const R* Sr = static_cast<const R*>(a.S);
    const R* Phr = static_cast<const R*>(a.phi);

    // tile geometry: interior start c0 along d, first line l0 and line count
    const int Nd = DIR == 0 ? P.nx : (DIR == 1 ? P.ny : P.nz);
    const int Nl = DIR == 0 ? P.ny : P.nx;
    int c0, l0, other;
    if (DIR == 0) { c0 = blockIdx.x * TC; l0 = blockIdx.y * TL; other = blockIdx.z; }
    else { l0 = blockIdx.x * TL; c0 = blockIdx.y * TC; other = blockIdx.z; }
    const int nc = min(TC, Nd - c0);
    const int nl = min(TL, Nl - l0);
    const long long stride = DIR == 0 ? 1 : (DIR == 1 ? (long long)P.nxt : (long long)P.nxt * P.nyt);
    // linear index of (line l, full position along d = g)
    auto cell = [&](int l, int g) -> long long {
        if (DIR == 0) return lin3(P, g, l0 + l + NG, other + NG);
        if (DIR == 1) return lin3(P, l0 + l + NG, g, other + NG);
        return lin3(P, l0 + l + NG, other + NG, g);
    };
    auto sidx = [&](int l, int p) { return DIR == 0 ? l * NP + p : p * TL + l; };
    auto fidx = [&](int l, int t) { return DIR == 0 ? l * NF + t : t * TL + l; };
    const long long pl = P.plane;

    if (threadIdx.x < 3) reinterpret_cast<int*>(sPhi + TL * NP)[2 * TL * NF + threadIdx.x] = 0;
    // ---- Phase A: split every cell the tile's stencils reach (positions 0..nc+7, full
    // index c0 + p along d).
    for (int it = threadIdx.x; it < TL * NP; it += SWEEP_THREADS) {
        int l, p;
        if (DIR == 0) { l = it / NP; p = it - l * NP; } else { p = it / TL; l = it - p * TL; }
        if (l >= nl || p >= nc + 8) continue;
        const long long c = cell(l, c0 + p);
        A q[6];
#pragma unroll
        for (int n = 0; n < 6; n++) q[n] = arith(Qr[c + n * pl]);
        A fp[5], fm[5];
        split_cell<A>(P.split, cst<R>(P), q, split_sound<A>(P, a, c, q), arith(Ar[0][c]), arith(Ar[1][c]),
                      arith(Ar[2][c]), arith(Hr[0][c]), arith(Hr[1][c]), arith(Hr[2][c]), arith(Sr[c]), fp, fm);
        const int s = sidx(l, p);
#pragma unroll
        for (int n = 0; n < 5; n++) {
            sFp[n * TL * NP + s] = plain(fp[n]);
            sFm[n * TL * NP + s] = plain(fm[n]);
        }
        if (hybrid) sPhi[s] = Phr[c];
    }
    __syncthreads();

    // ---- Phase B: faces t = 0..nc (face t lies between positions t+3 and t+4).
    // With the hybrid switch, NND2 faces are done at once and the WENO7 / WENO5 faces are queued
    // and then processed by consecutive threads: near a shock only a few faces of a warp take
    // the long WENO paths, and done in place they would run with the other lanes idle (and a
    // warp holding both kinds would run both paths). FP64 linear faces are done as integer strips
    // (f3d_fixed.cuh) where their coefficients allow it, others at once.
    auto do_face = [&](int l, int t, int br) {
        const long long cl = cell(l, c0 + t + 3), cr = cl + stride;
        A out[5];
        A s0 = A(0);
        if (FACES != WENO_LISTED && (br == 1 || br == 2)) s0 = A(2) / (arith(Sr[cl]) + arith(Sr[cr]));
        auto FP = [&](int n, int p) { return arith(sFp[n * TL * NP + sidx(l, p)]); };
        auto FM = [&](int n, int p) { return arith(sFm[n * TL * NP + sidx(l, p)]); };
        face_flux<FACES == WENO_CHAR || FACES == WENO_CHAR_REF32, A, FloatTile<FACES>::REF32>(P, a, br, t, s0, cl, cr, FP, FM, out);
        const int f = fidx(l, t);
#pragma unroll
        for (int n = 0; n < 5; n++) sF[n * TL * NF + f] = plain(out[n]);
    };
    auto face_lt = [&](int it, int& l, int& t) {
        if (DIR == 0) { l = it / NF; t = it - l * NF; } else { t = it / TL; l = it - t * TL; }
    };
    int* list7 = reinterpret_cast<int*>(sPhi + TL * NP);
    int* list5 = list7 + TL * NF;
    int* counts = list5 + TL * NF;  // WENO7 and WENO5 faces, next chunk
    unsigned char* sLin = reinterpret_cast<unsigned char*>(counts + 4);  // faces left to the strips
    const bool strips = sizeof(R) == 8 && P.lin_int;
    for (int it = threadIdx.x; it < TL * NF; it += SWEEP_THREADS) {
        int l, t;
        face_lt(it, l, t);
        if (strips) sLin[it] = 0;
        if (l >= nl || t > nc) continue;
        int br = P.fixed_branch;
        if (hybrid) {
            R ph[6];
#pragma unroll
            for (int o = 0; o < 6; o++) ph[o] = sPhi[sidx(l, t + 1 + o)];
            br = branch_of(P, ph);
            if (br == 1 || br == 2) {
                if constexpr (FACES == WENO_LISTED) {  // its flux is known (k_weno.cu)
                    const double* w = a.wflux + cell(l, c0 + t + 3);
#pragma unroll
                    for (int n = 0; n < 5; n++) sF[n * TL * NF + fidx(l, t)] = (R)w[n * pl];
                } else {
                    const int k = atomicAdd(&counts[br - 1], 1);
                    (br == 1 ? list7 : list5)[k] = it;
                }
                continue;
            }
        }
        if (strips && br == 0) {
            sLin[it] = 1;
            continue;
        }
        do_face(l, t, FACES == WENO_LISTED && br != 0 ? 3 : br);
    }
    if (hybrid || strips) {
        __syncthreads();
        const int n7 = counts[0], n5 = counts[1];
        if constexpr (sizeof(R) == 4) {
            for (int k = threadIdx.x; k < n7 + n5; k += SWEEP_THREADS) {
                int l, t;
                face_lt(k < n7 ? list7[k] : list5[k - n7], l, t);
                do_face(l, t, k < n7 ? 1 : 2);
            }
        } else {
            // chunks of 32 items taken by warps as they come free: the WENO faces first (~1300
            // FP64 instructions each), then the strips, so that no warp waits at the barrier
            // while another works through the block's WENO faces
            const int ns = (nc + LIN_STRIP) / LIN_STRIP, per = ns * (DIR == 0 ? nl : TL), items = 5 * per;
            const int ch7 = (n7 + 31) / 32, ch5 = (n5 + 31) / 32, chs = strips ? (items + 31) / 32 : 0;
            const int lane = threadIdx.x & 31;
            for (;;) {
                int ch = 0;
                if (lane == 0) ch = atomicAdd(&counts[2], 1);
                ch = __shfl_sync(0xffffffffu, ch, 0);
                if (ch >= ch7 + ch5 + chs) break;
                if (FACES != WENO_LISTED && ch < ch7 + ch5) {
                    const bool w7 = ch < ch7;
                    const int k = (w7 ? ch : ch - ch7) * 32 + lane;
                    if (k < (w7 ? n7 : n5)) {
                        int l, t;
                        face_lt(w7 ? list7[k] : list5[k], l, t);
                        do_face(l, t, w7 ? 1 : 2);
                    }
                    continue;
                }
                const int k = (ch - ch7 - ch5) * 32 + lane;
                if (k >= items) continue;
                const int n = k / per, r = k - n * per;
                int l, st;
                if (DIR == 0) { l = r / ns; st = r - l * ns; } else { st = r / TL; l = r - st * TL; }
                const int t0 = st * LIN_STRIP;
                unsigned want = 0u;
#pragma unroll
                for (int f = 0; f < LIN_STRIP; f++)
                    if (t0 + f < NF && sLin[fidx(l, t0 + f)]) want |= 1u << f;
                if (!want) continue;
                const R* fp = sFp + n * TL * NP;
                const R* fm = sFm + n * TL * NP;
                linear_strip(P, t0, nc + 7, want, [&](int p) { return (double)fp[sidx(l, p)]; },
                             [&](int p) { return (double)fm[sidx(l, p)]; },
                             [&](int f, double v) { sF[n * TL * NF + fidx(l, t0 + f)] = v; });
            }
        }
    }
    if (sizeof(R) == 8 && a.faces) {  // face-flux output in the reference's Fx/Fy/Fz shape
        __syncthreads();
        const long long fx = P.nx + (DIR == 0), fy = P.ny + (DIR == 1), fz = P.nz + (DIR == 2), nf = fx * fy * fz;
        for (int it = threadIdx.x; it < TL * NF; it += SWEEP_THREADS) {
            int l, t;
            face_lt(it, l, t);
            if (l >= nl || t > nc) continue;
            long long fi, fj, fk;
            if (DIR == 0) { fi = c0 + t; fj = l0 + l; fk = other; }
            else if (DIR == 1) { fi = l0 + l; fj = c0 + t; fk = other; }
            else { fi = l0 + l; fj = other; fk = c0 + t; }
            const long long fo = fi + fx * (fj + fy * fk);
#pragma unroll
            for (int n = 0; n < 5; n++) a.faces[fo + n * nf] = (double)sF[n * TL * NF + it];
        }
    }
    if (a.out_mode == OUT_FACES) return;
    __syncthreads();

    // ---- Phase C: differences, viscous terms and the accumulation of out_mode.
    sweep_epilogue<DIR, TL, TC, SWEEP_THREADS, R>(a, sF, c0, l0, other, nc, nl, cell, fidx);
}

template <int DIR, int FACES, class R> static cudaError_t configure_dir() {
    return cudaFuncSetAttribute(k_sweep<DIR, FACES, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sweep_smem_bytes<DIR, R>(true));
}

template <int FACES, class R> static cudaError_t configure_faces() {
    cudaError_t e = configure_dir<0, FACES, R>();
    if (e == cudaSuccess) e = configure_dir<1, FACES, R>();
    return e == cudaSuccess ? configure_dir<2, FACES, R>() : e;
}

// Dynamic shared memory above 48 KB must be enabled per kernel before the first launch
// (and outside stream capture): called from f3d_create.
cudaError_t sweep_configure() {
    cudaError_t e;
    if ((e = configure_faces<WENO_COMP, double>()) != cudaSuccess) return e;
    if ((e = configure_faces<WENO_CHAR, double>()) != cudaSuccess) return e;
    if ((e = configure_faces<WENO_LISTED, double>()) != cudaSuccess) return e;
    if ((e = configure_faces<WENO_COMP, float>()) != cudaSuccess) return e;
    if ((e = configure_faces<WENO_CHAR, float>()) != cudaSuccess) return e;
    if ((e = configure_faces<WENO_COMP_REF32, float>()) != cudaSuccess) return e;
    return configure_faces<WENO_CHAR_REF32, float>();
}

template <int DIR, int FACES, class R> static cudaError_t launch_dir(const SweepArgs& a, cudaStream_t st) {
    constexpr int TL = Tile<DIR, R>::TL, TC = Tile<DIR, R>::TC;
    const DevParams& P = a.P;
    const size_t smem = sweep_smem_bytes<DIR, R>(true);
    dim3 grid;
    if (DIR == 0) grid = dim3(cdiv(P.nx, TC), cdiv(P.ny, TL), P.nz);
    else if (DIR == 1) grid = dim3(cdiv(P.nx, TL), cdiv(P.ny, TC), P.nz);
    else grid = dim3(cdiv(P.nx, TL), cdiv(P.nz, TC), P.ny);
    k_sweep<DIR, FACES, R><<<grid, Tile<DIR, R, FACES>::NT, smem, st>>>(a);
    return cudaGetLastError();
}

template <int FACES, class R> static cudaError_t launch_faces(int dir, const SweepArgs& a, cudaStream_t st) {
    if (dir == 0) return launch_dir<0, FACES, R>(a, st);
    return dir == 1 ? launch_dir<1, FACES, R>(a, st) : launch_dir<2, FACES, R>(a, st);
}

// With the WENO faces listed (the hybrid switch in FP64), or a scheme without any, the sweep holds
// no WENO code: 56 registers a thread, and one instance for component- and characteristic-wise faces.
cudaError_t launch_sweep(int dir, const SweepArgs& a, cudaStream_t st) {
    const bool ch = a.P.character != 0;
    if (a.fp32 && a.P.ref32)
        return ch ? launch_faces<WENO_CHAR_REF32, float>(dir, a, st) : launch_faces<WENO_COMP_REF32, float>(dir, a, st);
    if (a.fp32) return ch ? launch_faces<WENO_CHAR, float>(dir, a, st) : launch_faces<WENO_COMP, float>(dir, a, st);
    const int fb = a.P.fixed_branch;
    if (fb == 0 || fb == 3 || (a.wflux && fb < 0)) return launch_faces<WENO_LISTED, double>(dir, a, st);
    return ch ? launch_faces<WENO_CHAR, double>(dir, a, st) : launch_faces<WENO_COMP, double>(dir, a, st);
}

}  // namespace f3d
