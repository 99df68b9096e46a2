// k_weno.cu — the WENO7 / WENO5 faces of the three sweeps, taken out of the tiles.
//
// What bounds it: the FP64 pipe. A characteristic WENO face costs ~1300 FP64 instructions against
// ~60 of a linear one, and shocks put them side by side: on the 256x64x64 shock tube 3% of the eta
// and zeta tiles hold nothing else and ran 8 to 12 times as long as the others, so the SMs that met
// one late worked on while the rest stood idle (FP64 pipe 46% busy over the sweep's duration, SMs
// occupied 73% of it; the xi sweep's WENO faces fill one warp of a tile at a time, whose single
// sub-core then bounds the tile). Here they are listed first and then spread evenly:
//   k_weno_list   one thread per cell: the branch of the faces on its upper side in the three
//                 directions (from the shock sensor, as the sweeps decide it); WENO faces are
//                 appended to one list a direction, WENO7 from its front and WENO5 from its back. The
//                 counts must be zero: the sensor's kernel, which every listing follows, clears them;
//   k_weno_faces  blocks of five warps take 32 faces of one list at a time: the warps split the
//                 eight stencil cells (one cell of 32 faces a warp) and form the face bases, then
//                 take one characteristic field (or component) each, then one flux component each.
//                 Every warp holds 32 faces in the same step, and a face's longest chain is a fifth
//                 of what one thread would run (32 faces: ~1800 FP64 warp instructions in chains
//                 of ~370, against one chain of ~1300 with the split taken from the tile). 171 us a stage
//                 of the tube on average, the FP64 pipe 96% busy (ncu).
// The fluxes go to arrays indexed by direction and left cell, where the sweeps find them: no result
// depends on the order in which faces entered a list.
#include "f3d_face.cuh"

namespace f3d {

// Branch of the face between cell c and the next along a line of stride s: the largest sensor of
// cells c - 2s .. c + 3s
__device__ __forceinline__ int face_branch(const DevParams& P, const double* phi, long long c, long long s) {
    double ph[6];
#pragma unroll
    for (int o = 0; o < 6; o++) ph[o] = phi[c + (o - 2) * s];
    return branch_of(P, ph);
}

__global__ void __launch_bounds__(256) k_weno_list(const DevParams P, const double* __restrict__ phi, const WenoList w) {
    after_previous();
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int g[3] = {0, 0, 0};
    const bool in_grid = c < P.plane;
    if (in_grid) split3(c, P.dnxt, P.dnyt, g[0], g[1], g[2]);
    const int N[3] = {P.nx, P.ny, P.nz};
    const long long st[3] = {1, (long long)P.nxt, (long long)P.nxt * P.nyt};
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        bool face = in_grid;
#pragma unroll
        for (int e = 0; e < 3; e++) face = face && (e == d ? g[e] >= NG - 1 : g[e] >= NG) && g[e] < N[e] + NG;
        const int br = face ? face_branch(P, phi, c, st[d]) : 0;
#pragma unroll
        for (int b = 1; b <= 2; b++) {
            const unsigned m = __ballot_sync(0xffffffffu, br == b);
            if (!m) continue;
            unsigned base = 0u;
            if (lane == __ffs((int)m) - 1) base = atomicAdd(&w.count[(b - 1) * 3 + d], (unsigned)__popc(m));
            base = __shfl_sync(0xffffffffu, base, __ffs((int)m) - 1);
            if (br == b) {
                const long long k = base + (unsigned)__popc(m & ((1u << lane) - 1u));
                w.list[d * P.plane + (b == 1 ? k : P.plane - 1 - k)] = (int)c;
            }
        }
    }
}

constexpr int WF_WARPS = 5, WF_FACES = 32;
struct WenoSmem {
    double f[10 * 8 * WF_FACES];        // Fp (5) and Fm (5) of the eight stencil cells
    CharBasis<F64> basis[WF_FACES];
    F64 flux[5 * WF_FACES];             // characteristic fluxes
    F64 s0[WF_FACES];
};

template <bool CHAR>
__global__ void __launch_bounds__(WF_WARPS * 32, 4) k_weno_faces(const WenoArgs a) {
    __shared__ WenoSmem sm;
    const DevParams& P = a.P;
    const WenoList& w = a.w;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const double* Q = a.Q;
    const long long pl = P.plane;
    int nf[6], nchunk = 0;
#pragma unroll
    for (int li = 0; li < 6; li++) {
        nf[li] = (int)w.count[li];
        nchunk += (nf[li] + WF_FACES - 1) / WF_FACES;
    }
    for (int ch = blockIdx.x; ch < nchunk; ch += gridDim.x) {
        int li = 0, first = ch * WF_FACES, have = 0;
        {
            int left = ch;
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const int n = (nf[q] + WF_FACES - 1) / WF_FACES;
                if (left >= 0 && left < n) { li = q; first = left * WF_FACES; have = min(WF_FACES, nf[q] - first); }
                left -= n;
            }
        }
        const int d = li % 3, br = li / 3 + 1;
        const long long stride = d == 0 ? 1 : (d == 1 ? (long long)P.nxt : (long long)P.nxt * P.nyt);
        const bool on = lane < have;
        const long long k = first + lane;
        const long long cl = on ? (long long)w.list[d * pl + (br == 1 ? k : pl - 1 - k)] : 0ll, cr = cl + stride;
        const double* A0 = a.A[3 * d];
        const double* A1 = a.A[3 * d + 1];
        const double* A2 = a.A[3 * d + 2];
        const double* S = a.S[d];
        double* out = w.flux + (5 * d + wp) * pl + cl;  // component wp of the face
        if (on) {
            for (int p = wp; p < 8; p += WF_WARPS) {
                if (br == 2 && (p == 0 || p == 7)) continue;  // WENO5 reads positions 1 .. 6
                const long long c = cl + (p - 3) * stride;
                F64 q[6], fp[5], fm[5];
#pragma unroll
                for (int n = 0; n < 6; n++) q[n] = f64(Q[c + n * pl]);
                split_cell<F64>(P.split, P.cd, q, f64(a.csnd[c]), f64(A0[c]), f64(A1[c]), f64(A2[c]),
                                f64(a.H[3 * d][c]), f64(a.H[3 * d + 1][c]), f64(a.H[3 * d + 2][c]), f64(S[c]), fp, fm);
#pragma unroll
                for (int n = 0; n < 5; n++) {
                    sm.f[(n * 8 + p) * WF_FACES + lane] = fp[n].v;
                    sm.f[((n + 5) * 8 + p) * WF_FACES + lane] = fm[n].v;
                }
            }
            if (wp == 3) {
                const F64 s0 = F64(2.0) / (f64(S[cl]) + f64(S[cr]));
                sm.s0[lane] = s0;
                auto as = [](const double* p) { return reinterpret_cast<const F64*>(p); };
                if (CHAR) char_basis<F64>(P, as(Q), as(A0), as(A1), as(A2), s0, cl, cr, sm.basis[lane]);
            }
        }
        __syncthreads();
        auto FP = [&](int n, int p) { return f64(sm.f[(n * 8 + p) * WF_FACES + lane]); };
        auto FM = [&](int n, int p) { return f64(sm.f[((n + 5) * 8 + p) * WF_FACES + lane]); };
        if (on) {
            const F64 s0 = sm.s0[lane];
            if (CHAR) sm.flux[wp * WF_FACES + lane] = char_field_flux<F64>(P, sm.basis[lane], wp, br, 0, s0, FP, FM);
            else *out = comp_field_flux<F64>(P, wp, br, 0, s0, FP, FM).v;
        }
        __syncthreads();
        if (CHAR) {
            if (on) {
                F64 flux[5];
#pragma unroll
                for (int n = 0; n < 5; n++) flux[n] = sm.flux[n * WF_FACES + lane];
                *out = char_right_row<F64>(sm.basis[lane], wp, flux).v;
            }
            __syncthreads();
        }
    }
}

cudaError_t launch_weno_list(const DevParams& P, const WenoList& w, const double* phi, cudaStream_t st) {
    launch_after(P, k_weno_list, cdiv(P.plane, 256), 256, st, P, phi, w);
    return cudaGetLastError();
}

// Four blocks of k_weno_faces per SM stay resident and share the lists out among themselves; a grid
// too small to fill them gets one block per 32 of its cells.
cudaError_t launch_weno(const WenoArgs& a, const double* phi, int sms, cudaStream_t st) {
    const long long most = (long long)a.P.nx * a.P.ny * a.P.nz / WF_FACES + 1;
    const int blocks = most < 4 * sms ? (int)most : 4 * sms;
    // without its lists the faces would be those of the state before
    const cudaError_t e = launch_weno_list(a.P, a.w, phi, st);
    if (e != cudaSuccess) return e;
    if (a.P.character) k_weno_faces<true><<<blocks, WF_WARPS * 32, 0, st>>>(a);
    else k_weno_faces<false><<<blocks, WF_WARPS * 32, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace f3d
