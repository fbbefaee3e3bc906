// The flux part of one FP64 right-hand side in one launch: the x, y and z
// sweeps and the viscous flux run side by side as blocks of different roles.
//
// On a small box the marching sweeps are bound by latency, not by any pipe:
// one thread splits S cells and reconstructs its faces one after the other, the
// launches depend on each other through T_acc, and a 32^3 box has 1024 lines
// for 148 SMs. Here a block takes a few whole periodic lines into shared
// memory: every thread splits one cell, then reconstructs the face on its right
// (no halo cells, no serial march), then differences. Each direction writes its
// own term, so nothing depends on another launch; the reader adds them in
// T_acc's order (acc_term). The operations per cell and face are those of the
// marching kernels: same bits. A thread takes the components of a face in a
// loop, so that the slot arithmetic is paid once for five (a step at 64^3 315 ->
// 266 us; the FP64 pipe was 54% busy, issue 62%).
//
// FP64 only: the FP32 form's reconstructions work on float deviations from an
// offset per marching segment, and its roundings belong to the marching kernels.
#pragma once

#include "ns3d_kernels.cuh"

namespace ns3d {

#ifndef NS3D_SMALL_T
#define NS3D_SMALL_T 128
#endif
constexpr int SMALL_T = NS3D_SMALL_T;  // threads per block
constexpr int SMALL_NC = 400;          // cells of a block's lines, at most (48 KB of shared memory)

// Launch shape: blocks per role (x, y, z, viscous), lines per block.
struct SmallShape {
    int nb[4], lb[3];
};

// `target` cells per block, four lines or more along y and z (32-byte rows) as
// far as `most` cells hold them: with 400 (300) extents above 100 (75) have three
// lines, above 200 (150) one, whose loads and stores use 8 bytes of a sector. That still beats
// the marching kernels (see small_box). `vth`: cells per block of the fourth role.
inline SmallShape small_shape(const DevParams& P, long long target, int most, int vth) {
    SmallShape sh{};
    for (int d = 0; d < 3; ++d) {
        const int len = d == 0 ? P.nx : (d == 1 ? P.ny : P.nz);
        const long long lines = d == 0 ? (long long)P.ny * P.nz : P.nx;
        long long lb = (target + len / 2) / len;
        if (d > 0 && lb < 4) lb = 4;
        if (lb > most / len) lb = most / len;
        if (lb > lines) lb = lines;
        if (lb < 1) lb = 1;
        sh.lb[d] = (int)lb;
        sh.nb[d] = (int)((lines + lb - 1) / lb) * (d == 0 ? 1 : (d == 1 ? P.nz : P.ny));
    }
    sh.nb[3] = (int)((P.n + vth - 1) / vth);
    return sh;
}
// Cells of the largest block of the shape, blocks of the launch.
inline int small_cells(const DevParams& P, const SmallShape& sh) {
    const int c[3] = {sh.lb[0] * P.nx, sh.lb[1] * P.ny, sh.lb[2] * P.nz};
    const int m = c[0] > c[1] ? c[0] : c[1];
    return m > c[2] ? m : c[2];
}
inline unsigned small_blocks(const SmallShape& sh) {
    return (unsigned)sh.nb[0] + (unsigned)sh.nb[1] + (unsigned)sh.nb[2] + (unsigned)sh.nb[3];
}

// The whole lines along DIR of block b of a role with lb lines per block: line
// l, position s is cell id0 + l dl + s ds and slot l cl + s cs of the block's
// nc = nl len slots (slots consecutive in memory order: coalesced).
template <int DIR>
struct LineTile {
    long long id0, dl, ds;
    int nl, len, cl, cs, nc;
    unsigned rd;  // ceil(2^32 / d), d the divisor of of_slot: c / d = umulhi(c, rd) for c, d < 2^16
    __device__ __forceinline__ LineTile(const DevParams& P, int b, int lb) {
        const int nx = P.nx, ny = P.ny, nz = P.nz;
        len = DIR == 0 ? nx : (DIR == 1 ? ny : nz);
        if constexpr (DIR == 0) {
            const int l0 = b * lb;
            nl = min(lb, ny * nz - l0);
            id0 = (long long)l0 * nx; dl = nx; ds = 1;
        } else {
            const int gx = (nx + lb - 1) / lb, o = b / gx, i0 = (b - o * gx) * lb;
            nl = min(lb, nx - i0);
            id0 = (DIR == 1 ? (long long)o * ny : (long long)o) * nx + i0;
            dl = 1;
            ds = DIR == 1 ? (long long)nx : (long long)nx * ny;
        }
        cl = DIR == 0 ? len : 1;
        cs = DIR == 0 ? 1 : nl;
        nc = nl * len;
        rd = 0xffffffffu / (unsigned)(DIR == 0 ? len : nl) + 1u;  // 0 for d = 1
    }
    __device__ __forceinline__ void of_slot(int c, int& l, int& s) const {
        if constexpr (DIR == 0) {
            l = (int)__umulhi((unsigned)c, rd);  // len >= 8
            s = c - l * len;
        } else {
            s = rd == 0u ? c : (int)__umulhi((unsigned)c, rd);
            l = c - s * nl;
        }
    }
    __device__ __forceinline__ long long id(int l, int s) const { return id0 + l * dl + s * ds; }
    // slot offset of position s (periodic, within a line length of the line)
    __device__ __forceinline__ int at(int s) const { return wrap1(s, len) * cs; }
};

// Shared doubles per cell: split fluxes (10), faces (5) and, for the
// characteristic-wise reconstruction, the Roe averages' terms (5); cells of a
// block's lines at most.
constexpr int small_doubles(bool chr) { return chr ? 20 : 15; }
constexpr int small_most(bool chr) { return chr ? 300 : SMALL_NC; }
constexpr int small_smem(int nc, bool chr) { return nc * small_doubles(chr) * (int)sizeof(double); }

// char_face with everything by the general code, for faces whose values come
// out infinite, NaN or huge below.
template <int DIR, int RC>
__device__ __noinline__ void char_face_cold(const DevParams& P, const double* wl, const double* wr,
                                            const double* F, int nc, const int* w, double* face) {
    char_face<DIR, double, RC>(P.gamma, wl, wr, [&](int m, int r) { return F[r * nc + w[m]]; },
                               [&](int m, int r) { return F[(5 + r) * nc + w[m]]; }, P.lin,
                               P.mdcd_disp, P.mdcd_diss, face);
}

// The face of char_face from the split fluxes F ([10][nc]) at slots w and the
// Roe terms g ([5][nc]: sqrt rho, u, v, w, H) of its two cells: the same
// operations in the same order, without the products with the eigenvectors'
// structural zeros and ones (each adds a zero or is the factor itself: 310
// instead of 500 operations for the projections) and with the branch-free
// quotients. One side's five projected windows are held at a time.
template <int DIR, int RC>
__device__ __forceinline__ void char_face_fast(const DevParams& P, const double* __restrict__ F,
                                               const double* __restrict__ g, int nc, const int* w,
                                               double face[5]) {
    constexpr int S = Stencil<RC>::S;
    constexpr int MID = (S - 1) / 2;
    const double gm1 = P.gamma - 1.0;
    const int cl = w[MID], cr = w[MID + 1];
    const double sl = g[cl], sr = g[cr];
    const double den = quot_mid(1.0, sl + sr);
    auto avg = [&](int k) { return (sl * g[k * nc + cl] + sr * g[k * nc + cr]) * den; };
    const double u0 = avg(1), v0 = avg(2), w0 = avg(3), h0 = avg(4);
    const double V = 0.5 * (u0 * u0 + v0 * v0 + w0 * w0);
    const double un = DIR == 0 ? u0 : (DIR == 1 ? v0 : w0);
    const double c = sqrt_mid(gm1 * (h0 - V));
    const double t2 = DIR == 0 ? v0 : (DIR == 1 ? w0 : u0);
    const double t3 = DIR == 0 ? w0 : (DIR == 1 ? u0 : v0);
    const double chi = quot_mid(0.5, c), K = quot_mid(gm1, c * c), K1 = 0.5 * K;
    // rows 0, 1, 4 of the left eigenvectors; rows 2 and 3 are (-t2, unit vector)
    // and (-t3, unit vector)
    const double ku[3] = {K1 * u0, K1 * v0, K1 * w0};
    double L0[5], L1[5], L4[5];
    L0[0] = K1 * V + chi * un;
    L4[0] = K1 * V - chi * un;
    L1[0] = 1.0 - K * V;
    L1[1] = K * u0; L1[2] = K * v0; L1[3] = K * w0; L1[4] = -K;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        L0[1 + d] = d == DIR ? -chi - ku[d] : -ku[d];
        L4[1 + d] = d == DIR ? chi - ku[d] : -ku[d];
    }
    L0[4] = K1;
    L4[4] = K1;
    constexpr int E2 = DIR == 0 ? 2 : (DIR == 1 ? 3 : 1);  // the unit component of rows 2, 3
    constexpr int E3 = DIR == 0 ? 3 : (DIR == 1 ? 1 : 2);
    double wc[5];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        double a[5][S];
#pragma unroll
        for (int m = 0; m < S; ++m) {
            // reconstruct_select reverses the minus window; WENO5 reads five values
            if (RC == RC_WENO5 && m == 5) continue;
            const int sl_ = w[side == 0 ? m : S - 1 - m];
            double f[5];
#pragma unroll
            for (int r = 0; r < 5; ++r) f[r] = F[(5 * side + r) * nc + sl_];
            double s0 = L0[0] * f[0], s1 = L1[0] * f[0], s4 = L4[0] * f[0];
#pragma unroll
            for (int r = 1; r < 5; ++r) {
                s0 += L0[r] * f[r];
                s1 += L1[r] * f[r];
                s4 += L4[r] * f[r];
            }
            a[0][m] = s0;
            a[1][m] = s1;
            a[2][m] = -t2 * f[0] + f[E2];
            a[3][m] = -t3 * f[0] + f[E3];
            a[4][m] = s4;
        }
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const double r = reconstruct<double, RC>(a[q], P.lin, P.mdcd_disp, P.mdcd_diss);
            wc[q] = side == 0 ? r : wc[q] + r;
        }
    }
    // the right eigenvectors' rows on wc
    const double uc = un * c, vel[3] = {u0, v0, w0};
    face[0] = (wc[0] + wc[1]) + wc[4];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double lo = d == DIR ? vel[d] - c : vel[d], hi = d == DIR ? vel[d] + c : vel[d];
        double t = lo * wc[0] + vel[d] * wc[1];
        if (1 + d == E2) t += wc[2];
        if (1 + d == E3) t += wc[3];
        face[1 + d] = t + hi * wc[4];
    }
    face[4] = (((h0 - uc) * wc[0] + V * wc[1]) + t2 * wc[2] + t3 * wc[3]) + (h0 + uc) * wc[4];
}

// The sweep along DIR of the lines of block b: out (5 blocks of n).
template <int DIR, int FVS, int RC, bool CHR>
__device__ __forceinline__ void small_sweep(const DevParams& P, const StateView& W,
                                            double* __restrict__ out, int b, int lb, double* sm) {
    constexpr int S = Stencil<RC>::S;
    constexpr int MID = (S - 1) / 2;
    const long long n = P.n;
    const LineTile<DIR> tl(P, b, lb);
    const int nc = tl.nc;
    double* F = sm;             // [10][nc]: F+0..4, F-0..4
    double* fl = sm + 10 * nc;  // [5][nc]: face right of each cell
    double* g = sm + 15 * nc;   // CHR [5][nc]: sqrt rho, u, v, w, H of each cell (roe_state)
    for (int c = threadIdx.x; c < nc; c += SMALL_T) {
        int l, s;
        tl.of_slot(c, l, s);
        const long long id = tl.id(l, s);
        const double raw[5] = {W.rho[id], W.u[id], W.v[id], W.w[id], W.p[id]};
        double Fp[5], Fm[5];
        split_fp64<FVS, RC, DIR == 0, DIR == 1, DIR == 2>(P, raw, Fp, Fm);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            F[q * nc + c] = Fp[q];
            F[(5 + q) * nc + c] = Fm[q];
        }
        if constexpr (CHR) {
            const double rho = raw[0], p = raw[4];
            const double E = rho * (0.5 * (raw[1] * raw[1] + raw[2] * raw[2] + raw[3] * raw[3]) +
                                    quot_mid(p, (P.gamma - 1.0) * rho));
            g[c] = sqrt_mid(rho);
            g[nc + c] = raw[1];
            g[2 * nc + c] = raw[2];
            g[3 * nc + c] = raw[3];
            g[4 * nc + c] = quot_mid(E + p, rho);
        }
    }
    __syncthreads();
    if constexpr (CHR) {
        for (int c = threadIdx.x; c < nc; c += SMALL_T) {
            int l, s, w[S];
            tl.of_slot(c, l, s);
#pragma unroll
            for (int m = 0; m < S; ++m) w[m] = tl.at(s - MID + m) + l * tl.cl;
            double face[5];
            char_face_fast<DIR, RC>(P, F, g, nc, w, face);
            if (any_huge(face)) {
                double wl[5], wr[5], fc[5];
                int wi[S];
                const long long il = tl.id(l, s), ir = tl.id(l, s + 1 == tl.len ? 0 : s + 1);
                wl[0] = W.rho[il]; wl[1] = W.u[il]; wl[2] = W.v[il]; wl[3] = W.w[il]; wl[4] = W.p[il];
                wr[0] = W.rho[ir]; wr[1] = W.u[ir]; wr[2] = W.v[ir]; wr[3] = W.w[ir]; wr[4] = W.p[ir];
#pragma unroll
                for (int m = 0; m < S; ++m) wi[m] = w[m];
                char_face_cold<DIR, RC>(P, wl, wr, F, nc, wi, fc);
#pragma unroll
                for (int q = 0; q < 5; ++q) face[q] = fc[q];
            }
#pragma unroll
            for (int q = 0; q < 5; ++q) fl[q * nc + c] = face[q];
        }
    } else {
        // a thread takes a face's components one after the other; of a block with no
        // more cells than half its threads two threads share them
        const bool two = nc <= SMALL_T / 2;
        const int half = two && threadIdx.x >= SMALL_T / 2 ? 1 : 0;
        const int q0 = half ? 3 : 0, q1 = two && !half ? 3 : 5;
        for (int c = threadIdx.x - half * (SMALL_T / 2); c < nc; c += SMALL_T) {
            // the face between positions s and s+1 of line l
            int l, s;
            tl.of_slot(c, l, s);
            int w[S];
#pragma unroll
            for (int m = 0; m < S; ++m) w[m] = tl.at(s - MID + m) + l * tl.cl;
#pragma unroll 1
            for (int q = q0; q < q1; ++q) {
                const double* fp = F + q * nc;
                const double* fm = fp + 5 * nc;
                double a[S], bm[S];
#pragma unroll
                for (int m = 0; m < S; ++m) {
                    a[m] = fp[w[m]];
                    bm[S - 1 - m] = fm[w[m]];  // reconstruct_select reverses for flag < 0
                }
                const double rp = reconstruct<double, RC>(a, P.lin, P.mdcd_disp, P.mdcd_diss);
                const double rm = reconstruct<double, RC>(bm, P.lin, P.mdcd_disp, P.mdcd_diss);
                double f = rp + rm;
                if constexpr (RC == RC_WENO5) {  // as in recon_face (the two may cancel)
                    if (face_huge(rp) || face_huge(rm))
                        f = weno5_ieee<double>(a[0], a[1], a[2], a[3], a[4]) +
                            weno5_ieee<double>(bm[0], bm[1], bm[2], bm[3], bm[4]);
                }
                fl[q * nc + c] = f;
            }
            if (two) break;
        }
    }
    __syncthreads();
    const double inv_h = DIR == 0 ? P.inv_dx : (DIR == 1 ? P.inv_dy : P.inv_dz);
    for (int c = threadIdx.x; c < nc; c += SMALL_T) {
        int l, s;
        tl.of_slot(c, l, s);
        const int left = l * tl.cl + tl.at(s - 1);
        double* o = out + tl.id(l, s);
#pragma unroll
        for (int q = 0; q < 5; ++q) o[q * n] = (fl[q * nc + c] - fl[q * nc + left]) * inv_h;
    }
}

// t3: 15 blocks of n, the x, y and z terms of the five components; fv: the
// viscous fluxes in store_fv's layout.
template <int FVS, int RC, bool CHR>
__global__ void __launch_bounds__(SMALL_T, (CHR ? 384 : 512) / SMALL_T)
k_flux_small(DevParams P, StateView W, double* __restrict__ t3, double* __restrict__ fv, SmallShape sh,
             const Ctrl* __restrict__ ctrl) {
    pdl_enter(P);
    if (ctrl && ctrl->stop) return;
    extern __shared__ double small_sm[];
    const long long n = P.n;
    int b = blockIdx.x;
    if (b < sh.nb[0]) {
        small_sweep<0, FVS, RC, CHR>(P, W, t3, b, sh.lb[0], small_sm);
        return;
    }
    b -= sh.nb[0];
    if (b < sh.nb[1]) {
        small_sweep<1, FVS, RC, CHR>(P, W, t3 + 5 * n, b, sh.lb[1], small_sm);
        return;
    }
    b -= sh.nb[1];
    if (b < sh.nb[2]) {
        small_sweep<2, FVS, RC, CHR>(P, W, t3 + 10 * n, b, sh.lb[2], small_sm);
        return;
    }
    b -= sh.nb[2];
    const int c = b * SMALL_T + threadIdx.x;
    if (c >= n) return;
    const int i = c % P.nx, jk = c / P.nx, j = jk % P.ny, k = jk / P.ny;
    if (P.vis_order == 4) visc_cell<double, 4>(P, W, fv, i, j, k);
    else if (P.vis_order == 6) visc_cell<double, 6>(P, W, fv, i, j, k);
    else visc_cell<double, 8>(P, W, fv, i, j, k);
}

// The rest of a stage (STAGE 1 to 3, k_update's operations) or of a right-hand
// side (STAGE 0, k_rhs_out's) of a small box: 32 cells by five warps. Warps 0 to
// 3 take the viscous divergence of one momentum or energy component each and
// the fifth the two conserved states, then the stage: a quarter of k_update's 96
// neighbour loads per thread one after the other, which is what bounds it there
// (a stage at 16^3: 6 us against 8; from 48^3 on k_update's larger number of
// cells in flight is the better one; between 32^3 and 48^3 not measured; four warps,
// with the stage in warp 0, measured 2% slower than five). STAGE 0 has no wider
// form: a right-hand side's kernels, marching ones with k_rhs_out -> k_flux_small with
// this: 48^3 136 -> 57 us, 100^3 534 -> 392 us, 200^3 3.21 -> 2.96 ms.
template <int ORD, int STAGE>
__global__ void __launch_bounds__(160)
k_update_small(DevParams P, StateView Wc, StateView W0, const double* __restrict__ t3,
               const double* __restrict__ fv, StateOut Wn, Ctrl* ctrl, double* __restrict__ rhs) {
    if constexpr (STAGE > 0) {
        pdl_enter(P);
        if (ctrl->stop) return;
    } else {
        if (P.pdl) pdl_wait();
    }
    __shared__ double rs[5][32];
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    const long long n = P.n;
    const int cell = blockIdx.x * 32 + lane;
    const bool live = cell < n;
    const long long id = live ? cell : 0;
    double r = 0.0;
    if (wq < 4) {
        const int nx = P.nx, ny = P.ny, nz = P.nz;
        const int i = (int)(id % nx), jk = (int)(id / nx), j = jk % ny, k = jk / ny;
        const long long sxy = (long long)nx * ny;
        // flux blocks of component wq + 1 along x, y, z (see cell_visc)
        const double* X = fv + (wq == 0 ? 0 : (wq == 1 ? 3 : (wq == 2 ? 4 : 6))) * n + id;
        const double* Y = fv + (wq == 0 ? 3 : (wq == 1 ? 1 : (wq == 2 ? 5 : 7))) * n + id;
        const double* Z = fv + (wq == 0 ? 4 : (wq == 1 ? 5 : (wq == 2 ? 2 : 8))) * n + id;
        r += dcentral_dir<double, ORD>(P, 0, [&](int o) { return X[wrap1(i + o, nx) - i]; }, P.dx);
        r += dcentral_dir<double, ORD>(P, 1, [&](int o) { return Y[(long long)(wrap1(j + o, ny) - j) * nx]; }, P.dy);
        r += dcentral_dir<double, ORD>(P, 2, [&](int o) { return Z[(long long)(wrap1(k + o, nz) - k) * sxy]; }, P.dz);
    }
    const int q = wq < 4 ? wq + 1 : 0;
    r += -acc_term<double, true>(t3, n, q, id);
    if constexpr (STAGE == 0) {
        if (live) rhs[q * n + id] = r;
    } else {
        double U0[5], U[5];
        if (wq == 4) stage_load<double, STAGE>(P, Wc, W0, id, U0, U);
        else rs[q][lane] = r;
        __syncthreads();
        if (wq < 4) return;
        const double rc[5] = {r, rs[1][lane], rs[2][lane], rs[3][lane], rs[4][lane]};
        double cand = CFL_INIT;
        if (live) stage_apply<double, STAGE>(P, U0, U, id, rc, ctrl->dt, Wn, ctrl, cand);
        if constexpr (STAGE == 3) {
            unsigned long long b = (cand == cand) ? pos_double_bits(cand) : ~0ull;  // NaN never wins
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long x = __shfl_xor_sync(0xffffffffu, b, o);
                b = x < b ? x : b;
            }
            if (lane == 0 && b != ~0ull) atomicMin(&ctrl->dtmin_bits, b);
        }
    }
}

}  // namespace ns3d
