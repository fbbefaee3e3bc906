// Discrete adjoint kernels (FP64): the vector-Jacobian product of the RHS and
// of one Shu-Osher stage with its cons<->prim conversions. No counterpart in
// the reference (it has no derivative code).
//
// RHS VJP, per direction d (R = V - sum_d inv_h_d (F_d(f) - F_d(f-1))):
//   lamF(f) = inv_h (lamR(f+1) - lamR(f))                     (face f = f+1/2)
//   reconstruction VJP of every face, lamF+-(c) = sum over the faces whose
//   windows hold c, then the transposed split Jacobian: k_adj_flux in shared
//   memory; for lines too long for that k_adj_face (the window cotangents into
//   G, 2 x S x 5 arrays) and k_adj_cell (the gather)
// Viscous part: lam of the fluxes = D^T lamR = -D lamR (antisymmetric central
// stencils on a periodic line), pointwise flux VJP (tau, q, mu(T)), then the
// gradient transpose -D again.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ns3d_adjoint.cuh"
#include "ns3d_internal.h"
#include "ns3d_kernels.cuh"

namespace ns3d {

namespace {

// index of the cell at line position s (wrapped) given the cell id at position p
struct Line {
    long long id;
    long long stride;
    int pos, len;
    __device__ long long at(int s) const { return id + (long long)(wrap1(s, len) - pos) * stride; }
};

template <int DIR>
__device__ __forceinline__ Line line_of(const DevParams& P, int i, int j, int k, long long id) {
    if constexpr (DIR == 0) return Line{id, 1, i, P.nx};
    else if constexpr (DIR == 1) return Line{id, (long long)P.nx, j, P.ny};
    else return Line{id, (long long)P.nx * P.ny, k, P.nz};
}

__device__ __forceinline__ void load_w5(const StateView& W, long long id, double* w) {
    double rr = W.rho[id];
    if (rr <= 0.0) rr = 1e-12;
    w[0] = rr;
    w[1] = W.u[id];
    w[2] = W.v[id];
    w[3] = W.w[id];
    w[4] = W.p[id];
}

// Forward split at the windows' cells, with Newton-refined reciprocal and
// square roots (split_fast, two steps: about an ulp).
template <int FVS, int DIR>
__device__ __forceinline__ void split_fwd(const double* w5, const DevParams& P, double* Fp,
                                          double* Fm) {
    split_fast<FVS, DIR == 0, DIR == 1, DIR == 2, 2>(P, 1.0 / (P.gamma - 1.0), 0.5 / P.gamma,
                                                     w5, Fp, Fm);
}

// Index of face/cell position f of a line in the split-flux cotangent array G.
// x lines (threads over j) use a j-fastest layout so that a warp's stores are
// contiguous; y and z lines (threads over i) use the cell index itself.
template <int DIR>
__device__ __forceinline__ long long g_index(const DevParams& P, int i, int j, int k) {
    if constexpr (DIR == 0) return ((long long)k * P.nx + i) * P.ny + j;
    else return ((long long)k * P.ny + j) * P.nx + i;
}

// Reconstruction VJP of every face: marches a line segment like k_sweep,
// holding the split fluxes of the face window in registers.
template <int DIR, int FVS, int RC>
__global__ void __launch_bounds__(128)
k_adj_face(DevParams P, StateView W, const double* __restrict__ lamR, double* __restrict__ G,
           int seg) {
    constexpr int S = Stencil<RC>::S;
    constexpr int MID = (S - 1) / 2;
    const int nx = P.nx, ny = P.ny;
    const long long n = P.n;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    long long base, stride;
    int len;
    if constexpr (DIR == 0) {
        if (t0 >= ny) return;
        base = ((long long)blockIdx.y * ny + t0) * nx; stride = 1; len = nx;
    } else if constexpr (DIR == 1) {
        if (t0 >= nx) return;
        base = (long long)blockIdx.y * ny * nx + t0; stride = nx; len = ny;
    } else {
        if (t0 >= nx) return;
        base = (long long)blockIdx.y * nx + t0; stride = (long long)nx * ny; len = P.nz;
    }
    const int c0 = blockIdx.z * seg;
    if (c0 >= len) return;
    const int c1 = min(c0 + seg, len);
    double lin[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) lin[m] = P.lin[m];
    const double inv_h = DIR == 0 ? P.inv_dx : (DIR == 1 ? P.inv_dy : P.inv_dz);
    auto idx = [&](int s) { return base + (long long)wrap1(s, len) * stride; };
    double fp[S][5], fm[S][5];
#pragma unroll
    for (int m = 0; m < S - 1; ++m) {
        double w5[5];
        load_w5(W, idx(c0 - MID + m), w5);
        split_fwd<FVS, DIR>(w5, P, fp[m], fm[m]);
    }
    double lr_here[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) lr_here[q] = lamR[q * n + idx(c0)];
    for (int f = c0; f < c1; ++f) {
        double w5[5];
        load_w5(W, idx(f - MID + S - 1), w5);
        split_fwd<FVS, DIR>(w5, P, fp[S - 1], fm[S - 1]);
        const long long nid = idx(f + 1);
        const long long fid = DIR == 0 ? g_index<0>(P, f, t0, blockIdx.y) : idx(f);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const double lr_next = lamR[q * n + nid];
            const double lamF = inv_h * (lr_next - lr_here[q]);
            lr_here[q] = lr_next;
            double a[S], b[S], ga[S], gb[S];
#pragma unroll
            for (int m = 0; m < S; ++m) {
                a[m] = fp[m][q];
                b[m] = fm[S - 1 - m][q];
                ga[m] = 0.0;
                gb[m] = 0.0;
            }
            reconstruct_vjp<RC>(a, lin, lamF, ga);
            reconstruct_vjp<RC>(b, lin, lamF, gb);
#pragma unroll
            for (int m = 0; m < S; ++m) {
                G[((long long)(0 * S + m) * 5 + q) * n + fid] = ga[m];
                G[((long long)(1 * S + m) * 5 + q) * n + fid] = gb[m];
            }
        }
#pragma unroll
        for (int m = 0; m < S - 1; ++m)
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                fp[m][q] = fp[m + 1][q];
                fm[m][q] = fm[m + 1][q];
            }
    }
}

// Gather of the split-flux cotangents of each cell and the transposed split
// Jacobian: lamW(c) += (dF+/dw)^T lamF+(c) + (dF-/dw)^T lamF-(c).
template <int DIR, int FVS, int RC>
__global__ void __launch_bounds__(128)
k_adj_cell(DevParams P, StateView W, const double* __restrict__ G, double* __restrict__ lamW) {
    constexpr int S = Stencil<RC>::S;
    constexpr int MID = (S - 1) / 2;
    // x: threads over j (G's x layout is j-fastest); y, z: threads over i
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (DIR == 0 ? P.ny : P.nx)) return;
    const int i = DIR == 0 ? (int)blockIdx.y : t, j = DIR == 0 ? t : (int)blockIdx.y;
    const int k = blockIdx.z;
    const long long n = P.n;
    const long long id = ((long long)k * P.ny + j) * P.nx + i;
    const int pos = DIR == 0 ? i : (DIR == 1 ? j : k);
    const int len = DIR == 0 ? P.nx : (DIR == 1 ? P.ny : P.nz);
    auto gat = [&](int s) {
        const int w = wrap1(s, len);
        return DIR == 0 ? g_index<0>(P, w, j, k) : (DIR == 1 ? g_index<1>(P, i, w, k)
                                                             : g_index<2>(P, i, j, w));
    };
    double gp[5], gm[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        double sp = 0.0, sm = 0.0;
#pragma unroll
        for (int m = 0; m < S; ++m) {
            // cell c = f - MID + m in the plus window of face f = c + MID - m
            sp += G[((long long)(0 * S + m) * 5 + q) * n + gat(pos + MID - m)];
            // cell c = f - MID + (S-1-m) in the minus window of face f = c + MID - S + 1 + m
            sm += G[((long long)(1 * S + m) * 5 + q) * n + gat(pos + MID - S + 1 + m)];
        }
        gp[q] = sp;
        gm[q] = sm;
    }
    double w5[5], gw[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    load_w5(W, id, w5);
    split_vjp<FVS, DIR>(w5, P.gamma, P.sw_eps, gp, gm, gw);
#pragma unroll
    for (int q = 0; q < 5; ++q) lamW[q * n + id] += gw[q];
}

// Viscous VJP, part 1: lam of the 12 gradients and the direct lam of u,v,w,T.
// lg blocks: 0..11 gradients (du/dx du/dy du/dz dv/.. dw/.. dT/..), 12..15 u,v,w,T.
template <int ORD>
__device__ __forceinline__ void adj_visc1_cell(const DevParams& P, const StateView& W,
                                               const double* __restrict__ lamR,
                                               double* __restrict__ lg, int i, int j, int k) {
    const long long n = P.n;
    const long long id = ((long long)k * P.ny + j) * P.nx + i;
    const Line Lx = line_of<0>(P, i, j, k, id), Ly = line_of<1>(P, i, j, k, id),
               Lz = line_of<2>(P, i, j, k, id);
    auto d = [&](const double* a, const Line& L, double h) {
        return dcentral<double, ORD>([&](int o) { return a[L.at(L.pos + o)]; }, h);
    };
    const double dx = P.dx, dy = P.dy, dz = P.dz;
    // lam of the fluxes (D^T = -D)
    double lF[4], lH[4], lGz[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double* lr = lamR + (long long)(m + 1) * n;
        lF[m] = -d(lr, Lx, dx);
        lH[m] = -d(lr, Ly, dy);
        lGz[m] = -d(lr, Lz, dz);
    }
    // forward gradients and stresses at the cell
    const double ux = d(W.u, Lx, dx), uy = d(W.u, Ly, dy), uz = d(W.u, Lz, dz);
    const double vx = d(W.v, Lx, dx), vy = d(W.v, Ly, dy), vz = d(W.v, Lz, dz);
    const double wx = d(W.w, Lx, dx), wy = d(W.w, Ly, dy), wz = d(W.w, Lz, dz);
    const double Tx = d(W.T, Lx, dx), Ty = d(W.T, Ly, dy), Tz = d(W.T, Lz, dz);
    const double T = W.T[id];
    const double mu = get_mu<double>(T, P.mu, P.sutherland_s);
    const double kq = P.Cp / P.Pr;
    const double div = ux + vy + wz;
    const double txx = 2.0 * mu * ux - 2.0 / 3.0 * mu * div;
    const double tyy = 2.0 * mu * vy - 2.0 / 3.0 * mu * div;
    const double tzz = 2.0 * mu * wz - 2.0 / 3.0 * mu * div;
    const double txy = mu * (uy + vx), txz = mu * (uz + wx), tyz = mu * (vz + wy);
    const double u = W.u[id], v = W.v[id], w = W.w[id];
    // flux entries: Fv = {txx, txy, txz, ex}, Hv = {txy, tyy, tyz, ey}, Gv = {txz, tyz, tzz, ez}
    double ltxx = lF[0], ltxy = lF[1] + lH[0], ltxz = lF[2] + lGz[0];
    double ltyy = lH[1], ltyz = lH[2] + lGz[1], ltzz = lGz[2];
    const double lex = lF[3], ley = lH[3], lez = lGz[3];
    // e_x = u txx + v txy + w txz + qx, e_y = u txy + v tyy + w tyz + qy, e_z = ...
    double lu = lex * txx + ley * txy + lez * txz;
    double lv = lex * txy + ley * tyy + lez * tyz;
    double lw = lex * txz + ley * tyz + lez * tzz;
    ltxx += lex * u; ltxy += lex * v + ley * u; ltxz += lex * w + lez * u;
    ltyy += ley * v; ltyz += ley * w + lez * v; ltzz += lez * w;
    // q_d = mu Cp/Pr dT_d
    double lmu = kq * (lex * Tx + ley * Ty + lez * Tz);
    const double lTx = lex * mu * kq, lTy = ley * mu * kq, lTz = lez * mu * kq;
    // stresses
    double lux = 2.0 * mu * ltxx, lvy = 2.0 * mu * ltyy, lwz = 2.0 * mu * ltzz;
    const double ldiv = -2.0 / 3.0 * mu * (ltxx + ltyy + ltzz);
    lux += ldiv; lvy += ldiv; lwz += ldiv;
    lmu += ltxx * (2.0 * ux - 2.0 / 3.0 * div) + ltyy * (2.0 * vy - 2.0 / 3.0 * div) +
           ltzz * (2.0 * wz - 2.0 / 3.0 * div);
    lmu += ltxy * (uy + vx) + ltxz * (uz + wx) + ltyz * (vz + wy);
    const double luy = mu * ltxy, lvx = mu * ltxy, luz = mu * ltxz, lwx = mu * ltxz;
    const double lvz = mu * ltyz, lwy = mu * ltyz;
    const double lT = lmu * dmu_dT(T, P.mu, P.sutherland_s);
    const double out[16] = {lux, luy, luz, lvx, lvy, lvz, lwx, lwy, lwz, lTx, lTy, lTz,
                            lu, lv, lw, lT};
#pragma unroll
    for (int q = 0; q < 16; ++q) lg[(long long)q * n + id] = out[q];
}

// Viscous VJP, part 2: gradient transpose (-D) plus the direct parts; T = p/(rho R).
// Added to the cotangent lw of one cell.
template <int ORD>
__device__ __forceinline__ void adj_visc2_cell(const DevParams& P, const StateView& W,
                                               const double* __restrict__ lg, int i, int j, int k,
                                               double lw[5]) {
    const long long n = P.n;
    const long long id = ((long long)k * P.ny + j) * P.nx + i;
    const Line Lx = line_of<0>(P, i, j, k, id), Ly = line_of<1>(P, i, j, k, id),
               Lz = line_of<2>(P, i, j, k, id);
    auto d = [&](int blk, const Line& L, double h) {
        const double* a = lg + (long long)blk * n;
        return dcentral<double, ORD>([&](int o) { return a[L.at(L.pos + o)]; }, h);
    };
    double lv4[4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
        lv4[m] = lg[(long long)(12 + m) * n + id] - d(3 * m, Lx, P.dx) - d(3 * m + 1, Ly, P.dy) -
                 d(3 * m + 2, Lz, P.dz);
    double rr = W.rho[id];
    if (rr <= 0.0) rr = 1e-12;
    const double T = W.T[id];
    lw[1] += lv4[0];
    lw[2] += lv4[1];
    lw[3] += lv4[2];
    lw[4] += lv4[3] / (rr * P.Rgas);
    lw[0] += -lv4[3] * T / rr;
}

// ---------------------------------------------------------------------------
// The RHS VJP in two launches.
//
// k_adj_flux: blocks of whole lines (LineTile) along x, y and z and, beside
// them, the first viscous part. A block splits its cells once into shared
// memory; then, one component at a time, every thread takes the
// reconstruction VJP of a face and, after a barrier, sums its cell's cotangents
// from the faces around it; the cell's ten sums end in the split Jacobian. The
// window cotangents (60 values per cell and direction) never leave the SM:
// writing and gathering them through memory was 126 + 126 MB per direction at
// 64^3, two thirds of the VJP's time. gw: 15 blocks of n, the x, y, z parts.
//
// k_adj_reduce: adds the parts and the second viscous part to a cell's
// cotangent and goes on, in the same thread, with what is pointwise after it:
// the end of a step (finish) and the next stage's adjoint.
// ---------------------------------------------------------------------------
constexpr int ADJ_T = 128;
constexpr int ADJ_NC = 300;  // cells of a block's lines, at most (48 KB of shared memory)

template <int RC>
constexpr int adj_smem(int nc) { return nc * (RC == RC_WENO5 ? 20 : 5) * (int)sizeof(double); }

template <int DIR, int FVS, int RC>
__device__ __forceinline__ void adj_lines(const DevParams& P, const StateView& W,
                                          const double* __restrict__ lamR, double* __restrict__ out,
                                          int b, int lb, double* sm) {
    constexpr int S = Stencil<RC>::S;
    constexpr int MID = (S - 1) / 2;
    const long long n = P.n;
    const LineTile<DIR> tl(P, b, lb);
    const int nc = tl.nc;
    const double inv_h = DIR == 0 ? P.inv_dx : (DIR == 1 ? P.inv_dy : P.inv_dz);
    // cotangent of the face between positions s and s+1, component q
    auto lam_face = [&](int l, int s, int q) {
        return inv_h * (lamR[q * n + tl.id(l, s + 1 == tl.len ? 0 : s + 1)] - lamR[q * n + tl.id(l, s)]);
    };
    auto split_jacobian = [&](int c, const double* gp, const double* gm) {
        int l, s;
        tl.of_slot(c, l, s);
        const long long id = tl.id(l, s);
        double w5[5], gw[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        load_w5(W, id, w5);
        split_vjp<FVS, DIR>(w5, P.gamma, P.sw_eps, gp, gm, gw);
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q * n + id] = gw[q];
    };
    if constexpr (RC == RC_WENO5) {
        double* F = sm;            // [10][nc]: F+0..4, F-0..4; then the cells' sums
        double* G = sm + 10 * nc;  // [10][nc]: window cotangents of one component, plus then minus
        for (int c = threadIdx.x; c < nc; c += ADJ_T) {
            int l, s;
            tl.of_slot(c, l, s);
            double w5[5], Fp[5], Fm[5];
            load_w5(W, tl.id(l, s), w5);
            split_fwd<FVS, DIR>(w5, P, Fp, Fm);
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                F[q * nc + c] = Fp[q];
                F[(5 + q) * nc + c] = Fm[q];
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int q = 0; q < 5; ++q) {
            for (int c = threadIdx.x; c < nc; c += ADJ_T) {
                int l, s;
                tl.of_slot(c, l, s);
                const double lam = lam_face(l, s, q);
                const double* fp = F + q * nc + l * tl.cl;
                const double* fm = fp + 5 * nc;
                double a[5], bm[5], ga[5] = {0, 0, 0, 0, 0}, gb[5] = {0, 0, 0, 0, 0};
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    a[m] = fp[tl.at(s - MID + m)];
                    bm[m] = fm[tl.at(s - MID + S - 1 - m)];
                }
                weno5_vjp(a, lam, ga);
                weno5_vjp(bm, lam, gb);
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    G[m * nc + c] = ga[m];
                    G[(5 + m) * nc + c] = gb[m];
                }
            }
            __syncthreads();
            for (int c = threadIdx.x; c < nc; c += ADJ_T) {
                int l, s;
                tl.of_slot(c, l, s);
                const double* g = G + l * tl.cl;
                double sp = 0.0, sq = 0.0;
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    // cell s = f - MID + m in the plus window of face f = s + MID - m,
                    // and f - MID + (S-1-m) in the minus window of f = s + MID - S + 1 + m
                    sp += g[m * nc + tl.at(s + MID - m)];
                    sq += g[(5 + m) * nc + tl.at(s + MID - S + 1 + m)];
                }
                F[q * nc + c] = sp;  // component q's split fluxes are not read again
                F[(5 + q) * nc + c] = sq;
            }
            __syncthreads();
        }
        for (int c = threadIdx.x; c < nc; c += ADJ_T) {
            double gp[5], gm[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                gp[q] = F[q * nc + c];
                gm[q] = F[(5 + q) * nc + c];
            }
            split_jacobian(c, gp, gm);
        }
    } else {
        // a linear scheme's window cotangents are its coefficients times the face's
        double* lf = sm;  // [5][nc]
        for (int t = threadIdx.x; t < 5 * nc; t += ADJ_T) {
            const int q = t / nc;
            int l, s;
            tl.of_slot(t - q * nc, l, s);
            lf[t] = lam_face(l, s, q);
        }
        __syncthreads();
        for (int c = threadIdx.x; c < nc; c += ADJ_T) {
            int l, s;
            tl.of_slot(c, l, s);
            double gp[5], gm[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const double* f = lf + q * nc + l * tl.cl;
                double sp = 0.0, sq = 0.0;
#pragma unroll
                for (int m = 0; m < S; ++m) {
                    const double c_m = RC == RC_LINEAR ? (m == 0 ? 1.0 : 0.0) : P.lin[m];
                    sp += c_m * f[tl.at(s + MID - m)];
                    sq += c_m * f[tl.at(s + MID - S + 1 + m)];
                }
                gp[q] = sp;
                gm[q] = sq;
            }
            split_jacobian(c, gp, gm);
        }
    }
}

template <int FVS, int RC>
__global__ void __launch_bounds__(ADJ_T, 4)
k_adj_flux(DevParams P, StateView W, const double* __restrict__ lamR, double* __restrict__ gw,
           double* __restrict__ lg, SmallShape sh) {
    pdl_enter(P);
    extern __shared__ double adj_sm[];
    const long long n = P.n;
    int b = blockIdx.x;
    if (b < sh.nb[0]) { adj_lines<0, FVS, RC>(P, W, lamR, gw, b, sh.lb[0], adj_sm); return; }
    b -= sh.nb[0];
    if (b < sh.nb[1]) { adj_lines<1, FVS, RC>(P, W, lamR, gw + 5 * n, b, sh.lb[1], adj_sm); return; }
    b -= sh.nb[1];
    if (b < sh.nb[2]) { adj_lines<2, FVS, RC>(P, W, lamR, gw + 10 * n, b, sh.lb[2], adj_sm); return; }
    b -= sh.nb[2];
    const long long c = (long long)b * ADJ_T + threadIdx.x;
    if (c >= n) return;
    const int i = (int)(c % P.nx), j = (int)(c / P.nx % P.ny), k = (int)(c / ((long long)P.nx * P.ny));
    if (P.vis_order == 4) adj_visc1_cell<4>(P, W, lamR, lg, i, j, k);
    else if (P.vis_order == 6) adj_visc1_cell<6>(P, W, lamR, lg, i, j, k);
    else adj_visc1_cell<8>(P, W, lamR, lg, i, j, k);
}

// Adjoint of one stage. Wk: the stage's output state, Wp: its input state.
// Stage coefficients (U_k = a U0 + bU U(Wp) + bR dt R(Wp)): (1, 0, 1),
// (3/4, 1/4, 1/4), (1/3, 2/3, 2/3). Writes lamR, initialises lamWp with the
// U(Wp) part and accumulates lamU0 (set at stage 3, the first one reversed).
__device__ __forceinline__ void adj_stage_cell(const DevParams& P, int stage, const double wk[5],
                                               const StateView& Wp, long long id, const double lw[5],
                                               double* __restrict__ lamU0, double* __restrict__ lamR,
                                               double* __restrict__ lamWp, double dt) {
    const long long n = P.n;
    const double a = stage == 1 ? 1.0 : (stage == 2 ? 0.75 : 1.0 / 3.0);
    const double bU = stage == 1 ? 0.0 : (stage == 2 ? 0.25 : 2.0 / 3.0);
    const double bR = stage == 1 ? 1.0 : bU;
    double lU[5];
    c2p_vjp(wk, P.gamma, lw, lU);
    double lp[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (stage != 1) {
        double wp[5], lUp[5];
        load_w5(Wp, id, wp);
#pragma unroll
        for (int q = 0; q < 5; ++q) lUp[q] = bU * lU[q];
        p2c_vjp(wp, P.gamma, lUp, lp);
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        if (stage == 3) lamU0[q * n + id] = a * lU[q];
        else lamU0[q * n + id] += a * lU[q];
        lamR[q * n + id] = bR * dt * lU[q];
        lamWp[q * n + id] = lp[q];
    }
}

// One stage reversed at the end of a segment (in the middle, k_adj_reduce).
__global__ void __launch_bounds__(256)
k_adj_stage(DevParams P, int stage, StateView Wk, StateView Wp, const double* lamWk,
            double* __restrict__ lamU0, double* __restrict__ lamR, double* lamWp, double dt) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= P.n) return;
    double wk[5], lw[5];
    load_w5(Wk, id, wk);
#pragma unroll
    for (int q = 0; q < 5; ++q) lw[q] = lamWk[q * P.n + id];
    adj_stage_cell(P, stage, wk, Wp, id, lw, lamU0, lamR, lamWp, dt);
}

// lamW (the cotangent of state W so far) += the parts of k_adj_flux (PARTS; the
// marching kernels have added theirs) and the second viscous part; finish:
// lamW += (dU0/dW)^T lamU0 (W is a step's start state); next > 0: that stage's
// adjoint, whose output state is W and whose input state is Wp, in place.
template <int ORD, bool PARTS>
__global__ void __launch_bounds__(128)
k_adj_reduce(DevParams P, StateView W, const double* __restrict__ gw, const double* __restrict__ lg,
             double* lamW, int finish, int next, StateView Wp, double* __restrict__ lamU0,
             double* __restrict__ lamR, double dt) {
    pdl_enter(P);
    const long long n = P.n;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    const int i = (int)(id % P.nx), j = (int)(id / P.nx % P.ny), k = (int)(id / ((long long)P.nx * P.ny));
    double lw[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        lw[q] = lamW[q * n + id];
        if constexpr (PARTS) lw[q] = ((lw[q] + gw[q * n + id]) + gw[(5 + q) * n + id]) + gw[(10 + q) * n + id];
    }
    adj_visc2_cell<ORD>(P, W, lg, i, j, k, lw);
    double w5[5];
    if (finish || next) load_w5(W, id, w5);
    if (finish) {
        double lU[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) lU[q] = lamU0[q * n + id];
        p2c_vjp(w5, P.gamma, lU, lw);
    }
    if (next) {
        adj_stage_cell(P, next, w5, Wp, id, lw, lamU0, lamR, lamW, dt);
    } else {
#pragma unroll
        for (int q = 0; q < 5; ++q) lamW[q * n + id] = lw[q];
    }
}

// The first viscous part alone, after the marching face kernels.
template <int ORD>
__global__ void __launch_bounds__(128)
k_adj_visc1(DevParams P, StateView W, const double* __restrict__ lamR, double* __restrict__ lg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.nx) return;
    adj_visc1_cell<ORD>(P, W, lamR, lg, i, blockIdx.y, blockIdx.z);
}

// d/dW of J = sum 0.5 rho |u|^2 dV (compute_total_energy, postprocess.cpp:103).
__global__ void __launch_bounds__(256)
k_adj_seed_ke(DevParams P, StateView W, double* __restrict__ lamW, double dV) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= P.n) return;
    const long long n = P.n;
    const double rho = W.rho[id], u = W.u[id], v = W.v[id], w = W.w[id];
    lamW[0 * n + id] = 0.5 * (u * u + v * v + w * w) * dV;
    lamW[1 * n + id] = rho * u * dV;
    lamW[2 * n + id] = rho * v * dV;
    lamW[3 * n + id] = rho * w * dV;
    lamW[4 * n + id] = 0.0;
}

// Boxes with a line too long for a block of k_adj_flux: the marching kernels.
bool long_lines(const DevParams& P) { return P.nx > ADJ_NC || P.ny > ADJ_NC || P.nz > ADJ_NC; }

template <int DIR, int FVS, int RC>
cudaError_t adj_dir(const LaunchCfg& L, StateView W, const double* lamR, double* G, double* lamW) {
    const DevParams& P = L.P;
    const int ext = DIR == 0 ? P.ny : P.nx;
    const int other = DIR == 2 ? P.ny : P.nz;
    const int len = DIR == 0 ? P.nx : (DIR == 1 ? P.ny : P.nz);
    const int seg = detail::segment_for(len, (long long)ext * other);
    const int th = detail::threads_for(ext);
    dim3 grid((ext + th - 1) / th, other, (len + seg - 1) / seg);
    k_adj_face<DIR, FVS, RC><<<grid, th, 0, L.stream>>>(P, W, lamR, G, seg);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int cext = DIR == 0 ? P.ny : P.nx;
    const int tc = detail::threads_for(cext);
    const dim3 cg((cext + tc - 1) / tc, DIR == 0 ? P.nx : P.ny, P.nz);
    k_adj_cell<DIR, FVS, RC><<<cg, tc, 0, L.stream>>>(P, W, G, lamW);
    return cudaGetLastError();
}

// G: the three directions' parts (15 blocks of n) for k_adj_reduce; for long
// lines the window cotangents (10 S blocks), whose sums are added to lamW here.
template <int FVS, int RC>
cudaError_t adj_flux(const LaunchCfg& L, StateView W, const double* lamR, double* G, double* lg, double* lamW) {
    const DevParams& P = L.P;
    if (!long_lines(P)) {
        // 64 to 256 cells a block, as in flux_small. With one line a block along y and z
        // (extents above 150) still faster than the marching kernels: a VJP's kernels,
        // WENO5, 200^3 12.8 -> 6.7 ms, 256^3 22.2 -> 13.0, 40x300x300 6.6 -> 2.9
        const long long target = std::min(256ll, std::max(64ll, 3 * P.n / (2 * 148)));
        const SmallShape sh = small_shape(P, target, ADJ_NC, ADJ_T);
        return launch_pdl(L, k_adj_flux<FVS, RC>, small_blocks(sh), ADJ_T, adj_smem<RC>(small_cells(P, sh)), P, W,
                          lamR, G, lg, sh);
    }
    cudaError_t e = adj_dir<0, FVS, RC>(L, W, lamR, G, lamW);
    if (e == cudaSuccess) e = adj_dir<1, FVS, RC>(L, W, lamR, G, lamW);
    if (e == cudaSuccess) e = adj_dir<2, FVS, RC>(L, W, lamR, G, lamW);
    if (e != cudaSuccess) return e;
    const int th = detail::threads_for(P.nx);
    const dim3 g = detail::cell_grid(P, th);
    if (P.vis_order == 4) k_adj_visc1<4><<<g, th, 0, L.stream>>>(P, W, lamR, lg);
    else if (P.vis_order == 6) k_adj_visc1<6><<<g, th, 0, L.stream>>>(P, W, lamR, lg);
    else k_adj_visc1<8><<<g, th, 0, L.stream>>>(P, W, lamR, lg);
    return cudaGetLastError();
}

template <int FVS>
cudaError_t adj_flux_rc(const LaunchCfg& L, StateView W, const double* lamR, double* G, double* lg, double* lamW) {
    switch (L.rc) {
    case RC_WENO5: return adj_flux<FVS, RC_WENO5>(L, W, lamR, G, lg, lamW);
    case RC_LINEAR: return adj_flux<FVS, RC_LINEAR>(L, W, lamR, G, lg, lamW);
    case RC_LIN6: return adj_flux<FVS, RC_LIN6>(L, W, lamR, G, lg, lamW);
    case RC_LIN8: return adj_flux<FVS, RC_LIN8>(L, W, lamR, G, lg, lamW);
    default: return cudaErrorNotSupported;
    }
}

}  // namespace

int adj_scratch_blocks(const LaunchCfg& L) {
    if (!long_lines(L.P)) return 15;
    const int S = L.rc == RC_LIN8 ? 8 : (L.rc == RC_LINEAR ? 2 : 6);
    return 2 * S * 5;
}

int adj_rhs_vjp_launches(const LaunchCfg& L) { return long_lines(L.P) ? 8 : 2; }

cudaError_t adj_rhs_vjp(const LaunchCfg& L, StateView W, double* G, double* lg, double* lamW, int finish, int next,
                        StateView Wp, double* lamU0, double* lamR, double dt) {
    const DevParams& P = L.P;
    cudaError_t e = L.fvs == FV_SW ? adj_flux_rc<FV_SW>(L, W, lamR, G, lg, lamW)
                                   : adj_flux_rc<FV_LF>(L, W, lamR, G, lg, lamW);
    if (e != cudaSuccess) return e;
    const unsigned b = (unsigned)((P.n + 127) / 128);
    auto reduce = [&](auto parts) {
        constexpr bool PARTS = decltype(parts)::value;
        auto go = [&](auto kernel) {
            return launch_pdl(L, kernel, b, 128, 0, P, W, G, lg, lamW, finish, next, Wp, lamU0, lamR, dt);
        };
        if (P.vis_order == 4) return go(k_adj_reduce<4, PARTS>);
        if (P.vis_order == 6) return go(k_adj_reduce<6, PARTS>);
        return go(k_adj_reduce<8, PARTS>);
    };
    return long_lines(P) ? reduce(std::false_type{}) : reduce(std::true_type{});
}

cudaError_t adj_stage(const LaunchCfg& L, int stage, StateView Wk, StateView Wp, const double* lamWk, double* lamU0,
                      double* lamR, double* lamWp, double dt) {
    k_adj_stage<<<(unsigned)((L.P.n + 255) / 256), 256, 0, L.stream>>>(L.P, stage, Wk, Wp, lamWk, lamU0, lamR, lamWp,
                                                                       dt);
    return cudaGetLastError();
}

cudaError_t adj_seed_ke(const LaunchCfg& L, StateView W, double* lamW, double dV) {
    k_adj_seed_ke<<<(unsigned)((L.P.n + 255) / 256), 256, 0, L.stream>>>(L.P, W, lamW, dV);
    return cudaGetLastError();
}

}  // namespace ns3d
