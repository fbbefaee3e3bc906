// Launchers for the stage kernels. Included by exactly one translation unit
// per compute type (ns3d_fp64.cu: double, -fmad=false; ns3d_fp32.cu: float),
// which instantiates them explicitly.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ns3d_kernels.cuh"
#include "ns3d_small.cuh"

namespace ns3d {

struct LaunchCfg {
    DevParams P;
    int fvs;      // FV_SW / FV_LF
    int rc;       // RC_* of the reconstruction
    int chr;      // 1: characteristic-wise reconstruction (char_recon)
    int seg[3];   // cells per thread segment along x, y, z
    cudaStream_t stream;
    int zb;       // planes per block of the 2.5-D viscous kernels (0: from the grid)
    int tiled;    // bit 0: 2.5-D visc_flux (when the box tiles); bit 1: its pipelined form
    long long small;  // FP64 boxes of at most so many cells take k_flux_small (see small_box)
    int rows;     // FP32 Lax-Friedrichs x sweep off the warp rows by k_sweep_x_rows: 1 always, 0 never, -1 where x_rows_box() holds
    int pipe;     // FP32 sweeps with the software-pipelined split: bit 0 the x sweep
                  // (k_sweep_x_pipe, rows of >= 128 cells), bit 1 the y / z sweeps (k_sweep_pipe)
};

// Launch-shape defaults, overridable by NS3D_TILE_ZB / NS3D_TILED / NS3D_SEG / NS3D_PIPE /
// NS3D_SMALL / NS3D_PDL / NS3D_XROWS for tuning.
void default_tiling(LaunchCfg& L);

// One inviscid sweep (dir 0, 1, 2 in this order per RHS evaluation).
template <class R>
cudaError_t launch_sweep(const LaunchCfg& L, int dir, StateView W, R* tacc, const Ctrl* ctrl);
template <class R>
cudaError_t launch_visc_flux(const LaunchCfg& L, StateView W, R* fv, const Ctrl* ctrl);
template <class R>
cudaError_t launch_update(const LaunchCfg& L, int stage, StateView Wc, StateView W0,
                          const R* tacc, const R* fv, StateOut Wn, Ctrl* ctrl);
template <class R>
cudaError_t launch_rhs_out(const LaunchCfg& L, const R* tacc, const R* fv, double* rhs);
// All fluxes of an FP64 right-hand side in one launch (k_flux_small): tacc (15
// blocks of n) and fv. For boxes of small_box() only.
cudaError_t launch_flux_small(const LaunchCfg& L, StateView W, double* tacc, double* fv, const Ctrl* ctrl);
constexpr long long kSmallUpdateCells = 33000;  // stages of larger boxes: k_update (see k_update_small)
// The rest of the stage (1 to 3; rhs unused) or of the right-hand side (stage 0;
// Wc, W0, Wn and ctrl unused) from launch_flux_small's terms.
cudaError_t launch_update_small(const LaunchCfg& L, int stage, StateView Wc, StateView W0, const double* tacc,
                                const double* fv, StateOut Wn, Ctrl* ctrl, double* rhs);

// A launch whose kernel calls pdl_wait: with P.pdl it may start while its
// predecessor in the stream drains.
template <class... K, class... A>
cudaError_t launch_pdl(const LaunchCfg& L, void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = L.stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = L.P.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}
// The z sweep fused with the stage update (k_sweep_ring<2, ..., FUSE>): T_acc
// holds the x + y terms, fv the viscous fluxes of Wc; writes Wn. Component-wise
// reconstruction only (L.chr == 0; cudaErrorNotSupported otherwise).
template <class R>
cudaError_t launch_sweep_z_update(const LaunchCfg& L, int stage, StateView Wc, StateView W0,
                                  const R* tacc, const R* fv, StateOut Wn, Ctrl* ctrl);

namespace detail {

inline int threads_for(int ext) { return ext >= 128 ? 128 : (ext >= 64 ? 64 : 32); }

inline dim3 cell_grid(const DevParams& P, int th) { return dim3((P.nx + th - 1) / th, P.ny, P.nz); }

// Cells per marching segment: long segments amortise the S-1 halo splits at
// the segment start, short ones give enough threads to fill 148 SMs. One cell
// per 1024 lines, within [1, 64] (and <= len): the fastest lengths measured on
// a B200 were 1 at 32^3 (1024 lines), 4 at 64^3, 16 at 128^3 and 64 at 256^3.
inline int segment_for(int len, long long lines) {
    long long seg = lines / 1024;
    seg = seg < 1 ? 1 : (seg > 64 ? 64 : seg);
    return seg > len ? len : (int)seg;
}

}  // namespace detail

// Whether an FP64 box takes launch_flux_small: every line short enough for a
// block's shared memory, no tuning override of the marching kernels, and few
// enough cells: L.small (1500000) where nx is a multiple of 32 and the x sweep
// marches a warp per row (a step at 64^3 356 -> 265 us, 112^3 1917 -> 1508 us
// WENO5 and 1214 -> 1044 us MDCD; 128^3 2092 -> 2102 and 1319 -> 1456; flat boxes just
// below the limit gain in WENO5, 32x216x216 1876 -> 1694, and lose in MDCD, 1182 -> 1323),
// six times as many elsewhere, where it marches a thread per row (100x75x90 1203 ->
// 773 us, 200^3 10.2 -> 8.6 ms WENO5, 6.6 -> 6.2 ms MDCD) and with characteristic-wise
// reconstruction (200^3 16.2 -> 12.9 ms, 12.5 -> 11.0). With one line a block along y and
// z: 30x390x390 6.25 -> 5.18 ms WENO5, 4.05 -> 4.06 MDCD; 300x300x90 10.0 -> 9.11, 6.62 ->
// 6.73; 210x210x200 11.0 -> 9.68, 7.34 -> 7.36; characteristic 100x290x300 17.8 -> 13.6, 14.0 ->
// 11.4, 160^3 8.41 -> 6.57, 6.32 -> 6.02. (Marching kernels -> k_flux_small throughout.)
inline bool small_box(const LaunchCfg& L) {
    const DevParams& P = L.P;
    const int most = small_most(L.chr != 0);
    return L.small && P.n <= (P.nx % 32 == 0 && !L.chr ? L.small : 6 * L.small) && P.nx <= most && P.ny <= most &&
           P.nz <= most;
}

// Boxes whose launches overlap by programmatic dependent launch: those whose
// kernels last some tens of microseconds (FP64 32^3 91 -> 76 us a step, 64^3
// 281 -> 266 us; FP32 8^3 101 -> 76 us, 64^3 243 -> 212 us, 96^3 616 -> 587 us). On
// larger ones the next kernel's waiting blocks cost more than the overlap gains
// (FP64 128^3 MDCD 1308 -> 1449 us, FP32 90x100x84 651 -> 665), in the FP32
// form's eight-point schemes earlier (75^3 455 -> 520 us, 64^3 228 -> 197). Two
// shapes of FP32 boxes inside those limits lose, both with launches of many
// 32-thread blocks whose lanes are not all live, each of which waits and signals:
// narrow ones with very many rows (10x500x100 C4th linear 570 -> 626 us, LF WENO5
// 1050 -> 1102; 9x130x121, 15730 rows, gains: 547 -> 519), and of the boxes with nx
// below 64 and no multiple of 32 those of 55000 to 140000 cells, with the C8th
// viscous terms or Lax-Friedrichs + WENO5 and all but the two-point scheme (LF MDCD
// 54x43x47 185 -> 209, 53x26x54 166 -> 183, 49x37x46 180 -> 192, LF WENO5 55x54x46 213 -> 238;
// smaller and larger ones gain, LF MDCD 34^3 153 -> 141, 52^3 207 -> 183).
// Characteristic-wise and MDCD_HYBRID boxes above 30000 cells are left out on no
// more than caution: overlapped they would gain on warp rows (64^3 FP64 369 -> 353 and
// 383 -> 368 us, FP32 373 -> 336 and 327 -> 294; 80^3 FP64 equal; 40^3 FP32 equal).
inline bool pdl_box(const LaunchCfg& L, bool fp64) {
    const DevParams& P = L.P;
    const long long n = P.n;
    if (n <= 30000) return true;
    if (L.chr || L.rc == RC_MDCD_HYBRID) return false;
    if (fp64) return n <= 300000;
    if ((long long)P.ny * P.nz > 30000) return false;
    if (P.nx < 64 && P.nx % 32 != 0 && n >= 55000 && n <= 140000 && L.rc != RC_LINEAR &&
        (P.vis_order == 8 || (L.rc == RC_WENO5 && L.fvs == FV_LF)))
        return false;
    return n <= 700000 && (L.rc != RC_LIN8 || (P.nx % 32 == 0 && n <= 300000));
}

#ifdef NS3D_LAUNCH_IMPL

namespace detail {

// Launch shape of a marching sweep along DIR (threads over the line index of
// `ext`, blockIdx.y over `other`, blockIdx.z over segments of `seg` cells).
struct MarchShape {
    dim3 grid;
    int th, seg;
};
template <int DIR>
inline MarchShape march_shape(const LaunchCfg& L, int max_threads) {
    const DevParams& P = L.P;
    const int ext = DIR == 0 ? P.ny : P.nx;        // thread dimension
    const int other = DIR == 2 ? P.ny : P.nz;     // blockIdx.y dimension
    const int len = DIR == 0 ? P.nx : (DIR == 1 ? P.ny : P.nz);
    MarchShape m;
    m.seg = L.seg[DIR] > 0 ? L.seg[DIR] : segment_for(len, (long long)ext * other);
    m.th = threads_for(ext);
    if (m.th > max_threads) m.th = max_threads;
    m.grid = dim3((ext + m.th - 1) / m.th, other, (len + m.seg - 1) / m.seg);
    return m;
}

// Whether the pipelined FP32 sweeps prefetch into L2: linear schemes on boxes
// whose sweep (60 bytes per cell) exceeds the 126 MB L2 (a step at 256^3 MDCD 5600
// -> 5220 us, linear 4980 -> 4810; 384^3 UPWIND_7TH 20.8 -> 20.5 ms; 128^3 876 -> 906).
template <int RC>
inline bool prefetched(const DevParams& P) {
    return (RC == RC_LINEAR || RC == RC_LIN6 || RC == RC_LIN8) && P.n > 2200000;
}
// f(entropy fix as a constant, prefetch as a constant) for the pipelined sweeps.
template <int FVS, int RC, class F>
cudaError_t by_split(const DevParams& P, F f) {
    auto by_pf = [&](auto ent) -> cudaError_t {
        if constexpr (RC != RC_WENO5 && RC != RC_MDCD_HYBRID) {
            if (prefetched<RC>(P)) return f(ent, std::true_type{});
        }
        return f(ent, std::false_type{});
    };
    if constexpr (FVS == FV_SW) {
        if (P.sw_eps > 0.0) return by_pf(std::integral_constant<int, 1>{});  // the entropy fix, compiled in
    }
    return by_pf(std::integral_constant<int, 0>{});
}

// Whether the FP32 Lax-Friedrichs x sweep off the warp rows takes k_sweep_x_rows: it
// copies eight columns of 128 rows at a time, so it needs cells enough for the
// grid (24^3 76 -> 81 us a step), more than a chunk or two of columns (10x500x100
// WENO5 1103 -> 1120 us, 17x90x100 equal, 20x155x154 UD7L 627 -> 581) and segments
// of several of them (rows/1024 cells each): with 5600 rows every scheme gains
// (75^3 WENO5 390 -> 373, UD7L 379 -> 366; 100x75x90 509 -> 467, 471 -> 436), with fewer
// the eight-point window's extra splits lose (70x51x41, 2091 rows, 216 -> 231,
// 130x40x40 273 -> 304; 4200 rows even) and long rows in WENO5 (501x60x60 1171 -> 1243,
// 250x60x70 666 -> 679; but 58x44x58 240 -> 200, 60^3 265 -> 249), and with 400 to 1800 rows
// the rest too (2001x20x20 MDCD 592 -> 672; 70x51x41 167 -> 164, 75x60x50 215 -> 204).
inline bool x_rows_box(const LaunchCfg& L) {
    if (L.rows >= 0) return L.rows != 0;
    const DevParams& P = L.P;
    const long long rows = (long long)P.ny * P.nz;
    if (P.n <= 140000 || P.nx < 16) return false;
    if (rows > 5000) return true;
    return rows > 2000 && L.rc != RC_LIN8 && (L.rc != RC_WENO5 || P.nx <= 100);
}

// k_sweep_x_rows: 62 KB of dynamic shared memory, opted in once per
// instantiation and device.
template <int FVS, int RC>
cudaError_t x_rows(const LaunchCfg& L, StateView W, float* tacc, int seg, const Ctrl* ctrl) {
    static bool opted[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !opted[dev]) {
        e = cudaFuncSetAttribute(k_sweep_x_rows<FVS, RC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)XR_SMEM);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) opted[dev] = true;
    }
    const dim3 grid((unsigned)(((long long)L.P.ny * L.P.nz + XR_T - 1) / XR_T), (L.P.nx + seg - 1) / seg);
    return launch_pdl(L, k_sweep_x_rows<FVS, RC>, grid, XR_T, XR_SMEM, L.P, W, tacc, seg, ctrl);
}

template <int DIR, class R, int FVS, int RC, bool CHR>
cudaError_t sweep_dir(const LaunchCfg& L, StateView W, R* tacc, const Ctrl* ctrl) {
    const DevParams& P = L.P;
    if (DIR == 0 && P.nx % 32 == 0) {
        const long long rows = (long long)P.ny * P.nz;
        const unsigned blocks = (unsigned)((rows + XW_WARPS - 1) / XW_WARPS);
        if constexpr (sizeof(R) == 4 && !CHR) {
            if ((L.pipe & 1) && P.nx >= 128) {
                return by_split<FVS, RC>(P, [&](auto ent, auto pf) {
                    return launch_pdl(L, k_sweep_x_pipe<FVS, RC, decltype(ent)::value, decltype(pf)::value>, blocks,
                                      32 * XW_WARPS, 0, P, W, tacc, ctrl);
                });
            }
            return launch_pdl(L, k_sweep_x_warp_f32<FVS, RC>, blocks, 32 * XW_WARPS, 0, P, W, tacc, ctrl);
        } else {
            return launch_pdl(L, k_sweep_x_warp<R, FVS, RC, CHR>, blocks, 32 * XW_WARPS, 0, P, W, tacc, ctrl);
        }
    }
    if constexpr (DIR != 0 && !CHR) {
        const MarchShape m = march_shape<DIR>(L, RingCfg<R>::T);
        if constexpr (sizeof(R) == 4) {
            if (L.pipe & 2) {
                return by_split<FVS, RC>(P, [&](auto ent, auto pf) {
                    return launch_pdl(L, k_sweep_pipe<DIR, FVS, RC, decltype(ent)::value, decltype(pf)::value>, m.grid,
                                      m.th, 0, P, W, tacc, m.seg, ctrl);
                });
            }
        }
        return launch_pdl(L, k_sweep_ring<DIR, R, FVS, RC, false>, m.grid, m.th, 0,
            P, W, tacc, m.seg, ctrl, FuseArgs<R>{});
    } else {
        const MarchShape m = march_shape<DIR>(L, 128);
        // Lax-Friedrichs only: beside another loop the compiler contracts the
        // Steger-Warming split's sums into other FMAs, and the float deviations'
        // roundings flip.
        if constexpr (sizeof(R) == 4 && !CHR && FVS == FV_LF) {
            if (x_rows_box(L)) return x_rows<FVS, RC>(L, W, tacc, m.seg, ctrl);
        }
        return launch_pdl(L, k_sweep<DIR, R, FVS, RC, CHR>, m.grid, m.th, 0, P, W, tacc, m.seg, ctrl);
    }
}

template <class R, int FVS, int RC>
cudaError_t sweep_z_update(const LaunchCfg& L, const FuseArgs<R>& F, StateView Wc,
                           const R* tacc) {
    const MarchShape m = march_shape<2>(L, RingCfg<R>::T);
    return launch_pdl(L, k_sweep_ring<2, R, FVS, RC, true>, m.grid, m.th, 0,
        L.P, Wc, const_cast<R*>(tacc), m.seg, F.ctrl, F);
}

// L.chr selects the characteristic-wise sweeps (du_inviscous_character).
template <class R, int FVS, int RC>
cudaError_t sweeps(const LaunchCfg& L, int dir, StateView W, R* tacc, const Ctrl* ctrl) {
    if (L.chr) {
        if (dir == 0) return sweep_dir<0, R, FVS, RC, true>(L, W, tacc, ctrl);
        if (dir == 1) return sweep_dir<1, R, FVS, RC, true>(L, W, tacc, ctrl);
        return sweep_dir<2, R, FVS, RC, true>(L, W, tacc, ctrl);
    }
    if (dir == 0) return sweep_dir<0, R, FVS, RC, false>(L, W, tacc, ctrl);
    if (dir == 1) return sweep_dir<1, R, FVS, RC, false>(L, W, tacc, ctrl);
    return sweep_dir<2, R, FVS, RC, false>(L, W, tacc, ctrl);
}

template <class R, int FVS>
cudaError_t sweeps_rc(const LaunchCfg& L, int dir, StateView W, R* tacc, const Ctrl* ctrl) {
    switch (L.rc) {
    case RC_WENO5: return sweeps<R, FVS, RC_WENO5>(L, dir, W, tacc, ctrl);
    case RC_LINEAR: return sweeps<R, FVS, RC_LINEAR>(L, dir, W, tacc, ctrl);
    case RC_LIN6: return sweeps<R, FVS, RC_LIN6>(L, dir, W, tacc, ctrl);
    case RC_MDCD_HYBRID: return sweeps<R, FVS, RC_MDCD_HYBRID>(L, dir, W, tacc, ctrl);
    case RC_LIN8: return sweeps<R, FVS, RC_LIN8>(L, dir, W, tacc, ctrl);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace detail

template <class R>
cudaError_t launch_sweep(const LaunchCfg& L, int dir, StateView W, R* tacc, const Ctrl* ctrl) {
    return L.fvs == FV_SW ? detail::sweeps_rc<R, FV_SW>(L, dir, W, tacc, ctrl)
                          : detail::sweeps_rc<R, FV_LF>(L, dir, W, tacc, ctrl);
}

template <class R>
cudaError_t launch_sweep_z_update(const LaunchCfg& L, int stage, StateView Wc, StateView W0,
                                  const R* tacc, const R* fv, StateOut Wn, Ctrl* ctrl) {
    if (L.chr) return cudaErrorNotSupported;
    const FuseArgs<R> F{stage, W0, fv, Wn, ctrl};
    auto by_rc = [&](auto fvs) -> cudaError_t {
        constexpr int FVS = decltype(fvs)::value;
        switch (L.rc) {
        case RC_WENO5: return detail::sweep_z_update<R, FVS, RC_WENO5>(L, F, Wc, tacc);
        case RC_LINEAR: return detail::sweep_z_update<R, FVS, RC_LINEAR>(L, F, Wc, tacc);
        case RC_LIN6: return detail::sweep_z_update<R, FVS, RC_LIN6>(L, F, Wc, tacc);
        case RC_MDCD_HYBRID: return detail::sweep_z_update<R, FVS, RC_MDCD_HYBRID>(L, F, Wc, tacc);
        case RC_LIN8: return detail::sweep_z_update<R, FVS, RC_LIN8>(L, F, Wc, tacc);
        default: return cudaErrorInvalidValue;
        }
    };
    return L.fvs == FV_SW ? by_rc(std::integral_constant<int, FV_SW>{})
                          : by_rc(std::integral_constant<int, FV_LF>{});
}

namespace detail {
template <class R>
inline bool tiles_25d(const LaunchCfg& L, int bit) {
    return (L.tiled & bit) && L.zb >= 0 && L.P.nx % VTile<R>::X == 0 && L.P.ny % VTile<R>::Y == 0;
}
// Planes per block of the 2.5-D kernels: L.zb when set, else 16 halved until
// the grid has at least 4 blocks per SM (32^3: 1 plane, 128^3: 8, 256^3: 16).
template <class R>
inline int zb_for(const LaunchCfg& L) {
    if (L.zb > 0) return L.zb;
    const long long tiles = (long long)(L.P.nx / VTile<R>::X) * (L.P.ny / VTile<R>::Y);
    int zb = 16;
    while (zb > 1 && tiles * ((L.P.nz + zb - 1) / zb) < 4 * 148) zb >>= 1;
    return zb;
}
template <class R>
inline dim3 grid_25d(const LaunchCfg& L) {
    const int zb = zb_for<R>(L);
    return dim3(L.P.nx / VTile<R>::X, L.P.ny / VTile<R>::Y, (L.P.nz + zb - 1) / zb);
}
// k_visc_flux_pipe<R, ORD>: more than 48 KB of dynamic shared memory, opted
// in once per instantiation and device (setting it twice is harmless).
template <class R, int ORD>
cudaError_t visc_pipe(const LaunchCfg& L, StateView W, R* fv, const Ctrl* ctrl) {
    constexpr int sm = (int)VPipe<R>::smem_bytes;
    static bool opted[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !opted[dev]) {
        e = cudaFuncSetAttribute(k_visc_flux_pipe<R, ORD>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) opted[dev] = true;
    }
    const dim3 g = grid_25d<R>(L), b(VTile<R>::X, VTile<R>::Y);
    return launch_pdl(L, k_visc_flux_pipe<R, ORD>, g, b, sm, L.P, W, fv, ctrl, zb_for<R>(L));
}
}  // namespace detail

template <class R>
cudaError_t launch_visc_flux(const LaunchCfg& L, StateView W, R* fv, const Ctrl* ctrl) {
    if (detail::tiles_25d<R>(L, 1) && (L.tiled & 2)) {
        switch (L.P.vis_order) {
        case 4: return detail::visc_pipe<R, 4>(L, W, fv, ctrl);
        case 6: return detail::visc_pipe<R, 6>(L, W, fv, ctrl);
        default: return detail::visc_pipe<R, 8>(L, W, fv, ctrl);
        }
    }
    if (detail::tiles_25d<R>(L, 1)) {
        const dim3 g = detail::grid_25d<R>(L), b(VTile<R>::X, VTile<R>::Y);
        switch (L.P.vis_order) {
        case 4: return launch_pdl(L, k_visc_flux_25d<R, 4>, g, b, 0, L.P, W, fv, ctrl, detail::zb_for<R>(L));
        case 6: return launch_pdl(L, k_visc_flux_25d<R, 6>, g, b, 0, L.P, W, fv, ctrl, detail::zb_for<R>(L));
        default: return launch_pdl(L, k_visc_flux_25d<R, 8>, g, b, 0, L.P, W, fv, ctrl, detail::zb_for<R>(L));
        }
    }
    const int th = detail::threads_for(L.P.nx);
    const dim3 g = detail::cell_grid(L.P, th);
    switch (L.P.vis_order) {
    case 4: return launch_pdl(L, k_visc_flux<R, 4>, g, th, 0, L.P, W, fv, ctrl);
    case 6: return launch_pdl(L, k_visc_flux<R, 6>, g, th, 0, L.P, W, fv, ctrl);
    default: return launch_pdl(L, k_visc_flux<R, 8>, g, th, 0, L.P, W, fv, ctrl);
    }
}

template <class R, int ORD>
static cudaError_t update_ord(const LaunchCfg& L, int stage, StateView Wc, StateView W0,
                              const R* tacc, const R* fv, StateOut Wn, Ctrl* ctrl) {
    const int th = detail::threads_for(L.P.nx);
    const dim3 g = detail::cell_grid(L.P, th);
    if (stage == 1) return launch_pdl(L, k_update<R, ORD, 1>, g, th, 0, L.P, Wc, W0, tacc, fv, Wn, ctrl);
    if (stage == 2) return launch_pdl(L, k_update<R, ORD, 2>, g, th, 0, L.P, Wc, W0, tacc, fv, Wn, ctrl);
    return launch_pdl(L, k_update<R, ORD, 3>, g, th, 0, L.P, Wc, W0, tacc, fv, Wn, ctrl);
}

template <class R>
cudaError_t launch_update(const LaunchCfg& L, int stage, StateView Wc, StateView W0,
                          const R* tacc, const R* fv, StateOut Wn, Ctrl* ctrl) {
    switch (L.P.vis_order) {
    case 4: return update_ord<R, 4>(L, stage, Wc, W0, tacc, fv, Wn, ctrl);
    case 6: return update_ord<R, 6>(L, stage, Wc, W0, tacc, fv, Wn, ctrl);
    default: return update_ord<R, 8>(L, stage, Wc, W0, tacc, fv, Wn, ctrl);
    }
}

template <class R>
cudaError_t launch_rhs_out(const LaunchCfg& L, const R* tacc, const R* fv, double* rhs) {
    const int th = detail::threads_for(L.P.nx);
    const dim3 g = detail::cell_grid(L.P, th);
    switch (L.P.vis_order) {
    case 4: k_rhs_out<R, 4><<<g, th, 0, L.stream>>>(L.P, tacc, fv, rhs); break;
    case 6: k_rhs_out<R, 6><<<g, th, 0, L.stream>>>(L.P, tacc, fv, rhs); break;
    default: k_rhs_out<R, 8><<<g, th, 0, L.stream>>>(L.P, tacc, fv, rhs); break;
    }
    return cudaGetLastError();
}

#ifdef NS3D_LAUNCH_SMALL
namespace detail {
template <int FVS, int RC, bool CHR>
cudaError_t flux_small(const LaunchCfg& L, StateView W, double* tacc, double* fv, const Ctrl* ctrl) {
    // 64 to 256 cells a block: the three sweeps together give two blocks per SM or
    // more from 6300 cells on (below, blocks of 64 cells are fewer)
    const long long target = std::min(256ll, std::max(64ll, 3 * L.P.n / (2 * 148)));
    const SmallShape sh = small_shape(L.P, target, small_most(CHR), SMALL_T);
    const int nc = small_cells(L.P, sh);
    const unsigned blocks = small_blocks(sh);
    return launch_pdl(L, k_flux_small<FVS, RC, CHR>, blocks, SMALL_T, small_smem(nc, CHR), L.P, W, tacc, fv, sh, ctrl);
}
}  // namespace detail

cudaError_t launch_flux_small(const LaunchCfg& L, StateView W, double* tacc, double* fv, const Ctrl* ctrl) {
    auto by_rc = [&](auto fvs, auto chr) -> cudaError_t {
        constexpr int FVS = decltype(fvs)::value;
        constexpr bool CHR = decltype(chr)::value;
        switch (L.rc) {
        case RC_WENO5: return detail::flux_small<FVS, RC_WENO5, CHR>(L, W, tacc, fv, ctrl);
        case RC_LINEAR: return detail::flux_small<FVS, RC_LINEAR, CHR>(L, W, tacc, fv, ctrl);
        case RC_LIN6: return detail::flux_small<FVS, RC_LIN6, CHR>(L, W, tacc, fv, ctrl);
        case RC_MDCD_HYBRID: return detail::flux_small<FVS, RC_MDCD_HYBRID, CHR>(L, W, tacc, fv, ctrl);
        case RC_LIN8: return detail::flux_small<FVS, RC_LIN8, CHR>(L, W, tacc, fv, ctrl);
        default: return cudaErrorInvalidValue;
        }
    };
    auto by_fvs = [&](auto chr) {
        return L.fvs == FV_SW ? by_rc(std::integral_constant<int, FV_SW>{}, chr)
                              : by_rc(std::integral_constant<int, FV_LF>{}, chr);
    };
    return L.chr ? by_fvs(std::true_type{}) : by_fvs(std::false_type{});
}

template <int ORD>
static cudaError_t update_small_ord(const LaunchCfg& L, int stage, StateView Wc, StateView W0, const double* tacc,
                                    const double* fv, StateOut Wn, Ctrl* ctrl, double* rhs) {
    const unsigned blocks = (unsigned)((L.P.n + 31) / 32);
    if (stage > 0 && L.P.n > kSmallUpdateCells) {
        const int th = detail::threads_for(L.P.nx);
        const dim3 g = detail::cell_grid(L.P, th);
        auto wide = [&](auto st) {
            return launch_pdl(L, k_update<double, ORD, decltype(st)::value, true>, g, th, 0, L.P, Wc, W0, tacc, fv, Wn,
                              ctrl);
        };
        if (stage == 1) return wide(std::integral_constant<int, 1>{});
        if (stage == 2) return wide(std::integral_constant<int, 2>{});
        return wide(std::integral_constant<int, 3>{});
    }
    auto go = [&](auto st) {
        return launch_pdl(L, k_update_small<ORD, decltype(st)::value>, blocks, 160, 0, L.P, Wc, W0, tacc, fv, Wn,
                          ctrl, rhs);
    };
    if (stage == 0) return go(std::integral_constant<int, 0>{});
    if (stage == 1) return go(std::integral_constant<int, 1>{});
    if (stage == 2) return go(std::integral_constant<int, 2>{});
    return go(std::integral_constant<int, 3>{});
}

cudaError_t launch_update_small(const LaunchCfg& L, int stage, StateView Wc, StateView W0, const double* tacc,
                                const double* fv, StateOut Wn, Ctrl* ctrl, double* rhs) {
    switch (L.P.vis_order) {
    case 4: return update_small_ord<4>(L, stage, Wc, W0, tacc, fv, Wn, ctrl, rhs);
    case 6: return update_small_ord<6>(L, stage, Wc, W0, tacc, fv, Wn, ctrl, rhs);
    default: return update_small_ord<8>(L, stage, Wc, W0, tacc, fv, Wn, ctrl, rhs);
    }
}
#endif  // NS3D_LAUNCH_SMALL

#define NS3D_INSTANTIATE_LAUNCHERS(R)                                                          \
    template cudaError_t launch_sweep<R>(const LaunchCfg&, int, StateView, R*, const Ctrl*);   \
    template cudaError_t launch_visc_flux<R>(const LaunchCfg&, StateView, R*, const Ctrl*);    \
    template cudaError_t launch_update<R>(const LaunchCfg&, int, StateView, StateView,         \
                                          const R*, const R*, StateOut, Ctrl*);                \
    template cudaError_t launch_rhs_out<R>(const LaunchCfg&, const R*, const R*, double*);   \
    template cudaError_t launch_sweep_z_update<R>(const LaunchCfg&, int, StateView, StateView, \
                                                  const R*, const R*, StateOut, Ctrl*);

#endif  // NS3D_LAUNCH_IMPL

}  // namespace ns3d
