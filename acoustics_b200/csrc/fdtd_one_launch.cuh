// fdtd_one_launch.cuh — a whole time step of a static scene in one launch.
//
// On a small grid no kernel of the region-split step fills the GPU, and the step
// is the sum of their latencies: at 64^3 (FP64) the shell's 68 CTAs march eight
// planes one after the other (12 us), the ghost list walks a chain of dependent
// loads (9 us), the sources wait for both interior and ghost list (4 us), and each
// link of the chain costs a launch.  Here one grid holds the step's CTAs side by
// side: ghost cells, PML cells (one per thread, no march), interior tiles (which
// add the sources to their own cells) and the listener rows of the step before.
// Consecutive steps are chained by programmatic dependent launches, so a step's
// CTAs are resident and decoded when the step before ends.
//   64^3 FP64 (one sphere, one source, 8 listeners)   16.5 -> 9.4 us a step
//   61x97x83 FP32 (three bodies)                       21.3 -> 6.7 us
// Without bodies and sources a 48^3 step takes 3.0 us (FP32); what is left is the
// latency of one CTA (tables, then state, then stores) times the waves of CTAs.
// 80 (FP64) and 64 (FP32) registers are the best of 2 to 4 (5) CTAs per SM.
// Where the line to the region-split step lies: one_launch_cells().
//
// The arithmetic of every cell is the region-split kernels', expression by
// expression, so the two give the same bits.
#pragma once
#include "fdtd_hot.cuh"
#include "fdtd_listeners.cuh"

// resident CTAs of 256 threads the kernel is compiled for
#ifndef FDTD_ONE_MINB_F32
#define FDTD_ONE_MINB_F32 4
#endif
#ifndef FDTD_ONE_MINB_F64
#define FDTD_ONE_MINB_F64 3
#endif

namespace fdtd {

// CTAs of one step: blocks [0, ghost) take the ghost cells, then shell[b] ..
// shell[b + 1] the cells of shell box b, then the interior's tiles, then the
// listeners.
struct OneLaunch {
    Box3 interior;
    ShellBoxes shell;
    int shell_first[SHELL_MAX_BOXES + 1];
    int ghost_blocks, int_first, int_tu, lis_first;
    SourceArgs src;
    const GhostPlan* plan;
    const int* ghost_count;
    int plan_cap;
    double h75, rho;
    const double* fc_x;
    int n_lis;
    const LisPlan* lis_plan;
    const LisRow* lis_rows;
    double* lis_row;  // row of the step before (null: none)
};

// split-pressure array of axis d where the cell keeps it
template <typename T>
__device__ __forceinline__ T* sh_pd_any(const KArgs<T>& A, bool cmp, int d) {
    return cmp ? A.zpd[d] : A.pd[d];
}

// Cell idx of shell box b: its face velocities and split pressures, as
// shell_tile_impl (full state) and shell_tile_red_impl (RED) update them.
template <typename T, bool RED>
__device__ __forceinline__ void shell_cell(const KArgs<T>& A, const ShellBoxes& B, int b, int idx) {
    const int na = B.zae[b] - B.za[b], nz = na + B.zbe[b] - B.zb[b];
    const int row = idx / nz, kz = idx - row * nz;
    const int xl = row / B.ny[b], yl = row - xl * B.ny[b];
    if (xl >= B.nx[b]) return;
    const bool first = kz < na;
    const int x = B.x0[b] + xl, y = B.y0[b] + yl, z = first ? B.za[b] + kz : B.zb[b] + kz - na;
    const int sx = (int)A.sx, sy = (int)A.sy;
    const unsigned c = (unsigned)x * A.sx + (unsigned)y * A.sy + z;
    const bool cmp = b == B.zbox;
    // compact storage of the z-slab pair (ShellBoxes): the cell's slot, and its high z face's
    unsigned q = c, qzh = c + 1;
    int qsx = sx, qsy = sy;
    if (cmp) {
        const int V = B.vz;
        const int g = first ? z / V - B.za[b] / V : B.gl[b] + z / V - B.zb[b] / V;
        const bool last_group = first ? g == B.gl[b] - 1 : g == B.ng[b] - 1;
        qsy = B.zrw;
        qsx = B.ny[b] * B.zrw;
        const unsigned r0 = (unsigned)xl * qsx + (unsigned)yl * qsy;
        q = r0 + g * V + z % V;
        qzh = (z % V == V - 1 && last_group) ? r0 + B.ng[b] * V + (first ? 0 : 1) : q + 1;
    }
    const bool x_end = xl + 1 == B.nx[b], y_end = yl + 1 == B.ny[b];

    const T* __restrict__ pc = A.pc;
    // tables: no results of the step before
    const uint8_t gx = __ldg(A.axflag[0] + x), gy = __ldg(A.axflag[1] + y), gz = __ldg(A.axflag[2] + z);
    const bool slab_x = !cmp && (__ldg(A.axflag[0] + B.x0[b]) & AXF_PML);
    const AxisCoef<T> cxl = A.coef[0][x], cxr = A.coef[0][x + 1];
    const AxisCoef<T> cyl = A.coef[1][y], cyr = A.coef[1][y + 1];
    const AxisCoef<T> czl = A.coef[2][z], czr = A.coef[2][z + 1];
    step_before_done();
    const T pz = pc[c];
    const T pxm = pc[x > 0 ? c - sx : c], pxp = pc[x + 1 < A.N0 ? c + sx : c];
    const T pym = pc[y > 0 ? c - sy : c], pyp = pc[y + 1 < A.N1 ? c + sy : c];
    const T pzm = pc[z > 0 ? c - 1 : c], pzp = pc[c + 1];
    const bool mx = gx & AXF_PML, my = gy & AXF_PML, mz = gz & AXF_PML;

    if constexpr (!RED) {
        const T* xlo = cmp ? A.zvo[0] + q : A.vo[0] + c;
        const T* xhi = cmp && !x_end ? A.zvo[0] + q + qsx : A.vo[0] + c + sx;
        const T* ylo = cmp ? A.zvo[1] + q : A.vo[1] + c;
        const T* yhi = cmp && !y_end ? A.zvo[1] + q + qsy : A.vo[1] + c + sy;
        const T* zlo = cmp ? A.zvo[2] + q : A.vo[2] + c;
        const T* zhi = cmp ? A.zvo[2] + qzh : A.vo[2] + c + 1;
        T* const pd0 = sh_pd_any(A, cmp, 0) + q;
        T* const pd1 = sh_pd_any(A, cmp, 1) + q;
        T* const pd2 = sh_pd_any(A, cmp, 2) + q;
        const T vx0 = *xlo, vx1 = *xhi, vy0 = *ylo, vy1 = *yhi, vz0 = *zlo, vz1 = *zhi;
        const T a0 = *pd0, a1 = *pd1, a2 = *pd2;
        // faces inside the PML, outer faces excluded; a high face is written by
        // this cell only when the cell beyond it is not a PML cell
        const bool fxl = (gx & AXF_FACE_LO) || ((gx & AXF_HAS_LO) && (my || mz));
        const bool fxr = (gx & AXF_FACE_HI) || ((gx & AXF_HAS_HI) && (my || mz));
        const bool fyl = (gy & AXF_FACE_LO) || ((gy & AXF_HAS_LO) && (mx || mz));
        const bool fyr = (gy & AXF_FACE_HI) || ((gy & AXF_HAS_HI) && (mx || mz));
        const bool fzl = (gz & AXF_FACE_LO) || ((gz & AXF_HAS_LO) && (mx || my));
        const bool fzr = (gz & AXF_FACE_HI) || ((gz & AXF_HAS_HI) && (mx || my));
        const T vx_l = fxl ? vel_update<T>(vx0, cxl.vupd, cxl.vgrad, pz, pxm) : vx0;
        const T vx_r = fxr ? vel_update<T>(vx1, cxr.vupd, cxr.vgrad, pxp, pz) : vx1;
        const T vy_l = fyl ? vel_update<T>(vy0, cyl.vupd, cyl.vgrad, pz, pym) : vy0;
        const T vy_r = fyr ? vel_update<T>(vy1, cyr.vupd, cyr.vgrad, pyp, pz) : vy1;
        const T vz_l = fzl ? vel_update<T>(vz0, czl.vupd, czl.vgrad, pz, pzm) : vz0;
        const T vz_r = fzr ? vel_update<T>(vz1, czr.vupd, czr.vgrad, pzp, pz) : vz1;
        const T ax = pd_update<T>(a0, cxl.pupd, cxl.pdiv, vx_r, vx_l, A.inv_h);
        const T ay = pd_update<T>(a1, cyl.pupd, cyl.pdiv, vy_r, vy_l, A.inv_h);
        const T az = pd_update<T>(a2, czl.pupd, czl.pdiv, vz_r, vz_l, A.inv_h);
        *pd0 = ax;
        *pd1 = ay;
        *pd2 = az;
        A.pn[c] = ax + ay + az;
        if (fxl) {
            (cmp ? A.zvn[0] + q : A.vn[0] + c)[0] = vx_l;
            if (cmp && xl == 0) A.vn[0][c] = vx_l;
        }
        if (fyl) {
            (cmp ? A.zvn[1] + q : A.vn[1] + c)[0] = vy_l;
            if (cmp && yl == 0) A.vn[1][c] = vy_l;
        }
        if (fzl) (cmp ? A.zvn[2] + q : A.vn[2] + c)[0] = vz_l;
        if (fxr && !((gx & AXF_NEXT_PML) || my || mz))
            (cmp && !x_end ? A.zvn[0] + q + qsx : A.vn[0] + c + sx)[0] = vx_r;
        if (fyr && !((gy & AXF_NEXT_PML) || mx || mz))
            (cmp && !y_end ? A.zvn[1] + q + qsy : A.vn[1] + c + sy)[0] = vy_r;
        if (fzr && !((gz & AXF_NEXT_PML) || mx || my)) (cmp ? A.zvn[2] + qzh : A.vn[2] + c + 1)[0] = vz_r;
    } else {
        // ex, ey, ez: the axes the cell absorbs along (fdtd_shell_red.cuh)
        const bool ex = slab_x, ey = !cmp && (!ex || my), ez = mz;
        T* const p0 = sh_pd_any(A, cmp, 0) + q;
        T* const p1 = A.pd[1] + c;
        T* const p2 = sh_pd_any(A, cmp, 2) + q;
        const bool use2 = (ex && ey) || ez;
        const T* const vz = cmp ? A.zvo[2] : A.vo[2];
        const T a0 = *p0, a1 = cmp ? (T)0 : *p1, a2 = use2 ? *p2 : (T)0;
        const T vx0 = ex ? A.vo[0][c] : (T)0, vx1 = ex ? A.vo[0][c + sx] : (T)0;
        const T vy0 = ey ? A.vo[1][c] : (T)0, vy1 = ey ? A.vo[1][c + sy] : (T)0;
        const T vz0 = ez ? vz[q] : (T)0, vz1 = ez ? vz[qzh] : (T)0;
        T lap = 0.0f, sn = 0.0f, so = 0.0f, o0 = 0.0f, o1 = 0.0f, az = 0.0f;
        if (ex) {
            const bool fl = (gx & AXF_FACE_LO) || ((gx & AXF_HAS_LO) && (my || mz));
            const bool fr = (gx & AXF_FACE_HI) || ((gx & AXF_HAS_HI) && (my || mz));
            const T vl = fl ? vel_update<T>(vx0, cxl.vupd, cxl.vgrad, pz, pxm) : vx0;
            const T vr = fr ? vel_update<T>(vx1, cxr.vupd, cxr.vgrad, pxp, pz) : vx1;
            const T a = pd_update<T>(a0, cxl.pupd, cxl.pdiv, vr, vl, A.inv_h);
            if (fl) A.vn[0][c] = vl;
            if (fr && !(gx & AXF_NEXT_PML)) A.vn[0][c + sx] = vr;
            o0 = a;
            sn = a;
            so = a0;
        } else {
            lap = lap + (pxp + pxm - 2.0f * pz);
        }
        if (ey) {
            const bool fl = (gy & AXF_FACE_LO) || ((gy & AXF_HAS_LO) && (ex || mz));
            const bool fr = (gy & AXF_FACE_HI) || ((gy & AXF_HAS_HI) && (ex || mz));
            const T vl = fl ? vel_update<T>(vy0, cyl.vupd, cyl.vgrad, pz, pym) : vy0;
            const T vr = fr ? vel_update<T>(vy1, cyr.vupd, cyr.vgrad, pyp, pz) : vy1;
            const T a = pd_update<T>(a1, cyl.pupd, cyl.pdiv, vr, vl, A.inv_h);
            if (fl) A.vn[1][c] = vl;
            if (fr && !(gy & AXF_NEXT_PML)) A.vn[1][c + sy] = vr;
            o1 = a;
            sn = sn + a;
            so = so + a1;
        } else {
            lap = lap + (pyp + pym - 2.0f * pz);
        }
        if (ez) {
            T* const vn = cmp ? A.zvn[2] : A.vn[2];
            const bool fl = (gz & AXF_FACE_LO) || ((gz & AXF_HAS_LO) && (ex || my));
            const bool fr = (gz & AXF_FACE_HI) || ((gz & AXF_HAS_HI) && (ex || my));
            const T vl = fl ? vel_update<T>(vz0, czl.vupd, czl.vgrad, pz, pzm) : vz0;
            const T vr = fr ? vel_update<T>(vz1, czr.vupd, czr.vgrad, pzp, pz) : vz1;
            az = pd_update<T>(a2, czl.pupd, czl.pdiv, vr, vl, A.inv_h);
            if (fl) vn[q] = vl;
            if (fr && !(gz & AXF_NEXT_PML)) vn[qzh] = vr;
            sn = sn + az;
            so = so + a2;
        } else {
            lap = lap + (pzp + pzm - 2.0f * pz);
        }
        // the increment of the plain axes (none for a corner cell)
        const T qold = ex ? (ey ? a2 : a1) : a0;
        const T qn = fmaf(lap * A.lap_scale, A.c2k2, qold);
        A.pn[c] = (sn + (pz - so)) + (ex && ey && ez ? 0.0f : qn);
        *p0 = ex ? o0 : qn;
        if (!cmp) *p1 = ey ? o1 : qn;
        if (use2) *p2 = ez ? az : qn;
    }
}

// A listener whose plan does not do (a NaN that the full fit leaves out), out of
// line: it is rare and takes more registers than the rest.
template <typename T>
__device__ __noinline__ void one_listener_unplanned(const SolveParams* P, int newp, int li, double* row) {
    listener_plan<T>(*P, newp, li, row);
    flag_nonfinite(*P, row, li);
}

// The ghost-neighbour list from its plans (every cell has one: plan_cap is the
// list's capacity where steps are one launch), the sources added too.
template <typename T, bool VISC>
__device__ __forceinline__ void one_ghost_cells(const KArgs<T>& A, const OneLaunch& L, int first) {
    const GhostArgs<T> G{A.pc, A.pn, A.dinc, VISC ? A.lapl : nullptr, A.lapc, A.sx, A.sy, A.c2k2, A.lap_scale, A.kcalp,
                         L.h75, L.rho, L.src.consts, L.fc_x};
    // the list is no result of the step before; its first plans are read beside the count
    const int stride = L.ghost_blocks * 256, q = threadIdx.x & 3;
    GhostLoad p{};
    if (first >> 2 < L.plan_cap) p = ghost_load(L.plan, first >> 2, q);
    const int planned = min(*L.ghost_count, L.plan_cap);
    step_before_done();
    for (int w = first & ~31; w < 4 * planned; w += stride) {  // whole warps, eight cells each
        const int g = (w + (int)threadIdx.x) >> 2;
        if (w != (first & ~31) || g >= planned) p = ghost_load(L.plan, min(g, planned - 1), q);
        ghost_cell_planned<T>(G, p, g < planned, &L.src);
    }
}

template <typename T, bool RED, bool VISC>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? FDTD_ONE_MINB_F32 : FDTD_ONE_MINB_F64) k_step_one(const __grid_constant__ KArgs<T> A,
                                                     const __grid_constant__ OneLaunch L) {
    const int blk = (int)blockIdx.x;
    const int tid = threadIdx.x + 32 * threadIdx.y;
    // the next step's CTAs may be placed as soon as all of this step's are; each
    // reads its tables, flags and plans before it waits for the step before
    asm volatile("griddepcontrol.launch_dependents;");
    if (blk < L.ghost_blocks) {
        one_ghost_cells<T, VISC>(A, L, blk * 256 + tid);
        if (blk == 0 && tid >= 224) advance_consts(*A.P, A.cur, tid - 224);
    } else if (blk < L.int_first) {
        int b = 0;
#pragma unroll
        for (int q = 1; q < SHELL_MAX_BOXES; ++q)
            if (q < L.shell.n && blk >= L.shell_first[q]) b = q;
        shell_cell<T, RED>(A, L.shell, b, (blk - L.shell_first[b]) * 256 + tid);
    } else if (blk < L.lis_first) {
        const int t = blk - L.int_first;
        interior_tile<T, 2, VISC, KArgs<T>, true>(A, L.interior, t % L.int_tu, t / L.int_tu, &L.src);
    } else {
        // row of the step before, from p^n (no stencil holds a ghost cell here)
        const int li = (blk - L.lis_first) * 8 + (int)threadIdx.y;
        if (li >= L.n_lis) return;  // whole warps
        const int lane = threadIdx.x;
        const LisPlan& pl = L.lis_plan[li];
        const int nc = pl.nc, n = pl.n, mode = pl.mode;
        const int cell = mode == 1 ? pl.cell : lane < nc ? pl.cells[lane & 7] : -1;
        const LisRow* rows = L.lis_rows + (size_t)li * 64;
        LisRow r0{}, r1{};
        if (mode == 0 && lane < n) r0 = rows[lane];
        if (mode == 0 && lane + 32 < n) r1 = rows[lane + 32];
        step_before_done();
        const double v = cell >= 0 ? (double)A.pc[cell] : 0.0;
        double acc = 0.0;
        if (mode == 0 && lane < n) acc += r0.w * (double)A.pc[r0.cell];
        if (mode == 0 && lane + 32 < n) acc += r1.w * (double)A.pc[r1.cell];
        const bool odd = mode == 2 || __any_sync(0xffffffffu, mode != 1 && cell >= 0 && isnan(v));
        if (odd) {
            one_listener_unplanned<T>(A.P, A.cur, li, L.lis_row);
            return;
        }
        acc = mode == 1 ? v : warp_sum(acc);
        if (lane == 0) {
            L.lis_row[li] = acc;
            if (!isfinite(acc)) atomicOr(A.P->dev_error, 1);
        }
    }
}

// Grid cells up to which a static solve steps by one launch: where the region-split
// step with 16-step graphs takes as long (us a step, one launch / split; a sphere
// and a box, one active source, 8 listeners, PML 8-10):
//   FP32  64^3 5.8 / 13.8, 112^3 13.3 / 14.5, 144x120x112 17.9 / 17.0, 160^3 29.6 / 25.5
//   FP64  64^3 8.0 / 14.0, 96^3 14.2 / 14.8, 112^3 20.3 / 17.4, 160^3 70.8 / 51.4
// Past it a thread per PML cell moves more bytes than the marching shell, which
// carries p and the low x face along.
#ifndef FDTD_ONE_LAUNCH_CELLS_F32
#define FDTD_ONE_LAUNCH_CELLS_F32 1600000
#endif
#ifndef FDTD_ONE_LAUNCH_CELLS_F64
#define FDTD_ONE_LAUNCH_CELLS_F64 1000000
#endif

template <typename T>
cudaError_t launch_one(const SolveParams* dP, const SolveParams& hP, const RegionLaunch& R, int cur, int n_ghost,
                       double* lis_row, cudaStream_t s, int* launches) {
    if (R.fc) {
        const cudaError_t e = launch_fc<T>(dP, hP, cur, s, true, launches);
        if (e != cudaSuccess) return e;
    }
    if (launches) *launches += 1;
    KArgs<T> A = make_kargs<T>(const_cast<SolveParams*>(dP), hP, cur);
    OneLaunch L{};
    L.interior = R.interior;
    L.shell = R.shell;
    const int cap = hP.ghost_cap;
    const int cells = n_ghost >= 0 ? std::min(n_ghost, cap) : cap;
    L.ghost_blocks = std::max(1, std::min((cells + 63) / 64, 148));  // four lanes a cell
    int blocks = L.ghost_blocks;
    for (int b = 0; b < R.shell.n; ++b) {
        const ShellBoxes& B = R.shell;
        L.shell_first[b] = blocks;
        const long long c = (long long)B.nx[b] * B.ny[b] * (B.zae[b] - B.za[b] + B.zbe[b] - B.zb[b]);
        blocks += (int)((c + 255) / 256);
    }
    L.int_first = blocks;
    const Box3& I = R.interior;
    const int nx = I.hi[0] - I.lo[0];
    L.int_tu = interior_unit_tiles(I, 16 / (int)sizeof(T));
    if (nx > 0 && L.int_tu > 0) blocks += L.int_tu * ((nx + 1) / 2);
    L.lis_first = blocks;
    if (lis_row && hP.n_lis > 0) blocks += (hP.n_lis + 7) / 8;
    L.src = source_args(hP, R, cur);
    L.plan = hP.ghost_plan;
    L.ghost_count = hP.ghost_count;
    L.plan_cap = hP.plan_ready ? hP.plan_cap : 0;
    L.h75 = 0.75 * hP.h;
    L.rho = hP.rho;
    L.fc_x = R.fc ? hP.fc_x + (size_t)cur * hP.fc_n : nullptr;
    L.n_lis = hP.n_lis;
    L.lis_plan = hP.lis_plan;
    L.lis_rows = hP.lis_rows;
    L.lis_row = lis_row;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(32, 8);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if constexpr (sizeof(T) == 4) {
        if (R.red && hP.visc) return cudaLaunchKernelEx(&cfg, k_step_one<T, true, true>, A, L);
        if (R.red) return cudaLaunchKernelEx(&cfg, k_step_one<T, true, false>, A, L);
    }
    if (hP.visc) return cudaLaunchKernelEx(&cfg, k_step_one<T, false, true>, A, L);
    return cudaLaunchKernelEx(&cfg, k_step_one<T, false, false>, A, L);
}

}  // namespace fdtd
