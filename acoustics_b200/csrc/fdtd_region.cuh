// fdtd_region.cuh — the step split by region, one lean kernel per region:
//
//   k_interior   non-PML cells, box [lo, hi): ghost-aware Laplacian, leapfrog /
//                compensated increment, Gaussian sources
//                (MAC_Grid.cpp:187-299 + :921-944).  Only pressure words move:
//                p^n (neighbours from the CTA's rows), p^{n-1} or the increment,
//                p^{n+1}, plus one classification byte.
//   k_pml_shell  the PML shell's boxes (two x and two y slabs, the pair of z slabs
//                between them): face velocities (MAC_Grid.cpp:461-479) and
//                split-field pressures (:496-508).
//
// Face ownership: a PML face is written by the cell to its right; the one face
// layer whose right cell is not a PML cell (x = W h on the low side) is written
// by its left (PML) cell, so the interior kernel never touches velocities.
//
// Cells next to a solid (a compact list built by the classification) have a kernel
// of their own, so the interior kernel is a pure 7-point leapfrog.  Both add the
// Gaussian sources, while they are active, to the cells they own (k_sources does
// it after them where the interior takes an explicit chunk of x planes).
//
// Interior mapping: a CTA takes 256 consecutive units of the box, one per thread;
// a unit is a z group (16 bytes: 4 FP32 or 2 FP64 cells) of one (x, y) row, at XB
// consecutive x planes.  All loads of the XB planes (p^n at XB+2 planes, y
// neighbours, p^{n-1}/increment, classification) are issued before any arithmetic
// so that every thread keeps ~5*XB independent HBM requests in flight; z neighbours
// come from the lanes beside it with shuffles (interior_tile).
#pragma once
#include "fdtd_device.cuh"
#include "fdtd_coupled.cuh"
#include "fdtd_geometry.cuh"
#include "fdtd_stencil.cuh"

namespace fdtd {

// Ghost-aware Laplacian of one bulk cell with at least one solid neighbour
// (MAC_Grid.cpp:267-297); returns the unscaled sum and the number of axes with
// ghost cells on both sides.
template <typename T>
__device__ __noinline__ T ghost_laplacian(const SolveParams& P, long long c, const int idx[3], unsigned mask, T p0,
                                          const T nbp[3], const T nbm[3], double t, int par, int* surrounded) {
    const long long strides[3] = {P.SX, P.SY, 1};
    T lap = 0.0;
    int s = 0;
    for (int d = 0; d < 3; ++d) {
        const bool gn = (mask >> (2 * d)) & 1u;
        const bool gp = (mask >> (2 * d + 1)) & 1u;
        T gpv = 0, gnv = 0;
        if (gp || gn) {
            double own[3] = {P.cpos[0][idx[0]], P.cpos[1][idx[1]], P.cpos[2][idx[2]]};
            // FULLY_COUPLED: the solved ghost pressures of this step; RASTERIZE: pg
            if (gp) {
                own[d] = P.cpos[d][idx[d] + 1];
                gpv = P.fc_rows ? (T)fc_ghost(P, par, c + strides[d], 2 * d, (double)p0)
                                : (T)ghost_pressure(P, P.gobj[c + strides[d]], own, d, -1, (double)p0, t);
            }
            if (gn) {
                own[d] = P.cpos[d][idx[d] - 1];
                gnv = P.fc_rows ? (T)fc_ghost(P, par, c - strides[d], 2 * d + 1, (double)p0)
                                : (T)ghost_pressure(P, P.gobj[c - strides[d]], own, d, +1, (double)p0, t);
            }
        }
        if (gp && gn) {
            lap = lap + (gpv + gnv - (T)2.0 * p0) / (T)(9.0 / 16.0);
            ++s;
        } else if (gp) {
            lap = lap + (gpv + (T)0.75 * nbm[d] - (T)(7.0 / 4.0) * p0) / (T)(21.0 / 32.0);
        } else if (gn) {
            lap = lap + ((T)0.75 * nbp[d] + gnv - (T)(7.0 / 4.0) * p0) / (T)(21.0 / 32.0);
        } else {
            lap = lap + (nbp[d] + nbm[d] - (T)2.0 * p0);
        }
    }
    *surrounded = s;
    return lap;
}

// Full update of non-PML bulk cell c next to a solid (ghost-aware Laplacian,
// cavity freeze), everything re-read from memory.  Sources are added by
// k_sources afterwards, as the reference adds them after the update
// (MAC_Grid.cpp:938-944).
template <typename T>
__device__ __forceinline__ void ghost_cell(const SolveParams& P, int cur, long long c) {
    const long long sx = P.SX, sy = P.SY;
    const T* __restrict__ pc = (const T*)P.p[cur];
    T* __restrict__ pn = (T*)P.p[cur ^ 1];
    const double t = P.consts[cur].t;
    int x, y, z;
    cell_ijk(P, c, x, y, z);
    const uint8_t code = P.cls[c];
    const T p0 = pc[c];
    const T nbp[3] = {pc[c + sx], pc[c + sy], pc[c + 1]};
    const T nbm[3] = {pc[c - sx], pc[c - sy], pc[c - 1]};
    const int idx[3] = {x, y, z};
    int surrounded = 0;
    T lap = ghost_laplacian<T>(P, c, idx, code & CLS_MASK, p0, nbp, nbm, t, cur, &surrounded);
    lap = lap * (T)P.lap_scale;
    const bool cavity = (surrounded > 1) && (code & CLS_VALID);
    // air viscosity on cells with a valid history (MAC_Grid.cpp:926-930)
    const bool visc = P.visc && (code & CLS_VALID);
    T lapl = 0;
    if (P.visc) {
        lapl = ((const T*)P.lapv[cur ^ 1])[c];
        ((T*)P.lapv[cur])[c] = lap;
    }
    if constexpr (sizeof(T) == 8) {
        if (cavity) pn[c] = p0;
        else if (visc) pn[c] = (T)2.0 * p0 - pn[c] - lapl * (T)P.kcalp + lap * (T)(P.c2k2 + P.kcalp);
        else pn[c] = (T)2.0 * p0 - pn[c] + lap * (T)P.c2k2;
    } else {
        float d = cavity ? 0.0f : P.dinc[c] + (float)(lap * (T)P.c2k2);
        if (!cavity && visc) d = fmaf((float)P.kcalp, (float)(lap - lapl), d);
        P.dinc[c] = d;
        pn[c] = p0 + d;
    }
}

// Pointers and scalars of the planned update, by value or read from the
// solve's parameters once.
template <typename T>
struct GhostArgs {
    const T* pc;
    T* pn;
    float* dinc;
    const T* lapl;  // air viscosity, else null
    T* lapc;
    unsigned sx, sy;
    T c2k2, lap_scale, kcalp;
    double h75, rho;              // 0.75 h, rho
    const StepConsts* consts;     // of this step
    const double* fc_x;           // FULLY_COUPLED: this step's ghost pressures by row
};

template <typename T>
__device__ __forceinline__ GhostArgs<T> ghost_args(const SolveParams& P, int cur) {
    return GhostArgs<T>{(const T*)P.p[cur], (T*)P.p[cur ^ 1], P.dinc, P.visc ? (const T*)P.lapv[cur ^ 1] : nullptr,
                        (T*)P.lapv[cur], (unsigned)P.SX, (unsigned)P.SY, (T)P.c2k2, (T)P.lap_scale, (T)P.kcalp,
                        0.75 * P.h, P.rho, P.consts + cur, P.fc_rows ? P.fc_x + (size_t)cur * P.fc_n : nullptr};
}

// ghost_cell from the cells' plans, four lanes a cell: an axis of the Laplacian
// each (its two faces and its division) and, in the last, what the cell keeps of
// p^{n-1} and the sources.  One lane alone would take the axes' divisions in turn
// at the end of every small step.  The terms are summed in axis order, and every
// expression is ghost_cell's (boundary_accel, ghost_pressure, ghost_laplacian), so
// the bits are the same.
struct GhostLoad {
    uint4 h0, h1;  // words 0-7 of the plan
    double2 u;     // this lane's axis
};
__device__ __forceinline__ GhostLoad ghost_load(const GhostPlan* plan, int g, int q) {
    const uint4* w = reinterpret_cast<const uint4*>(plan + g);
    GhostLoad r;
    r.h0 = w[0];
    r.h1 = w[1];
    r.u = *reinterpret_cast<const double2*>(&w[2 + (q < 3 ? q : 0)]);
    return r;
}

__host__ __device__ __forceinline__ SourceArgs source_args(const SolveParams& P, const Box3& region, int n, int cur) {
    SourceArgs S{};
    S.region = region;
    S.n = n;
    for (int d = 0; d < 3; ++d) {
        S.N[d] = P.N[d];
        S.ax[d] = P.src_ax[d];
    }
    S.consts = P.consts + cur;
    S.k = P.k;
    return S;
}

// sum_s G_s(x, t + k/2) at cell (x, y, z), as source_term (the factors' loads do
// not wait for the time factor)
__device__ __forceinline__ double source_at(const SourceArgs& S, int x, int y, int z) {
    double src = 0.0;
    for (int s = 0; s < S.n; ++s) {
        const double f = (S.ax[0][s * S.N[0] + x] * S.ax[1][s * S.N[1] + y]) * S.ax[2][s * S.N[2] + z];
        const double tf = S.consts->src_tf[s];
        if (tf != 0.0) src += f * tf;
    }
    return src;
}

// Called by whole warps; lanes with on = false work on some plan and store nothing.
// S: the sources to add (null: k_sources does).
template <typename T>
__device__ __forceinline__ void ghost_cell_planned(const GhostArgs<T>& A, const GhostLoad& G, bool on,
                                                   const SourceArgs* S) {
    const int q = threadIdx.x & 3;
    const unsigned c = G.h0.x;
    const uint32_t code = G.h0.y;
    const T* __restrict__ pc = A.pc + c;
    const unsigned st = q == 0 ? A.sx : q == 1 ? A.sy : 1u;
    const T p0 = pc[0];
    // lanes 0-2: the neighbours along the axis; lane 3: p^{n-1} or the increment, the last Laplacian
    const T pp = q < 3 ? pc[st] : sizeof(T) == 8 ? A.pn[c] : (T)A.dinc[c];
    const T pm = q < 3 ? *(pc - st) : A.lapl ? A.lapl[c] : (T)0;
    const bool gn = q < 3 && ((code >> (2 * q)) & 1u), gp = q < 3 && ((code >> (2 * q + 1)) & 1u);
    // bodies of the axis' two faces: bytes 8-13 of the plan
    const uint32_t bodies = q == 0 ? G.h0.z : q == 1 ? G.h0.z >> 16 : G.h0.w;
    const unsigned on_n = bodies & 0xFFu, on_p = (bodies >> 8) & 0xFFu;
    // a face's body's acceleration, or its solved pressure
    auto face = [&](bool here, unsigned o, double u) {
        if (!here || o == GHOST_STILL) return 0.0;
        return o == GHOST_COUPLED ? A.fc_x[(int)u] : A.consts->obj_g[o];
    };
    const double gt_n = face(gn, on_n, G.u.x), gt_p = face(gp, on_p, G.u.y);
    double add = 0.0;
    bool add_src = false;
    if (S && S->n > 0 && q == 3) {
        const int x = (int)(G.h1.x & 0xFFFFu), y = (int)(G.h1.x >> 16), z = (int)(G.h1.y & 0xFFFFu);
        const Box3& r = S->region;
        add_src = x >= r.lo[0] && x < r.hi[0] && y >= r.lo[1] && y < r.hi[1] && z >= r.lo[2] && z < r.hi[2];
        if (add_src) add = source_at(*S, x, y, z) * S->k;
    }
    double vn = (double)p0, vp = (double)p0;
    if (gn && on_n != GHOST_STILL) vn = on_n == GHOST_COUPLED ? gt_n : vn - A.h75 * (G.u.x * gt_n * (-A.rho));
    // the face toward + has its normal toward this cell, along -
    if (gp && on_p != GHOST_STILL) vp = on_p == GHOST_COUPLED ? gt_p : vp - A.h75 * (G.u.y * gt_p * (-A.rho) * -1.0);
    const T pgn = (T)vn, pgp = (T)vp;
    T num, den;
    if (gp && gn) {
        num = pgp + pgn - (T)2.0 * p0;
        den = (T)(9.0 / 16.0);
    } else if (gp) {
        num = pgp + (T)0.75 * pm - (T)(7.0 / 4.0) * p0;
        den = (T)(21.0 / 32.0);
    } else if (gn) {
        num = (T)0.75 * pp + pgn - (T)(7.0 / 4.0) * p0;
        den = (T)(21.0 / 32.0);
    } else {
        num = pp + pm - (T)2.0 * p0;
        den = (T)1.0;
    }
    const T term = gp || gn ? num / den : num;
    const unsigned both = __ballot_sync(0xffffffffu, gp && gn);
    const int base = threadIdx.x & 28;
    T lap = 0.0;
    lap = lap + __shfl_sync(0xffffffffu, term, base);
    lap = lap + __shfl_sync(0xffffffffu, term, base + 1);
    lap = lap + __shfl_sync(0xffffffffu, term, base + 2);
    if (q != 3 || !on) return;
    const T prev = pp, lapl = pm;
    lap = lap * A.lap_scale;
    const bool valid = code & CLS_VALID;
    const bool cavity = __popc((both >> base) & 7u) > 1 && valid;
    const bool visc = A.lapl && valid;
    if (A.lapl) A.lapc[c] = lap;
    if constexpr (sizeof(T) == 8) {
        T v;
        if (cavity) v = p0;
        else if (visc) v = (T)2.0 * p0 - prev - lapl * A.kcalp + lap * (A.c2k2 + A.kcalp);
        else v = (T)2.0 * p0 - prev + lap * A.c2k2;
        if (add_src) v += add;
        A.pn[c] = v;
    } else {
        float d = cavity ? 0.0f : prev + (float)(lap * A.c2k2);
        if (!cavity && visc) d = fmaf((float)A.kcalp, (float)(lap - lapl), d);
        if (add_src) d = d + (float)add;
        A.dinc[c] = d;
        A.pn[c] = p0 + d;
    }
}

// The cells of the ghost-neighbour list, by plan where there is one.
template <typename T>
__device__ __forceinline__ void ghost_cells_body(const SolveParams& P, int cur, int bid, int nblocks, bool plans,
                                                 const SourceArgs* S = nullptr) {
    const int n = min(list_counts(P, cur)[0], P.ghost_cap);
    const int planned = plans ? min(n, P.plan_cap) : 0;
    const int first = bid * blockDim.x + threadIdx.x, stride = nblocks * blockDim.x;
    if (planned > 0) {
        const GhostArgs<T> A = ghost_args<T>(P, cur);
        // whole warps, eight cells each
        for (int w = first & ~31; w < 4 * planned; w += stride) {
            const int g = (w + (int)(threadIdx.x & 31)) >> 2;
            ghost_cell_planned<T>(A, ghost_load(P.ghost_plan, min(g, planned - 1), threadIdx.x & 3), g < planned,
                                  S);
        }
    }
    for (int g = planned + first; g < n; g += stride) {
        const long long c = P.ghost_list[g];
        ghost_cell<T>(P, cur, c);
        if (!S || S->n == 0) continue;
        // (outside the supports' bounding box a source's factors are zero)
        int x, y, z;
        cell_ijk(P, c, x, y, z);
        const double src = source_at(*S, x, y, z);
        T* __restrict__ pn = (T*)P.p[cur ^ 1];
        if constexpr (sizeof(T) == 8) {
            pn[c] += src * S->k;
        } else {
            const float d = P.dinc[c] + (float)(src * S->k);
            P.dinc[c] = d;
            pn[c] = ((const T*)P.p[cur])[c] + d;
        }
    }
}

// Face (d, s) of a plan: toward the solid cell idx + (s ? 1 : -1) e_d, whose
// closest object is o (GHOST_STILL: none, or a constraint).
__device__ __forceinline__ void plan_face(const SolveParams& P, GhostPlan& G, const int idx[3], int d, int s, unsigned o) {
    if (o >= (unsigned)P.n_obj || P.obj[o].accel_kind == 0) return;
    const int sgn = s ? 1 : -1;
    // the face a quarter cell from the solid cell's centre (ghost_pressure)
    double pos[3] = {P.cpos[0][idx[0]], P.cpos[1][idx[1]], P.cpos[2][idx[2]]};
    pos[d] = P.cpos[d][idx[d] + sgn];
    pos[d] += (sgn > 0 ? -1.0 : 1.0) * 0.25 * P.h;
    const DevObject& O = P.obj[o];
    if (O.accel_kind == 1) {
        G.u[d][s] = O.dir[d];
    } else {
        const double r0 = pos[0] - O.c[0], r1 = pos[1] - O.c[1], r2 = pos[2] - O.c[2];
        const double len = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
        const double r[3] = {r0, r1, r2};
        G.u[d][s] = len > 0.0 ? r[d] / len : 0.0;
    }
    G.obj[2 * d + s] = (uint8_t)o;
}
__device__ __forceinline__ GhostPlan empty_plan(int c, uint8_t code, const int idx[3]) {
    GhostPlan G{};
    G.c = c;
    G.code = code;
    for (int f = 0; f < 6; ++f) G.obj[f] = GHOST_STILL;
    for (int d = 0; d < 3; ++d) G.ijk[d] = (uint16_t)idx[d];
    return G;
}

// Plans of the ghost-neighbour list of the current classification (static scenes).
static __global__ void __launch_bounds__(128) k_ghost_prep(const SolveParams* __restrict__ Pp) {
    const SolveParams& P = *Pp;
    const int n = min(min(*P.ghost_count, P.ghost_cap), P.plan_cap);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int c = P.ghost_list[q];
        int idx[3];
        cell_ijk(P, c, idx[0], idx[1], idx[2]);
        GhostPlan G = empty_plan(c, P.cls[c], idx);
        const long long strides[3] = {P.SX, P.SY, 1};
        for (int f = 0; f < 6; ++f) {
            if (!((G.code >> f) & 1u)) continue;
            const int d = f >> 1, s = f & 1;
            const long long nb = c + (s ? 1 : -1) * strides[d];
            if (P.fc_rows) {
                const int row = fc_row(P, nb, 2 * d + (s ? 0 : 1));
                if (row >= 0) {  // (else, which classification rules out, the cell's own pressure)
                    G.obj[f] = GHOST_COUPLED;
                    G.u[d][s] = (double)row;
                }
                continue;
            }
            const unsigned gobj = P.gobj[nb];
            if (!(gobj & GOBJ_CONSTRAINT)) plan_face(P, G, idx, d, s, gobj & 0x7F);
        }
        P.ghost_plan[q] = G;
    }
}

// pNext += k * sum_s G_s(x, t + k/2) over the bounding box of the source
// supports clipped to the non-PML box (GaussianPressureSource.cpp:6-30), with
// G_s = (product of the per-axis spatial factors) * (time factor of the step).
template <typename T>
__device__ __forceinline__ void sources_body(const SolveParams& P, int cur, const Box3& region, int bid, int nblocks) {
    const StepConsts& sc = P.consts[cur];
    bool any_src = false;
    for (int s = 0; s < P.n_src; ++s) any_src |= (sc.src_tf[s] != 0.0);
    if (!any_src) return;
    const int nx = region.hi[0] - region.lo[0], ny = region.hi[1] - region.lo[1], nz = region.hi[2] - region.lo[2];
    const long long total = (long long)nx * ny * nz;
    const T* __restrict__ pc = (const T*)P.p[cur];
    T* __restrict__ pn = (T*)P.p[cur ^ 1];
    for (long long t = bid * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)nblocks * blockDim.x) {
        const int z = region.lo[2] + (int)(t % nz);
        const int y = region.lo[1] + (int)((t / nz) % ny);
        const int x = region.lo[0] + (int)(t / ((long long)nz * ny));
        const long long c = cidx(P, x, y, z);
        if (!(P.cls[c] & CLS_BULK)) continue;
        const double src = source_term(P, cur, x, y, z);
        if constexpr (sizeof(T) == 8) {
            pn[c] += src * P.k;
        } else {
            const float d = P.dinc[c] + (float)(src * P.k);
            P.dinc[c] = d;
            pn[c] = pc[c] + d;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(128) k_ghost_cells(const SolveParams* __restrict__ Pp, int cur,
                                                     bool plans, const __grid_constant__ SourceArgs S) {
    ghost_cells_body<T>(*Pp, cur, blockIdx.x, gridDim.x, plans, &S);
}

template <typename T>
__global__ void __launch_bounds__(256) k_sources(const SolveParams* __restrict__ Pp, int cur, Box3 region) {
    sources_body<T>(*Pp, cur, region, blockIdx.x, gridDim.x);
}

}  // namespace fdtd
