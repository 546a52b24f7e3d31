// fdtd_fetch.cu — read-back of cells and fields.
//
// Cells (PML_WaveSolver::FetchCell and SampleAxisAlignedSlice,
// PML_WaveSolver.cpp:439-458, MAC_Grid.cpp:1941-1963, MAC_Grid::GetCell
// :4182-4258): one thread per cell finds its words where the solve keeps them,
// evaluates the ghost-face pressures of the last step with the step's own device
// functions, and makes the whole fdtd_cell, in mapped host memory.  The host made nine addresses per
// cell, a request array and the geometry of every record before: a 192 x 160
// slice took 4.9 ms, now 1.9.
//
// Fields: one thread per element of the dense order, as doubles, straight into
// mapped host memory (consecutive threads write consecutive words, so the bus
// sees whole lines).  The host copied the padded arrays and walked them element
// by element: 192 x 160 x 144 FP32 8.2 ms, now 2.5.
// Compiled with -fmad=false like the step kernels, so the ghost-face pressures
// are the ones the step used, bit for bit.
#include <cfloat>
#include <cmath>

#include "fdtd_coupled.cuh"
#include "fdtd_geometry.cuh"
#include "fdtd_launch.hpp"

namespace fdtd {

// Index into the compact z-slab arrays of the PML state (ShellBoxes::zbox) of
// the split pressure of cell (x, y, z) (dface < 0) or of its low face along
// dface; -1 when that element lies in the padded arrays (zslab_index, fdtd_step.cpp).
__device__ __forceinline__ long long zslab_slot(const ShellBoxes& B, int N2, int dface, int x, int y, int z) {
    const int b = B.zbox, V = B.vz;
    if (b < 0) return -1;
    if (x < B.x0[b] || x >= B.x0[b] + B.nx[b] || y < B.y0[b] || y >= B.y0[b] + B.ny[b]) return -1;
    if (dface != 2 && z >= N2) return -1;
    auto slot = [&](int zz) -> int {
        if (zz >= B.za[b] && zz < B.zae[b]) return (zz / V - B.za[b] / V) * V + zz % V;
        if (zz >= B.zb[b] && zz < B.zbe[b]) return (B.gl[b] + zz / V - B.zb[b] / V) * V + zz % V;
        return -1;
    };
    int q = slot(z);
    if (dface == 2 && q < 0 && z == B.zae[b] && z > 0)  // the face after the first range
        q = ((z - 1) % V != V - 1) ? slot(z - 1) + 1 : B.ng[b] * V;
    if (q < 0) return -1;
    return ((long long)(x - B.x0[b]) * B.ny[b] + (y - B.y0[b])) * B.zrw + q;
}

constexpr int FETCH_THREADS = 128;

// cur: the parity of the next step (the solver's current one); the last step
// ran with cur ^ 1, read p^n and wrote p^{n+1} into p[cur].
template <typename T>
__global__ void __launch_bounds__(FETCH_THREADS) k_fetch_cells(const SolveParams* __restrict__ Pp, int cur,
                                                     const __grid_constant__ FetchArgs F, long long first, int n,
                                                     fdtd_cell* __restrict__ out) {
    // the CTA's records, written out together as consecutive words
    static_assert(sizeof(fdtd_cell) % 8 == 0, "copied as 8-byte words");
    __shared__ fdtd_cell made[FETCH_THREADS];
    const SolveParams& P = *Pp;
    const int q0 = blockIdx.x * FETCH_THREADS;
    const int here = min(FETCH_THREADS, n - q0);
    // (threads past the end make the last cell again)
    const int q = q0 + min((int)threadIdx.x, here - 1);
    int idx[3];
    if (F.dim < 0) {
        dense_ijk(P, F.cell, idx[0], idx[1], idx[2]);
    } else {
        const long long t = first + q;
        const int d1 = (F.dim + 1) % 3, d2 = (F.dim + 2) % 3;
        idx[F.dim] = F.k;
        idx[d1] = (int)(t / P.N[d2]);
        idx[d2] = (int)(t % P.N[d2]);
    }
    const int i = idx[0], j = idx[1], k = idx[2];
    const long long c = cidx(P, i, j, k);
    const T* __restrict__ pc = (const T*)P.p[cur];
    // p^n of the last step: the other buffer (FP64) or p^{n+1} less the compensated increment (FP32)
    auto prev = [&](long long x) -> double {
        if constexpr (sizeof(T) == 8) return ((const double*)P.p[cur ^ 1])[x];
        else return (double)pc[x] - (double)P.dinc[x];
    };
    // an element of the PML state; NaN where the solve does not hold it
    auto element = [&](const void* base, const void* zbase, int dface, int x, int y, int z) -> double {
        if (F.reduced || !base) return NAN;
        const long long s = P.zcount > 0 ? zslab_slot(F.shell, P.N[2], dface, x, y, z) : -1;
        return s >= 0 ? (double)((const T*)zbase)[s] : (double)((const T*)base)[cidx(P, x, y, z)];
    };
    const uint8_t code = P.cls[c], gobj = P.gobj[c];
    const bool bulk = code & CLS_BULK;
    const bool pml = P.pml_cell[0][i] || P.pml_cell[1][j] || P.pml_cell[2][k];
    int flags = 0;  // cell_flags (fdtd_step.cpp)
    if (bulk) flags |= FDTD_CELL_BULK;
    if (!bulk && (code & CLS_MASK)) flags |= FDTD_CELL_GHOST;
    if (code & CLS_VALID) flags |= FDTD_CELL_VALID_HISTORY;
    if (pml) flags |= FDTD_CELL_PML;
    if (!bulk && (gobj & GOBJ_CONSTRAINT)) flags |= FDTD_CELL_CONSTRAINT;

    fdtd_cell C;
    C.index = (int32_t)(((long long)i * P.N[1] + j) * P.N[2] + k);
    C.n_gc_value = 0;
    // PressureCellType (MAC_Grid.cpp:3977-3997)
    if (pml) {
        double m = DBL_MIN;
        for (int d = 0; d < 3; ++d) {
            const double s = F.csig[d][idx[d]];
            m = m < s ? s : m;
        }
        C.r_identity = -0.5 * m / F.pml_strength;
    } else if (bulk) {
        C.r_identity = 0.5;
    } else if (!(flags & FDTD_CELL_GHOST)) {
        C.r_identity = 1.0;
    } else {
        C.r_identity = -1.0;
        C.n_gc_value = 6;
    }
    double pos[3];
    for (int d = 0; d < 3; ++d) {
        pos[d] = P.cpos[d][idx[d]];
        C.indices[d] = idx[d];
        C.centroid[d] = pos[d];
        C.lower_corner[d] = pos[d] - P.h / 2.0;
        C.upper_corner[d] = pos[d] + P.h / 2.0;
    }
    // ghost faces (MAC_Grid.cpp:4210-4227): toward -x, +x, -y, +y, -z, +z, where
    // the neighbour is bulk; they hold zero until the first step computes them, then
    // RASTERIZE pressures as MAC_Grid.cpp:1188-1281 gives them, FULLY_COUPLED the
    // solved values of the last step
    const unsigned mask = C.n_gc_value ? (unsigned)(code & CLS_MASK) : 0u;
    const long long strides[3] = {P.SX, P.SY, 1};
    const int par = cur ^ 1;
    const double t = P.consts[par].t;
    for (int f = 0; f < 6; ++f) {
        C.gc_value[f] = -1.0;
        if (!((mask >> f) & 1u)) continue;
        const int d = f >> 1;
        const int dir = (f & 1) ? +1 : -1;
        const int nb = idx[d] + dir;
        if (F.step_index == 0) {
            C.gc_value[f] = 0.0;
            continue;
        }
        if (nb < 0 || nb >= P.N[d]) continue;  // the classification sets no face off the grid
        const double pn = prev(c + dir * strides[d]);
        C.gc_value[f] = P.fc_rows ? fc_ghost(P, par, c, f, pn) : ghost_pressure(P, gobj, pos, d, dir, pn, t);
    }
    double v[6];
    for (int d = 0; d < 3; ++d) {
        int up[3] = {i, j, k};
        up[d] += 1;  // the upper face index never exceeds N[d] (MAC_Grid.cpp:4247-4249)
        C.p_directional[d] = element(P.pd[d], P.zpd[d], -1, i, j, k);
        v[2 * d] = element(P.v[F.vbuf][d], P.zv[F.vbuf][d], d, i, j, k);
        v[2 * d + 1] = element(P.v[F.vbuf][d], P.zv[F.vbuf][d], d, up[0], up[1], up[2]);
    }
    C.p_full = (double)pc[c];
    C.vx[0] = v[0], C.vx[1] = v[1];
    C.vy[0] = v[2], C.vy[1] = v[3];
    C.vz[0] = v[4], C.vz[1] = v[5];
    if (!F.reduced) flags |= FDTD_CELLINFO_PML_STATE;
    C.h = P.h;
    // the Laplacian kept for the next step: the phased path keeps the reference's
    // (every cell, every step); the fused kernels keep it on the non-PML cells of
    // a static scene (its other cells stay zero)
    if (F.step_index == 0) {
        C.laplacian = 0.0;
        flags |= FDTD_CELLINFO_LAPLACIAN;
    } else if (P.visc && (F.phased || (!F.moving && !pml))) {
        C.laplacian = P.lapv[cur] ? (double)((const T*)P.lapv[cur])[c] : NAN;
        flags |= FDTD_CELLINFO_LAPLACIAN;
    } else {
        C.laplacian = NAN;
    }
    C.flags = flags;
    made[threadIdx.x] = C;
    __syncthreads();
    constexpr int W = (int)sizeof(fdtd_cell) / 8;
    const unsigned long long* from = reinterpret_cast<const unsigned long long*>(made);
    unsigned long long* to = reinterpret_cast<unsigned long long*>(out + q0);
    for (int w = threadIdx.x; w < here * W; w += FETCH_THREADS) to[w] = from[w];
}

cudaError_t launch_fetch_cells(const SolveParams* dP, bool fp64, int cur, const FetchArgs& F, long long first, int n,
                               fdtd_cell* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int blocks = (n + FETCH_THREADS - 1) / FETCH_THREADS;
    if (fp64) k_fetch_cells<double><<<blocks, FETCH_THREADS, 0, s>>>(dP, cur, F, first, n, out);
    else k_fetch_cells<float><<<blocks, FETCH_THREADS, 0, s>>>(dP, cur, F, first, n, out);
    return cudaGetLastError();
}

template <typename T>
__global__ void __launch_bounds__(256) k_field_dense(const __grid_constant__ FieldArgs F, long long first, long long n,
                                                     double* __restrict__ out) {
    const unsigned e1 = (unsigned)F.ext[1], e2 = (unsigned)F.ext[2];
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const unsigned o = (unsigned)(first + q);  // fewer than 2^31 elements
        const unsigned row = o / e2, k = o - row * e2;
        const unsigned i = row / e1, j = row - i * e1;
        const long long c = i * F.SX + j * F.SY + k;
        const long long z = F.zsrc ? zslab_slot(F.shell, F.N[2], F.dface, (int)i, (int)j, (int)k) : -1;
        double v = z >= 0 ? (double)((const T*)F.zsrc)[z] : (double)((const T*)F.src)[c];
        if (F.inc) v = v - (double)F.inc[c];
        out[q] = v;
    }
}

cudaError_t launch_field_dense(const FieldArgs& F, bool fp64, long long first, long long n, double* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const long long blocks = (n + 255) / 256;
    const unsigned grid = (unsigned)(blocks < 148 * 8 ? blocks : 148 * 8);
    if (fp64) k_field_dense<double><<<grid, 256, 0, s>>>(F, first, n, out);
    else k_field_dense<float><<<grid, 256, 0, s>>>(F, first, n, out);
    return cudaGetLastError();
}

}  // namespace fdtd
