// fdtd_coupled.cuh — per-step part of the FULLY_COUPLED ghost cells
// (MAC_Grid::PML_pressureUpdateGhostCells, MAC_Grid.cpp:1131-1425): the
// right-hand side of the fixed sparse system of a static scene (rows built by
// fdtd_coupled.cpp) and its solution by BiCGSTAB with the diagonal
// preconditioner and a tolerance of one machine epsilon relative to the
// right-hand side, the reference's solver and settings (MAC_Grid.cpp:1409-1412),
// in a cluster of eight CTAs (one CTA for more rows than it holds).  The ghost pressures of a step land in fc_x[parity]; the
// ghost-cell Laplacian and the listeners of that step read them there.
#pragma once
#include "fdtd_device.cuh"
#include "fdtd_geometry.cuh"

namespace fdtd {

// Row of the ghost face of solid cell `owner` towards direction f = 2 dim +
// (sign > 0); -1 when the cell has no ghost face there.
FDTD_HD int fc_row(const SolveParams& P, long long owner, int f) {
    const int e = P.fc_idx[owner];
    if (e < 0 || !((e >> f) & 1)) return -1;
    int below = 0;
    for (int q = 0; q < f; ++q) below += (e >> q) & 1;
    return (e >> 6) + below;
}

// Ghost pressure of that face in the step of parity `par` (fallback when the
// cell has no face there, which classification rules out).
FDTD_HD double fc_ghost(const SolveParams& P, int par, long long owner, int f, double fallback) {
    const int r = fc_row(P, owner, f);
    return r < 0 ? fallback : P.fc_x[(size_t)par * P.fc_n + r];
}

// Right-hand side of row R from the pressures p, in the step of constants C.
template <typename T>
__device__ __forceinline__ double fc_rhs(const SolveParams& P, const FcRow& R, const T* __restrict__ p,
                                         const StepConsts& C) {
    const double p_neig = (double)p[R.nbr];
    if (R.kind == 1) return p_neig;
    double a[3];
    boundary_accel_g(P.obj[R.obj], R.bp, C.obj_g[R.obj], a);
    double g[3];
    for (int i = 0; i < 3; ++i) g[i] = a[i] * (-P.rho);
    double n[3] = {0.0, 0.0, 0.0};
    n[R.dim] = (R.sign > 0 ? 1.0 : -1.0);
    const double g_nr = g[0] * n[0] + g[1] * n[1] + g[2] * n[2];
    const double pg = p_neig - 0.75 * P.h * g_nr;
    if (R.kind == 0) return pg;
    if (R.kind == 3) return -pg;
    const double g_ne = g[0] * R.ne[0] + g[1] * R.ne[1] + g[2] * R.ne[2];
    double b = -(g_ne * R.fdw);
    for (int q = 0; q < 8; ++q)
        if (R.cell[q] >= 0) b -= R.w[q] * (double)p[R.cell[q]];
    if (R.si >= 0) b -= R.w[R.si] * (g_ne * P.h);
    return b;
}

template <typename T>
__global__ void __launch_bounds__(256) k_fc_rhs(const SolveParams* __restrict__ Pp, int cur) {
    const SolveParams& P = *Pp;
    const T* __restrict__ p = (const T*)P.p[cur];
    for (int ri = blockIdx.x * blockDim.x + threadIdx.x; ri < P.fc_n; ri += gridDim.x * blockDim.x)
        P.fc_b[ri] = fc_rhs<T>(P, P.fc_rows[ri], p, P.consts[cur]);
}

// Sum over the CTA (1024 threads) of one value per thread.
__device__ __forceinline__ double fc_block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? red[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (l == 0) red[32] = v;
    }
    __syncthreads();
    return red[32];
}

// diagonal of row r: +1 (kinds 0, 1) or -1 (kinds 2, 3); the preconditioner is its inverse
__device__ __forceinline__ double fc_diag(const FcRow& R) { return R.kind <= 1 ? 1.0 : -1.0; }

// out = A (D^-1 in), D the diagonal
__device__ __forceinline__ void fc_apply_precond(const SolveParams& P, const double* in, double* out) {
    for (int r = threadIdx.x; r < P.fc_n; r += blockDim.x) {
        const FcRow& R = P.fc_rows[r];
        double y = in[r];  // diag * (in / diag)
        if (R.kind == 2)
            for (int q = 0; q < 8; ++q)
                if (R.unk[q] >= 0) y += R.w[q] * (in[R.unk[q]] / fc_diag(P.fc_rows[R.unk[q]]));
        out[r] = y;
    }
}

// One CTA of 1024 threads.  BiCGSTAB from x = 0 with the right preconditioned
// update of the reference's solver; stops once |r|^2 <= eps^2 |b|^2 or after
// fc_maxit iterations (status: iterations, or -iterations when not converged).
static __global__ void __launch_bounds__(1024) k_fc_solve(const SolveParams* __restrict__ Pp, int cur) {
    const SolveParams& P = *Pp;
    __shared__ double red[33];
    const int n = P.fc_n;
    double* x = P.fc_x + (size_t)cur * n;
    double* r = P.fc_work;
    double* r0 = r + n;
    double* pv = r0 + n;
    double* v = pv + n;
    double* sv = v + n;
    double* tv = sv + n;
    const double* b = P.fc_b;
    double bb = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        x[i] = 0.0;
        r[i] = b[i];
        r0[i] = b[i];
        pv[i] = 0.0;
        v[i] = 0.0;
        bb += b[i] * b[i];
    }
    const double rhs2 = fc_block_sum(bb, red);
    if (rhs2 == 0.0) {
        if (threadIdx.x == 0) P.fc_status[0] = 0;
        return;
    }
    const double eps = 2.220446049250313e-16;
    const double tol2 = eps * eps * rhs2;
    double r0_sq = rhs2, rr = rhs2;
    double rho = 1.0, alpha = 1.0, w = 1.0;
    int it = 0, restarts = 0;
    while (rr > tol2 && it < P.fc_maxit) {
        const double rho_old = rho;
        double part = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) part += r0[i] * r[i];
        rho = fc_block_sum(part, red);
        if (fabs(rho) < eps * eps * r0_sq) {
            // the basis became orthogonal to r0: restart from the current residual
            __syncthreads();
            part = 0.0;
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const FcRow& R = P.fc_rows[i];
                double ax = fc_diag(R) * x[i];
                if (R.kind == 2)
                    for (int q = 0; q < 8; ++q)
                        if (R.unk[q] >= 0) ax += R.w[q] * x[R.unk[q]];
                r[i] = b[i] - ax;
                r0[i] = r[i];
                part += r[i] * r[i];
            }
            rho = r0_sq = fc_block_sum(part, red);
            if (restarts++ == 0) it = 0;
        }
        const double beta = (rho / rho_old) * (alpha / w);
        for (int i = threadIdx.x; i < n; i += blockDim.x) pv[i] = r[i] + beta * (pv[i] - w * v[i]);
        __syncthreads();
        fc_apply_precond(P, pv, v);  // v = A y, y = D^-1 p
        __syncthreads();
        part = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) part += r0[i] * v[i];
        alpha = rho / fc_block_sum(part, red);
        for (int i = threadIdx.x; i < n; i += blockDim.x) sv[i] = r[i] - alpha * v[i];
        __syncthreads();
        fc_apply_precond(P, sv, tv);  // t = A z, z = D^-1 s
        __syncthreads();
        double tt = 0.0, ts = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            tt += tv[i] * tv[i];
            ts += tv[i] * sv[i];
        }
        const double tt_all = fc_block_sum(tt, red);
        const double ts_all = fc_block_sum(ts, red);
        w = tt_all > 0.0 ? ts_all / tt_all : 0.0;
        part = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const double dinv = 1.0 / fc_diag(P.fc_rows[i]);
            x[i] += alpha * (pv[i] * dinv) + w * (sv[i] * dinv);
            r[i] = sv[i] - w * tv[i];
            part += r[i] * r[i];
        }
        rr = fc_block_sum(part, red);
        ++it;
    }
    if (threadIdx.x == 0) P.fc_status[0] = rr > tol2 ? -it : it;
}

// ---------------------------------------------------------------------------
// The same system by a cluster of eight CTAs, right-hand side included.  One CTA
// read every row (216 bytes) from L2 twice an iteration through one SM and met at
// six barriers of 1024 threads: 111 us for 1968 rows and 5 iterations, and 8 for the
// right-hand side before it.  Here a thread owns R rows and keeps their vectors in
// registers; of the matrix it reads the off-diagonal entries only (fc_w, fc_u: by
// entry, then by row), and every CTA has the whole of the vector being multiplied
// in its shared memory, written by its owners into all eight.  Two exchanges and
// three sums an iteration, five cluster barriers.  The sums add the CTAs' parts
// in order of rank in every CTA, so all take the same branches.
//   1968 rows: k_fc_rhs + k_fc_solve 119 us -> 31 us (80^3 FP64 step 120 -> 37 us, its
// other cells in one launch).
// More rows than FC_CLUSTER_ROWS (their vector would not fit shared memory
// comfortably) keep the one-CTA kernels.
constexpr int FC_CTAS = 8;
constexpr int FC_CLUSTER_ROWS = 4 * FC_CTAS * 512;

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// store v at the place of this CTA's shared address `a` in CTA `rank` of the cluster
__device__ __forceinline__ void cluster_store(unsigned a, unsigned rank, double v) {
    unsigned m;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(m), "d"(v) : "memory");
}

struct FcClusterSums {
    double part[16][2];                // of this CTA's warps
    double all[2][FC_CTAS][2];         // of the CTAs, two sums in flight
};

// Sums of a and b over the cluster (a barrier for everything before it too).
template <int THREADS>
__device__ __forceinline__ void fc_cluster_sum(FcClusterSums& S, unsigned rank, int& turn, double& a, double& b) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
        S.part[w][0] = a;
        S.part[w][1] = b;
    }
    __syncthreads();
    if (w == 0) {
        double s[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            s[k] = lane < THREADS / 32 ? S.part[lane][k] : 0.0;
#pragma unroll
            for (int o = THREADS / 64; o > 0; o >>= 1) s[k] += __shfl_down_sync(0xffffffffu, s[k], o);
            s[k] = __shfl_sync(0xffffffffu, s[k], 0);
        }
        if (lane < 2 * FC_CTAS) {
            const unsigned at = (unsigned)__cvta_generic_to_shared(&S.all[turn][rank][lane & 1]);
            cluster_store(at, lane >> 1, (lane & 1) ? s[1] : s[0]);
        }
    }
    cluster_barrier();
    a = b = 0.0;
#pragma unroll
    for (int c = 0; c < FC_CTAS; ++c) {
        a += S.all[turn][c][0];
        b += S.all[turn][c][1];
    }
    turn ^= 1;
}

template <typename T, int R, int THREADS>
__global__ void __cluster_dims__(FC_CTAS, 1, 1) __launch_bounds__(THREADS, 1)
    k_fc_cluster(const SolveParams* __restrict__ Pp, int cur) {
    extern __shared__ double fc_vec[];  // [fc_n] the vector being multiplied
    __shared__ FcClusterSums sums;
    asm volatile("griddepcontrol.launch_dependents;");  // the kernel after may be placed
    const SolveParams& P = *Pp;
    const int n = P.fc_n, width = P.fc_width;
    const unsigned rank = cluster_rank();
    const int first = (int)rank * THREADS + threadIdx.x;
    constexpr int STRIDE = FC_CTAS * THREADS;
    int turn = 0;
    // one row a thread: its entries in registers (unused ones at column 0 with weight 0)
    double ew[8];
    int eu[8];
    if constexpr (R == 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int u = e < width && first < n ? P.fc_u[(size_t)e * n + first] : -1;
            eu[e] = u < 0 ? 0 : u;
            ew[e] = u < 0 ? 0.0 : P.fc_w[(size_t)e * n + first];
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the step before is complete from here on
    double b[R], x[R], r[R], r0[R], pv[R], v[R], sv[R], tv[R], dg[R];
    auto exchange = [&](const double (&in)[R]) {  // fc_vec <- in, everywhere
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int i = first + k * STRIDE;
            if (i >= n) continue;
            const unsigned at = (unsigned)__cvta_generic_to_shared(fc_vec + i);
#pragma unroll
            for (unsigned c = 0; c < FC_CTAS; ++c) cluster_store(at, c, in[k]);
        }
        cluster_barrier();
    };
    auto apply = [&](const double (&in)[R], double (&out)[R]) {  // out = A (D^-1 in), in exchanged
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int i = first + k * STRIDE;
            double y = in[k];
            if constexpr (R == 1) {
#pragma unroll
                for (int e = 0; e < 8; ++e) y += ew[e] != 0.0 ? ew[e] * fc_vec[eu[e]] : 0.0;
            } else if (i < n) {
#pragma unroll 4
                for (int e = 0; e < width; ++e) {
                    const int u = P.fc_u[(size_t)e * n + i];
                    const double a = P.fc_w[(size_t)e * n + i];
                    y += u >= 0 ? a * fc_vec[u] : 0.0;
                }
            }
            out[k] = y;
        }
    };
    const T* __restrict__ p = (const T*)P.p[cur];
    const StepConsts& C = P.consts[cur];
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int i = first + k * STRIDE;
        b[k] = 0.0;
        dg[k] = 1.0;
        if (i < n) {
            const FcRow& row = P.fc_rows[i];
            dg[k] = fc_diag(row);
            b[k] = fc_rhs<T>(P, row, p, C);
        }
        x[k] = pv[k] = v[k] = 0.0;
        r[k] = r0[k] = b[k];
        s0 += b[k] * b[k];
    }
    // (the barrier also orders the CTAs' starts before the first remote store of a vector)
    cluster_barrier();
    fc_cluster_sum<THREADS>(sums, rank, turn, s0, s1);
    const double rhs2 = s0;
    const double eps = 2.220446049250313e-16;
    const double tol2 = eps * eps * rhs2;
    double r0_sq = rhs2, rr = rhs2, rho_next = rhs2;  // rho_next: r0 . r
    double rho = 1.0, alpha = 1.0, w = 1.0;
    int it = 0, restarts = 0;
    while (rr > tol2 && it < P.fc_maxit) {
        const double rho_old = rho;
        rho = rho_next;
        if (fabs(rho) < eps * eps * r0_sq) {
            // the basis became orthogonal to r0: restart from the current residual
            double xd[R], ax[R];
#pragma unroll
            for (int k = 0; k < R; ++k) xd[k] = x[k] * dg[k];  // apply() divides by the diagonal
            exchange(xd);
            apply(xd, ax);
            s0 = s1 = 0.0;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                r[k] = b[k] - ax[k];
                r0[k] = r[k];
                s0 += r[k] * r[k];
            }
            fc_cluster_sum<THREADS>(sums, rank, turn, s0, s1);
            rho = r0_sq = s0;
            if (restarts++ == 0) it = 0;
        }
        const double beta = (rho / rho_old) * (alpha / w);
#pragma unroll
        for (int k = 0; k < R; ++k) pv[k] = r[k] + beta * (pv[k] - w * v[k]);
        exchange(pv);
        apply(pv, v);  // v = A y, y = D^-1 p
        s0 = s1 = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k) s0 += r0[k] * v[k];
        fc_cluster_sum<THREADS>(sums, rank, turn, s0, s1);
        alpha = rho / s0;
#pragma unroll
        for (int k = 0; k < R; ++k) sv[k] = r[k] - alpha * v[k];
        exchange(sv);
        apply(sv, tv);  // t = A z, z = D^-1 s
        s0 = s1 = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            s0 += tv[k] * tv[k];
            s1 += tv[k] * sv[k];
        }
        fc_cluster_sum<THREADS>(sums, rank, turn, s0, s1);
        w = s0 > 0.0 ? s1 / s0 : 0.0;
        s0 = s1 = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            x[k] += alpha * (pv[k] * dg[k]) + w * (sv[k] * dg[k]);  // the diagonal is its own inverse
            r[k] = sv[k] - w * tv[k];
            s0 += r[k] * r[k];
            s1 += r0[k] * r[k];
        }
        fc_cluster_sum<THREADS>(sums, rank, turn, s0, s1);
        rr = s0;
        rho_next = s1;
        ++it;
    }
    double* out = P.fc_x + (size_t)cur * n;
#pragma unroll
    for (int k = 0; k < R; ++k)
        if (first + k * STRIDE < n) out[first + k * STRIDE] = x[k];
    if (rank == 0 && threadIdx.x == 0) P.fc_status[0] = rr > tol2 ? -it : it;
    cluster_barrier();  // no CTA's shared memory ends before the others' last stores to it
}

// Ghost pressures of a FULLY_COUPLED step of parity cur on stream s; chained: the
// step before is one kernel launched before it on s (a programmatic dependent of it).
template <typename T>
cudaError_t launch_fc(const SolveParams* dP, const SolveParams& hP, int cur, cudaStream_t s, bool chained,
                      int* launches) {
    if (hP.fc_n > FC_CLUSTER_ROWS) {
        k_fc_rhs<T><<<64, 256, 0, s>>>(dP, cur);
        k_fc_solve<<<1, 1024, 0, s>>>(dP, cur);
        if (launches) *launches += 2;
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(FC_CTAS);
    cfg.blockDim = dim3(hP.fc_n <= FC_CTAS * 256 ? 256 : 512);
    cfg.dynamicSmemBytes = (size_t)hP.fc_n * sizeof(double);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    if (launches) *launches += 1;
    if (hP.fc_n <= FC_CTAS * 256) return cudaLaunchKernelEx(&cfg, k_fc_cluster<T, 1, 256>, dP, cur);
    if (hP.fc_n <= FC_CTAS * 512) return cudaLaunchKernelEx(&cfg, k_fc_cluster<T, 1, 512>, dP, cur);
    if (hP.fc_n <= 2 * FC_CTAS * 512) return cudaLaunchKernelEx(&cfg, k_fc_cluster<T, 2, 512>, dP, cur);
    return cudaLaunchKernelEx(&cfg, k_fc_cluster<T, 4, 512>, dP, cur);
}

// shared-memory limits of the cluster kernels on the current device
template <typename T>
cudaError_t prepare_fc() {
    const int most = FC_CLUSTER_ROWS * (int)sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(k_fc_cluster<T, 2, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, most / 2);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fc_cluster<T, 4, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e;
}

}  // namespace fdtd
