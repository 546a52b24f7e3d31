// fdtd_launch.hpp — host-callable launchers of the device kernels.
#pragma once
#include <cuda_runtime.h>

#include "../../include/fdtd_c.h"
#include "fdtd_device.cuh"

namespace fdtd {

// Streams of one step.  The step is enqueued on s and ends on s; in between the
// ghost-cell list runs on s3 (launched first: a few latency-bound CTAs next to
// the interior's), the interior on s2 (then the sources, where the two do not add
// them), the PML shell on s.
// s2 / s3 may be null (everything on s).
struct StepStreams {
    cudaStream_t s, s2, s3;
    cudaEvent_t fork, join, ghost;
};

// region-split step: PML shell, interior, ghost-neighbour list and (while active) sources
cudaError_t launch_step_regions_fp64(const SolveParams* dP, const SolveParams& hP, const RegionLaunch& R, int cur,
                                     const StepStreams& S, int* launches);
cudaError_t launch_step_regions_fp32(const SolveParams* dP, const SolveParams& hP, const RegionLaunch& R, int cur,
                                     const StepStreams& S, int* launches);

// a static solve's step in one launch (fdtd_one_launch.cuh): n_ghost cells of the
// ghost-neighbour list (< 0: not known on the host), the listener row of the step
// before to lis_row (null: none)
cudaError_t launch_one_fp64(const SolveParams* dP, const SolveParams& hP, const RegionLaunch& R, int cur,
                            int n_ghost, double* lis_row, cudaStream_t s, int* launches);
cudaError_t launch_one_fp32(const SolveParams* dP, const SolveParams& hP, const RegionLaunch& R, int cur,
                            int n_ghost, double* lis_row, cudaStream_t s, int* launches);
// grid cells up to which a static solve steps that way
long long one_launch_cells(int precision);

// batched step of many members (fdtd_batch.cuh)
cudaError_t launch_batch_fp64(const BatchLaunch& L, const StepStreams& S, int* launches);
cudaError_t launch_batch_fp32(const BatchLaunch& L, const StepStreams& S, int* launches);
// listener rows / advance of a batched step, for either field type (FP64 unit)
cudaError_t launch_batch_listeners_any(int precision, const BatchLaunch& L, cudaStream_t s, int* launches);
cudaError_t launch_batch_advance_any(int precision, const BatchLaunch& L, cudaStream_t s, int* launches);

// fdtd_fp64.cu (compiled with -fmad=false)
cudaError_t launch_prologue_fp64(const SolveParams* dP, int cur, int advance, int n_solid_pml, cudaStream_t s);
// listener fits and ghost-cell plans of a static scene's classification (once)
cudaError_t launch_static_prep(SolveParams* dP, int precision, int newp, int n_lis, int plan_cap, cudaStream_t s);
cudaError_t launch_consts_init(const SolveParams* dP, double t0, cudaStream_t s);
cudaError_t launch_listeners(const SolveParams* dP, int precision, int newp, int n_lis, double* out_row,
                             cudaStream_t s);
// cell classification over the boxes B (a copy of dP->boxes): the box solid
// test, the sweep over the units no box reaches and the one over those it does
// (3 launches; the last only when some box has cells).  With `prev` (the boxes
// of the classification before, when every cell outside them is known to hold
// the default flags) the first sweep visits only the units those reached.
// `meshes`: the scene's mesh bodies (the solid test by warps).
// Analytic bodies then take one launch (k_cls_tiles).  cur: the step's parity.
cudaError_t launch_classify(const SolveParams* dP, const int N[3], const ClsBoxes& B, bool collect_fresh, ClsMeshes meshes,
                            int cur, cudaStream_t s, int* launches, const ClsBoxes* prev = nullptr);
cudaError_t launch_cls_history(const SolveParams* dP, long long ncell, int* count, int* list, int cap, cudaStream_t s);
// held: where the PML cells' p^{n-1} is read (null: where p^{n+1} goes; FP64)
cudaError_t launch_fresh_cells(const SolveParams* dP, int precision, int cur, long long ncell, int* d_status,
                               cudaStream_t s, const double* held = nullptr);

// plain FP64 path, one kernel per reference phase
cudaError_t launch_phased_fp64(const SolveParams* dP, const int N[3], int cur, double* lap, cudaStream_t s,
                               int* launches);

// fdtd_fetch.cu: read-back of cells (FetchCell / SampleAxisAlignedSlice) and fields.
// Cells first, first + 1, ... of a request: the cell `cell` (dim < 0), or the plane
// k of axis dim with i over N[(dim+1)%3] outer, j over N[(dim+2)%3] inner.
struct FetchArgs {
    int dim, k;
    long long cell;
    long long step_index;
    double pml_strength;
    bool reduced, phased, moving;
    int vbuf;                 // face-velocity buffer of the current state
    const double* csig[3];    // absorption at the cell centres
    ShellBoxes shell;
};
cudaError_t launch_fetch_cells(const SolveParams* dP, bool fp64, int cur, const FetchArgs& F, long long first, int n,
                               fdtd_cell* out, cudaStream_t s);  // out may be mapped host memory
// Elements first .. first + n of a dense field (extents ext) as doubles to out:
// src (and, where the PML state is compact, zsrc) hold it; inc: subtracted (FP32
// p^{n-1}); dface: the faces' axis, -1 for cells.  out may be mapped host memory.
struct FieldArgs {
    const void* src;
    const float* inc;
    const void* zsrc;
    int ext[3], N[3], dface;
    long long SX, SY;
    ShellBoxes shell;
};
cudaError_t launch_field_dense(const FieldArgs& F, bool fp64, long long first, long long n, double* out, cudaStream_t s);

// fdtd_fp32.cu
cudaError_t prepare_fp32_kernels();
// fdtd_fp64.cu: shared-memory limits of the FP64 kernels that stage loads
cudaError_t prepare_fp64_kernels();
cudaError_t launch_prologue_fp32(const SolveParams* dP, int cur, int advance, int n_solid_pml, cudaStream_t s);

}  // namespace fdtd
