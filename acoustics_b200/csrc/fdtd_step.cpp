// fdtd_step.cpp — the step loop (SimWorld::StepWorld -> RunForSteps(1) ->
// PML_WaveSolver::stepSystem -> FetchPressureData, SimWorld.cpp:507-600), CUDA
// graph capture of static scenes, read-back and snapshot/restore.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <exception>
#include <string>
#include <thread>
#include <vector>

#include "../../include/fdtd_c.h"
#include "fdtd_device.cuh"
#include "fdtd_internal.hpp"
#include "fdtd_launch.hpp"

using namespace fdtd;

#define CUDA_TRY(s, expr)                                                                   \
    do {                                                                                    \
        cudaError_t _e = (expr);                                                            \
        if (_e != cudaSuccess) {                                                            \
            set_error((s), std::string("CUDA: ") + cudaGetErrorString(_e) + " at " #expr); \
            return _e == cudaErrorMemoryAllocation ? FDTD_ERR_OOM : FDTD_ERR_CUDA;          \
        }                                                                                   \
    } while (0)

namespace {

// Classification over the boxes already in s->hP.boxes.
void classification_launches(fdtd_solver* s, int cur, fdtd_status& st, const ClsBoxes* prev) {
    const ClsBoxes& B = s->hP.boxes;
    // pageable source: the copy is staged before the call returns
    cudaError_t e = fdtd::counted_copyAsync(s, &s->dP->boxes, &B, sizeof(ClsBoxes), cudaMemcpyHostToDevice, s->stream);
    int l = 0;
    if (e == cudaSuccess) e = launch_classify(s->dP, s->N, B, s->moving, cls_meshes(s), cur, s->stream, &l, prev);
    s->launches += l;
    if (e != cudaSuccess) {
        set_error(s, std::string("classification launch: ") + cudaGetErrorString(e));
        st = FDTD_ERR_CUDA;
    }
}

// Every box with cells lies inside the non-PML box, `cells` cells from its faces.
// The classification writes pressures only at solid cells (in the boxes of
// this step) and fresh cells (in those of the step before); the shell kernel
// reads and writes the PML cells and reads one cell beyond them.
bool boxes_clear_of_shell(const fdtd_solver* s, const ClsBoxes& B, int cells = 2) {
    for (int b = 0; b < B.n; ++b) {
        if (B.first[b + 1] == B.first[b]) continue;
        for (int d = 0; d < 3; ++d)
            if (B.lo[b][d] < s->interior.lo[d] + cells || B.lo[b][d] + B.rg[b][d] > s->interior.hi[d] - cells)
                return false;
    }
    return true;
}

// How many cells from a fresh cell, along an axis, the cells of its fit may lie:
// they enclose the image of the cell's centre behind the nearest body's surface,
// as far beyond the cell as the surface is away (reflect_against_boundary).  The
// cell was solid at the last classification, its centre within h/4 of a point of a
// body that has since moved; so the surface is no farther than h/4 and the way that
// point went, and the nearest body's no farther than that.  What a body adds:
//   - an ellipsoid, whose distance is an estimate, too small by its axes' ratio at most;
//   - a mesh, whose closest point is one of the nearest triangle's, but not always
//     its nearest (tri_closest_ref): its longest edge.
// FRESH_ANYWHERE: a cell may have left the scaled box of the body that held it; its
// value then comes from the first body, wherever that is (lowest_object).
constexpr int FRESH_ANYWHERE = 1 << 30;
int fresh_reach(const fdtd_solver* s) {
    if (s->cls_objs.size() != s->objs.size()) return FRESH_ANYWHERE;
    double way = 0.0, ratio = 1.0, edge = 0.0;
    for (size_t i = 0; i < s->objs.size(); ++i) {
        const HostObject &was = s->cls_objs[i], &now = s->objs[i];
        if (now.d.shape == FDTD_SHAPE_MESH) edge = std::max(edge, s->meshes[now.d.mesh].edge);
        if (now.d.shape == FDTD_SHAPE_ELLIPSOID) {
            const double* a = now.d.size;
            ratio = std::max(ratio, std::max({a[0], a[1], a[2]}) / std::min({a[0], a[1], a[2]}));
        }
        if (now.d.motion == FDTD_MOTION_STATIC) continue;
        // (solid cells of a mesh that bounds no solid may lie far from its surface)
        if (now.d.shape == FDTD_SHAPE_MESH && !s->meshes[now.d.mesh].solid) return FRESH_ANYWHERE;
        double c2 = 0.0, turn2 = 0.0, r2 = 0.0;
        for (int d = 0; d < 3; ++d) {
            const double dc = now.c[d] - was.c[d];
            const double e = now.d.shape == FDTD_SHAPE_MESH ? std::max(std::fabs(was.mlo[d]), std::fabs(was.mhi[d]))
                                                            : now.d.size[d];
            c2 += dc * dc;
            r2 += e * e;
            // where distance_to_mesh evaluates the distance (AABB_CHECK_TOLERANCE_SCALE)
            const double mid = (now.bmax[d] + now.bmin[d]) / 2.0, half = 1.1 * (now.bmax[d] - now.bmin[d]);
            const double out = 0.25 * s->h * (1.0 + 1e-6);
            if (!(was.bmin[d] - out > mid - half && was.bmax[d] + out < mid + half)) return FRESH_ANYWHERE;
        }
        for (int k = 0; k < 9; ++k) {
            const double dr = now.d.rotation[k] - was.d.rotation[k];
            turn2 += dr * dr;
        }
        if (now.d.shape == FDTD_SHAPE_SPHERE) turn2 = 0.0;
        way = std::max(way, std::sqrt(c2) + std::sqrt(turn2 * r2));
    }
    const double cells = ((way + 0.25 * s->h) * ratio + edge) / s->h * (1.0 + 1e-6);
    return cells < 1e6 ? (int)cells + 1 : FRESH_ANYWHERE;  // (NaN and all)
}

// True when a Gaussian source may contribute at a step starting at time t:
// exp(-u^2/2) underflows to zero for |u| > 38.6 (GaussianPressureSource.cpp:21-24).
bool sources_active(const fdtd_solver* s, double t) {
    const double ts = t + 0.5 * s->k;
    for (const auto& g : s->sources)
        if (std::fabs((ts - g.offset_time) / g.width_time) < 40.0) return true;
    return false;
}

// Sources active at any step of [t, t + n k)
bool sources_active_window(const fdtd_solver* s, double t, int n) {
    for (const auto& g : s->sources) {
        const double a = (t + 0.5 * s->k - g.offset_time) / g.width_time;
        const double b = (t + (n - 0.5) * s->k - g.offset_time) / g.width_time;
        if (b > -40.0 && a < 40.0) return true;
    }
    return false;
}

// The Laplacian array of the phased path: with air viscosity the one of the
// step's parity (the previous step's stays for the update), else the single one.
double* phased_lap(const fdtd_solver* s, int cur) {
    return s->hP.visc ? (double*)s->hP.lapv[cur] : s->d_lap;
}

StepStreams step_streams(const fdtd_solver* s) {
    return StepStreams{s->stream, s->stream2, s->stream3, s->ev_fork, s->ev_join, s->ev_ghost};
}

// True when no listener stencil (the cells its MLS may read, two cells around
// them) meets a classification box: the classification of the next step writes
// flags and pressures only inside its boxes, its fresh cells lie in the boxes of
// this step.
}  // namespace
namespace fdtd {
bool listeners_clear_of(const fdtd_solver* s, const ClsBoxes& B) {
    for (int l = 0; l < s->L; ++l) {
        int lo[3], hi[3];
        for (int d = 0; d < 3; ++d) {
            const double diff = (s->listeners[3 * (size_t)l + d] - s->bmin[d]) - s->h / 2.0;
            const int a0 = std::min(std::max((int)(diff / s->h), 0), s->N[d] - 1);
            lo[d] = a0 - 2;
            hi[d] = a0 + 4;
        }
        for (int b = 0; b < B.n; ++b) {
            if (B.first[b + 1] == B.first[b]) continue;
            bool meet = true;
            for (int d = 0; d < 3; ++d) meet = meet && lo[d] < B.lo[b][d] + B.rg[b][d] && B.lo[b][d] < hi[d];
            if (meet) return false;
        }
    }
    return true;
}
}  // namespace fdtd
namespace {

// The listener rows of a step run on stream4 beside the next step while every
// listener stencil is clear of this step's classification boxes (static scenes
// after their first step; for moving bodies the next step waits for the rows if
// its own boxes reach a stencil).  A stencil that holds a ghost cell is not: its
// rows also read p^n beside the solid, in the buffer the next step writes.  Not
// with Engquist cells either (the step after writes the exterior cells of the
// pressure they read) or solids in the PML (re-zeroed at the start of every step).
bool listeners_aside(const fdtd_solver* s, bool classify) {
    if (!s->stream4 || s->n_solid_pml != 0 || !s->eng.empty()) return false;
    return s->moving ? listeners_clear_of(s, s->hP.boxes) : (!classify && s->lis_clear);
}

// Make the solver stream wait for every listener launch on stream4.
fdtd_status join_listeners(fdtd_solver* s) {
    if (!s->lis_pending[0] && !s->lis_pending[1]) return FDTD_OK;
    CUDA_TRY(s, cudaEventRecord(s->ev_lis_join, s->stream4));
    CUDA_TRY(s, cudaStreamWaitEvent(s->stream, s->ev_lis_join, 0));
    s->lis_pending[0] = s->lis_pending[1] = false;
    return FDTD_OK;
}

// The interior's x planes by their distance from the boxes of this step's and the
// last step's classification: `near` those within PLANES_REACH, `far` the others;
// both empty when the far ones are too few to start apart.  The classification
// touches cells one beyond a box, a fresh cell lies in the last step's box and its
// fit reads p^n and p^{n-1} at most fresh_reach() cells from it (near planes go as
// far where that is farther), and the cells of both are read one cell further.
// Only where the interior is long enough to hide the classification behind and the
// shell leaves it room (us a step, together / apart; two spheres):
//   FP32  96^3 56.9 / 57.0, 160x150x170 66.7 / 62.9, 256^3 112.6 / 105.5,
//         320x320x256 140.3 / 131.5, 384x384x256 172.0 / 169.8
//   FP64 (a shell CTA leaves one interior CTA's registers, which run beside it
//         anyway)  224x200x210 120.2 / 122.6, 256^3 158.7 / 167.2
constexpr int PLANES_REACH = 6;
constexpr long long PLANES_CELLS = 2000000;
void planes_ahead(const fdtd_solver* s, const ClsBoxes& prev, int fresh, XRanges& far, XRanges& near) {
    if (s->precision == FDTD_PRECISION_FP64 || s->n_interior < PLANES_CELLS) return;
    const int lo = s->region.interior.lo[0], hi = s->region.interior.hi[0];
    if (hi <= lo || fresh >= hi - lo) return;
    const int around = std::max(PLANES_REACH, fresh);
    std::vector<char> reach(hi - lo, 0);
    for (const ClsBoxes* B : {&prev, &s->hP.boxes})
        for (int b = 0; b < B->n; ++b) {
            if (B->first[b + 1] == B->first[b]) continue;
            const int a = std::max(lo, B->lo[b][0] - around);
            const int e = std::min(hi, B->lo[b][0] + B->rg[b][0] + around);
            for (int x = a; x < e; ++x) reach[x - lo] = 1;
        }
    auto push = [](XRanges& X, int a, int e) {
        X.lo[X.n] = a;
        X.hi[X.n++] = e;
    };
    int n_far = 0;
    for (int x = lo; x < hi;) {
        int e = x;
        while (e < hi && reach[e - lo] == reach[x - lo]) ++e;
        if (!reach[x - lo]) n_far += e - x;
        XRanges& X = reach[x - lo] ? near : far;
        if (X.n == MAX_X_RANGES) n_far = -hi;  // (cannot be: a range per box at most, and one more)
        else push(X, x, e);
        x = e;
    }
    // (no near plane: nothing waits for the classification, and a range is needed to say so)
    if (4 * n_far < hi - lo || near.n == 0) far.n = near.n = 0;
}

// Room to hold p^{n-1} (FP64); false: none to be had.
bool make_held(fdtd_solver* s) {
    void* d = nullptr;
    if (cudaMalloc(&d, (size_t)s->np * 8) != cudaSuccess ||
        (!s->ev_held && cudaEventCreateWithFlags(&s->ev_held, cudaEventDisableTiming) != cudaSuccess)) {
        cudaGetLastError();
        if (d) cudaFree(d);
        return false;
    }
    s->held = (double*)d;
    s->arena_bytes += (size_t)s->np * 8;
    return true;
}

// The row a one-launch step left to its successor; newp: the parity of the
// current pressure.
fdtd_status flush_lag(fdtd_solver* s, int newp) {
    if (!s->lag_row) return FDTD_OK;
    CUDA_TRY(s, launch_listeners(s->dP, s->precision, newp, s->L, s->lag_row, s->stream));
    s->launches++;
    s->lag_row = nullptr;
    return FDTD_OK;
}

// Listener fits and ghost-cell plans of a static scene's classification.
fdtd_status static_prep(fdtd_solver* s, int newp) {
    CUDA_TRY(s, launch_static_prep(s->dP, s->precision, newp, s->L, s->hP.plan_cap, s->stream));
    s->launches += 1 + (s->L > 0) + (s->hP.plan_cap > 0);
    // host mirrors of the flags the prep sets (later uploads keep them)
    s->hP.lis_ready = 1;
    s->hP.plan_ready = s->hP.plan_cap > 0;
    return FDTD_OK;
}

// Enqueue one time step with the pressure parity `cur`; listener row to dev_row.
fdtd_status enqueue_step(fdtd_solver* s, int cur, double* dev_row, bool classify, bool src) {
    s->region.sources = src ? 1 : 0;
    fdtd_status st = FDTD_OK;
    // this step writes the pressure slot the listeners of the step before last read
    if (s->lis_pending[cur]) {
        CUDA_TRY(s, cudaStreamWaitEvent(s->stream, s->ev_lis[cur], 0));
        s->lis_pending[cur] = false;
    }
    const bool fused = s->opt.kernel == FDTD_KERNEL_FUSED;
    bool shell_ahead = false;
    XRanges near{};  // interior planes left to this step's classification (n = 0: all)
    if (classify) {
        // MAC_Grid::classifyCells_FAST + InterpolateFreshPressureCell (PML_WaveSolver.cpp:807-812)
        const ClsBoxes prev = s->hP.boxes;
        classification_boxes(s, s->hP.boxes);
        // the rows of the step before still being read beside this step: this
        // step's classification must not write under a listener stencil first
        if (s->lis_pending[cur ^ 1] && !listeners_clear_of(s, s->hP.boxes)) {
            CUDA_TRY(s, cudaStreamWaitEvent(s->stream, s->ev_lis[cur ^ 1], 0));
            s->lis_pending[cur ^ 1] = false;
        }
        if (s->moving && s->region.red && !boxes_clear_of_shell(s, s->hP.boxes)) {
            // past the end time the bodies were checked for: the reduced PML state no longer holds
            set_error(s, "a moving body came within two cells of the PML of a reduced-state solve (past its end_time)");
            return FDTD_ERR_UNSUPPORTED;
        }
        // Interior planes out of reach of the bodies' boxes hold no cell the
        // classification or the fresh cells touch or read: they start first, on
        // stream6, beside both.
        const int fresh = s->moving && s->cls_boxes_current ? fresh_reach(s) : FRESH_ANYWHERE;
        if (s->moving) s->cls_objs = s->objs;
        XRanges far{};
        if (s->moving && fused && s->cls_boxes_current && !s->hP.visc && s->eng.empty() && s->stream6 &&
            s->boundary_handling == FDTD_BOUNDARY_RASTERIZE && s->region.xb == 2)
            planes_ahead(s, prev, fresh, far, near);
        // Moving bodies clear of the PML: the shell kernel reads nothing the
        // classification writes, so it starts first too.  In FP64 it writes p^{n+1} over
        // p^{n-1}, which a fresh cell's fit that lies in the PML (a body gone many cells
        // in this step) then reads from a copy made before.
        shell_ahead = s->moving && fused && s->cls_boxes_current && s->n_solid_pml == 0 && !s->hP.visc &&
                      s->eng.empty() &&
                      s->stream5 && s->interior.hi[0] > s->interior.lo[0] && boxes_clear_of_shell(s, prev) &&
                      boxes_clear_of_shell(s, s->hP.boxes);
        const bool hold = shell_ahead && s->precision == FDTD_PRECISION_FP64 &&
                          !(fresh < FRESH_ANYWHERE && boxes_clear_of_shell(s, prev, fresh));
        if (hold && !s->held) shell_ahead = make_held(s);
        const double* held = hold && shell_ahead ? s->held : nullptr;
        if (shell_ahead || far.n > 0) {
            CUDA_TRY(s, cudaEventRecord(s->ev_sfork, s->stream));
            const auto ahead = [&](cudaStream_t on, cudaEvent_t done, int skip, const XRanges& planes) -> fdtd_status {
                RegionLaunch R = s->region;
                R.skip |= 4 | skip;  // no ghost list
                R.x = planes;
                if (skip & 1) R.sources = 0;
                R.fc = 0;
                const StepStreams S{on, nullptr, nullptr, s->ev_fork, s->ev_join, s->ev_ghost};
                CUDA_TRY(s, cudaStreamWaitEvent(on, s->ev_sfork, 0));
                int l = 0;
                if (s->precision == FDTD_PRECISION_FP64)
                    CUDA_TRY(s, launch_step_regions_fp64(s->dP, s->hP, R, cur, S, &l));
                else
                    CUDA_TRY(s, launch_step_regions_fp32(s->dP, s->hP, R, cur, S, &l));
                s->launches += l;
                CUDA_TRY(s, cudaEventRecord(done, on));
                return FDTD_OK;
            };
            // (the interior first: its CTAs are short, so the classification's find room sooner)
            if (far.n > 0) {
                const fdtd_status fst = ahead(s->stream6, s->ev_fdone, 2, far);
                if (fst != FDTD_OK) return fst;
            }
            if (held) {
                // (the classification zeroes cells of bodies meanwhile, which are not PML cells)
                CUDA_TRY(s, cudaStreamWaitEvent(s->stream5, s->ev_sfork, 0));
                CUDA_TRY(s, cudaMemcpyAsync(s->held, s->hP.p[cur ^ 1], (size_t)s->np * 8, cudaMemcpyDeviceToDevice, s->stream5));
                CUDA_TRY(s, cudaEventRecord(s->ev_held, s->stream5));
            }
            if (shell_ahead) {
                const fdtd_status sst = ahead(s->stream5, s->ev_sdone, 1, XRanges{});
                if (sst != FDTD_OK) return sst;
                s->overlapped_steps++;
            }
        }
        // moving bodies after a classification of the step before: only the units
        // its boxes reached can hold flags other than the defaults
        classification_launches(s, cur, st, (s->moving && s->cls_boxes_current) ? &prev : nullptr);
        // (the one-launch classification of analytic bodies makes the ghost list's plans)
        if (s->moving) s->hP.plan_ready = s->cls_boxes_current && s->hP.plan_cap > 0;
        s->cls_boxes_current = true;
        if (st != FDTD_OK) return st;
        if (s->moving) {
            if (held) CUDA_TRY(s, cudaStreamWaitEvent(s->stream, s->ev_held, 0));
            CUDA_TRY(s, launch_fresh_cells(s->dP, s->precision, cur, s->ncell, s->d_status, s->stream, held));
            s->launches++;
            if (s->boundary_handling == FDTD_BOUNDARY_FULLY_COUPLED) {
                // the coupled rows of this step's ghost faces (host build from the new flags)
                st = build_fully_coupled(s);
                if (st != FDTD_OK) return st;
                s->region.fc = s->hP.fc_n > 0 ? 1 : 0;
                CUDA_TRY(s, fdtd::counted_copyAsync(s, s->dP, &s->hP, sizeof(SolveParams), cudaMemcpyHostToDevice,
                                                    s->stream));
            }
        }
        if (!s->moving) {
            // static classification: the listener fits become fixed weights, the
            // ghost list's cells plans
            const fdtd_status pst = static_prep(s, cur ^ 1);
            if (pst != FDTD_OK) return pst;
        }
    }
    if (s->region.one) {
        int l = 0;
        cudaError_t e = s->precision == FDTD_PRECISION_FP64
                            ? launch_one_fp64(s->dP, s->hP, s->region, cur, s->n_ghost, s->lag_row, s->stream, &l)
                            : launch_one_fp32(s->dP, s->hP, s->region, cur, s->n_ghost, s->lag_row, s->stream, &l);
        CUDA_TRY(s, e);
        s->launches += l;
        s->lag_row = nullptr;
        if (s->L > 0 && dev_row) {
            if (s->lis_clear) {
                s->lag_row = dev_row;  // by the next step's launch, or flush_lag
            } else {
                CUDA_TRY(s, launch_listeners(s->dP, s->precision, cur ^ 1, s->L, dev_row, s->stream));
                s->launches++;
            }
        }
        return FDTD_OK;
    }
    // the region-split path advances the step constants inside its shell kernel;
    // the prologue then only runs to re-zero solid cells inside the PML, or to
    // advance the constants of a grid without PML cells
    RegionLaunch R = s->region;
    if (shell_ahead) R.skip |= 2;
    R.x = near;
    const bool no_shell = R.shell.block_first[R.shell.n] == 0;
    const int advance = (!fused || no_shell) ? 1 : 0;
    if (s->precision == FDTD_PRECISION_FP64) {
        if (advance || s->n_solid_pml > 0) {
            CUDA_TRY(s, launch_prologue_fp64(s->dP, cur, advance, s->n_solid_pml, s->stream));
            s->launches++;
        }
        int l = 0;
        if (s->opt.kernel == FDTD_KERNEL_PHASED) {
            CUDA_TRY(s, launch_phased_fp64(s->dP, s->N, cur, phased_lap(s, cur), s->stream, &l));
        } else {
            CUDA_TRY(s, launch_step_regions_fp64(s->dP, s->hP, R, cur, step_streams(s), &l));
        }
        s->launches += l;
    } else {
        if (advance || s->n_solid_pml > 0) {
            CUDA_TRY(s, launch_prologue_fp32(s->dP, cur, advance, s->n_solid_pml, s->stream));
            s->launches++;
        }
        int l = 0;
        CUDA_TRY(s, launch_step_regions_fp32(s->dP, s->hP, R, cur, step_streams(s), &l));
        s->launches += l;
    }
    if (shell_ahead) CUDA_TRY(s, cudaStreamWaitEvent(s->stream, s->ev_sdone, 0));
    if (near.n > 0) CUDA_TRY(s, cudaStreamWaitEvent(s->stream, s->ev_fdone, 0));
    if (s->L > 0 && dev_row) {
        // the phased path keeps p^{n+1} in the same slot as the fused one
        if (listeners_aside(s, classify)) {
            CUDA_TRY(s, cudaEventRecord(s->ev_step, s->stream));
            CUDA_TRY(s, cudaStreamWaitEvent(s->stream4, s->ev_step, 0));
            CUDA_TRY(s, launch_listeners(s->dP, s->precision, cur ^ 1, s->L, dev_row, s->stream4));
            CUDA_TRY(s, cudaEventRecord(s->ev_lis[cur], s->stream4));
            s->lis_pending[cur] = true;
        } else {
            CUDA_TRY(s, launch_listeners(s->dP, s->precision, cur ^ 1, s->L, dev_row, s->stream));
        }
        s->launches++;
    }
    return FDTD_OK;
}

// Host bookkeeping after a step: parity, clock mirror, object animation
// (SimWorld::UpdateObjectState(t + dt), SimWorld.cpp:596-600).
fdtd_status after_step(fdtd_solver* s) {
    s->cur ^= 1;
    s->step_index++;
    s->time += s->k;
    if (s->moving) {
        s->state_time += s->k;
        for (size_t i = 0; i < s->objs.size(); ++i) {
            auto& o = s->objs[i];
            if (o.d.motion == FDTD_MOTION_STATIC) continue;
            host_object_pose(o, s->state_time);
            host_update_bbox(o);
        }
        to_dev_objects(s);
        CUDA_TRY(s, fdtd::counted_copyAsync(s, &s->dP->obj[0], &s->hP.obj[0], sizeof(DevObject) * s->objs.size(),
                                    cudaMemcpyHostToDevice, s->stream));
    }
    return FDTD_OK;
}

fdtd_status check_device_errors(fdtd_solver* s) {
    // the error flags, the status words and the list lengths in one copy to pinned
    // memory and one wait (three copies to pageable memory and two waits: 64^3 FP64
    // stepped one by one 69 us a step instead of 31)
    CUDA_TRY(s, fdtd::counted_copyAsync(s, s->h_status, s->hP.dev_error, status_bytes(s), cudaMemcpyDeviceToHost, s->stream));
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    const int dev_error = s->h_status[0];
    const int* status = s->h_status + (s->d_status - s->hP.dev_error);
    const int* counts = s->h_status + (s->d_ghost_count - s->hP.dev_error);  // list_counts
    const int ghosts = s->moving ? std::max(counts[0], counts[2]) : counts[0];
    if (!s->moving) s->n_ghost = ghosts;
    if (ghosts > s->region.ghost_cap) {
        set_error(s, "ghost-neighbour list overflow (" + std::to_string(ghosts) + " > " +
                         std::to_string(s->region.ghost_cap) + ")");
        return FDTD_ERR_OOM;
    }
    if (status[0] == 2) {
        set_error(s, "fresh cell inside an object (MAC_Grid.cpp:2050-2053)");
        return FDTD_ERR_GEOMETRY;
    }
    if (dev_error & 1) {
        set_error(s, "listener sample not finite, or a degenerate listener stencil (no cell or rank-deficient MLS)");
        return FDTD_ERR_NUMERIC;
    }
    if (dev_error & fdtd::DEV_ERR_ENGQUIST) {
        set_error(s, "a solid cell reaches the stencil of an Engquist-Majda boundary cell (the ghost-pressure forms of "
                     "MAC_Grid.cpp:533-920 are not built): keep bodies and constraints three cells from sides without PML");
        return FDTD_ERR_UNSUPPORTED;
    }
    if (dev_error & fdtd::FDTD_DEV_ERR_TMA_TIMEOUT) {
        set_error(s, "a tensor copy of the PML-shell kernel did not complete within its bounded wait");
        return FDTD_ERR_TIMEOUT;
    }
    return FDTD_OK;
}

// Capture `n` steps starting at parity `cur` into a graph (static scenes only).
fdtd_status capture_graph(fdtd_solver* s, int cur, int n, bool src, cudaGraphExec_t* out) {
    cudaGraph_t g = nullptr;
    fdtd_status st = join_listeners(s);  // no dependency on work outside the capture
    if (st != FDTD_OK) return st;
    CUDA_TRY(s, cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    int c = cur;
    for (int i = 0; i < n && st == FDTD_OK; ++i) {
        st = enqueue_step(s, c, s->d_lis + (size_t)i * s->L, false, src);
        c ^= 1;
    }
    if (st == FDTD_OK) st = flush_lag(s, c);
    if (st == FDTD_OK) st = join_listeners(s);  // the graph ends with every row written
    s->lis_pending[0] = s->lis_pending[1] = false;
    cudaError_t e = cudaStreamEndCapture(s->stream, &g);
    if (st != FDTD_OK) {
        if (g) cudaGraphDestroy(g);
        return st;
    }
    if (e != cudaSuccess) {
        set_error(s, std::string("graph capture: ") + cudaGetErrorString(e));
        return FDTD_ERR_CUDA;
    }
    e = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    // the graph's device-side setup now, not at its first launch
    if (e == cudaSuccess) e = cudaGraphUpload(*out, s->stream);
    if (e != cudaSuccess) {
        set_error(s, std::string("graph instantiate: ") + cudaGetErrorString(e));
        return FDTD_ERR_CUDA;
    }
    return FDTD_OK;
}

// Run n steps; listener rows land in the device ring d_lis (chunks of at most
// lis_cap_steps) and are passed to `sink(first_step, count)` after each chunk.
// Static scenes replay captured graphs of graph_steps steps once the first
// step (which classifies) has run.
template <typename Sink>
fdtd_status run_steps(fdtd_solver* s, int n, Sink sink) {
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    const long long launches0 = s->launches;
    const int G = s->opt.graph_steps;
    int done = 0;
    while (done < n) {
        const int remaining = n - done;
        const bool classify_now = s->moving || s->step_index == 0;
        if (!classify_now && G > 0 && remaining >= G) {
            const bool src = sources_active_window(s, s->time, G);
            const int key = s->cur + (src ? 2 : 0);
            if (!s->graph_exec[key]) {
                const long long l0 = s->launches;
                fdtd_status st = capture_graph(s, s->cur, G, src, &s->graph_exec[key]);
                if (st != FDTD_OK) return st;
                s->graph_launches_per_exec = s->launches - l0;
                s->launches = l0;
            }
            CUDA_TRY(s, cudaGraphLaunch(s->graph_exec[key], s->stream));
            s->launches += s->graph_launches_per_exec;
            for (int q = 0; q < G; ++q) {
                fdtd_status st = after_step(s);
                if (st != FDTD_OK) return st;
            }
            fdtd_status st = sink(done, G);
            if (st != FDTD_OK) return st;
            done += G;
            continue;
        }
        int m = std::min(remaining, s->lis_cap_steps);
        if (G > 0 && !s->moving && classify_now) m = 1;
        for (int i = 0; i < m; ++i) {
            const bool classify = s->moving || s->step_index == 0;
            fdtd_status st = enqueue_step(s, s->cur, s->d_lis + (size_t)i * s->L, classify, sources_active(s, s->time));
            if (st != FDTD_OK) return st;
            st = after_step(s);
            if (st != FDTD_OK) return st;
        }
        fdtd_status st = flush_lag(s, s->cur);
        if (st == FDTD_OK) st = join_listeners(s);
        if (st != FDTD_OK) return st;
        st = sink(done, m);
        if (st != FDTD_OK) return st;
        done += m;
    }
    s->last_launches = s->launches - launches0;
    return FDTD_OK;
}

// FDTD_CELL_* bits of cell (i, j, k) from its classification and ghost-object bytes.
uint8_t cell_flags(const fdtd_solver* s, uint8_t code, uint8_t gobj, int i, int j, int k) {
    const bool bulk = code & CLS_BULK;
    uint8_t f = 0;
    if (bulk) f |= FDTD_CELL_BULK;
    if (!bulk && (code & CLS_MASK)) f |= FDTD_CELL_GHOST;
    if (code & CLS_VALID) f |= FDTD_CELL_VALID_HISTORY;
    if (s->tab[0].pml_cell[i] || s->tab[1].pml_cell[j] || s->tab[2].pml_cell[k]) f |= FDTD_CELL_PML;
    if (!bulk && (gobj & GOBJ_CONSTRAINT)) f |= FDTD_CELL_CONSTRAINT;
    return f;
}

}  // namespace

extern "C" {

fdtd_status fdtd_solver_step(fdtd_solver* s, int32_t n_steps, double* listener_out) {
    if (!s || n_steps < 0) return (set_error(s, "invalid arguments"), FDTD_ERR_INVALID_ARG);
    const int L = s->L;
    // rows of consecutive chunks gather in the pinned staging buffer (copies in
    // stream order, before the next chunk rewrites the device ring); the host
    // waits only when the buffer is full and at the end
    int staged = 0, staged_first = 0;
    auto flush = [&]() -> fdtd_status {
        if (staged == 0) return FDTD_OK;
        CUDA_TRY(s, cudaStreamSynchronize(s->stream));
        std::memcpy(listener_out + (size_t)staged_first * L, s->h_lis_stage, (size_t)staged * L * 8);
        staged = 0;
        return FDTD_OK;
    };
    fdtd_status st = run_steps(s, n_steps, [&](int first, int count) -> fdtd_status {
        if (listener_out && L > 0) {
            if (staged + count > s->lis_cap_steps) {
                const fdtd_status f = flush();
                if (f != FDTD_OK) return f;
            }
            if (staged == 0) staged_first = first;
            CUDA_TRY(s, fdtd::counted_copyAsync(s, s->h_lis_stage + (size_t)staged * L, s->d_lis, (size_t)count * L * 8,
                                        cudaMemcpyDeviceToHost, s->stream));
            staged += count;
        }
        return FDTD_OK;
    });
    if (st != FDTD_OK) return st;
    st = flush();
    if (st != FDTD_OK) return st;
    st = check_device_errors(s);
    if (st != FDTD_OK) return st;
    if (s->end_time > 0.0 && s->time >= s->end_time) return FDTD_END_OF_TIME;
    return FDTD_OK;
}

fdtd_status fdtd_solver_step_device(fdtd_solver* s, int32_t n_steps, void* device_listener_out) {
    if (!s || n_steps < 0) return (set_error(s, "invalid arguments"), FDTD_ERR_INVALID_ARG);
    const int L = s->L;
    double* out = (double*)device_listener_out;
    fdtd_status st = run_steps(s, n_steps, [&](int first, int count) -> fdtd_status {
        if (out && L > 0)
            CUDA_TRY(s, fdtd::counted_copyAsync(s, out + (size_t)first * L, s->d_lis, (size_t)count * L * 8,
                                        cudaMemcpyDeviceToDevice, s->stream));
        return FDTD_OK;
    });
    return st;
}

fdtd_status fdtd_solver_fetch_listeners(fdtd_solver* s, double* out) {
    if (!s || (!out && s->L > 0)) return (set_error(s, "invalid arguments"), FDTD_ERR_INVALID_ARG);
    if (s->L == 0) return FDTD_OK;
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    CUDA_TRY(s, launch_listeners(s->dP, s->precision, s->cur, s->L, s->d_lis, s->stream));
    // (pinned staging: a step leaves nothing in it)
    CUDA_TRY(s, fdtd::counted_copyAsync(s, s->h_lis_stage, s->d_lis, (size_t)s->L * 8, cudaMemcpyDeviceToHost, s->stream));
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    std::memcpy(out, s->h_lis_stage, (size_t)s->L * 8);
    return FDTD_OK;
}

fdtd_status fdtd_solver_time_kernel(fdtd_solver* s, int32_t which, int32_t n_launches, float* elapsed_ms) {
    if (!s || n_launches <= 0 || !elapsed_ms || which < 0 || which > 4)
        return (set_error(s, "invalid arguments"), FDTD_ERR_INVALID_ARG);
    if (which > 0 && s->opt.kernel != FDTD_KERNEL_FUSED)
        return (set_error(s, "single-kernel timing needs the region-split (fused) path"), FDTD_ERR_INVALID_ARG);
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    cudaEvent_t e0, e1;
    CUDA_TRY(s, cudaEventCreate(&e0));
    CUDA_TRY(s, cudaEventCreate(&e1));
    RegionLaunch R = s->region;
    R.sources = 0;
    if (which == 1) R.skip = 2 | 4;
    if (which == 2) R.skip = 1 | 4;
    if (which == 3) R.skip = 1 | 2;
    // the launches are captured into a graph and the graph is timed: device time
    // only, whatever the host's launch rate (a step forks to three streams)
    fdtd_status jst = join_listeners(s);
    if (jst != FDTD_OK) return jst;
    // moving bodies: the list of the last classification, whose lengths are those of
    // its parity, in the launches of both (the next step's pair is empty again below)
    int* const counts = s->d_ghost_count;
    if (s->moving)
        CUDA_TRY(s, cudaMemcpyAsync(counts + 2 * s->cur, counts + 2 * (s->cur ^ 1), 2 * sizeof(int),
                                    cudaMemcpyDeviceToDevice, s->stream));
    const bool one = which == 0 && s->region.one;
    CUDA_TRY(s, cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    int c = s->cur;
    for (int i = 0; i < n_launches; ++i) {
        cudaError_t e;
        if (which == 4) {
            e = launch_listeners(s->dP, s->precision, c, s->L, s->d_lis, s->stream);
        } else if (one) {
            e = s->precision == FDTD_PRECISION_FP64
                    ? launch_one_fp64(s->dP, s->hP, R, c, s->n_ghost, nullptr, s->stream, nullptr)
                    : launch_one_fp32(s->dP, s->hP, R, c, s->n_ghost, nullptr, s->stream, nullptr);
        } else if (s->precision == FDTD_PRECISION_FP64) {
            if (s->opt.kernel == FDTD_KERNEL_PHASED) e = launch_phased_fp64(s->dP, s->N, c, phased_lap(s, c), s->stream, nullptr);
            else e = launch_step_regions_fp64(s->dP, s->hP, R, c, step_streams(s), nullptr);
        } else {
            e = launch_step_regions_fp32(s->dP, s->hP, R, c, step_streams(s), nullptr);
        }
        if (e != cudaSuccess) {
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(s->stream, &g);
            if (g) cudaGraphDestroy(g);
            set_error(s, std::string("stencil launch: ") + cudaGetErrorString(e));
            return FDTD_ERR_CUDA;
        }
        if (which != 4) c ^= 1;
    }
    cudaGraph_t g = nullptr;
    CUDA_TRY(s, cudaStreamEndCapture(s->stream, &g));
    cudaGraphExec_t x = nullptr;
    cudaError_t ge = cudaGraphInstantiate(&x, g, 0);
    cudaGraphDestroy(g);
    if (ge != cudaSuccess) {
        set_error(s, std::string("stencil graph: ") + cudaGetErrorString(ge));
        return FDTD_ERR_CUDA;
    }
    // one untimed replay, one timed: 2 n launches, so the parity comes back
    ge = cudaGraphLaunch(x, s->stream);
    if (ge == cudaSuccess) ge = cudaEventRecord(e0, s->stream);
    if (ge == cudaSuccess) ge = cudaGraphLaunch(x, s->stream);
    if (ge == cudaSuccess) ge = cudaEventRecord(e1, s->stream);
    if (ge == cudaSuccess) ge = cudaEventSynchronize(e1);
    if (ge == cudaSuccess) ge = cudaEventElapsedTime(elapsed_ms, e0, e1);
    if (ge == cudaSuccess && s->moving) ge = cudaMemsetAsync(counts + 2 * s->cur, 0, 2 * sizeof(int), s->stream);
    cudaGraphExecDestroy(x);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (ge != cudaSuccess) {
        set_error(s, std::string("stencil timing: ") + cudaGetErrorString(ge));
        return FDTD_ERR_CUDA;
    }
    return FDTD_OK;
}

fdtd_status fdtd_solver_time_stencil(fdtd_solver* s, int32_t n_launches, float* elapsed_ms) {
    return fdtd_solver_time_kernel(s, 0, n_launches, elapsed_ms);
}

fdtd_status fdtd_solver_synchronize(fdtd_solver* s) {
    if (!s) return FDTD_ERR_INVALID_ARG;
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    return FDTD_OK;
}

void* fdtd_solver_stream(fdtd_solver* s) { return s ? (void*)s->stream : nullptr; }

const char* fdtd_solver_last_error(fdtd_solver* s) { return s ? s->err.c_str() : ""; }

int64_t fdtd_solver_last_launch_count(fdtd_solver* s) { return s ? s->last_launches : 0; }

int64_t fdtd_solver_overlapped_steps(fdtd_solver* s) { return s ? s->overlapped_steps : 0; }

int32_t fdtd_solver_shell_staging(fdtd_solver* s) {
    if (!s || !s->region.red) return -1;
    return s->region.tma ? FDTD_SHELL_STAGING_TMA : FDTD_SHELL_STAGING_RING;
}

fdtd_status fdtd_solver_transfer_bytes(fdtd_solver* s, int64_t* host_to_device, int64_t* device_to_host) {
    if (!s || !host_to_device || !device_to_host) return (set_error(s, "invalid arguments"), FDTD_ERR_INVALID_ARG);
    *host_to_device = s->bytes_h2d;
    *device_to_host = s->bytes_d2h;
    return FDTD_OK;
}

fdtd_status fdtd_solver_prepare_graphs(fdtd_solver* s) {
    if (!s) return FDTD_ERR_INVALID_ARG;
    const int G = s->opt.graph_steps;
    if (G <= 0 || s->moving || s->step_index == 0) return FDTD_OK;
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    const bool src = sources_active_window(s, s->time, G);
    const int key = s->cur + (src ? 2 : 0);
    if (s->graph_exec[key]) return FDTD_OK;
    const long long l0 = s->launches;
    fdtd_status st = capture_graph(s, s->cur, G, src, &s->graph_exec[key]);
    if (st != FDTD_OK) return st;
    s->graph_launches_per_exec = s->launches - l0;
    s->launches = l0;
    return FDTD_OK;
}

int32_t fdtd_solver_pml_state(fdtd_solver* s) {
    return (s && s->region.red) ? FDTD_PML_STATE_AUTO : FDTD_PML_STATE_FULL;
}

fdtd_status fdtd_solver_info_get(fdtd_solver* s, fdtd_solver_info* info) {
    if (!s || !info) return FDTD_ERR_INVALID_ARG;
    std::memset(info, 0, sizeof(*info));
    for (int d = 0; d < 3; ++d) info->divisions[d] = s->N[d];
    info->n_listeners = s->L;
    info->n_cells = s->ncell;
    info->n_pml_cells = s->n_pml;
    info->n_interior_cells = s->n_interior;
    info->device_bytes = (int64_t)s->arena_bytes;
    info->step_index = s->step_index;
    info->time = s->time;
    info->time_step = s->k;
    const double w = s->precision == FDTD_PRECISION_FP64 ? 8.0 : 4.0;
    info->algorithmic_bytes_per_step = w * (3.0 * (double)s->n_interior + 14.0 * (double)s->n_pml);
    return FDTD_OK;
}

fdtd_status fdtd_solver_get_classification(fdtd_solver* s, uint8_t* flags, fdtd_ghost_face* faces, int64_t* n_faces) {
    if (!s) return FDTD_ERR_INVALID_ARG;
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    std::vector<uint8_t> pcls(s->np), pgobj(s->np);
    CUDA_TRY(s, fdtd::counted_copyAsync(s, pcls.data(), s->hP.cls, s->np, cudaMemcpyDeviceToHost, s->stream));
    CUDA_TRY(s, fdtd::counted_copyAsync(s, pgobj.data(), s->hP.gobj, s->np, cudaMemcpyDeviceToHost, s->stream));
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    // dense (reference) order and indices
    std::vector<uint8_t> cls(s->ncell), gobj(s->ncell);
    {
        long long c = 0;
        for (int i = 0; i < s->N[0]; ++i)
            for (int j = 0; j < s->N[1]; ++j)
                for (int k = 0; k < s->N[2]; ++k, ++c) {
                    cls[c] = pcls[i * s->SX + j * s->SY + k];
                    gobj[c] = pgobj[i * s->SX + j * s->SY + k];
                }
    }
    const long long sx = (long long)s->N[1] * s->N[2];
    int64_t count = 0;
    const int64_t cap = (faces && n_faces) ? *n_faces : 0;
    for (long long c = 0; c < s->ncell; ++c) {
        const uint8_t code = cls[c];
        const bool bulk = code & CLS_BULK;
        const unsigned mask = code & CLS_MASK;
        const int i = (int)(c / sx), j = (int)((c / s->N[2]) % s->N[1]), k = (int)(c % s->N[2]);
        if (flags) flags[c] = cell_flags(s, code, gobj[c], i, j, k);
        if (bulk || !mask) continue;
        // faces in key order: neighbour flat index ascending (-x, -y, -z, +z, +y, +x)
        static const int od[6] = {0, 1, 2, 2, 1, 0};
        static const int os[6] = {-1, -1, -1, +1, +1, +1};
        const long long strides[3] = {sx, s->N[2], 1};
        for (int f = 0; f < 6; ++f) {
            if (!((mask >> (2 * od[f] + (os[f] > 0))) & 1u)) continue;
            if (count < cap) {
                fdtd_ghost_face& g = faces[count];
                std::memset(&g, 0, sizeof(g));
                g.owner_cell = (int32_t)c;
                g.neighbour_cell = (int32_t)(c + os[f] * strides[od[f]]);
                g.topology = os[f] * (od[f] + 1);
                g.type = (gobj[c] & GOBJ_CONSTRAINT) ? 1 : 0;
                const int o = gobj[c] & 0x7F;
                g.boundary_object = (o == GOBJ_NONE) ? -1 : o;
                g.key = szudzik(g.owner_cell, g.neighbour_cell);
            }
            ++count;
        }
    }
    if (n_faces) *n_faces = count;
    return FDTD_OK;
}

}  // extern "C"

namespace {

// Index into the compact z-slab arrays of the PML state (ShellBoxes::zbox) of
// the split pressure of cell (x, y, z) (dface < 0) or of its low face along
// dface; -1 when that element lives in the padded arrays.
long long zslab_index(const fdtd_solver* s, int dface, int x, int y, int z) {
    const ShellBoxes& B = s->shell;
    const int b = B.zbox, V = B.vz;
    if (s->hP.zcount <= 0 || b < 0) return -1;
    if (x < B.x0[b] || x >= B.x0[b] + B.nx[b] || y < B.y0[b] || y >= B.y0[b] + B.ny[b]) return -1;
    if (dface != 2 && z >= s->N[2]) return -1;
    auto slot = [&](int zz) -> long long {  // compact slot of the cell (or its low face) zz in the row
        if (zz >= B.za[b] && zz < B.zae[b]) return (long long)(zz / V - B.za[b] / V) * V + zz % V;
        if (zz >= B.zb[b] && zz < B.zbe[b]) return (long long)(B.gl[b] + zz / V - B.zb[b] / V) * V + zz % V;
        return -1;
    };
    long long q = slot(z);
    if (dface == 2 && q < 0 && z == B.zae[b] && z > 0) {
        // boundary face after the first range: high face of its last cell
        const long long qc = slot(z - 1);
        q = ((z - 1) % V != V - 1) ? qc + 1 : (long long)B.ng[b] * V;
    }
    if (q < 0) return -1;
    return ((long long)(x - B.x0[b]) * B.ny[b] + (y - B.y0[b])) * B.zrw + q;
}

// Where field `which` lies on the device: padded array, the compact z-slab array
// of the PML state (or null) and the extents of its dense form.  FP32 PRESSURE_PREV
// is p^n - d (d the compensated increment).
struct FieldPlace {
    void* src = nullptr;
    void* zsrc = nullptr;
    int ext[3] = {0, 0, 0};
    int dface = -1;
    bool fp32_prev = false;
};

fdtd_status field_place(fdtd_solver* s, int32_t which, int64_t count, FieldPlace& f) {
    const SolveParams& P = s->hP;
    const bool f64 = s->precision == FDTD_PRECISION_FP64;
    long long n = s->ncell;
    const int vbuf = s->opt.kernel == FDTD_KERNEL_PHASED ? 0 : s->cur;
    switch (which) {
        case FDTD_FIELD_PRESSURE: f.src = P.p[s->cur]; break;
        case FDTD_FIELD_PRESSURE_PREV: f.src = f64 ? P.p[s->cur ^ 1] : P.p[s->cur]; break;
        case FDTD_FIELD_PML_PX: case FDTD_FIELD_PML_PY: case FDTD_FIELD_PML_PZ: f.src = P.pd[which - FDTD_FIELD_PML_PX]; break;
        case FDTD_FIELD_VX: case FDTD_FIELD_VY: case FDTD_FIELD_VZ:
            f.src = P.v[vbuf][which - FDTD_FIELD_VX];
            n = s->vcount[which - FDTD_FIELD_VX];
            break;
        default: return (set_error(s, "unknown field"), FDTD_ERR_INVALID_ARG);
    }
    if (count != n) return (set_error(s, "count does not match the field size"), FDTD_ERR_INVALID_ARG);
    if (s->region.red && which >= FDTD_FIELD_PML_PX)
        return (set_error(s, "this FP32 solve keeps the reduced PML state (no split pressures or face velocities "
                             "along axes without absorption); create it with pml_state = FDTD_PML_STATE_FULL to "
                             "access them"),
                FDTD_ERR_UNSUPPORTED);
    for (int d = 0; d < 3; ++d) f.ext[d] = s->N[d];
    if (which >= FDTD_FIELD_VX) {
        f.dface = which - FDTD_FIELD_VX;
        f.ext[f.dface] += 1;
    }
    f.fp32_prev = !f64 && which == FDTD_FIELD_PRESSURE_PREV;
    if (P.zcount > 0 && which >= FDTD_FIELD_PML_PX)
        f.zsrc = which <= FDTD_FIELD_PML_PZ ? P.zpd[which - FDTD_FIELD_PML_PX] : P.zv[vbuf][which - FDTD_FIELD_VX];
    return FDTD_OK;
}

// A dense host array into a field (fdtd_solver_set_field).  Writing FP32
// PRESSURE_PREV sets d from the p^n already on the device, so write PRESSURE first.
fdtd_status field_write(fdtd_solver* s, int32_t which, const double* dense, int64_t count) {
    if (!s || !dense) return FDTD_ERR_INVALID_ARG;
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    const SolveParams& P = s->hP;
    FieldPlace f;
    const fdtd_status st = field_place(s, which, count, f);
    if (st != FDTD_OK) return st;
    const bool f64 = s->precision == FDTD_PRECISION_FP64;
    const size_t w = f64 ? 8 : 4;
    const long long np = s->np;
    std::vector<char> raw(np * w), zraw;
    std::vector<float> inc;
    CUDA_TRY(s, fdtd::counted_copyAsync(s, raw.data(), f.src, np * w, cudaMemcpyDeviceToHost, s->stream));
    if (f.fp32_prev) {
        inc.resize(np);
        CUDA_TRY(s, fdtd::counted_copyAsync(s, inc.data(), P.dinc, np * 4, cudaMemcpyDeviceToHost, s->stream));
    }
    // the z-slab box keeps its PML state in compact arrays (ShellBoxes)
    const ShellBoxes& B = s->shell;
    if (f.zsrc) {
        zraw.resize(P.zcount * w);
        CUDA_TRY(s, fdtd::counted_copyAsync(s, zraw.data(), f.zsrc, P.zcount * w, cudaMemcpyDeviceToHost, s->stream));
    }
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    double* r64 = (double*)raw.data();
    float* r32 = (float*)raw.data();
    long long o = 0;
    for (int i = 0; i < f.ext[0]; ++i)
        for (int j = 0; j < f.ext[1]; ++j)
            for (int k = 0; k < f.ext[2]; ++k, ++o) {
                const long long c = i * s->SX + j * s->SY + k;
                if (f64) r64[c] = dense[o];
                else if (f.fp32_prev) inc[c] = (float)((double)r32[c] - dense[o]);
                else r32[c] = (float)dense[o];
            }
    if (f.fp32_prev) {
        CUDA_TRY(s, fdtd::counted_copyAsync(s, P.dinc, inc.data(), np * 4, cudaMemcpyHostToDevice, s->stream));
    } else {
        if (f.zsrc) {
            // every (padded grid index, compact index) pair of the z-slab box
            const int b = B.zbox;
            for (int x = B.x0[b]; x < B.x0[b] + B.nx[b]; ++x)
                for (int y = B.y0[b]; y < B.y0[b] + B.ny[b]; ++y)
                    for (int z = 0; z <= s->N[2]; ++z) {
                        const long long q = zslab_index(s, f.dface, x, y, z);
                        if (q >= 0) std::memcpy(zraw.data() + q * w, raw.data() + (x * s->SX + y * s->SY + z) * w, w);
                    }
        }
        CUDA_TRY(s, fdtd::counted_copyAsync(s, f.src, raw.data(), np * w, cudaMemcpyHostToDevice, s->stream));
        if (f.zsrc)
            CUDA_TRY(s, fdtd::counted_copyAsync(s, f.zsrc, zraw.data(), P.zcount * w, cudaMemcpyHostToDevice, s->stream));
    }
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    return FDTD_OK;
}

// total items of item_bytes to out: launch(first, n, buffer) makes a chunk of them
// in the mapped host buffer given (enqueued on the solver stream), which is then
// copied out.  The device makes the chunks at the bus's rate; what takes long is
// the first touch of the caller's fresh memory (35 MB: 7.5 ms with one thread, 1.3
// with eight), so several threads take chunks in turn, each with its own buffer.
// The buffers are pinned memory of the kept blocks, no more than the solver's calls need,
// and given back with it: a 4 MiB allocation of its own, for one cell too, made the first
// view of every solver (field and slice of 192 x 160 x 144) 10.5 ms, now 4.7, and a
// first cell 2.5 to 6, now 0.05.  (Given back after each call, one block served all
// solvers, but the device writes slower to lines that a core has just read: with
// three solvers in turn a slice 1.4 ms instead of 1.1.)
template <typename Launch>
fdtd_status read_back(fdtd_solver* s, long long total, size_t item_bytes, void* out, Launch launch) {
    const long long chunk = (long long)(fdtd::READBACK_BYTES / item_bytes);
    const long long chunks = (total + chunk - 1) / chunk;
    const unsigned cores = std::thread::hardware_concurrency();
    const int workers = (int)std::min<long long>({chunks, (long long)fdtd::READBACK_WORKERS, cores ? (long long)cores : 1});
    if (workers < 1) return FDTD_OK;
    for (int w = 0; w < workers; ++w)
        if (!s->rb_done[w]) CUDA_TRY(s, cudaEventCreateWithFlags(&s->rb_done[w], cudaEventDisableTiming));
    // (powers of two, so that the kept blocks fit one another's calls)
    size_t each = (size_t)64 << 10;
    while (each < fdtd::READBACK_BYTES && each < (size_t)total * item_bytes) each *= 2;
    if (s->rb_bytes < (size_t)workers * each) {
        host_release(s->rb_stage, s->rb_bytes);
        s->rb_stage = nullptr;
        s->rb_bytes = 0;
        CUDA_TRY(s, host_acquire((size_t)workers * each, &s->rb_stage, &s->rb_bytes));
    }
    std::atomic<long long> next{0};
    std::atomic<int> failed{(int)cudaSuccess};
    auto work = [&](int w) {
        char* buf = (char*)s->rb_stage + (size_t)w * each;
        cudaError_t e = w > 0 ? cudaSetDevice(s->opt.device) : cudaSuccess;
        for (long long c; e == cudaSuccess && failed.load() == (int)cudaSuccess && (c = next.fetch_add(1)) < chunks;) {
            const long long first = c * chunk, n = std::min(chunk, total - first);
            e = launch(first, n, buf);
            if (e == cudaSuccess) e = cudaEventRecord(s->rb_done[w], s->stream);
            if (e == cudaSuccess) e = cudaEventSynchronize(s->rb_done[w]);
            if (e == cudaSuccess) std::memcpy((char*)out + (size_t)first * item_bytes, buf, (size_t)n * item_bytes);
        }
        int none = (int)cudaSuccess;
        if (e != cudaSuccess) failed.compare_exchange_strong(none, (int)e);
    };
    std::vector<std::thread> others;
    try {
        for (int w = 1; w < workers; ++w) others.emplace_back(work, w);
    } catch (const std::exception&) {
        // no thread to be had: the ones there are take all chunks
    }
    work(0);
    for (auto& t : others) t.join();
    if (failed.load() != (int)cudaSuccess) cudaStreamSynchronize(s->stream);  // nothing writes to the buffers any more
    CUDA_TRY(s, (cudaError_t)failed.load());
    fdtd::count_transfer(s, (size_t)total * item_bytes, cudaMemcpyDeviceToHost);
    return FDTD_OK;
}

// A field as a dense host array of doubles (fdtd_solver_get_field).
fdtd_status field_read(fdtd_solver* s, int32_t which, double* dense, int64_t count) {
    if (!s || !dense) return FDTD_ERR_INVALID_ARG;
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    FieldPlace f;
    const fdtd_status st = field_place(s, which, count, f);
    if (st != FDTD_OK) return st;
    const SolveParams& P = s->hP;
    FieldArgs F{};
    F.src = f.src;
    F.inc = f.fp32_prev ? P.dinc : nullptr;
    F.zsrc = f.zsrc;
    F.dface = f.dface;
    for (int d = 0; d < 3; ++d) {
        F.ext[d] = f.ext[d];
        F.N[d] = s->N[d];
    }
    F.SX = s->SX;
    F.SY = s->SY;
    F.shell = s->shell;
    return read_back(s, count, sizeof(double), dense, [&](long long first, long long n, void* buf) {
        return launch_field_dense(F, s->precision == FDTD_PRECISION_FP64, first, n, (double*)buf, s->stream);
    });
}

// MAC_Grid::GetCell (MAC_Grid.cpp:4182-4258) + the stored Laplacian of
// PML_WaveSolver::FetchCell (PML_WaveSolver.cpp:439-447): cell `cell` (dim < 0)
// or the `total` cells of plane k of axis dim, made by the device (k_fetch_cells).
fdtd_status fetch_cells(fdtd_solver* s, int dim, int k, long long cell, long long total, fdtd_cell* out) {
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    FetchArgs F{};
    F.dim = dim;
    F.k = k;
    F.cell = cell;
    F.step_index = s->step_index;
    F.pml_strength = s->pml_strength;
    F.reduced = s->region.red != 0;
    F.phased = s->opt.kernel == FDTD_KERNEL_PHASED;
    F.moving = s->moving;
    F.vbuf = F.phased ? 0 : s->cur;
    for (int d = 0; d < 3; ++d) F.csig[d] = s->d_csig[d];
    F.shell = s->shell;
    s->launches += (total + (long long)(fdtd::READBACK_BYTES / sizeof(fdtd_cell)) - 1) /
                   (long long)(fdtd::READBACK_BYTES / sizeof(fdtd_cell));
    return read_back(s, total, sizeof(fdtd_cell), out, [&](long long first, long long n, void* buf) {
        return launch_fetch_cells(s->dP, s->precision == FDTD_PRECISION_FP64, s->cur, F, first, (int)n, (fdtd_cell*)buf,
                                  s->stream);
    });
}

}  // namespace

extern "C" {

fdtd_status fdtd_solver_get_field(fdtd_solver* s, int32_t which, double* out, int64_t count) {
    // the read-back stages the field in host memory
    if (s && fdtd::inject_failure(FDTD_INJECT_HOST_ALLOC))
        return (set_error(s, "host staging buffer of the field read-back: allocation failed"), FDTD_ERR_OOM);
    return field_read(s, which, out, count);
}

fdtd_status fdtd_solver_set_field(fdtd_solver* s, int32_t which, const double* in, int64_t count) {
    return field_write(s, which, in, count);
}

fdtd_status fdtd_solver_domain(fdtd_solver* s, double min_bound[3], double max_bound[3]) {
    if (!s || !min_bound || !max_bound) return FDTD_ERR_INVALID_ARG;
    for (int d = 0; d < 3; ++d) {
        min_bound[d] = s->bmin[d];
        max_bound[d] = s->bmax[d];
    }
    return FDTD_OK;
}

fdtd_status fdtd_solver_fetch_cell(fdtd_solver* s, int64_t cell_index, fdtd_cell* out) {
    if (!s || !out) return FDTD_ERR_INVALID_ARG;
    if (cell_index < 0 || cell_index >= s->ncell)
        return (set_error(s, "cell_index out of range"), FDTD_ERR_INVALID_ARG);
    return fetch_cells(s, -1, 0, cell_index, 1, out);
}

fdtd_status fdtd_solver_sample_slice(fdtd_solver* s, int32_t dim, double offset, fdtd_cell* out, int64_t capacity,
                                     int64_t* count) {
    if (!s || !count) return FDTD_ERR_INVALID_ARG;
    if (dim < 0 || dim > 2) return (set_error(s, "dim must be 0, 1 or 2"), FDTD_ERR_INVALID_ARG);
    const int d1 = (dim + 1) % 3, d2 = (dim + 2) % 3;
    const int64_t n = (int64_t)s->N[d1] * s->N[d2];
    *count = n;
    if (!out) return FDTD_OK;
    if (capacity < n) return (set_error(s, "capacity below the slice's cell count"), FDTD_ERR_INVALID_ARG);
    // the face grid along dim starts half a cell below the cells (MAC_Grid.cpp:103-113)
    const double lower = s->bmin[dim] - s->h / 2.0;
    const double r = (offset - lower) / s->h;
    if (!(r > -1.0) || !(r < 2147483647.0))
        return (set_error(s, "offset outside the grid along dim"), FDTD_ERR_INVALID_ARG);
    const int k = std::min((int)r, s->N[dim] - 1);
    return fetch_cells(s, dim, k, 0, n, out);
}

// ---------------------------------------------------------------------------
// snapshot / restore (FDTD_AcousticSimulator::_SaveSimulationSnapshot, :381-415)
// ---------------------------------------------------------------------------
namespace {
struct SnapHeader {
    uint64_t magic;
    int64_t ncell;
    int32_t precision, kernel, cur, n_obj;
    int64_t step_index;
    double time, state_time;
    int64_t total;  // bytes, this header's too
};
// The regions are raw copies, so a change of what they hold (StepConsts, HostObject, the
// arrays of a solve) is another layout and takes another number.
const uint64_t SNAP_MAGIC = 0x324e53445446ULL;  // "FTDSN2"

size_t snap_total(fdtd_solver* s, const std::vector<std::pair<void*, size_t>>& regs) {
    size_t total = sizeof(SnapHeader) + s->objs.size() * sizeof(HostObject);
    for (const auto& r : regs) total += r.second;
    return total;
}

std::vector<std::pair<void*, size_t>> snap_regions(fdtd_solver* s) {
    const SolveParams& P = s->hP;
    const size_t w = s->precision == FDTD_PRECISION_FP64 ? 8 : 4;
    std::vector<std::pair<void*, size_t>> r;
    const size_t np = (size_t)s->np;  // the padded arrays as they are
    r.push_back({P.p[0], np * w});
    r.push_back({P.p[1], np * w});
    if (P.dinc) r.push_back({P.dinc, np * 4});
    for (int d = 0; d < 3; ++d) r.push_back({P.pd[d], np * w});
    for (int b = 0; b < 2; ++b)
        for (int d = 0; d < 3; ++d)
            if (P.v[b][d]) r.push_back({P.v[b][d], np * w});
    r.push_back({P.cls, np});
    r.push_back({P.gobj, np});
    if (P.zcount > 0)
        for (int d = 0; d < 3; ++d) {
            r.push_back({P.zpd[d], (size_t)P.zcount * w});
            r.push_back({P.zv[0][d], (size_t)P.zcount * w});
            r.push_back({P.zv[1][d], (size_t)P.zcount * w});
        }
    for (int b = 0; b < 2; ++b)
        if (P.lapv[b]) r.push_back({P.lapv[b], np * (s->precision == FDTD_PRECISION_FP64 ? 8 : 4)});
    if (P.eng_buf) r.push_back({P.eng_buf, s->eng.size() * ENG_BUF * 8});
    r.push_back({P.consts, 2 * sizeof(StepConsts)});
    r.push_back({P.dev_error, sizeof(int)});
    return r;
}
}  // namespace

}  // extern "C"

namespace fdtd {
// Moving bodies that stay two cells clear of the PML at every step of
// [start_time, end_time]: the per-step classification boxes of the whole run,
// posed and unioned as the step driver does, are checked on the host.  Then no
// PML cell is ever solid or next to a solid, and the reduced PML state is exact.
bool moving_clear_of_pml(fdtd_solver* s) {
    if (!s->moving || !(s->end_time > s->start_time) || !(s->k > 0)) return false;
    const double nsteps = std::ceil((s->end_time - s->start_time) / s->k) + 2.0;
    if (nsteps > 2.0e7) return false;
    std::vector<HostObject> objs = s->objs;
    double t = s->start_time;
    for (auto& o : objs) {
        host_object_pose(o, t);
        host_update_bbox(o);
        host_reset_union(o);
    }
    bool clear = true;
    std::swap(s->objs, objs);  // classification_boxes reads s->objs
    ClsBoxes B;
    for (long long i = 0; i <= (long long)nsteps && clear; ++i) {
        if (i > 0) {
            t += s->k;
            for (auto& o : s->objs) {
                if (o.d.motion == FDTD_MOTION_STATIC) continue;
                host_object_pose(o, t);
                host_update_bbox(o);
            }
        }
        classification_boxes(s, B);
        clear = boxes_clear_of_shell(s, B);
    }
    std::swap(s->objs, objs);
    return clear;
}

// Listener plans (fixed MLS weights) and ghost-cell plans of a static solve from
// its current classification, as its first step builds them; used after a restore.
fdtd_status rebuild_listener_plans(fdtd_solver* s) {
    if (s->moving) return FDTD_OK;
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    const fdtd_status st = static_prep(s, s->cur);
    if (st != FDTD_OK) return st;
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    return FDTD_OK;
}
}  // namespace fdtd

extern "C" {

fdtd_status fdtd_solver_snapshot(fdtd_solver* s, void* buffer, int64_t* bytes) {
    if (!s || !bytes) return FDTD_ERR_INVALID_ARG;
    auto regs = snap_regions(s);
    const size_t total = snap_total(s, regs);
    if (!buffer) {
        *bytes = (int64_t)total;
        return FDTD_OK;
    }
    if (*bytes < (int64_t)total) return (set_error(s, "snapshot buffer too small"), FDTD_ERR_INVALID_ARG);
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    SnapHeader h{SNAP_MAGIC, s->ncell, s->precision, s->opt.kernel, s->cur, (int32_t)s->objs.size(),
                 s->step_index, s->time, s->state_time, (int64_t)total};
    char* p = (char*)buffer;
    std::memcpy(p, &h, sizeof(h));
    p += sizeof(h);
    std::memcpy(p, s->objs.data(), s->objs.size() * sizeof(HostObject));
    p += s->objs.size() * sizeof(HostObject);
    for (auto& r : regs) {
        CUDA_TRY(s, fdtd::counted_copyAsync(s, p, r.first, r.second, cudaMemcpyDeviceToHost, s->stream));
        p += r.second;
    }
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    *bytes = (int64_t)total;
    return FDTD_OK;
}

fdtd_status fdtd_solver_restore(fdtd_solver* s, const void* buffer, int64_t bytes) {
    if (!s || !buffer) return FDTD_ERR_INVALID_ARG;
    SnapHeader h;
    if (bytes < (int64_t)sizeof(h)) return (set_error(s, "snapshot truncated"), FDTD_ERR_INVALID_ARG);
    std::memcpy(&h, buffer, sizeof(h));
    auto regs = snap_regions(s);
    const size_t total = snap_total(s, regs);
    if (h.magic != SNAP_MAGIC || h.ncell != s->ncell || h.precision != s->precision || h.kernel != s->opt.kernel ||
        h.n_obj != (int32_t)s->objs.size() || h.total != (int64_t)total)
        return (set_error(s, "snapshot does not match this solver"), FDTD_ERR_INVALID_ARG);
    if (bytes < (int64_t)total) return (set_error(s, "snapshot truncated"), FDTD_ERR_INVALID_ARG);
    CUDA_TRY(s, cudaSetDevice(s->opt.device));
    CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    const char* p = (const char*)buffer + sizeof(h);
    // the pose state comes from the snapshot; what points into this solver's own
    // storage (device meshes, keyframe tracks, mesh vertices) stays this solver's
    const std::vector<HostObject> own = s->objs;
    std::memcpy(s->objs.data(), p, s->objs.size() * sizeof(HostObject));
    for (size_t i = 0; i < s->objs.size(); ++i) {
        s->objs[i].mview = own[i].mview;
        s->objs[i].kf = own[i].kf;
        s->objs[i].mv = own[i].mv;
    }
    p += s->objs.size() * sizeof(HostObject);
    for (auto& r : regs) {
        CUDA_TRY(s, fdtd::counted_copy(s, r.first, p, r.second, cudaMemcpyHostToDevice));
        p += r.second;
    }
    s->cur = h.cur;
    s->step_index = h.step_index;
    s->time = h.time;
    s->state_time = h.state_time;
    s->cls_boxes_current = false;  // the flags came from the snapshot, not from hP.boxes
    to_dev_objects(s);
    CUDA_TRY(s, fdtd::counted_copy(s, s->dP, &s->hP, sizeof(SolveParams), cudaMemcpyHostToDevice));
    // the fixed listener weights of the restored classification (a first step
    // classifies and derives them itself)
    if (s->step_index > 0) return rebuild_listener_plans(s);
    return FDTD_OK;
}

}  // extern "C"
