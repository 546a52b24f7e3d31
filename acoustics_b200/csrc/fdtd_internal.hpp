// fdtd_internal.hpp — host-side state of one solver handle.
#pragma once
#include <cuda_runtime.h>

#include <array>
#include <functional>
#include <string>
#include <vector>

#include "../../include/fdtd_c.h"
#include "fdtd_device.cuh"
#include "fdtd_tma.hpp"

namespace fdtd {

constexpr size_t READBACK_BYTES = (size_t)512 << 10;
constexpr int READBACK_WORKERS = 8;

struct HostObject {
    fdtd_object_desc d;
    double c[3] = {0, 0, 0};
    double bmin[3] = {0, 0, 0}, bmax[3] = {0, 0, 0};  // _bboxWorld
    double umin[3] = {0, 0, 0}, umax[3] = {0, 0, 0};  // _bboxWorldUnion2Steps
    double mlo[3] = {0, 0, 0}, mhi[3] = {0, 0, 0};    // mesh: extent of rotation * v about the centre
    MeshView mview{};                                 // mesh: device hierarchy and triangles
    // FDTD_MOTION_KEYFRAMED: the track (solver-owned frames) and the rest rotation it turns
    const double* kf = nullptr;
    int kf_n = 0;
    double kf_step = 0;
    double R0[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    // meshes: object-frame vertices (solver-owned) for the extent of a turned mesh
    const double* mv = nullptr;
    int mv_n = 0;
};

// A validated mesh with its pseudo-normals and hierarchy (fdtd_mesh.cpp).
struct MeshHost {
    std::vector<MeshNode> nodes;
    std::vector<MeshTri> tris;  // leaf order
    std::vector<int> top;       // MeshView::top
    std::vector<double> vertices;
    double edge = 0;            // longest edge
    bool solid = false;         // MeshView::solid
};
bool build_mesh(const fdtd_mesh_desc& md, MeshHost& out, std::string& err);
// MeshView::solid of a mesh that build_mesh made of md; false where in doubt
bool mesh_bounds_solid(const fdtd_mesh_desc& md, const MeshHost& M);
void mesh_extent(const double* verts, size_t nv, const double R[9], double lo[3], double hi[3]);
// A host object of scene object i at rest (mesh extent set; pose and box not yet).
HostObject make_host_object(const fdtd_scene_desc* sc, int i);
bool read_obj(const char* path, double scale, std::vector<double>& verts, std::vector<int32_t>& tris, std::string& err);

struct AxisTables {
    std::vector<uint8_t> pml_cell, pml_face;
    std::vector<double> cpos, fpos, pupd, pdiv, vupd, vgrad;
    std::vector<double> csig;  // absorption coefficient at the cell centres
};

void host_object_pose(HostObject& o, double t);
// keyframed pose at time t: centre and the rotation that turns the rest pose (fdtd_kinematics.cpp)
void keyframe_pose(const double* frames, int n, double step, double t, double com[3], double R[9]);
bool read_kinematics(const char* path, std::vector<double>& frames, std::string& err);
void host_update_bbox(HostObject& o);
void host_reset_union(HostObject& o);

}  // namespace fdtd

struct fdtd_solver {
    fdtd_options opt{};
    int precision = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t stream2 = nullptr;   // second stream: interior kernel concurrent with the shell
    cudaStream_t stream3 = nullptr;   // third stream: ghost-cell list beside the interior
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_ghost = nullptr;
    // listener rows of step n run on stream4 beside step n+1; step n+2, which
    // overwrites the pressure they read, waits on ev_lis[parity of step n]
    cudaStream_t stream4 = nullptr;
    cudaEvent_t ev_step = nullptr, ev_lis[2] = {nullptr, nullptr}, ev_lis_join = nullptr;
    bool lis_pending[2] = {false, false};
    // moving bodies clear of the PML: the shell kernel of a step runs on stream5
    // beside that step's classification
    cudaStream_t stream5 = nullptr;
    cudaEvent_t ev_sfork = nullptr, ev_sdone = nullptr;
    // and the interior planes out of the bodies' reach on stream6 (planes_ahead)
    cudaStream_t stream6 = nullptr;
    cudaEvent_t ev_fdone = nullptr;
    // hP.boxes are the boxes of the classification the cell flags hold (the
    // solid cells lie in them); cleared when the flags are loaded from elsewhere
    bool cls_boxes_current = false;
    std::vector<fdtd::HostObject> cls_objs;  // moving scenes: the bodies as that classification found them
    // FP64, made when first needed: p^{n-1} for fits that may lie in the PML, whose shell
    // starts ahead and writes over it
    double* held = nullptr;
    cudaEvent_t ev_held = nullptr;
    bool lis_clear = false;         // listeners_clear_of the boxes of the last reset
    long long overlapped_steps = 0;
    // geometry
    double h = 0, c = 0, rho = 0, k = 0, end_time = 0, start_time = 0;
    double pml_strength = 0;
    int N[3] = {0, 0, 0};
    long long ncell = 0, n_pml = 0, n_interior = 0;
    long long SX = 0, SY = 0, np = 0;  // padded strides and elements per device array
    long long vcount[3] = {0, 0, 0};
    double bmin[3] = {0, 0, 0}, bmax[3] = {0, 0, 0};
    fdtd::AxisTables tab[3];
    std::vector<fdtd::HostObject> objs;
    std::vector<fdtd::MeshHost> meshes;     // the scene's meshes (those objects use)
    std::vector<std::vector<double>> kf_store;  // keyframe tracks of the objects (empty: none)
    std::vector<void*> mesh_alloc;          // their device copies
    std::vector<fdtd_plane_desc> planes;
    std::vector<fdtd_gaussian_source_desc> sources;
    std::vector<double> listeners;
    int L = 0;
    bool moving = false;
    int preset = 0;                 // boundary_condition_preset
    std::vector<fdtd::EngCell> eng;  // Engquist-Majda cells (sides without PML)
    int boundary_handling = 0;              // FDTD_BOUNDARY_*
    std::vector<void*> fc_alloc;            // device arrays of the FULLY_COUPLED rows
    long long fc_immersed = 0, fc_fallback = 0;
    // device
    fdtd::SolveParams hP{};
    fdtd::SolveParams* dP = nullptr;
    void* arena = nullptr;
    size_t arena_bytes = 0;
    size_t arena_block = 0;         // bytes of the device block holding the arena (>= its carve)
    int* d_solid_pml = nullptr;
    int n_solid_pml = 0;
    double* d_lap = nullptr;
    int* d_status = nullptr;
    double* d_lis = nullptr;
    double* h_lis_stage = nullptr;  // (pinned; followed by h_status)
    size_t h_lis_bytes = 0;
    int main_priority = 0, side_priority = 0;  // of stream; of stream2 and stream3
    int* h_status = nullptr;         // host side of what a call reads at its end: dev_error ... d_ghost_count
    int lis_cap_steps = 0;
    int xb = 4;                       // planes per thread of the interior kernel
    fdtd::Box3 interior{};            // non-PML box
    fdtd::ShellBoxes shell{};         // PML shell boxes
    fdtd::RegionLaunch region{};      // launch description of the region-split step
    // one-launch steps: the listener row of the last step, written by the next
    // step's launch (or by flush_lag), and the cells of the ghost list once known
    double* lag_row = nullptr;
    int n_ghost = -1;
    int* d_ghost_list = nullptr;
    int* d_ghost_count = nullptr;
    // stepping state
    int cur = 0;
    long long step_index = 0;
    double time = 0.0;        // simulation time of the next step (host mirror of the device clock)
    double state_time = 0.0;  // SimWorld::_state.time for object animation
    bool classified_after_first_step = false;
    cudaGraphExec_t graph_exec[4] = {nullptr, nullptr, nullptr, nullptr};  // [parity + 2*sources]
    long long launches = 0;
    long long last_launches = 0;
    long long graph_launches_per_exec = 0;
    fdtd::TmaStep* tma = nullptr;     // tiles and tensor maps of the TMA-staged shell (reduced state)
    // read-backs (fields, cells): pinned staging as large as any so far needed, a part
    // and an event per worker
    void* rb_stage = nullptr;
    size_t rb_bytes = 0;
    cudaEvent_t rb_done[fdtd::READBACK_WORKERS] = {};
    const double* d_csig[3] = {nullptr, nullptr, nullptr};  // absorption at the cell centres
    // bytes this handle copied between host and device memory since creation
    long long bytes_h2d = 0, bytes_d2h = 0;
    std::string err;
};

namespace fdtd {
// Host<->device copies of a solver handle, added to its transfer totals
// (fdtd_solver_transfer_bytes); s may be NULL.
inline void count_transfer(fdtd_solver* s, size_t n, cudaMemcpyKind kind) {
    if (!s) return;
    if (kind == cudaMemcpyHostToDevice) s->bytes_h2d += (long long)n;
    else if (kind == cudaMemcpyDeviceToHost) s->bytes_d2h += (long long)n;
}
// A copy in the order of the solver's stream, done on return.  (The default stream
// orders nothing before kernels on non-blocking streams: cudaMemcpy from pageable
// memory may return before the device has the data, and cudaMemset always.)
inline cudaError_t counted_copy(fdtd_solver* s, void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
    count_transfer(s, n, kind);
    const cudaError_t e = cudaMemcpyAsync(dst, src, n, kind, s->stream);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s->stream);
}
inline cudaError_t counted_copyAsync(fdtd_solver* s, void* dst, const void* src, size_t n, cudaMemcpyKind kind,
                                     cudaStream_t stream) {
    count_transfer(s, n, kind);
    return cudaMemcpyAsync(dst, src, n, kind, stream);
}
// bytes of the arena from the error flags to the list lengths (carve_arena)
inline size_t status_bytes(const fdtd_solver* s) {
    return (size_t)((const char*)(s->d_ghost_count + 4) - (const char*)s->hP.dev_error);
}
void set_error(fdtd_solver* s, const std::string& msg);
inline ClsMeshes cls_meshes(const fdtd_solver* s) {
    ClsMeshes k = CLS_MESHES_NONE;
    for (const MeshHost& m : s->meshes)
        if (!m.tris.empty()) k = m.solid && k != CLS_MESHES_LOOSE ? CLS_MESHES_SOLID : CLS_MESHES_LOOSE;
    return k;
}
// no listener stencil meets a classification box (fdtd_step.cpp)
bool listeners_clear_of(const fdtd_solver* s, const ClsBoxes& B);
// moving bodies two cells clear of the PML through [start_time, end_time]
bool moving_clear_of_pml(fdtd_solver* s);
// A batch member made outside the batch: its solver created and its first step
// run (or its snapshot restored), ready to be placed between two batched steps
// (fdtd_batch.cpp).  batch_prepare touches no batch state, so a server prepares
// members on another host thread while its batch steps.
struct PreparedMember {
    fdtd_solver* s = nullptr;
    int64_t total = 0, done = 0;
    std::vector<double> rows;
};
fdtd_status batch_prepare(const fdtd_options& batch_opt, const fdtd_scene_desc* scene, int32_t steps_total,
                          const void* snapshot, int64_t snapshot_bytes, const double* rows, int64_t steps_done,
                          PreparedMember* out, std::string* err, const std::function<void()>& on_memory = nullptr);
// fdtd_solver_create; on_memory is called as soon as the solver holds its device block
fdtd_status solver_create(const fdtd_scene_desc* sc, const fdtd_options* opt, fdtd_solver** out,
                          const std::function<void()>& on_memory);
int32_t batch_place(fdtd_batch* b, PreparedMember&& pm);
// Device blocks for solver arenas, kept after a solver is destroyed for the next
// one on the same device (fdtd_api.cpp)
cudaError_t arena_acquire(int device, size_t bytes, void** ptr, size_t* block_bytes);
void arena_release(int device, void* ptr, size_t block_bytes);
cudaError_t stream_acquire(int device, int priority, cudaStream_t* out);
void stream_release(int device, int priority, cudaStream_t st);
cudaError_t host_acquire(size_t bytes, void** ptr, size_t* block_bytes);
void host_release(void* ptr, size_t block_bytes);
// listener plans of a static solve from its current classification (after a restore)
fdtd_status rebuild_listener_plans(fdtd_solver* s);
// fdtd_debug_inject_failure: true when this allocation of kind `what` is to fail
bool inject_failure(int what);
// TMA-staged PML shell (fdtd_tma.cpp)
bool tma_encoder_available();
fdtd_status build_shell_tma(fdtd_solver* s);
void free_shell_tma(fdtd_solver* s);
fdtd_status solver_init_geometry(fdtd_solver* s, const fdtd_scene_desc* sc);
void classification_boxes(const fdtd_solver* s, ClsBoxes& B);
void to_dev_objects(fdtd_solver* s);
fdtd_status build_fully_coupled(fdtd_solver* s);
void free_fully_coupled(fdtd_solver* s);
}  // namespace fdtd
