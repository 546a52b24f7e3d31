// fdtd_mesh.cpp — host side of triangle-mesh bodies: validation of a mesh
// (closed and consistently oriented, as the reference's signed distance field
// requires, AdaptiveDistanceField.cpp:92-96), pseudo-normals of faces, edges
// and vertices [Baerentzen 2002], the bounding-volume hierarchy the device
// queries walk (fdtd_mesh.cuh), and the Wavefront .obj reader
// (MeshObjReader::read with a scale, FDTD_RigidObject.cpp:84-93).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <map>
#include <sstream>
#include <string>
#include <utility>
#include <vector>

#include "../../include/fdtd_c.h"
#include "fdtd_internal.hpp"

namespace fdtd {

namespace {

void sub3(const double* a, const double* b, double* r) {
    for (int i = 0; i < 3; ++i) r[i] = a[i] - b[i];
}
void cross3(const double* a, const double* b, double* r) {
    r[0] = a[1] * b[2] - a[2] * b[1];
    r[1] = a[2] * b[0] - a[0] * b[2];
    r[2] = a[0] * b[1] - a[1] * b[0];
}
double dot3(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
double norm3(const double* a) { return std::sqrt(dot3(a, a)); }

struct Builder {
    const std::vector<MeshTri>* all;
    std::vector<int> order;
    std::vector<MeshNode> nodes;
    int max_depth = 0;

    void bounds(int lo, int hi, double* mn, double* mx) const {
        for (int d = 0; d < 3; ++d) {
            mn[d] = HUGE_VAL;
            mx[d] = -HUGE_VAL;
        }
        for (int k = lo; k < hi; ++k) {
            const MeshTri& t = (*all)[order[k]];
            for (int v = 0; v < 3; ++v)
                for (int d = 0; d < 3; ++d) {
                    mn[d] = std::min(mn[d], t.p[v][d]);
                    mx[d] = std::max(mx[d], t.p[v][d]);
                }
        }
    }

    // node `at` covers order[lo, hi)
    void build(int at, int lo, int hi, int depth) {
        max_depth = std::max(max_depth, depth);
        double mn[3], mx[3];
        bounds(lo, hi, mn, mx);
        // widen the box a little: a triangle's rounded distance is then never below its box's
        double ext = 0.0;
        for (int d = 0; d < 3; ++d) ext = std::max(ext, mx[d] - mn[d]);
        for (int d = 0; d < 3; ++d) {
            const double pad = 1e-9 * (ext + std::max(std::fabs(mn[d]), std::fabs(mx[d])));
            nodes[at].lo[d] = mn[d] - pad;
            nodes[at].hi[d] = mx[d] + pad;
        }
        if (hi - lo <= 4 || depth >= 48) {
            nodes[at].first = lo;
            nodes[at].count = hi - lo;
            return;
        }
        // median split of the centroids along the widest centroid extent
        double cmn[3] = {HUGE_VAL, HUGE_VAL, HUGE_VAL}, cmx[3] = {-HUGE_VAL, -HUGE_VAL, -HUGE_VAL};
        auto centroid = [&](int t, int d) {
            const MeshTri& T = (*all)[t];
            return (T.p[0][d] + T.p[1][d] + T.p[2][d]) / 3.0;
        };
        for (int k = lo; k < hi; ++k)
            for (int d = 0; d < 3; ++d) {
                cmn[d] = std::min(cmn[d], centroid(order[k], d));
                cmx[d] = std::max(cmx[d], centroid(order[k], d));
            }
        int axis = 0;
        for (int d = 1; d < 3; ++d)
            if (cmx[d] - cmn[d] > cmx[axis] - cmn[axis]) axis = d;
        const int mid = (lo + hi) / 2;
        std::nth_element(order.begin() + lo, order.begin() + mid, order.begin() + hi, [&](int a, int b) {
            const double ca = centroid(a, axis), cb = centroid(b, axis);
            return ca < cb || (ca == cb && a < b);
        });
        const int left = (int)nodes.size();
        nodes.resize(nodes.size() + 2);
        nodes[at].first = left;
        nodes[at].count = 0;
        build(left, lo, mid, depth + 1);
        build(left + 1, mid, hi, depth + 1);
    }
};

}  // namespace

bool build_mesh(const fdtd_mesh_desc& md, MeshHost& out, std::string& err) {
    const int nv = md.n_vertices, nt = md.n_triangles;
    if (nv < 4 || nt < 4 || !md.vertices || !md.triangles) {
        err = "mesh: at least 4 vertices and 4 triangles are needed";
        return false;
    }
    for (int i = 0; i < 3 * nv; ++i)
        if (!std::isfinite(md.vertices[i])) {
            err = "mesh: non-finite vertex coordinate";
            return false;
        }
    std::vector<MeshTri> tris(nt);
    std::map<std::pair<int, int>, std::vector<std::pair<int, int>>> edges;  // (a, b) directed -> (tri, local edge)
    for (int t = 0; t < nt; ++t) {
        MeshTri& T = tris[t];
        std::memset(&T, 0, sizeof(T));
        T.id = t;
        int v[3];
        for (int k = 0; k < 3; ++k) {
            v[k] = md.triangles[3 * t + k];
            if (v[k] < 0 || v[k] >= nv) {
                err = "mesh: triangle " + std::to_string(t) + " has a vertex index out of range";
                return false;
            }
            for (int d = 0; d < 3; ++d) T.p[k][d] = md.vertices[3 * v[k] + d];
        }
        if (v[0] == v[1] || v[1] == v[2] || v[0] == v[2]) {
            err = "mesh: triangle " + std::to_string(t) + " repeats a vertex";
            return false;
        }
        double e1[3], e2[3], n[3];
        sub3(T.p[1], T.p[0], e1);
        sub3(T.p[2], T.p[0], e2);
        cross3(e1, e2, n);
        const double ln = norm3(n);
        if (!(ln > 0.0)) {
            err = "mesh: triangle " + std::to_string(t) + " has zero area";
            return false;
        }
        for (int d = 0; d < 3; ++d) T.nf[d] = n[d] / ln;
        for (int k = 0; k < 3; ++k) edges[{v[k], v[(k + 1) % 3]}].push_back({t, k});
    }
    // closed and consistently oriented: each directed edge once, its reverse once
    for (const auto& e : edges) {
        if (e.second.size() != 1) {
            err = "mesh: an edge is used twice in the same direction (inconsistent orientation or non-manifold)";
            return false;
        }
        const auto r = edges.find({e.first.second, e.first.first});
        if (r == edges.end()) {
            err = "mesh has a boundary (an edge with one triangle); a closed surface is required";
            return false;
        }
        const int t = e.second[0].first, k = e.second[0].second, u = r->second[0].first;
        for (int d = 0; d < 3; ++d) tris[t].ne[k][d] = tris[t].nf[d] + tris[u].nf[d];
    }
    // vertices: sum of the incident unit face normals weighted by the incident angle
    std::vector<double> vn(3 * (size_t)nv, 0.0);
    for (int t = 0; t < nt; ++t) {
        for (int k = 0; k < 3; ++k) {
            const double* p = tris[t].p[k];
            double a[3], b[3];
            sub3(tris[t].p[(k + 1) % 3], p, a);
            sub3(tris[t].p[(k + 2) % 3], p, b);
            double c = dot3(a, b) / (norm3(a) * norm3(b));
            c = std::max(-1.0, std::min(1.0, c));
            const double ang = std::acos(c);
            const int v = md.triangles[3 * t + k];
            for (int d = 0; d < 3; ++d) vn[3 * v + d] += ang * tris[t].nf[d];
        }
    }
    for (int t = 0; t < nt; ++t)
        for (int k = 0; k < 3; ++k) {
            const int v = md.triangles[3 * t + k];
            for (int d = 0; d < 3; ++d) tris[t].nv[k][d] = vn[3 * v + d];
        }
    // hierarchy
    Builder B;
    B.all = &tris;
    B.order.resize(nt);
    for (int t = 0; t < nt; ++t) B.order[t] = t;
    B.nodes.resize(1);
    B.build(0, 0, nt, 0);
    if (B.max_depth + 2 >= MESH_STACK) {
        err = "mesh: hierarchy too deep";
        return false;
    }
    out.nodes = B.nodes;
    // the nodes five levels down, with the leaves above them
    out.top.assign(1, 0);
    for (int level = 0; level < 5; ++level) {
        std::vector<int> next;
        for (int n : out.top) {
            if (out.nodes[n].count > 0) {
                next.push_back(n);
            } else {
                next.push_back(out.nodes[n].first);
                next.push_back(out.nodes[n].first + 1);
            }
        }
        out.top.swap(next);
    }
    out.tris.resize(nt);
    for (int k = 0; k < nt; ++k) out.tris[k] = tris[B.order[k]];
    out.edge = 0.0;
    for (const MeshTri& T : tris)
        for (int k = 0; k < 3; ++k) {
            double e[3];
            sub3(T.p[(k + 1) % 3], T.p[k], e);
            out.edge = std::max(out.edge, norm3(e));
        }
    out.vertices.assign(md.vertices, md.vertices + 3 * (size_t)nv);
    return true;
}

namespace {

struct Corners {
    const double* p[3];
    const int32_t* v;  // vertex indices
};

void unit3(const double* a, double* r) {
    const double n = norm3(a);
    for (int i = 0; i < 3; ++i) r[i] = n > 0.0 ? a[i] / n : 0.0;
}

// Triangles without a common vertex: some axis (the normals, the cross products of
// their edges, and in a common plane the edges' normals) shows a gap of more than eps.
bool apart(const Corners& A, const Corners& B, double eps) {
    double ea[3][3], eb[3][3], na[3], nb[3];
    for (int i = 0; i < 3; ++i) {
        sub3(A.p[(i + 1) % 3], A.p[i], ea[i]);
        sub3(B.p[(i + 1) % 3], B.p[i], eb[i]);
    }
    cross3(ea[0], ea[1], na);
    cross3(eb[0], eb[1], nb);
    auto gap = [&](const double* axis) {
        double a[2] = {HUGE_VAL, -HUGE_VAL}, b[2] = {HUGE_VAL, -HUGE_VAL}, u[3];
        unit3(axis, u);
        for (int i = 0; i < 3; ++i) {
            const double x = dot3(u, A.p[i]), y = dot3(u, B.p[i]);
            a[0] = std::min(a[0], x), a[1] = std::max(a[1], x);
            b[0] = std::min(b[0], y), b[1] = std::max(b[1], y);
        }
        return b[0] - a[1] > eps || a[0] - b[1] > eps;
    };
    if (gap(na) || gap(nb)) return true;
    double x[3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            cross3(ea[i], eb[j], x);
            if (gap(x)) return true;
        }
    for (int i = 0; i < 3; ++i) {
        cross3(na, ea[i], x);
        if (gap(x)) return true;
        cross3(nb, eb[i], x);
        if (gap(x)) return true;
    }
    return false;
}

// Sines of angles: below the first a direction lies in a plane but for rounding,
// above the second it does not.
constexpr double IN_PLANE = 1e-12, OFF_PLANE = 1e-8;

// Triangles with one common vertex (corner i of A, j of B) and no other point in
// common: some plane through it has A's other corners on one side and B's on the
// other, with at most one of each in it, on different rays.
bool only_corner(const Corners& A, int i, const Corners& B, int j) {
    double d[2][2][3], n[2][3];  // unit directions from the corner, normals
    for (int k = 0; k < 2; ++k) {
        double e[3];
        sub3(A.p[(i + 1 + k) % 3], A.p[i], e);
        unit3(e, d[0][k]);
        sub3(B.p[(j + 1 + k) % 3], B.p[j], e);
        unit3(e, d[1][k]);
    }
    for (int q = 0; q < 2; ++q) cross3(d[q][0], d[q][1], n[q]);
    auto plane = [&](const double* normal) {
        double u[3], s[2][2];
        if (!(norm3(normal) > OFF_PLANE)) return false;
        unit3(normal, u);
        for (int q = 0; q < 2; ++q)
            for (int k = 0; k < 2; ++k) s[q][k] = dot3(u, d[q][k]);
        for (int q = 0; q < 2; ++q)          // the triangle strictly on one side (but for one ray)
            for (int sg = -1; sg <= 1; sg += 2) {
                const double *f = s[q], *g = s[q ^ 1];
                const bool other = sg * g[0] <= IN_PLANE && sg * g[1] <= IN_PLANE;  // the other one on the other
                if (!other) continue;
                if (sg * f[0] > OFF_PLANE && sg * f[1] > OFF_PLANE) return true;
                for (int k = 0; k < 2; ++k) {
                    if (!(sg * f[k ^ 1] > OFF_PLANE && std::fabs(f[k]) <= IN_PLANE)) continue;
                    // ray k of this one in the plane: the other's there, one at most, elsewhere
                    bool clear = true;
                    for (int m = 0; m < 2; ++m) {
                        if (sg * g[m] < -OFF_PLANE) continue;
                        double x[3];
                        cross3(d[q][k], d[q ^ 1][m], x);
                        const bool same = dot3(d[q][k], d[q ^ 1][m]) > 0.0 && !(norm3(x) > OFF_PLANE);
                        const bool between = sg * g[m ^ 1] >= -OFF_PLANE;  // a sector in the plane
                        clear = clear && !same && !between;
                    }
                    if (clear) return true;
                }
            }
        return false;
    };
    if (plane(n[0]) || plane(n[1])) return true;
    double x[3];
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b) {
            cross3(d[0][a], d[1][b], x);
            if (plane(x)) return true;
        }
    for (int q = 0; q < 2; ++q)
        for (int k = 0; k < 2; ++k) {
            cross3(n[q], d[q][k], x);
            if (plane(x)) return true;
        }
    return false;
}

// Triangles with a common edge p q, not folded onto one another (x, y: the third corners).
bool only_edge(const double* p, const double* q, const double* x, const double* y) {
    double e[3], u[3], f[2][3];
    sub3(q, p, e);
    unit3(e, u);
    const double* c[2] = {x, y};
    for (int k = 0; k < 2; ++k) {
        double r[3];
        sub3(c[k], p, r);
        const double a = dot3(r, u);
        for (int d = 0; d < 3; ++d) r[d] -= a * u[d];
        unit3(r, f[k]);
    }
    double z[3];
    cross3(f[0], f[1], z);
    return dot3(f[0], f[1]) < 0.0 || norm3(z) > 1e-6;
}

// The two triangles share their common vertices or edge only.
bool only_shared(const Corners& A, const Corners& B, double eps) {
    int n = 0, ia[3], ib[3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            if (A.v[i] == B.v[j] && n < 3) {
                ia[n] = i;
                ib[n++] = j;
            }
    if (n == 0) return apart(A, B, eps);
    if (n == 1) return only_corner(A, ia[0], B, ib[0]);
    if (n == 2) return only_edge(A.p[ia[0]], A.p[ia[1]], A.p[3 - ia[0] - ia[1]], B.p[3 - ib[0] - ib[1]]);
    return false;
}

}  // namespace

// The sign of a mesh's distance, read from the nearest feature's pseudo-normal, tells
// inside from outside where the mesh is the boundary of a solid: no two triangles meet
// but in common vertices and edges, the triangles round a vertex form one fan, and the
// parts, each turned outward, lie side by side (their boxes apart).  A closed mesh need
// not be: parts may overlap, lie inside one another or be turned inside out, and then the sign
// also changes half way between two of their surfaces.  Says no where in doubt (rounding,
// and a true hollow, one part inside another turned inward): those take the general path.
// 1280 triangles: 1.9 ms, once a mesh and creation (the hierarchy 1.8).
bool mesh_bounds_solid(const fdtd_mesh_desc& md, const MeshHost& M) {
    const int nt = md.n_triangles, nv = md.n_vertices;
    auto corners = [&](int leaf) {
        const MeshTri& T = M.tris[leaf];
        return Corners{{T.p[0], T.p[1], T.p[2]}, md.triangles + 3 * (size_t)T.id};
    };
    // directed edges, sorted: the triangle on the other side of each
    struct Edge {
        int a, b, t;
        bool operator<(const Edge& o) const { return a != o.a ? a < o.a : b < o.b; }
    };
    std::vector<Edge> edges;
    std::vector<int> degree(nv, 0), any(nv, -1);
    for (int t = 0; t < nt; ++t)
        for (int k = 0; k < 3; ++k) {
            const int a = md.triangles[3 * (size_t)t + k], b = md.triangles[3 * (size_t)t + (k + 1) % 3];
            edges.push_back({a, b, t});
            ++degree[a];
            any[a] = t;
        }
    std::sort(edges.begin(), edges.end());
    auto across = [&](int a, int b) {  // triangle with the directed edge a b (every one exists)
        return std::lower_bound(edges.begin(), edges.end(), Edge{a, b, 0})->t;
    };
    // one fan round each vertex
    for (int v = 0; v < nv; ++v) {
        if (degree[v] == 0) continue;
        int t = any[v], n = 0;
        do {
            const int32_t* q = md.triangles + 3 * (size_t)t;
            const int k = q[0] == v ? 0 : q[1] == v ? 1 : 2;
            t = across(v, q[(k + 2) % 3]);  // the edge (previous corner, v), from its other side
            ++n;
        } while (t != any[v] && n <= degree[v]);
        if (n != degree[v]) return false;
    }
    // parts: enclosed volume and box of each
    std::vector<int> part(nt, -1), todo;
    std::vector<std::vector<double>> box;
    for (int s = 0; s < nt; ++s) {
        if (part[s] >= 0) continue;
        std::vector<double> b{HUGE_VAL, HUGE_VAL, HUGE_VAL, -HUGE_VAL, -HUGE_VAL, -HUGE_VAL};
        double volume = 0.0, size = 0.0;
        const double* o = md.vertices + 3 * (size_t)md.triangles[3 * (size_t)s];
        part[s] = (int)box.size();
        todo.assign(1, s);
        while (!todo.empty()) {
            const int t = todo.back();
            todo.pop_back();
            const int32_t* q = md.triangles + 3 * (size_t)t;
            double r[3][3], n[3];
            for (int k = 0; k < 3; ++k) {
                const double* p = md.vertices + 3 * (size_t)q[k];
                sub3(p, o, r[k]);
                for (int d = 0; d < 3; ++d) {
                    b[d] = std::min(b[d], p[d]);
                    b[3 + d] = std::max(b[3 + d], p[d]);
                }
                const int u = across(q[(k + 1) % 3], q[k]);
                if (part[u] < 0) {
                    part[u] = part[s];
                    todo.push_back(u);
                }
            }
            cross3(r[1], r[2], n);
            volume += dot3(r[0], n);
            size += std::fabs(dot3(r[0], n));
        }
        if (!(volume > 1e-9 * size)) return false;
        for (const auto& c : box) {
            bool meet = true;
            for (int d = 0; d < 3; ++d) meet = meet && b[d] <= c[3 + d] && c[d] <= b[3 + d];
            if (meet) return false;
        }
        box.push_back(b);
        if (box.size() > 64) return false;
    }
    // no two triangles meet elsewhere
    double extent = 0.0;
    for (int d = 0; d < 3; ++d)
        extent = std::max({extent, std::fabs(M.nodes[0].lo[d]), std::fabs(M.nodes[0].hi[d])});
    const double eps = 1e-12 * extent;
    auto boxes_meet = [&](const MeshNode& a, const MeshNode& b) {
        for (int d = 0; d < 3; ++d)
            if (a.lo[d] > b.hi[d] + eps || b.lo[d] > a.hi[d] + eps) return false;
        return true;
    };
    auto tris_meet = [&](const MeshTri& a, const MeshTri& b) {
        for (int d = 0; d < 3; ++d) {
            if (std::min({a.p[0][d], a.p[1][d], a.p[2][d]}) > std::max({b.p[0][d], b.p[1][d], b.p[2][d]}) + eps) return false;
            if (std::min({b.p[0][d], b.p[1][d], b.p[2][d]}) > std::max({a.p[0][d], a.p[1][d], a.p[2][d]}) + eps) return false;
        }
        return true;
    };
    std::vector<std::pair<int, int>> pairs(1, {0, 0});
    while (!pairs.empty()) {
        const auto [na, nb] = pairs.back();
        pairs.pop_back();
        const MeshNode &a = M.nodes[na], &b = M.nodes[nb];
        if (na != nb && !boxes_meet(a, b)) continue;
        if (na == nb && a.count == 0) {
            pairs.insert(pairs.end(), {{a.first, a.first}, {a.first + 1, a.first + 1}, {a.first, a.first + 1}});
        } else if (a.count == 0) {
            pairs.insert(pairs.end(), {{a.first, nb}, {a.first + 1, nb}});
        } else if (b.count == 0) {
            pairs.insert(pairs.end(), {{na, b.first}, {na, b.first + 1}});
        } else {
            for (int i = a.first; i < a.first + a.count; ++i)
                for (int j = na == nb ? i + 1 : b.first; j < b.first + b.count; ++j)
                    if (tris_meet(M.tris[i], M.tris[j]) && !only_shared(corners(i), corners(j), eps)) return false;
        }
    }
    return true;
}

// (for tests without a device) 1 / 0: mesh_bounds_solid, negative: not a valid mesh
extern "C" int fdtd_debug_mesh_bounds_solid(const fdtd_mesh_desc* mesh) {
    MeshHost M;
    std::string err;
    if (!mesh || !build_mesh(*mesh, M, err)) return -1;
    return mesh_bounds_solid(*mesh, M) ? 1 : 0;
}

// Extent of rotation * v over the vertices: the world box of the body is
// centre + [lo, hi] (FDTD_RigidObject::UpdateBoundingBox, FDTD_RigidObject.cpp:190-226).
void mesh_extent(const double* verts, size_t nv, const double R[9], double lo[3], double hi[3]) {
    for (int d = 0; d < 3; ++d) {
        lo[d] = HUGE_VAL;
        hi[d] = -HUGE_VAL;
    }
    for (size_t v = 0; v < nv; ++v) {
        const double* p = &verts[3 * v];
        for (int d = 0; d < 3; ++d) {
            const double w = R[d * 3 + 0] * p[0] + R[d * 3 + 1] * p[1] + R[d * 3 + 2] * p[2];
            lo[d] = std::min(lo[d], w);
            hi[d] = std::max(hi[d], w);
        }
    }
}

bool read_obj(const char* path, double scale, std::vector<double>& verts, std::vector<int32_t>& tris, std::string& err) {
    std::ifstream f(path);
    if (!f) {
        err = std::string("cannot open mesh file ") + path;
        return false;
    }
    verts.clear();
    tris.clear();
    std::string line;
    int lineno = 0;
    while (std::getline(f, line)) {
        ++lineno;
        if (line.size() < 2) continue;
        std::istringstream ss(line);
        std::string tag;
        ss >> tag;
        if (tag == "v") {
            double x, y, z;
            if (!(ss >> x >> y >> z)) {
                err = std::string(path) + ":" + std::to_string(lineno) + ": bad vertex";
                return false;
            }
            verts.push_back(x * scale);
            verts.push_back(y * scale);
            verts.push_back(z * scale);
        } else if (tag == "f") {
            std::vector<int32_t> idx;
            std::string tok;
            while (ss >> tok) {
                // "i", "i/t", "i//n", "i/t/n"; negative indices count from the end
                const long v = std::strtol(tok.c_str(), nullptr, 10);
                const long nvs = (long)(verts.size() / 3);
                const long z = v > 0 ? v - 1 : nvs + v;
                if (v == 0 || z < 0) {
                    err = std::string(path) + ":" + std::to_string(lineno) + ": bad face index";
                    return false;
                }
                idx.push_back((int32_t)z);
            }
            if (idx.size() < 3) {
                err = std::string(path) + ":" + std::to_string(lineno) + ": face with fewer than 3 vertices";
                return false;
            }
            for (size_t k = 1; k + 1 < idx.size(); ++k) {  // fan
                tris.push_back(idx[0]);
                tris.push_back(idx[k]);
                tris.push_back(idx[k + 1]);
            }
        }
    }
    for (int32_t t : tris)
        if (t >= (int32_t)(verts.size() / 3)) {
            err = std::string(path) + ": face index beyond the vertices";
            return false;
        }
    return true;
}

}  // namespace fdtd

extern "C" fdtd_status fdtd_read_obj(const char* path, double scale, int32_t* n_vertices, int32_t* n_triangles,
                                     double* vertices, int32_t* triangles) {
    if (!path || !n_vertices || !n_triangles) return FDTD_ERR_INVALID_ARG;
    std::vector<double> v;
    std::vector<int32_t> t;
    std::string err;
    if (!fdtd::read_obj(path, scale, v, t, err)) {
        fdtd::set_error(nullptr, err);
        return FDTD_ERR_IO;
    }
    *n_vertices = (int32_t)(v.size() / 3);
    *n_triangles = (int32_t)(t.size() / 3);
    if (vertices) std::memcpy(vertices, v.data(), v.size() * sizeof(double));
    if (triangles) std::memcpy(triangles, t.data(), t.size() * sizeof(int32_t));
    return FDTD_OK;
}

extern "C" fdtd_status fdtd_mesh_signed_distance(const fdtd_mesh_desc* mesh, int64_t n, const double* points,
                                                 double* out) {
    if (!mesh || n < 0 || (n > 0 && (!points || !out))) return FDTD_ERR_INVALID_ARG;
    fdtd::MeshHost M;
    std::string err;
    if (!fdtd::build_mesh(*mesh, M, err)) {
        fdtd::set_error(nullptr, err);
        return FDTD_ERR_GEOMETRY;
    }
    const fdtd::MeshView v{M.nodes.data(), M.tris.data(), (int)M.nodes.size(), (int)M.tris.size(), nullptr, 0, 0};
    for (int64_t i = 0; i < n; ++i) out[i] = fdtd::mesh_sdf(v, points + 3 * i);
    return FDTD_OK;
}
