// kpt_trace.cuh -- two-level BVH2 traversal (closest hit and any hit).
//
// Follows TLAS::intersect / TLAS::intersectP (shaders/tlas.cu:8-125),
// BLAS2::intersect / BLAS2::intersectP (shaders/blas.cuh:198-336),
// Bounds3f::intersectP (maths/bounds.cuh:38-57) and Triangle::intersect
// (shaders/triangle.cuh:66-102): the same visiting order (near child popped
// first, children culled against the closest hit so far), the same absolute
// epsilons, IEEE arithmetic.  Differences from the reference, none of which
// changes a result:
//   * child boxes live in the parent node, so the boxes tested when a node
//     is popped are the ones the reference tests, read in one record;
//   * the stacks hold 48 (BLAS) and 32 (TLAS) entries instead of 16 (the
//     reference overflows its 16-entry stacks on deep trees, which is
//     undefined behaviour); a ray that would overflow stops and is counted
//     in `overflow`.
#pragma once
#include <cooperative_groups.h>

#include "kpt_device.cuh"
#include "kpt_index.h"
#include "kpt_internal.h"

namespace kpt {

namespace cg = cooperative_groups;

struct XRay { float3 o, d, inv; };

__device__ __forceinline__ XRay make_xray(float3 o, float3 d) {
    XRay r;
    r.o = o;
    r.d = d;
    r.inv = make_float3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
    return r;
}

// Ray::transform (shaders/ray.cuh:28-31): object ray = M (o,1), M (d,0),
// direction not renormalised so that t is shared with the world ray.
__device__ __forceinline__ XRay transform_xray(const XRay& r, const float4* inv) {
    float3 o = make_float3(xrow(inv[0], r.o, 1.0f), xrow(inv[1], r.o, 1.0f), xrow(inv[2], r.o, 1.0f));
    float3 d = make_float3(xrow(inv[0], r.d, 0.0f), xrow(inv[1], r.d, 0.0f), xrow(inv[2], r.d, 0.0f));
    return make_xray(o, d);
}

// Slab test against one child box of a node.
__device__ __forceinline__ bool slab(float lx, float ly, float lz, float hx, float hy, float hz,
                                     const XRay& r, float tmin, float tmax, float* tenter_out) {
    float t0x = xm(xs(lx, r.o.x), r.inv.x), t1x = xm(xs(hx, r.o.x), r.inv.x);
    float t0y = xm(xs(ly, r.o.y), r.inv.y), t1y = xm(xs(hy, r.o.y), r.inv.y);
    float t0z = xm(xs(lz, r.o.z), r.inv.z), t1z = xm(xs(hz, r.o.z), r.inv.z);
    float tenter = fmaxf(fmaxf(fminf(t0x, t1x), fminf(t0y, t1y)), fminf(t0z, t1z));
    float texit = fminf(fminf(fmaxf(t0x, t1x), fmaxf(t0y, t1y)), fmaxf(t0z, t1z));
    bool hit = (tenter <= texit) && (texit >= tmin) && (tenter <= tmax);
    *tenter_out = hit ? tenter : __int_as_float(0x7f800000);
    return hit;
}

__device__ __forceinline__ void node_slabs(const BvhNode& n, const XRay& r, float tmin, float tmax,
                                           bool* h1, float* t1, bool* h2, float* t2) {
    *h1 = slab(n.a.x, n.a.y, n.a.z, n.a.w, n.b.x, n.b.y, r, tmin, tmax, t1);
    *h2 = slab(n.b.z, n.b.w, n.c.x, n.c.y, n.c.z, n.c.w, r, tmin, tmax, t2);
}

__device__ __forceinline__ BvhNode load_node(const BvhNode* p) {
    BvhNode n;
    const float4* q = reinterpret_cast<const float4*>(p);
    n.a = __ldg(q);
    n.b = __ldg(q + 1);
    n.c = __ldg(q + 2);
    n.d = __ldg(reinterpret_cast<const int4*>(q + 3));
    return n;
}

// Moeller-Trumbore with the reference's epsilons; returns t or +inf.
__device__ __forceinline__ float tri_test(const float4* tri, const XRay& r, float tmin, float tmax,
                                          float* bu, float* bv, int* local_id) {
    float4 a = __ldg(tri), b = __ldg(tri + 1), c = __ldg(tri + 2);
    float3 v0 = make_float3(a.x, a.y, a.z);
    float3 e1 = make_float3(b.x, b.y, b.z);
    float3 e2 = make_float3(c.x, c.y, c.z);
    const float INF = __int_as_float(0x7f800000);
    float3 pv = xcross(r.d, e2);
    float det = xdot(e1, pv);
    if (det > -TRI_EPS && det < TRI_EPS) return INF;
    float inv = __frcp_rn(det);
    float3 tv = xsub3(r.o, v0);
    float u = xm(inv, xdot(tv, pv));
    if (u < 0.0f || u > 1.0f) return INF;
    float3 qv = xcross(tv, e1);
    float v = xm(inv, xdot(r.d, qv));
    if (v < 0.0f || xa(u, v) > 1.0f) return INF;
    float t = xm(inv, xdot(e2, qv));
    if (t > TRI_EPS && t < tmax && t > tmin) {
        *bu = u;
        *bv = v;
        *local_id = __float_as_int(a.w);
        return t;
    }
    return INF;
}

struct Hit {
    float t;
    int inst;       // instance, -1: miss
    int tri;        // local triangle id (mesh order)
    float u, v;
};

struct TraceStats {
    unsigned box_tests, tri_tests, inst_xforms, overflow;
};

// Stack entries: >= 0 interior node index; < 0 leaf, encoded as
// -(2 * parent + slot) - 1, whose triangle range is read back from the
// parent node when it is popped (the node is still in L1).
__device__ __forceinline__ int leaf_code(int parent, int slot) { return -(2 * parent + slot) - 1; }

// BLAS2::intersect (blas.cuh:261-336) for one instance, merged into `best`
// the way TLAS::intersect does (tlas.cu:116-121).
__device__ __forceinline__ void blas_closest(const SceneView& s, int inst, const XRay& wr, float tmin, float tmax,
                                             Hit& best, TraceStats& st, int* stack) {
    const InstRec& ir = s.inst[inst];
    const MeshRec m = s.meshes[ir.mesh];
    float4 inv[3] = {__ldg(&ir.inv[0]), __ldg(&ir.inv[1]), __ldg(&ir.inv[2])};
    XRay r = transform_xray(wr, inv);
    st.inst_xforms++;
    Hit loc;
    loc.t = __int_as_float(0x7f800000);
    loc.tri = -1;
    loc.u = loc.v = 0.0f;
    int sp = 0;
    int first = m.leaf_first, count = m.leaf_count;
    bool leaf = m.node_root < 0;
    if (!leaf) stack[sp++] = m.node_root;
    for (;;) {
        if (!leaf) {
            if (sp == 0) break;
            int e = stack[--sp];
            if (e < 0) {
                int c = -e - 1;
                int4 d = __ldg(reinterpret_cast<const int4*>(s.nodes + (c >> 1)) + 3);
                first = (c & 1) ? d.z : d.x;
                count = (c & 1) ? d.w : d.y;
                leaf = true;
            } else {
                BvhNode n = load_node(s.nodes + e);
                bool h1, h2;
                float t1, t2;
                node_slabs(n, r, tmin, tmax, &h1, &t1, &h2, &t2);
                st.box_tests += 2;
                bool p1 = h1 && t1 < loc.t, p2 = h2 && t2 < loc.t;
                if (sp + 2 > BLAS_STACK) { st.overflow++; break; }
                int c1 = n.d.y ? leaf_code(e, 0) : n.d.x;
                int c2 = n.d.w ? leaf_code(e, 1) : n.d.z;
                if (t1 > t2) {
                    if (p1) stack[sp++] = c1;
                    if (p2) stack[sp++] = c2;
                } else {
                    if (p2) stack[sp++] = c2;
                    if (p1) stack[sp++] = c1;
                }
                continue;
            }
        }
        for (int i = 0; i < count; ++i) {
            float u, v;
            int lid;
            float t = tri_test(s.tris + 3 * (size_t)(first + i), r, tmin, tmax, &u, &v, &lid);
            st.tri_tests++;
            if (t < loc.t) {
                loc.t = t;
                loc.tri = lid;
                loc.u = u;
                loc.v = v;
                tmax = t;
            }
        }
        leaf = false;
        if (m.node_root < 0) break;
    }
    if (loc.t < best.t) {
        best = loc;
        best.inst = inst;
    }
}

// TLAS::intersect (tlas.cu:60-125).
__device__ __forceinline__ Hit trace_closest(const SceneView& s, const XRay& r, float tmin, float tmax,
                                             TraceStats& st, int* stack) {
    Hit best;
    best.t = __int_as_float(0x7f800000);
    best.inst = -1;
    best.tri = -1;
    best.u = best.v = 0.0f;
    float te;
    st.box_tests++;
    if (s.ninst == 0 ||
        !slab(s.tlas_lo.x, s.tlas_lo.y, s.tlas_lo.z, s.tlas_hi.x, s.tlas_hi.y, s.tlas_hi.z, r, tmin, tmax, &te))
        return best;
    if (s.tlas_root_leaf) {
        blas_closest(s, 0, r, tmin, tmax, best, st, stack);
        return best;
    }
    int* tstack = stack + BLAS_STACK;
    int sp = 0;
    tstack[sp++] = 0;
    while (sp > 0) {
        int e = tstack[--sp];
        if (e >= 0) {
            BvhNode n = load_node(s.tlas + e);
            bool h1, h2;
            float t1, t2;
            node_slabs(n, r, tmin, tmax, &h1, &t1, &h2, &t2);
            st.box_tests += 2;
            bool p1 = h1 && t1 < best.t, p2 = h2 && t2 < best.t;
            if (sp + 2 > TLAS_STACK) { st.overflow++; break; }
            int c1 = n.d.y ? -n.d.x - 1 : n.d.x;   // TLAS leaves hold one instance
            int c2 = n.d.w ? -n.d.z - 1 : n.d.z;
            if (t1 > t2) {
                if (p1) tstack[sp++] = c1;
                if (p2) tstack[sp++] = c2;
            } else {
                if (p2) tstack[sp++] = c2;
                if (p1) tstack[sp++] = c1;
            }
        } else {
            blas_closest(s, -e - 1, r, tmin, tmax, best, st, stack);
        }
    }
    return best;
}

// BLAS2::intersectP (blas.cuh:198-259).
__device__ __forceinline__ bool blas_any(const SceneView& s, int inst, const XRay& wr, float tmin, float tmax,
                                         TraceStats& st, int* stack) {
    const InstRec& ir = s.inst[inst];
    const MeshRec m = s.meshes[ir.mesh];
    float4 inv[3] = {__ldg(&ir.inv[0]), __ldg(&ir.inv[1]), __ldg(&ir.inv[2])};
    XRay r = transform_xray(wr, inv);
    st.inst_xforms++;
    int sp = 0;
    int first = m.leaf_first, count = m.leaf_count;
    bool leaf = m.node_root < 0;
    if (!leaf) stack[sp++] = m.node_root;
    for (;;) {
        if (!leaf) {
            if (sp == 0) return false;
            int e = stack[--sp];
            if (e < 0) {
                int c = -e - 1;
                int4 d = __ldg(reinterpret_cast<const int4*>(s.nodes + (c >> 1)) + 3);
                first = (c & 1) ? d.z : d.x;
                count = (c & 1) ? d.w : d.y;
            } else {
                BvhNode n = load_node(s.nodes + e);
                bool h1, h2;
                float t1, t2;
                node_slabs(n, r, tmin, tmax, &h1, &t1, &h2, &t2);
                st.box_tests += 2;
                if (sp + 2 > BLAS_STACK) { st.overflow++; return false; }
                int c1 = n.d.y ? leaf_code(e, 0) : n.d.x;
                int c2 = n.d.w ? leaf_code(e, 1) : n.d.z;
                // near child pushed last, popped first
                if (t1 > t2) {
                    if (h1) stack[sp++] = c1;
                    if (h2) stack[sp++] = c2;
                } else {
                    if (h2) stack[sp++] = c2;
                    if (h1) stack[sp++] = c1;
                }
                continue;
            }
        }
        for (int i = 0; i < count; ++i) {
            float u, v;
            int lid;
            float t = tri_test(s.tris + 3 * (size_t)(first + i), r, tmin, tmax, &u, &v, &lid);
            st.tri_tests++;
            if (t < __int_as_float(0x7f800000)) return true;
        }
        leaf = false;
        if (m.node_root < 0) return false;
    }
}

// TLAS::intersectP (tlas.cu:8-58).
__device__ __forceinline__ bool trace_any(const SceneView& s, const XRay& r, float tmin, float tmax,
                                          TraceStats& st, int* stack) {
    float te;
    st.box_tests++;
    if (s.ninst == 0 ||
        !slab(s.tlas_lo.x, s.tlas_lo.y, s.tlas_lo.z, s.tlas_hi.x, s.tlas_hi.y, s.tlas_hi.z, r, tmin, tmax, &te))
        return false;
    if (s.tlas_root_leaf) return blas_any(s, 0, r, tmin, tmax, st, stack);
    int* tstack = stack + BLAS_STACK;
    int sp = 0;
    tstack[sp++] = 0;
    while (sp > 0) {
        int e = tstack[--sp];
        if (e >= 0) {
            BvhNode n = load_node(s.tlas + e);
            bool h1, h2;
            float t1, t2;
            node_slabs(n, r, tmin, tmax, &h1, &t1, &h2, &t2);
            st.box_tests += 2;
            if (sp + 2 > TLAS_STACK) { st.overflow++; return false; }
            int c1 = n.d.y ? -n.d.x - 1 : n.d.x;
            int c2 = n.d.w ? -n.d.z - 1 : n.d.z;
            if (t1 > t2) {
                if (h1) tstack[sp++] = c1;
                if (h2) tstack[sp++] = c2;
            } else {
                if (h2) tstack[sp++] = c2;
                if (h1) tstack[sp++] = c1;
            }
        } else if (blas_any(s, -e - 1, r, tmin, tmax, st, stack)) {
            return true;
        }
    }
    return false;
}

// ---------------------------------------------------------------------------
// Queue traversal: persistent warps walk a queue of rays.  Each lane owns one
// ray and, when it is done, fetches the next queue entry, so no lane waits
// for the longest ray of its warp.  The warp alternates between three kinds of
// work, each run for many lanes at a time:
//   * interior nodes: every lane whose next entry is a node steps through
//     nodes until it reaches something else; the loop ends for the warp when
//     fewer than half of its live lanes are still in it;
//   * leaves: the warp tests the pending leaves together, four lanes to a
//     leaf (eight while at most four leaves are pending), one triangle each,
//     the rays read from shared memory; the group's closest hit goes back to
//     the lane that owns the ray;
//   * instances: lanes entering or leaving one change the ray's space.
// What bounds it: instruction issue (72% of cycles at 21 of 32 lanes active
// per instruction) and the L1 data pipe (78%: 64-byte nodes and 48-byte
// triangles at unrelated addresses).  One step of any kind per loop iteration
// with leaves tested by their own lane, as before, ran 11.7 lanes per
// instruction: the extension rays of the 1920x1080x16 frame (depth 8) took
// 11.15 ms and its shadow rays 5.86 ms, now 6.41 and 2.82; 1M bounce chains
// in 2M triangles 2.29 ms, now 1.25.  Measured on the way (the same frame's
// extension rays): nodes and leaves in loops of their own 8.99, each left
// early 7.94, node records in two 32-byte loads 7.61, the stack's first 16
// entries in shared memory 7.44 (conflict-free; a divergent local pop spreads
// over lines), leaves shared by the warp 6.74, results reduced only in rounds
// with a hit 6.33.  Not kept: the entry distance beside each stack entry, to
// drop far nodes without loading them (9.15: twice the stack traffic);
// four-wide nodes for the any-hit rays (the same time).
//
// The visiting order and culling are those of trace_closest / trace_any above
// (the BLAS keeps its local closest hit and culls against it, and is merged
// into the ray's closest hit when left; among equal distances of a leaf the
// first triangle wins), so every result is identical to theirs.
//
// Src supplies the queue:  float tmin();       (one value for the whole queue)
//                          void ray(int i, float3& o, float3& d, float& tmax);
//                          bool closest(int i, const Hit& h, float3& o, float3& d);   (ANY == false)
//                          void any(int i, bool occluded);      (ANY == true)
// closest() may return true with the next ray of entry i (a bounce chain):
// the lane traces it next, with the same tmax.  ROOTS: the queue spans
// several scenes merged into `s` (a batch), each entry's TLAS root supplied by
//                          void root(int i, float4& lo, float4& hi, int& root, int& ninst);
// (root: a node index of s.tlas, or ~instance for a single-instance scene).
// The block has TRACE_BLOCK threads; the stack never overflows (a scene
// deeper than BLAS_STACK - 1 or TLAS_STACK - 1 is refused when committed, and
// a node pushes one entry).

constexpr int STACK_SHARED = 16;   // stack entries per ray in shared memory (8: 7.49 ms, 24 and 32: as 16)

// Two 16-byte quarters of a 64-byte node in one load.
__device__ __forceinline__ void load_half_node(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// The bound b' with (t < b') == (t <= b) for every t (denormals are zero here).
__device__ __forceinline__ float next_up(float b) {
    if (!(fabsf(b) < __int_as_float(0x7f800000))) return b;   // infinities and NaN
    if (fabsf(b) < 1.17549435e-38f) return 1.17549435e-38f;
    return __int_as_float(__float_as_int(b) + (b > 0.0f ? 1 : -1));
}

// The hit of local triangle record `slot` (leaf order) of instance `inst` by
// the world ray o, d, at the distance t found by the traversal: its
// barycentrics by the same operations as tri_test.
__device__ __forceinline__ Hit hit_at(const SceneView& s, int inst, int slot, float t, float3 o, float3 d) {
    const InstRec& ir = s.inst[inst];
    const float4 inv[3] = {__ldg(&ir.inv[0]), __ldg(&ir.inv[1]), __ldg(&ir.inv[2])};
    const float3 ro = make_float3(xrow(inv[0], o, 1.0f), xrow(inv[1], o, 1.0f), xrow(inv[2], o, 1.0f));
    const float3 rd = make_float3(xrow(inv[0], d, 0.0f), xrow(inv[1], d, 0.0f), xrow(inv[2], d, 0.0f));
    const float4* tri = s.tris + 3 * (size_t)slot;
    const float4 a = __ldg(tri), b = __ldg(tri + 1), c = __ldg(tri + 2);
    const float3 e1 = make_float3(b.x, b.y, b.z), e2 = make_float3(c.x, c.y, c.z);
    const float3 pv = xcross(rd, e2);
    const float rdet = __frcp_rn(xdot(e1, pv));
    const float3 tv = xsub3(ro, make_float3(a.x, a.y, a.z));
    Hit h;
    h.t = t;
    h.inst = inst;
    h.tri = __float_as_int(a.w);
    h.u = xm(rdet, xdot(tv, pv));
    h.v = xm(rdet, xdot(rd, xcross(tv, e1)));
    return h;
}

// Shared memory of a block's rays.
struct TraceShared {
    float world[9][TRACE_BLOCK];    // world ray: origin, reciprocal direction, direction
    float object[6][TRACE_BLOCK];   // ray in its instance: origin, direction
    int top[STACK_SHARED][TRACE_BLOCK];
    int owners[TRACE_BLOCK];
};

// What the rays of a queue are: closest hits, any hits, or each its own kind.
enum RayKind { RAYS_CLOSEST, RAYS_ANY, RAYS_MIXED };

// One lane's ray and the steps of its warp (every lane of a full warp calls
// step() together).
template <RayKind KIND>
struct Traversal {
    static constexpr unsigned FULL = 0xffffffffu;
    // what a lane does next (cur, and the entries of its stack): an interior
    // node (>= 0), a leaf (~its first triangle, or ~instance in the TLAS), or
    // leave the instance, store the result, nothing more (the queue is empty)
    static constexpr int LEAVE = (int)0x80000000, DONE = (int)0x80000001, DEAD = (int)0x80000002;
    const SceneView& s;
    TraceShared& sh;
    TraceStats& st;                     // (RAYS_MIXED: of the closest-hit rays)
    TraceStats& st_any;                 // RAYS_MIXED: of the any-hit rays
    int* stack;
    const float tmin;
    const int tid, lane;
    int cur;
    int inst = -1;                      // instance being traversed, -1: in the TLAS
    int sp = 0;
    float tmax;
    float bound0, bound;                // boxes entered at or beyond are culled: of the ray, now
    float best_t;                       // closest hit of the ray: instance, triangle record
    int best_inst = -1, best_slot = -1;
    int slot = -1;                      // closest hit in the instance (its distance is `bound`), -1: none
    bool occluded = false;              // any hit: a triangle blocked the ray
    bool any = KIND == RAYS_ANY;
    const BvhNode* nodes;
    float3 o, inv, d;                   // the ray in the space being traversed

    __device__ __forceinline__ Traversal(const SceneView& s_, TraceShared& sh_, TraceStats& st_, TraceStats& st_any_,
                                         int* stack_, float tmin_, bool alive)
        : s(s_), sh(sh_), st(st_), st_any(st_any_), stack(stack_), tmin(tmin_), tid(threadIdx.x),
          lane(threadIdx.x & 31), cur(alive ? DONE : DEAD) {
        tmax = bound0 = bound = best_t = __int_as_float(0x7f800000);
        nodes = s.tlas;
        o = inv = d = make_float3(0.0f, 0.0f, 0.0f);
    }
    __device__ __forceinline__ void push(int e) {
        if (sp < STACK_SHARED) sh.top[sp][tid] = e;
        else stack[sp] = e;
        ++sp;
    }
    __device__ __forceinline__ int pop() {
        --sp;
        int e;
        if (sp < STACK_SHARED) e = sh.top[sp][tid];
        else e = stack[sp];
        return e;
    }
    __device__ __forceinline__ bool is_leaf() const { return cur < 0 && cur > DEAD && inst >= 0; }
    __device__ __forceinline__ bool any_hit() const { return KIND == RAYS_MIXED ? any : KIND == RAYS_ANY; }

    // a new ray: the TLAS root box (TLAS::intersect, tlas.cu:60-75), then its root
    __device__ __forceinline__ void start(float3 wo, float3 wd, float4 lo, float4 hi, int root, int ninst) {
        const XRay w = make_xray(wo, wd);
        o = w.o;
        inv = w.inv;
        d = w.d;
        sh.world[0][tid] = o.x; sh.world[1][tid] = o.y; sh.world[2][tid] = o.z;
        sh.world[3][tid] = inv.x; sh.world[4][tid] = inv.y; sh.world[5][tid] = inv.z;
        sh.world[6][tid] = d.x; sh.world[7][tid] = d.y; sh.world[8][tid] = d.z;
        best_t = __int_as_float(0x7f800000);
        best_inst = -1;
        bound = bound0;
        inst = -1;
        occluded = false;
        nodes = s.tlas;
        sp = 0;
        push(DONE);
        cur = DONE;
        float te;
        (KIND == RAYS_MIXED && any ? st_any : st).box_tests++;
        if (ninst > 0 && slab(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, w, tmin, tmax, &te)) cur = root;
    }
    __device__ __forceinline__ void start(float3 wo, float3 wd) {
        start(wo, wd, s.tlas_lo, s.tlas_hi, s.tlas_root_leaf ? ~0 : 0, s.ninst);
    }

    // the closest hit of the ray that is done
    __device__ __forceinline__ Hit result() const {
        Hit h;
        h.t = best_t;
        h.inst = h.tri = -1;
        h.u = h.v = 0.0f;
        if (best_inst >= 0)
            h = hit_at(s, best_inst, best_slot, best_t,
                       make_float3(sh.world[0][tid], sh.world[1][tid], sh.world[2][tid]),
                       make_float3(sh.world[6][tid], sh.world[7][tid], sh.world[8][tid]));
        return h;
    }

    // nodes, leaves, instances; live: lanes of the warp with a ray on its way
    __device__ __forceinline__ void step(int live) {
        const float INF = __int_as_float(0x7f800000);
        const int warp0 = tid & ~31;
        // ---- interior nodes of the TLAS or of an instance's BLAS, until fewer
        // than half of the live lanes step (3/8: 6.38 ms, 5/8: as 1/2, none: 7.4)
        while (cur >= 0) {
            float4 a, b, c, refs;
            const float4* q = reinterpret_cast<const float4*>(nodes + cur);
            load_half_node(q, a, b);
            load_half_node(q + 2, c, refs);
            // slab() of both child boxes (the ray's bound in one comparison)
            const float l1x = xm(xs(a.x, o.x), inv.x), l1y = xm(xs(a.y, o.y), inv.y), l1z = xm(xs(a.z, o.z), inv.z);
            const float h1x = xm(xs(a.w, o.x), inv.x), h1y = xm(xs(b.x, o.y), inv.y), h1z = xm(xs(b.y, o.z), inv.z);
            const float l2x = xm(xs(b.z, o.x), inv.x), l2y = xm(xs(b.w, o.y), inv.y), l2z = xm(xs(c.x, o.z), inv.z);
            const float h2x = xm(xs(c.y, o.x), inv.x), h2y = xm(xs(c.z, o.y), inv.y), h2z = xm(xs(c.w, o.z), inv.z);
            const float t1 = fmaxf(fmaxf(fminf(l1x, h1x), fminf(l1y, h1y)), fminf(l1z, h1z));
            const float x1 = fminf(fminf(fmaxf(l1x, h1x), fmaxf(l1y, h1y)), fmaxf(l1z, h1z));
            const float t2 = fmaxf(fmaxf(fminf(l2x, h2x), fminf(l2y, h2y)), fminf(l2z, h2z));
            const float x2 = fminf(fminf(fmaxf(l2x, h2x), fmaxf(l2y, h2y)), fmaxf(l2z, h2z));
            const bool p1 = t1 <= x1 && x1 >= tmin && t1 < bound;
            const bool p2 = t2 <= x2 && x2 >= tmin && t2 < bound;
            (KIND == RAYS_MIXED && any ? st_any : st).box_tests += 2;
            const int r1 = __float_as_int(refs.x), r2 = __float_as_int(refs.z);
            const int c1 = __float_as_int(refs.y) ? ~r1 : r1, c2 = __float_as_int(refs.w) ? ~r2 : r2;
            // the near child is next, the far one on the stack
            const bool first = p1 && !(p2 && t1 > t2);
            if (p1 && p2) push(first ? c2 : c1);
            if (p1 || p2) cur = first ? c1 : c2;
            else cur = pop();
            if (2 * __popc(__activemask()) < live) break;
        }
        __syncwarp(FULL);
        // ---- leaves, until fewer than an eighth of the live lanes have one
        unsigned leaves = __ballot_sync(FULL, is_leaf());
        while (leaves) {
            const int nleaf = __popc(leaves);
            const int shift = nleaf <= 4 ? 3 : 2, width = 1 << shift;
            const unsigned gmask = (1u << width) - 1u;
            const int rank = __popc(leaves & ((1u << lane) - 1u));
            const bool mine = is_leaf() && rank < (32 >> shift);   // this lane's leaf is in the round
            if (mine) sh.owners[warp0 + rank] = lane;
            __syncwarp(FULL);
            const int g = lane >> shift, j = lane & (width - 1);   // group of lanes, its triangle
            const bool act = g < nleaf;
            const int owner = act ? sh.owners[warp0 + g] : 0;
            const int k = ~__shfl_sync(FULL, cur, owner) + j;
            // BLAS2::intersect tests against min(tmax, closest so far), intersectP against tmax
            const float limit = __shfl_sync(FULL, any_hit() ? tmax : fminf(tmax, bound), owner);
            float t = INF;
            bool last = false, hit = false;
            if (act) {
                // tri_test of record k (past the end of a leaf: another leaf's, or the array's padding)
                const float4* tri = s.tris + 3 * (size_t)k;
                const float4 a = __ldg(tri), b = __ldg(tri + 1), c = __ldg(tri + 2);
                const int ow = warp0 + owner;
                last = b.w != 0.0f;
                const float3 e1 = make_float3(b.x, b.y, b.z), e2 = make_float3(c.x, c.y, c.z);
                const float3 rd = make_float3(sh.object[3][ow], sh.object[4][ow], sh.object[5][ow]);
                const float3 pv = xcross(rd, e2);
                const float det = xdot(e1, pv);
                const float rdet = __frcp_rn(det);
                const float3 tv = make_float3(xs(sh.object[0][ow], a.x), xs(sh.object[1][ow], a.y),
                                              xs(sh.object[2][ow], a.z));
                const float u = xm(rdet, xdot(tv, pv));
                const float3 qv = xcross(tv, e1);
                const float v = xm(rdet, xdot(rd, qv));
                t = xm(rdet, xdot(e2, qv));
                hit = !(det > -TRI_EPS && det < TRI_EPS) && !(u < 0.0f || u > 1.0f) &&
                      !(v < 0.0f || xa(u, v) > 1.0f) && t > TRI_EPS && t < limit && t > tmin;
            }
            const unsigned ends = __ballot_sync(FULL, last);
            const bool tested = act && !((ends >> (lane - j)) & ((1u << j) - 1u));   // the leaf reaches this lane
            hit = hit && tested;
            const unsigned hits = __ballot_sync(FULL, hit);
            const int from = mine ? rank << shift : 0;                  // first lane of this lane's leaf's group
            const bool my_hit = mine && ((hits >> from) & gmask), my_end = (ends >> from) & gmask;
            if constexpr (KIND == RAYS_MIXED) {   // counted for the ray's kind, by its owner
                const unsigned t_mask = __ballot_sync(FULL, tested);
                if (mine) (any ? st_any : st).tri_tests += __popc((t_mask >> from) & gmask);
            } else if (tested) {
                st.tri_tests++;
            }
            const int first = ~cur;
            if (mine) {
                if (any_hit() && my_hit) {
                    occluded = true;
                    cur = DONE;
                } else if (my_end) {
                    cur = pop();
                } else {
                    cur -= width;   // the leaf's next triangles
                }
            }
            if (KIND != RAYS_ANY && hits) {
                // the group's closest hit, the first among equals
                if (!hit) t = INF;
                int jm = j;
                for (int w = 1; w < width; w <<= 1) {
                    const float t2 = __shfl_xor_sync(FULL, t, w);
                    const int j2 = __shfl_xor_sync(FULL, jm, w);
                    if (t2 < t || (t2 == t && j2 < jm)) {
                        t = t2;
                        jm = j2;
                    }
                }
                const float ht = __shfl_sync(FULL, t, from);
                const int hj = __shfl_sync(FULL, jm, from);
                if (my_hit && !any_hit()) {
                    bound = ht;
                    slot = first + hj;
                }
            }
            leaves = __ballot_sync(FULL, is_leaf());
            if (8 * __popc(leaves) < live) break;
        }
        // ---- instances
        if (cur == LEAVE) {
            // merge its closest hit (tlas.cu:116-121), back to the world ray
            if (KIND != RAYS_ANY) {
                if (slot >= 0 && bound < best_t) {
                    best_t = bound;
                    best_inst = inst;
                    best_slot = slot;
                }
                bound = fminf(bound0, best_t);
            }
            inst = -1;
            nodes = s.tlas;
            o = make_float3(sh.world[0][tid], sh.world[1][tid], sh.world[2][tid]);
            inv = make_float3(sh.world[3][tid], sh.world[4][tid], sh.world[5][tid]);
            d = make_float3(sh.world[6][tid], sh.world[7][tid], sh.world[8][tid]);
            cur = pop();
        } else if (cur < 0 && cur > DEAD && inst < 0) {
            // entering one (TLAS leaf): object-space ray (Ray::transform)
            inst = ~cur;
            const InstRec& ir = s.inst[inst];
            const float4 m[3] = {__ldg(&ir.inv[0]), __ldg(&ir.inv[1]), __ldg(&ir.inv[2])};
            XRay w;
            w.o = o;
            w.d = d;
            const XRay r = transform_xray(w, m);
            o = r.o;
            inv = r.inv;
            d = r.d;
            sh.object[0][tid] = o.x; sh.object[1][tid] = o.y; sh.object[2][tid] = o.z;
            sh.object[3][tid] = d.x; sh.object[4][tid] = d.y; sh.object[5][tid] = d.z;
            (KIND == RAYS_MIXED && any ? st_any : st).inst_xforms++;
            push(LEAVE);
            nodes = s.nodes;
            bound = bound0;
            slot = -1;
            cur = ir.root;
        }
    }
};

// Lanes of a warp that take rays of a queue of n: a queue of fewer rays than
// the grid has lanes is spread over all its warps -- short queues are bound
// by the latency of their longest rays, which other rays of the warp prolong
// (1021 rays 88 -> 27 us, the 65k paths of a 256x256 frame 0.85 -> 0.42 ms
// with this and the above).
__device__ __forceinline__ int queue_lanes(int n) {
    return lanes_of_queue(n, gridDim.x * (TRACE_BLOCK / 32));
}

template <bool ANY, class Src, bool ROOTS = false>
__device__ __forceinline__ void trace_queue(const SceneView& s, int n, int* next, Src& src, TraceStats& st,
                                            int* stack) {
    constexpr unsigned FULL = 0xffffffffu;
    using T = Traversal<ANY ? RAYS_ANY : RAYS_CLOSEST>;
    __shared__ TraceShared sh;
    if (n <= 0) return;
    const int lane = threadIdx.x & 31;
    T r(s, sh, st, st, stack, src.tmin(), lane < queue_lanes(n));
    int ray = -1;   // queue entry
    for (;;) {
        // rays that are done wait until fetch_batch lanes of the warp are (or
        // nobody else works), then store their results and fetch and set up
        // their next rays together
        const unsigned idle = __ballot_sync(FULL, r.cur == T::DONE), dead = __ballot_sync(FULL, r.cur == T::DEAD);
        if (idle && ((idle | dead) == FULL || __popc(idle) >= s.fetch_batch)) {
            bool more = false;
            float3 wo, wd;
            if (r.cur == T::DONE && ray >= 0) {
                if (ANY) src.any(ray, r.occluded);
                else more = src.closest(ray, r.result(), wo, wd);
            }
            const unsigned want = __ballot_sync(FULL, r.cur == T::DONE && !more);
            int base = 0;
            if (lane == 0 && want) base = atomicAdd(next, __popc(want));
            base = __shfl_sync(FULL, base, 0);
            if (r.cur == T::DONE) {
                if (!more) {
                    ray = queue_entry(base, __popc(want & ((1u << lane) - 1u)));
                    if (queued(ray, n)) {
                        src.ray(ray, wo, wd, r.tmax);
                        r.bound0 = next_up(r.tmax);
                        more = true;
                    } else {
                        r.cur = T::DEAD;
                    }
                }
                if (more) {
                    if constexpr (ROOTS) {
                        float4 lo, hi;
                        int root, ninst;
                        src.root(ray, lo, hi, root, ninst);
                        r.start(wo, wd, lo, hi, root, ninst);
                    } else {
                        r.start(wo, wd);
                    }
                }
            }
            continue;
        }
        if (dead == FULL) break;
        r.step(32 - __popc(idle | dead));
    }
}

}  // namespace kpt
