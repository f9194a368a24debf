// Device code shared by the single-request wavefront renderer (wavefront.cu) and the
// multi-request server (server.cu): the SoA path pool, two-level traversal, light
// sampling, and the per-path stages (camera, extend, shade, shadow).
//
// Every stage restates the reference's per-path arithmetic (paths relative to src/):
// camera integrator/wavefront_kernels.cu:234-270 with the draw order of
// cpu_path_tracer.cpp:532-542; extend wavefront_kernels.cu:272-354; shade
// cpu_path_tracer.cpp:403-498 (emission + MIS, pass-through, NEE, BSDF sample, RR);
// shadow cpu_path_tracer.cpp:27-73.  A path's step count (extends so far) is its scatter
// depth plus its pass-through depth, so paths of different depths can share one queue.
#pragma once

#include <cuda_runtime.h>

#include "../../include/lux_gpu.h"
#include "lux_wide.cuh"
#include "pt_device.cuh"

namespace lux {
namespace pt {

constexpr int kThreads = 256;
constexpr int kStack = 72;
constexpr int kShadowSegments = 1024;

// Path state and queues.  A path's records are read and written at places that the queues
// pick, so what is used together lies together, in whole 32-byte sectors moved by one
// instruction each.
//   state   4 words of 16 bytes a path: throughput.rgb and eta scale; previous sample's
//           position and pdf; PCG state lo/hi, depth | passthrough << 16, measure | flags << 8;
//           pixel, sample, PCG increment lo/hi (the last does not change)
//   ray     2: origin and t_min; direction and t_max
//   shadow  4: origin and t_max; direction and ignored primitive (int bits); then, in a scene
//           without pass-through surfaces, the radiance to add when the ray arrives; else
//           contribution.rgb and MIS weight, and the throughput at the vertex
struct PathPool {
    int capacity = 0;
    float4* state = nullptr;
    float4* ray = nullptr;
    float4* shadow = nullptr;
    float4* rad = nullptr;          // radiance.rgb
    float4* hit = nullptr;          // t, u, v, primitive (int bits)
    int* qray[2] = {nullptr, nullptr};
    int* qshadow = nullptr;
};

// Device buffers of a pool (wavefront.cu), without the ray queues if the paths need no order
// of their own; adds what they take to *bytes.
int path_pool_alloc(PathPool& pool, int capacity, bool ray_queues, int64_t* bytes = nullptr);
void path_pool_free(PathPool& pool);

namespace {

LUX_D unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// 32 bytes from a 32-byte aligned address that this kernel may also write.
LUX_D void ld8(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z),
                   "=f"(b.w) : "l"(p) : "memory");
}

// Warp-aggregated append: lanes with the same queue share one atomic.
LUX_D int append(int* counter_base, int queue, bool active) {
    unsigned mask = __ballot_sync(0xffffffffu, active);
    if (!active) return -1;
    unsigned peers = __match_any_sync(mask, queue);
    int leader = __ffs(peers) - 1;
    int base = 0;
    if (static_cast<int>(threadIdx.x & 31) == leader) base = atomicAdd(counter_base + queue, __popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + __popc(peers & lanemask_lt());
}

LUX_D f3 xyz(const float4& v) { return make_f3(v.x, v.y, v.z); }

// ------------------------------------------------------------------ traversal

struct SceneHit {
    int prim = -1;
    float t = 0, u = 0, v = 0;
};

// transform_point / transform_vector with the implicit row (0 0 0 1)
// (core/mat4.cuh:173-199).
LUX_D f3 xform_point(const float* m, f3 p) {
    float x = add(add(add(mul(m[0], p.x), mul(m[1], p.y)), mul(m[2], p.z)), m[3]);
    float y = add(add(add(mul(m[4], p.x), mul(m[5], p.y)), mul(m[6], p.z)), m[7]);
    float z = add(add(add(mul(m[8], p.x), mul(m[9], p.y)), mul(m[10], p.z)), m[11]);
    float w = add(add(add(mul(0.0f, p.x), mul(0.0f, p.y)), mul(0.0f, p.z)), 1.0f);
    return w == 1.0f ? make_f3(x, y, z) : make_f3(x / w, y / w, z / w);
}
LUX_D f3 xform_vector(const float* m, f3 v) {
    return make_f3(add(add(mul(m[0], v.x), mul(m[1], v.y)), mul(m[2], v.z)),
                   add(add(mul(m[4], v.x), mul(m[5], v.y)), mul(m[6], v.z)),
                   add(add(mul(m[8], v.x), mul(m[9], v.y)), mul(m[10], v.z)));
}

// Node visits and triangle tests of a walk in the reference's visit order: each box the
// reference's stackless walk tests (the root's, and both children's of every node it
// enters: bvh/bvh_device.cuh:43-90) and each triangle it tests; instances: TLAS leaves
// whose BLAS was searched.  Filled only by the kCount variants below.
struct WalkCounts {
    unsigned long long boxes = 0, tris = 0, instances = 0;
};

// Closest hit inside one BLAS in object space, reference order (bvh/bvh_device.cuh:92-134
// with GpuMeshPrimitiveIntersector, scene/gpu_scene_bvh.cuh:15-42).  best_t enters as the
// current bound; returns the local triangle id or -1.  kCount adds to *wc.
template <bool kCount = false>
LUX_D int blas_closest(const BvhView& b, f3 o, f3 d, float tmin, float& best_t, float& bu,
                       float& bv, int ignored_local, int* error, WalkCounts* wc = nullptr) {
    if (b.n <= 0) return -1;
    ray3 r{o, tmin, d, best_t};
    slab_ray sr = make_slab_ray(r);
    float tn;
    if (kCount) wc->boxes += 1;
    if (!slab_hit(sr, load_root(b.root), best_t, tn)) return -1;
    int2 stack[kStack];  // (node ref, entry t bits): one 8-byte access per entry
    int sp = 0;
    int cur = b.n == 1 ? ~0 : 0;
    int best = -1;
    const long long bound = 2ll * b.n + 64;
    for (long long step = 0;; ++step) {
        if (step > bound || cur >= b.n - 1 || ~cur >= b.n) {
            atomicOr(error, kErrLoopBound);
            return -1;
        }
        bool pop = true;
        if (cur >= 0) {
            BvhNode nd = load_node(b.nodes, cur);
            float tl, tr;
            if (kCount) wc->boxes += 2;
            bool hl = slab_hit(sr, node_left_box(nd), best_t, tl);
            bool hr = slab_hit(sr, node_right_box(nd), best_t, tr);
            if (hl) {
                if (hr) {
                    if (sp >= kStack) {
                        atomicOr(error, kErrStackOverflow);
                        return -1;
                    }
                    stack[sp] = make_int2(nd.ch.y, __float_as_int(tr));
                    ++sp;
                }
                cur = nd.ch.x;
                pop = false;
            } else if (hr) {
                cur = nd.ch.y;
                pop = false;
            }
        } else {
            const float4* tp = reinterpret_cast<const float4*>(b.tris + ~cur);
            float4 p0 = __ldg(tp);
            int local = __float_as_int(p0.w);
            if (local != ignored_local) {
                if (kCount) wc->tris += 1;
                float4 p1 = __ldg(tp + 1);
                float4 p2 = __ldg(tp + 2);
                float t, u, v;
                if (moller_trumbore(o, d, xyz(p0), xyz(p1), xyz(p2), t, u, v) && t > tmin
                    && t < best_t) {
                    best = local;
                    best_t = t;
                    bu = u;
                    bv = v;
                }
            }
        }
        if (pop) {
            bool resumed = false;
            while (sp > 0) {
                --sp;
                const int2 e = stack[sp];
                if (!(__int_as_float(e.y) > best_t)) {
                    cur = e.x;
                    resumed = true;
                    break;
                }
            }
            if (!resumed) break;
        }
    }
    return best;
}

// Two-level closest hit (intersect_scene_bvh_device, scene/gpu_scene_bvh.cuh:44-135):
// TLAS over instance boxes in reference order; at each instance leaf the ray is taken
// to object space and its BLAS searched with t_max = the current best.  ignored: scene
// triangle id skipped (shadow rays leaving a surface), -1 none.  kCount adds the
// walk's node visits and triangle tests (both levels) to *wc.
template <bool kCount = false>
LUX_D SceneHit scene_closest(const SceneView& sc, f3 o, f3 d, float tmin, float tmax,
                             int ignored, int* error, WalkCounts* wc = nullptr) {
    SceneHit h;
    h.t = tmax;
    if (!sc.has_two_level) return h;
    const BvhView& tl = sc.tlas;
    ray3 r{o, tmin, d, tmax};
    slab_ray sr = make_slab_ray(r);
    float tn;
    if (kCount) wc->boxes += 1;
    if (!slab_hit(sr, load_root(tl.root), h.t, tn)) return h;
    int ign_instance = -1, ign_local = -1;
    if (ignored >= 0) {
        float4 v1 = __ldg(&sc.tris[ignored].v1);
        float4 v2 = __ldg(&sc.tris[ignored].v2);
        ign_instance = __float_as_int(v1.w);
        ign_local = __float_as_int(v2.w);
    }
    int2 stack[kStack];  // (node ref, entry t bits): one 8-byte access per entry
    int sp = 0;
    int cur = tl.n == 1 ? ~0 : 0;
    const long long bound = 2ll * tl.n + 64;
    for (long long step = 0;; ++step) {
        if (step > bound || cur >= tl.n - 1 || ~cur >= tl.n) {
            atomicOr(error, kErrLoopBound);
            return SceneHit{-1, tmax, 0, 0};
        }
        bool pop = true;
        if (cur >= 0) {
            BvhNode nd = load_node(tl.nodes, cur);
            float a, b;
            if (kCount) wc->boxes += 2;
            bool hl = slab_hit(sr, node_left_box(nd), h.t, a);
            bool hr = slab_hit(sr, node_right_box(nd), h.t, b);
            if (hl) {
                if (hr) {
                    if (sp >= kStack) {
                        atomicOr(error, kErrStackOverflow);
                        return SceneHit{-1, tmax, 0, 0};
                    }
                    stack[sp] = make_int2(nd.ch.y, __float_as_int(b));
                    ++sp;
                }
                cur = nd.ch.x;
                pop = false;
            } else if (hr) {
                cur = nd.ch.y;
                pop = false;
            }
        } else {
            int inst_id = sc.tlas_instance[tl.sorted_ids[~cur]];
            const Instance& inst = sc.instances[inst_id];
            f3 lo = xform_point(inst.inv, o);
            f3 ld = xform_vector(inst.inv, d);
            float best = h.t;
            float u = 0, v = 0;
            if (kCount) wc->instances += 1;
            int local = blas_closest<kCount>(sc.blas[inst.blas], lo, ld, tmin, best, u, v,
                                             inst_id == ign_instance ? ign_local : -1, error,
                                             wc);
            if (local >= 0 && best < h.t) {
                h.prim = inst.first_primitive + local;
                h.t = best;
                h.u = u;
                h.v = v;
            }
        }
        if (pop) {
            bool resumed = false;
            while (sp > 0) {
                --sp;
                const int2 e = stack[sp];
                if (!(__int_as_float(e.y) > h.t)) {
                    cur = e.x;
                    resumed = true;
                    break;
                }
            }
            if (!resumed) break;
        }
    }
    return h;
}

// scene_closest as a resumable walk, for kernels whose warps interleave many walks.  The
// TLAS is walked over its binary nodes (a TLAS of at most kFlatTlas instances is entered
// leaf by leaf: its leaf boxes are tested in leaf order when the walk starts), each BLAS
// over its quantised 4-wide nodes (lux_wide.cuh: every leaf the binary walk reaches is
// reached in the same left-first order and accepted by the exact test of its own box, the
// triangle's box formed from its record), so the leaves tested and the best hit after each
// are those of scene_closest / blas_closest above and the result is the same.  (The TLAS
// over its 4-wide nodes: 257 instances 2 % faster, Cornell 4 % and the heavy scene 6 %
// slower, by the spills of a second node test in the kernel.)
//
// A walk is at a BLAS node (cur >= 0), waits at a BLAS leaf (leaf, and perhaps a second one
// in cur), or is done with its BLAS (at_rest).  A leaf may wait while nodes are tested: node
// tests only have to keep every leaf the reference reaches, which they do under any bound
// not below the current one, and leaves are tested in order under the bound of their turn.
// The world-space ray is not kept: tlas() is handed it again when a BLAS is left.  The
// stacks live apart from the scalar state, which then stays in registers.
constexpr int kWideStackPt = 100;     // as kWideStack, of 30-bit codes: 60 nodes, 30 * 3 = 90
constexpr int kFlatTlas = 4;          // TLAS leaves tested together when a walk starts

struct WalkStacks {  // deferred (node ref, entry t bits), TLAS and BLAS
    int2 t[kStack];
    int2 b[kWideStackPt];
};

struct WalkRay {
    f3 o, d;
    float tmin, tmax;
    int ignored;                  // scene triangle skipped, -1 none
};

struct TwoLevelWalk {
    SceneHit hit;                 // best so far (hit.t is the current bound)
    // The BLAS being walked, and the ray in its space.
    slab_ray lsr;
    f3 ld;
    unsigned oct;                 // octant of the object-space ray (wide_octant)
    const WideNode* wide;
    const TriRecord* tris;
    int n, ignored, first;
    int cur, leaf;
    unsigned steps;               // bounded by 2n + 64 per BLAS
    WideTop top;
    WideTop t_top;                // deferred TLAS children

    LUX_D bool at_rest() const { return cur == kNoNode && leaf == kNoNode; }

    LUX_D void fail(int* error, int bit) {
        atomicOr(error, bit);
        hit = SceneHit{};
        hit.t = INFINITY;
        cur = leaf = kNoNode;
        top.clear();
        t_top.clear();
    }
    LUX_D void stop() {  // an occlusion walk ends at its first accepted triangle
        cur = leaf = kNoNode;
        top.clear();
        t_top.clear();
    }

    // Goes through the TLAS, from its root (fresh) or from the last deferred child, until a
    // BLAS is entered (true) or nothing is left (false).
    LUX_D bool tlas(const SceneView& sc, WalkStacks& k, const WalkRay& r, bool fresh,
                    int* error) {
        const BvhView& tl = sc.tlas;
        const slab_ray sr = make_slab_ray(ray3{r.o, r.tmin, r.d, r.tmax});
        int at = kNoNode;
        if (fresh) {
            hit = SceneHit{};
            hit.t = r.tmax;
            stop();
            if (!sc.has_two_level) return false;
            if (tl.n <= kFlatTlas) {
                // Every leaf box is tested here, in leaf order (the binary walk's left-first
                // order), and the passing leaves after the first are deferred with their
                // entry t as the walk defers children, so the walk enters the same instances
                // under the same bounds without stepping through the TLAS's internal nodes
                // (a leaf box passes under a bound exactly when every box above it does).
                float at_t = 0.0f;
                for (int j = tl.n - 1; j >= 0; --j) {
                    float te;
                    if (slab_hit(sr, leaf_box(tl, j), hit.t, te)) {
                        if (at != kNoNode) t_top.push(k.t, at, at_t);
                        at = ~j;
                        at_t = te;
                    }
                }
            } else {
                float tn;
                if (!slab_hit(sr, load_root(tl.root), hit.t, tn)) return false;
                at = 0;
            }
        } else {
            at = t_top.pop(k.t, hit.t);
        }
        const unsigned bound = 2u * static_cast<unsigned>(tl.n) + 64u;
        for (unsigned step = 0; at != kNoNode; ++step) {
            if (step > bound || at >= tl.n - 1 || ~at >= tl.n) {
                fail(error, kErrLoopBound);
                return false;
            }
            if (at >= 0) {
                const BvhNode nd = load_node(tl.nodes, at);
                float ta, tb;
                const bool hl = slab_hit(sr, node_left_box(nd), hit.t, ta);
                const bool hr = slab_hit(sr, node_right_box(nd), hit.t, tb);
                if (hl && hr) {
                    if (t_top.full(kStack)) {
                        fail(error, kErrStackOverflow);
                        return false;
                    }
                    t_top.push(k.t, nd.ch.y, tb);
                }
                at = hl ? nd.ch.x : hr ? nd.ch.y : kNoNode;
            } else {
                if (enter(sc, ~at, r, sr)) return true;
                at = kNoNode;
            }
            if (at == kNoNode) at = t_top.pop(k.t, hit.t);
        }
        return false;
    }

    // Enters the instance of TLAS leaf j: the ray in its object space and the BLAS root's
    // test; true when the walk goes on in the BLAS.
    LUX_D bool enter(const SceneView& sc, int j, const WalkRay& r, const slab_ray& sr) {
        const int inst_id = sc.tlas_instance[sc.tlas.sorted_ids[j]];
        const Instance& inst = sc.instances[inst_id];
        const BvhView& b = sc.blas[inst.blas];
        if (b.n <= 0) return false;
        const f3 lo = xform_point(inst.inv, r.o);
        ld = xform_vector(inst.inv, r.d);
        if (ld.x == r.d.x && ld.y == r.d.y && ld.z == r.d.z) {
            lsr = sr;   // a translation: the same direction, so the same reciprocals
            lsr.o = lo;
        } else {
            lsr = make_slab_ray(ray3{lo, r.tmin, ld, hit.t});
        }
        float tn;
        if (!slab_hit(lsr, load_root(b.root), hit.t, tn)) return false;
        oct = wide_octant(lsr);
        wide = b.wide;
        tris = b.tris;
        n = b.n;
        steps = 0;
        first = inst.first_primitive;
        ignored = -1;
        if (r.ignored >= 0 &&
            __float_as_int(__ldg(&sc.tris[r.ignored].v1.w)) == inst_id)
            ignored = __float_as_int(__ldg(&sc.tris[r.ignored].v2.w));
        top.clear();
        cur = b.n == 1 ? kNoNode : 0;
        leaf = b.n == 1 ? ~0 : kNoNode;
        return true;
    }
    // Tests BLAS node cur and moves on to the next node; a leaf on the way goes to the free
    // place, a second one stops the walk until the first has been tested.
    LUX_D void node_step(WalkStacks& k, int* error) {
        // One branch for the three checks: with one each, renders took 0.2 to 2 % longer.
        if ((++steps > 2u * static_cast<unsigned>(n) + 64u) | (cur >= n - 1) |
            top.full(kWideStackPt)) {
            fail(error, top.full(kWideStackPt) ? kErrStackOverflow : kErrLoopBound);
            return;
        }
        const WideNode w = load_wide(wide, cur);
        float t[4];
        bool p[4];
        wide_test(w, lsr, oct, hit.t, t, p);
        cur = wide_descend(w, t, p, k.b, top);
        wide_move_on(cur, leaf, k.b, top, hit.t);
    }

    // Tests the waiting leaf: its exact box (the triangle's box) under the current best t,
    // then the triangle.
    LUX_D void leaf_step(WalkStacks& k, bool any_hit, int* error) {
        const int j = ~leaf;
        leaf = kNoNode;
        if (j >= n) {
            fail(error, kErrLoopBound);
            return;
        }
        const float4* tp = reinterpret_cast<const float4*>(tris + j);
        const float4 p0 = __ldg(tp);
        const int local = __float_as_int(p0.w);
        if (local != ignored) {
            const float4 p1 = __ldg(tp + 1);
            const float4 p2 = __ldg(tp + 2);
            float tn, t, u, v;
            const octant_ray lorr = make_octant_ray(lsr);
            if (child_hit(triangle_box(xyz(p0), xyz(p1), xyz(p2)), lsr, lorr, hit.t, tn)
                && moller_trumbore(lsr.o, ld, xyz(p0), xyz(p1), xyz(p2), t, u, v)
                && t > lsr.tmin && t < hit.t) {
                hit.prim = first + local;
                hit.t = t;
                hit.u = u;
                hit.v = v;
                if (any_hit) {
                    stop();
                    return;
                }
            }
        }
        wide_move_on(cur, leaf, k.b, top, hit.t);
    }
};

// ------------------------------------------------------------------ lights

// sample_alias_table_index (light/light_sampler.h:71-82).
LUX_D int sample_alias(const AliasEntry* table, int count, float u) {
    float scaled = mul(fminf(u, 0.99999994f), static_cast<float>(count));
    int column = static_cast<int>(scaled);
    if (column >= count) column = count - 1;
    float threshold = sub(scaled, static_cast<float>(column));
    const AliasEntry& e = table[column];
    int index = threshold < e.probability ? column : e.alias;
    return index >= 0 && index < count ? index : -1;
}

// ---- light tree (light/light_sampler.h:90-348).  Every walk is bounded by the node
// count, as the reference's.

// light_bvh_node_importance with squared_distance_to_bounds: power over the squared
// distance from p to the node's box, the distance kept at least kRayEpsilon.
LUX_D float light_node_importance(const SceneView& sc, int i, f3 p) {
    if (i < 0 || i >= sc.light_tree_count) return 0;
    const LightNode& n = sc.light_tree[i];
    if (n.power <= 0 || n.lo.x > n.hi.x || n.lo.y > n.hi.y || n.lo.z > n.hi.z) return 0;
    const float pa[3] = {p.x, p.y, p.z};
    const float lo[3] = {n.lo.x, n.lo.y, n.lo.z};
    const float hi[3] = {n.hi.x, n.hi.y, n.hi.z};
    float d2 = 0;
    for (int a = 0; a < 3; ++a) {
        float delta = 0;
        if (pa[a] < lo[a]) delta = sub(lo[a], pa[a]);
        else if (pa[a] > hi[a]) delta = sub(pa[a], hi[a]);
        d2 = add(d2, mul(delta, delta));
    }
    d2 = fmaxf(d2, mul(kRayEpsilon, kRayEpsilon));
    return n.power / d2;
}

// light_bvh_child_probability: the child's share of its parent's two importances.
LUX_D float light_child_probability(const SceneView& sc, int parent, int child, f3 p) {
    const int count = sc.light_tree_count;
    if (parent < 0 || parent >= count || child < 0 || child >= count) return 0;
    const LightNode& n = sc.light_tree[parent];
    if (child != n.left && child != n.right) return 0;
    const float l = light_node_importance(sc, n.left, p);
    const float r = light_node_importance(sc, n.right, p);
    const float total = add(l, r);
    if (total <= 0) return 0;
    const float lp = l / total;
    return child == n.left ? lp : sub(1.0f, lp);
}

// sample_light_bvh: root to leaf, the draw rescaled at each step.
LUX_D int sample_light_tree(const SceneView& sc, f3 p, float select_u, float& pmf) {
    pmf = 0;
    const int count = sc.light_tree_count;
    int node = sc.light_tree_root;
    if (!sc.light_tree || node < 0 || node >= count) return -1;
    float u = fminf(select_u, 0.99999994f);
    pmf = 1;
    for (int depth = 0; depth < count; ++depth) {
        const LightNode& n = sc.light_tree[node];
        if (n.light >= 0) return n.light;
        const float lp = light_child_probability(sc, node, n.left, p);
        if (lp <= 0) {
            node = n.right;
        } else if (lp >= 1) {
            node = n.left;
        } else if (u < lp) {
            pmf = mul(pmf, lp);
            u = u / lp;
            node = n.left;
        } else {
            const float rp = sub(1.0f, lp);
            pmf = mul(pmf, rp);
            u = sub(u, lp) / rp;
            node = n.right;
        }
        if (node < 0 || node >= count) {
            pmf = 0;
            return -1;
        }
    }
    pmf = 0;
    return -1;
}

// light_bvh_pmf: the product of child probabilities from the light's leaf to the root.
LUX_D float light_tree_pmf(const SceneView& sc, f3 p, int light) {
    const int count = sc.light_tree_count;
    if (!sc.light_tree || !sc.light_leaf || light < 0 || light >= sc.light_count) return 0;
    int node = sc.light_leaf[light];
    if (node < 0 || node >= count) return 0;
    float pmf = 1;
    for (int depth = 0; depth < count; ++depth) {
        const int parent = sc.light_tree[node].parent;
        if (parent < 0) return pmf;
        const float pr = light_child_probability(sc, parent, node, p);
        if (pr <= 0) return 0;
        pmf = mul(pmf, pr);
        node = parent;
        if (node >= count) return 0;
    }
    return 0;
}

// The tree's share of the total power and the other table's power
// (sample_light_bvh_mixture / light_bvh_mixture_pmf, light/light_sampler.h:265-359).
LUX_D bool light_tree_split(const SceneView& sc, float& tree_p, float& other) {
    const float tree_power = sc.light_tree[sc.light_tree_root].power;
    if (tree_power <= 0) return false;
    other = sc.other_count > 0 ? fmaxf(0.0f, sc.other_power) : 0.0f;
    const float total = add(tree_power, other);
    if (total <= 0) return false;
    tree_p = tree_power / total;
    return true;
}

// sample_indexed_discrete_light over the other table's alias entries.
LUX_D int sample_other_light(const SceneView& sc, float u, float& pmf) {
    pmf = 0;
    if (!sc.other_lights || !sc.other_alias || sc.other_count <= 0 || sc.other_power <= 0)
        return -1;
    const int slot = sample_alias(sc.other_alias, sc.other_count, u);
    if (slot < 0) return -1;
    pmf = sc.other_alias[slot].pmf;
    return pmf > 0 ? sc.other_lights[slot] : -1;
}

LUX_D int sample_light_mixture(const SceneView& sc, f3 p, float select_u, float& pmf) {
    pmf = 0;
    float tree_p, other;
    if (!light_tree_split(sc, tree_p, other)) return -1;
    if (other <= 0 || tree_p >= 1) return sample_light_tree(sc, p, select_u, pmf);
    if (tree_p <= 0) return sample_other_light(sc, select_u, pmf);
    const float u = fminf(select_u, 0.99999994f);
    float part = 0;
    int index;
    if (u < tree_p) {
        index = sample_light_tree(sc, p, u / tree_p, part);
        pmf = mul(tree_p, part);
    } else {
        const float other_p = sub(1.0f, tree_p);
        index = sample_other_light(sc, sub(u, tree_p) / other_p, part);
        pmf = mul(other_p, part);
    }
    return pmf > 0 ? index : -1;
}

LUX_D float light_mixture_pmf(const SceneView& sc, f3 p, int light) {
    float tree_p, other;
    if (light < 0 || !light_tree_split(sc, tree_p, other)) return 0;
    if (light < sc.light_count && sc.light_leaf[light] >= 0)
        return mul(tree_p, light_tree_pmf(sc, p, light));
    const int slot = light < sc.light_count && sc.light_other_slot ? sc.light_other_slot[light] : -1;
    if (slot < 0 || other <= 0 || !sc.other_alias) return 0;
    return mul(sub(1.0f, tree_p), sc.other_alias[slot].pmf);
}

LUX_D bool use_light_tree(const SceneView& sc, int sampler) {
    return sampler == 2 && sc.light_tree && sc.light_leaf && sc.light_tree_count > 0 &&
           sc.light_tree_root >= 0 && sc.light_tree_root < sc.light_tree_count;
}

// light_pmf (gpu_scene_light_sampler.cuh:9-45): the selection probability of a light at
// shading position p; p matters to the tree sampler only.
LUX_D float light_pmf(const SceneView& sc, int sampler, f3 p, int index) {
    if (index < 0 || index >= sc.light_count || sc.total_light_power <= 0) return 0;
    if (sampler == 0) return 1.0f / static_cast<float>(sc.light_count);
    if (use_light_tree(sc, sampler)) return light_mixture_pmf(sc, p, index);
    return sc.light_alias ? sc.light_alias[index].pmf : 0.0f;
}

// sample_scene_light (gpu_scene_light_sampler.cuh:47-96): the light picked by select_u
// at shading position p and its pmf (the tree walk's own, else light_pmf); -1 when none.
LUX_D int select_light(const SceneView& sc, int sampler, f3 p, float select_u, float& pmf) {
    pmf = 0;
    if (sc.light_count <= 0 || sc.total_light_power <= 0) return -1;
    int index;
    float selected = 0;
    if (sampler == 0) {
        index = static_cast<int>(mul(fminf(select_u, 0.99999994f), static_cast<float>(sc.light_count)));
        if (index >= sc.light_count) index = sc.light_count - 1;
    } else if (use_light_tree(sc, sampler)) {
        index = sample_light_mixture(sc, p, select_u, selected);
    } else {
        if (!sc.light_alias) return -1;
        index = sample_alias(sc.light_alias, sc.light_count, select_u);
    }
    if (index < 0) return -1;
    pmf = selected > 0 ? selected : light_pmf(sc, sampler, p, index);
    return index;
}

struct LightLi {
    f3 wi, position, radiance;
    float distance = INFINITY;
    float pdf = 0;
    int measure = kMeasureSolidAngle;
    bool valid = false;
};

LUX_D f3 sample_triangle_area(f3 v0, f3 v1, f3 v2, float ux, float uy) {  // light_sampler.h:361-367
    float s = sqrtf(ux);
    float b0 = sub(1.0f, s);
    float b1 = mul(s, sub(1.0f, uy));
    float b2 = mul(s, uy);
    return (v0 * b0 + v1 * b1) + v2 * b2;
}

LUX_D float solid_angle_pdf(f3 lpos, f3 lnormal, int two_sided, float pdf_area, f3 ref) {
    f3 to = lpos - ref;  // pdf_solid_angle (light/light_sampler.h:380-390)
    float d2 = length2(to);
    if (d2 <= mul(kRayEpsilon, kRayEpsilon) || pdf_area <= 0) return 0;
    f3 wi = vdiv(to, sqrtf(d2));
    float c = emission_cosine(lnormal, -wi, two_sided);
    if (c <= 0) return 0;
    return mul(pdf_area, d2) / c;
}

// ------------------------------------------------------------------ image infinite lights
// direction_to_latlong_uv / latlong_uv_to_direction / image_env_lookup /
// image_infinite_pdf_for_texel / sample_image_infinite_light / image_infinite_pdf
// (light/light.h:144-269).

LUX_D float2 env_uv(f3 wi) {
    f3 w = normalize(wi);
    float phi = atan2f(w.z, w.x);
    if (phi < 0) phi = add(phi, 2.0f * kPi);
    float theta = acosf(fmaxf(-1.0f, fminf(1.0f, w.y)));
    return make_float2(mul(phi, 0.5f * kInvPi), mul(theta, kInvPi));
}

LUX_D int env_texel(const EnvLight& e, float2 uv) {
    int x = static_cast<int>(fminf(static_cast<float>(e.width - 1), floorf(mul(uv.x, static_cast<float>(e.width)))));
    int y = static_cast<int>(fminf(static_cast<float>(e.height - 1), floorf(mul(uv.y, static_cast<float>(e.height)))));
    return y * e.width + x;
}

LUX_D f3 env_lookup(const EnvLight& e, f3 wi) {
    if (!e.pixels || e.width <= 0 || e.height <= 0) return splat(0);
    const int i = env_texel(e, env_uv(wi));
    const float* p = e.pixels + 3 * static_cast<size_t>(i);
    return make_f3(p[0], p[1], p[2]) * e.scale;
}

LUX_D float env_pdf_texel(const EnvLight& e, int index, float v) {
    if (!e.cdf || e.width <= 0 || e.height <= 0 || e.total <= 0) return 0;
    const int count = e.width * e.height;
    if (index < 0 || index >= count) return 0;
    float w = index == 0 ? e.cdf[0] : sub(e.cdf[index], e.cdf[index - 1]);
    if (w <= 0) return 0;
    float theta = mul(kPi, v);
    float sin_theta = fmaxf(1e-6f, sinf(theta));
    float uv_pdf = mul(w / e.total, static_cast<float>(count));
    return uv_pdf / mul(mul(mul(2.0f, kPi), kPi), sin_theta);
}

LUX_D float env_pdf(const EnvLight& e, f3 wi) {
    if (!e.pixels || !e.cdf || e.width <= 0 || e.height <= 0 || e.total <= 0) return 0;
    const float2 uv = env_uv(wi);
    return env_pdf_texel(e, env_texel(e, uv), uv.y);
}

// Texel by the running sums (the first texel whose sum reaches the target; a binary
// search finds the same texel as the reference's linear scan), then a uniform point in
// it.
LUX_D LightLi env_sample(const EnvLight& e, float select_u, float ux, float uy) {
    LightLi li;
    if (!e.pixels || !e.cdf || e.width <= 0 || e.height <= 0 || e.total <= 0) return li;
    const int count = e.width * e.height;
    const float target = mul(fminf(select_u, 0.99999994f), e.total);
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (target <= e.cdf[mid]) hi = mid;
        else lo = mid + 1;
    }
    const int index = target <= e.cdf[lo] ? lo : count - 1;
    const int x = index % e.width, y = index / e.width;
    const float u = add(static_cast<float>(x), ux) / static_cast<float>(e.width);
    const float v = add(static_cast<float>(y), uy) / static_cast<float>(e.height);
    const float phi = mul(mul(2.0f, kPi), u);
    const float theta = mul(kPi, v);
    const float st = sinf(theta);
    li.wi = make_f3(mul(cosf(phi), st), cosf(theta), mul(sinf(phi), st));
    li.distance = INFINITY;
    li.radiance = env_lookup(e, li.wi);
    li.pdf = env_pdf_texel(e, index, v);
    li.measure = kMeasureSolidAngle;
    li.valid = max_component(li.radiance) > 0 && li.pdf > 0;
    return li;
}

// ------------------------------------------------------------------ image emission
// image_asset_lookup_nearest (scene/scene_data.h:164-173): the texel under the wrapped
// texture coordinates, times scale.
LUX_D f3 image_lookup(const SceneView& sc, int image, float tu, float tv, f3 scale) {
    if (!sc.images || image < 0) return splat(0);
    const ImageView im = sc.images[image];
    if (!im.pixels || im.width <= 0 || im.height <= 0) return splat(0);
    const float u = sub(tu, floorf(tu));
    const float v = sub(tv, floorf(tv));
    const int x = static_cast<int>(fminf(static_cast<float>(im.width - 1), floorf(mul(u, static_cast<float>(im.width)))));
    const int y = static_cast<int>(fminf(static_cast<float>(im.height - 1), floorf(mul(v, static_cast<float>(im.height)))));
    const float* p = im.pixels + 3 * (static_cast<size_t>(y) * im.width + x);
    return make_f3(mul(p[0], scale.x), mul(p[1], scale.y), mul(p[2], scale.z));
}

// interpolate_triangle_uv (scene/scene_data.h:230-233) at barycentrics (u, v).
LUX_D void triangle_uv(const SceneTriShading& sh, float u, float v, float& tu, float& tv) {
    const float w = sub(sub(1.0f, u), v);
    tu = add(add(mul(w, sh.n0.w), mul(u, sh.n2.w)), mul(v, sh.uv.y));
    tv = add(add(mul(w, sh.n1.w), mul(u, sh.uv.x)), mul(v, sh.uv.z));
}

// gpu_diffuse_area_light_emission_value (gpu_scene_light_sampler.cuh:216-223).
LUX_D f3 area_light_emission(const SceneView& sc, const Light& L, int prim, float u, float v) {
    if (L.image < 0) return L.emission;
    float tu, tv;
    triangle_uv(sc.shading[prim], u, v, tu, tv);
    return image_lookup(sc, L.image, tu, tv, L.image_scale);
}

// sample_light_li (scene/scene_light_sampler.h:212-265 / gpu_scene_light_sampler.cuh:133-193).
LUX_D LightLi sample_light(const SceneView& sc, int sampler, f3 p, float select_u, float comp_u, float ux,
                           float uy) {
    LightLi li;
    float pmf;
    const int index = select_light(sc, sampler, p, select_u, pmf);
    if (index < 0 || !(pmf > 0)) return li;
    const Light L = sc.lights[index];
    if (L.kind == 0) {
        const SceneTri& t = sc.tris[L.primitive];
        f3 v0 = xyz(t.v0), v1 = xyz(t.v1), v2 = xyz(t.v2);
        f3 pos = sample_triangle_area(v0, v1, v2, ux, uy);
        f3 n = triangle_normal(v0, v1, v2);
        float pdf_area = L.area > 0 ? 1.0f / L.area : 0.0f;
        f3 to = pos - p;
        float d2 = length2(to);
        if (d2 <= mul(kRayEpsilon, kRayEpsilon)) return li;
        li.distance = sqrtf(d2);
        li.wi = vdiv(to, li.distance);
        li.position = pos;
        // sample_triangle_barycentric_uv (light/light_sampler.h:369-374) for the texel.
        const float s0 = sqrtf(ux);
        const f3 le = area_light_emission(sc, L, L.primitive, mul(s0, sub(1.0f, uy)), mul(s0, uy));
        li.radiance = eval_emission(le, L.two_sided, n, -li.wi);
        li.pdf = mul(pmf, solid_angle_pdf(pos, n, L.two_sided, pdf_area, p));
        li.measure = kMeasureSolidAngle;
        li.valid = max_component(li.radiance) > 0 && li.pdf > 0;
        return li;
    }
    if (L.kind == 1) {  // sample_point_light (light/light.h:161-175)
        f3 to = L.vec - p;
        float d2 = length2(to);
        if (d2 <= mul(kRayEpsilon, kRayEpsilon)) return li;
        li.distance = sqrtf(d2);
        li.wi = vdiv(to, li.distance);
        li.position = L.vec;
        li.radiance = vdiv(L.emission, d2);
        li.pdf = 1.0f;
        li.measure = kMeasureDiscrete;
        li.valid = max_component(li.radiance) > 0;
    } else if (L.kind == 2) {  // sample_distant_light (light/light.h:177-187)
        li.wi = normalize(L.vec);
        li.distance = INFINITY;
        li.radiance = L.emission;
        li.pdf = 1.0f;
        li.measure = kMeasureDiscrete;
        li.valid = max_component(li.radiance) > 0;
    } else if (L.kind == 4) {  // image infinite: the component draw picks the texel
        if (!sc.env || L.primitive < 0) return li;
        li = env_sample(sc.env[L.primitive], comp_u, ux, uy);
    } else {  // uniform infinite (light/light.h:144-150, 189-197)
        float z = sub(1.0f, mul(2.0f, ux));
        float r = sqrtf(fmaxf(0.0f, sub(1.0f, mul(z, z))));
        float phi = mul(mul(2.0f, kPi), uy);
        li.wi = make_f3(mul(r, cosf(phi)), z, mul(r, sinf(phi)));
        li.distance = INFINITY;
        li.radiance = L.emission;
        li.pdf = 1.0f / mul(4.0f, kPi);
        li.measure = kMeasureSolidAngle;
        li.valid = max_component(li.radiance) > 0;
    }
    li.pdf = mul(li.pdf, pmf);
    return li;
}

LUX_D f3 infinite_le(const SceneView& sc, f3 dir) {  // infinite_lights_le
    f3 le = splat(0);
    for (int i = 0; i < sc.light_count; ++i) {
        const Light& L = sc.lights[i];
        if (L.kind == 3) le = le + L.emission;
        else if (L.kind == 4 && sc.env && L.primitive >= 0) le = le + env_lookup(sc.env[L.primitive], dir);
    }
    return le;
}

LUX_D float infinite_pdf(const SceneView& sc, int sampler, f3 dir) {  // infinite_lights_pdf_li
    float pdf = 0;
    for (int i = 0; i < sc.light_count; ++i) {
        const Light& L = sc.lights[i];
        if (L.kind == 3) {
            pdf = add(pdf, mul(light_pmf(sc, sampler, splat(0.0f), i), 1.0f / mul(4.0f, kPi)));
        } else if (L.kind == 4 && sc.env && L.primitive >= 0) {
            pdf = add(pdf, mul(light_pmf(sc, sampler, splat(0.0f), i), env_pdf(sc.env[L.primitive], dir)));
        }
    }
    return pdf;
}

// ------------------------------------------------------------------ path state helpers

struct PathState {
    f3 thr;
    float eta;
    f3 prev_pos;
    float prev_pdf;
    int pixel, sample, depth, passthrough, measure;
    unsigned flags;
    Pcg rng;
};

LUX_D PathState load_state(const PathPool& rt, int p) {
    PathState s;
    float4 a, b, c, d;
    ld8(rt.state + 4 * static_cast<size_t>(p), a, b);
    ld8(rt.state + 4 * static_cast<size_t>(p) + 2, c, d);
    s.thr = xyz(a);
    s.eta = a.w;
    s.prev_pos = xyz(b);
    s.prev_pdf = b.w;
    s.rng.state = static_cast<uint64_t>(__float_as_uint(c.x)) |
                  (static_cast<uint64_t>(__float_as_uint(c.y)) << 32);
    const int depths = __float_as_int(c.z), mode = __float_as_int(c.w);
    s.depth = depths & 0xffff;
    s.passthrough = (depths >> 16) & 0xffff;
    s.measure = mode & 0xff;
    s.flags = static_cast<unsigned>(mode) >> 8;
    s.pixel = __float_as_int(d.x);
    s.sample = __float_as_int(d.y);
    s.rng.inc = static_cast<uint64_t>(__float_as_uint(d.z)) |
                (static_cast<uint64_t>(__float_as_uint(d.w)) << 32);
    return s;
}

LUX_D float4 state_word2(const PathState& s) {
    return make_float4(__uint_as_float(static_cast<unsigned>(s.rng.state)),
                       __uint_as_float(static_cast<unsigned>(s.rng.state >> 32)),
                       __int_as_float(s.depth | (s.passthrough << 16)),
                       __int_as_float(s.measure | static_cast<int>(s.flags << 8)));
}
LUX_D float4 state_word3(const PathState& s) {
    return make_float4(__int_as_float(s.pixel), __int_as_float(s.sample),
                       __uint_as_float(static_cast<unsigned>(s.rng.inc)),
                       __uint_as_float(static_cast<unsigned>(s.rng.inc >> 32)));
}

// What changes of a path's state; store_new_state: all of it.
LUX_D void store_state(const PathPool& rt, int p, const PathState& s) {
    float4* o = rt.state + 4 * static_cast<size_t>(p);
    stg8(o, make_float4(s.thr.x, s.thr.y, s.thr.z, s.eta),
         make_float4(s.prev_pos.x, s.prev_pos.y, s.prev_pos.z, s.prev_pdf));
    o[2] = state_word2(s);
}
LUX_D void store_new_state(const PathPool& rt, int p, const PathState& s) {
    float4* o = rt.state + 4 * static_cast<size_t>(p);
    stg8(o, make_float4(s.thr.x, s.thr.y, s.thr.z, s.eta),
         make_float4(s.prev_pos.x, s.prev_pos.y, s.prev_pos.z, s.prev_pdf));
    stg8(o + 2, state_word2(s), state_word3(s));
}

LUX_D int path_pixel(const PathPool& rt, int p) {
    return __float_as_int(rt.state[4 * static_cast<size_t>(p) + 3].x);
}

LUX_D void load_ray(const PathPool& rt, int p, float4& o, float4& d) {
    ld8(rt.ray + 2 * static_cast<size_t>(p), o, d);
}
LUX_D void store_ray(const PathPool& rt, int p, f3 o, f3 d) {
    stg8(rt.ray + 2 * static_cast<size_t>(p), make_float4(o.x, o.y, o.z, kRayEpsilon),
         make_float4(d.x, d.y, d.z, INFINITY));
}

LUX_D void add_radiance(const PathPool& rt, int p, f3 v) {
    float4 r = rt.rad[p];
    rt.rad[p] = make_float4(add(r.x, v.x), add(r.y, v.y), add(r.z, v.z), 0.0f);
}

// Moves path p's state (everything but the per-bounce hit and shadow records) from pool
// src to slot q of pool dst.
LUX_D void copy_path(const PathPool& src, int p, const PathPool& dst, int q) {
    float4 a, b;
    for (int k = 0; k < 4; k += 2) {
        ld8(src.state + 4 * static_cast<size_t>(p) + k, a, b);
        stg8(dst.state + 4 * static_cast<size_t>(q) + k, a, b);
    }
    load_ray(src, p, a, b);
    stg8(dst.ray + 2 * static_cast<size_t>(q), a, b);
    dst.rad[q] = src.rad[p];
}

LUX_D int material_of(const SceneView& sc, int prim) {
    return __float_as_int(__ldg(&sc.tris[prim].v0.w));
}

// Emission seen at a hit (surface_light_le + area_light_pdf_solid_angle,
// scene/scene_light_sampler.h:318-465) at barycentrics (u, v).
LUX_D f3 surface_le(const SceneView& sc, int prim, const Material& m, f3 ng, f3 wo, float u,
                    float v) {
    int li = sc.primitive_light[prim];
    if (li >= 0 && li < sc.light_count && sc.lights[li].kind == 0) {
        const Light& L = sc.lights[li];
        return eval_emission(area_light_emission(sc, L, prim, u, v), L.two_sided, ng, wo);
    }
    if (m.emission_image >= 0) {  // gpu_eval_emission of an image-emissive material
        float tu, tv;
        triangle_uv(sc.shading[prim], u, v, tu, tv);
        return eval_emission(image_lookup(sc, m.emission_image, tu, tv, m.emission_scale),
                             m.two_sided, ng, wo);
    }
    if (max_component(m.emission) <= 0) return splat(0);
    return eval_emission(m.emission, m.two_sided, ng, wo);
}

LUX_D float surface_light_pdf(const SceneView& sc, int sampler, int prim, f3 ng, f3 pos,
                              f3 ref) {
    int li = sc.primitive_light[prim];
    if (li >= 0 && li < sc.light_count && sc.lights[li].kind == 0 && sc.lights[li].area > 0) {
        const Light& L = sc.lights[li];
        return mul(light_pmf(sc, sampler, ref, li), solid_angle_pdf(pos, ng, L.two_sided, 1.0f / L.area, ref));
    }
    return 0.0f;
}
// ------------------------------------------------------------------ per-path stages

struct CameraParams {
    int width, height;
    uint64_t seed;
    int frame_index, sample_offset;
};

// New camera path in slot p (generate_camera_rays_kernel; draw order jitter x, jitter y,
// lens 2D, time).
LUX_D void init_path(const PathPool& rt, const Camera& cam, int p, int pixel, int sample,
                     const CameraParams& c) {
    int x = pixel % c.width;
    int y = pixel / c.width;
    Pcg g = make_sampler(c.seed, c.frame_index, pixel, sample + c.sample_offset);
    float jx = g.next_float();
    float jy = g.next_float();
    float u = add(static_cast<float>(x), jx) / static_cast<float>(c.width);
    float v = add(static_cast<float>(c.height - 1 - y), jy) / static_cast<float>(c.height);
    float lx = g.next_float();
    float ly = g.next_float();
    (void)g.next_float();  // time
    f3 o, d;
    camera_ray(cam, u, v, lx, ly, o, d);
    PathState s;
    s.thr = splat(1.0f);
    s.eta = 1.0f;
    s.prev_pos = splat(0.0f);
    s.prev_pdf = 0.0f;
    s.pixel = pixel;
    s.sample = sample;
    s.depth = 0;
    s.passthrough = 0;
    s.measure = kMeasureNone;
    s.flags = 0;
    s.rng = g;
    store_new_state(rt, p, s);
    rt.rad[p] = make_float4(0, 0, 0, 0);
    store_ray(rt, p, o, d);
}

// Records the closest hit h of path p's ray (primitive -1 on a miss).
LUX_D void store_hit(const PathPool& rt, int p, const SceneHit& h) {
    rt.hit[p] = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
}

// The environment's radiance along path p's ray, which hit nothing, with its weight
// (cpu_path_tracer.cpp:415-428); false when there is none.
LUX_D bool miss_radiance(const PathPool& rt, const SceneView& sc, int sampler, int p, f3& add_v) {
    const f3 dir = xyz(rt.ray[2 * static_cast<size_t>(p) + 1]);
    f3 le = infinite_le(sc, dir);
    if (!(max_component(le) > 0)) return false;
    PathState s = load_state(rt, p);
    if (s.depth == 0 || is_delta(s.flags)) {
        add_v = s.thr * le;
        return true;
    }
    if (s.measure == kMeasureSolidAngle && s.prev_pdf > 0) {
        float w = power_heuristic(s.prev_pdf, infinite_pdf(sc, sampler, dir));
        add_v = (s.thr * le) * w;
        return true;
    }
    return false;
}

// store_hit, and on a miss the environment's radiance.
LUX_D void extend_finish(const PathPool& rt, const SceneView& sc, int sampler, int p,
                         const SceneHit& h) {
    store_hit(rt, p, h);
    f3 v;
    if (h.prim < 0 && miss_radiance(rt, sc, sampler, p, v)) add_radiance(rt, p, v);
}

// A path whose ray hit nothing, in place of shading.  (Not at the end of the walk: only the
// shadow rays walked beside it may add to a path's radiance there.)
LUX_D void finish_missed(const PathPool& rt, const SceneView& sc, int sampler, int p) {
    f3 v;
    if (miss_radiance(rt, sc, sampler, p, v)) add_radiance(rt, p, v);
}

// Material class of path p's hit, kMissed when it has none.
constexpr int kMissed = kClasses, kNoPath = kClasses + 1;
LUX_D int hit_class(const PathPool& rt, const SceneView& sc, int p) {
    const int prim = __float_as_int(rt.hit[p].w);
    return prim >= 0 ? material_class(sc.materials[material_of(sc, prim)].type) : kMissed;
}

// A block's paths in order of class, the order of their places within a class, so that its
// warps shade one material each (all but those at the seams) and the block still reads its
// paths' records where the queue has them side by side.  (Appended to a queue per material
// as their walks ended, paths came out of all order, and shading took 1.7 times as long.)
// The block sorts up to kSortRounds paths a thread at a time and its warps take 32 of them
// after 32 as they come free: with one path a thread and a warp for each 32, the warps waited
// for the slowest a third of the time (the heavy scene's 512x512, 16 spp: 10.29 -> 9.82 ms).
constexpr int kSortRounds = 4;
constexpr int kBlockWarps = kThreads / 32;

struct ClassSort {
    int place[kNoPath * kSortRounds * kBlockWarps];   // by class, then by round and warp
    int path[kSortRounds * kThreads];
    int total, taken;

    // Sorts path_of(0 .. rounds * kThreads - 1) (-1: none) by class_of(path).  Called by
    // every thread of the block.
    template <typename PathOf, typename ClassOf>
    LUX_D void sort(int rounds, PathOf path_of, ClassOf class_of) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const unsigned lt = lanemask_lt();
        int p[kSortRounds], cls[kSortRounds], rank[kSortRounds];
#pragma unroll
        for (int r = 0; r < kSortRounds; ++r)
            p[r] = r < rounds ? path_of(r * kThreads + static_cast<int>(threadIdx.x)) : -1;
#pragma unroll
        for (int r = 0; r < kSortRounds; ++r) cls[r] = p[r] >= 0 ? class_of(p[r]) : kNoPath;
#pragma unroll
        for (int r = 0; r < kSortRounds; ++r) {
            rank[r] = 0;
#pragma unroll
            for (int c = 0; c < kNoPath; ++c) {
                const unsigned m = __ballot_sync(0xffffffffu, cls[r] == c);
                if (cls[r] == c) rank[r] = __popc(m & lt);
                if (lane == 0) place[(c * kSortRounds + r) * kBlockWarps + warp] = __popc(m);
            }
        }
        if (threadIdx.x == 0) taken = 0;
        __syncthreads();
        if (warp == 0) {   // exclusive sums of the counts
            constexpr int kEach = kNoPath * kSortRounds * kBlockWarps / 32;
            static_assert(kEach * 32 == kNoPath * kSortRounds * kBlockWarps, "counts per lane");
            int v[kEach], sum = 0;
#pragma unroll
            for (int k = 0; k < kEach; ++k) {
                v[k] = place[lane * kEach + k];
                sum += v[k];
            }
            int incl = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += o;
            }
            int run = incl - sum;
#pragma unroll
            for (int k = 0; k < kEach; ++k) {
                place[lane * kEach + k] = run;
                run += v[k];
            }
            if (lane == 31) total = incl;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortRounds; ++r)
            if (cls[r] < kNoPath)
                path[place[(cls[r] * kSortRounds + r) * kBlockWarps + warp] + rank[r]] = p[r];
        __syncthreads();
    }

    // The next 32 paths for the calling warp: its lane's path and class (-1 and kNoPath past
    // the last); false when none are left.
    LUX_D bool next(int& p, int& cls) {
        const int lane = threadIdx.x & 31;
        int g = 0;
        if (lane == 0) g = atomicAdd(&taken, 1);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (32 * g >= total) return false;
        const int k = 32 * g + lane;
        p = -1;
        cls = kNoPath;
        if (k < total) {
            p = path[k];
            cls = 0;
#pragma unroll
            for (int c = 1; c < kNoPath; ++c)
                if (k >= place[c * kSortRounds * kBlockWarps]) cls = c;
        }
        return true;
    }
};

// Paths a thread for a sort: as many as leave every block something to do.
LUX_D int sort_rounds(int n) {
    return max(1, min(kSortRounds, n / static_cast<int>(kThreads * gridDim.x)));
}

// Closest hit of path p's ray (one walk to completion).
LUX_D void extend_path(const PathPool& rt, const SceneView& sc, int p, int* error) {
    float4 a, b;
    load_ray(rt, p, a, b);
    store_hit(rt, p, scene_closest(sc, xyz(a), xyz(b), a.w, b.w, -1, error));
}

// What path p's shadow ray adds with transmittance tr: throughput * ((contribution * tr) *
// mis), formed at shading where tr is always 1 (whole: the record has the factors).
LUX_D f3 shadow_value(const PathPool& rt, int p, f3 tr, bool whole) {
    const float4* rec = rt.shadow + 4 * static_cast<size_t>(p) + 2;
    if (!whole) return xyz(rec[0]);
    float4 c, t;
    ld8(rec, c, t);
    return xyz(t) * ((xyz(c) * tr) * c.w);
}

// Walks of n items by persistent warps; item(k) names the k-th (any number from 0).  Lanes
// without a walk take the next item through one warp-aggregated atomic on *next_item, so no
// lane idles behind the longest walk of a static warp; and the warp takes one kind of step
// at a time, so that most lanes execute it:
//   * BLAS nodes are tested (at most `budget` rounds) until more lanes wait at a leaf than
//     are at a node, or kRestShare of the lanes are between BLASes;
//   * the waiting leaves are tested;
//   * at kRestShare, finished walks hand over their hits, items are fetched, and the TLAS is
//     walked for all lanes that are between BLASes.  These take several dependent loads
//     whatever their number.
// One step of whatever kind per lane and round, all kinds one after another in every round,
// kept 9-10 of 32 lanes active.  Measured on whole renders (Cornell 256x256 at 64 spp, the
// heavy scene 512x512 at 16, 257 instances 401x301 at 7), that against this: 4.99, 16.41,
// 12.85 against 4.32, 11.64, 9.55 ms.  kRestShare 12/32: 4.85, 12.66, 9.90; 16: 4.66, 12.24,
// 9.75; 20: 4.51, 11.99, 9.62; 24: 4.43, 12.03, 9.60; 28: 4.42, 12.47, 9.97 ms.  Leaves once
// waiting lanes are more than 3, 2, 1, 1/2 times those at nodes (in a later build): 4.15,
// 9.96, 7.66; 4.15, 9.79, 7.64; 4.16, 9.64, 7.40; 4.22, 9.65, 7.34 ms.
//
// tag_of(p) picks an item's scene once (view(tag) returns it); ray(p) is its ray in world
// space; any_hit(scene, p): end at the first accepted triangle.  finish(p, tag, hit) is called
// by every lane of the warp after each round in which some lane finished, with p = -1 for
// lanes that did not, so it may use warp-collective operations (and must do nothing for
// p = -1); it returns true for a walk that goes on from ray(p), which it has changed.
#ifndef LUX_WALK_REST
#define LUX_WALK_REST 24
#endif
constexpr int kRestShare = LUX_WALK_REST;   // of 32
template <typename Item, typename TagOf, typename View, typename Ray, typename AnyHit,
          typename Finish>
LUX_D void walk_items(Item item, int n, int* next_item, int budget, int* error, TagOf tag_of,
                      View view, Ray ray, AnyHit any_hit, Finish finish) {
    const unsigned lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    // Fewer items than lanes are spread over all warps: what counts then is the longest walk
    // plus the steps its warp takes for other lanes (an 8 spp 320x240 render of 8 bounces:
    // 1.67 ms; at least 24, 16, 8, 1 lanes a warp: 1.58, 1.55, 1.49, 1.45).
    const int warps = static_cast<int>(gridDim.x * (blockDim.x >> 5));
    const int lanes = max(1, min(32, (n + warps - 1) / warps));
    // >= 0 active item, -1 needs one, -2 none left
    int p = static_cast<int>(lane) < lanes ? -1 : -2;
    int tag = 0;
    bool fresh = false;
    int alive = lanes;          // lanes that are not out of items
    TwoLevelWalk w;
    w.hit = SceneHit{};
    w.n = 0;
    w.stop();
    WalkStacks stacks;
    for (;;) {
        // Nodes
        int on = 0, waiting = 0, resting = 0;
        for (int s = 0; s < budget; ++s) {
            on = __popc(__ballot_sync(0xffffffffu, w.cur >= 0));
            waiting = __popc(__ballot_sync(0xffffffffu, w.cur < 0 && w.leaf != kNoNode));
            resting = alive - on - waiting;
            if (on == 0 || waiting > on || resting * 32 >= alive * kRestShare) break;
            if (w.cur >= 0) w.node_step(stacks, error);
        }
        if (waiting > 0 && resting * 32 < alive * kRestShare) {
            if (w.leaf != kNoNode) w.leaf_step(stacks, any_hit(view(tag), p), error);
            continue;
        }
        // Lanes between BLASes: those whose walk is over hand over its hit, lanes without
        // an item take one, and the TLAS is walked on.
        const bool done = p >= 0 && !fresh && w.at_rest() && w.t_top.h == kNoNode;
        if (__any_sync(0xffffffffu, done)) {
            SceneHit h = w.hit;
            if (h.prim < 0) h.t = INFINITY;
            const bool again = finish(done ? p : -1, tag, h);
            if (done) {
                fresh = again;
                if (!again) p = -1;
            }
        }
        const bool need = p == -1;
        const unsigned m = __ballot_sync(0xffffffffu, need);
        if (m) {
            const int leader = __ffs(m) - 1;
            int base = 0;
            if (static_cast<int>(lane) == leader) base = atomicAdd(next_item, __popc(m));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (need) {
                const int idx = base + __popc(m & lt);
                if (idx >= n) {
                    p = -2;
                } else {
                    p = item(idx);
                    tag = tag_of(p);
                    fresh = true;
                }
            }
            alive = __popc(__ballot_sync(0xffffffffu, p != -2));
            if (alive == 0) break;
        }
        if (p >= 0 && w.at_rest()) {
            w.tlas(view(tag), stacks, ray(p), fresh, error);
            fresh = false;
        }
    }
}

LUX_D WalkRay path_ray(const PathPool& rt, int p) {
    float4 a, b;
    load_ray(rt, p, a, b);
    return WalkRay{xyz(a), xyz(b), a.w, b.w, -1};
}
LUX_D WalkRay shadow_ray(const PathPool& rt, int p) {
    float4 a, b;
    ld8(rt.shadow + 4 * static_cast<size_t>(p), a, b);
    return WalkRay{xyz(a), xyz(b), kRayEpsilon, a.w, __float_as_int(b.w)};
}

// The segments of path p's shadow ray through pass-through surfaces, exactly as shadow_path
// takes them, one walk per segment: the state of a lane's ray between its walks.  In a scene
// without pass-through materials the first hit already blocks the ray, and a hit exists
// exactly when a closest hit does, so the walk may end at the first accepted triangle.
struct ShadowSegments {
    f3 tr = splat(1.0f);
    int seg = 0;
    bool blocked = false;

    // Takes the closest hit of a segment; true when the ray goes on (path p's shadow record is
    // then the next segment's ray).
    LUX_D bool go_on(const PathPool& rt, const SceneView& sc, int p, const SceneHit& h,
                     int* error) {
        if (h.prim < 0) return false;
        const Material mat = sc.materials[material_of(sc, h.prim)];
        if (!is_passthrough(mat)) {
            blocked = true;
            return false;
        }
        tr = tr * passthrough_transmittance(mat);
        float4* rec = rt.shadow + 4 * static_cast<size_t>(p);
        float4 a, b;
        ld8(rec, a, b);
        const float adv = add(h.t, kRayEpsilon);
        if (!(max_component(tr) > 0) || adv >= a.w) return false;
        if (++seg >= kShadowSegments) {
            atomicOr(error, kErrLoopBound);
            blocked = true;
            return false;
        }
        const f3 o = xyz(a) + xyz(b) * adv;
        stg8(rec, make_float4(o.x, o.y, o.z, sub(a.w, adv)),
             make_float4(b.x, b.y, b.z, __int_as_float(-1)));
        return true;
    }
    LUX_D bool arrives() const { return !blocked && max_component(tr) > 0; }
};

struct ShadeOut {
    bool spawn = false;   // the pool's ray p is the next ray
    bool shadow = false;  // the pool's shadow record p is a shadow ray
};

// ------------------------------------------------------------------ debug images
// The reference wavefront tracer's debug images (integrator/wavefront_debug.cuh,
// wavefront_kernels.cu:287-305, 475-482, 586-592), per-pixel sums over samples:
//   ng / ns   at the camera ray's hit: 0.5 * (normalize(n) + 1) of the geometric normal /
//             of the shading normal turned to the geometric side; nothing on a miss;
//   shadow    at the path's first scattering hit (depth 0, after pass-through surfaces),
//             when it samples a light: orange (1, 0.5, 0) when the light sample is
//             invalid, purple (0.5, 0, 1) when the unoccluded estimate is, else the
//             classification of its shadow ray (shadow_aov_color).
//   path log  (on when log_count is set) one lux_path_log_record per surface vertex a
//             path reaches (integrator/pathstate.cuh:41-96), at an atomically taken
//             index; the index keeps counting past capacity so the host learns the size
//             needed.
struct DebugTargets {
    float* shadow = nullptr;
    float* ng = nullptr;
    float* ns = nullptr;
    lux_path_log_record* log = nullptr;
    unsigned long long* log_count = nullptr;
    long long log_capacity = 0;
    int sample_offset = 0;
    // Traversal totals (box tests, triangle tests, instance visits) of every extension
    // and shadow walk, or null.
    unsigned long long* walk_counts = nullptr;
};

// What the shading of one vertex decided, for its path log record
// (SurfaceStageLogState, integrator/wavefront_kernels.cu:140-151).
struct VertexLog {
    f3 wi = make_f3(0, 0, 0);
    float bsdf_pdf = 0, light_pdf = 0;
    int bsdf_measure = kMeasureNone, light_measure = kMeasureNone, source = 0;
    unsigned bsdf_flags = 0;
    unsigned events = LUX_PATH_EVENT_SURFACE_HIT;
};

constexpr int kSourceBsdf = 2;  // SampleSource::BSDF

// record_surface_vertex / record_path_vertex (integrator/wavefront_kernels.cu:84-138,
// integrator/pathstate.cuh:82-96) for the vertex at hit prim of path state s.
LUX_D void log_vertex(const DebugTargets& dbg, const SceneView& sc, const PathState& s,
                      int vertex, int depth, int prim, f3 pos, f3 ng, f3 ns, f3 wo, f3 thr_before,
                      f3 thr_after, const VertexLog& v, unsigned termination) {
    if (!dbg.log_count) return;
    const unsigned long long index = atomicAdd(dbg.log_count, 1ull);
    if (index >= static_cast<unsigned long long>(dbg.log_capacity)) return;
    const SceneTri tri = sc.tris[prim];
    lux_path_log_record r;
    r.pixel_index = s.pixel;
    r.sample_index = dbg.sample_offset + s.sample;
    r.depth = depth;
    r.triangle_id = prim;
    r.instance_id = __float_as_int(tri.v1.w);
    r.mesh_id = sc.instances[r.instance_id].blas;
    r.local_primitive_id = __float_as_int(tri.v2.w);
    r.primitive_kind = 1;
    r.material_id = __float_as_int(tri.v0.w);
    r.vertex = vertex;
    const f3 vecs[7] = {pos, ng, ns, wo, v.wi, thr_before, thr_after};
    float* dst[7] = {r.position, r.ng, r.ns, r.wo, r.wi, r.throughput_before, r.throughput_after};
    for (int k = 0; k < 7; ++k) {
        dst[k][0] = vecs[k].x;
        dst[k][1] = vecs[k].y;
        dst[k][2] = vecs[k].z;
    }
    r.bsdf_pdf = v.bsdf_pdf;
    r.guide_pdf = 0.0f;
    r.light_pdf = v.light_pdf;
    r.bsdf_pdf_measure = static_cast<uint8_t>(v.bsdf_measure);
    r.guide_pdf_measure = 0;
    r.light_pdf_measure = static_cast<uint8_t>(v.light_measure);
    r.sample_source = static_cast<uint8_t>(v.source);
    r.bsdf_flags = v.bsdf_flags;
    r.termination_flags = termination;
    r.event_flags = v.events | (termination ? LUX_PATH_EVENT_TERMINATED : 0u);
    dbg.log[index] = r;
}

LUX_D void aov_add(float* image, int pixel, f3 c) {
    atomicAdd(image + 3 * size_t(pixel), c.x);
    atomicAdd(image + 3 * size_t(pixel) + 1, c.y);
    atomicAdd(image + 3 * size_t(pixel) + 2, c.z);
}

LUX_D f3 encode_normal_color(f3 n) { return (normalize(n) + splat(1.0f)) * 0.5f; }

// primary_normal_debug_color for the camera ray's closest hit h of path p.
LUX_D void aov_primary(const PathPool& rt, const SceneView& sc, int p, const SceneHit& h,
                       const DebugTargets& aov) {
    const float4 mode = rt.state[4 * static_cast<size_t>(p) + 2];
    if (__float_as_int(mode.z) != 0 || h.prim < 0) return;  // depth and pass-through count both zero
    const int pixel = path_pixel(rt, p);
    const SceneTri tri = sc.tris[h.prim];
    const f3 ng = triangle_normal(xyz(tri.v0), xyz(tri.v1), xyz(tri.v2));
    if (aov.ng) aov_add(aov.ng, pixel, encode_normal_color(ng));
    if (aov.ns) {
        f3 ns = shading_normal(sc.shading[h.prim], ng, h.u, h.v);
        if (dot(ng, ns) < 0) ns = -ns;
        aov_add(aov.ns, pixel, encode_normal_color(ns));
    }
}

// shadow_debug_classification_color: red when the shading normal faces the light but
// the geometric normal does not; unblocked: blue-ish after pass-through surfaces, else
// dark grey; blocked by the source's own material within 16 epsilon: yellow; by a back
// face of it: blue (magenta near a mesh boundary edge, which these scenes do not carry);
// by a front face of it: cyan; by another material: green.
LUX_D f3 shadow_aov_color(const SceneView& sc, int source_prim, f3 ng, f3 ns, f3 dir,
                          int occluder, float hit_t, int passthrough_hits) {
    const float shading_cos = dot(ns, dir);
    const float geometric_cos = dot(ng, dir);
    if (shading_cos > 0 && geometric_cos <= 0) return make_f3(1, 0, 0);
    if (occluder < 0) return passthrough_hits > 0 ? make_f3(0, 0.35f, 0.8f) : splat(0.03f);
    const bool same = material_of(sc, occluder) == material_of(sc, source_prim);
    if (same && hit_t < mul(16.0f, kRayEpsilon)) return make_f3(1, 1, 0);
    if (same) {
        const SceneTri o = sc.tris[occluder];
        const bool back = dot(triangle_normal(xyz(o.v0), xyz(o.v1), xyz(o.v2)), -dir) <= 0;
        return back ? make_f3(0, 0, 1) : make_f3(0, 1, 1);
    }
    return make_f3(0, 1, 0);
}

// Shading of the hit stored for path p (cpu_path_tracer.cpp:430-497).  With kAov, also
// the shadow debug image's light-sample verdict at depth 0, shadow rays at depth 0 are
// marked (1 in the record's last word) for classification, and the vertex goes to the path log at each
// exit evaluate_hit_kernel records one (integrator/wavefront_kernels.cu:397-555).
template <bool kAov = false>
LUX_D ShadeOut shade_path(const PathPool& rt, const SceneView& sc, int sampler, int max_depth,
                          int p, const DebugTargets& aov = DebugTargets{}) {
    ShadeOut out;
    float4 ra, rb;
    load_ray(rt, p, ra, rb);
    const float4 hh = rt.hit[p];
    f3 ro = xyz(ra), rd = xyz(rb);
    int prim = __float_as_int(hh.w);
    float t = hh.x, hu = hh.y, hv = hh.z;
    const SceneTri tri = sc.tris[prim];
    f3 v0 = xyz(tri.v0), v1 = xyz(tri.v1), v2 = xyz(tri.v2);
    const Material m = sc.materials[__float_as_int(tri.v0.w)];
    PathState s = load_state(rt, p);
    const int step = s.depth + s.passthrough;
    f3 pos = ro + rd * t;                    // Ray::at
    f3 ng = triangle_normal(v0, v1, v2);
    f3 wo = -rd;
    const bool logging = kAov && aov.log_count != nullptr;
    const f3 thr0 = s.thr;
    VertexLog vl;
    // Logs this vertex with throughput_after thr1 and the given termination.
    auto log = [&](f3 thr1, unsigned termination) {
        if (!logging) return;
        f3 n = shading_normal(sc.shading[prim], ng, hu, hv);
        if (dot(ng, n) < 0) n = -n;
        log_vertex(aov, sc, s, step, s.depth, prim, pos, ng, n, wo, thr0, thr1, vl, termination);
    };
    // Emission with MIS (cpu_path_tracer.cpp:434-447).
    f3 le = surface_le(sc, prim, m, ng, wo, hu, hv);
    if (max_component(le) > 0) {
        if (s.depth == 0 || is_delta(s.flags)) {
            add_radiance(rt, p, s.thr * le);
            vl.events |= LUX_PATH_EVENT_EMISSION;
        } else if (s.measure == kMeasureSolidAngle && s.prev_pdf > 0) {
            float lpdf = surface_light_pdf(sc, sampler, prim, ng, pos, s.prev_pos);
            add_radiance(rt, p, (s.thr * le) * power_heuristic(s.prev_pdf, lpdf));
            vl.events |= LUX_PATH_EVENT_EMISSION;
        }
    }
    if (is_passthrough(m)) {  // cpu_path_tracer.cpp:449-455
        s.thr = s.thr * passthrough_transmittance(m);
        vl.events |= LUX_PATH_EVENT_PASSTHROUGH | LUX_PATH_EVENT_DELTA;
        vl.wi = normalize(-wo);
        vl.bsdf_pdf = 1.0f;
        vl.bsdf_measure = kMeasureDiscrete;
        vl.source = kSourceBsdf;
        vl.bsdf_flags = kFlagDeltaTransmission | kFlagTransmission;
        if (max_component(s.thr) > 0 && step < max_depth) {
            vl.events |= LUX_PATH_EVENT_SPAWNED_RAY;
            log(s.thr, 0);
            s.passthrough += 1;
            f3 no = pos + rd * kRayEpsilon;
            store_ray(rt, p, no, rd);
            store_state(rt, p, s);
            out.spawn = true;
        } else {
            log(s.thr, max_component(s.thr) <= 0 ? LUX_PATH_END_ZERO_THROUGHPUT
                                                 : LUX_PATH_END_MAX_DEPTH);
        }
        return out;
    }
    if (!is_scattering(m)) {
        log(thr0, LUX_PATH_END_NON_SCATTERING);
        return out;
    }
    if (step >= max_depth || s.depth >= max_depth) {
        log(thr0, LUX_PATH_END_MAX_DEPTH);
        return out;
    }
    SceneTriShading sh = sc.shading[prim];
    f3 ns = shading_normal(sh, ng, hu, hv);
    if (dot(ng, ns) < 0) ns = -ns;   // make_surface_interaction
    Interaction it{pos, ng, ns, wo};
    Pcg& g = s.rng;
    if (has_direct_lighting_lobe(m)) {  // estimate_direct_light, :122-158
        float su = g.next_float();
        float cu = g.next_float();
        float lx = g.next_float();
        float ly = g.next_float();
        LightLi li = sample_light(sc, sampler, pos, su, cu, lx, ly);
        int verdict = 0;  // 0 light sample invalid, 1 estimate invalid, 2 valid
        if (li.valid) vl.events |= LUX_PATH_EVENT_DIRECT_LIGHT_SAMPLED;
        if (li.valid && li.pdf > 0) {
            verdict = 1;
            vl.light_pdf = li.pdf;  // pdf_light_solid_angle, logged as a solid angle
            vl.light_measure = kMeasureSolidAngle;
            f3 f = eval_bsdf(m, it, li.wi);
            float cs = abs_cosine(ns, li.wi);
            float pb = pdf_bsdf(m, it, li.wi);
            if (max_component(f) > 0 && max_component(li.radiance) > 0 && cs > 0) {
                verdict = 2;
                vl.events |= LUX_PATH_EVENT_DIRECT_LIGHT_VALID;
                f3 contrib = (f * li.radiance) * (cs / li.pdf);
                float mis = li.measure == kMeasureDiscrete ? 1.0f : power_heuristic(li.pdf, pb);
                f3 off = dot(li.wi, ng) >= 0 ? ng : -ng;
                f3 so = pos + off * kRayEpsilon;
                f3 sd = li.wi;
                float smax = INFINITY;
                bool ok = true;
                if (li.distance < INFINITY) {  // trace_shadow(from, to)
                    f3 to = li.position - so;
                    float dist = length(to);
                    if (dist <= kRayEpsilon) {
                        ok = false;
                    } else {
                        sd = vdiv(to, dist);
                        smax = sub(dist, kRayEpsilon);
                    }
                }
                const bool mark = kAov && aov.shadow && s.depth == 0 && sc.light_count > 0 &&
                                  sc.total_light_power > 0;
                if (!ok && mark) {  // make_shadow_work_item_li: a zero-length ray, no light
                    sd = li.wi;
                    smax = kRayEpsilon;
                    contrib = splat(0.0f);
                    ok = true;
                }
                if (ok) {
                    out.shadow = true;
                    float4* shadow = rt.shadow + 4 * static_cast<size_t>(p);
                    stg8(shadow, make_float4(so.x, so.y, so.z, smax),
                         make_float4(sd.x, sd.y, sd.z, __int_as_float(prim)));
                    if (kAov || sc.has_passthrough) {
                        stg8(shadow + 2, make_float4(contrib.x, contrib.y, contrib.z, mis),
                             make_float4(s.thr.x, s.thr.y, s.thr.z, mark ? 1.0f : 0.0f));
                    } else {
                        const f3 value = s.thr * (contrib * mis);   // as shadow_value, tr = 1
                        shadow[2] = make_float4(value.x, value.y, value.z, 0.0f);
                    }
                }
            }
        }
        if (kAov && aov.shadow && s.depth == 0 && verdict < 2 && sc.light_count > 0 &&
            sc.total_light_power > 0)
            aov_add(aov.shadow, s.pixel, verdict == 0 ? make_f3(1, 0.5f, 0) : make_f3(0.5f, 0, 1));
    }
    float bx = g.next_float();
    float by = g.next_float();
    BsdfSample bs = sample_bsdf(m, it, bx, by);
    vl.wi = bs.wi;
    vl.bsdf_flags = bs.flags;
    vl.events |= LUX_PATH_EVENT_BSDF_SAMPLED | (is_delta(bs.flags) ? LUX_PATH_EVENT_DELTA : 0u);
    if (bs.pdf > 0) {
        vl.bsdf_pdf = bs.pdf;
        vl.bsdf_measure = bs.measure;
    }
    if (!(bs.pdf > 0 && max_component(bs.weight) > 0)) log(thr0, LUX_PATH_END_INVALID_BSDF);
    if (bs.pdf > 0 && max_component(bs.weight) > 0) {
        f3 nthr = s.thr * bs.weight;
        float neta = mul(s.eta, is_transmission(bs.flags) && bs.eta > 0 ? mul(bs.eta, bs.eta) : 1.0f);
        bool alive = true;
        vl.source = kSourceBsdf;
        if (s.depth > 2) {  // path_transport.cuh:58-84
            float prob = fminf(0.95f, mul(max_component(nthr), neta));
            float ru = g.next_float();
            if (ru <= prob) nthr = vdiv(nthr, prob);
            else alive = false;
        }
        if (!alive) log(nthr, LUX_PATH_END_RUSSIAN_ROULETTE);
        if (alive) {
            vl.events |= LUX_PATH_EVENT_SPAWNED_RAY;
            log(nthr, 0);
            s.thr = nthr;
            s.eta = neta;
            s.prev_pdf = bs.pdf;
            s.measure = bs.measure;
            s.flags = bs.flags;
            s.prev_pos = pos;
            s.depth += 1;
            f3 off = dot(bs.wi, ng) >= 0 ? ng : -ng;   // spawn_scatter_ray
            f3 no = pos + off * kRayEpsilon;
            store_ray(rt, p, no, bs.wi);
            store_state(rt, p, s);
            out.spawn = true;
        }
    }
    return out;
}

// Shadow ray of path p through pass-through surfaces (trace_shadow,
// cpu_path_tracer.cpp:27-73); adds throughput * ((contribution * T) * mis).  With kAov,
// a ray marked at shading adds its classification colour to the shadow debug image.
template <bool kAov = false>
LUX_D void shadow_path(const PathPool& rt, const SceneView& sc, int p, int* error,
                       unsigned long long& segments, const DebugTargets& aov = DebugTargets{}) {
    float4 a, b;
    ld8(rt.shadow + 4 * static_cast<size_t>(p), a, b);
    f3 o = xyz(a), d = xyz(b);
    float tmax = a.w;
    float tmin = kRayEpsilon;
    int ignored = __float_as_int(b.w);
    f3 tr = splat(1.0f);
    bool blocked = false;
    int occluder = -1, crossed = 0;
    float occluder_t = 0;
    for (int seg = 0;; ++seg) {
        if (seg >= kShadowSegments) {
            atomicOr(error, kErrLoopBound);
            blocked = true;
            break;
        }
        ++segments;
        SceneHit h;
        if (kAov && aov.walk_counts) {
            WalkCounts wc;
            h = scene_closest<true>(sc, o, d, tmin, tmax, ignored, error, &wc);
            atomicAdd(aov.walk_counts, wc.boxes);
            atomicAdd(aov.walk_counts + 1, wc.tris);
            atomicAdd(aov.walk_counts + 2, wc.instances);
        } else {
            h = scene_closest(sc, o, d, tmin, tmax, ignored, error);
        }
        if (h.prim < 0) break;
        const Material m = sc.materials[material_of(sc, h.prim)];
        if (!is_passthrough(m)) {
            blocked = true;
            occluder = h.prim;
            occluder_t = h.t;
            break;
        }
        ++crossed;
        tr = tr * passthrough_transmittance(m);
        if (max_component(tr) <= 0) break;
        float adv = add(h.t, kRayEpsilon);
        if (adv >= tmax) break;
        o = o + d * adv;
        tmax = sub(tmax, adv);
        tmin = kRayEpsilon;
        ignored = -1;
    }
    if (!blocked && max_component(tr) > 0)
        add_radiance(rt, p, shadow_value(rt, p, tr, kAov || sc.has_passthrough));
    if (kAov && aov.shadow && rt.shadow[4 * static_cast<size_t>(p) + 3].w == 1.0f) {
        const int source = __float_as_int(b.w);
        const SceneTri tri = sc.tris[source];
        const f3 ng = triangle_normal(xyz(tri.v0), xyz(tri.v1), xyz(tri.v2));
        const float4 hh = rt.hit[p];
        f3 ns = shading_normal(sc.shading[source], ng, hh.y, hh.z);
        if (dot(ng, ns) < 0) ns = -ns;
        aov_add(aov.shadow, path_pixel(rt, p),
                shadow_aov_color(sc, source, ng, ns, d, occluder, occluder_t, crossed));
    }
}

LUX_D void warp_add(unsigned long long* counter, unsigned long long v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(counter, v);
}

}  // namespace
}  // namespace pt
}  // namespace lux
