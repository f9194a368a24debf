// Ray walk over the 4-wide nodes (WideNode), shared by the LBVH ray queries and the path
// tracer's TLAS and BLAS searches.
//
// Results are those of the reference's stackless walk (intersect_bvh_device_impl,
// bvh/bvh_device.cuh:43-90): leaves in left-first order, a box accepted when its slab
// entry does not exceed min(exit, best t), a triangle when t_min < t < best t.  The walk
// descends through the decoded (outward-rounded) child boxes, entering the first child
// that passes and deferring the others with their entry distances, resumed while the
// entry does not exceed the best t.  Decoded boxes contain the exact ones and the slab
// bounds are monotone in the box, so every leaf the reference reaches is reached here, in
// the same order; each leaf is then accepted by the exact test of its own box under the
// best t of that moment, which is the reference's verdict (its ancestors' exact boxes
// pass whenever the leaf's does).  The leaves tested and the best hit after each are
// therefore the reference's, so hit ids and t agree bit for bit.
#pragma once

#include "lux_bvh.cuh"

namespace lux {

// Deferred children of the deepest walk.  A path has at most 93 binary nodes (prefix lengths
// 1 to 63 of 63-bit codes, then 30 more of up to 2^30 equal ones' indices), a wide node takes
// two or more of them and defers at most three: 47 * 3 = 141.  (Room that is not used costs
// nothing: 2,048 to 4,194,304 rays of a 1M-triangle tree take the same at 116, 144 and 160.)
constexpr int kWideStack = 144;

LUX_D WideNode load_wide(const WideNode* wide, int i) {
    WideNode w;
    ldg8(wide + i, w.q0, w.q1);
    ldg8(reinterpret_cast<const float4*>(wide + i) + 2, w.q2, w.q3);
    return w;
}

LUX_D int wide_ref(const WideNode& w, int c) {
    return __float_as_int(c == 0 ? w.q2.z : c == 1 ? w.q2.w : c == 2 ? w.q3.x : w.q3.y);
}

// Slab verdict of one box under t_max (octant form when no axis is parallel).
LUX_D bool child_hit(const box3& b, const slab_ray& sr, const octant_ray& orr, float tmax,
                     float& tn) {
    return sr.parallel == 0 ? octant_hit(orr, b, tmax, tn) : slab_hit(sr, b, tmax, tn);
}

// Octant bits of a ray for wide_test (bit a: 1/d_a < 0), or kWideGeneral for a ray whose
// planes it may not take through the fused form: a parallel axis, or a direction so long
// that 1/d times a grid step could underflow.
constexpr unsigned kWideGeneral = 8u;
LUX_D unsigned wide_octant(const slab_ray& sr) {
    if (sr.parallel != 0) return kWideGeneral;
    const float least = fminf(fminf(fabsf(sr.inv.x), fabsf(sr.inv.y)), fabsf(sr.inv.z));
    if (!(least >= 8.6736174e-19f)) return kWideGeneral;   // 2^-60
    return (sr.inv.x < 0.0f ? 1u : 0u) | (sr.inv.y < 0.0f ? 2u : 0u) |
           (sr.inv.z < 0.0f ? 4u : 0u);
}

// r0 = q0 * a + b, r1 = q1 * a + b, each rounded once, by one packed instruction.
LUX_D void fma2(float q0, float q1, float a, float b, float& r0, float& r1) {
    asm("{.reg .b64 q, a, b, r;\n mov.b64 q, {%2, %3};\n mov.b64 a, {%4, %4};\n mov.b64 b, {%5, %5};\n"
        "fma.rn.f32x2 r, q, a, b;\n mov.b64 {%0, %1}, r;}"
        : "=f"(r0), "=f"(r1) : "f"(q0), "f"(q1), "f"(a), "f"(b));
}

// Hit verdicts p[c] of the node's child boxes under tmax, and for each child a bound tn[c]
// not above the entry t that the exact slab test computes for its exact box.  A child
// whose exact box passes passes here; one whose exact box fails may pass too (the walk's
// leaves are accepted by their exact boxes).
//
// A plane's t is one fused multiply-add, fma(2^15 + q, s * inv, (c - o) * inv), where the
// exact test subtracts and multiplies: with u = 2^-24 the two differ by at most
// 8u |t| + 0.016 |s * inv|.  The second term is half of what the planes were moved outward
// (kWideMargin); the first is taken off tn and put onto the exit t (2^-20 of each).
LUX_D void wide_test(const WideNode& w, const slab_ray& sr, unsigned oct, float tmax,
                     float tn[4], bool p[4]) {
    const unsigned lx = __float_as_uint(w.q1.x), ly = __float_as_uint(w.q1.y);
    const unsigned lz = __float_as_uint(w.q1.z), hx = __float_as_uint(w.q1.w);
    const unsigned hy = __float_as_uint(w.q2.x), hz = __float_as_uint(w.q2.y);
    const float sx = w.q3.z, sy = w.q3.w, sz = w.q0.w;
    const bool has2 = __float_as_int(w.q3.x) != kNoNode, has3 = __float_as_int(w.q3.y) != kNoNode;
    if (oct != kWideGeneral) {
        const unsigned nxq = (oct & 1u) ? hx : lx, fxq = (oct & 1u) ? lx : hx;
        const unsigned nyq = (oct & 2u) ? hy : ly, fyq = (oct & 2u) ? ly : hy;
        const unsigned nzq = (oct & 4u) ? hz : lz, fzq = (oct & 4u) ? lz : hz;
        const float ax = mul(sx, sr.inv.x), bx = mul(sub(w.q0.x, sr.o.x), sr.inv.x);
        const float ay = mul(sy, sr.inv.y), by = mul(sub(w.q0.y, sr.o.y), sr.inv.y);
        const float az = mul(sz, sr.inv.z), bz = mul(sub(w.q0.z, sr.o.z), sr.inv.z);
        constexpr float kSlack = 9.5367431640625e-07f;   // 2^-20
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float nx, fx, ny, fy, nz, fz;
            fma2(wide_biased(nxq, c), wide_biased(fxq, c), ax, bx, nx, fx);
            fma2(wide_biased(nyq, c), wide_biased(fyq, c), ay, by, ny, fy);
            fma2(wide_biased(nzq, c), wide_biased(fzq, c), az, bz, nz, fz);
            const float te = fmaxf(fmaxf(nx, ny), nz);
            const float tx = fminf(fminf(fx, fy), fz);
            tn[c] = fmaxf(sr.tmin, __fmaf_rn(fabsf(te), -kSlack, te));
            const float tf = fminf(tmax, __fmaf_rn(fabsf(tx), kSlack, tx));
            p[c] = !(tn[c] > tf);
        }
    } else {
        const octant_ray orr = make_octant_ray(sr);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const box3 b{make_f3(wide_decode(w.q0.x, lx, c, sx), wide_decode(w.q0.y, ly, c, sy),
                                 wide_decode(w.q0.z, lz, c, sz)),
                         make_f3(wide_decode(w.q0.x, hx, c, sx), wide_decode(w.q0.y, hy, c, sy),
                                 wide_decode(w.q0.z, hz, c, sz))};
            p[c] = child_hit(b, sr, orr, tmax, tn[c]);
        }
    }
    p[2] = p[2] && has2;
    p[3] = p[3] && has3;
}

// Deferred children of a walk, last in first out: the last one in registers, the others in
// memory as 8-byte (handle, entry t) records above a kNoNode record that ends the stack.
// With the last one at hand a pop does not wait for memory unless the record is skipped:
// its load of the next one is in flight while the walk tests the popped node.
struct WideTop {
    int h;
    float t;
    int sp;      // records in memory
    LUX_D void clear() {
        h = kNoNode;
        t = -INFINITY;
        sp = 0;
    }
    LUX_D bool full(int capacity) const { return sp + 3 > capacity; }
    LUX_D void push(int2* stack, int handle, float entry) {
        stack[sp] = make_int2(h, __float_as_int(t));
        ++sp;
        h = handle;
        t = entry;
    }
    // Takes the last record off; its handle when it still passes under best_t, kNoNode when
    // it does not (or when none is left).
    LUX_D int take(const int2* stack, float best_t) {
        if (h == kNoNode) return kNoNode;
        const int handle = t > best_t ? kNoNode : h;
        --sp;
        const int2 e = stack[sp];
        h = e.x;
        t = __int_as_float(e.y);
        return handle;
    }
    LUX_D int pop(const int2* stack, float best_t) {
        int handle = kNoNode;
        while (handle == kNoNode && h != kNoNode) handle = take(stack, best_t);
        return handle;
    }
};

// Goes down from node w: the first child that passes is returned (kNoNode when none does)
// and the others are deferred from right to left.  The caller has room for three records.
LUX_D int wide_descend(const WideNode& w, const float tn[4], const bool p[4], int2* stack,
                       WideTop& top) {
    if (p[3] && (p[0] || p[1] || p[2])) top.push(stack, wide_ref(w, 3), tn[3]);
    if (p[2] && (p[0] || p[1])) top.push(stack, wide_ref(w, 2), tn[2]);
    if (p[1] && p[0]) top.push(stack, wide_ref(w, 1), tn[1]);
    return p[0] ? wide_ref(w, 0)
                : p[1] ? wide_ref(w, 1) : p[2] ? wide_ref(w, 2) : p[3] ? wide_ref(w, 3) : kNoNode;
}

// Moves a walk that is past cur on: a leaf in cur goes to the free place `leaf`, and cur
// becomes the next deferred record that passes; it stops at a node, at a second leaf, or
// with nothing left (cur == kNoNode).
LUX_D void wide_move_on(int& cur, int& leaf, const int2* stack, WideTop& top, float best_t) {
    for (;;) {
        if (cur < 0 && cur != kNoNode && leaf == kNoNode) {
            leaf = cur;
            cur = kNoNode;
        }
        if (cur != kNoNode || top.h == kNoNode) return;
        cur = top.take(stack, best_t);
    }
}

// The reference's verdict on sorted leaf k's own box under the current best t.
LUX_D bool leaf_hit(const BvhView& b, int k, const slab_ray& sr, const octant_ray& orr,
                    float best_t) {
    float tn;
    return child_hit(leaf_box(b, k), sr, orr, best_t, tn);
}

// Sorted leaf k's triangle record (p0, p1, p2) and the verdict on the leaf's exact box.
// In a BVH built from triangles the leaf box is the triangle's own box, formed here from
// the record's vertices exactly as the build formed it, so the leaf costs one 48-byte
// record load and no parent-slot load.
LUX_D bool leaf_record_hit(const BvhView& b, int k, const slab_ray& sr, const octant_ray& orr,
                           float best_t, float4& p0, float4& p1, float4& p2) {
    const float4* tp = reinterpret_cast<const float4*>(b.tris + k);
    p0 = __ldg(tp);
    p1 = __ldg(tp + 1);
    p2 = __ldg(tp + 2);
    if (!b.leaf_is_triangle_box) return leaf_hit(b, k, sr, orr, best_t);
    float tn;
    return child_hit(triangle_box(make_f3(p0.x, p0.y, p0.z), make_f3(p1.x, p1.y, p1.z),
                                  make_f3(p2.x, p2.y, p2.z)),
                     sr, orr, best_t, tn);
}

// Walks bvh from its root for a ray with slab constants sr; leaf(k, p0, p1, p2, best_t)
// tests sorted leaf k (its triangle record p0..p2), may lower best_t, and returns true to
// end the walk (any-hit).  Returns false after setting an error bit (loop bound or stack
// overflow).
template <typename Leaf>
LUX_D bool wide_walk(const BvhView& b, const slab_ray& sr, float& best_t, int* error,
                     Leaf&& leaf) {
    if (b.n <= 0) return true;
    float tn0;
    if (!slab_hit(sr, load_root(b.root), best_t, tn0)) return true;
    const octant_ray orr = make_octant_ray(sr);
    const unsigned oct = wide_octant(sr);
    int2 stack[kWideStack];  // (node ref, entry t bits)
    WideTop top;
    top.clear();
    int cur = b.n == 1 ? ~0 : 0;
    const long long bound = 2ll * b.n + 64;
    for (long long step = 0; cur != kNoNode; ++step) {
        if (step > bound || cur >= b.n - 1 || ~cur >= b.n) {
            atomicOr(error, kErrLoopBound);
            return false;
        }
        int next = kNoNode;
        if (cur >= 0) {
            if (top.full(kWideStack)) {
                atomicOr(error, kErrStackOverflow);
                return false;
            }
            const WideNode w = load_wide(b.wide, cur);
            float t[4];
            bool p[4];
            wide_test(w, sr, oct, best_t, t, p);
            next = wide_descend(w, t, p, stack, top);
        } else {
            float4 p0, p1, p2;
            if (leaf_record_hit(b, ~cur, sr, orr, best_t, p0, p1, p2) &&
                leaf(~cur, p0, p1, p2, best_t))
                return true;
        }
        cur = next != kNoNode ? next : top.pop(stack, best_t);
    }
    return true;
}

}  // namespace lux
