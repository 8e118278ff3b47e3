// Occlusion of a whole tile by one triangle.
//
// The segments from a point (or a short line) to the receivers of a tile form
// a thin convex shaft.  When one triangle cuts every segment between the
// shaft's end vertices strictly inside its edges, it cuts every segment in
// between: for a fixed end the crossing point is a projective map of the other
// end, so it stays in the hull of the crossings at the vertices, which lies in
// the (convex) triangle.  One lane then settles a pair of 32 segments with one
// traversal of the shaft's centre line, and a warp tests 32 shafts at a time;
// only shafts without such a triangle go on to the per-cell traversal.
//
// The test answers "blocked" only with margins far above the FP32 error of the
// per-cell traversal (positions within about 5e-7 M, M the largest coordinate
// 1-norm, over the sine of the angle to the triangle's plane), so it never
// changes a visibility bit.
#pragma once

#include "traverse.cuh"

namespace wcb {

struct Shaft {
    V3<float> a[2];      // vertices of the near end
    int na;
    float lo[3], hi[3];  // box of the far end
    float size;          // largest coordinate 1-norm of both ends
    // occluders must lie on the far end's side of this plane (side 0: no plane)
    float pn[3], poff, side;
};

WCB_D float norm1(V3<float> v) { return fabsf(v.x) + fabsf(v.y) + fabsf(v.z); }

// Does triangle (v0, v1, v2) cut every segment between a[.] and the box?
WCB_D bool triangle_cuts_shaft(const Shaft& s, V3<float> v0, V3<float> v1, V3<float> v2) {
    const float size = fmaxf(s.size, fmaxf(norm1(v0), fmaxf(norm1(v1), norm1(v2))));
    const float margin = 1e-4f + 2e-5f * size;
    if (s.side != 0.f) {
        const V3<float> pn = v3(s.pn[0], s.pn[1], s.pn[2]);
        if (!(s.side * (dot(pn, v0) - s.poff) > margin && s.side * (dot(pn, v1) - s.poff) > margin &&
              s.side * (dot(pn, v2) - s.poff) > margin))
            return false;
    }
    const V3<float> e0 = v1 - v0, e1 = v2 - v1, e2 = v0 - v2;
    V3<float> n = cross(e0, v2 - v0);
    const float nl = dot(n, n);
    if (!(nl > 1e-12f)) return false;
    n = n * rsqrtf(nl);
    // the near end strictly on one side, the box on the other
    float ha[2];
    ha[0] = dot(n, s.a[0] - v0);
    ha[1] = s.na > 1 ? dot(n, s.a[1] - v0) : ha[0];
    const float sg = ha[0] > 0.f ? 1.f : -1.f;
    if (!(sg * ha[0] > margin && sg * ha[1] > margin)) return false;
    const float hc = dot(n, v3(0.5f * (s.lo[0] + s.hi[0]), 0.5f * (s.lo[1] + s.hi[1]), 0.5f * (s.lo[2] + s.hi[2])) - v0);
    const float hr = 0.5f * (fabsf(n.x) * (s.hi[0] - s.lo[0]) + fabsf(n.y) * (s.hi[1] - s.lo[1]) +
                             fabsf(n.z) * (s.hi[2] - s.lo[2]));
    if (!(sg * hc + hr < -margin)) return false;
    // inward edge normals in the triangle's plane
    V3<float> m[3] = {cross(n, e0), cross(n, e1), cross(n, e2)};
    float off[3];
    m[0] = m[0] * rsqrtf(dot(e0, e0));
    m[1] = m[1] * rsqrtf(dot(e1, e1));
    m[2] = m[2] * rsqrtf(dot(e2, e2));
    const int layers = s.lo[2] < s.hi[2] ? 2 : 1;
#pragma unroll 1
    for (int k = 0; k < s.na; ++k) {
        const V3<float> a = s.a[k];
        off[0] = dot(m[0], v0 - a);
        off[1] = dot(m[1], v1 - a);
        off[2] = dot(m[2], v2 - a);
#pragma unroll 1
        for (int q = 0; q < 4 * layers; ++q) {
            const V3<float> d = v3((q & 1) ? s.hi[0] : s.lo[0], (q & 2) ? s.hi[1] : s.lo[1],
                                   (q & 4) ? s.hi[2] : s.lo[2]) - a;
            // crossing at a + d t, t = ha / -(n.d)
            const float fall = -dot(n, d);
            const float inv = __fdividef(1.f, fall);
            const float t = ha[k] * inv;
            const float pad = 1e-4f + 1e-5f * size * fabsf(inv) * norm1(d);
            if (!(dot(m[0], d) * t - off[0] > pad && dot(m[1], d) * t - off[1] > pad && dot(m[2], d) * t - off[2] > pad))
                return false;
        }
    }
    return true;
}

// Search of the shaft's centre line for a triangle outside `ig` that cuts the
// whole shaft, in resumable pieces: node() descends to the next leaves, test()
// tries one leaf.  A warp that settles many shafts runs the two apart, so the
// long triangle test is taken by many lanes at once, and a lane that is done
// takes its next shaft.
struct ShaftSearch {
    V3<float> o, inv;
    int next, sp;      // next node or (single-triangle scene) leaf; kNone when nothing is left
    int leaf0, leaf1;  // leaves to try (0: none)
    static constexpr int kNone = 0x7fffffff;

    WCB_D void start(const SceneDev& sc, V3<float> p0, V3<float> p1) {
        const Ray<float> r = make_ray<float>(p0, p1 - p0, 1e-6f, 1.f - 1e-6f);
        o = r.o;
        inv = r.inv;
        sp = 0;
        leaf1 = 0;
        leaf0 = sc.root < 0 ? sc.root : 0;
        next = sc.root < 0 ? kNone : sc.root;
    }
    WCB_D bool done() const { return leaf0 == 0 && next == kNone; }

    WCB_D void node(const SceneDev& sc, int* stack) {
        Ray<float> r;
        r.o = o;
        r.inv = inv;
        r.tmin = 1e-6f;
        const int stride = blockDim.x, lane = threadIdx.x;
        float4 a, b, c;
        int4 d;
        load_node(sc.nodes, next, a, b, c, d);
        float n0, n1;
        const bool h0 = box_hit(r, a.x, a.y, a.z, a.w, b.x, b.y, 1.f - 1e-6f, &n0);
        const bool h1 = box_hit(r, b.z, b.w, c.x, c.y, c.z, c.w, 1.f - 1e-6f, &n1);
        const int l0 = h0 && d.x < 0 ? d.x : 0, l1 = h1 && d.y < 0 ? d.y : 0;
        leaf0 = l0 ? l0 : l1;
        leaf1 = l0 ? l1 : 0;
        const bool in0 = h0 && d.x >= 0, in1 = h1 && d.y >= 0;
        // a full stack drops the far child: it can only leave the shaft unsettled
        if (in0 && in1 && sp < sc.stack_entries) stack[sp++ * stride + lane] = d.y;
        if (in0 || in1) next = in0 ? d.x : d.y;
        else next = sp > 0 ? stack[--sp * stride + lane] : kNone;
    }

    // Does the next leaf's triangle cut the shaft?
    WCB_D bool test(const SceneDev& sc, const Ignore& ig, const Shaft& s) {
        const int slot = ~leaf0;
        leaf0 = leaf1;
        leaf1 = 0;
        const float4 a = __ldg(sc.tri + 3 * slot + 0);
        const float4 b = __ldg(sc.tri + 3 * slot + 1);
        const float4 c = __ldg(sc.tri + 3 * slot + 2);
        return !ignored(ig, __float_as_int(a.w), __float_as_int(b.w)) &&
               triangle_cuts_shaft(s, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z));
    }
};

WCB_D bool shaft_blocked(const SceneDev& sc, V3<float> p0, V3<float> p1, const Ignore& ig, const Shaft& s, int* stack) {
    if (sc.num_faces == 0) return false;
    ShaftSearch q;
    q.start(sc, p0, p1);
    while (!q.done()) {
        while (q.leaf0 == 0 && q.next != ShaftSearch::kNone) q.node(sc, stack);
        if (q.leaf0 != 0 && q.test(sc, ig, s)) return true;
    }
    return false;
}

}  // namespace wcb
