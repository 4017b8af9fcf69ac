// The discrete triangle distance (tri_tri_dist, comparison_dist.h:12-189) with
// the sub-tests that cannot matter left out.
//
// tri_tri_dist takes the closest of 15 features (six vertex-plane projections,
// nine edge pairs), lets six edge-plane intersections override it, and its
// callers read the result only when the distance is below a limit.  One FP64
// instruction costs as much as 64 FP32 ones on this GPU, so every feature is
// first bounded in FP32 from coordinates relative to a's first vertex:
//   * an intersection is evaluated unless both ends of the edge are on one side
//     of the plane, or the crossing point is outside the triangle, by more than
//     the errors involved;
//   * a projection is left out when its barycentric coordinates are outside,
//     an edge pair or projection when a lower bound of its distance passes the
//     limit or a distance already found.  The lower bound is the gap between
//     the two features along some direction, which holds whatever the
//     direction is; FP32 only has to find a good one.
// What is left (2 to 3 features of 21 for separate triangles) is evaluated by
// the FP64 code of tri_tri_dist and the closest taken in its order (the first
// of equal distances), so P, Q and the distance are the same bits whenever the
// distance is below the limit; otherwise the returned distance is only known
// to be no smaller than the limit (or NaN).
//
// tri_tri_dist of two triangles none of whose features has a distance (a
// triangle that is a point, coordinates that are not finite) is 0 at the
// origin: what all its comparisons leave.  Triangles that are not tri_regular,
// or kFarSizes away, take the plain function, which alone knows.
#pragma once
#include "d2g_geom.cuh"

namespace d2g {

struct F3 {
    float x, y, z;
};
D2G_HD F3 f3(float x, float y, float z) {
    F3 r;
    r.x = x;
    r.y = y;
    r.z = z;
    return r;
}
D2G_HD F3 operator-(F3 a, F3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
// Fused where that saves an instruction: only a bound's quality depends on it.
D2G_HD F3 fma3(F3 d, float s, F3 p) { return f3(fmaf(d.x, s, p.x), fmaf(d.y, s, p.y), fmaf(d.z, s, p.z)); }
D2G_HD float dot3(F3 a, F3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }
D2G_HD F3 cross3(F3 a, F3 b) {
    return f3(fmaf(a.y, b.z, -(a.z * b.y)), fmaf(a.z, b.x, -(a.x * b.z)), fmaf(a.x, b.y, -(a.y * b.x)));
}
// x / y to a few ulps.
D2G_HD float div_fast(float x, float y) {
#ifdef __CUDA_ARCH__
    return __fdividef(x, y);
#else
    return x / y;
#endif
}
D2G_HD float clampf01(float t) { return t > 0.f ? (t < 1.f ? t : 1.f) : 0.f; }  // NaN: 0
D2G_HD F3 rel3(V3 p, V3 o) { return f3((float)(p.x - o.x), (float)(p.y - o.y), (float)(p.z - o.z)); }
D2G_HD float maxabs3(F3 a) { return fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)); }

// The closest points of segments S0 S1 and E0 E1 (approximately): the vector
// between them and its squared length.
D2G_HD F3 seg_vector(F3 S0, F3 S1, F3 E0, F3 E1, float& d2) {
    const F3 u = S1 - S0, v = E1 - E0, w = S0 - E0;
    const float a = dot3(u, u), b = dot3(u, v), c = dot3(v, v), d = dot3(u, w), e = dot3(v, w);
    const float s = clampf01(div_fast(fmaf(b, e, -(c * d)), fmaf(a, c, -(b * b))));
    const float t = clampf01(div_fast(fmaf(b, s, e), c));
    const float s2 = clampf01(div_fast(fmaf(b, t, -d), a));
    const F3 n = fma3(v, t, E0) - fma3(u, s2, S0);
    d2 = dot3(n, n);
    return n;
}

// Edges p[][0] p[][1] and p[][2] p[][3] at the start and at the end of a motion
// on straight lines: further apart than lim all along, because the gap along
// the direction between their closest points at the start, concave in time, is
// so at both ends.  Closest points within 1e-15 give no direction: the length
// of one below 1e-20 underflows, and any gap would pass for a large one.
D2G_HD bool edges_stay_apart(const F3 (&p)[2][4], float lim) {
    float d2, g[2];
    const F3 d = seg_vector(p[0][0], p[0][1], p[0][2], p[0][3], d2);
    for (int m = 0; m < 2; m++)
        g[m] = fminf(dot3(d, p[m][2]), dot3(d, p[m][3])) - fmaxf(dot3(d, p[m][0]), dot3(d, p[m][1]));
    return d2 > 1e-30f && fminf(g[0], g[1]) > lim * sqrtf(d2);
}

// Two of the triangle's edges, taken from its vertices relative to the other's,
// are neither points nor out of range: with another such triangle some edge
// pair has a finite distance.  s: the squared lengths of the edges at the first
// vertex.
D2G_HD bool tri_regular(float s) { return s > 1e-30f && s < 1e30f; }  // false for NaN
// A triangle further from the origin than this many of its sizes: FP64 rounding
// at its place, 1e-16 of the distance, comes near the bounds' margin of its
// barycentric coordinates (1e-5).
constexpr float kFarSizes = 1e10f;

// tri_tri_dist, out of line: hardly ever called beside the bounds.
#ifdef __CUDA_ARCH__
static __device__ __noinline__
#else
inline
#endif
double tri_tri_dist_plain(const Tri& a, const Tri& b, V3& P, V3& Q) { return tri_tri_dist(a, b, P, Q); }

// What the bounds read of a triangle's plane.
struct PlaneBound {
    F3 o, v0, v1, n;      // first vertex, edges, v0 x v1
    float d00, d01, d11, inv, len;  // dots, 1 / (d00 d11 - d01^2), |n|
    float mb;             // margin of a barycentric coordinate
    float eh;             // margin of a height n . (p - o), per unit of max(|p - o|, edges)
    float flat;           // largest height of the triangle's own vertices over n
    bool ok;              // conditioned well enough for the bounds
};
// rho: the largest relative coordinate of the two triangles.  The barycentric
// margin covers the reference's float barycentrics, whose error grows with the
// triangle's conditioning k = d00 d11 / det, and the FP32 coordinates here.
D2G_HD PlaneBound plane_bound(F3 a, F3 b, F3 c, float rho) {
    PlaneBound p;
    p.o = a;
    p.v0 = b - a;
    p.v1 = c - a;
    p.n = cross3(p.v0, p.v1);
    p.d00 = dot3(p.v0, p.v0);
    p.d01 = dot3(p.v0, p.v1);
    p.d11 = dot3(p.v1, p.v1);
    const float det = p.d00 * p.d11 - p.d01 * p.d01;
    p.inv = 1.f / det;
    const float l0 = sqrtf(p.d00), l1 = sqrtf(p.d11);
    const float k = p.d00 * p.d11 * p.inv, s = 1.f + rho / fminf(l0, l1);
    p.mb = 1e-5f * k * s;
    p.len = sqrtf(dot3(p.n, p.n));
    p.eh = 2e-6f * (l0 * l1 + rho * (l0 + l1));
    p.flat = fmaxf(fabsf(dot3(p.n, p.v0)), fabsf(dot3(p.n, p.v1)));
    p.ok = det > 0.f && k >= 0.f && p.mb < 0.05f && p.len > 0.f;  // false for NaN
    return p;
}
D2G_HD void plane_bary(const PlaneBound& p, F3 q, float& u, float& v, float& w) {
    const float d20 = dot3(q, p.v0), d21 = dot3(q, p.v1);
    v = (p.d11 * d20 - p.d01 * d21) * p.inv;
    w = (p.d00 * d21 - p.d01 * d20) * p.inv;
    u = 1.f - v - w;
}
// The crossing of edge s e (heights hs, he over T's plane) certainly not
// inside T.
D2G_HD bool no_crossing(const PlaneBound& p, F3 s, F3 e, float hs, float he) {
    if (!p.ok) return false;
    const F3 qs = s - p.o, qe = e - p.o;
    const float r = fmaxf(maxabs3(qs), maxabs3(qe));
    const float err = 2.f * p.eh * r + 1e-30f;
    if ((hs > err && he > err) || (hs < -err && he < -err)) return true;
    const float dh = fabsf(hs - he);
    if (!(dh > 8.f * err)) return false;
    const float t = hs / (hs - he), dt = 4.f * err / dh;
    float u, v, w;
    plane_bary(p, fma3(qe - qs, t, qs), u, v, w);
    // the crossing point moves by dt along the edge at most; its barycentric
    // coordinates by that over the edges' heights
    const F3 D = qe - qs;
    const float lmin = sqrtf(fminf(p.d00, p.d11));
    const float m = p.mb + dt * sqrtf(dot3(D, D)) * (p.d00 * p.d11 * p.inv) / lmin * 2.f;
    return u < -m || v < -m || w < -m;  // false for NaN
}

D2G_HD int lowest_bit(unsigned m) {
#ifdef __CUDA_ARCH__
    return __ffs((int)m) - 1;
#else
    return __builtin_ctz(m);
#endif
}

// tri_tri_dist(a, b, P, Q) where the result is below `limit`; else a distance
// of at least `limit` (or NaN), with P and Q meaningless.
D2G_HD double tri_tri_dist_below(const Tri& a, const Tri& b, double limit, V3& P, V3& Q) {
    const V3 o = a.A;
    F3 A[3], B[3];
    A[0] = f3(0.f, 0.f, 0.f);
    A[1] = rel3(a.B, o);
    A[2] = rel3(a.C, o);
    B[0] = rel3(b.A, o);
    B[1] = rel3(b.B, o);
    B[2] = rel3(b.C, o);
    float rho = 0.f;
    for (int i = 0; i < 3; i++) rho = fmaxf(rho, fmaxf(maxabs3(A[i]), maxabs3(B[i])));
    // the FP32 coordinates' error, and the FP64 evaluation's at world scale
    const float mag = (float)(fabs(o.x) + fabs(o.y) + fabs(o.z));
    const float margin = 4e-6f * rho + 1e-13f * mag + 1e-30f;
    const PlaneBound pa = plane_bound(A[0], A[1], A[2], rho), pb = plane_bound(B[0], B[1], B[2], rho);
    const float sa = pa.d00 + pa.d11, sb = pb.d00 + pb.d11;
    if (!(tri_regular(sa) && tri_regular(sb) && mag < kFarSizes * sqrtf(fminf(sa, sb)))) {
        const Tri ca = a, cb = b;  // (in memory for the call; a, b, P and Q stay in registers)
        V3 p, q;
        const double d = tri_tri_dist_plain(ca, cb, p, q);
        P = p;
        Q = q;
        return d;
    }
    float hB[3], hA[3];  // heights of b's vertices over a's plane and of a's over b's
#pragma unroll
    for (int i = 0; i < 3; i++) {
        hB[i] = dot3(pa.n, B[i] - pa.o);
        hA[i] = dot3(pb.n, A[i] - pb.o);
    }
    const float flimit = (float)limit * (1.f + 1e-6f);
    // ---- intersections: the last one found decides
    unsigned cross = 0;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int j1 = j == 2 ? 0 : j + 1;
        if (!no_crossing(pa, B[j], B[j1], hB[j], hB[j1])) cross |= 1u << j;
        if (!no_crossing(pb, A[j], A[j1], hA[j], hA[j1])) cross |= 8u << j;
    }
    bool any = false;
    V3 X = mk(0, 0, 0);
    while (cross) {
        const int k = lowest_bit(cross);
        cross &= cross - 1;
        double t;
        bool t_inf, isInt;
        const bool on_a = k < 3;
        const Edge e = tedge(on_a ? b : a, on_a ? k : k - 3);
        tri_intersect_segment(on_a ? a : b, e.A, e.B, t, t_inf, isInt);
        if (isInt) {
            X = lerp(e.A, e.B, t);
            any = true;
        }
    }
    if (any) {
        P = X;
        Q = X;
        return norm(X - X);
    }
    // ---- lower bounds of the 15 features, and the most promising one
    float lb[15];
    float best_est = 3.4e38f;
    int first = 6;
#pragma unroll
    for (int i = 0; i < 6; i++) {  // 0-2: b's vertices on a's plane, 3-5: a's on b's
        const PlaneBound& p = i < 3 ? pa : pb;
        const F3 q = (i < 3 ? B[i] : A[i - 3]) - p.o;
        const float h = fabsf(i < 3 ? hB[i] : hA[i - 3]);
        lb[i] = 0.f;
        if (p.ok) {
            float u, v, w;
            plane_bary(p, q, u, v, w);
            const float m = p.mb;
            if (u < -m || v < -m || w < -m) {
                lb[i] = 3.4e38f;
            } else {
                const float gap = (h - p.flat - p.eh * rho) / p.len;
                lb[i] = gap - margin - 2.f * m * sqrtf(fmaxf(p.d00, p.d11));
                if (u > m && v > m && w > m && h < best_est * p.len) {
                    best_est = h / p.len;
                    first = i;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const F3 S0 = A[i], S1 = A[i == 2 ? 0 : i + 1], E0 = B[j], E1 = B[j == 2 ? 0 : j + 1];
            float d2;
            const F3 n = seg_vector(S0, S1, E0, E1, d2);
            const float d = sqrtf(d2);
            const float gap = (fminf(dot3(n, E0), dot3(n, E1)) - fmaxf(dot3(n, S0), dot3(n, S1))) / d;
            lb[6 + 3 * i + j] = gap > 0.f && d2 > 1e-30f ? gap - margin : 0.f;  // NaN: 0 (edges_stay_apart)
            if (d < best_est) {
                best_est = d;
                first = 6 + 3 * i + j;
            }
        }
    // ---- the most promising feature, then those it and the limit leave
    V3 Pc = mk(0, 0, 0), Qc = mk(0, 0, 0);
    double dc = 1.0 / 0.0;
    int at = 15;
    unsigned todo = 1u << first, done = 0;
    for (int round = 0; round < 2; round++) {
        if (round) {
            const float lim = fminf((float)dc * (1.f + 1e-6f), flimit);
            todo = 0;
#pragma unroll
            for (int k = 0; k < 15; k++)
                if (!(lb[k] > lim)) todo |= 1u << k;  // NaN limit or bound: kept
            todo &= ~done;
        } else if (!(lb[0] <= flimit) && !(lb[1] <= flimit) && !(lb[2] <= flimit) && !(lb[3] <= flimit) &&
                   !(lb[4] <= flimit) && !(lb[5] <= flimit) && !(lb[6] <= flimit) && !(lb[7] <= flimit) &&
                   !(lb[8] <= flimit) && !(lb[9] <= flimit) && !(lb[10] <= flimit) && !(lb[11] <= flimit) &&
                   !(lb[12] <= flimit) && !(lb[13] <= flimit) && !(lb[14] <= flimit) && flimit == flimit) {
            return 1.0 / 0.0;  // no feature below the limit
        }
        done |= todo;
        unsigned v = todo & 63u, e = todo >> 6;
        while (v) {
            const int k = lowest_bit(v);
            v &= v - 1;
            const bool on_a = k < 3;
            const V3 p = on_a ? tvert(b, k) : tvert(a, k - 3);
            bool in;
            const V3 on = tri_project_to_plane(on_a ? a : b, p, in);
            if (!in) continue;
            const V3 Pk = on_a ? on : p, Qk = on_a ? p : on;
            const double d = norm(Pk - Qk);
            if (d < dc || (d == dc && k < at && at < 15)) {
                Pc = Pk;
                Qc = Qk;
                dc = d;
                at = k;
            }
        }
        while (e) {
            const int k = lowest_bit(e);
            e &= e - 1;
            const Edge ea = tedge(a, k / 3), eb = tedge(b, k % 3);
            V3 Pk, Qk;
            const double d = edge_closest(ea.A, ea.B, eb.A, eb.B, Pk, Qk);
            if (d < dc || (d == dc && 6 + k < at && at < 15)) {
                Pc = Pk;
                Qc = Qk;
                dc = d;
                at = 6 + k;
            }
        }
    }
    P = Pc;
    Q = Qc;
    return at < 15 ? norm(Pc - Qc) : 1.0 / 0.0;
}

}  // namespace d2g
