// Level-synchronous surrogate-tree traversal on the GPU, for all body pairs
// of a call at once.
//
// The reference walks one body pair at a time, level by level
// (collision_detection/full_tree_comparison.h:13-219).  Here every frontier
// holds the node pairs of ALL body pairs, sorted by body pair and, within a
// pair, in the reference's order; every expansion is an ordered compaction
// (prefix sums), so the contacts of each pair come out in exactly the order
// the reference's sequential loops produce them.
//
// The descent only needs to know which node pairs have a hit; leaf pairs end
// it.  So a level decides its node pairs (FP32 where the answer is certain,
// the FP64 tests until the first hit where it is not) and puts the leaf pairs
// it opens onto one list, and all leaf pairs of the call are tested in FP64 at
// once after the last level: one chain of the slowest tests instead of one per
// level, and enough tests to fill the GPU.
// All arithmetic is FP64 with -fmad=false, in the order declared in
// d2g_geom.cuh, so results equal the CPU restatement bit for bit.
#include <cub/cub.cuh>

#include <mutex>
#include <string>

#include "d2g_geom.cuh"
#include "d2g_internal.hpp"
#include "d2g_limits.hpp"
#include "d2g_prune.cuh"

namespace d2g {

namespace {

constexpr int kBlock = 128;

inline int nblocks(long long n, int b = kBlock) { return (int)((n + b - 1) / b); }

__device__ __forceinline__ int4 ld_node(const int4* nodes, int g) { return nodes[g]; }

// ------------------------------------------------------------- CCD prep ----
// Projects both futures over the pair's max_time (model/state.cpp:90-102,
// full_tree_comparison.h:78-79) and forms the pose matrices.
// Per pair: the futures over max_time, the pose matrices (pair_mats) and the
// root frontier entry.  Four lanes per pair: lanes 1 and 3 extrapolate a and
// b, lane k forms transform k (a start, a end, b start, b end) and then the
// product inverse(transform k^2) * transform k, so the four 4x4 inverses and
// products run side by side.
__global__ void k_ccd_prep(int n, const int32_t* __restrict__ pairs, const double* __restrict__ max_time,
                           const double* __restrict__ cur, const double* __restrict__ ii,
                           const int32_t* __restrict__ mesh, const int32_t* __restrict__ mesh_node_off,
                           const double* __restrict__ geo_eps, double* __restrict__ pm, double* __restrict__ pfut,
                           float* __restrict__ search, Entry* __restrict__ soup) {
    const int p = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 2);
    const int k = threadIdx.x & 3;
    if (p >= n) return;  // uniform per quad
    const unsigned qm = 0xFu << (threadIdx.x & 28);
    const int body = pairs[2 * p + (k >> 1)];
    const State c = load_state(cur + 14 * (size_t)body);
    State st = c;
    if (k & 1) {
        st = extrapolate(c, max_time[p], ii + 9 * (size_t)body);
        store_state(pfut + 28 * (size_t)p + 14 * (k >> 1), st);
    }
    double* M = pm + (size_t)PM_SIZE * p;
    double T[16], O[16], inv[16], R[16];
    transformation(st.q, st.x, T);
#pragma unroll
    for (int i = 0; i < 16; i++) {
        M[16 * k + i] = T[i];
        O[i] = __shfl_xor_sync(qm, T[i], 2);
    }
    mat_inverse(O, inv);
    mat_mul(inv, T, R);
#pragma unroll
    for (int i = 0; i < 16; i++) M[PM_ABS + 16 * k + i] = R[i];
    if (k == 0) {
        const int a = pairs[2 * p], b = pairs[2 * p + 1];
        search[p] = (float)(geo_eps[a] + geo_eps[b]);
        Entry e;
        e.pair = p;
        e.na = mesh_node_off[mesh[a]];
        e.nb = mesh_node_off[mesh[b]];
        soup[p] = e;
    }
}

// Discrete narrow phase prep: future transforms of a and b (comparison_dist.h:225,229).
// A pose's rotation comes from the state's quaternion as it is, which a caller
// may have set to any length: it keeps distances (to 3e-6 of themselves) when
// its columns are orthonormal to 2e-6, FP32 rounding taking 3e-7 of that.
__device__ __forceinline__ bool keeps_distances(const double* __restrict__ M) {
    const F3 x = f3((float)M[0], (float)M[4], (float)M[8]), y = f3((float)M[1], (float)M[5], (float)M[9]),
             z = f3((float)M[2], (float)M[6], (float)M[10]);
    const float d = fmaxf(fmaxf(fabsf(dot3(x, y)), fabsf(dot3(y, z))), fabsf(dot3(z, x)));
    const float l = fabsf(dot3(x, x) - 1.f) + fabsf(dot3(y, y) - 1.f) + fabsf(dot3(z, z) - 1.f);
    return d < 2e-6f && l < 2e-6f;  // false for NaN: l is one then
}

// The discrete phase's FP32 poses: rows 0-2 of both, then whether both keep
// distances.
constexpr int kNpPose32 = 25;
__global__ void k_np_prep(int n, const int32_t* __restrict__ pairs, const double* __restrict__ fut,
                          const int32_t* __restrict__ mesh, const int32_t* __restrict__ mesh_node_off,
                          const double* __restrict__ geo_eps, double* __restrict__ pm, float* __restrict__ search,
                          Entry* __restrict__ front, float* __restrict__ pm32, const int32_t* __restrict__ err) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n || (err && *err)) return;
    const int a = pairs[2 * p], b = pairs[2 * p + 1];
    const State fa = load_state(fut + 14 * (size_t)a);
    const State fb = load_state(fut + 14 * (size_t)b);
    double* M = pm + 32 * (size_t)p;
    transformation(fa.q, fa.x, M);
    transformation(fb.q, fb.x, M + 16);
    if (pm32) {
        for (int k = 0; k < 12; k++) {
            pm32[kNpPose32 * (size_t)p + k] = (float)M[k];
            pm32[kNpPose32 * (size_t)p + 12 + k] = (float)M[16 + k];
        }
        pm32[kNpPose32 * (size_t)p + 24] = keeps_distances(M) && keeps_distances(M + 16) ? 1.f : 0.f;
    }
    search[p] = (float)(geo_eps[a] + geo_eps[b]);
    Entry e;
    e.pair = p;
    e.na = mesh_node_off[mesh[a]];
    e.nb = mesh_node_off[mesh[b]];
    front[p] = e;
}

// ------------------------------------------------------------ soup stage ---
__global__ void k_compact(int n, const int32_t* __restrict__ flags, const int32_t* __restrict__ off,
                          int32_t* __restrict__ items) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (flags[i]) items[off[i]] = i;
}

__device__ __forceinline__ void put_result(PrimResult& r, double dist, V3 A, V3 B, double toc) {
    r.dist = dist;
    r.P[0] = A.x;
    r.P[1] = A.y;
    r.P[2] = A.z;
    r.Q[0] = B.x;
    r.Q[1] = B.y;
    r.Q[2] = B.z;
    r.toc = toc;
}

// ------------------------------------------- flattened primitive tests -----
// One level of the CCD as two homogeneous work lists: every point-triangle
// test and every edge-edge test of the level, from the soup stage (the 15
// sub-tests of each surviving triangle pair, continuous_comparison.h:692-777)
// and from the connected stage (all tests of each leaf pair, :855-907).
// Point-triangle list: 6 per soup triangle pair, then 6*na*nb per leaf pair;
// edge-edge list: 9 per soup triangle pair, then 9*na*nb per leaf pair.  The
// soup sub-results are folded afterwards in the reference's order.
constexpr int kPrimBlock = 64;

__global__ void k_conn_nn(int n, const Entry* __restrict__ conn, const int32_t* __restrict__ ntris,
                          int32_t* __restrict__ cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Entry e = conn[i];
    cnt[i] = ntris[e.na] * ntris[e.nb];
}

// The leaf pair of every leaf-pair triangle pair: tp[off[e] .. off[e + 1]) = e,
// a warp per leaf pair.  Test j of a list with m tests per triangle pair
// belongs to leaf pair tp[j / m] (a search of off in every test kernel before).
__global__ void k_tp_fill(int n, const int32_t* __restrict__ off, int32_t* __restrict__ tp) {
    const int e = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    if (e >= n) return;
    for (int k = off[e] + (threadIdx.x & 31); k < off[e + 1]; k += 32) tp[k] = e;
}

__device__ __forceinline__ void store_prim(PrimResult* __restrict__ r, double dist, V3 A, V3 B, double toc) {
    r->dist = dist;
    r->P[0] = A.x;
    r->P[1] = A.y;
    r->P[2] = A.z;
    r->Q[0] = B.x;
    r->Q[1] = B.y;
    r->Q[2] = B.z;
    r->toc = toc;
}

// ---------------------------------------------- FP32 candidate filtering ---
// Every primitive CCD test returns a distance between a point of a box built
// from its inputs and a point of a second box: for edgeEdgeCCD the world
// positions of the two edges' endpoints at the start and the end; for
// pointTriCCDLinear the point carried into the triangle's frame at the start
// and the end, then through the triangle body's start and end transforms, and
// the triangle's vertices through the same two transforms (the returned
// points are lerps of those).  A box gap above the hit threshold means the
// test cannot hit (a soup sub-test with such a distance can never be the best
// of a triangle pair that hits), so the test is recorded as no contact (+inf)
// and left out of the FP64 work list.  The gap is computed in FP32 and only
// used beyond a margin (point-triangle 1 mm, edge-edge 20 um, plus 4e-6 of the
// largest coordinate involved) far above the FP32 and FP64 rounding at scene scale.

struct Box32 {
    float lo[3], hi[3];
};
__device__ __forceinline__ void box_init(Box32& b) {
    for (int k = 0; k < 3; k++) {
        b.lo[k] = 3.4e38f;
        b.hi[k] = -3.4e38f;
    }
}
// adds M (3x4 rows, FP32) applied to (x, y, z); returns the point in o
__device__ __forceinline__ void box_add(Box32& b, const float* M, float x, float y, float z, float* o, float& mag) {
    for (int r = 0; r < 3; r++) {
        const float v = M[4 * r] * x + M[4 * r + 1] * y + M[4 * r + 2] * z + M[4 * r + 3];
        o[r] = v;
        b.lo[r] = fminf(b.lo[r], v);
        b.hi[r] = fmaxf(b.hi[r], v);
        mag = fmaxf(mag, fabsf(v));
    }
}
__device__ __forceinline__ float box_gap(const Box32& a, const Box32& b) {
    float g2 = 0.f;
    for (int k = 0; k < 3; k++) {
        const float g = fmaxf(b.lo[k] - a.hi[k], a.lo[k] - b.hi[k]);
        if (g > 0.f) g2 += g * g;
    }
    return sqrtf(g2);
}

// Indices of PM_* matrices in the FP32 pose block: 8 x 12 floats per pair, then
// for the poses AS, AE, BS, BE whether they keep distances.
constexpr int kPose32 = 100;
__device__ __forceinline__ const float* pm32_of(const float* pm32, int pair, int which) {
    return pm32 + (size_t)kPose32 * pair + 12 * which;
}
enum { P32_AS = 0, P32_AE, P32_BS, P32_BE, P32_ABS, P32_ABE, P32_BAS, P32_BAE };

__global__ void k_ccd_pm32(int n, const double* __restrict__ pm, float* __restrict__ pm32) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * kPose32) return;
    const int p = i / kPose32, w = (i % kPose32) / 12, r = i % kPose32 - 12 * w;
    const double* M = pm + (size_t)PM_SIZE * p;
    pm32[i] = w < 8 ? (float)M[16 * w + r] : (keeps_distances(M + 16 * r) ? 1.f : 0.f);
}

// The swept-AABB prefilter of every (triangle of a, triangle of b) slot of a
// soup node pair (continuous_comparison.h:804-812), one warp per node pair, and
// what the descent needs of the pair.  A node pair of the soup stage has an
// inner node, emits nothing and is opened when any of its triangle pairs has a
// test with a distance below the search distance.  Every edge-edge test
// returns at most its distance at the start (edgeEdgeCCD evaluates it first)
// or at most 1e-8, so a slot whose triangles' vertices, or else edges, are
// closer than the search distance there by a margin (20 um plus 4e-6 of the
// coordinates, above their FP32 rounding) certainly hits: the node pair is
// marked and done.  The slots of the others go onto `list` for k_soup_slots,
// marked when a gap over the motion clears all their edge-edge tests.  Two bodies that are
// single leaves meet at the root: their slots are counted (`lc`) and tested
// with the leaf pairs (k_soup_filter).  The box stage:
// lanes 0-7 form the swept boxes of a's triangles, lanes 8-15 those of b's,
// once each, and every lane then tests two of the 64 slots from shuffled
// boxes.  flags[64 * entry + 8 * ta + tb] = 1 where the boxes overlap.  The
// boxes are first formed in FP32 (FP32 poses and triangles): a slot whose
// boxes are apart, or overlap, by more than a margin (1e-4 m plus 4e-6 of the
// largest coordinate, far above the FP32 rounding of the box edges) has the
// answer the FP64 boxes give; a warp with any slot inside the margin (or a
// NaN) forms the FP64 boxes and decides those slots exactly.
// res[h]: the swept boxes of slot lane + 32 h overlap.  verts: the warp's 16
// triangles (a's, then b's) in FP32 at the start, [16][9], ends: at the end;
// mags: the largest coordinate of each, for the margins (infinite where a
// triangle's edges could vanish or its coordinates pass FP32's range: then
// nothing is certain).
__device__ __forceinline__ void swept_slots(const Entry& e, const int32_t* __restrict__ pairs,
                                            const double* __restrict__ pm, const float* __restrict__ pm32,
                                            const int32_t* __restrict__ ntris, const double* __restrict__ tris,
                                            const float* __restrict__ tri32, const double* __restrict__ geo_eps,
                                            int (&res)[2], float (*verts)[9], float (*ends)[9], float* mags) {
    const int lane = threadIdx.x & 31;
    const int na = ntris[e.na], nb = ntris[e.nb];
    const bool side_b = lane >= 8;
    const int t = lane & 7;
    const bool own = lane < 16 && t < (side_b ? nb : na);
    const int body = pairs[2 * e.pair + (side_b ? 1 : 0)];
    const int node = side_b ? e.nb : e.na;
    Box32 b32;
    box_init(b32);
    float mag = 0.f;
    if (own) {
        const float* tv = tri32 + ((size_t)node * 8 + t) * 9;
        const float* MS = pm32_of(pm32, e.pair, side_b ? P32_BS : P32_AS);
        const float* ME = pm32_of(pm32, e.pair, side_b ? P32_BE : P32_AE);
        float o[3], oe[3][3];
        mag = fmaxf(fmaxf(fmaxf(fabsf(MS[3]), fabsf(MS[7])), fabsf(MS[11])),
                    fmaxf(fmaxf(fabsf(ME[3]), fabsf(ME[7])), fabsf(ME[11])));
#pragma unroll
        for (int v = 0; v < 3; v++) {
            box_add(b32, MS, tv[3 * v], tv[3 * v + 1], tv[3 * v + 2], o, mag);
            if (verts) {
                verts[lane][3 * v] = o[0];
                verts[lane][3 * v + 1] = o[1];
                verts[lane][3 * v + 2] = o[2];
            }
            box_add(b32, ME, tv[3 * v], tv[3 * v + 1], tv[3 * v + 2], oe[v], mag);
            if (verts) {
                ends[lane][3 * v] = oe[v][0];
                ends[lane][3 * v + 1] = oe[v][1];
                ends[lane][3 * v + 2] = oe[v][2];
            }
        }
        const float e32 = (float)geo_eps[body];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            b32.lo[k] -= e32;
            b32.hi[k] += e32;
        }
        mag += e32;
        if (mags) {
            // a distance is certain to be returned only while none of the
            // triangle's edges can vanish on its way: no edge is shorter than
            // 0.1 mm or changes by more than half
            const float* q = verts[lane];
            bool steady = true;
#pragma unroll
            for (int v = 0; v < 3; v++) {
                const int v1 = (v + 1) % 3;
                float l2 = 0.f, c2 = 0.f;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const float l = q[3 * v1 + k] - q[3 * v + k], c = (oe[v1][k] - oe[v][k]) - l;
                    l2 += l * l;
                    c2 += c * c;
                }
                steady = steady && l2 > 1e-8f && c2 < 0.2f * l2;
            }
            mags[lane] = steady ? mag : INFINITY;
        }
    }
    bool border = false;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int sl = lane + 32 * h, ta = sl >> 3, tb = sl & 7;
        float alo[3], ahi[3], blo[3], bhi[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            alo[k] = __shfl_sync(0xffffffffu, b32.lo[k], ta);
            ahi[k] = __shfl_sync(0xffffffffu, b32.hi[k], ta);
            blo[k] = __shfl_sync(0xffffffffu, b32.lo[k], 8 + tb);
            bhi[k] = __shfl_sync(0xffffffffu, b32.hi[k], 8 + tb);
        }
        const float m = 1e-4f + 4e-6f * fmaxf(__shfl_sync(0xffffffffu, mag, ta), __shfl_sync(0xffffffffu, mag, 8 + tb));
        res[h] = 0;
        if (ta < na && tb < nb) {
            bool apart = false, over = true;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                apart = apart || blo[k] > ahi[k] + m || alo[k] > bhi[k] + m;
                over = over && blo[k] < ahi[k] - m && alo[k] < bhi[k] - m;
            }
            res[h] = apart ? 0 : (over ? 1 : 2);
            border = border || res[h] == 2;
        }
    }
    if (__any_sync(0xffffffffu, border)) {
        Box bx;
#pragma unroll
        for (int k = 0; k < 3; k++) bx.lo[k] = bx.hi[k] = 0.0;
        if (own) {
            const double* M = pm + (size_t)PM_SIZE * e.pair;
            const Tri tri = load_tri(tris + (size_t)node * 72 + t * 9);
            bx = side_b ? swept_box(tri, M + PM_BS, M + PM_BE, geo_eps[body])
                        : swept_box(tri, M + PM_AS, M + PM_AE, geo_eps[body]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int sl = lane + 32 * h, ta = sl >> 3, tb = sl & 7;
            Box A, B;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                A.lo[k] = __shfl_sync(0xffffffffu, bx.lo[k], ta);
                A.hi[k] = __shfl_sync(0xffffffffu, bx.hi[k], ta);
                B.lo[k] = __shfl_sync(0xffffffffu, bx.lo[k], 8 + tb);
                B.hi[k] = __shfl_sync(0xffffffffu, bx.hi[k], 8 + tb);
            }
            if (res[h] == 2) res[h] = box_overlap(A, B) ? 1 : 0;
        }
    }
}

// Counters of a traversal, on the device.
enum { LC_LIST = 0, LC_NEXT, LC_LEAF, LC_ROOT, LC_TRI = 8, LC_TRI_N = 32, LC_SIZE = LC_TRI + LC_TRI_N };

__device__ __forceinline__ void warp_append(int j, bool keep, int32_t* list, int32_t* count);

__device__ __forceinline__ float vert_min(const float* a, const float* b) {
    float m = 3.4e38f;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const float dx = a[3 * i] - b[3 * j], dy = a[3 * i + 1] - b[3 * j + 1], dz = a[3 * i + 2] - b[3 * j + 2];
            m = fminf(m, fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
        }
    return sqrtf(m);
}
// The closest edge pair: its distance, and the vector between its points.
__device__ __forceinline__ float edge_min(const float* a, const float* b, F3& dir) {
    float m = 3.4e38f;
    dir = f3(0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int i1 = (i + 1) % 3, j1 = (j + 1) % 3;
            float d2;
            const F3 d =
                seg_vector(f3(a[3 * i], a[3 * i + 1], a[3 * i + 2]), f3(a[3 * i1], a[3 * i1 + 1], a[3 * i1 + 2]),
                           f3(b[3 * j], b[3 * j + 1], b[3 * j + 2]), f3(b[3 * j1], b[3 * j1 + 1], b[3 * j1 + 2]), d2);
            if (d2 < m) {
                m = d2;
                dir = d;
            }
        }
    return sqrtf(m);
}

// The gap between the triangles along d (d need not be a unit vector).
__device__ __forceinline__ float axis_gap9(F3 d, const float* a, const float* b) {
    const float nn = sqrtf(dot3(d, d));
    if (!(nn > 1e-20f)) return 0.f;
    float a0 = 3.4e38f, a1 = -3.4e38f, b0 = 3.4e38f, b1 = -3.4e38f;
#pragma unroll
    for (int v = 0; v < 3; v++) {
        const float pa = dot3(d, f3(a[3 * v], a[3 * v + 1], a[3 * v + 2]));
        const float pb = dot3(d, f3(b[3 * v], b[3 * v + 1], b[3 * v + 2]));
        a0 = fminf(a0, pa);
        a1 = fmaxf(a1, pa);
        b0 = fminf(b0, pb);
        b1 = fmaxf(b1, pb);
    }
    return fmaxf(b0 - a1, a0 - b1) / nn;
}
// A lower bound of two triangles' distance: along any direction it is at least
// the gap between the projections, whatever the direction, so one computed in
// FP32 still bounds.  Separate triangles are closest between two edges, in the
// direction d of their closest edge pair, or between a vertex and a face, along
// its normal.  Over a motion: points move on straight lines from their start to
// their end positions, so the gap along a fixed direction is concave in time
// and at least the smaller of the two ends'.  Bounds every distance between
// points of the triangles at one time (every edge-edge distance of
// edgeEdgeCCD).
__device__ __forceinline__ float axis_gap_motion(F3 d, const float* a, const float* b, const float* ae,
                                                 const float* be) {
    const float nn = sqrtf(dot3(d, d));
    if (!(nn > 1e-20f)) return 0.f;
    float g[2][2];  // [pose][side]
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float *A = k ? ae : a, *B = k ? be : b;
        float a0 = 3.4e38f, a1 = -3.4e38f, b0 = 3.4e38f, b1 = -3.4e38f;
#pragma unroll
        for (int v = 0; v < 3; v++) {
            const float pa = dot3(d, f3(A[3 * v], A[3 * v + 1], A[3 * v + 2]));
            const float pb = dot3(d, f3(B[3 * v], B[3 * v + 1], B[3 * v + 2]));
            a0 = fminf(a0, pa);
            a1 = fmaxf(a1, pa);
            b0 = fminf(b0, pb);
            b1 = fmaxf(b1, pb);
        }
        g[k][0] = b0 - a1;
        g[k][1] = a0 - b1;
    }
    return fmaxf(fminf(g[0][0], g[1][0]), fminf(g[0][1], g[1][1])) / nn;
}
__device__ __forceinline__ float tri_gap_motion(F3 d, const float* a, const float* b, const float* ae,
                                                const float* be) {
    const F3 na = cross3(f3(a[3] - a[0], a[4] - a[1], a[5] - a[2]), f3(a[6] - a[0], a[7] - a[1], a[8] - a[2]));
    const F3 nb = cross3(f3(b[3] - b[0], b[4] - b[1], b[5] - b[2]), f3(b[6] - b[0], b[7] - b[1], b[8] - b[2]));
    return fmaxf(axis_gap_motion(d, a, b, ae, be),
                 fmaxf(axis_gap_motion(na, a, b, ae, be), axis_gap_motion(nb, a, b, ae, be)));
}

// Marks a slot of k_ccd_level's list whose edge-edge tests are all clear.
constexpr int kEdgesClear = kSlotMark;

__global__ void __launch_bounds__(kBlock) k_ccd_level(
    int n_soup, const Entry* __restrict__ soup, const int32_t* __restrict__ pairs, const double* __restrict__ pm,
    const float* __restrict__ pm32, const int32_t* __restrict__ ntris, const double* __restrict__ tris,
    const float* __restrict__ tri32, const double* __restrict__ geo_eps, const float* __restrict__ search,
    const int4* __restrict__ nodes, const uint8_t* __restrict__ skip, const uint8_t* __restrict__ eskip,
    int use_bounds, int certificates, int32_t* __restrict__ entry_hits, int32_t* __restrict__ list,
    int32_t* __restrict__ lc, const int32_t* __restrict__ n_dev) {
    __shared__ float s_verts[kBlock / 32][16][9];
    __shared__ float s_ends[kBlock / 32][16][9];
    __shared__ float s_mag[kBlock / 32][16];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    if (n_dev) n_soup = *n_dev;
    for (int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5); w < n_soup;  // uniform per warp
         w += (int)((gridDim.x * (size_t)blockDim.x) >> 5)) {
        __syncwarp();
        const Entry e = soup[w];
        // a pair the root certificate proved contact-free, or a node pair its
        // separation witness proved clear: no slot goes on
        if ((skip && skip[e.pair]) || (eskip && eskip[w])) {
            if (lane == 0) entry_hits[w] = 0;
            continue;
        }
        int res[2];
        swept_slots(e, pairs, pm, pm32, ntris, tris, tri32, geo_eps, res, s_verts[wi], s_ends[wi], s_mag[wi]);
        const int k = __popc(__ballot_sync(0xffffffffu, res[0])) + __popc(__ballot_sync(0xffffffffu, res[1]));
        if (lane == 0 && k) atomicAdd(lc + LC_TRI + (w & (LC_TRI_N - 1)), k);
        bool sure = false;
        if (ld_node(nodes, e.na).z || ld_node(nodes, e.nb).z) {
            __syncwarp();
            const float thr = search[e.pair];
            float room[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int sl = lane + 32 * h, ta = sl >> 3, tb = sl & 7;
                room[h] = -1.f;
                if (!res[h] || !use_bounds || !(thr > 1e-6f)) continue;
                room[h] = thr - (2e-5f + 4e-6f * (fmaxf(s_mag[wi][ta], s_mag[wi][8 + tb]) + thr));
                sure = sure || vert_min(s_verts[wi][ta], s_verts[wi][8 + tb]) < room[h];
            }
            sure = __any_sync(0xffffffffu, sure);
            if (!sure) {
                bool clear[2] = {false, false};
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int sl = lane + 32 * h, ta = sl >> 3, tb = sl & 7;
                    if (!res[h] || !use_bounds) continue;
                    F3 d;
                    const float m = edge_min(s_verts[wi][ta], s_verts[wi][8 + tb], d);
                    if (m < room[h]) sure = true;
                    // (s_mag is infinite for an unsteady triangle: never clear either)
                    clear[h] = certificates &&
                               tri_gap_motion(d, s_verts[wi][ta], s_verts[wi][8 + tb], s_ends[wi][ta],
                                              s_ends[wi][8 + tb]) >
                                   thr + (2e-5f + 4e-6f * (fmaxf(s_mag[wi][ta], s_mag[wi][8 + tb]) + thr));
                }
                sure = __any_sync(0xffffffffu, sure);
                if (!sure) {
                    warp_append((64 * w + lane) | (clear[0] ? kEdgesClear : 0), res[0] != 0, list, lc + LC_LIST);
                    warp_append((64 * w + lane + 32) | (clear[1] ? kEdgesClear : 0), res[1] != 0, list, lc + LC_LIST);
                }
            }
        } else if (lane == 0 && k) {
            atomicAdd(lc + LC_ROOT, 1);
        }
        if (lane == 0) entry_hits[w] = sure ? 1 : 0;
    }
}

// The swept-box flags of the root node pairs that are two leaves (the soup
// stage's only emitting ones); 0 for every other node pair's slots.
__global__ void k_soup_filter(int n_soup, const Entry* __restrict__ soup, const int32_t* __restrict__ pairs,
                              const double* __restrict__ pm, const float* __restrict__ pm32,
                              const int32_t* __restrict__ ntris, const double* __restrict__ tris,
                              const float* __restrict__ tri32, const double* __restrict__ geo_eps,
                              const int4* __restrict__ nodes, const uint8_t* __restrict__ skip,
                              int32_t* __restrict__ flags) {
    const int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= n_soup) return;  // uniform per warp
    const Entry e = soup[w];
    int res[2] = {0, 0};
    if (!(skip && skip[e.pair]) && !ld_node(nodes, e.na).z && !ld_node(nodes, e.nb).z)
        swept_slots(e, pairs, pm, pm32, ntris, tris, tri32, geo_eps, res, nullptr, nullptr, nullptr);
    flags[64 * (size_t)w + lane] = res[0];
    flags[64 * (size_t)w + lane + 32] = res[1];
}


__global__ void k_add_u64(unsigned long long* __restrict__ v, unsigned long long x) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *v += x;
}

// ------------------------------------------------- learned proposal --------
// Features of a CCD pair query for the proposal network, from the bodies'
// current states: B's pose in A's frame (R_a^T R_b row major, R_a^T (x_b -
// x_a)), the relative motion over the query's horizon in A's frame
// (R_a^T (v_b - v_a) max_time, R_a^T (w_b - w_a) max_time with w = R I^-1 R^T L)
// and the two bounding radii; FP64, stored as FP32.
__global__ void k_ccd_features(int n, const int32_t* __restrict__ pairs, const double* __restrict__ max_time,
                               const double* __restrict__ cur, const double* __restrict__ ii,
                               const double* __restrict__ radius, float* __restrict__ feat) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int ia = pairs[2 * p], ib = pairs[2 * p + 1];
    const State a = load_state(cur + 14 * (size_t)ia), b = load_state(cur + 14 * (size_t)ib);
    double Ra[9], Rb[9], Ia[9], Ib[9];
    qmat(a.q, Ra);
    qmat(b.q, Rb);
    world_inv_inertia(a.q, ii + 9 * (size_t)ia, Ia);
    world_inv_inertia(b.q, ii + 9 * (size_t)ib, Ib);
    const V3 wa = m3_vec(Ia, a.L), wb = m3_vec(Ib, b.L);
    const double mt = max_time[p];
    float* f = feat + 20 * (size_t)p;
    auto at = [&](V3 v, int r) { return (Ra[r] * v.x + Ra[3 + r] * v.y) + Ra[6 + r] * v.z; };  // (R_a^T v)_r
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) f[3 * r + c] = (float)((Ra[r] * Rb[c] + Ra[3 + r] * Rb[3 + c]) + Ra[6 + r] * Rb[6 + c]);
    for (int r = 0; r < 3; r++) {
        f[9 + r] = (float)at(b.x - a.x, r);
        f[12 + r] = (float)(at(b.v - a.v, r) * mt);
        f[15 + r] = (float)(at(wb - wa, r) * mt);
    }
    f[18] = (float)radius[ia];
    f[19] = (float)radius[ib];
}

// The root certificate of a pair query the network predicts contact-free: a
// warp per pair proves that no slot of the root node pair can hit, so the
// query has no contacts (compareTreesFullContinuous expands only node pairs
// with hits).  A slot is proven clear when the reference's swept-box test
// rejects it (continuous_comparison.h:804-812; decided in FP32 beyond a
// margin, as the swept-box filter decides it, else in FP64), or when the
// two triangles' vertices, each on a straight line from its start to its end
// position, stay apart over the motion:
//   * along an axis n fixed at the start (the centroid difference, either
//     face normal), min_j n.b_j(t) - max_i n.a_i(t) is concave in t, so its
//     minimum over [0, 1] is at t = 0 or 1; the gap over |n| bounds every
//     edge-edge distance edgeEdgeCCD evaluates (points of the two edges at
//     one time), and the point-to-triangle distances at t = 0 and 1;
//   * pointTriCCDLinear returns 0 only when a vertex's start and end lie on
//     opposite sides of the other triangle's plane (its start and end frames),
//     and otherwise the vertex's distance to that plane at t = 0 or 1 when its
//     projection falls inside (decided with float barycentrics) or nothing:
//     so every vertex must keep its side, and the gap carries a margin for a
//     projection the float test puts inside by mistake (6e-7 of the
//     triangle's size times its conditioning (L0 L1 / 2 area)^2).
// A query whose every root slot is proven clear is skipped: it would produce
// no contact.  Any slot not proven leaves the query to the exact traversal.
// stats: [2] predicted clear, [3] certified, [4] not certified, [5] seen.
__device__ __forceinline__ double axis_gap(V3 n, const V3* A0, const V3* A1, const V3* B0, const V3* B1) {
    double g = -1e300;
    for (int sg = 0; sg < 2; sg++) {
        const V3 m = sg ? -n : n;
        double gmin = 1e300;
        for (int t = 0; t < 2; t++) {
            const V3* A = t ? A1 : A0;
            const V3* B = t ? B1 : B0;
            const double amax = fmax(fmax(dot(m, A[0]), dot(m, A[1])), dot(m, A[2]));
            const double bmin = fmin(fmin(dot(m, B[0]), dot(m, B[1])), dot(m, B[2]));
            gmin = fmin(gmin, bmin - amax);
        }
        g = fmax(g, gmin);
    }
    const double nn = norm(n);
    return nn > 0.0 ? g / nn : -1e300;
}
// every vertex of P keeps a side of T's plane (start and end frames), with
// distances far above rounding
__device__ __forceinline__ bool keeps_side(const V3* P0, const V3* P1, const V3* T0, const V3* T1, double tol) {
    const V3 n0 = cross(T0[1] - T0[0], T0[2] - T0[0]), n1 = cross(T1[1] - T1[0], T1[2] - T1[0]);
    const double l0 = norm(n0), l1 = norm(n1);
    if (!(l0 > 0.0) || !(l1 > 0.0)) return false;
    for (int i = 0; i < 3; i++) {
        const double h0 = dot(n0, P0[i] - T0[0]) / l0, h1 = dot(n1, P1[i] - T1[0]) / l1;
        if (!(h0 * h1 > 0.0) || !(fabs(h0) > tol) || !(fabs(h1) > tol)) return false;
    }
    return true;
}
__device__ __forceinline__ double tri_conditioning(const V3* T, double& lmax) {
    const double l0 = norm(T[1] - T[0]), l1 = norm(T[2] - T[0]), l2 = norm(T[2] - T[1]);
    lmax = fmax(fmax(l0, l1), l2);
    const double a2 = norm(cross(T[1] - T[0], T[2] - T[0]));
    if (!(a2 > 0.0)) return 1e300;
    const double k = (l0 * l1) / a2;
    return k * k;
}
// ------------------------------------------------ separation witnesses -----
// Temporal coherence of the CCD traversal (the separation witnesses of
// collision_detection/contact_state.cpp:14-150 and full_tree_comparison.cpp:
// 7-198, rebuilt so that results cannot change).  A witness is an axis, in
// body a's frame, that separated a soup node pair at an earlier call.  At the
// next call the node pair is skipped when that axis (through a's current
// rotation) still proves every slot of the pair clear over the query's motion,
// by the same proof as the root certificate (swept-box rejection, or
// side-keeping vertices and a separating gap beyond the search distance);
// a skipped node pair has no hit, so the reference would neither expand it
// nor emit from it.  Node pairs without hits get a new witness (the axis
// between their buckets' vertex centroids) when it proves them clear.  A
// stale or foreign witness can only fail its check.  Table: open addressing,
// 64-bit keys (bodies < 2^19, node ids local to their tree < 2^12; other
// node pairs get no witness), at most 32 probes.
__device__ __forceinline__ unsigned long long witness_key(int a, int b, int la, int lb) {
    if (a < 0 || b < 0 || a >= (1 << 19) || b >= (1 << 19) || la < 0 || lb < 0 || la >= 4096 || lb >= 4096)
        return 0ull;
    return (1ull << 63) | ((unsigned long long)a << 43) | ((unsigned long long)b << 24) |
           ((unsigned long long)la << 12) | (unsigned long long)lb;
}
__device__ __forceinline__ unsigned int witness_hash(unsigned long long k, int log2cap) {
    return (unsigned int)((k * 0x9E3779B97F4A7C15ull) >> (64 - log2cap));
}

// Every slot of node pair (na, nb) proven clear (warp-collective).  Lanes
// 0-7 hold a's triangles and lanes 8-15 b's: each forms its triangle's world
// vertices at the start and end and the reference's swept box once; every
// lane then takes two slots, rejected by the boxes or proven by the
// certificate from shuffled vertices.  With `axis` non-null only that world
// axis is tried (a witness); otherwise the slot's centroid difference and
// both face normals.
__device__ bool slots_clear(int na_node, int nb_node, const double* M, const float* pm32, int pair,
                            const int32_t* ntris, const double* tris, const float* tri32, double eps_a, double eps_b,
                            double S, const V3* axis) {
    const int lane = threadIdx.x & 31;
    const int na = ntris[na_node], nb = ntris[nb_node];
    const bool side_b = lane >= 8;
    const int t = lane & 7;
    const bool own = lane < 16 && t < (side_b ? nb : na);
    // The swept boxes first in FP32, as the swept-box filter forms them: a slot
    // whose boxes are apart by more than the margin is rejected as the FP64
    // boxes would reject it; only when some slot is not the warp goes on in FP64.
    bool apart32[2];
    {
        Box32 b32;
        box_init(b32);
        float mag = 0.f;
        if (own) {
            const float* tv = tri32 + ((size_t)(side_b ? nb_node : na_node) * 8 + t) * 9;
            const float* MS = pm32_of(pm32, pair, side_b ? P32_BS : P32_AS);
            const float* ME = pm32_of(pm32, pair, side_b ? P32_BE : P32_AE);
            float o[3];
            for (int v = 0; v < 3; v++) {
                box_add(b32, MS, tv[3 * v], tv[3 * v + 1], tv[3 * v + 2], o, mag);
                box_add(b32, ME, tv[3 * v], tv[3 * v + 1], tv[3 * v + 2], o, mag);
            }
            const float e32 = (float)(side_b ? eps_b : eps_a);
            for (int k = 0; k < 3; k++) {
                b32.lo[k] -= e32;
                b32.hi[k] += e32;
            }
            mag += e32;
        }
        bool any_near = false;
        for (int h = 0; h < 2; h++) {
            const int sl = lane + 32 * h, ta = sl >> 3, tb = sl & 7;
            bool apart = false;
            const float m = 1e-4f + 4e-6f * fmaxf(__shfl_sync(0xffffffffu, mag, ta),
                                                  __shfl_sync(0xffffffffu, mag, 8 + tb));
            for (int k = 0; k < 3; k++) {
                const float alo = __shfl_sync(0xffffffffu, b32.lo[k], ta), ahi = __shfl_sync(0xffffffffu, b32.hi[k], ta);
                const float blo = __shfl_sync(0xffffffffu, b32.lo[k], 8 + tb),
                            bhi = __shfl_sync(0xffffffffu, b32.hi[k], 8 + tb);
                apart = apart || blo > ahi + m || alo > bhi + m;
            }
            apart32[h] = apart;
            any_near = any_near || (ta < na && tb < nb && !apart);
        }
        if (!__any_sync(0xffffffffu, any_near)) return true;  // every slot rejected by the swept boxes
    }
    V3 v0[3], v1[3];
    Box bx;
    for (int k = 0; k < 3; k++) bx.lo[k] = bx.hi[k] = 0.0;
    for (int i = 0; i < 3; i++) v0[i] = v1[i] = mk(0, 0, 0);
    if (own) {
        const Tri T = load_tri(tris + (size_t)(side_b ? nb_node : na_node) * 72 + t * 9);
        const double* MS = M + (side_b ? PM_BS : PM_AS);
        const double* ME = M + (side_b ? PM_BE : PM_AE);
        bx = swept_box(T, MS, ME, side_b ? eps_b : eps_a);
        v0[0] = xform_rigid(T.A, MS);
        v0[1] = xform_rigid(T.B, MS);
        v0[2] = xform_rigid(T.C, MS);
        v1[0] = xform_rigid(T.A, ME);
        v1[1] = xform_rigid(T.B, ME);
        v1[2] = xform_rigid(T.C, ME);
    }
    auto sh3 = [&](V3 v, int src) {
        return mk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                  __shfl_sync(0xffffffffu, v.z, src));
    };
    bool clear = true;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int sl = lane + 32 * h, ta = sl >> 3, tb = sl & 7;
        Box A, B;
        for (int k = 0; k < 3; k++) {
            A.lo[k] = __shfl_sync(0xffffffffu, bx.lo[k], ta);
            A.hi[k] = __shfl_sync(0xffffffffu, bx.hi[k], ta);
            B.lo[k] = __shfl_sync(0xffffffffu, bx.lo[k], 8 + tb);
            B.hi[k] = __shfl_sync(0xffffffffu, bx.hi[k], 8 + tb);
        }
        V3 A0[3], A1[3], B0[3], B1[3];
        for (int i = 0; i < 3; i++) {
            A0[i] = sh3(v0[i], ta);
            A1[i] = sh3(v1[i], ta);
            B0[i] = sh3(v0[i], 8 + tb);
            B1[i] = sh3(v1[i], 8 + tb);
        }
        if (ta >= na || tb >= nb || !clear || apart32[h] || !box_overlap(A, B)) continue;
        double mag = 0.0;
        for (int i = 0; i < 3; i++)
            mag = fmax(mag, fmax(fmax(fmax(fabs(A0[i].x), fabs(A0[i].y)), fabs(A0[i].z)),
                                 fmax(fmax(fabs(B0[i].x), fabs(B0[i].y)), fabs(B0[i].z))));
        double la, lb;
        const double ka = tri_conditioning(A0, la), kb = tri_conditioning(B0, lb);
        if (!(ka < 1e4) || !(kb < 1e4)) {
            clear = false;
            continue;
        }
        const double tol = 1e-9 + 1e-12 * mag;
        const double margin = (1e-5 + 1e-9 * mag) + 6e-7 * fmax(ka * la, kb * lb);
        if (!keeps_side(A0, A1, B0, B1, tol) || !keeps_side(B0, B1, A0, A1, tol)) {
            clear = false;
            continue;
        }
        double g;
        if (axis) {
            g = axis_gap(*axis, A0, A1, B0, B1);
        } else {
            const V3 ca = (A0[0] + A0[1]) + A0[2], cb = (B0[0] + B0[1]) + B0[2];
            g = axis_gap(cb - ca, A0, A1, B0, B1);
            g = fmax(g, axis_gap(cross(A0[1] - A0[0], A0[2] - A0[0]), A0, A1, B0, B1));
            g = fmax(g, axis_gap(cross(B0[1] - B0[0], B0[2] - B0[0]), A0, A1, B0, B1));
        }
        if (!(g >= S + margin)) clear = false;
    }
    return __all_sync(0xffffffffu, clear);
}

__global__ void k_root_certify(int n, const int32_t* __restrict__ pairs, const double* __restrict__ pm,
                               const float* __restrict__ pm32, const float* __restrict__ tri32,
                               const int32_t* __restrict__ mesh, const int32_t* __restrict__ mesh_node_off,
                               const int32_t* __restrict__ ntris, const double* __restrict__ tris,
                               const double* __restrict__ geo_eps, const float* __restrict__ search,
                               const float* __restrict__ pred, float logit_cut, uint8_t* __restrict__ skip,
                               unsigned long long* __restrict__ stats) {
    const int p = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (p >= n) return;  // uniform per warp
    const bool gated = pred[2 * (size_t)p + 1] < logit_cut;  // NaN: not gated
    if (!gated) {
        if (lane == 0) skip[p] = 0;
        return;
    }
    const int ia = pairs[2 * p], ib = pairs[2 * p + 1];
    const bool all = slots_clear(mesh_node_off[mesh[ia]], mesh_node_off[mesh[ib]], pm + (size_t)PM_SIZE * p, pm32, p,
                                 ntris, tris, tri32, geo_eps[ia], geo_eps[ib], (double)search[p], nullptr);
    if (lane == 0) {
        skip[p] = all ? 1 : 0;
        atomicAdd(stats + 2, 1ull);
        atomicAdd(stats + (all ? 3 : 4), 1ull);
    }
}

__global__ void k_witness_check(int n, const Entry* __restrict__ soup, const int32_t* __restrict__ pairs,
                                const double* __restrict__ pm, const float* __restrict__ pm32,
                                const float* __restrict__ tri32, const int32_t* __restrict__ mesh,
                                const int32_t* __restrict__ mesh_node_off, const int32_t* __restrict__ ntris,
                                const double* __restrict__ tris, const double* __restrict__ geo_eps,
                                const float* __restrict__ search, const WitnessSlot* __restrict__ table,
                                int log2cap, uint8_t* __restrict__ wflag, unsigned long long* __restrict__ stats) {
    const int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= n) return;  // uniform per warp
    const Entry e = soup[w];
    const int a = pairs[2 * e.pair], b = pairs[2 * e.pair + 1];
    const unsigned long long key =
        witness_key(a, b, e.na - mesh_node_off[mesh[a]], e.nb - mesh_node_off[mesh[b]]);
    int found = -1;
    if (key) {
        const unsigned int mask = (1u << log2cap) - 1u;
        unsigned int h = witness_hash(key, log2cap);
        for (int probe = 0; probe < 32; probe++, h = (h + 1) & mask) {
            const unsigned long long k = table[h].key;
            if (k == key) {
                found = (int)h;
                break;
            }
            if (k == 0ull) break;
        }
    }
    bool clear = false;
    if (found >= 0) {
        const double* M = pm + (size_t)PM_SIZE * e.pair;
        const WitnessSlot& W = table[found];
        // the axis through a's rotation at the start (rows 0-2 of its start transform)
        const V3 loc = mk((double)W.ax, (double)W.ay, (double)W.az);
        const V3 n_world = mk((M[PM_AS + 0] * loc.x + M[PM_AS + 1] * loc.y) + M[PM_AS + 2] * loc.z,
                              (M[PM_AS + 4] * loc.x + M[PM_AS + 5] * loc.y) + M[PM_AS + 6] * loc.z,
                              (M[PM_AS + 8] * loc.x + M[PM_AS + 9] * loc.y) + M[PM_AS + 10] * loc.z);
        clear = norm(n_world) > 0.0 && slots_clear(e.na, e.nb, M, pm32, e.pair, ntris, tris, tri32, geo_eps[a],
                                                   geo_eps[b], (double)search[e.pair], &n_world);
    }
    if (lane == 0) {
        wflag[w] = clear ? 1 : 0;
        if (clear) atomicAdd(stats + 6, 1ull);
    }
}

__global__ void k_witness_make(int n, const Entry* __restrict__ soup, const int32_t* __restrict__ entry_hits,
                               const uint8_t* __restrict__ wflag, const uint8_t* __restrict__ skip,
                               const int32_t* __restrict__ pairs, const double* __restrict__ pm,
                               const float* __restrict__ pm32, const float* __restrict__ tri32,
                               const int32_t* __restrict__ mesh, const int32_t* __restrict__ mesh_node_off,
                               const int32_t* __restrict__ ntris, const double* __restrict__ tris,
                               const double* __restrict__ geo_eps, const float* __restrict__ search,
                               WitnessSlot* __restrict__ table, int log2cap, unsigned long long* __restrict__ stats) {
    const int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= n) return;  // uniform per warp
    const Entry e = soup[w];
    if (entry_hits[w] > 0 || wflag[w] || (skip && skip[e.pair])) return;
    const int a = pairs[2 * e.pair], b = pairs[2 * e.pair + 1];
    const unsigned long long key =
        witness_key(a, b, e.na - mesh_node_off[mesh[a]], e.nb - mesh_node_off[mesh[b]]);
    if (!key) return;
    const double* M = pm + (size_t)PM_SIZE * e.pair;
    // the axis between the two buckets' vertex centroids at the start
    const int na = ntris[e.na], nb = ntris[e.nb];
    V3 c = mk(0, 0, 0);
    if (lane < 16) {
        const int t = lane & 7;
        const bool side_b = lane >= 8;
        if (t < (side_b ? nb : na)) {
            const Tri T = load_tri(tris + (size_t)(side_b ? e.nb : e.na) * 72 + t * 9);
            const double* Ms = M + (side_b ? PM_BS : PM_AS);
            const V3 s = (xform_rigid(T.A, Ms) + xform_rigid(T.B, Ms)) + xform_rigid(T.C, Ms);
            c = s * (side_b ? 1.0 / nb : -1.0 / na);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        c.x += __shfl_xor_sync(0xffffffffu, c.x, o);
        c.y += __shfl_xor_sync(0xffffffffu, c.y, o);
        c.z += __shfl_xor_sync(0xffffffffu, c.z, o);
    }
    if (!(norm(c) > 0.0) ||
        !slots_clear(e.na, e.nb, M, pm32, e.pair, ntris, tris, tri32, geo_eps[a], geo_eps[b], (double)search[e.pair],
                     &c))
        return;
    if (lane == 0) {
        // store the axis in a's frame: R_a^T n
        const V3 loc = mk((M[PM_AS + 0] * c.x + M[PM_AS + 4] * c.y) + M[PM_AS + 8] * c.z,
                          (M[PM_AS + 1] * c.x + M[PM_AS + 5] * c.y) + M[PM_AS + 9] * c.z,
                          (M[PM_AS + 2] * c.x + M[PM_AS + 6] * c.y) + M[PM_AS + 10] * c.z);
        const unsigned int mask = (1u << log2cap) - 1u;
        unsigned int h = witness_hash(key, log2cap);
        for (int probe = 0; probe < 32; probe++, h = (h + 1) & mask) {
            const unsigned long long old = atomicCAS(&table[h].key, 0ull, key);
            if (old == 0ull || old == key) {
                table[h].ax = (float)loc.x;
                table[h].ay = (float)loc.y;
                table[h].az = (float)loc.z;
                atomicAdd(stats + 7, 1ull);
                break;
            }
        }
    }
}

// Point-triangle work item j (the decoding of k_prim_pt): which pair, which
// point (body-local), which triangle (body-local) and which transforms.
struct PtWork {
    int pair, pt_node, pt_tri, pt_vert, tri_node, tri_idx, mC, mT;  // mC: point frame pair, mT: triangle body
    PrimResult* out;
    int32_t* hit;
};
__device__ __forceinline__ PtWork decode_pt(int j, int n_tp, const int32_t* items, const Entry* soup,
                                            const Entry* conn, const int32_t* nn_off, const int32_t* tp,
                                            const int32_t* ntris, PrimResult* sub, PrimResult* cres, int32_t* chit) {
    PtWork w;
    w.hit = nullptr;
    if (j < 6 * n_tp) {
        const int k = j / 6, q = j % 6;
        const int slot = items[k];
        const Entry e = soup[slot >> 6];
        const int i = q >> 1;
        w.pair = e.pair;
        if (q & 1) {
            w.pt_node = e.nb, w.pt_tri = slot & 7, w.tri_node = e.na, w.tri_idx = (slot >> 3) & 7;
            w.mC = P32_BAS, w.mT = P32_AS;
        } else {
            w.pt_node = e.na, w.pt_tri = (slot >> 3) & 7, w.tri_node = e.nb, w.tri_idx = slot & 7;
            w.mC = P32_ABS, w.mT = P32_BS;
        }
        w.pt_vert = i;
        w.out = sub + 15 * (size_t)k + 5 * i + (q & 1);
        return w;
    }
    const int jp = j - 6 * n_tp;
    const int ei = tp[jp / 6];
    const Entry e = conn[ei];
    const int l = jp - 6 * nn_off[ei];
    const int na = ntris[e.na], nb = ntris[e.nb];
    const int n1 = 3 * na * nb;
    w.pair = e.pair;
    if (l < n1) {
        const int vi = l / nb, jj = l % nb;
        w.pt_node = e.na, w.pt_tri = vi / 3, w.pt_vert = vi % 3, w.tri_node = e.nb, w.tri_idx = jj;
        w.mC = P32_ABS, w.mT = P32_BS;
    } else {
        const int m = l - n1;
        const int vi = m / na, jj = m % na;
        w.pt_node = e.nb, w.pt_tri = vi / 3, w.pt_vert = vi % 3, w.tri_node = e.na, w.tri_idx = jj;
        w.mC = P32_BAS, w.mT = P32_AS;
    }
    const size_t item = 15 * (size_t)nn_off[ei] + l;
    w.out = cres + item;
    w.hit = chit + item;
    return w;
}

// Edge-edge work item j, as the edge-edge mask and CCD kernels decode it.
struct EeWork {
    int pair, na, nb, aTri, aEdge, bTri, bEdge;
    PrimResult* out;
    int32_t* hit;
};
__device__ __forceinline__ EeWork decode_ee(int j, int n_tp, const int32_t* items, const Entry* soup,
                                            const Entry* conn, const int32_t* nn_off, const int32_t* tp,
                                            const int32_t* ntris, PrimResult* sub, PrimResult* cres, int32_t* chit) {
    EeWork w;
    w.hit = nullptr;
    Entry e;
    if (j < 9 * n_tp) {
        const int k = j / 9, q = j % 9;
        const int slot = items[k];
        e = soup[slot >> 6];
        w.aTri = (slot >> 3) & 7;
        w.bTri = slot & 7;
        w.aEdge = q / 3;
        w.bEdge = q % 3;
        w.out = sub + 15 * (size_t)k + 5 * w.aEdge + 2 + w.bEdge;
    } else {
        const int jp = j - 9 * n_tp;
        const int ei = tp[jp / 9];
        e = conn[ei];
        const int m = jp - 9 * nn_off[ei];
        const int na = ntris[e.na], nb = ntris[e.nb];
        const int ea = m / (3 * nb), eb = m % (3 * nb);
        w.aTri = ea / 3;
        w.aEdge = ea % 3;
        w.bTri = eb / 3;
        w.bEdge = eb % 3;
        const size_t item = 15 * (size_t)nn_off[ei] + 6 * (size_t)na * nb + m;
        w.out = cres + item;
        w.hit = chit + item;
    }
    w.pair = e.pair;
    w.na = e.na;
    w.nb = e.nb;
    return w;
}

__device__ __forceinline__ void record_no_contact(PrimResult* out, int32_t* hit) {
    store_prim(out, 1.0 / 0.0, mk(0, 0, 0), mk(0, 0, 0), 1.0);
    if (hit) *hit = 0;
}

// A warp's surviving tests appended to list (lane order within the warp,
// warps in arrival order; the tests' results do not depend on the order), the
// list's length in *count.
__device__ __forceinline__ void warp_append(int j, bool keep, int32_t* list, int32_t* count) {
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) list[base + __popc(m & ((1u << lane) - 1u))] = j;
}

// FP32 bounds of a point-triangle test (pointTriCCDLinear): certainly no
// distance below thr.  Either the boxes are apart; or the point keeps its side
// of the triangle's plane, so that only its start and end count, and at each
// its projection is outside the triangle or it is too far above the plane.
// Both in FP32 with margins: the box's as for k_ccd_mask_ee; the plane's in
// the triangle's frame (PlaneBound, which covers the reference's single-
// precision barycentrics), whose heights are distances only under poses that
// keep them, and those come with the FP64 rounding of the world coordinates.
__device__ __forceinline__ bool pt_apart(const float* __restrict__ pm32, int pair, int mC, int mT, const float* pt,
                                         const float* tv, float thr) {
    const float *Cs = pm32_of(pm32, pair, mC), *Ce = pm32_of(pm32, pair, mC + 1);
    const float *tS = pm32_of(pm32, pair, mT), *tE = pm32_of(pm32, pair, mT + 1);
    float mag = 0.f, ps[3], pe[3], o[3];
    Box32 bp, bq, scratch;
    box_init(bp);
    box_init(bq);
    box_init(scratch);
    box_add(scratch, Cs, pt[0], pt[1], pt[2], ps, mag);
    box_add(scratch, Ce, pt[0], pt[1], pt[2], pe, mag);
    const float local = fmaxf(mag, fmaxf(fmaxf(fmaxf(fabsf(Cs[3]), fabsf(Cs[7])), fabsf(Cs[11])),
                                         fmaxf(fmaxf(fabsf(Ce[3]), fabsf(Ce[7])), fabsf(Ce[11]))));
    box_add(bp, tS, ps[0], ps[1], ps[2], o, mag);
    box_add(bp, tS, pe[0], pe[1], pe[2], o, mag);
    box_add(bp, tE, ps[0], ps[1], ps[2], o, mag);
    box_add(bp, tE, pe[0], pe[1], pe[2], o, mag);
    for (int v = 0; v < 3; v++) {
        box_add(bq, tS, tv[3 * v], tv[3 * v + 1], tv[3 * v + 2], o, mag);
        box_add(bq, tE, tv[3 * v], tv[3 * v + 1], tv[3 * v + 2], o, mag);
    }
    if (box_gap(bp, bq) > thr + (1e-3f + 4e-6f * (mag + thr))) return true;  // NaN: not certain
    const float* keeps = pm32_of(pm32, pair, 8);
    if (keeps[mT] == 0.f || keeps[mT + 1] == 0.f) return false;
    const F3 T0 = f3(tv[0], tv[1], tv[2]), T1 = f3(tv[3], tv[4], tv[5]), T2 = f3(tv[6], tv[7], tv[8]);
    const F3 p0 = f3(ps[0], ps[1], ps[2]), p1 = f3(pe[0], pe[1], pe[2]);
    // the frame's coordinates carry an error of 4e-7 of their size, 1e-6 here
    const float rho = fmaxf(fmaxf(local, fmaxf(maxabs3(T0), fmaxf(maxabs3(T1), maxabs3(T2)))), 1e-3f);
    const PlaneBound P = plane_bound(T0, T1, T2, 8.f * rho);
    if (!P.ok) return false;
    const F3 q[2] = {p0 - T0, p1 - T0};
    const float h0 = dot3(P.n, q[0]), h1 = dot3(P.n, q[1]);
    const float err = 2.f * P.eh * 8.f * rho;
    if (!((h0 > err && h1 > err) || (h0 < -err && h1 < -err))) return false;
    const float lim = (thr + (2e-5f + 1e-13f * mag + 4e-6f * (8.f * rho + thr))) * P.len + err;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        float u, v, w;
        plane_bary(P, q[k], u, v, w);
        if (!(u < -P.mb || v < -P.mb || w < -P.mb) && !(fabsf(k ? h1 : h0) > lim)) return false;
    }
    return true;
}

__global__ void __launch_bounds__(kBlock) k_ccd_mask_pt(int n_tp, int n_total, const int32_t* __restrict__ items,
                                                        const Entry* __restrict__ soup, const Entry* __restrict__ conn,
                                                        const int32_t* __restrict__ nn_off, const int32_t* __restrict__ tp,
                                                        const float* __restrict__ pm32,
                                                        const int32_t* __restrict__ ntris,
                                                        const float* __restrict__ tri32,
                                                        const float* __restrict__ search, PrimResult* __restrict__ sub,
                                                        PrimResult* __restrict__ cres, int32_t* __restrict__ chit,
                                                        int32_t* __restrict__ list, int32_t* __restrict__ count,
                                                        int use_bounds) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    bool keep = false;
    if (j < n_total) {
        const PtWork w = decode_pt(j, n_tp, items, soup, conn, nn_off, tp, ntris, sub, cres, chit);
        const float* pt = tri32 + ((size_t)w.pt_node * 8 + w.pt_tri) * 9 + 3 * w.pt_vert;
        const float* tv = tri32 + ((size_t)w.tri_node * 8 + w.tri_idx) * 9;
        keep = !use_bounds || !pt_apart(pm32, w.pair, w.mC, w.mT, pt, tv, search[w.pair]);
        if (!keep) record_no_contact(w.out, w.hit);
    }
    warp_append(j, keep, list, count);
}

__global__ void __launch_bounds__(kBlock) k_ccd_mask_ee(int n_tp, int n_total, const int32_t* __restrict__ items,
                                                        const Entry* __restrict__ soup, const Entry* __restrict__ conn,
                                                        const int32_t* __restrict__ nn_off, const int32_t* __restrict__ tp,
                                                        const float* __restrict__ pm32,
                                                        const int32_t* __restrict__ ntris,
                                                        const float* __restrict__ tri32,
                                                        const float* __restrict__ search, PrimResult* __restrict__ sub,
                                                        PrimResult* __restrict__ cres, int32_t* __restrict__ chit,
                                                        int32_t* __restrict__ list, int32_t* __restrict__ count,
                                                        int use_bounds, int certificates,
                                                        unsigned long long* __restrict__ cut_counts) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    bool keep = false, cut = false;
    if (j < n_total) {
        const EeWork w = decode_ee(j, n_tp, items, soup, conn, nn_off, tp, ntris, sub, cres, chit);
        const float* ta = tri32 + ((size_t)w.na * 8 + w.aTri) * 9;
        const float* tb = tri32 + ((size_t)w.nb * 8 + w.bTri) * 9;
        const int a0 = w.aEdge, a1 = w.aEdge == 2 ? 0 : w.aEdge + 1;
        const int b0 = w.bEdge, b1 = w.bEdge == 2 ? 0 : w.bEdge + 1;
        float mag = 0.f, o[2][4][3];  // [start, end][a0 a1 b0 b1]
        Box32 ba, bb;
        box_init(ba);
        box_init(bb);
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const float* MA = pm32_of(pm32, w.pair, P32_AS + m);
            const float* MB = pm32_of(pm32, w.pair, P32_BS + m);
            mag = fmaxf(mag, fmaxf(fmaxf(fmaxf(fabsf(MA[3]), fabsf(MA[7])), fabsf(MA[11])),
                                   fmaxf(fmaxf(fabsf(MB[3]), fabsf(MB[7])), fabsf(MB[11]))));
            box_add(ba, MA, ta[3 * a0], ta[3 * a0 + 1], ta[3 * a0 + 2], o[m][0], mag);
            box_add(ba, MA, ta[3 * a1], ta[3 * a1 + 1], ta[3 * a1 + 2], o[m][1], mag);
            box_add(bb, MB, tb[3 * b0], tb[3 * b0 + 1], tb[3 * b0 + 2], o[m][2], mag);
            box_add(bb, MB, tb[3 * b1], tb[3 * b1 + 1], tb[3 * b1 + 2], o[m][3], mag);
        }
        const float thr = search[w.pair];
        const float lim = thr + (2e-5f + 4e-6f * (mag + thr));
        keep = !use_bounds || !(box_gap(ba, bb) > lim);
        if (keep && use_bounds && certificates) {
            F3 p[2][4];
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int v = 0; v < 4; v++) p[m][v] = f3(o[m][v][0], o[m][v][1], o[m][v][2]);
            cut = edges_stay_apart(p, lim);
            keep = !cut;
        }
        if (!keep) record_no_contact(w.out, w.hit);
    }
    const unsigned n_cut = __popc(__ballot_sync(0xffffffffu, cut));
    if (n_cut && (threadIdx.x & 31) == 0)
        atomicAdd(cut_counts + (blockIdx.x % kCutCounters), (unsigned long long)n_cut);
    warp_append(j, keep, list, count);
}

__global__ void __launch_bounds__(kPrimBlock) k_prim_pt(int n_tp, int n_total, const int32_t* __restrict__ items,
                                                        const Entry* __restrict__ soup, const Entry* __restrict__ conn,
                                                        const int32_t* __restrict__ nn_off, const int32_t* __restrict__ tp,
                                                        const double* __restrict__ pm,
                                                        const int32_t* __restrict__ ntris,
                                                        const double* __restrict__ tris,
                                                        const float* __restrict__ search,
                                                        PrimResult* __restrict__ sub, PrimResult* __restrict__ cres,
                                                        int32_t* __restrict__ chit, const int32_t* __restrict__ list,
                                                        const int32_t* __restrict__ n_list) {
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    if (kk >= n_total || kk >= *n_list) return;
    const int j = list[kk];
    if (j < 6 * n_tp) {
        const int k = j / 6, w = j % 6;
        const int slot = items[k];
        const Entry e = soup[slot >> 6];
        const double* M = pm + (size_t)PM_SIZE * e.pair;
        const Tri ta = load_tri(tris + (size_t)e.na * 72 + ((slot >> 3) & 7) * 9);
        const Tri tb = load_tri(tris + (size_t)e.nb * 72 + (slot & 7) * 9);
        const int i = w >> 1;
        const Ccd r = (w & 1) ? point_tri_ccd(tvert(tb, i), M + PM_BAS, M + PM_BAE, ta, M + PM_AS, M + PM_AE)
                              : point_tri_ccd(tvert(ta, i), M + PM_ABS, M + PM_ABE, tb, M + PM_BS, M + PM_BE);
        store_prim(sub + 15 * (size_t)k + 5 * i + (w & 1), r.dist, r.P, r.Q, r.toc);
        return;
    }
    const int jp = j - 6 * n_tp;
    const int ei = tp[jp / 6];
    const Entry e = conn[ei];
    const int l = jp - 6 * nn_off[ei];
    const int na = ntris[e.na], nb = ntris[e.nb];
    const double* M = pm + (size_t)PM_SIZE * e.pair;
    const double* pa = tris + (size_t)e.na * 72;
    const double* pb = tris + (size_t)e.nb * 72;
    const int n1 = 3 * na * nb;
    Ccd r;
    V3 A, B;
    if (l < n1) {
        const int vi = l / nb, jj = l % nb;
        r = point_tri_ccd(tvert(load_tri(pa + (vi / 3) * 9), vi % 3), M + PM_ABS, M + PM_ABE, load_tri(pb + jj * 9),
                          M + PM_BS, M + PM_BE);
        A = r.P;
        B = r.Q;
    } else {
        const int m = l - n1;
        const int vi = m / na, jj = m % na;
        r = point_tri_ccd(tvert(load_tri(pb + (vi / 3) * 9), vi % 3), M + PM_BAS, M + PM_BAE, load_tri(pa + jj * 9),
                          M + PM_AS, M + PM_AE);
        A = r.Q;
        B = r.P;
    }
    const size_t item = 15 * (size_t)nn_off[ei] + l;
    store_prim(cres + item, r.dist, A, B, r.toc);
    chit[item] = r.dist < (double)search[e.pair] ? 1 : 0;
}

// Edge-edge CCD in two passes over the surviving tests.  GB300's FP64 pipe
// takes one warp instruction per 64 cycles per SM sub-partition (SMSP),
// dependent or not and whatever the number of active lanes (a division costs
// ~9 such slots, a square root ~10), so a warp's time is the instruction count
// of its longest lane.  62% of the tests end within two Newton iterations (~230
// slots each on one lane) and 20% run all ten; 0.5% bisect (~370 slots, which
// every warp of the first pass that has one would wait for).  So:
//   k_ee_first   one test per lane: the edges and at most two
//                Newton iterations; the tests still running and those that
//                bisect are saved and listed.
//   k_ee_rest4   the listed tests on four lanes each (below), ~190 slots an
//                iteration: while the list gives each SMSP at most a warp or
//                two, latency is what counts.
//   k_ee_rest1   the listed tests on one lane each, when there are more than
//                kRestWide: a quarter of the warps at 1.2 times the slots (noisy
//                spheres, 71,000 listed tests: 1,225 us on four lanes, 636 on
//                one; 520 with the shortened iteration).
// Each test performs exactly the operations of edge_edge_ccd, in order.
// The first pass's iteration cap is the context setting D2G_TUNE_EE_FIRST_ITERS (default 2).
constexpr int kRestWide = 7000;
constexpr int kEeRec = 10;  // saved test: t, min_dist, P, Q, toc, iterations done or -1: bisect (the edges are recomputed)
struct EeArgs {
    int n_tp;
    const int32_t* items;
    const Entry* soup;
    const Entry* conn;
    const int32_t* nn_off;
    const int32_t* tp;
    const int32_t* ntris;
    const float* search;
    PrimResult* sub;
    PrimResult* cres;
    int32_t* chit;
    const double* pm;
    const double* tris;
    double* rec;     // kEeRec per listed test
    int32_t* work;   // the listed test's work item
    int32_t* count;  // [0] listed tests
    int first_iters;  // Newton iterations in the first pass
    int bounds;       // the FP32 bounds dropped tests before this
    int certificates;  // conservative-advancement cut-off of the first pass (results unchanged)
    unsigned long long* ca_stats;  // [0] tests cut, [1] Newton iterations they did not run
};

// Conservative advancement over an edge-edge test's linear motion: every
// endpoint moves on a straight line, so the points of the two edges at any
// time t' are within V |t' - t| of where they were at time t, V being the
// largest relative endpoint displacement |(aE.i - aS.i) - (bE.j - bS.j)| over
// the four endpoint pairs (a point of an edge is a convex combination of its
// endpoints, and so is its displacement).  Every distance edgeEdgeCCD
// evaluates after time t is therefore at least dist(t) - V max(t, 1 - t).
// When that and every distance evaluated so far are at least the search
// distance (plus a margin far above FP64 rounding), the test cannot hit, and
// a sub-test that cannot hit is never the best of a triangle pair that hits:
// it is recorded as no contact, as the FP32 and box bounds record theirs.
__device__ __forceinline__ double ee_motion_bound(const Edge& aS, const Edge& aE, const Edge& bS, const Edge& bE) {
    const V3 da0 = aE.A - aS.A, da1 = aE.B - aS.B, db0 = bE.A - bS.A, db1 = bE.B - bS.B;
    const V3 d00 = da0 - db0, d01 = da0 - db1, d10 = da1 - db0, d11 = da1 - db1;
    const double m = fmax(fmax(dot(d00, d00), dot(d01, d01)), fmax(dot(d10, d10), dot(d11, d11)));
    return sqrt(m);
}

// The gap between the boxes of the two edges' endpoints, start and end, passes lim.
__device__ __forceinline__ bool ee_boxes_apart(const Edge& aS, const Edge& aE, const Edge& bS, const Edge& bE,
                                               double lim) {
    auto gap = [](double a0, double a1, double a2, double a3, double b0, double b1, double b2, double b3) {
        return fmax(fmin(fmin(b0, b1), fmin(b2, b3)) - fmax(fmax(a0, a1), fmax(a2, a3)),
                    fmin(fmin(a0, a1), fmin(a2, a3)) - fmax(fmax(b0, b1), fmax(b2, b3)));
    };
    const double gx = fmax(0.0, gap(aS.A.x, aS.B.x, aE.A.x, aE.B.x, bS.A.x, bS.B.x, bE.A.x, bE.B.x));
    const double gy = fmax(0.0, gap(aS.A.y, aS.B.y, aE.A.y, aE.B.y, bS.A.y, bS.B.y, bE.A.y, bE.B.y));
    const double gz = fmax(0.0, gap(aS.A.z, aS.B.z, aE.A.z, aE.B.z, bS.A.z, bS.B.z, bE.A.z, bE.B.z));
    return (gx * gx + gy * gy) + gz * gz > lim * lim;
}

__device__ __forceinline__ void ee_store_at(const EeArgs& a, int o, float thr, const Ccd& r) {
    if (o < 0) {  // leaf-pair test: P and Q swapped (continuous_comparison.h:881-896)
        store_prim(a.cres + (-1 - o), r.dist, r.Q, r.P, r.toc);
        a.chit[-1 - o] = r.dist < (double)thr ? 1 : 0;
    } else {
        store_prim(a.sub + o, r.dist, r.P, r.Q, r.toc);
    }
}

// The gap between the edges along Q - P (of length d), at the start and at the
// end, is at least lim plus a margin (1 um and 1e-9 of the coordinates): no
// distance of the motion is below lim (the gap of linearly moving points is
// concave in time).
__device__ __forceinline__ bool ee_gap_clear(const Edge& aS, const Edge& aE, const Edge& bS, const Edge& bE, V3 P,
                                             V3 Q, double d, double lim) {
    const V3 n = Q - P;
    const double g0 = fmin(dot(n, bS.A), dot(n, bS.B)) - fmax(dot(n, aS.A), dot(n, aS.B));
    const double g1 = fmin(dot(n, bE.A), dot(n, bE.B)) - fmax(dot(n, aE.A), dot(n, aE.B));
    const double mag = fmax(fmax(fmax(fabs(aS.A.x), fabs(aS.A.y)), fabs(aS.A.z)),
                            fmax(fmax(fabs(bS.A.x), fabs(bS.A.y)), fabs(bS.A.z)));
    return fmin(g0, g1) >= ((lim + 1e-6) + 1e-9 * mag) * d;
}

// No point of the motion shortens the edge to nothing: its change is less than
// half of it.
__device__ __forceinline__ bool ee_steady(const Edge& S, const Edge& E) {
    const V3 v = S.B - S.A, w = (E.B - E.A) - v;
    return dot(w, w) < 0.25 * dot(v, v);
}

// The undecided slots of a level (list of node pair * 64 + slot): whether any
// of their 15 sub-tests (continuous_comparison.h:692-777) returns a distance
// below the search distance; a hit marks the node pair and ends its other
// slots.  A level leaves some ten to a few thousand slots, so the kernel lasts
// as long as one slot's chain of FP64 instructions (64 cycles each): a warp a
// slot, the vertices' start and end positions a component per lane, then the
// nine edge pairs on lanes 0-8 and the six point-triangle tests on lanes
// 16-21.  An edge pair is decided by its distance at the start (edgeEdgeCCD
// evaluates it first, and returns no more than it or at most 1e-8), or, as a
// certificate, by the
// gap along the direction between its points there, the smaller of the start's
// and the end's (the gap of linearly moving points is concave in time); the
// rest runs edgeEdgeCCD's iterates until a distance is below the limit, and its
// bisection (~370 FP64 instructions) last.  A thread per sub-test took 51 us a
// level on the 1,024-hull step.
__global__ void __launch_bounds__(kBlock) k_soup_slots(const int32_t* __restrict__ list,
                                                       const int32_t* __restrict__ n_list,
                                                       const Entry* __restrict__ soup, const double* __restrict__ pm,
                                                       const float* __restrict__ pm32, const double* __restrict__ tris,
                                                       const float* __restrict__ tri32,
                                                       const float* __restrict__ search, int32_t* entry_hits,
                                                       int certificates) {
    __shared__ double s_v[kBlock / 32][2][6][3];  // start, end; a's vertices, b's
    const int n = *n_list;
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    double(*v)[6][3] = s_v[wi];
    for (int k = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5); k < n;
         k += (int)((gridDim.x * (size_t)blockDim.x) >> 5)) {
        const int item = list[k], slot = item & ~kEdgesClear;
        const bool edges = !(item & kEdgesClear);
        if (__any_sync(0xffffffffu, ((volatile int32_t*)entry_hits)[slot >> 6] != 0)) continue;
        const Entry e = soup[slot >> 6];
        const int ta = (slot >> 3) & 7, tb = slot & 7;
        const float thr = search[e.pair];
        const double lim = (double)thr;
        const double* M = pm + (size_t)PM_SIZE * e.pair;
        const double* da = tris + (size_t)e.na * 72 + ta * 9;
        const double* db = tris + (size_t)e.nb * 72 + tb * 9;
        // the point-triangle tests the FP32 bounds leave
        bool pt = false;
        if (lane >= 16 && lane < 22) {
            const int i = (lane - 16) >> 1;
            const bool pb = (lane & 1) != 0;  // a vertex of b against a, else of a against b
            const float* fa = tri32 + ((size_t)e.na * 8 + ta) * 9;
            const float* fb = tri32 + ((size_t)e.nb * 8 + tb) * 9;
            pt = !pt_apart(pm32, e.pair, pb ? P32_BAS : P32_ABS, pb ? P32_AS : P32_BS, (pb ? fb : fa) + 3 * i,
                           pb ? fa : fb, thr);
        }
        if (!edges && !__any_sync(0xffffffffu, pt)) continue;
        for (int r = lane; r < 36; r += 32) {  // xform_rigid, a row each
            const int pose = r / 18, i = r % 18 / 3, c = r % 3;
            const double* T = M + (i < 3 ? (pose ? PM_AE : PM_AS) : (pose ? PM_BE : PM_BS)) + 4 * c;
            const double* p = i < 3 ? da + 3 * i : db + 3 * (i - 3);
            v[pose][i][c] = ((T[0] * p[0] + T[1] * p[1]) + T[2] * p[2]) + T[3] * 1.0;
        }
        __syncwarp();
        auto at = [&](int pose, int i) { return mk(v[pose][i][0], v[pose][i][1], v[pose][i][2]); };
        Edge aS, aE, bS, bE;
        V3 P, Q;
        EdgeDiv div;
        bool hit = false, open = edges && lane < 9, steady = false;
        if (open) {
            const int ia = lane / 3, ib = lane % 3, a1 = ia == 2 ? 0 : ia + 1, b1 = ib == 2 ? 0 : ib + 1;
            aS.A = at(0, ia);
            aS.B = at(0, a1);
            aE.A = at(1, ia);
            aE.B = at(1, a1);
            bS.A = at(0, 3 + ib);
            bS.B = at(0, 3 + b1);
            bE.A = at(1, 3 + ib);
            bE.B = at(1, 3 + b1);
            // while no edge can vanish on its way every distance is a number, and
            // any one below the limit makes the result one
            steady = thr > 1e-6f && ee_steady(aS, aE) && ee_steady(bS, bE);
            if (steady) {
                const double d0 = edge_closest(aS.A, aS.B, bS.A, bS.B, P, Q, div);
                hit = d0 < lim;
                open = !hit && !(certificates && ee_gap_clear(aS, aE, bS, bE, P, Q, d0, lim));
            }
        }
        bool any = __any_sync(0xffffffffu, hit);
        if (!any && __any_sync(0xffffffffu, open)) {
            if (open && steady) {
                // edgeEdgeCCD's iterates from the start's closest points, up to
                // the first below the limit or one whose gap clears the test
                double t = 0.0;
                Edge a = aS, b = bS;
                for (int iter = 1; iter < kEeNewtonIters && open; iter++) {
                    const double t_prev = t;
                    t = ee_newton_step(aS, aE, bS, bE, a, b, P, Q, div, t);
                    if (t == t_prev || t != t) break;
                    a.A = lerp(aS.A, aE.A, t);
                    a.B = lerp(aS.B, aE.B, t);
                    b.A = lerp(bS.A, bE.A, t);
                    b.B = lerp(bS.B, bE.B, t);
                    const double d = edge_closest(a.A, a.B, b.A, b.B, P, Q, div);
                    hit = d < lim;
                    open = !hit && !(certificates && ee_gap_clear(aS, aE, bS, bE, P, Q, d, lim));
                }
            }
            any = __any_sync(0xffffffffu, hit);
        }
        if (!any && pt) {
            const int i = (lane - 16) >> 1;
            const bool pb = (lane & 1) != 0;
            const double* p = (pb ? db : da) + 3 * i;
            hit = point_tri_ccd(mk(p[0], p[1], p[2]), M + (pb ? PM_BAS : PM_ABS), M + (pb ? PM_BAE : PM_ABE),
                                load_tri(pb ? da : db), M + (pb ? PM_AS : PM_BS), M + (pb ? PM_AE : PM_BE))
                      .dist < lim;
        }
        any = any || __any_sync(0xffffffffu, hit);
        if (!any && __any_sync(0xffffffffu, open)) {
            // the bisection's distance, and the whole of an unsteady test
            if (open) {
                Ccd r;
                double best = DBL_MAX;
                const double dot_start = ee_coplanarity(aS, bS);
                if (dot_start * ee_coplanarity(aE, bE) < 0.0) best = ee_bisect(aS, aE, bS, bE, dot_start, r);
                hit = best < lim;
                if (!steady && !hit && best > 1e-8) {
                    double t = 0.0;
                    for (int iter = 0; iter < kEeNewtonIters; iter++)
                        if (ee_newton_iter(aS, aE, bS, bE, t, best, r)) break;
                    hit = best < lim;
                }
            }
            any = __any_sync(0xffffffffu, hit);
        }
        if (any && lane == 0) entry_hits[slot >> 6] = 1;
        __syncwarp();
    }
}

// The same without FP32 bounds (the list holds every slot of the level), a
// thread a test; without the certificates too, each the reference's whole one.
__global__ void __launch_bounds__(kPrimBlock) k_soup_tests(const int32_t* __restrict__ list,
                                                           const int32_t* __restrict__ n_list,
                                                           const Entry* __restrict__ soup,
                                                           const double* __restrict__ pm,
                                                           const double* __restrict__ tris,
                                                           const float* __restrict__ search, int32_t* entry_hits,
                                                           int certificates) {
    const int n = *n_list;
    const long long n_ee = 9LL * n, total = 15LL * n;
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < total;
         j += (long long)gridDim.x * blockDim.x) {
        const bool ee = j < n_ee;
        const int k = (int)(ee ? j / 9 : (j - n_ee) / 6), q = (int)(ee ? j % 9 : (j - n_ee) % 6);
        const int slot = list[k] & ~kEdgesClear;
        if (((volatile int32_t*)entry_hits)[slot >> 6]) continue;
        const Entry e = soup[slot >> 6];
        const double* M = pm + (size_t)PM_SIZE * e.pair;
        const Tri A = load_tri(tris + (size_t)e.na * 72 + ((slot >> 3) & 7) * 9);
        const Tri B = load_tri(tris + (size_t)e.nb * 72 + (slot & 7) * 9);
        double dist;
        if (ee) {
            const Edge ea = tedge(A, q / 3), eb = tedge(B, q % 3);
            Edge aS, aE, bS, bE;
            aS.A = xform_rigid(ea.A, M + PM_AS);
            aS.B = xform_rigid(ea.B, M + PM_AS);
            bS.A = xform_rigid(eb.A, M + PM_BS);
            bS.B = xform_rigid(eb.B, M + PM_BS);
            aE.A = xform_rigid(ea.A, M + PM_AE);
            aE.B = xform_rigid(ea.B, M + PM_AE);
            bE.A = xform_rigid(eb.A, M + PM_BE);
            bE.B = xform_rigid(eb.B, M + PM_BE);
            const double lim = (double)search[e.pair];
            V3 P, Q;
            // as in k_soup_slots, else the whole test
            const bool brief = certificates && lim > 1e-6 && ee_steady(aS, aE) && ee_steady(bS, bE);
            dist = brief ? edge_closest(aS.A, aS.B, bS.A, bS.B, P, Q) : lim;
            if (!(dist < lim) && !(brief && ee_gap_clear(aS, aE, bS, bE, P, Q, dist, lim)))
                dist = edge_edge_ccd(aS, aE, bS, bE).dist;
        } else if (q & 1) {
            dist = point_tri_ccd(tvert(B, q >> 1), M + PM_BAS, M + PM_BAE, A, M + PM_AS, M + PM_AE).dist;
        } else {
            dist = point_tri_ccd(tvert(A, q >> 1), M + PM_ABS, M + PM_ABE, B, M + PM_BS, M + PM_BE).dist;
        }
        if (dist < (double)search[e.pair]) entry_hits[slot >> 6] = 1;
    }
}

__global__ void __launch_bounds__(kPrimBlock) k_ee_first(int n_total, const int32_t* __restrict__ list,
                                                         const int32_t* __restrict__ n_list,
                                                         const double* __restrict__ pm,
                                                         const double* __restrict__ tris, EeArgs a) {
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    bool keep = false;
    int o = 0;
    float thr = 0.f;
    Edge aS, aE, bS, bE;
    Ccd r;
    double min_dist = DBL_MAX, t = 0.0;
    int iters = 0;
    if (kk < n_total && kk < *n_list) {
        const int j = list[kk];
        const EeWork w = decode_ee(j, a.n_tp, a.items, a.soup, a.conn, a.nn_off, a.tp, a.ntris, a.sub, a.cres,
                                   a.chit);
        o = w.hit ? -1 - (int)(w.out - a.cres) : (int)(w.out - a.sub);
        thr = a.search[w.pair];
        const double* M = pm + (size_t)PM_SIZE * w.pair;
        const Edge ea = tedge(load_tri(tris + (size_t)w.na * 72 + w.aTri * 9), w.aEdge);
        const Edge eb = tedge(load_tri(tris + (size_t)w.nb * 72 + w.bTri * 9), w.bEdge);
        aS.A = xform_rigid(ea.A, M + PM_AS);
        aS.B = xform_rigid(ea.B, M + PM_AS);
        aE.A = xform_rigid(ea.A, M + PM_AE);
        aE.B = xform_rigid(ea.B, M + PM_AE);
        bS.A = xform_rigid(eb.A, M + PM_BS);
        bS.B = xform_rigid(eb.B, M + PM_BS);
        bE.A = xform_rigid(eb.A, M + PM_BE);
        bE.B = xform_rigid(eb.B, M + PM_BE);
        // Without the FP32 bounds: every distance edgeEdgeCCD can return is
        // between points of the two swept segments, which lie in the boxes of
        // their four endpoint positions, so a box gap beyond the search distance
        // (plus 1e-7 m, far above FP64 rounding at scene scale) means no hit.
        if (!a.bounds && ee_boxes_apart(aS, aE, bS, bE, (double)thr + 1e-7)) {
            record_no_contact(w.out, w.hit);
        } else {
            r.P = mk(0, 0, 0);
            r.Q = mk(0, 0, 0);
            r.toc = 0.0;
            const double dot_start = ee_coplanarity(aS, bS);
            const double dot_end = ee_coplanarity(aE, bE);
            const bool bisect = dot_start * dot_end < 0.0;
            bool done = false, cut = false;
            if (bisect) {
                iters = -1;  // in the second pass
            } else {
                for (; iters < a.first_iters; iters++) {
                    const double t_at = t;
                    double d_at;
                    if (ee_newton_iter(aS, aE, bS, bE, t, min_dist, r, &d_at)) {
                        done = true;
                        break;
                    }
                    if (a.certificates && min_dist >= (double)thr) {
                        const double V = ee_motion_bound(aS, aE, bS, bE);
                        const double mag = fmax(fmax(fmax(fabs(aS.A.x), fabs(aS.A.y)), fabs(aS.A.z)),
                                                fmax(fmax(fabs(bS.A.x), fabs(bS.A.y)), fabs(bS.A.z)));
                        const double lim = ((double)thr + 1e-6) + 1e-12 * (mag + V);
                        if (min_dist >= lim && d_at - V * fmax(t_at, 1.0 - t_at) >= lim) {
                            cut = true;
                            iters++;
                            break;
                        }
                    }
                }
            }
            if (cut) {
                record_no_contact(w.out, w.hit);
                atomicAdd(a.ca_stats, 1ull);
                atomicAdd(a.ca_stats + 1, (unsigned long long)(kEeNewtonIters - iters));
            } else if (done) {
                r.dist = min_dist;
                ee_store_at(a, o, thr, r);
            } else {
                keep = true;  // the rest runs in the second pass
            }
        }
    }
    // warp-aggregated append of the tests still running
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (m) {
        const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
        int base = 0;
        if (lane == lead) base = atomicAdd(a.count, __popc(m));
        base = __shfl_sync(0xffffffffu, base, lead);
        if (keep) {
            const int slot = base + __popc(m & ((1u << lane) - 1u));
            double* R = a.rec + (size_t)kEeRec * slot;
            const double st[kEeRec] = {t, min_dist, r.P.x, r.P.y, r.P.z, r.Q.x, r.Q.y, r.Q.z, r.toc, (double)iters};
#pragma unroll
            for (int k = 0; k < kEeRec; k++) R[k] = st[k];
            a.work[slot] = list[kk];
        }
    }
}

// ---- the Newton phase on four lanes per test ------------------------------
// GB300 issues an FP64 warp instruction at the same cost whatever the number
// of active lanes, and a level has far fewer surviving edge-edge tests than
// the GPU has lanes, so a test's time is the number of FP64 instructions on
// its path.  Here each test runs on a quad of lanes: lane c < 3 holds
// component c of every point (lane 3 mirrors x), vector operations are one
// instruction for all three components, a dot product is one multiply and the
// two adds (x + y) + z of the reference's order, and independent divisions
// share one instruction stream on different lanes.  Scalars are computed
// identically on all four lanes, so every branch is uniform within a quad.
// Every value is produced by the same operations, in the same order, as in
// edge_edge_ccd.
struct Quad {
    unsigned m;  // the quad's lanes
    int base;    // its first lane
    int c;       // this lane's component (3: mirror of x)
};
__device__ __forceinline__ double q_at(const Quad& q, double v, int k) { return __shfl_sync(q.m, v, q.base + k); }
__device__ __forceinline__ double q_dot(const Quad& q, double a, double b) {
    const double p = a * b;
    const double px = q_at(q, p, 0), py = q_at(q, p, 1), pz = q_at(q, p, 2);
    return (px + py) + pz;
}
__device__ __forceinline__ double q_lerp(double A, double B, double t) {
    const double u = 1 - t;
    return A * u + B * t;
}
// components differ anywhere (vne)
__device__ __forceinline__ bool q_ne(const Quad& q, double a, double b) {
    const unsigned bal = __ballot_sync(q.m, q.c < 3 && m_ne(a, b));
    return ((bal >> q.base) & 7u) != 0u;
}
// m_div_recip by the squared length of an edge (rl: its reciprocal), clamped.
__device__ __forceinline__ double q_lerp_at(double A, double B, double n, double l, double rl) {
    return q_lerp(A, B, clamp01(m_div_recip(n, l, rl)));
}
// edge_closest(SA, SB, EA, EB, P, Q): one component per lane.  The squared
// lengths of the edges and their reciprocals (one division, on different
// lanes) serve all five divisions by them.
struct QuadDiv {
    double S, rS, E, rE;  // of (SA, SB) and (EA, EB)
};
__device__ __forceinline__ double q_edge_closest(const Quad& q, double SA, double SB, double EA, double EB, double& P,
                                                 double& Qo, QuadDiv& d) {
    const double segDC = EB - EA, segAB = SB - SA;
    d.E = q_dot(q, segDC, segDC);
    d.S = q_dot(q, segAB, segAB);
    const double rl = 1.0 / ((q.c & 1) ? d.S : d.E);
    d.rE = q_at(q, rl, 0);
    d.rS = q_at(q, rl, 1);
    const double segAC = SA - EA;
    const double segBC = SB - EA;
    const double nA = q_dot(q, segAC, segDC), nB = q_dot(q, segBC, segDC);
    const double s2 = m_div_recip((q.c & 1) ? nB : nA, d.E, d.rE);  // lanes 0, 2: A; 1, 3: B
    const double sA = q_at(q, s2, 0), sB = q_at(q, s2, 1);
    const double inPlaneA = SA - sA * segDC;
    const double inPlaneB = SB - sB * segDC;
    const double inPlaneBA = inPlaneB - inPlaneA;
    double t = q_dot(q, EA - inPlaneA, inPlaneBA) / q_dot(q, inPlaneBA, inPlaneBA);
    t = q_ne(q, inPlaneA, inPlaneB) ? t : 0.0;
    const double segABtoLineCD = q_lerp(SA, SB, clamp01(t));
    Qo = q_lerp_at(EA, EB, q_dot(q, segABtoLineCD - EA, segDC), d.E, d.rE);
    P = q_lerp_at(SA, SB, q_dot(q, Qo - SA, segAB), d.S, d.rS);
    const double v = Qo - P;
    return sqrt(q_dot(q, v, v));
}

// ee_coplanarity of edges (aA, aB), (bA, bB), one component per lane
__device__ __forceinline__ double q_coplanarity(const Quad& q, double aA, double aB, double bA, double bB) {
    const int c1 = q.c == 1 ? 2 : (q.c == 2 ? 0 : 1), c2 = q.c == 1 ? 0 : (q.c == 2 ? 1 : 2);
    const double u = aB - aA, v = bA - aA, w = bB - aA;
    return q_dot(q, w, q_at(q, u, c1) * q_at(q, v, c2) - q_at(q, u, c2) * q_at(q, v, c1));
}

// ee_cubic, one component per lane.
__device__ __forceinline__ EeCubic q_cubic(const Quad& q, double aSA, double aSB, double bSA, double bSB, double aEA,
                                           double aEB, double bEA, double bEB) {
    const int c1 = q.c == 1 ? 2 : (q.c == 2 ? 0 : 1), c2 = q.c == 1 ? 0 : (q.c == 2 ? 1 : 2);
    const double u0 = aSB - aSA, v0 = bSA - aSA, w0 = bSB - aSA;
    const double uE = aEB - aEA, vE = bEA - aEA, wE = bEB - aEA;
    const double u1 = uE - u0, v1 = vE - v0, w1 = wE - w0;
    const double u01 = q_at(q, u0, c1), u02 = q_at(q, u0, c2), v01 = q_at(q, v0, c1), v02 = q_at(q, v0, c2);
    const double u11 = q_at(q, u1, c1), u12 = q_at(q, u1, c2), v11 = q_at(q, v1, c1), v12 = q_at(q, v1, c2);
    const double n0 = u01 * v02 - u02 * v01, n2 = u11 * v12 - u12 * v11;
    const double n1 = (u01 * v12 - u02 * v11) + (u11 * v02 - u12 * v01);
    auto sum = [&](double p) { return (q_at(q, p, 0) + q_at(q, p, 1)) + q_at(q, p, 2); };
    EeCubic c;
    c.c0 = sum(w0 * n0);
    c.c1 = sum(w0 * n1 + w1 * n0);
    c.c2 = sum(w0 * n2 + w1 * n1);
    c.c3 = sum(w1 * n2);
    const uint32_t l = max_hi3(max_hi3(0, mk(u0, v0, w0)), mk(uE, vE, wE));
    const uint32_t m = m_max_hi(m_max_hi(max_hi3(max_hi3(0, mk(aSA, aSB, bSA)), mk(aEA, aEB, bEA)), bSB), bEB);
    c.err = ee_cubic_err(__reduce_max_sync(q.m, m), __reduce_max_sync(q.m, l));
    return c;
}

__global__ void __launch_bounds__(kBlock) k_ee_rest4(EeArgs a) {
    const int n = a.count[0];
    if (n > kRestWide) return;  // k_ee_rest1
    Quad q;
    q.m = 0xFu << (threadIdx.x & 28);
    q.base = threadIdx.x & 28;
    q.c = threadIdx.x & 3;
    const int comp = q.c < 3 ? q.c : 0;
    const int n_quads = (gridDim.x * blockDim.x) >> 2;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; i < n; i += n_quads) {
        const double* R = a.rec + (size_t)kEeRec * i;
        const EeWork w = decode_ee(a.work[i], a.n_tp, a.items, a.soup, a.conn, a.nn_off, a.tp, a.ntris, a.sub,
                                   a.cres, a.chit);
        // this lane's component of the edges' endpoints at start and end
        // (xform_rigid's row `comp`, the same operations in the same order)
        const double* M = a.pm + (size_t)PM_SIZE * w.pair;
        const double* ta = a.tris + (size_t)w.na * 72 + w.aTri * 9;
        const double* tb = a.tris + (size_t)w.nb * 72 + w.bTri * 9;
        const double* va0 = ta + 3 * w.aEdge;
        const double* va1 = ta + 3 * (w.aEdge == 2 ? 0 : w.aEdge + 1);
        const double* vb0 = tb + 3 * w.bEdge;
        const double* vb1 = tb + 3 * (w.bEdge == 2 ? 0 : w.bEdge + 1);
        auto row = [&](const double* T, const double* v) {
            const double* m = T + 4 * comp;
            return ((m[0] * v[0] + m[1] * v[1]) + m[2] * v[2]) + m[3] * 1.0;
        };
        const double aSA = row(M + PM_AS, va0), aSB = row(M + PM_AS, va1);
        const double aEA = row(M + PM_AE, va0), aEB = row(M + PM_AE, va1);
        const double bSA = row(M + PM_BS, vb0), bSB = row(M + PM_BS, vb1);
        const double bEA = row(M + PM_BE, vb0), bEB = row(M + PM_BE, vb1);
        double t = R[0], min_dist = R[1];
        double rP = R[2 + comp], rQ = R[5 + comp], toc = R[8];
        int iter = (int)R[9];
        QuadDiv div;
        if (iter < 0) {  // ee_bisect
            iter = 0;
            const double dot_start = q_coplanarity(q, aSA, aSB, bSA, bSB);
            const EeCubic cubic = q_cubic(q, aSA, aSB, bSA, bSB, aEA, aEB, bEA, bEB);
            double lo = 0.0, hi = 1.0;
            for (int k = 0; k < 20; k++) {
                const double mid = (lo + hi) / 2.0;
                int side = ee_bisect_side(cubic.at(mid), cubic.err, dot_start);
                if (side < 0) {
                    const double dm = q_coplanarity(q, q_lerp(aSA, aEA, mid), q_lerp(aSB, aEB, mid),
                                                    q_lerp(bSA, bEA, mid), q_lerp(bSB, bEB, mid));
                    side = fabs(dm) < 1e-8 ? 1 : (dot_start * dm < 0.0 ? 2 : 0);
                }
                if (side == 1) {
                    lo = mid;
                    hi = mid;
                    break;
                } else if (side == 2) {
                    hi = mid;
                } else {
                    lo = mid;
                }
            }
            toc = (lo + hi) / 2.0;
            min_dist = q_edge_closest(q, q_lerp(aSA, aEA, toc), q_lerp(aSB, aEB, toc), q_lerp(bSA, bEA, toc),
                                      q_lerp(bSB, bEB, toc), rP, rQ, div);
            if (!(min_dist > 1e-8)) iter = kEeNewtonIters;
        }
        for (; iter < kEeNewtonIters; iter++) {
            const double atA = q_lerp(aSA, aEA, t), atB = q_lerp(aSB, aEB, t);
            const double btA = q_lerp(bSA, bEA, t), btB = q_lerp(bSB, bEB, t);
            double P, Qv;
            const double dist = q_edge_closest(q, atA, atB, btA, btB, P, Qv, div);
            if (dist < min_dist) {
                min_dist = dist;
                rP = P;
                rQ = Qv;
                toc = t;
            }
            // edge_project(atA, atB, P) and edge_project(btA, btB, Q), divided on lanes 0 / 1
            const double na = q_dot(q, P - atA, atB - atA), nb = q_dot(q, Qv - btA, btB - btA);
            const double pr = m_div_recip((q.c & 1) ? nb : na, (q.c & 1) ? div.E : div.S, (q.c & 1) ? div.rE : div.rS);
            const double pa = q_at(q, pr, 0), pb = q_at(q, pr, 1);
            // ee_newton_terms, component per lane
            const double omt = 1 - t, ompa = 1 - pa, ompb = 1 - pb, pbm1 = pb - 1;
            const double f = ((pa * (aEB + aSB * omt) - pb * (bEB + bSB * omt)) + ompa * atA) - ompb * btA;
            const double p1 = aSB * pa, p2 = bSB * pb, p3 = ompa * (aEA - aSA), p4 = (bEA - bSA) * pbm1;
            const double G = ((p2 - p1) + p3) + p4;
            double gf2 = G * f, gh = G * G;
            const double ff = f * f;
            if (__any_sync(q.m, !(m_scalable(p1) && m_scalable(p2) && m_scalable(p3) && m_scalable(p4) &&
                                  m_scalable(gf2) && (!m_is_zero(gf2) || m_is_zero(G) || m_is_zero(f))))) {
                const double g = ((-2 * aSB * pa + 2 * bSB * pb) + 2 * ompa * (aEA - aSA)) + 2 * (bEA - bSA) * pbm1;
                const double h = ((-aSB * pa / 2 + bSB * pb / 2) + ompa * (aEA - aSA) / 2) + (bEA - bSA) * pbm1 / 2;
                gf2 = g * f / 2;
                gh = g * h;
            }
            const double gf = (q_at(q, gf2, 0) + q_at(q, gf2, 1)) + q_at(q, gf2, 2);
            const double S = (q_at(q, ff, 0) + q_at(q, ff, 1)) + q_at(q, ff, 2);
            const double GH = (q_at(q, gh, 0) + q_at(q, gh, 1)) + q_at(q, gh, 2);
            const double sS = sqrt(S);
            // gf / sS, GH / sS and (-gf * gf) / pow15(S) on lanes 0, 1, 2
            const double num = q.c == 1 ? GH : (q.c == 2 ? (-gf) * gf : gf);
            const double den = q.c == 2 ? m_pow15(S) : sS;
            const double quo = num / den;
            const double t_diff = q_at(q, quo, 0);
            const double t_diff2 = q_at(q, quo, 1) + q_at(q, quo, 2);
            const double t_prev = t;
            t = t - t_diff / t_diff2;
            t = clamp01(t);
            if (t == t_prev || t != t) break;
        }
        const double Px = q_at(q, rP, 0), Py = q_at(q, rP, 1), Pz = q_at(q, rP, 2);
        const double Qx = q_at(q, rQ, 0), Qy = q_at(q, rQ, 1), Qz = q_at(q, rQ, 2);
        if (q.c == 0) {
            Ccd r;
            r.dist = min_dist;
            r.P = mk(Px, Py, Pz);
            r.Q = mk(Qx, Qy, Qz);
            r.toc = toc;
            ee_store_at(a, w.hit ? -1 - (int)(w.out - a.cres) : (int)(w.out - a.sub), a.search[w.pair], r);
        }
    }
}

__global__ void __launch_bounds__(kPrimBlock) k_ee_rest1(EeArgs a) {
    const int n = a.count[0];
    if (n <= kRestWide) return;  // k_ee_rest4
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double* R = a.rec + (size_t)kEeRec * i;
        const EeWork w = decode_ee(a.work[i], a.n_tp, a.items, a.soup, a.conn, a.nn_off, a.tp, a.ntris, a.sub, a.cres,
                                   a.chit);
        const double* M = a.pm + (size_t)PM_SIZE * w.pair;
        const Edge ea = tedge(load_tri(a.tris + (size_t)w.na * 72 + w.aTri * 9), w.aEdge);
        const Edge eb = tedge(load_tri(a.tris + (size_t)w.nb * 72 + w.bTri * 9), w.bEdge);
        Edge aS, aE, bS, bE;
        aS.A = xform_rigid(ea.A, M + PM_AS);
        aS.B = xform_rigid(ea.B, M + PM_AS);
        aE.A = xform_rigid(ea.A, M + PM_AE);
        aE.B = xform_rigid(ea.B, M + PM_AE);
        bS.A = xform_rigid(eb.A, M + PM_BS);
        bS.B = xform_rigid(eb.B, M + PM_BS);
        bE.A = xform_rigid(eb.A, M + PM_BE);
        bE.B = xform_rigid(eb.B, M + PM_BE);
        double t = R[0], min_dist = R[1];
        Ccd r;
        r.P = mk(R[2], R[3], R[4]);
        r.Q = mk(R[5], R[6], R[7]);
        r.toc = R[8];
        int iter = (int)R[9];
        if (iter < 0) {
            iter = 0;
            min_dist = ee_bisect(aS, aE, bS, bE, ee_coplanarity(aS, bS), r);
            if (!(min_dist > 1e-8)) iter = kEeNewtonIters;
        }
        for (; iter < kEeNewtonIters; iter++)
            if (ee_newton_iter(aS, aE, bS, bE, t, min_dist, r)) break;
        r.dist = min_dist;
        ee_store_at(a, w.hit ? -1 - (int)(w.out - a.cres) : (int)(w.out - a.sub), a.search[w.pair], r);
    }
}

// triTriCCDLinear's sequential (dist, toc) selection over its 15 sub-tests
// (continuous_comparison.h:682-778), then the soup hit test (:817).
__global__ void k_soup_fold(int K, const int32_t* __restrict__ items, const Entry* __restrict__ soup,
                            const PrimResult* __restrict__ sub, const float* __restrict__ search,
                            PrimResult* __restrict__ res, int32_t* __restrict__ hit) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    PrimResult best;
    best.dist = 1.0 / 0.0;
    best.P[0] = best.P[1] = best.P[2] = 0.0;
    best.Q[0] = best.Q[1] = best.Q[2] = 0.0;
    best.toc = 1.0;
    for (int s = 0; s < 15; s++) {
        const PrimResult c = sub[15 * (size_t)k + s];
        if (c.dist < best.dist || (c.dist == best.dist && c.toc < best.toc)) best = c;
    }
    res[k] = best;
    const Entry e = soup[items[k] >> 6];
    hit[k] = best.dist < (double)search[e.pair] ? 1 : 0;
}

// ----------------------------------------------------------- discrete -----
// Candidate slots of the discrete narrow phase.  A (node pair, ta, tb) slot
// can only hit (comparison_dist.h:231-233) when the triangles are closer than
// thr = search + eps_a + eps_b.  Lower bounds on that distance: the bounding
// spheres' |c_a - c_b| - r_a - r_b (centroid, radius rounded up), the gap
// between the boxes of the transformed triangles and, for slots those keep,
// the gaps along the two face normals and the direction between the closest
// edges.  The largest is evaluated in FP32 and a slot is dropped
// only when it exceeds thr by a margin
// (20 um plus 4e-6 of the magnitudes involved) far above the FP32 rounding of
// the bound (3e-7 of them) and the FP64 rounding of the exact test, so every
// slot that hits survives.  Dropped slots produce nothing in the reference
// either.  (A triangle that is a point, or not finite, is the exception: the
// reference's distance to it can be 0 with no feature at all (d2g_prune.cuh),
// wherever the other triangle is.  Such slots are kept within 1 mm of the limit
// by the spheres and boxes, and decided by the whole distance.)
//
// A warp per node pair: lanes 0-7 transform a's triangles, 8-15 b's, once each
// into shared memory, with their normals; every lane takes two of the 64 slots
// through the spheres, boxes and normals; what is left is packed onto the first
// lanes for the edges, ~400 instructions of the ~700.  Bounded by issue (67%)
// at 34% occupancy: 1,024 hulls' 355,000 leaf pairs 258 us, their four levels
// 207 us (323 and 257 with the edges before the normals, two slots a lane and
// unfused products; a thread per slot, transforming both triangles of each:
// 870 us).  Rejecting by spheres before the other bounds are prepared, or a
// cap of 64 registers, gained nothing.
//
// LEAF: the node pair's contacts are wanted; the survivors as two mask words
// and counts.  Otherwise the pair has an inner node and emits nothing: all the
// descent needs of it is whether some slot hits.  The exact distance is at most
// that of any edge pair, so a slot whose vertices, or else edges, are closer
// than thr by the same margin certainly hits (unless a triangle is almost a
// point, whose edges return no distance); the pair is marked and done, and only
// the survivors of the others go onto `list` for k_np_slots.
__device__ __forceinline__ float box_gap9(const float* a, const float* b) {
    float gap2 = 0.f;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const float alo = fminf(fminf(a[r], a[3 + r]), a[6 + r]), ahi = fmaxf(fmaxf(a[r], a[3 + r]), a[6 + r]);
        const float blo = fminf(fminf(b[r], b[3 + r]), b[6 + r]), bhi = fmaxf(fmaxf(b[r], b[3 + r]), b[6 + r]);
        const float g = fmaxf(blo - ahi, alo - bhi);
        if (g > 0.f) gap2 += g * g;
    }
    return sqrtf(gap2);
}

// The gap along a triangle's unit normal (n: the normal, the triangle's range
// along it) to the triangle v.
__device__ __forceinline__ float normal_gap(const float* n, const float* v) {
    const F3 d = f3(n[0], n[1], n[2]);
    const float p0 = dot3(d, f3(v[0], v[1], v[2])), p1 = dot3(d, f3(v[3], v[4], v[5])),
                p2 = dot3(d, f3(v[6], v[7], v[8]));
    return fmaxf(fminf(p0, fminf(p1, p2)) - n[4], n[3] - fmaxf(p0, fmaxf(p1, p2)));
}

// Marks a slot of k_np_filter's list that only the whole distance decides: a
// triangle that is a point or not finite, or one that is kFarSizes away.
constexpr int kWholeTest = kSlotMark;

template <bool LEAF>
__global__ void __launch_bounds__(kBlock, LEAF ? 7 : 6) k_np_filter(int n, const Entry* __restrict__ front,
                                                      const float* __restrict__ pm32, const int32_t* __restrict__ ntris,
                                                      const float4* __restrict__ sph, const float* __restrict__ tri32,
                                                      const float* __restrict__ eps_up,
                                                      const float* __restrict__ search,
                                                      const int4* __restrict__ nodes, int use_bounds,
                                                      uint32_t* __restrict__ mask, int32_t* __restrict__ cnt,
                                                      int32_t* __restrict__ entry_hits, int32_t* __restrict__ list,
                                                      int32_t* __restrict__ lc, const int32_t* __restrict__ n_dev) {
    __shared__ float s_v[kBlock / 32][16][9];
    // centre, radius, eps, magnitude, size (0 for a triangle that is a point or
    // not finite), unit normal, the triangle's own range along it
    __shared__ float s_c[kBlock / 32][16][13];
    __shared__ uint8_t s_slot[kBlock / 32][64];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    if (!LEAF && n_dev) n = *n_dev;
    for (int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5); w < n;  // uniform per warp
         w += (int)((gridDim.x * (size_t)blockDim.x) >> 5)) {
        __syncwarp();
        const Entry e = front[w];
        if (!LEAF && !ld_node(nodes, e.na).z && !ld_node(nodes, e.nb).z) {
            // a root pair of two leaves goes onto the list of leaf pairs as it is
            if (lane == 0) {
                entry_hits[w] = 1;
                atomicAdd(lc + LC_ROOT, 1);
            }
            continue;
        }
        const int na = ntris[e.na], nb = ntris[e.nb];
        const float* PA = pm32 + kNpPose32 * (size_t)e.pair;
        const float* PB = PA + 12;
        if (lane < 16 && (lane & 7) < (lane < 8 ? na : nb)) {
            const size_t t = (size_t)(lane < 8 ? e.na : e.nb) * 8 + (lane & 7);
            const float* M = lane < 8 ? PA : PB;
            const float* tv = tri32 + t * 9;
            float* v = s_v[wi][lane];
            float* c = s_c[wi][lane];
            const float4 sp = sph[t];
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float m0 = M[4 * r], m1 = M[4 * r + 1], m2 = M[4 * r + 2], m3 = M[4 * r + 3];
                c[r] = fmaf(m0, sp.x, fmaf(m1, sp.y, fmaf(m2, sp.z, m3)));
#pragma unroll
                for (int k = 0; k < 3; k++) v[3 * k + r] = fmaf(m0, tv[3 * k], fmaf(m1, tv[3 * k + 1], fmaf(m2, tv[3 * k + 2], m3)));
            }
            c[3] = sp.w;
            c[4] = eps_up[t];
            c[5] = fabsf(sp.x) + fabsf(sp.y) + fabsf(sp.z) + sp.w;
            float ext = 0.f;
#pragma unroll
            for (int r = 0; r < 3; r++) ext = fmaxf(ext, fmaxf(fabsf(v[3 + r] - v[r]), fabsf(v[6 + r] - v[r])));
            c[6] = ext > 1e-5f && ext < 1e15f ? ext : 0.f;
            F3 nn = cross3(f3(v[3] - v[0], v[4] - v[1], v[5] - v[2]), f3(v[6] - v[0], v[7] - v[1], v[8] - v[2]));
            const float len = sqrtf(dot3(nn, nn)), inv = len > 1e-20f ? 1.f / len : 0.f;
            nn = f3(nn.x * inv, nn.y * inv, nn.z * inv);
            const float p0 = dot3(nn, f3(v[0], v[1], v[2])), p1 = dot3(nn, f3(v[3], v[4], v[5])),
                        p2 = dot3(nn, f3(v[6], v[7], v[8]));
            c[7] = nn.x;
            c[8] = nn.y;
            c[9] = nn.z;
            c[10] = fminf(p0, fminf(p1, p2));
            c[11] = fmaxf(p0, fmaxf(p1, p2));
        }
        if (lane == 0) atomicAdd(lc + LC_TRI + (w & (LC_TRI_N - 1)), na * nb);
        const float se = search[e.pair];
        const bool rigid = PA[24] != 0.f;  // else the spheres' radii are not the triangles'
        const float tm = fabsf(PA[3]) + fabsf(PA[7]) + fabsf(PA[11]) + fabsf(PB[3]) + fabsf(PB[7]) + fabsf(PB[11]);
        __syncwarp();
        // the bounds that each triangle's own data give, two slots a lane
        const int ta0 = lane >> 3, tb0 = lane & 7;
        unsigned m[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int ta = ta0 + 4 * h;
            bool keep = ta < na && tb0 < nb;
            if (keep && use_bounds) {
                const float *ca = s_c[wi][ta], *cb = s_c[wi][8 + tb0], *va = s_v[wi][ta], *vb = s_v[wi][8 + tb0];
                const float dx = ca[0] - cb[0], dy = ca[1] - cb[1], dz = ca[2] - cb[2];
                const float thr = se + ca[4] + cb[4];
                const bool plain = !(fminf(ca[6], cb[6]) > 0.f);
                const float lim = thr + ((plain ? 1e-3f : 2e-5f) + 4e-6f * (tm + ca[5] + cb[5] + thr));
                keep = !(rigid && sqrtf(dx * dx + dy * dy + dz * dz) - ca[3] - cb[3] > lim) &&  // NaN keeps the slot
                       !(box_gap9(va, vb) > lim) &&
                       (plain || (!(normal_gap(ca + 7, vb) > lim) && !(normal_gap(cb + 7, va) > lim)));
            }
            m[h] = __ballot_sync(0xffffffffu, keep);
        }
        const int k0 = __popc(m[0]), K = k0 + __popc(m[1]);
        if (use_bounds && K > 0) {
            // the others, packed, a slot a lane
            const unsigned low = (1u << lane) - 1u;
            if ((m[0] >> lane) & 1u) s_slot[wi][__popc(m[0] & low)] = (uint8_t)lane;
            if ((m[1] >> lane) & 1u) s_slot[wi][k0 + __popc(m[1] & low)] = (uint8_t)(32 + lane);
            __syncwarp();
            auto room = [&](const float* ca, const float* cb) {
                const float thr = se + ca[4] + cb[4];
                return fminf(ca[6], cb[6]) > 0.f ? thr - (2e-5f + 4e-6f * (tm + ca[5] + cb[5] + thr)) : -1.f;
            };
            if (!LEAF) {
                bool sure = false;
                for (int k = lane; k < K; k += 32) {
                    const int ta = s_slot[wi][k] >> 3, tb = 8 + (s_slot[wi][k] & 7);
                    const float rm = room(s_c[wi][ta], s_c[wi][tb]);
                    sure = sure || (rm > 0.f && vert_min(s_v[wi][ta], s_v[wi][tb]) < rm);
                }
                if (__any_sync(0xffffffffu, sure)) {
                    if (lane == 0) entry_hits[w] = 1;
                    continue;
                }
            }
            m[0] = m[1] = 0;
            bool sure = false;
            for (int base = 0; base < K; base += 32) {
                const int k = min(base + lane, K - 1), sl = s_slot[wi][k], ta = sl >> 3, tb = 8 + (sl & 7);
                const float *ca = s_c[wi][ta], *cb = s_c[wi][tb], *va = s_v[wi][ta], *vb = s_v[wi][tb];
                F3 d;
                const float dist = edge_min(va, vb, d);
                if (!LEAF && __any_sync(0xffffffffu, dist < room(ca, cb))) {
                    sure = true;
                    break;
                }
                const float thr = se + ca[4] + cb[4], lim = thr + (2e-5f + 4e-6f * (tm + ca[5] + cb[5] + thr));
                const bool kept = !(fminf(ca[6], cb[6]) > 0.f) || !(axis_gap9(d, va, vb) > lim);
                const unsigned bit = kept ? 1u << (sl & 31) : 0u;
                m[0] |= __reduce_or_sync(0xffffffffu, sl < 32 ? bit : 0u);
                m[1] |= __reduce_or_sync(0xffffffffu, sl < 32 ? 0u : bit);
            }
            if (!LEAF && sure) {
                if (lane == 0) entry_hits[w] = 1;
                continue;
            }
        }
        if (!LEAF && lane == 0) entry_hits[w] = 0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (LEAF) {
                if (lane == 0) {
                    mask[2 * (size_t)w + h] = m[h];
                    cnt[2 * (size_t)w + h] = __popc(m[h]);
                }
            } else {
                const bool keep = (m[h] >> lane) & 1u;
                const bool whole = keep && use_bounds &&
                                   !(tm < 0.1f * kFarSizes * fminf(s_c[wi][ta0 + 4 * h][6], s_c[wi][8 + tb0][6]));
                warp_append((64 * w + lane + 32 * h) | (whole ? kWholeTest : 0), keep, list, lc + LC_LIST);
            }
        }
        if (LEAF) break;  // a warp a node pair
    }
}

// The undecided slots of a descent's level: whether a triangle pair is closer
// than its limit, until the node pair is marked.  As k_soup_slots: some ten to
// a few hundred slots, a warp a slot (a thread a slot took 20 to 60 us a
// level); the vertices a component per lane, then the nine edge pairs on lanes
// 0-8 and, if none is below the limit, the six projections on lanes 9-14 and
// the six edge crossings on lanes 16-21 that the FP32 bounds leave.  A marked
// slot's distance is the reference's whole one, on one lane.
__global__ void __launch_bounds__(kBlock) k_np_slots(const int32_t* __restrict__ list,
                                                     const int32_t* __restrict__ n_list,
                                                     const Entry* __restrict__ front, const double* __restrict__ pm,
                                                     const double* __restrict__ tris, const double* __restrict__ eps,
                                                     const float* __restrict__ search, int32_t* entry_hits) {
    __shared__ double s_v[kBlock / 32][6][3];
    const int n = *n_list;
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    double(*v)[3] = s_v[wi];
    for (int k = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5); k < n;
         k += (int)((gridDim.x * (size_t)blockDim.x) >> 5)) {
        const int item = list[k], slot = item & ~kWholeTest;
        if (__any_sync(0xffffffffu, ((volatile int32_t*)entry_hits)[slot >> 6] != 0)) continue;
        const Entry e = front[slot >> 6];
        const int ta = (slot >> 3) & 7, tb = slot & 7;
        const double* M = pm + 32 * (size_t)e.pair;
        if (lane < 18) {  // tri_xform_rigid, a row each
            const int i = lane / 3, c = lane % 3;
            const double* T = M + (i < 3 ? 0 : 16) + 4 * c;
            const double* p = i < 3 ? tris + (size_t)e.na * 72 + ta * 9 + 3 * i : tris + (size_t)e.nb * 72 + tb * 9 + 3 * (i - 3);
            v[i][c] = ((T[0] * p[0] + T[1] * p[1]) + T[2] * p[2]) + T[3] * 1.0;
        }
        __syncwarp();
        const double thr = ((double)search[e.pair] + eps[(size_t)e.na * 8 + ta]) + eps[(size_t)e.nb * 8 + tb];
        auto at = [&](int i) { return mk(v[i][0], v[i][1], v[i][2]); };
        bool hit = false, any;
        if (item & kWholeTest) {
            V3 P, Q;
            if (lane == 0) hit = tri_tri_dist_plain(Tri{at(0), at(1), at(2)}, Tri{at(3), at(4), at(5)}, P, Q) < thr;
            any = __any_sync(0xffffffffu, hit);
            if (any && lane == 0) entry_hits[slot >> 6] = 1;
            __syncwarp();
            continue;
        }
        if (lane < 9) {
            const int ia = lane / 3, ib = lane % 3;
            V3 P, Q;
            hit = edge_closest(at(ia), at(ia == 2 ? 0 : ia + 1), at(3 + ib), at(ib == 2 ? 3 : 4 + ib), P, Q) < thr;
        }
        any = __any_sync(0xffffffffu, hit);
        if (!any && lane >= 9 && lane < 22 && lane != 15) {
            // T: the triangle whose plane is used, the feature is the other's
            const int q = lane < 15 ? lane - 9 : lane - 16;
            const int t0 = q < 3 ? 0 : 3, o0 = 3 - t0, i = q < 3 ? q : q - 3, i1 = i == 2 ? 0 : i + 1;
            const V3 o = at(0);
            F3 r[6];
            float rho = 0.f;
#pragma unroll
            for (int j = 0; j < 6; j++) {
                r[j] = rel3(at(j < 3 ? t0 + j : o0 + j - 3), o);
                rho = fmaxf(rho, maxabs3(r[j]));
            }
            const F3 ri = i == 0 ? r[3] : (i == 1 ? r[4] : r[5]), ri1 = i1 == 0 ? r[3] : (i1 == 1 ? r[4] : r[5]);
            const PlaneBound p = plane_bound(r[0], r[1], r[2], rho);
            const float h = dot3(p.n, ri - p.o);
            const Tri T{at(t0), at(t0 + 1), at(t0 + 2)};
            if (lane < 15) {
                bool out = false;
                if (p.ok) {
                    float bu, bv, bw;
                    plane_bary(p, ri - p.o, bu, bv, bw);
                    out = bu < -p.mb || bv < -p.mb || bw < -p.mb;
                }
                if (!out) {
                    const V3 pt = at(o0 + i);
                    bool in;
                    const V3 on = tri_project_to_plane(T, pt, in);
                    hit = in && norm(on - pt) < thr;
                }
            } else if (!no_crossing(p, ri, ri1, h, dot3(p.n, ri1 - p.o))) {
                double t;
                bool t_inf;
                tri_intersect_segment(T, at(o0 + i), at(o0 + i1), t, t_inf, hit);
                hit = hit && 0.0 < thr;
            }
        }
        any = any || __any_sync(0xffffffffu, hit);
        if (any && lane == 0) entry_hits[slot >> 6] = 1;
        __syncwarp();
    }
}

// The same with the whole FP64 test of every slot (bounds off), a thread a slot.
__global__ void __launch_bounds__(kBlock) k_np_level_tests(const int32_t* __restrict__ list,
                                                           const int32_t* __restrict__ n_list,
                                                           const Entry* __restrict__ front,
                                                           const double* __restrict__ pm,
                                                           const double* __restrict__ tris,
                                                           const double* __restrict__ eps,
                                                           const float* __restrict__ search, int32_t* entry_hits) {
    const int n = *n_list;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int slot = list[k];
        if (((volatile int32_t*)entry_hits)[slot >> 6]) continue;
        const Entry e = front[slot >> 6];
        const int ta = (slot >> 3) & 7, tb = slot & 7;
        const double* M = pm + 32 * (size_t)e.pair;
        const Tri A = tri_xform_rigid(load_tri(tris + (size_t)e.na * 72 + ta * 9), M);
        const Tri B = tri_xform_rigid(load_tri(tris + (size_t)e.nb * 72 + tb * 9), M + 16);
        const double thr = ((double)search[e.pair] + eps[(size_t)e.na * 8 + ta]) + eps[(size_t)e.nb * 8 + tb];
        V3 P, Q;
        if (tri_tri_dist(A, B, P, Q) < thr) entry_hits[slot >> 6] = 1;
    }
}

// Ordered compaction of the surviving slots (slot order = the reference's
// triangle-pair order within each node pair), a thread per mask word.
__global__ void k_np_items(int n_words, const uint32_t* __restrict__ mask, const int32_t* __restrict__ off,
                           int32_t* __restrict__ items) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_words) return;
    int o = off[i];
    for (unsigned m = mask[i]; m; m &= m - 1) items[o++] = 32 * i + __ffs(m) - 1;
}

// One surviving slot a thread: the FP64 triangle distance and the hit test.
// Bound by the FP64 pipe; tri_tri_dist_below evaluates 2 to 3 of the 21
// features (1,024 packed hulls' leaf pairs: 352 us with the pipe 80% busy;
// with all features, 825 us a level).
__global__ void __launch_bounds__(kBlock) k_np(int n_slots, const Entry* __restrict__ front,
                                               const int32_t* __restrict__ pairs, const double* __restrict__ pm,
                                               const int32_t* __restrict__ ntris, const double* __restrict__ tris,
                                               const double* __restrict__ eps, const double* __restrict__ inner_eps,
                                               const double* __restrict__ geo_eps,
                                               const float* __restrict__ search, PrimResult* __restrict__ res,
                                               double* __restrict__ res_eps, int32_t* __restrict__ hit,
                                               int32_t* __restrict__ entry_hits, const int32_t* __restrict__ items,
                                               int use_bounds) {
    // Work item k tests slot items[k]; results are stored per item.
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_slots) return;
    const int i = items[k];
    const Entry e = front[i >> 6];
    const int ta = (i >> 3) & 7, tb = i & 7;
    int h = 0;
    if (ta < ntris[e.na] && tb < ntris[e.nb]) {
        const double* M = pm + 32 * (size_t)e.pair;
        const Tri A = tri_xform_rigid(load_tri(tris + (size_t)e.na * 72 + ta * 9), M);
        const Tri B = tri_xform_rigid(load_tri(tris + (size_t)e.nb * 72 + tb * 9), M + 16);
        V3 P, Q;
        const double ea = eps[(size_t)e.na * 8 + ta], eb = eps[(size_t)e.nb * 8 + tb];
        const double thr = ((double)search[e.pair] + ea) + eb;
        const double d = use_bounds ? tri_tri_dist_below(A, B, thr, P, Q) : tri_tri_dist(A, B, P, Q);
        h = d < thr ? 1 : 0;
        if (h) {
            const int a = pairs[2 * e.pair], b = pairs[2 * e.pair + 1];
            put_result(res[k], d, P, Q, 0.0);
            res_eps[4 * (size_t)k + 0] = geo_eps[a] + ea;
            res_eps[4 * (size_t)k + 1] = geo_eps[b] + eb;
            res_eps[4 * (size_t)k + 2] = inner_eps[(size_t)e.na * 8 + ta];
            res_eps[4 * (size_t)k + 3] = inner_eps[(size_t)e.nb * 8 + tb];
            atomicAdd(&entry_hits[i >> 6], 1);
        }
    }
    hit[k] = h;
}

// Frontier entries of one body pair (pair index 0) from a list of node pairs.
__global__ void k_bucket_entries(int n, const int32_t* __restrict__ node_pairs, Entry* __restrict__ front) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Entry e;
    e.pair = 0;
    e.na = node_pairs[2 * i];
    e.nb = node_pairs[2 * i + 1];
    front[i] = e;
}

// --------------------------------------------------- finals / expansion ----
// A result as a contact record (collision_detection/contact.h).
__device__ __forceinline__ void write_record(const PrimResult& r, const double* re, int a, int b,
                                             const double* __restrict__ geo_eps, double* __restrict__ o) {
    o[0] = r.P[0];
    o[1] = r.P[1];
    o[2] = r.P[2];
    o[3] = r.Q[0];
    o[4] = r.Q[1];
    o[5] = r.Q[2];
    if (re) {
        o[6] = re[0];
        o[7] = re[1];
        o[8] = re[2];
        o[9] = re[3];
    } else {
        o[6] = geo_eps[a];
        o[7] = geo_eps[b];
        o[8] = 0.0;
        o[9] = 0.0;
    }
    o[10] = r.toc;
    o[11] = (double)a;
    o[12] = (double)b;
    o[13] = 0.0;
}

// Append flagged results as contact records.
__global__ void k_emit(int n, const int32_t* __restrict__ flags, const int32_t* __restrict__ off,
                       const int32_t* __restrict__ items, int slot_shift, const Entry* __restrict__ front,
                       const int32_t* __restrict__ tp, const int32_t* __restrict__ pairs,
                       const PrimResult* __restrict__ res, const double* __restrict__ res_eps,
                       const double* __restrict__ geo_eps, double* __restrict__ rec, int32_t* __restrict__ rec_pair,
                       int base) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || !flags[k]) return;
    const int ei = tp ? tp[k / 15] : (items ? items[k] : k) >> slot_shift;
    const Entry e = front[ei];
    write_record(res[k], res_eps ? res_eps + 4 * (size_t)k : nullptr, pairs[2 * e.pair], pairs[2 * e.pair + 1],
                 geo_eps, rec + 14 * (size_t)(base + off[k]));
    rec_pair[base + off[k]] = e.pair;
}

// Expansion rule of full_tree_comparison.h:27-59: leaf-leaf keeps its hits,
// otherwise the shallower inner side (b on ties, the inner one when the other
// is a leaf) is replaced by its children.
// A level's expansion for the descents: children with an inner node to next
// [0 ..), leaf pairs to leaf [leaf0 ..) (with self_leaf also a marked pair of
// two leaves itself), in order; the totals to lc.  prev: the counters of the
// level before, when the host does not know them yet (n and leaf0 are its
// totals, the launch is for a bound).  A thread per node pair.  Up to kExpandOneBlock
// node pairs one block does it all; larger levels take two launches,
// k_expand_sums for the blocks' totals and k_expand_level, whose blocks add up
// the totals before theirs (three launches and a library scan before).
constexpr int kExpandThreads = 256, kExpandOneThreads = 1024, kExpandOneBlock = 2048;
struct Opened {
    Entry e;
    int4 P;           // the opened node (two leaves: y = self_leaf)
    int rule;
    unsigned leaves;  // bit per child: a leaf pair
};
__device__ __forceinline__ bool open_pair(const Entry& e, const int4* __restrict__ nodes, int self_leaf, Opened& o) {
    const int4 A = ld_node(nodes, e.na), B = ld_node(nodes, e.nb);
    o.e = e;
    o.rule = !A.z && !B.z ? 0 : (!A.z ? 2 : (!B.z ? 1 : (A.w < B.w ? 1 : 2)));
    o.P = o.rule == 1 ? A : B;
    o.leaves = 0;
    if (!o.rule) {
        o.P.y = self_leaf;
        o.leaves = 1;
        return self_leaf != 0;
    }
    if (!(o.rule == 1 ? B : A).z) {
#pragma unroll
        for (int ch = 0; ch < 8; ch++)
            if (ch < o.P.y && !ld_node(nodes, o.P.x + ch).z) o.leaves |= 1u << ch;
    }
    return true;
}
// Exclusive prefix sums of (s, c) over the block, and its totals (every thread).
template <int THREADS>
__device__ __forceinline__ int2 block_scan2(int s, int c, int2& total) {
    __shared__ int2 wsum[THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int xs = s, xc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ys = __shfl_up_sync(0xffffffffu, xs, o), yc = __shfl_up_sync(0xffffffffu, xc, o);
        if (lane >= o) {
            xs += ys;
            xc += yc;
        }
    }
    __syncthreads();
    if (lane == 31) wsum[w] = make_int2(xs, xc);
    __syncthreads();
    int2 before = make_int2(xs - s, xc - c);
    total = make_int2(0, 0);
#pragma unroll
    for (int k = 0; k < THREADS / 32; k++) {
        const int2 v = wsum[k];
        if (k < w) {
            before.x += v.x;
            before.y += v.y;
        }
        total.x += v.x;
        total.y += v.y;
    }
    return before;
}
__global__ void __launch_bounds__(kExpandThreads) k_expand_sums(int n, const Entry* __restrict__ front,
                                                                const int32_t* __restrict__ entry_hits,
                                                                const int4* __restrict__ nodes, int self_leaf,
                                                                int2* __restrict__ sums,
                                                                const int32_t* __restrict__ prev) {
    if (prev) n = prev[LC_NEXT];
    const int i = blockIdx.x * kExpandThreads + threadIdx.x;
    Opened o;
    int s = 0, c = 0;
    if (i < n && entry_hits[i] > 0 && open_pair(front[i], nodes, self_leaf, o)) {
        c = __popc(o.leaves);
        s = o.P.y - c;
    }
    int2 total;
    block_scan2<kExpandThreads>(s, c, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_expand_level(int n, const Entry* __restrict__ front,
                                                                 const int32_t* __restrict__ entry_hits,
                                                                 const int4* __restrict__ nodes, int self_leaf,
                                                                 const int2* __restrict__ sums,
                                                                 Entry* __restrict__ next, Entry* __restrict__ leaf,
                                                                 int leaf0, int32_t* __restrict__ lc,
                                                                 const int32_t* __restrict__ prev) {
    if (prev) {
        n = prev[LC_NEXT];
        leaf0 = prev[LC_LEAF];
    }
    int2 base = make_int2(0, leaf0);
    if (sums) {  // the blocks before this one
        int s = 0, c = 0;
        for (int k = threadIdx.x; k < (int)blockIdx.x; k += THREADS) {
            s += sums[k].x;
            c += sums[k].y;
        }
        int2 total;
        block_scan2<THREADS>(s, c, total);
        base.x += total.x;
        base.y += total.y;
    }
    // one block walks the level, else one pass (with n from the device some
    // blocks have nothing)
    for (int i0 = sums ? blockIdx.x * THREADS : 0; i0 < n; i0 += sums ? INT32_MAX / 2 : THREADS) {
        const int i = i0 + threadIdx.x;
        Opened o;
        int s = 0, c = 0;
        if (i < n && entry_hits[i] > 0 && open_pair(front[i], nodes, self_leaf, o)) {
            c = __popc(o.leaves);
            s = o.P.y - c;
        }
        int2 total;
        const int2 at = block_scan2<THREADS>(s, c, total);
        if (s + c > 0) {
            Entry* ps = next + base.x + at.x;
            Entry* pc = leaf + base.y + at.y;
            for (int ch = 0; ch < o.P.y; ch++) {
                Entry x;
                x.pair = o.e.pair;
                x.na = o.rule == 1 ? o.P.x + ch : o.e.na;
                x.nb = o.rule == 2 ? o.P.x + ch : o.e.nb;
                if ((o.leaves >> ch) & 1u)
                    *pc++ = x;
                else
                    *ps++ = x;
            }
        }
        base.x += total.x;
        base.y += total.y;
    }
    if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) {
        lc[LC_NEXT] = base.x;
        lc[LC_LEAF] = base.y;
    }
}

// ---------------------------------------------------------- output sort ----
__global__ void k_iota(int n, int32_t* __restrict__ v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}
// First record of every pair in the sorted pair ids: out[p] for p in [0, n_pairs].
__global__ void k_pair_offsets(int n, int p0, int n_pairs, const int32_t* __restrict__ rec_pair,
                               int32_t* __restrict__ out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > n_pairs) return;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (rec_pair[mid] < p0 + p)
            lo = mid + 1;
        else
            hi = mid;
    }
    out[p] = lo;
}
__global__ void k_gather(int n, const int32_t* __restrict__ idx, const double* __restrict__ in,
                         double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int j = idx[i];
    if (j < 0 || j >= n) return;
    const double* s = in + 14 * (size_t)j;
    double* d = out + 14 * (size_t)i;
#pragma unroll
    for (int k = 0; k < 14; k++) d[k] = s[k];
}

// Future state left on each body: the projection of the last pair containing it.
__global__ void k_last_pair(int n, const int32_t* __restrict__ pairs, int32_t* __restrict__ last) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    atomicMax(&last[pairs[2 * p]], p);
    atomicMax(&last[pairs[2 * p + 1]], p);
}
__global__ void k_write_fut(int n, const int32_t* __restrict__ pairs, const int32_t* __restrict__ last,
                            const double* __restrict__ pfut, double* __restrict__ fut) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int a = pairs[2 * p], b = pairs[2 * p + 1];
    if (last[a] == p)
        for (int k = 0; k < 14; k++) fut[14 * (size_t)a + k] = pfut[28 * (size_t)p + k];
    if (last[b] == p)
        for (int k = 0; k < 14; k++) fut[14 * (size_t)b + k] = pfut[28 * (size_t)p + 14 + k];
}

__global__ void k_fill(int n, int32_t* __restrict__ v, int32_t x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = x;
}

// ------------------------------------------------------------ host side ----
#define LAUNCH(kern, n, ...)                                                \
    do {                                                                    \
        kern<<<nblocks(n), kBlock, 0, ctx->stream>>>(__VA_ARGS__);          \
        ctx->eng.launches++;                                                \
    } while (0)

// Profiling mode: an event pair around a dominant kernel's launch; the
// elapsed times are collected at the next stream synchronisation.
int prof_begin(d2g_ctx* ctx, int kind, long long items, cudaStream_t st = nullptr) {
    Engine& E = ctx->eng;
    if (!E.profiling) return -1;
    cudaEvent_t ev[2];
    for (int i = 0; i < 2; i++) {
        if (!E.event_pool.empty()) {
            ev[i] = E.event_pool.back();
            E.event_pool.pop_back();
        } else if (cudaEventCreate(&ev[i]) != cudaSuccess) {
            return -1;
        }
    }
    cudaEventRecord(ev[0], st ? st : ctx->stream);
    E.pending.push_back(Engine::Pending{kind, ev[0], ev[1], items});
    return (int)E.pending.size() - 1;
}
void prof_end(d2g_ctx* ctx, int idx, cudaStream_t st = nullptr) {
    if (idx >= 0) cudaEventRecord(ctx->eng.pending[idx].e1, st ? st : ctx->stream);
}
// Call only after the stream has been synchronised.
void prof_collect(d2g_ctx* ctx) {
    Engine& E = ctx->eng;
    for (auto& p : E.pending) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, p.e0, p.e1) == cudaSuccess) {
            E.prof_ms[p.kind] += ms;
            E.prof_launches[p.kind] += 1;
            E.prof_items[p.kind] += p.items;
        }
        E.event_pool.push_back(p.e0);
        E.event_pool.push_back(p.e1);
    }
    E.pending.clear();
}

// Exclusive prefix sum of a small int32 array in one 1024-thread block:
// out[0..n] with out[n] = total.  The array is
// staged in shared memory in chunks of kScanChunk (coalesced), each thread
// sums its kScanPer contiguous elements, and a shuffle scan over the thread
// sums gives every thread its offset.
constexpr int kScanThreads = 1024, kScanPer = 8, kScanChunk = kScanThreads * kScanPer;
static_assert(kScanThreads == 32 * 32, "the warp-sum scan assumes 32 warps");
constexpr int kScanOneBlock = 4 * kScanChunk;  // larger arrays go to cub
__global__ void __launch_bounds__(kScanThreads) k_scan1(const int32_t* __restrict__ in, int32_t* __restrict__ out,
                                                        int n) {
    __shared__ int32_t buf[kScanChunk];
    __shared__ int32_t wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += kScanChunk) {
        const int m = min(kScanChunk, n - base);
        for (int i = tid; i < kScanChunk; i += kScanThreads) buf[i] = i < m ? in[base + i] : 0;
        __syncthreads();
        int v[kScanPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kScanPer; k++) {
            v[k] = buf[tid * kScanPer + k];
            sum += v[k];
        }
        int x = sum;  // inclusive warp scan of the thread sums
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            int z = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, z, o);
                if (lane >= o) z += y;
            }
            wsum[lane] = z;  // inclusive over warps
        }
        __syncthreads();
        int run = carry + (w > 0 ? wsum[w - 1] : 0) + (x - sum);
#pragma unroll
        for (int k = 0; k < kScanPer; k++) {
            buf[tid * kScanPer + k] = run;
            run += v[k];
        }
        const int chunk_total = wsum[31];
        __syncthreads();
        for (int i = tid; i < m; i += kScanThreads) out[base + i] = buf[i];
        carry += chunk_total;
        __syncthreads();
    }
    if (tid == 0) out[n] = carry;
}

int scan_on(cudaStream_t st, DBuf<uint8_t>& tmp, const int32_t* in, int32_t* out, int n) {
    if (n <= kScanOneBlock) {
        k_scan1<<<1, kScanThreads, 0, st>>>(in, out, n);
        return D2G_OK;
    }
    D2G_CUDA(cudaMemsetAsync(out, 0, sizeof(int32_t), st));
    size_t bytes = 0;
    D2G_CUDA(cub::DeviceScan::InclusiveSum(nullptr, bytes, in, out + 1, n, st));
    if (int rc = tmp.ensure(bytes + 16)) return rc;
    D2G_CUDA(cub::DeviceScan::InclusiveSum(tmp.p, bytes, in, out + 1, n, st));
    return D2G_OK;
}
int scan(d2g_ctx* ctx, const int32_t* in, int32_t* out, int n) {
    if (n <= kScanOneBlock) ctx->eng.launches++;  // this library's scan kernel (larger ones are cub's)
    return scan_on(ctx->stream, ctx->eng.cub_tmp, in, out, n);
}
// Read k device int32 scalars (after the stream's pending work).
int read_scalars(d2g_ctx* ctx, const int32_t* const* src, int k, int32_t* dst) {
    for (int i = 0; i < k; i++)
        D2G_CUDA(cudaMemcpyAsync(ctx->h_pinned + i, src[i], sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    D2G_CUDA(cudaStreamSynchronize(ctx->stream));
    prof_collect(ctx);
    for (int i = 0; i < k; i++) dst[i] = ctx->h_pinned[i];
    return D2G_OK;
}

#define RC(x)                     \
    do {                          \
        if (int rc_ = (x)) return rc_; \
    } while (0)

// Sort records by pair (stable) into rec_sorted and write offsets [n_pairs+1].
// Pairs [p0, p0 + n_pairs): the records' pair ids lie in that range and the
// offsets are indexed from p0.
int finish_records(d2g_ctx* ctx, int n_pairs, int n_rec, int p0 = 0) {
    Engine& E = ctx->eng;
    RC(E.out_off.ensure(n_pairs + 1));
    RC(E.rec_sorted.ensure(14 * (size_t)n_rec + 14));
    if (n_rec > 0) {
        RC(E.rec_idx.ensure(n_rec));
        RC(E.rec_idx_sorted.ensure(n_rec));
        RC(E.rec_pair_sorted.ensure(n_rec));
        LAUNCH(k_iota, n_rec, n_rec, E.rec_idx.p);
        int bits = 1;
        while ((1LL << bits) < (long long)p0 + n_pairs + 1 && bits < 31) bits++;
        size_t bytes = 0;
        D2G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, E.rec_pair.p, E.rec_pair_sorted.p, E.rec_idx.p,
                                                 E.rec_idx_sorted.p, n_rec, 0, bits, ctx->stream));
        RC(E.cub_tmp.ensure(bytes + 16));
        D2G_CUDA(cub::DeviceRadixSort::SortPairs(E.cub_tmp.p, bytes, E.rec_pair.p, E.rec_pair_sorted.p, E.rec_idx.p,
                                                 E.rec_idx_sorted.p, n_rec, 0, bits, ctx->stream));
        LAUNCH(k_gather, n_rec, n_rec, E.rec_idx_sorted.p, E.rec.p, E.rec_sorted.p);
    }
    LAUNCH(k_pair_offsets, n_pairs + 1, n_rec, p0, n_pairs, E.rec_pair_sorted.p, E.out_off.p);
    return D2G_OK;
}

}  // namespace

// Profiling marks for kernels launched outside this file.
int prof_mark_begin(d2g_ctx* ctx, int kind, long long items) { return prof_begin(ctx, kind, items); }
void prof_mark_end(d2g_ctx* ctx, int idx) { prof_end(ctx, idx); }
void prof_mark_collect(d2g_ctx* ctx) { prof_collect(ctx); }

// Launch with an explicit block size.
#define LAUNCHB(kern, n, block, ...)                                                  \
    do {                                                                              \
        kern<<<nblocks(n, block), block, 0, ctx->stream>>>(__VA_ARGS__);              \
        ctx->eng.launches++;                                                          \
    } while (0)

// Append flagged results (already scanned into `off`) as contact records at `base`.
void emit_records(d2g_ctx* ctx, int n, const int32_t* flags, const int32_t* off, const int32_t* items, int shift,
                  const Entry* front, const int32_t* tp, const int32_t* d_pairs, const PrimResult* res, int base) {
    Engine& E = ctx->eng;
    LAUNCH(k_emit, n, n, flags, off, items, shift, front, tp, d_pairs, res, nullptr, ctx->geo_eps.p,
           E.rec.p, E.rec_pair.p, base);
}

// Grid of k_ee_rest4: it reads its list size from device memory, so the grid
// is fixed (every block resident, grid-stride; the first quads take the
// tests, so a short list occupies the first blocks, one warp per SMSP).
int ee_grid_size(d2g_ctx* ctx, int* grid) {
    Engine& E = ctx->eng;
    if (E.ee_grid == 0) {
        int per_sm = 0;
        D2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ee_rest4, kBlock, 0));
        E.ee_grid = std::max(1, ctx->n_sms * std::max(1, per_sm));
    }
    *grid = E.ee_grid;
    return D2G_OK;
}

// Grid of the kernels that test a level's undecided slots, whose number they
// read from device memory too: a few warps per SM sub-partition.
int slot_grid_size(d2g_ctx* ctx) { return 3 * ctx->n_sms; }

// Bytes a traversal level may use for its buffers: a sixth of the device
// memory (the rest holds the scene, the contact records with their sorted
// copy, and other stages).  d2g_ctx_set_level_budget overrides it.
double level_budget(d2g_ctx* ctx) {
    Engine& E = ctx->eng;
    if (E.level_budget > 0) return (double)E.level_budget;
    if (E.device_bytes == 0) {  // queried once: the driver call is not free
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return 1e30;
        E.device_bytes = total_b;
    }
    return (double)E.device_bytes / 6.0;
}

// The proposal's 20 features of n pair queries over the context's device
// bodies, into E.pp_feat.
int run_ccd_features(d2g_ctx* ctx, const int32_t* d_pairs, const double* d_max_time, int n) {
    Engine& E = ctx->eng;
    RC(E.pp_feat.ensure(20 * (size_t)n + 1));
    if (n > 0)
        LAUNCH(k_ccd_features, n, n, d_pairs, d_max_time, ctx->cur.p, ctx->inv_inertia.p, ctx->bounding_radius.p,
               E.pp_feat.p);
    D2G_CUDA(cudaGetLastError());
    return D2G_OK;
}

// The separation-witness table: allocated on first use and cleared when the
// witnesses written since the last clearing could fill half of it (stale
// entries only cost a failed check; clearing keeps the probes short).
int ensure_witness_table(d2g_ctx* ctx) {
    Engine& E = ctx->eng;
    const size_t cap = (size_t)1 << E.wt_log2cap;
    if (!E.wt_table.p || E.wt_inserts > (long long)(cap / 2)) {
        RC(E.wt_table.ensure(cap));
        D2G_CUDA(cudaMemsetAsync(E.wt_table.p, 0, sizeof(WitnessSlot) * cap, ctx->stream));
        E.wt_inserts = 0;
    }
    return D2G_OK;
}

// Body indices of a device pair list inside [0, n_bodies): one flag, one read.
__global__ void k_check_pairs(int n, const int32_t* __restrict__ pairs, int n_bodies, int32_t* __restrict__ bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * n) return;
    const int v = pairs[i];
    if (v < 0 || v >= n_bodies) atomicMin(bad, i >> 1);
}

int check_device_pairs(d2g_ctx* ctx, const int32_t* d_pairs, int n) {
    Engine& E = ctx->eng;
    if (n <= 0) return D2G_OK;
    RC(E.scratch_i32.ensure(1));
    ctx->h_pinned[0] = INT32_MAX;
    D2G_CUDA(cudaMemcpyAsync(E.scratch_i32.p, ctx->h_pinned, sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
    LAUNCH(k_check_pairs, 2LL * n, n, d_pairs, ctx->n_bodies, E.scratch_i32.p);
    int32_t bad = 0;
    const int32_t* src = E.scratch_i32.p;
    RC(read_scalars(ctx, &src, 1, &bad));
    if (bad != INT32_MAX) {
        set_error("device pair " + std::to_string(bad) + " names a body outside [0, " +
                  std::to_string(ctx->n_bodies) + ")");
        return D2G_ERR_INVALID;
    }
    return D2G_OK;
}

// The CCD counters live on the device across calls (one read when asked).
int ensure_ccd_stats(d2g_ctx* ctx) {
    Engine& E = ctx->eng;
    if (!E.ccd_stats.p) {
        RC(E.ccd_stats.ensure(kCcdStats + kCutCounters));
        D2G_CUDA(cudaMemsetAsync(E.ccd_stats.p, 0, sizeof(unsigned long long) * (kCcdStats + kCutCounters),
                                 ctx->stream));
    }
    return D2G_OK;
}

int read_ccd_stats(d2g_ctx* ctx, int64_t* out, int n, bool reset) {
    Engine& E = ctx->eng;
    RC(ensure_ccd_stats(ctx));
    unsigned long long h[kCcdStats + kCutCounters];
    D2G_CUDA(cudaMemcpyAsync(h, E.ccd_stats.p, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    if (reset) D2G_CUDA(cudaMemsetAsync(E.ccd_stats.p, 0, sizeof(h), ctx->stream));
    D2G_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int i = kCcdStats; i < kCcdStats + kCutCounters; i++) {  // cut before their first iterate
        h[0] += h[i];
        h[1] += kEeNewtonIters * h[i];
    }
    for (int i = 0; i < n && i < kCcdStats; i++) out[i] = (int64_t)h[i];
    return D2G_OK;
}

// A descent's outcome: whether it passed the byte budget, the node pairs
// and swept (or valid) triangle pairs it saw, its levels and the leaf pairs it
// left in E.conn, in level order.
struct Traversal {
    bool abandon = false;
    double peak = 0.0;
    int64_t nodes = 0, tri = 0, levels = 0;
    int n_leaf = 0, n_root = 0;  // n_root: root pairs of two leaves (CCD: with candidate slots)
};

// Descends from the n node pairs in E.soup: per level `decide` marks the node
// pairs with a hit in E.entry_hits, and their children go to the next level
// or, two leaves, onto E.conn (with self_leaf also marked root pairs that are
// two leaves).
//
// Reading a level's counts drains the GPU for the launches of the next (~30 us
// a level of an icosphere descent's 8), so up to kAhead levels are launched per
// read: for the first the host knows the node pairs, the others take the count
// from the level before on the device and are launched for a bound, eight
// children a node pair.  Levels run ahead only while the bound is below
// kAheadPairs, whose buffers (~2.4 KB a node pair) fit the budget, and while
// the meshes' depths allow another level; levels above are long enough to
// hide the read.  decide gets the level's first node pair and their number (or
// a bound), its counters and, running ahead, where its count is; a single body
// pair's level that a slot list cannot number, or that passes the budget, is
// decided in ranges (level_range).
constexpr int kAhead = 4, kAheadPairs = 1 << 16;
template <class F>
int descend(d2g_ctx* ctx, int n, bool self_leaf, double budget, bool may_abandon, Traversal& T, F decide) {
    Engine& E = ctx->eng;
    cudaStream_t s = ctx->stream;
    RC(E.lc.ensure(kAhead * LC_SIZE));
    int new_leaf = 0;
    const int max_levels = 2 * ctx->max_depth;  // a level opens one side, and stops at two leaves
    while (n > 0) {
        // past the budget (768 bytes a node pair: its slot list and its
        // children; 18 a leaf pair so far), or past what a slot list numbers
        const double need = 64.0 * 8.0 * 1.5 * n + 1.5 * sizeof(Entry) * T.n_leaf;
        const bool wide = 8LL * n + T.n_leaf > (long long)INT32_MAX;  // counts are 32-bit
        if ((need > budget || n > kMaxListPairs || wide) && may_abandon) {
            T.abandon = true;
            return D2G_OK;
        }
        if (wide) {
            set_error("a traversal level of one body pair with " + std::to_string(n) +
                      " node pairs exceeds the 32-bit node pair count");
            return D2G_ERR_INVALID;
        }
        // (profiling counts slots, witnesses keep a table a level)
        const int most = E.profiling || E.witnesses ? 1 : std::min<int64_t>(kAhead, max_levels - T.levels);
        int bound[kAhead] = {n}, K = 1;
        for (; K < most; K++) {
            const long long b = 8LL * bound[K - 1];
            if (b > kAheadPairs || 2400.0 * 1.5 * (double)b > budget) break;
            bound[K] = (int)b;
        }
        const size_t top = (size_t)bound[K - 1];
        const int range = K > 1 ? bound[K - 1] : level_range(n, budget);
        size_t leaves = (size_t)T.n_leaf + 1;
        for (int k = 0; k < K; k++) leaves += 8 * (size_t)bound[k];  // a node has at most 8 children
        RC(E.entry_hits.ensure(top + 1));
        RC(E.ccd_list.ensure(64 * (size_t)range));
        RC(E.soup_next.ensure(8 * top + 1));
        RC(E.soup.ensure_keep(K > 1 ? 8 * top + 1 : (size_t)n + 1, (size_t)n, s));
        RC(E.conn.ensure_keep(leaves, (size_t)T.n_leaf, s));
        D2G_CUDA(cudaMemsetAsync(E.lc.p, 0, sizeof(int32_t) * LC_SIZE * K, s));
        for (int k = 0; k < K; k++) {
            int32_t* lc = E.lc.p + k * LC_SIZE;
            const int32_t* prev = k ? lc - LC_SIZE : nullptr;
            const int m = bound[k];
            for (int r0 = 0; r0 < m; r0 += range) {
                if (r0 > 0) D2G_CUDA(cudaMemsetAsync(lc + LC_LIST, 0, sizeof(int32_t), s));
                RC(decide(r0, std::min(range, m - r0), lc, k ? prev + LC_NEXT : nullptr));
            }
            const bool one = m <= kExpandOneBlock;
            const int blocks = one ? 1 : nblocks(m, kExpandThreads);
            if (!one) {
                RC(E.sums.ensure(2 * (size_t)blocks));
                k_expand_sums<<<blocks, kExpandThreads, 0, s>>>(m, E.soup.p, E.entry_hits.p, ctx->nodes.p,
                                                                self_leaf ? 1 : 0, (int2*)E.sums.p, prev);
                E.launches++;
            }
            if (one)
                k_expand_level<kExpandOneThreads><<<1, kExpandOneThreads, 0, s>>>(
                    m, E.soup.p, E.entry_hits.p, ctx->nodes.p, self_leaf ? 1 : 0, nullptr, E.soup_next.p, E.conn.p,
                    T.n_leaf, lc, prev);
            else
                k_expand_level<kExpandThreads><<<blocks, kExpandThreads, 0, s>>>(
                    m, E.soup.p, E.entry_hits.p, ctx->nodes.p, self_leaf ? 1 : 0, (const int2*)E.sums.p,
                    E.soup_next.p, E.conn.p, T.n_leaf, lc, prev);
            E.launches++;
            std::swap(E.soup, E.soup_next);
        }
        D2G_CUDA(cudaMemcpyAsync(ctx->h_pinned, E.lc.p, sizeof(int32_t) * LC_SIZE * K, cudaMemcpyDeviceToHost, s));
        D2G_CUDA(cudaStreamSynchronize(s));
        prof_collect(ctx);
        for (int k = 0; k < K && n > 0; k++) {
            const int32_t* lc = ctx->h_pinned + k * LC_SIZE;
            T.peak = std::max(T.peak, (64.0 * 8.0 * 1.5 * n + 1.5 * sizeof(Entry) * T.n_leaf) / budget);
            if (T.levels == 0) T.n_root = lc[LC_ROOT];
            T.levels++;
            T.nodes += n;
            n = lc[LC_NEXT];
            new_leaf = lc[LC_LEAF] - T.n_leaf;
            T.n_leaf = lc[LC_LEAF];
            for (int q = 0; q < LC_TRI_N; q++) T.tri += (uint32_t)lc[LC_TRI + q];
        }
    }
    D2G_CUDA(cudaMemsetAsync(E.lc.p + LC_TRI, 0, sizeof(int32_t) * LC_TRI_N, s));
    // the last level's leaf pairs are a level of the reference's (root pairs of
    // two leaves belong to the first)
    if (new_leaf > (self_leaf && T.levels == 1 ? T.n_root : 0)) T.levels++;
    return D2G_OK;
}
// Blocks for a level's kernels, a warp a node pair: running ahead, eight an SM,
// about what is resident at once (the kernels stride).
int level_blocks(d2g_ctx* ctx, int n, bool ahead) {
    return ahead ? std::min(nblocks(32LL * n), 8 * ctx->n_sms) : nblocks(32LL * n);
}

// The FP64 tests of the descent's leaf pairs (E.conn, in level order), and of
// the chunk's root pairs that are two leaves (soup stage: the best of a
// triangle pair's 15 tests); their contacts are appended to E.rec.  Large lists
// run in ranges that keep the test buffers within the budget; `full` is called
// between ranges with the records so far, and may take them.
template <class F>
int ccd_leaf_tests(d2g_ctx* ctx, const int32_t* d_pairs, const uint8_t* skip, int p0, int p1, Traversal& T,
                   double budget, int& n_rec, long long* n_pp, bool* abandon, F full) {
    Engine& E = ctx->eng;
    cudaStream_t s = ctx->stream;
    int ee_grid = 0;
    RC(ee_grid_size(ctx, &ee_grid));
    // ~1900 bytes of test buffers per triangle pair (x1.5 growth slack), at most 64 in a leaf pair
    const int range = (int)std::min(1.0e6, std::max(256.0, budget / (1.5 * 1900.0 * 64.0)));
    for (int c0 = T.n_root > 0 ? -1 : 0; c0 < T.n_leaf; c0 = c0 < 0 ? 0 : c0 + range) {
        // c0 = -1: the roots; else the leaf pairs [c0, c0 + n_conn)
        const int n_soup = c0 < 0 ? p1 - p0 : 0, n_conn = c0 < 0 ? 0 : std::min(range, T.n_leaf - c0);
        const Entry* soup = E.roots.p + p0;
        const Entry* conn = E.conn.p + (c0 < 0 ? 0 : c0);
        const int n_slots = 64 * n_soup;
        int K = 0, P = 0;  // soup triangle pairs, leaf-pair triangle pairs
        if (n_soup > 0) {
            if (64LL * n_soup > (long long)INT32_MAX / 2 && p1 - p0 > 1) {
                *abandon = true;
                return D2G_OK;
            }
            RC(E.flags.ensure(n_slots + 1));
            RC(E.flag_off.ensure(n_slots + 1));
            LAUNCH(k_soup_filter, 32LL * n_soup, n_soup, soup, d_pairs, E.pm.p, E.pm32c.p, ctx->ntris.p, ctx->tris.p,
                   ctx->tri32.p, ctx->geo_eps.p, ctx->nodes.p, skip, E.flags.p);
            RC(scan(ctx, E.flags.p, E.flag_off.p, n_slots));
            const int32_t* src = E.flag_off.p + n_slots;
            RC(read_scalars(ctx, &src, 1, &K));
        } else {
            RC(E.nn_cnt.ensure(n_conn + 1));
            RC(E.nn_off.ensure(n_conn + 1));
            LAUNCH(k_conn_nn, n_conn, n_conn, conn, ctx->ntris.p, E.nn_cnt.p);
            RC(scan(ctx, E.nn_cnt.p, E.nn_off.p, n_conn));
            const int32_t* src = E.nn_off.p + n_conn;
            RC(read_scalars(ctx, &src, 1, &P));
            RC(E.tp.ensure((size_t)P + 1));
            LAUNCH(k_tp_fill, 32LL * n_conn, n_conn, E.nn_off.p, E.tp.p);
            *n_pp += P;
        }
        if (15LL * K + 15LL * P > (long long)INT32_MAX || 1.5 * 1900.0 * (double)K > budget) {
            if (p1 - p0 > 1) {  // test indices are 32-bit; the budget
                *abandon = true;
                return D2G_OK;
            }
            if (15LL * K + 15LL * P > (long long)INT32_MAX) {
                set_error("CCD call with " + std::to_string(K) + " + " + std::to_string(P) +
                          " triangle pairs in one body pair exceeds the 32-bit test index range");
                return D2G_ERR_INVALID;
            }
        }
        T.peak = std::max(T.peak, 1.5 * 1900.0 * K / budget);
        if (K + P == 0) continue;
        RC(E.items.ensure(K + 1));
        RC(E.sub.ensure(15 * (size_t)K + 1));
        RC(E.res.ensure(K + 1));
        RC(E.hit.ensure(K + 1));
        RC(E.cres.ensure(15 * (size_t)P + 1));
        RC(E.chit.ensure(15 * (size_t)P + 1));
        RC(E.cflag_off.ensure(15 * (size_t)P + 1));
        RC(E.tp.ensure((size_t)P + 1));
        if (n_soup > 0) LAUNCH(k_compact, n_slots, n_slots, E.flags.p, E.flag_off.p, E.items.p);
        const int n_pt = 6 * K + 6 * P, n_ee = 9 * K + 9 * P;
        // FP32 bounds drop the tests that cannot hit; the FP64 kernels run on
        // the survivors, which the bound kernels append to their lists
        RC(E.ccd_cnt.ensure(3));
        RC(E.ccd_list.ensure((size_t)n_pt + n_ee + 2));
        int32_t* cnt_pt = E.ccd_cnt.p;
        int32_t* cnt_ee = E.ccd_cnt.p + 1;
        int32_t* cnt_rest = E.ccd_cnt.p + 2;  // edge-edge tests continued by k_ee_rest4
        int32_t* list_pt = E.ccd_list.p;
        int32_t* list_ee = E.ccd_list.p + n_pt;
        D2G_CUDA(cudaMemsetAsync(E.ccd_cnt.p, 0, 3 * sizeof(int32_t), s));
        RC(E.ee_rec.ensure((size_t)kEeRec * n_ee));
        RC(E.ee_work.ensure(n_ee));
        // The point-triangle and edge-edge chains touch disjoint outputs: the
        // edge-edge chain runs on the second stream beside the other.
        cudaStream_t s_ee = ctx->stream2;
        D2G_CUDA(cudaEventRecord(ctx->ev_fork, s));
        D2G_CUDA(cudaStreamWaitEvent(s_ee, ctx->ev_fork, 0));
        k_ccd_mask_ee<<<nblocks(n_ee), kBlock, 0, s_ee>>>(K, n_ee, E.items.p, soup, conn, E.nn_off.p, E.tp.p,
                                                          E.pm32c.p, ctx->ntris.p, ctx->tri32.p, E.search.p, E.sub.p,
                                                          E.cres.p, E.chit.p, list_ee, cnt_ee, E.fp32_bounds ? 1 : 0,
                                                          E.certificates ? 1 : 0, E.ccd_stats.p + kCcdStats);
        const int pfe = prof_begin(ctx, PROF_CONN, n_ee, s_ee);
        EeArgs ea;
        ea.n_tp = K;
        ea.items = E.items.p;
        ea.soup = soup;
        ea.conn = conn;
        ea.nn_off = E.nn_off.p;
        ea.tp = E.tp.p;
        ea.ntris = ctx->ntris.p;
        ea.search = E.search.p;
        ea.sub = E.sub.p;
        ea.cres = E.cres.p;
        ea.chit = E.chit.p;
        ea.pm = E.pm.p;
        ea.tris = ctx->tris.p;
        ea.rec = E.ee_rec.p;
        ea.work = E.ee_work.p;
        ea.count = cnt_rest;
        ea.first_iters = E.tune[D2G_TUNE_EE_FIRST_ITERS];
        ea.bounds = E.fp32_bounds ? 1 : 0;
        ea.certificates = E.certificates ? 1 : 0;
        ea.ca_stats = E.ccd_stats.p;
        k_ee_first<<<nblocks(n_ee, kPrimBlock), kPrimBlock, 0, s_ee>>>(n_ee, list_ee, cnt_ee, E.pm.p, ctx->tris.p,
                                                                      ea);
        k_ee_rest4<<<ee_grid, kBlock, 0, s_ee>>>(ea);
        if (n_ee > kRestWide) {  // (the list is read on the device; a shorter one cannot be that long)
            k_ee_rest1<<<2 * ee_grid, kPrimBlock, 0, s_ee>>>(ea);
            ctx->eng.launches++;
        }
        ctx->eng.launches += 3;
        prof_end(ctx, pfe, s_ee);
        LAUNCH(k_ccd_mask_pt, n_pt, K, n_pt, E.items.p, soup, conn, E.nn_off.p, E.tp.p, E.pm32c.p, ctx->ntris.p,
               ctx->tri32.p, E.search.p, E.sub.p, E.cres.p, E.chit.p, list_pt, cnt_pt, E.fp32_bounds ? 1 : 0);
        const int pfp = prof_begin(ctx, PROF_SOUP_CCD, n_pt);
        LAUNCHB(k_prim_pt, n_pt, kPrimBlock, K, n_pt, E.items.p, soup, conn, E.nn_off.p, E.tp.p, E.pm.p, ctx->ntris.p,
                ctx->tris.p, E.search.p, E.sub.p, E.cres.p, E.chit.p, list_pt, cnt_pt);
        prof_end(ctx, pfp);
        D2G_CUDA(cudaEventRecord(ctx->ev_join, s_ee));
        D2G_CUDA(cudaStreamWaitEvent(s, ctx->ev_join, 0));
        // contacts, in order
        int32_t fin = 0;
        const int32_t* src;
        if (n_soup > 0) {
            LAUNCH(k_soup_fold, K, K, E.items.p, soup, E.sub.p, E.search.p, E.res.p, E.hit.p);
            RC(scan(ctx, E.hit.p, E.flag_off.p, K));
            src = E.flag_off.p + K;
        } else {
            RC(scan(ctx, E.chit.p, E.cflag_off.p, 15 * P));
            src = E.cflag_off.p + 15 * P;
        }
        RC(read_scalars(ctx, &src, 1, &fin));
        RC(E.rec.ensure_keep(14 * (size_t)(n_rec + fin + 1), 14 * (size_t)n_rec, s));
        RC(E.rec_pair.ensure_keep((size_t)(n_rec + fin + 1), (size_t)n_rec, s));
        if (fin > 0 && n_soup > 0)
            emit_records(ctx, K, E.hit.p, E.flag_off.p, E.items.p, 6, soup, nullptr, d_pairs, E.res.p, n_rec);
        else if (fin > 0)
            emit_records(ctx, 15 * P, E.chit.p, E.cflag_off.p, nullptr, 0, conn, E.tp.p, d_pairs, E.cres.p, n_rec);
        n_rec += fin;
        RC(full());
    }
    return D2G_OK;
}

int run_ccd(d2g_ctx* ctx, const int32_t* d_pairs, const double* d_max_time, int n_pairs, int* n_out,
            int64_t* counters, const CcdSink* sink) {
    Engine& E = ctx->eng;
    cudaStream_t s = ctx->stream;
    int64_t c_node = 0, c_tri = 0, c_leaf = 0, c_levels = 0;
    RC(ensure_ccd_stats(ctx));
    if (E.witnesses) RC(ensure_witness_table(ctx));
    RC(E.pm.ensure((size_t)PM_SIZE * n_pairs + 1));
    RC(E.pfut.ensure(28 * (size_t)n_pairs + 1));
    RC(E.search.ensure(n_pairs + 1));
    RC(E.soup.ensure(n_pairs + 1));
    const int test_grid = slot_grid_size(ctx);
    int n_rec = 0;
    long long n_streamed = 0;  // records handed to the sink
    if (n_pairs > 0)
        LAUNCH(k_ccd_prep, 4LL * n_pairs, n_pairs, d_pairs, d_max_time, ctx->cur.p, ctx->inv_inertia.p, ctx->mesh.p,
               ctx->mesh_node_off.p, ctx->geo_eps.p, E.pm.p, E.pfut.p, E.search.p, E.soup.p);
    RC(E.pm32c.ensure((size_t)kPose32 * n_pairs + 1));
    if (n_pairs > 0) LAUNCH(k_ccd_pm32, (long long)kPose32 * n_pairs, n_pairs, E.pm.p, E.pm32c.p);  // FP32 poses, once per call
    // The learned proposal: the network predicts which queries have no
    // contact; the root certificate proves it for those it can, and the
    // proven ones are skipped (their outputs are empty either way).
    const uint8_t* skip = nullptr;
    if (E.proposal && n_pairs > 0) {
        RC(E.pp_feat.ensure(20 * (size_t)n_pairs));
        RC(E.pp_skip.ensure(n_pairs + 1));
        LAUNCH(k_ccd_features, n_pairs, n_pairs, d_pairs, d_max_time, ctx->cur.p, ctx->inv_inertia.p,
               ctx->bounding_radius.p, E.pp_feat.p);
        const float* pred = nullptr;
        RC(mlp_forward_device(E.proposal, E.pp_feat.p, n_pairs, &pred));
        LAUNCH(k_root_certify, 32LL * n_pairs, n_pairs, d_pairs, E.pm.p, E.pm32c.p, ctx->tri32.p, ctx->mesh.p,
               ctx->mesh_node_off.p,
               ctx->ntris.p, ctx->tris.p, ctx->geo_eps.p, E.search.p, pred, E.proposal_logit, E.pp_skip.p,
               E.ccd_stats.p);
        LAUNCH(k_add_u64, 1, E.ccd_stats.p + 5, (unsigned long long)n_pairs);
        skip = E.pp_skip.p;
    }
    // Pair chunks: the traversal of a range of body pairs runs to the end
    // before the next range starts.  A level whose buffers would pass the
    // budget abandons its chunk (its records are dropped) and the chunk is
    // halved.  A pair's records come from one chunk and are sorted by pair at
    // the end, so the results do not depend on the chunking.
    RC(E.roots.ensure(n_pairs + 1));
    if (n_pairs > 0)
        D2G_CUDA(cudaMemcpyAsync(E.roots.p, E.soup.p, sizeof(Entry) * n_pairs, cudaMemcpyDeviceToDevice, s));
    const double budget = level_budget(ctx);
    // start from the chunk size that fitted last time (abandoning a chunk
    // wastes its finished levels), growing it when the last call used under
    // a third of the budget
    int chunk = E.ccd_chunk > 0 ? std::min(n_pairs, E.ccd_chunk) : n_pairs;
    double peak = 0.0;  // largest level need / budget among finished chunks
    for (int p0 = 0; p0 < n_pairs;) {
        const int p1 = std::min(n_pairs, p0 + chunk);
        const int rec_start = n_rec;
        Traversal T;
        RC(E.soup.ensure((size_t)(p1 - p0) + 1));  // the frontiers swap every level: this one may be the smaller
        D2G_CUDA(cudaMemcpyAsync(E.soup.p, E.roots.p + p0, sizeof(Entry) * (p1 - p0), cudaMemcpyDeviceToDevice, s));
        RC(descend(ctx, p1 - p0, false, budget, p1 - p0 > 1, T, [&](int r0, int n_soup, int32_t* lc,
                                                                    const int32_t* n_dev) -> int {
            const Entry* soup = E.soup.p + r0;
            int32_t* hits = E.entry_hits.p + r0;
            const int pff = prof_begin(ctx, PROF_SOUP_FILTER, 64LL * n_soup);
            const uint8_t* eskip = nullptr;
            if (E.witnesses) {
                RC(E.wt_flag.ensure(n_soup + 1));
                LAUNCH(k_witness_check, 32LL * n_soup, n_soup, soup, d_pairs, E.pm.p, E.pm32c.p, ctx->tri32.p,
                       ctx->mesh.p, ctx->mesh_node_off.p, ctx->ntris.p, ctx->tris.p, ctx->geo_eps.p, E.search.p,
                       E.wt_table.p, E.wt_log2cap, E.wt_flag.p, E.ccd_stats.p);
                eskip = E.wt_flag.p;
            }
            k_ccd_level<<<level_blocks(ctx, n_soup, n_dev != nullptr), kBlock, 0, s>>>(
                n_soup, soup, d_pairs, E.pm.p, E.pm32c.p, ctx->ntris.p, ctx->tris.p, ctx->tri32.p, ctx->geo_eps.p,
                E.search.p, ctx->nodes.p, skip, eskip, E.fp32_bounds ? 1 : 0, E.certificates ? 1 : 0, hits,
                E.ccd_list.p, lc, n_dev);
            E.launches++;
            prof_end(ctx, pff);
            if (E.fp32_bounds)
                k_soup_slots<<<test_grid, kBlock, 0, s>>>(E.ccd_list.p, lc + LC_LIST, soup, E.pm.p, E.pm32c.p,
                                                          ctx->tris.p, ctx->tri32.p, E.search.p, hits,
                                                          E.certificates ? 1 : 0);
            else
                k_soup_tests<<<4 * test_grid, kPrimBlock, 0, s>>>(E.ccd_list.p, lc + LC_LIST, soup, E.pm.p,
                                                                  ctx->tris.p, E.search.p, hits,
                                                                  E.certificates ? 1 : 0);
            E.launches++;
            if (E.witnesses) {
                LAUNCH(k_witness_make, 32LL * n_soup, n_soup, soup, hits, E.wt_flag.p, skip, d_pairs,
                       E.pm.p, E.pm32c.p, ctx->tri32.p, ctx->mesh.p, ctx->mesh_node_off.p, ctx->ntris.p, ctx->tris.p,
                       ctx->geo_eps.p, E.search.p, E.wt_table.p, E.wt_log2cap, E.ccd_stats.p);
                E.wt_inserts += n_soup;
            }
            return D2G_OK;
        }));
        bool abandon = T.abandon;
        long long n_pp = 0;  // leaf pairs' triangle pairs
        bool first = true;
        // the records so far, sorted by pair, go to the consumer and are dropped
        auto hand_over = [&]() -> int {
            RC(finish_records(ctx, p1 - p0, n_rec, p0));
            RC(sink->consume(ctx, sink->user, p0, p1, first));
            first = false;
            n_streamed += n_rec;
            n_rec = 0;
            return D2G_OK;
        };
        // ~240 bytes a record with its sorted copy (x1.5 growth slack): a
        // streamed chunk keeps about half the budget of them
        auto full = [&]() -> int { return sink && 360.0 * n_rec > 0.5 * budget ? hand_over() : D2G_OK; };
        if (!abandon)
            RC(ccd_leaf_tests(ctx, d_pairs, skip, p0, p1, T, budget, n_rec, &n_pp, &abandon, full));
        if (abandon) {
            n_rec = rec_start;
            chunk = std::max(1, (p1 - p0) / 2);
            continue;
        }
        c_node += T.nodes + T.n_leaf;
        c_tri += T.tri + 15 * n_pp;
        c_leaf += T.n_leaf;
        c_levels += T.levels;
        peak = std::max(peak, T.peak);
        if (sink) RC(hand_over());
        p0 = p1;
    }
    if (n_pairs > 0) E.ccd_chunk = chunk >= n_pairs ? 0 : (peak < 1.0 / 3.0 ? 2 * chunk : chunk);
    if (!sink) RC(finish_records(ctx, n_pairs, n_rec));
    if (n_pairs > 0) {
        RC(E.last_pair.ensure(ctx->n_bodies + 1));
        LAUNCH(k_fill, ctx->n_bodies, ctx->n_bodies, E.last_pair.p, -1);
        LAUNCH(k_last_pair, n_pairs, n_pairs, d_pairs, E.last_pair.p);
        LAUNCH(k_write_fut, n_pairs, n_pairs, d_pairs, E.last_pair.p, E.pfut.p, ctx->fut.p);
    }
    D2G_CUDA(cudaGetLastError());
    *n_out = sink ? (int)n_streamed : n_rec;
    if (counters) {
        counters[0] = c_node;
        counters[1] = c_tri;
        counters[2] = c_leaf;
        counters[3] = c_levels;
    }
    return D2G_OK;
}

// The surviving slots of n node pairs at `front` (k_np_filter), tested; the
// item list, hit flags and results stay in E.items, E.hit, E.res and res_eps
// (E.pfut).  One read, of the survivors' count.
int np_slot_tests(d2g_ctx* ctx, const int32_t* d_pairs, const Entry* front, int n, int* n_items_out) {
    Engine& E = ctx->eng;
    DBuf<double>& res_eps = E.pfut;  // per-slot eps record buffer
    const int n_slots = 64 * n, n_words = 2 * n;
    RC(E.np_mask.ensure(n_words + 1));
    RC(E.np_cnt.ensure(n_words + 1));
    RC(E.np_off.ensure(n_words + 1));
    RC(E.lc.ensure(kAhead * LC_SIZE));
    LAUNCH(k_np_filter<true>, 32LL * n, n, front, E.pm32.p, ctx->ntris.p, ctx->tri_sph.p, ctx->tri32.p, ctx->eps_up.p,
           E.search.p, ctx->nodes.p, E.fp32_bounds ? 1 : 0, E.np_mask.p, E.np_cnt.p, (int32_t*)nullptr, (int32_t*)nullptr, E.lc.p,
           (const int32_t*)nullptr);
    RC(scan(ctx, E.np_cnt.p, E.np_off.p, n_words));
    int32_t n_items = 0;
    const int32_t* src = E.np_off.p + n_words;
    RC(read_scalars(ctx, &src, 1, &n_items));
    *n_items_out = n_items;
    if (n_items == 0) return D2G_OK;
    RC(E.items.ensure(n_items + 1));
    RC(E.res.ensure(n_items));
    RC(res_eps.ensure(4 * (size_t)n_items));
    RC(E.hit.ensure(n_items));
    LAUNCH(k_np_items, n_words, n_words, E.np_mask.p, E.np_off.p, E.items.p);
    const int pf = prof_begin(ctx, PROF_NP, n_slots);
    LAUNCH(k_np, n_items, n_items, front, d_pairs, E.pm.p, ctx->ntris.p, ctx->tris.p, ctx->eps.p, ctx->inner_eps.p,
           ctx->geo_eps.p, E.search.p, E.res.p, res_eps.p, E.hit.p, E.entry_hits.p, E.items.p, E.fp32_bounds ? 1 : 0);
    prof_end(ctx, pf);
    return D2G_OK;
}

int run_narrowphase(d2g_ctx* ctx, const int32_t* d_pairs, int n_pairs, int* n_out, int64_t* counters) {
    Engine& E = ctx->eng;
    cudaStream_t s = ctx->stream;
    int64_t c_node = 0, c_tri = 0, c_levels = 0;
    RC(E.pm.ensure(32 * (size_t)n_pairs + 1));
    RC(E.search.ensure(n_pairs + 1));
    RC(E.roots.ensure(n_pairs + 1));
    RC(E.pm32.ensure(kNpPose32 * (size_t)n_pairs + 1));
    if (n_pairs > 0)
        LAUNCH(k_np_prep, n_pairs, n_pairs, d_pairs, ctx->fut.p, ctx->mesh.p, ctx->mesh_node_off.p, ctx->geo_eps.p,
               E.pm.p, E.search.p, E.roots.p, E.pm32.p, nullptr);
    const int test_grid = slot_grid_size(ctx);
    int n_rec = 0;
    // pair chunks, as in run_ccd
    const double budget = level_budget(ctx);
    // a leaf pair's slots take ~110 bytes each (x1.5 growth slack)
    const int range = (int)std::min(8.0e6, std::max(1024.0, budget / (1.5 * 110.0 * 64.0)));
    int chunk = E.np_chunk > 0 ? std::min(n_pairs, E.np_chunk) : n_pairs;
    double peak = 0.0;
    for (int p0 = 0; p0 < n_pairs;) {
        const int p1 = std::min(n_pairs, p0 + chunk);
        Traversal T;
        RC(E.soup.ensure((size_t)(p1 - p0) + 1));
        D2G_CUDA(cudaMemcpyAsync(E.soup.p, E.roots.p + p0, sizeof(Entry) * (p1 - p0), cudaMemcpyDeviceToDevice, s));
        RC(descend(ctx, p1 - p0, true, budget, p1 - p0 > 1, T, [&](int r0, int n, int32_t* lc,
                                                                   const int32_t* n_dev) -> int {
            const Entry* front = E.soup.p + r0;
            int32_t* hits = E.entry_hits.p + r0;
            k_np_filter<false><<<level_blocks(ctx, n, n_dev != nullptr), kBlock, 0, s>>>(
                n, front, E.pm32.p, ctx->ntris.p, ctx->tri_sph.p, ctx->tri32.p, ctx->eps_up.p, E.search.p,
                ctx->nodes.p, E.fp32_bounds ? 1 : 0, nullptr, nullptr, hits, E.ccd_list.p, lc, n_dev);
            E.launches++;
            if (E.fp32_bounds)
                k_np_slots<<<test_grid, kBlock, 0, s>>>(E.ccd_list.p, lc + LC_LIST, front, E.pm.p, ctx->tris.p,
                                                        ctx->eps.p, E.search.p, hits);
            else
                k_np_level_tests<<<4 * test_grid, kBlock, 0, s>>>(E.ccd_list.p, lc + LC_LIST, front, E.pm.p,
                                                                  ctx->tris.p, ctx->eps.p, E.search.p,
                                                                  hits);
            E.launches++;
            return D2G_OK;
        }));
        if (T.abandon) {
            chunk = std::max(1, (p1 - p0) / 2);
            continue;
        }
        // contacts of the leaf pairs, in level order, in ranges within the budget
        for (int c0 = 0; c0 < T.n_leaf; c0 += range) {
            const int n = std::min(range, T.n_leaf - c0);
            const Entry* front = E.conn.p + c0;
            RC(E.entry_hits.ensure(n + 1));  // (counted by k_np, read by the bucket comparison only)
            int n_items = 0;
            RC(np_slot_tests(ctx, d_pairs, front, n, &n_items));
            if (n_items == 0) continue;
            RC(E.flag_off.ensure(n_items + 1));
            RC(scan(ctx, E.hit.p, E.flag_off.p, n_items));
            RC(E.rec.ensure_keep(14 * (size_t)(n_rec + n_items + 1), 14 * (size_t)n_rec, s));
            RC(E.rec_pair.ensure_keep((size_t)(n_rec + n_items + 1), (size_t)n_rec, s));
            LAUNCH(k_emit, n_items, n_items, E.hit.p, E.flag_off.p, E.items.p, 6, front, (const int32_t*)nullptr,
                   d_pairs, E.res.p, E.pfut.p, ctx->geo_eps.p, E.rec.p, E.rec_pair.p, n_rec);
            int32_t hits = 0;
            const int32_t* src = E.flag_off.p + n_items;
            RC(read_scalars(ctx, &src, 1, &hits));
            n_rec += hits;
        }
        if (T.n_leaf > 0) {  // the leaf pairs' slots, counted by k_np_filter
            D2G_CUDA(cudaMemcpyAsync(ctx->h_pinned, E.lc.p, sizeof(int32_t) * LC_SIZE, cudaMemcpyDeviceToHost, s));
            D2G_CUDA(cudaStreamSynchronize(s));
            for (int k = 0; k < LC_TRI_N; k++) T.tri += (uint32_t)ctx->h_pinned[LC_TRI + k];
        }
        c_node += T.nodes + T.n_leaf - T.n_root;  // root pairs of two leaves are in both
        c_tri += T.tri;
        c_levels += T.levels;
        peak = std::max(peak, T.peak);
        p0 = p1;
    }
    if (n_pairs > 0) E.np_chunk = chunk >= n_pairs ? 0 : (peak < 1.0 / 3.0 ? 2 * chunk : chunk);
    RC(finish_records(ctx, n_pairs, n_rec));
    D2G_CUDA(cudaGetLastError());
    *n_out = n_rec;
    if (counters) {
        counters[0] = c_node;
        counters[1] = c_tri;
        counters[2] = 0;
        counters[3] = c_levels;
    }
    return D2G_OK;
}

// findContactsBucketComparison (comparison_dist.h:205-240) as the reference's
// strategy interface issues it: one body pair, the node pairs of one level of
// compareTreesFull (full_tree_comparison.h:25).  The level runs as a level of
// run_narrowphase does (FP32 candidate bounds, then one FP64 triangle
// distance per surviving slot), except that every hit is emitted, in slot
// order, and the per-node-pair hit counts are summed into the reference's
// cumulative pair_used_out.
int run_bucket_comparison(d2g_ctx* ctx, const int32_t* d_pair, const int32_t* d_node_pairs, int n, int* n_hits) {
    Engine& E = ctx->eng;
    cudaStream_t s = ctx->stream;
    RC(E.pm.ensure(33));
    RC(E.search.ensure(2));
    RC(E.pm32.ensure(kNpPose32));
    RC(E.roots.ensure(2));
    LAUNCH(k_np_prep, 1, 1, d_pair, ctx->fut.p, ctx->mesh.p, ctx->mesh_node_off.p, ctx->geo_eps.p, E.pm.p,
           E.search.p, E.roots.p, E.pm32.p, nullptr);
    RC(E.soup.ensure(n + 1));
    RC(E.off_a.ensure(n + 1));
    RC(E.entry_hits.ensure(n + 1));
    D2G_CUDA(cudaMemsetAsync(E.entry_hits.p, 0, sizeof(int32_t) * (n + 1), s));
    *n_hits = 0;
    if (n == 0) {
        D2G_CUDA(cudaMemsetAsync(E.off_a.p, 0, sizeof(int32_t), s));
        return D2G_OK;
    }
    LAUNCH(k_bucket_entries, n, n, d_node_pairs, E.soup.p);
    int n_items = 0;
    RC(np_slot_tests(ctx, d_pair, E.soup.p, n, &n_items));
    RC(E.flag_off.ensure(n_items + 1));
    RC(scan(ctx, E.hit.p, E.flag_off.p, n_items));
    RC(scan(ctx, E.entry_hits.p, E.off_a.p, n));
    int32_t tot = 0;
    {
        const int32_t* src = E.off_a.p + n;
        RC(read_scalars(ctx, &src, 1, &tot));
    }
    RC(E.rec.ensure(14 * (size_t)tot + 14));
    RC(E.rec_pair.ensure((size_t)tot + 1));
    if (tot > 0)
        LAUNCH(k_emit, n_items, n_items, E.hit.p, E.flag_off.p, E.items.p, 6, E.soup.p, (const int32_t*)nullptr,
               d_pair, E.res.p, E.pfut.p, ctx->geo_eps.p, E.rec.p, E.rec_pair.p, 0);
    D2G_CUDA(cudaGetLastError());
    *n_hits = tot;
    return D2G_OK;
}

}  // namespace d2g

// ============================================================================
// Allocation-free discrete narrow phase.
//
// For callers that may not allocate device memory while they run: a host that
// hands this library a fixed memory budget up front (game or robotics loops
// with real-time limits, where an allocation can stall or fail mid-frame), or
// an embedding runtime that owns every allocation itself.  Every intermediate
// buffer of the traversal is carved out of the file-scope array below, which
// each GPU that loads this library holds until the process exits.
//
// Limits (larger requests are rejected with D2G_ERR_INVALID and a message,
// before the traversal or at the level that would pass them):
//   body pairs per call          <= D2G_NOALLOC_MAX_PAIRS      (2048; each pair
//                                   puts its root node pair in the first level)
//   node pairs per tree level    <= D2G_NOALLOC_MAX_NODE_PAIRS (2048)
//   contacts found per call      <= D2G_NOALLOC_MAX_CONTACTS   (32768)
// All calls share the array and it keeps the previous call's contents: the
// counters that must start at zero are cleared on every call, and two calls
// whose work overlaps on the GPU (different streams, or different threads)
// race on it.  The call reads each level's sizes back to the host, so it
// synchronizes its stream once per tree level and once at the end.  The first
// call on a device looks up the array's device address (cudaGetSymbolAddress)
// and caches it; make that first call before any stream capture.
// ============================================================================
namespace d2g {
namespace {

constexpr size_t kNoAllocBytes = (size_t)24 << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
void* g_noalloc_ptr[64] = {nullptr};

// Device address of the scratch array on the current device.
int noalloc_base(void** out) {
    int dev = 0;
    D2G_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_error("device index beyond the allocation-free path's table");
        return D2G_ERR_INVALID;
    }
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            set_error(std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
            return D2G_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return D2G_OK;
}

// Bump carve-out of 256-byte aligned pieces.
struct Carve {
    unsigned char* base;
    size_t used, cap;
    template <class T>
    T* take(size_t n) {
        const size_t off = (used + 255) & ~(size_t)255;
        const size_t bytes = n * sizeof(T);
        if (off + bytes > cap) return nullptr;
        used = off + bytes;
        return (T*)(base + off);
    }
};

// Index checks of the caller's device inputs: pair body ids, their mesh ids,
// node links and bucket sizes.  Sets *err to 1 on any violation.
__global__ void k_noalloc_validate(int n_pairs, const int32_t* __restrict__ pairs, int n_bodies,
                                   const int32_t* __restrict__ mesh, int n_meshes,
                                   const int32_t* __restrict__ mesh_node_off, int n_nodes,
                                   const int4* __restrict__ nodes, const int32_t* __restrict__ ntris,
                                   int32_t* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_meshes && (mesh_node_off[i] < 0 || mesh_node_off[i] >= n_nodes)) atomicExch(err, 1);
    if (i < n_pairs) {
        const int a = pairs[2 * i], b = pairs[2 * i + 1];
        if (a < 0 || a >= n_bodies || b < 0 || b >= n_bodies)
            atomicExch(err, 1);
        else if (mesh[a] < 0 || mesh[a] >= n_meshes || mesh[b] < 0 || mesh[b] >= n_meshes)
            atomicExch(err, 1);
    }
    if (i < n_nodes) {
        const int4 nd = nodes[i];
        if (ntris[i] < 0 || ntris[i] > 8 || nd.y < 0 || nd.y > 8 || (nd.z && (nd.x < 0 || nd.x > n_nodes - nd.y)))
            atomicExch(err, 1);
    }
}

// A level of the allocation-free traversal in three launches and one read of
// its sizes (before: 13 launches and copies, two reads; 8 cubes 448 us).
// k_na_slots: 64 threads per node pair, a slot each.  They first transform the
// two buckets' 48 vertices into shared memory, one each: transforming both
// triangles in every slot was 216 FP64 instructions of a node pair's two
// warps, 46 of 70 us a level of 2,048 node pairs, instead of 36.  Contacts are
// wanted of leaf pairs only: their hits go into a mask word per warp.
__global__ void __launch_bounds__(kBlock) k_na_slots(int n, const int32_t* __restrict__ err,
                                                     const Entry* __restrict__ front,
                                                     const int32_t* __restrict__ pairs, const double* __restrict__ pm,
                                                     const int4* __restrict__ nodes,
                                                     const int32_t* __restrict__ ntris,
                                                     const double* __restrict__ tris, const double* __restrict__ eps,
                                                     const double* __restrict__ inner_eps,
                                                     const double* __restrict__ geo_eps,
                                                     const float* __restrict__ search, PrimResult* __restrict__ res,
                                                     double* __restrict__ res_eps, uint32_t* __restrict__ mask,
                                                     int32_t* __restrict__ any) {
    __shared__ double s_v[kBlock / 64][48][3];
    const int w = (int)(blockIdx.x * (kBlock / 64) + (threadIdx.x >> 6)), l = threadIdx.x & 63;
    const bool in = w < n && !*err;
    Entry e{0, 0, 0};
    int na = 0, nb = 0;
    double(*v)[3] = s_v[threadIdx.x >> 6];
    if (in) {
        e = front[w];
        na = ntris[e.na];
        nb = ntris[e.nb];
        const int t = l % 24 / 3, node = l < 24 ? e.na : e.nb;
        if (l < 48 && t < (l < 24 ? na : nb)) {
            const double* p = tris + (size_t)node * 72 + 3 * (l % 24);
            const V3 x = xform_rigid(mk(p[0], p[1], p[2]), pm + 32 * (size_t)e.pair + (l < 24 ? 0 : 16));
            v[l][0] = x.x;
            v[l][1] = x.y;
            v[l][2] = x.z;
        }
    }
    __syncthreads();
    const int ta = l >> 3, tb = l & 7;
    bool h = false, leaf = false;
    if (in && ta < na && tb < nb) {
        auto at = [&](int i) { return mk(v[i][0], v[i][1], v[i][2]); };
        const Tri A{at(3 * ta), at(3 * ta + 1), at(3 * ta + 2)};
        const Tri B{at(24 + 3 * tb), at(24 + 3 * tb + 1), at(24 + 3 * tb + 2)};
        const double ea = eps[(size_t)e.na * 8 + ta], eb = eps[(size_t)e.nb * 8 + tb];
        const double thr = ((double)search[e.pair] + ea) + eb;
        V3 P, Q;
        const double d = tri_tri_dist_below(A, B, thr, P, Q);
        h = d < thr;
        leaf = !ld_node(nodes, e.na).z && !ld_node(nodes, e.nb).z;
        if (h && leaf) {
            const size_t k = 64 * (size_t)w + l;
            put_result(res[k], d, P, Q, 0.0);
            res_eps[4 * k + 0] = geo_eps[pairs[2 * e.pair]] + ea;
            res_eps[4 * k + 1] = geo_eps[pairs[2 * e.pair + 1]] + eb;
            res_eps[4 * k + 2] = inner_eps[(size_t)e.na * 8 + ta];
            res_eps[4 * k + 3] = inner_eps[(size_t)e.nb * 8 + tb];
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, h && leaf), hits = __ballot_sync(0xffffffffu, h);
    if (w < n && (l & 31) == 0) {
        mask[2 * (size_t)w + (l >> 5)] = m;
        any[2 * (size_t)w + (l >> 5)] = hits ? 1 : 0;
    }
}

// One block: the records' offsets and the next level's node pairs
// (full_tree_comparison.h:27-59, as k_expand_level), both from one scan, two
// node pairs a thread.  out: records, node pairs (written when they fit), err.
constexpr int kNaLevel = 1024;
__global__ void __launch_bounds__(kNaLevel) k_na_level(int n, const int32_t* __restrict__ err,
                                                       const Entry* __restrict__ front,
                                                       const int4* __restrict__ nodes,
                                                       const uint32_t* __restrict__ mask,
                                                       const int32_t* __restrict__ any, int32_t* __restrict__ off,
                                                       Entry* __restrict__ next, int max_next,
                                                       int32_t* __restrict__ out) {
    static_assert(2 * kNaLevel >= D2G_NOALLOC_MAX_NODE_PAIRS, "two node pairs a thread");
    __shared__ unsigned long long s_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (*err) {
        if (threadIdx.x < 3) out[threadIdx.x] = threadIdx.x == 2 ? 1 : 0;
        return;
    }
    int cnt[2][2], kids[2] = {0, 0}, first[2] = {0, 0};
    bool open_a[2] = {false, false};
    unsigned long long sum = 0;  // records, and node pairs in the high half
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int w = 2 * threadIdx.x + q;
        cnt[q][0] = w < n ? __popc(mask[2 * w]) : 0;
        cnt[q][1] = w < n ? __popc(mask[2 * w + 1]) : 0;
        if (w < n && (any[2 * w] | any[2 * w + 1])) {
            const int4 A = ld_node(nodes, front[w].na), B = ld_node(nodes, front[w].nb);
            if (A.z || B.z) {
                open_a[q] = A.z && (!B.z || A.w < B.w);
                kids[q] = open_a[q] ? A.y : B.y;
                first[q] = open_a[q] ? A.x : B.x;
            }
        }
        sum += (unsigned long long)(cnt[q][0] + cnt[q][1]) + ((unsigned long long)kids[q] << 32);
    }
    unsigned long long inc = sum;
    for (int o = 1; o < 32; o *= 2) {
        const unsigned long long x = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += x;
    }
    if (lane == 31) s_sum[warp] = inc;
    __syncthreads();
    unsigned long long before = inc - sum, total = 0;
    for (int i = 0; i < 32; i++) {
        if (i < warp) before += s_sum[i];
        total += s_sum[i];
    }
    const int nn = (int)(total >> 32);
    int at = (int)(unsigned)before, to = (int)(before >> 32);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int w = 2 * threadIdx.x + q;
        if (w >= n) break;
        off[2 * w] = at;
        off[2 * w + 1] = at + cnt[q][0];
        at += cnt[q][0] + cnt[q][1];
        if (nn > max_next) continue;
        Entry x = front[w];
        for (int c = 0; c < kids[q]; c++) {
            (open_a[q] ? x.na : x.nb) = first[q] + c;
            next[to++] = x;
        }
    }
    if (threadIdx.x == 0) {
        out[0] = (int)(unsigned)total;
        out[1] = nn;
        out[2] = 0;
    }
}

__global__ void k_na_emit(int n_slots, const uint32_t* __restrict__ mask, const int32_t* __restrict__ off,
                          const Entry* __restrict__ front, const int32_t* __restrict__ pairs,
                          const PrimResult* __restrict__ res, const double* __restrict__ res_eps,
                          const double* __restrict__ geo_eps, double* __restrict__ rec, int32_t* __restrict__ rec_pair,
                          int base) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_slots) return;
    const uint32_t m = mask[k >> 5], bit = 1u << (k & 31);
    if (!(m & bit)) return;
    const int o = base + off[k >> 5] + __popc(m & (bit - 1u));
    const Entry e = front[k >> 6];
    write_record(res[k], res_eps + 4 * (size_t)k, pairs[2 * e.pair], pairs[2 * e.pair + 1], geo_eps,
                 rec + 14 * (size_t)o);
    rec_pair[o] = e.pair;
}

int noalloc_read(cudaStream_t s, const int32_t* src, int32_t* dst, int n) {
    D2G_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    D2G_CUDA(cudaStreamSynchronize(s));
    return D2G_OK;
}

#define NA_LAUNCH(kern, n, ...) kern<<<nblocks(n), kBlock, 0, s>>>(__VA_ARGS__)

}  // namespace
}  // namespace d2g

extern "C" int d2g_compare_trees_full_noalloc(const d2g_device_scene* sc, const int32_t* d_pairs, int32_t n_pairs,
                                              double* d_contacts, int32_t capacity, int32_t* d_offsets,
                                              int32_t* n_contacts, void* stream) {
    using namespace d2g;
    cudaStream_t s = (cudaStream_t)stream;
    if (!sc || !d_offsets || !n_contacts || n_pairs < 0 || (n_pairs > 0 && !d_pairs) || capacity < 0 ||
        (capacity > 0 && !d_contacts) || sc->n_meshes <= 0 || sc->n_bodies <= 0 || !sc->mesh_node_off ||
        !sc->nodes || !sc->ntris || !sc->tris || !sc->eps || !sc->inner_eps || !sc->mesh || !sc->fut ||
        !sc->geo_eps || sc->n_nodes <= 0) {
        set_error("invalid allocation-free narrow-phase arguments");
        return D2G_ERR_INVALID;
    }
    if (n_pairs > D2G_NOALLOC_MAX_PAIRS) {
        set_error("allocation-free narrow phase: " + std::to_string(n_pairs) + " pairs exceed the limit of " +
                  std::to_string(D2G_NOALLOC_MAX_PAIRS));
        return D2G_ERR_INVALID;
    }
    void* base = nullptr;
    if (int rc = noalloc_base(&base)) return rc;
    const int MP = D2G_NOALLOC_MAX_PAIRS, MN = D2G_NOALLOC_MAX_NODE_PAIRS, MR = D2G_NOALLOC_MAX_CONTACTS;
    static_assert(D2G_NOALLOC_MAX_PAIRS <= D2G_NOALLOC_MAX_NODE_PAIRS,
                  "the first tree level holds one root node pair per body pair");
    Carve cv{(unsigned char*)base, 0, kNoAllocBytes};
    double* pm = cv.take<double>(32 * (size_t)MP);
    float* search = cv.take<float>(MP);
    Entry* front = cv.take<Entry>(MN);
    Entry* next = cv.take<Entry>(MN);
    uint32_t* mask = cv.take<uint32_t>(2 * (size_t)MN);
    int32_t* any = cv.take<int32_t>(2 * (size_t)MN);
    int32_t* off = cv.take<int32_t>(2 * (size_t)MN);
    PrimResult* res = cv.take<PrimResult>(64 * (size_t)MN);
    double* res_eps = cv.take<double>(4 * 64 * (size_t)MN);
    double* rec = cv.take<double>(14 * (size_t)MR);
    int32_t* rec_pair = cv.take<int32_t>(MR);
    int32_t* rec_pair_sorted = cv.take<int32_t>(MR);
    int32_t* rec_idx = cv.take<int32_t>(MR);
    int32_t* rec_idx_sorted = cv.take<int32_t>(MR);
    int32_t* err = cv.take<int32_t>(1);
    int32_t* out = cv.take<int32_t>(3);
    const size_t tmp_bytes = kNoAllocBytes - ((cv.used + 255) & ~(size_t)255) - 256;
    void* tmp = cv.take<unsigned char>(tmp_bytes);
    if (!tmp || !err || !out) {
        set_error("allocation-free scratch layout does not fit");
        return D2G_ERR_INVALID;
    }
    const int4* nodes = (const int4*)sc->nodes;
    int32_t h_err = 0;
    D2G_CUDA(cudaMemsetAsync(err, 0, sizeof(int32_t), s));
    int nv = n_pairs > sc->n_nodes ? n_pairs : sc->n_nodes;
    nv = nv > sc->n_meshes ? nv : sc->n_meshes;
    NA_LAUNCH(k_noalloc_validate, nv, n_pairs, d_pairs, sc->n_bodies, sc->mesh, sc->n_meshes, sc->mesh_node_off,
              sc->n_nodes, nodes, sc->ntris, err);
    // (the kernels below do nothing once err is set: its read comes with the
    // first level's)
    auto refused = [&]() {
        set_error("allocation-free narrow phase: a body, mesh or node index is out of range");
        return D2G_ERR_INVALID;
    };
    if (n_pairs > 0) {
        NA_LAUNCH(k_np_prep, n_pairs, n_pairs, d_pairs, sc->fut, sc->mesh, sc->mesh_node_off, sc->geo_eps, pm, search,
                  front, nullptr, err);
    } else {
        if (int rc = noalloc_read(s, err, &h_err, 1)) return rc;
        if (h_err) return refused();
    }
    int n = n_pairs, n_rec = 0, level = 0;
    while (n > 0) {
        NA_LAUNCH(k_na_slots, 64 * n, n, err, front, d_pairs, pm, nodes, sc->ntris, sc->tris, sc->eps, sc->inner_eps,
                  sc->geo_eps, search, res, res_eps, mask, any);
        k_na_level<<<1, kNaLevel, 0, s>>>(n, err, front, nodes, mask, any, off, next, MN, out);
        int32_t got[3] = {0, 0, 0};
        if (int rc = noalloc_read(s, out, got, 3)) return rc;
        if (got[2]) return refused();
        const int tot = got[0], nn = got[1];
        if (n_rec + tot > MR) {
            set_error("allocation-free narrow phase: contacts exceed the limit of " + std::to_string(MR));
            return D2G_ERR_INVALID;
        }
        if (tot > 0)
            NA_LAUNCH(k_na_emit, 64 * n, 64 * n, mask, off, front, d_pairs, res, res_eps, sc->geo_eps, rec, rec_pair,
                      n_rec);
        n_rec += tot;
        if (nn > MN) {
            set_error("allocation-free narrow phase: " + std::to_string(nn) + " node pairs at level " +
                      std::to_string(level + 1) + " exceed the limit of " + std::to_string(MN));
            return D2G_ERR_INVALID;
        }
        Entry* t = front;
        front = next;
        next = t;
        n = nn;
        level++;
    }
    if (n_rec > 0) {
        NA_LAUNCH(k_iota, n_rec, n_rec, rec_idx);
        int bits = 1;
        while ((1 << bits) < n_pairs + 1 && bits < 31) bits++;
        size_t need = 0;
        D2G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, need, rec_pair, rec_pair_sorted, rec_idx, rec_idx_sorted,
                                                 n_rec, 0, bits, s));
        if (need > tmp_bytes) {
            set_error("allocation-free scratch: sort temporary storage too small");
            return D2G_ERR_INVALID;
        }
        size_t avail = tmp_bytes;
        D2G_CUDA(cub::DeviceRadixSort::SortPairs(tmp, avail, rec_pair, rec_pair_sorted, rec_idx, rec_idx_sorted,
                                                 n_rec, 0, bits, s));
        if (n_rec <= capacity) NA_LAUNCH(k_gather, n_rec, n_rec, rec_idx_sorted, rec, d_contacts);
    }
    NA_LAUNCH(k_pair_offsets, n_pairs + 1, n_rec, 0, n_pairs, rec_pair_sorted, d_offsets);
    D2G_CUDA(cudaGetLastError());
    D2G_CUDA(cudaStreamSynchronize(s));
    *n_contacts = n_rec;
    if (n_rec > capacity) {
        set_error("contact capacity " + std::to_string(capacity) + " < " + std::to_string(n_rec));
        return D2G_CAPACITY;
    }
    return D2G_OK;
}
