// Contact filtering and the per-cluster sequential-impulse solve.
//
// filterContacts (collision_detection/contact.h:44-69): one block per body
// pair, a sort by (eps_a + eps_b, |A - B|, input order) and the greedy
// de-duplication of contact midpoints.
//
// SequentialImpulses::solve (strategies/contact_force/sequential_impulses.cpp:
// 104-638): one block, a thread-block cluster or a grid per cluster.  The
// reference's Gauss-Seidel sweep visits the contacts in sorted order and
// integrates both bodies after each one; a contact only reads and writes its
// own two bodies, so contacts are grouped into waves: a contact's wave is one
// past the last wave that touched either of its moving bodies.  Within a wave
// the bodies are disjoint and the contacts run in parallel; every body still
// sees its contacts in sorted order, so every floating-point operation happens
// in the reference's order (static bodies are never integrated; the impulse
// sum the convergence test reads for them is accumulated from per-contact
// deltas in sorted order).
#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "d2g_geom.cuh"
#include "d2g_internal.hpp"
#include "d2g_limits.hpp"

namespace d2g {

namespace {

constexpr int kBlock = 128;
constexpr int kSolveBlock = 256;
constexpr int kGridMinContacts = 128;    // a cluster this large may take a cooperative grid
constexpr int kGridMaxClusters = 8;      // ... with more parts than D2G_TUNE_GRID_MIN_PARTS,
                                         // when at most this many clusters qualify
constexpr int kClusterMinContacts = 32;  // a cluster this large may take a thread-block cluster
constexpr int kOneBlockParts = 32;       // ... and more particles than this
constexpr int kSolveSmemMax = 200 * 1024;  // dynamic shared memory of a solve block at most
inline int nblocks(long long n, int b = kBlock) { return (int)((n + b - 1) / b); }

// -------------------------------------------------------- segment sorts ---
// Contacts are sorted within a body pair (the filter) or a cluster (the
// solve), never across: a block sorts a segment where it lies, in shared
// memory up to the kernel's capacity and in global memory above.  Ascending by
// (a, b, id), or by (a, id) without TWO: ids are distinct, so ties keep their
// input order.  A bitonic network whose merges start with a mirrored step, so
// that all exchanges put the smaller element first and places from n on need
// not exist.  A comparator t of a step within 64 elements belongs to the warp
// that owns them, and needs no block barrier before the next such step.
// (Library segmented sorts took 22 launches and ~175 us of a 296 us filter
// call on 4,000 contacts in 300 pairs, and 12 launches in a solve.)  The filter
// call by its groups, the caller's host copies included, before and now (ms):
//   100,000 of 3                    5.1 / 5.1      1 of 20,000,  21 kept      7.8 / 1.6
//   64 of 2,000, 983 kept each     27.5 / 1.4      1 of 20,000, 1,901 kept     575 / 8.2
//   8 of 8,000, 1,600 kept each     198 / 2.5      1 of 262,144,   21 kept    95.5 / 23.4
//   8 of 9,000 (global memory)      232 / 3.5      1 of 262,144, 2,549 kept  9,118 / 145
constexpr int kSegSmall = 1024;        // elements of the 128-thread kernels' shared memory
constexpr int kSegLarge = 8192;        // ... of the 1,024-thread kernels'
constexpr int kSegSmallBlock = 128, kSegLargeBlock = 1024;
constexpr int kSegLargeSmem = 20 * kSegLarge, kOrderSmem = 12 * kSegLarge;
typedef unsigned long long u64;

template <bool TWO>
__device__ void sort_segment(int n, u64* a, u64* b, int32_t* id) {
    const int nt = (int)blockDim.x;
    int half = 1;  // comparators of a step: half the padded size
    while (2 * half < n) half *= 2;
    auto exchange = [&](int i, int j) {
        if (j >= n) return;
        const u64 ai = a[i], aj = a[j], bi = TWO ? b[i] : 0, bj = TWO ? b[j] : 0;
        const int32_t di = id[i], dj = id[j];
        if (ai < aj || (ai == aj && (bi < bj || (bi == bj && di < dj)))) return;
        a[i] = aj;
        a[j] = ai;
        if (TWO) {
            b[i] = bj;
            b[j] = bi;
        }
        id[i] = dj;
        id[j] = di;
    };
    __syncthreads();
    for (int h = 1; h <= half; h *= 2) {  // sorted runs of h become runs of 2 h
        for (int t = threadIdx.x; t < half; t += nt) {
            const int base = 2 * (t & ~(h - 1)), o = t & (h - 1);
            exchange(base + o, base + 2 * h - 1 - o);
        }
        if (h > 32)
            __syncthreads();
        else
            __syncwarp();
        for (int w = h / 2; w > 0; w /= 2) {
            for (int t = threadIdx.x; t < half; t += nt) {
                const int i = 2 * (t & ~(w - 1)) + (t & (w - 1));
                exchange(i, i + w);
            }
            if (w > 32)
                __syncthreads();
            else
                __syncwarp();
        }
        if (h >= 32) __syncthreads();  // the next merge crosses warps
    }
    __syncthreads();
}

// Segments above the small kernels' capacity go to the large ones' list
// (list[0] counts them): true when the block is to leave segment p.
__device__ __forceinline__ bool leave_segment(int p, int n, int32_t* list) {
    if (n <= kSegSmall) return false;
    if (threadIdx.x == 0) list[1 + atomicAdd(list, 1)] = p;
    return true;
}

// ------------------------------------------------------------ filtering ---
// The midpoint of a contact, and filterContacts' test (contact.h:49-66): h's
// within eps_a + eps_b + margin (c's own) of c's.
__device__ __forceinline__ V3 contact_mid(const double* c) {
    return mk((c[0] + c[3]) / 2, (c[1] + c[4]) / 2, (c[2] + c[5]) / 2);
}
__device__ __noinline__ bool contact_near_exact(const double* c, const double* h, double margin) {
    return norm(contact_mid(c) - contact_mid(h)) < (c[6] + c[7]) + margin;
}

// The same in FP32 on midpoints relative to the pair's first contact: a
// distance further from the search radius than both roundings can move it (a
// component of the difference by 2^-24 (|x| + |y| + |x - y|), the root by a
// few 2^-24 of itself, the radius by 2^-24 of itself) decides; the rest, and
// whatever is not finite, goes to the FP64 test.
struct NearF {
    float x, y, z, s;
};
__device__ __forceinline__ bool contact_near(const NearF& c, const NearF& h, const double* cr, const double* hr,
                                             double margin) {
    const float dx = c.x - h.x, dy = c.y - h.y, dz = c.z - h.z;
    const float d = sqrtf(dx * dx + dy * dy + dz * dz);
    const float m = 5e-7f * (fabsf(c.x) + fabsf(c.y) + fabsf(c.z) + fabsf(h.x) + fabsf(h.y) + fabsf(h.z)) + 1e-15f;
    if (d + m < c.s * 0.999999f) return true;
    if (d - m > c.s * 1.000001f && d < 1e18f) return false;
    return contact_near_exact(cr, hr, margin);
}

// filterContacts of one body pair's contacts, one block: sorted by
// compareContacts (contact.h:32-40: (eps_a + eps_b, |A - B|), both
// non-negative doubles, whose bit patterns order like the values), then the
// greedy pass (contact.h:49-66): a contact is kept unless near an already kept
// one.  Contacts are taken 32 at a time: every warp tests them against its
// share of the kept ones, then warp 0 resolves the 32 in order (the lowest
// surviving lane is kept and eliminates the later lanes near it).  The kept
// contacts' FP32 midpoints and ids are compacted to the segment's front.
// Bounded by the serial chain of kept contacts, ~60 instructions each; with
// FP64 distances it was ~20 FP64 instructions at 64 cycles.
struct FilterArgs {
    const int32_t* off;
    const double* rec;
    double margin;
    u64 *ga, *gb;        // global working arrays of the largest segments
    int32_t *order, *cnt, *list;
};
__device__ void filter_segment(const FilterArgs& f, int p, int n, u64* a, u64* b, int32_t* id) {
    const int c0 = f.off[p], nt = (int)blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = nt >> 5;
    for (int i = threadIdx.x; i < n; i += nt) {
        const double* c = f.rec + 14 * (size_t)(c0 + i);
        a[i] = (u64)__double_as_longlong(c[6] + c[7]);
        b[i] = (u64)__double_as_longlong(norm(mk(c[0] - c[3], c[1] - c[4], c[2] - c[5])));
        id[i] = c0 + i;
    }
    sort_segment<true>(n, a, b, id);
    const V3 o = n > 0 ? contact_mid(f.rec + 14 * (size_t)c0) : mk(0, 0, 0);
    for (int i = threadIdx.x; i < n; i += nt) {  // the keys' places take the midpoints
        const double* c = f.rec + 14 * (size_t)id[i];
        const V3 m = contact_mid(c) - o;
        *(float2*)(a + i) = make_float2((float)m.x, (float)m.y);
        *(float2*)(b + i) = make_float2((float)m.z, (float)((c[6] + c[7]) + f.margin));
    }
    __shared__ unsigned s_dead[kSegLargeBlock / 32];
    __shared__ int s_kept;
    __syncthreads();
    auto at = [&](int i) {
        const float2 u = *(const float2*)(a + i), v = *(const float2*)(b + i);
        return NearF{u.x, u.y, v.x, v.y};
    };
    int nk = 0;
    for (int base = 0; base < n; base += 32) {
        const int j = base + lane;
        const bool in = j < n;
        const NearF me = at(in ? j : base);
        const int32_t my = id[in ? j : base];
        const double* mr = f.rec + 14 * (size_t)my;
        bool alive = in;
        for (int t = warp; t < nk && alive; t += nw)
            if (contact_near(me, at(t), mr, f.rec + 14 * (size_t)id[t], f.margin)) alive = false;
        const unsigned dead = __ballot_sync(0xffffffffu, !alive);
        if (lane == 0) s_dead[warp] = dead;
        __syncthreads();  // every warp has read this chunk: kept contacts may take its places
        if (warp == 0) {
            unsigned d = lane < nw ? s_dead[lane] : 0u;
            d = __reduce_or_sync(0xffffffffu, d);
            alive = !((d >> lane) & 1u);
            unsigned kept = 0, live = __ballot_sync(0xffffffffu, alive);
            while (live) {
                const int src = __ffs(live) - 1;
                kept |= 1u << src;
                const NearF h{__shfl_sync(0xffffffffu, me.x, src), __shfl_sync(0xffffffffu, me.y, src),
                              __shfl_sync(0xffffffffu, me.z, src), 0.0f};
                const int32_t hid = __shfl_sync(0xffffffffu, my, src);
                if (alive && lane > src && contact_near(me, h, mr, f.rec + 14 * (size_t)hid, f.margin)) alive = false;
                live = __ballot_sync(0xffffffffu, alive) & ~((2u << src) - 1u);
            }
            if ((kept >> lane) & 1u) {
                const int k = nk + __popc(kept & ((1u << lane) - 1u));
                *(float2*)(a + k) = make_float2(me.x, me.y);
                *(float2*)(b + k) = make_float2(me.z, me.s);
                id[k] = my;
            }
            if (lane == 0) s_kept = nk + __popc(kept);
        }
        __syncthreads();
        nk = s_kept;
    }
    for (int i = threadIdx.x; i < nk; i += nt) f.order[c0 + i] = id[i];
    if (threadIdx.x == 0) f.cnt[p] = nk;
    __syncthreads();
}

__global__ void __launch_bounds__(kSegSmallBlock) k_filter(FilterArgs f) {
    __shared__ u64 a[kSegSmall], b[kSegSmall];
    __shared__ int32_t id[kSegSmall];
    const int p = blockIdx.x, n = f.off[p + 1] - f.off[p];
    if (!leave_segment(p, n, f.list)) filter_segment(f, p, n, a, b, id);
}
__global__ void __launch_bounds__(kSegLargeBlock) k_filter_large(FilterArgs f) {
    extern __shared__ __align__(16) unsigned char dyn[];
    u64 *a = (u64*)dyn, *b = a + kSegLarge;
    int32_t* id = (int32_t*)(b + kSegLarge);
    for (int q = blockIdx.x; q < f.list[0]; q += gridDim.x) {
        const int p = f.list[1 + q], c0 = f.off[p], n = f.off[p + 1] - c0;
        if (n <= kSegLarge)
            filter_segment(f, p, n, a, b, id);
        else
            filter_segment(f, p, n, f.ga + c0, f.gb + c0, f.order + c0);
    }
}

// Kept contacts, in sorted order per pair, to their scanned positions: a warp
// per pair copies its 14-double records in one run.
__global__ void k_filter_write(int n_pairs, const int32_t* __restrict__ off, const int32_t* __restrict__ order,
                               const int32_t* __restrict__ out_off, const double* __restrict__ rec,
                               double* __restrict__ out) {
    const int p = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    if (p >= n_pairs) return;
    const int o0 = out_off[p], n = 14 * (out_off[p + 1] - o0);
    const int32_t* ids = order + off[p];
    double* d = out + 14 * (size_t)o0;
    for (int e = threadIdx.x & 31; e < n; e += 32) d[e] = rec[14 * (size_t)ids[e / 14] + e % 14];
}

// ---------------------------------------------------------------- solve ---
// What a sweep of the reference really recomputes.  updateState
// (sequential_impulses.cpp:46-70) integrates a body's state from its impulse
// sums: v from imp, x from ioff, L from rimp, and q from roff.  roff only ever
// receives the friction loop's zero updates, so q, the rotation and with it
// R * local of every contact are constants of a solve; updateStateImmediate's
// state is read by nothing that reaches a result.  A contact's update is
// therefore two short chains: a position half (x, ioff, the offset impulse
// and the penetration test) that reads nothing of the other, and a velocity
// half (v, L, imp, rimp, the normal impulse) that reads the position half's
// lever arms and test.  Every value is produced by the reference's operations
// in the reference's order.
//
// The halves run on different warps, the position half one wave ahead:
// GB300 issues an FP64 warp instruction every 64 cycles per SM sub-partition
// whatever the number of active lanes, so a wave costs the longest warp's
// FP64 instruction count, 28 for the velocity half and 21 for the position
// half, against ~143 when one warp formed both with the quaternion integration
// of two states.  A contact takes eight lanes of each (side A or B, component).
// Where a block has a single task of at most four contacts in a wave its four
// sub-partitions have room for sixteen lanes a contact: products, divisions and
// the linear and angular sums run side by side, 20 instructions either half,
// with the next wave's constants loaded before the barrier.
// Bodies live in shared memory (spread over the blocks of a thread-block
// cluster, read and written through distributed shared memory) and a contact
// in the shared memory of the block that always processes it, both in global
// memory where they do not fit or the blocks form a cooperative grid.
//
// A wave of one contact in one block takes 1.3 us (7.2 before); the table at
// run_solve has the layouts.

struct BodyS {  // one body's working state
    double x[3], v[3], w[3];  // position, velocity, body inverse inertia * L
    double imp[3], rimp[3], ioff[3], last_imp[3];
    double fx[3], fv[3], fL[3];  // the input future state
    double ii[9], m, rm;  // rm = 1 / m, for div_by
    int32_t is_static, rbad;  // rbad: friction iteration (1-based) whose lever arm was not finite, 0 = none
};

struct ConS {  // one contact's working state in the normal loop
    double rl[2][3], n[3];  // R * local per side, the normal
    double r[2][3];         // lever arms p1 - x, from the position half to the velocity half
    double imp, off, outer, m, slop, damp_m;
    BodyS* body[2];
    double* sd;          // where its impulse delta on a static body goes, or null
    int32_t ci;          // the contact in sorted order, -1: an unused place
    int16_t near_, sneg;  // d1 < outer (position half); the delta is -u (the static body is b)
};

struct BodyG {  // per body, written once per solve (global memory)
    double Ti[16];     // inverse transform of the input future state
    double R0[9];      // its rotation
    double q[4], R[9];  // the solved state's quaternion and rotation
};

struct ConG {  // per contact in sorted order (global memory)
    double local[2][3], n[3], outer, mass_eff, slop, damp_m, impulse;
    double rl[2][3], rF[2][3];  // R * local; contact point - input position
    double u[3], rf[2][2][3], lf[3];  // body update, torques (by iteration parity and side), friction impulse
    double mu, cnt, rcnt;
    int32_t a, b;  // particle indices within the cluster
};

__device__ __forceinline__ V3 ld3(const double* p) { return mk(p[0], p[1], p[2]); }
__device__ __forceinline__ void st3(double* p, V3 v) {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
}
__device__ __forceinline__ V3 calc_torque(V3 force, V3 point, V3 com) { return cross(-force, point - com); }
__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
// v with its sign flipped where f (an integer operation)
__device__ __forceinline__ double neg_if(double v, bool f) {
    return __hiloint2double(__double2hiint(v) ^ (f ? (int)0x80000000 : 0), __double2loint(v));
}
// Comparisons of the hot loops on bit patterns: the FP64 pipe takes a
// comparison at the price of an addition.
__device__ __forceinline__ bool is_pos(double v) {  // v > 0 (false for NaN)
    const long long b = __double_as_longlong(v);
    return b > 0 && b <= 0x7ff0000000000000ll;
}
__device__ __forceinline__ double max0(double v) {  // dmax(v, 0.0): v unless v < 0
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull ? 0.0 : v;
}
// sqrt(s) > 1e-6 and sqrt(s) > 1e-4 for s >= 0 without the root: the rounded
// square root is monotone, and these are the largest doubles whose root does
// not pass the bound (false for NaN).
constexpr double kSqMax1e6 = 1e-12, kSqMax1e4 = 1.0000000000000002e-08;
__device__ __forceinline__ bool sq_above(double s, double lim) {
    const long long b = __double_as_longlong(s);
    return b > __double_as_longlong(lim) && b <= 0x7ff0000000000000ll;
}

// x / y given ry = 1 / y: m_div_recip (same result), its three operations
// issued ahead of the range checks, which run beside them.
__device__ __forceinline__ double div_by(double x, double y, double ry) {
    const double q = x * ry;
    const double r = fma(-q, y, x);
    double res = fma(r, ry, q);
    const bool yok = (unsigned)(m_exp_field(y) - 573) <= 900u;
    if (!(yok && (unsigned)(m_exp_field(q) - 573) <= 900u)) {
        if (yok && m_is_zero(x))
            res = q;
        else
            res = x / y;
    }
    return res;
}

// Synchronisation of one cluster's solve: the threads of one block, the
// blocks of a thread-block cluster (the hardware cluster barrier), or every
// thread of a cooperative grid (all blocks resident) for a very large
// cluster.  The grid barrier is a 64-bit arrival counter in global memory:
// each block's thread 0 adds 1 with release semantics and waits, with
// acquire loads, until the count reaches the blocks times the barriers
// passed; the wait is bounded, and a barrier that gives up records the fact
// so the kernel can stop and report it.
enum SyncMode : int { kSyncBlock = 0, kSyncGrid = 1, kSyncCluster = 2 };

// A cluster's small integers (shared memory of a block, else global memory
// zeroed before the launch).
enum { kFlFail = 0, kFlLevels, kFlTasks, kFlAny0, kFlAny1, kFlSpin, kFlStatics, kFlCursor, kFlags };

struct SolveSync {
    unsigned long long* count;  // grid barrier arrivals (monotonic within a launch)
    unsigned long long* passed;  // grid: the block's barriers passed so far (shared memory)
    int32_t* flags;
    unsigned int spin_limit;  // polls before a grid barrier wait gives up
};

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_add_release_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed_i32(const int32_t* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Every thread of the thread-block cluster; release / acquire at cluster
// scope order the blocks' global and shared memory accesses across it.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Grid barrier: after __syncthreads each block's thread 0 arrives with a
// release add (releasing its block's writes) and polls with acquire loads
// until every block has arrived as often as it has, then __syncthreads
// hands the acquired writes to the block.  The barriers passed so far are
// counted per block in shared memory (every block passes the same ones).
template <int MODE>
__device__ __forceinline__ bool solve_sync(const SolveSync& S) {
    if (MODE == kSyncBlock) {
        __syncthreads();
        return true;
    }
    if (MODE == kSyncCluster) {
        __syncwarp();
        cluster_barrier();
        return true;
    }
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        red_add_release_u64(S.count, 1ull);
        const unsigned long long target = (unsigned long long)gridDim.x * ++*S.passed;
        unsigned int spins = 0;
        while (ld_acquire_u64(S.count) < target) {
            if (++spins > S.spin_limit) {  // seconds at the default: the other blocks are gone
                atomicExch(S.flags + kFlSpin, 1);
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// true when any thread of the cluster's solve passes v; flag 0 or 1 by the
// call's parity (the other one is cleared for the next call by the first
// block, gb = 0).
template <int MODE>
__device__ __forceinline__ bool solve_any(const SolveSync& S, bool v, int parity, int gb, bool* ok) {
    const bool blk = __syncthreads_or(v ? 1 : 0) != 0;
    if (MODE == kSyncBlock) return blk;
    if (threadIdx.x == 0 && blk) atomicOr(S.flags + kFlAny0 + parity, 1);
    *ok = solve_sync<MODE>(S) && *ok;
    const bool r = ld_relaxed_i32(S.flags + kFlAny0 + parity) != 0;
    if (gb == 0 && threadIdx.x == 0) S.flags[kFlAny0 + (parity ^ 1)] = 0;
    return r;
}

// Arguments of a cluster solve.
struct SolveArgs {
    const int32_t *cl_part_off, *cl_parts, *cl_con_off, *order;
    const double* rec;
    const int32_t* pair_cnt;
    const double *warm, *cl_step;
    const uint8_t* is_static;
    const double *mass, *ii, *mu;
    double* fut;
    double gravity_z;
    // work arrays: per particle of the call, per contact, and the waves' tasks
    BodyG* bg;
    BodyS* bs;    // bodies that are not in shared memory
    ConG* cg;
    ConS* cs;     // contacts that are not in shared memory (four places per contact)
    int32_t *slot, *deg, *boff, *statics;  // per body; per particle
    int2* ab;          // contacts' particles, bit 30 marks a static one
    int32_t *blist, *lpos, *prev, *level;  // two per contact (level: one)
    int32_t *tcon, *tl;  // contacts of the waves' tasks, first task of every wave
    double* sdelta;      // per entry of blist: a contact's impulse delta on a static body
    int32_t *status, *iters;
    double* out_impulse;
    int32_t* out_ab;
    const int32_t* con_pair;
    double* pair_warm;
    int smem;   // dynamic shared memory, bytes
    int lanes;  // D2G_TUNE_SOLVE_LANES
};

constexpr int kStaticBit = 1 << 30;
constexpr int kWaveCache = 1024;  // wave bounds kept in shared memory

// Body p of the cluster: block p % G's shared memory, or global memory.
template <int MODE>
__device__ __forceinline__ BodyS* body_at(int p, BodyS* sm, BodyS* gl, bool in_smem, int G) {
    if (!in_smem) return gl + p;
    if (MODE == kSyncBlock) return sm + p;
    unsigned long long out;
    asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"((unsigned long long)(sm + p / G)), "r"(p % G));
    return (BodyS*)out;
}

// The position half of one contact (sequential_impulses.cpp:239-378): eight
// lanes, side = lane bit 2, component = lane bits 0-1 (the fourth lane repeats
// x and writes nothing).
__device__ __forceinline__ void position_half(ConS& C, bool act, int side, int c, double t, double rt) {
    const int lane = threadIdx.x & 31, cc = c < 3 ? c : 0, base = lane & ~3;
    BodyS& B = *C.body[side];
    const double x = B.x[cc], ioff = B.ioff[cc], fx = B.fx[cc], m = B.m, rm = B.rm;
    const double n = C.n[cc];
    const bool st = B.is_static != 0;
    const double p1 = C.rl[side][cc] + x;
    const double r = p1 - x;
    const double pr = p1 * n;
    const double dv = (shfl_d(pr, base) + shfl_d(pr, base | 1)) + shfl_d(pr, base | 2);
    const double ot = shfl_d(dv, lane ^ 4);
    const double d1 = (side ? dv : ot) - (side ? ot : dv);  // n.p1B - n.p1A
    const double pen = C.outer - d1;
    const bool near_ = is_pos(pen);  // d1 < outer
    const double e = pen - C.slop;
    const double off0 = C.off;
    const double dn = div_by(C.damp_m * (is_pos(e) ? e : 0.0), t, rt);
    const double off1 = max0(off0 + (near_ ? dn : neg_if(off0, true)));
    const double uo = neg_if(n, true) * (off1 - off0);
    const double io = ioff + neg_if(uo, side);
    const double xn = fx + div_by(io, m, rm) * t;
    __syncwarp();
    if (act && c < 3) {
        C.r[side][c] = r;
        if (!st) {
            B.ioff[c] = io;
            B.x[c] = xn;
        }
        if ((side | c) == 0) {
            C.off = off1;
            C.near_ = near_ ? 1 : 0;
        }
    }
}

// The velocity half, lanes as above, with the lever arms and the test that
// the position half left in the contact.
__device__ __forceinline__ void velocity_half(ConS& C, bool act, int side, int c) {
    const int lane = threadIdx.x & 31, cc = c < 3 ? c : 0, base = lane & ~3;
    const int c1 = cc == 2 ? 0 : cc + 1, c2 = cc == 0 ? 2 : cc - 1;
    BodyS& B = *C.body[side];
    const double w1 = B.w[c1], w2 = B.w[c2], r1 = C.r[side][c1], r2 = C.r[side][c2];
    const double v = B.v[cc], n = C.n[cc];
    const double imp_b = B.imp[cc], rimp_b = B.rimp[cc], fv = B.fv[cc], fL = B.fL[cc], m = B.m, rm = B.rm;
    const double i0 = B.ii[3 * cc], i1 = B.ii[3 * cc + 1], i2 = B.ii[3 * cc + 2];
    const bool st = B.is_static != 0;
    const double vs = v + (w1 * r2 - w2 * r1);  // v + (ii L) x (p1 - x)
    const double pr = vs * n;
    const double dv = (shfl_d(pr, base) + shfl_d(pr, base | 1)) + shfl_d(pr, base | 2);
    const double ot = shfl_d(dv, lane ^ 4);
    const double v1 = (side ? ot : dv) - (side ? dv : ot);  // n.v1A - n.v1B
    const double imp0 = C.imp;
    const double dn = (v1 * C.m) * 0.1;
    const double imp1 = max0(imp0 + (C.near_ ? dn : neg_if(imp0, true)));
    const double u = neg_if(n, true) * (imp1 - imp0);
    const double us = neg_if(u, side);
    const double nus = neg_if(us, true);
    const double n1 = shfl_d(nus, base | c1), n2 = shfl_d(nus, base | c2);
    const double rimp = rimp_b + (n1 * r2 - n2 * r1);
    const double L = fL + rimp;
    const double imp = imp_b + us;
    const double L0 = shfl_d(L, base), L1 = shfl_d(L, base | 1), L2 = shfl_d(L, base | 2);
    const double vn = fv + div_by(imp, m, rm);
    const double w = (i0 * L0 + i1 * L1) + i2 * L2;
    __syncwarp();
    if (act && c < 3) {
        if (!st) {
            B.imp[c] = imp;
            B.rimp[c] = rimp;
            B.v[c] = vn;
            B.w[c] = w;
        }
        if (side == 0) {
            if (C.sd) C.sd[c] = neg_if(u, C.sneg != 0);
            if (c == 0) C.imp = imp1;
        }
    }
}

// The sixteen-lane forms (a warp has two contacts): lane bits 0-1 component,
// bit 2 k, bit 3 side, bit 4 contact.  Lanes that differ in k run different
// operations of one instruction stream: x + y as fma(x, 1, y) and x y as
// fma(x, y, -0), each the same single rounding, so an addition, a product or a
// fused step of div_by can share an instruction: 20 FP64 instructions for the
// velocity half instead of 28 and 20 for the position half instead of 21, 64
// cycles each.  What no other warp writes is loaded one interval ahead
// (HalfPre).  100 cubes on 16 blocks: 164 -> 140 us per iteration.
struct HalfPre {
    ConS* C;
    BodyS* B;
    double* sd;
    bool act, moving, sneg;  // the lane's contact exists; its body is not static; the sign of sd
    double q[9];
};

__device__ __forceinline__ HalfPre velocity16_load(ConS* task, int half) {
    const int lane = threadIdx.x & 31, c = lane & 3, cc = c < 3 ? c : 0, k = (lane >> 2) & 1, side = (lane >> 3) & 1;
    const int c1 = cc == 2 ? 0 : cc + 1, c2 = cc == 0 ? 2 : cc - 1;
    HalfPre t;
    ConS* C = task + 2 * half + (lane >> 4);
    t.act = C->ci >= 0;
    if (!t.act) C = task;  // (a task's first contact exists)
    BodyS& B = *C->body[side];
    t.C = C;
    t.B = &B;
    t.moving = t.act && c < 3 && !B.is_static;
    t.sd = t.act && c < 3 && k && side == 0 ? C->sd : nullptr;
    t.sneg = C->sneg != 0;
    t.q[0] = C->n[k ? c2 : c1];
    t.q[1] = C->n[cc];
    t.q[2] = B.ii[3 * cc + k];
    t.q[3] = B.ii[3 * cc + 2];
    t.q[4] = C->m;
    t.q[5] = B.fv[cc];
    t.q[6] = B.fL[cc];
    t.q[7] = B.m;
    t.q[8] = B.rm;
    return t;
}
__device__ __forceinline__ void velocity_half16(const HalfPre& t) {
    const int lane = threadIdx.x & 31, c = lane & 3, cc = c < 3 ? c : 0, k = (lane >> 2) & 1, side = (lane >> 3) & 1;
    const int c1 = cc == 2 ? 0 : cc + 1, c2 = cc == 0 ? 2 : cc - 1, base = lane & ~7;
    ConS& C = *t.C;
    BodyS& B = *t.B;
    const double wx = B.w[k ? c2 : c1], rx = C.r[side][k ? c1 : c2], v = B.v[cc];
    const double sum = k ? B.imp[cc] : B.rimp[cc], imp0 = C.imp;
    const bool near_ = C.near_ != 0;
    // (w1 r2 on k = 0) - (w2 r1 on k = 1)
    const double p = wx * rx, po = shfl_d(p, lane ^ 4);
    const double vs = v + ((k ? po : p) - (k ? p : po));
    const double pr = vs * t.q[1];
    const double dv = (shfl_d(pr, base) + shfl_d(pr, base | 1)) + shfl_d(pr, base | 2);
    const double ot = shfl_d(dv, lane ^ 8);
    const double v1 = (side ? ot : dv) - (side ? dv : ot);
    const double dn = (v1 * t.q[4]) * 0.1;
    const double imp1 = max0(imp0 + (near_ ? dn : neg_if(imp0, true)));
    const double du = imp1 - imp0;
    // nus = -us in component c1 (k = 0) or c2, times r2 or r1
    const double nus = neg_if(neg_if(t.q[0], true) * du, !side);
    const double g = nus * rx, go = shfl_d(g, lane ^ 4);
    const double nn = neg_if(t.q[1], true);
    const double x1 = fma(k ? nn : g, k ? du : 1.0, k ? -0.0 : neg_if(go, true));  // torque | u
    const double x2 = sum + neg_if(x1, k & side);                                  // rimp | imp
    const double x3 = fma(x2, k ? t.q[8] : 1.0, k ? -0.0 : t.q[6]);                // L | imp / m: q
    const double La = shfl_d(x3, base | k), L2 = shfl_d(x3, base | 2);
    const double P = t.q[2] * La;                                                  // i0 L0 | i1 L1
    const double Po = shfl_d(P, lane ^ 4);
    const double x4 = fma(k ? neg_if(x3, true) : t.q[3], k ? t.q[7] : L2, k ? x2 : -0.0);  // i2 L2 | residual
    const double x5 = fma(k ? x4 : P, k ? t.q[8] : 1.0, k ? x3 : Po);              // i0 L0 + i1 L1 | imp / m
    double im = x5;
    if (k && t.moving) {  // div_by's range checks
        const bool yok = (unsigned)(m_exp_field(t.q[7]) - 573) <= 900u;
        if (!(yok && (unsigned)(m_exp_field(x3) - 573) <= 900u)) im = yok && m_is_zero(x2) ? x3 : x2 / t.q[7];
    }
    const double x6 = (k ? t.q[5] : x5) + (k ? im : x4);                           // w | v
    __syncwarp();
    if (t.moving) {
        (k ? B.imp : B.rimp)[c] = x2;
        (k ? B.v : B.w)[c] = x6;
    }
    if (t.sd) t.sd[c] = neg_if(x1, t.sneg);
    if (t.act && (lane & 15) == 4) C.imp = imp1;
}
__device__ __forceinline__ HalfPre position16_load(ConS* task, int half) {
    const int lane = threadIdx.x & 31, c = lane & 3, cc = c < 3 ? c : 0, side = (lane >> 3) & 1;
    HalfPre t;
    ConS* C = task + 2 * half + (lane >> 4);
    t.act = C->ci >= 0;
    if (!t.act) C = task;
    BodyS& B = *C->body[side];
    t.C = C;
    t.B = &B;
    t.moving = t.act && c < 3 && !B.is_static;
    t.sd = nullptr;
    t.sneg = false;
    t.q[0] = C->rl[side][cc];
    t.q[1] = C->n[cc];
    t.q[2] = C->outer;
    t.q[3] = C->slop;
    t.q[4] = C->damp_m;
    t.q[5] = B.fx[cc];
    t.q[6] = B.m;
    t.q[7] = B.rm;
    t.q[8] = 0.0;
    return t;
}
__device__ __forceinline__ void position_half16(const HalfPre& h, double t, double rt) {
    const int lane = threadIdx.x & 31, c = lane & 3, cc = c < 3 ? c : 0, k = (lane >> 2) & 1, side = (lane >> 3) & 1;
    const int base = lane & ~7;
    ConS& C = *h.C;
    BodyS& B = *h.B;
    const double x = B.x[cc], ioff = B.ioff[cc], off0 = C.off;
    const double p1 = h.q[0] + x;
    const double y = fma(k ? x : p1, k ? -1.0 : h.q[1], k ? p1 : -0.0);  // p1 n | p1 - x
    const double dv = (shfl_d(y, base) + shfl_d(y, base | 1)) + shfl_d(y, base | 2);
    const double ot = shfl_d(dv, lane ^ 8);
    const double d1 = (side ? dv : ot) - (side ? ot : dv);
    const double pen = h.q[2] - d1;
    const bool near_ = is_pos(pen);
    const double e = pen - h.q[3];
    const double dn = div_by(h.q[4] * (is_pos(e) ? e : 0.0), t, rt);
    const double off1 = max0(off0 + (near_ ? dn : neg_if(off0, true)));
    const double uo = neg_if(h.q[1], true) * (off1 - off0);
    const double io = ioff + neg_if(uo, side);
    const double xn = h.q[5] + div_by(io, h.q[6], h.q[7]) * t;
    __syncwarp();
    if (k) {
        if (h.act && c < 3) C.r[side][c] = y;
    } else if (h.moving) {
        B.ioff[c] = io;
        B.x[c] = xn;
    }
    if (h.act && (lane & 15) == 0) {
        C.off = off1;
        C.near_ = near_ ? 1 : 0;
    }
}

// Body p's impulse sums over its contacts in sorted order
// (sequential_impulses.cpp:193-215 and :560-607: imp +- u, rimp - last + new),
// then updateState: eight lanes, lane bit 2 picks imp or rimp, bits 0-1 the
// component.  par: the torques' parity; the other one holds the last ones.
// The list's entries are loaded eight at a time: their latency, not the two
// additions of an entry, would be the cost.
__device__ __forceinline__ void accumulate_body(BodyS& B, const int32_t* __restrict__ list, int n, const ConG* cg,
                                                int par, bool act, bool with_x, double t) {
    constexpr int kChunk = 8;
    const int lane = threadIdx.x & 31, kind = (lane >> 2) & 1, c = lane & 3, cc = c < 3 ? c : 0, base = lane & ~3;
    double acc = kind ? B.rimp[cc] : B.imp[cc];
    if (!act) n = 0;
    for (int k = 0; k < n; k += kChunk) {
        int e[kChunk];
        double s1[kChunk], s2[kChunk];
#pragma unroll
        for (int q = 0; q < kChunk; q++) e[q] = k + q < n ? list[k + q] : -1;
#pragma unroll
        for (int q = 0; q < kChunk; q++) {
            if (e[q] < 0) continue;
            const ConG& C = cg[e[q] >> 1];
            const int role = e[q] & 1;
            s1[q] = kind ? neg_if(C.rf[par ^ 1][role][cc], true) : neg_if(C.u[cc], role != 0);
            s2[q] = C.rf[par][role][cc];
        }
#pragma unroll
        for (int q = 0; q < kChunk; q++) {
            if (e[q] < 0) continue;
            acc = acc + s1[q];
            if (kind) acc = acc + s2[q];
        }
    }
    __syncwarp();
    const double L = B.fL[cc] + acc;  // rimp lanes
    const double L0 = shfl_d(L, base), L1 = shfl_d(L, base | 1), L2 = shfl_d(L, base | 2);
    if (act && c < 3) {
        if (kind) {
            B.rimp[c] = acc;
            B.w[c] = (B.ii[3 * c] * L0 + B.ii[3 * c + 1] * L1) + B.ii[3 * c + 2] * L2;
        } else {
            B.imp[c] = acc;
            B.v[c] = B.fv[c] + div_by(acc, B.m, B.rm);
            if (with_x) B.x[c] = B.fx[c] + div_by(B.ioff[c], B.m, B.rm) * t;
        }
    }
}

// A static body's impulse sum: s plus n deltas in order, one warp; lane c < 3
// returns component c.  get(k, d) loads delta k.  A zero delta changes
// nothing but a zero's sign, which no test reads.
template <class F>
__device__ __forceinline__ double static_sum(double s, int n, F get) {
    const int lane = threadIdx.x & 31;
    for (int b = 0; b < n; b += 32) {
        double d[3] = {0.0, 0.0, 0.0};
        if (b + lane < n) get(b + lane, d);
        unsigned live =
            __ballot_sync(0xffffffffu, !(m_is_zero(d[0]) && m_is_zero(d[1]) && m_is_zero(d[2])));
        while (live) {
            const int k = __ffs(live) - 1;
            live &= live - 1;
            const double a = shfl_d(d[0], k), e = shfl_d(d[1], k), f = shfl_d(d[2], k);
            s = s + (lane == 0 ? a : (lane == 1 ? e : f));
        }
    }
    return s;
}

#define SYNC()                           \
    do {                                 \
        if (!solve_sync<MODE>(S)) {      \
            if (tid == 0) a.status[k] = 3; \
            return;                      \
        }                                \
    } while (0)

// SequentialImpulses::solve of cluster k by G blocks of kSolveBlock threads;
// gb is this block's index among them.  Thread, body and task indices
// interleave the blocks.
template <int MODE>
__device__ void solve_body(int k, int gb, int G, const SolveSync& S, const SolveArgs& a) {
    extern __shared__ __align__(16) unsigned char dyn[];
    const int tid = (int)threadIdx.x * G + gb, nt = kSolveBlock * G;
    const int lane = threadIdx.x & 31, warp = (int)(threadIdx.x >> 5);
    const int p0 = a.cl_part_off[k], np = a.cl_part_off[k + 1] - p0;
    const int c0 = a.cl_con_off[k], nc = a.cl_con_off[k + 1] - c0;
    const double t = a.cl_step[k];
    const double rt = 1.0 / t;  // for div_by
    bool ok = true;
    const int32_t* parts = a.cl_parts + p0;
    volatile int32_t* fl = S.flags;
    ConG* cg = a.cg + c0;
    const int nloc = np > gb ? (np - gb + G - 1) / G : 0;  // bodies of this block
    const size_t body_bytes = sizeof(BodyS) * (size_t)((np + G - 1) / G);
    const bool bodies_in = MODE != kSyncGrid && 2 * body_bytes <= (size_t)a.smem;
    BodyS* bsm = (BodyS*)dyn;
    BodyS* bgl = a.bs + p0;
    unsigned char* rest = dyn + (bodies_in ? body_bytes : 0);
    const size_t rest_bytes = (size_t)a.smem - (bodies_in ? body_bytes : 0);
    auto body = [&](int p) { return body_at<MODE>(p, bsm, bgl, bodies_in, G); };
    auto own_body = [&](int s) { return bodies_in ? bsm + s : bgl + (s * G + gb); };

    // ---- bodies (:178-188), the inverse transforms on the first half of the
    // block's warps, the integrated orientation on the second
    if (MODE == kSyncBlock) {
        if (threadIdx.x < kFlags) S.flags[threadIdx.x] = 0;
        __syncthreads();
    }
    for (int s = threadIdx.x & (kSolveBlock / 2 - 1); s < nloc; s += kSolveBlock / 2) {
        const int p = s * G + gb, g = parts[p];
        const double* F = a.fut + 14 * (size_t)g;
        BodyG& W = a.bg[p0 + p];
        const bool st = a.is_static[g] != 0;
        const State f = load_state(F);
        if (threadIdx.x < kSolveBlock / 2) {
            double T[16];
            transformation(f.q, f.x, T);
            mat_inverse(T, W.Ti);
            for (int r = 0; r < 3; r++)
                for (int q = 0; q < 3; q++) W.R0[3 * r + q] = T[4 * r + q];
            a.deg[p0 + p] = 0;
            if (st)
                a.statics[p0 + atomicAdd(S.flags + kFlStatics, 1)] = p;
            else
                a.slot[g] = p;
        } else {
            BodyS& B = *own_body(s);
            const double m = a.mass[g];
            const double* ii = a.ii + 9 * (size_t)g;
            B.m = m;
            B.rm = 1.0 / m;
            B.is_static = st ? 1 : 0;
            B.rbad = 0;
            for (int q = 0; q < 9; q++) B.ii[q] = ii[q];
            st3(B.fx, f.x);
            st3(B.fv, f.v);
            st3(B.fL, f.L);
            st3(B.x, f.x);
            st3(B.v, f.v);
            st3(B.w, m3_vec(ii, f.L));
            st3(B.imp, mk(m * 0.0, m * 0.0, m * a.gravity_z) * t);
            for (int q = 0; q < 3; q++) B.rimp[q] = B.ioff[q] = 0.0;
            Quat q = f.q;
            if (!st) {
                double Iinv[9];
                world_inv_inertia(f.q, ii, Iinv);
                const V3 omega = m3_vec(Iinv, f.L + t * mk(0.0, 0.0, 0.0));  // roff = 0
                q = qmul(qexp((0.5 * omega) * t), f.q);
            }
            W.q[0] = q.w;
            W.q[1] = q.x;
            W.q[2] = q.y;
            W.q[3] = q.z;
            qmat(q, W.R);
        }
    }
    SYNC();
    const int n_static = fl[kFlStatics];
    // ---- contacts in sorted order: local frames, normal mass, failure test
    // (:109-168) and warm-start impulses (:193-215), two lanes per contact
    for (int b2 = 32 * (warp * G + gb); b2 < 2 * nc; b2 += nt) {
        const int i = (b2 + lane) >> 1, side = lane & 1;
        const bool act = i < nc;
        double term = 0.0;
        int p = 0;
        bool st = false;
        V3 gn = mk(0, 0, 0), A = gn, Bp = gn;
        const double* h = nullptr;
        int oi = 0, g = 0;
        if (act) {
            ConG& C = cg[i];
            oi = a.order[c0 + i];
            h = a.rec + 14 * (size_t)oi;
            A = ld3(h);
            Bp = ld3(h + 3);
            g = (int)h[11 + side];
            st = a.is_static[g] != 0;
            if (st) {
                for (int q = 0; q < n_static; q++) {
                    const int cand = a.statics[p0 + q];
                    if (parts[cand] == g) {
                        p = cand;
                        break;
                    }
                }
            } else {
                p = a.slot[g];
            }
            const BodyG& W = a.bg[p0 + p];
            const double* F = a.fut + 14 * (size_t)g;
            const V3 P = side ? Bp : A, fx = ld3(F + 8);
            const V3 loc = xform_general(P, W.Ti);
            st3(C.local[side], loc);
            const V3 rF = P - fx;
            st3(C.rF[side], rF);
            gn = (Bp - A) / 2.0;
            const V3 rn = cross(rF, gn);
            term = 1.0 / a.mass[g] + quad_form(rn, a.ii + 9 * (size_t)g);
            const double wv = a.warm[oi];
            const double impulse = wv == wv ? wv * 0.75 : 0.0;
            const V3 n = normalized(gn);
            const V3 u = (-n) * impulse;
            // p1 = T_FS local with the input future state's transform
            const V3 p1 = mk(((W.R0[0] * loc.x + W.R0[1] * loc.y) + W.R0[2] * loc.z) + fx.x * 1.0,
                             ((W.R0[3] * loc.x + W.R0[4] * loc.y) + W.R0[5] * loc.z) + fx.y * 1.0,
                             ((W.R0[6] * loc.x + W.R0[7] * loc.y) + W.R0[8] * loc.z) + fx.z * 1.0);
            st3(C.rf[0][side], calc_torque(side ? -u : u, p1, fx));
            for (int q = 0; q < 3; q++) C.rf[1][side][q] = 0.0;
            a.prev[2 * (c0 + i) + side] = -1;
            if (side == 0) {
                st3(C.u, u);
                st3(C.n, n);
                C.impulse = impulse;
                for (int q = 0; q < 3; q++) C.lf[q] = 0.0;
                const int cnt = a.pair_cnt[oi];
                C.cnt = (double)cnt;
                C.rcnt = 1.0 / (double)cnt;
                C.outer = (h[6] + h[7]) * 0.25;
                // the normal loop's slop and damp * m (:260-287) depend on the contact alone
                const double start_dist = norm(A - Bp);
                if (start_dist < 1e-6 && t > 1e-4) atomicExch(S.flags + kFlFail, 1);
                C.slop = lerp1(dmax(C.outer * 0.2, C.outer - start_dist), C.outer * 0.2, 0.3);
            }
        }
        const double tB = shfl_d(term, lane | 1);
        const int pB = __shfl_sync(0xffffffffu, p, lane | 1), gB = __shfl_sync(0xffffffffu, g, lane | 1);
        const bool sB = __shfl_sync(0xffffffffu, st ? 1 : 0, lane | 1) != 0;
        if (act && side == 0) {
            ConG& C = cg[i];
            double kn = 0.0;
            if (!st) kn += term;
            if (!sB) kn += tB;
            C.mass_eff = kn < 1e-6 ? 0.0 : 1.0 / kn;
            C.damp_m = 0.1 * C.mass_eff;
            C.mu = dmin(a.mu[g], a.mu[gB]);
            C.a = p;
            C.b = pB;
            a.ab[c0 + i] = make_int2(p | (st ? kStaticBit : 0), pB | (sB ? kStaticBit : 0));
            // lists: a moving body has every contact that names it, a static one
            // those of which it is a, or b beside a moving a
            atomicAdd(a.deg + p0 + p, 1);
            if ((!sB && pB != p) || (sB && !st)) atomicAdd(a.deg + p0 + pB, 1);
        }
    }
    SYNC();
    if (fl[kFlFail]) {
        if (tid == 0) a.status[k] = 1;
        return;
    }
    // ---- every body's contacts in sorted order, a warp per body: a warp reads
    // the cluster's contacts, coalesced 8-byte loads, up to the body's last one,
    // which needs neither a sort nor an order of arrival (bodies times contacts:
    // 4,096 hulls with 13,466 contacts on the grid solve in 35 ms, 86 before)
    for (int p = warp * G + gb; p < np; p += (kSolveBlock / 32) * G) {
        const int n = a.deg[p0 + p];
        int base = 0;
        if (lane == 0) base = atomicAdd(S.flags + kFlCursor, n);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane == 0) a.boff[p0 + p] = base;
        const bool st = a.is_static[parts[p]] != 0;
        int cnt = 0, carry = -1;
        for (int b = 0; b < nc && cnt < n; b += 32) {
            const int i = b + lane;
            const int2 q = i < nc ? a.ab[c0 + i] : make_int2(-1, -1);
            const bool isa = i < nc && (q.x & ~kStaticBit) == p, isb = i < nc && (q.y & ~kStaticBit) == p;
            const bool in = st ? isa || (isb && !(q.x & kStaticBit)) : isa || isb;
            const unsigned m = __ballot_sync(0xffffffffu, in), low = m & ((1u << lane) - 1u);
            if (in) {
                const int role = isa ? 0 : 1, at = base + cnt + __popc(low);
                a.blist[2 * c0 + at] = 2 * i + role;
                a.lpos[2 * (c0 + i) + role] = at;
                if (!st) a.prev[2 * (c0 + i) + role] = low ? b + 31 - __clz(low) : carry;
            }
            if (m) carry = b + 31 - __clz(m);
            cnt += __popc(m);
        }
    }
    SYNC();
    // ---- the warm-start sums of every body, then updateState
    auto accumulate = [&](int par, bool with_x) {
        const int grp = (int)threadIdx.x >> 3;
        for (int s0 = 0; s0 < nloc; s0 += kSolveBlock / 8) {
            if (s0 + (warp << 2) >= nloc) break;  // uniform per warp
            const int s = s0 + grp;
            const bool in = s < nloc;
            BodyS& B = *own_body(in ? s : s0 + (warp << 2));
            const int p = in ? s * G + gb : gb;
            accumulate_body(B, a.blist + 2 * (size_t)c0 + a.boff[p0 + p], a.deg[p0 + p], cg, par,
                            in && !B.is_static, with_x, t);
        }
    };
    accumulate(0, true);
    for (int q = gb; q < n_static; q += G) {  // static bodies' running sums, by their block's first warp
        const int p = a.statics[p0 + q];
        if (warp != 0) continue;
        double* imp = body(p)->imp;
        const int32_t* list = a.blist + 2 * (size_t)c0 + a.boff[p0 + p];
        const double s = static_sum(lane < 3 ? imp[lane] : 0.0, a.deg[p0 + p], [&](int j, double* d) {
            const int i = list[j] >> 1;
            const bool neg = (a.ab[c0 + i].y & kStaticBit) != 0;  // -u on a static b
            for (int e = 0; e < 3; e++) d[e] = neg_if(cg[i].u[e], neg);
        });
        if (lane < 3) imp[lane] = s;
    }
    // ---- wave schedule, by the first block: round l takes the contacts whose
    // predecessors on both moving bodies lie in earlier rounds; a wave's
    // contacts are dealt to tasks of four
    if (gb == 0 && nc > 0) {
        __shared__ int s_cnt;
        const bool in = 12 * (size_t)nc <= rest_bytes;
        int32_t* lv = in ? (int32_t*)rest : a.level + c0;
        const int32_t* pv = in ? (int32_t*)rest + nc : a.prev + 2 * (size_t)c0;
        for (int i = threadIdx.x; i < nc; i += kSolveBlock) {
            lv[i] = -1;
            if (in) {
                ((int32_t*)rest)[nc + 2 * i] = a.prev[2 * (c0 + i)];
                ((int32_t*)rest)[nc + 2 * i + 1] = a.prev[2 * (c0 + i) + 1];
            }
        }
        int total = 0, l = 0, T = 0;
        volatile int32_t* vlv = lv;
        while (total < nc) {
            if (threadIdx.x == 0) s_cnt = 0;
            __syncthreads();
            for (int i = threadIdx.x; i < nc; i += kSolveBlock) {
                if (vlv[i] >= 0) continue;
                const int pa = pv[2 * i], pb = pv[2 * i + 1];
                const int la = pa < 0 ? -2 : vlv[pa], lb = pb < 0 ? -2 : vlv[pb];
                if (la == -1 || la >= l || lb == -1 || lb >= l) continue;
                vlv[i] = l;
                a.tcon[4 * (size_t)(c0 + T) + atomicAdd(&s_cnt, 1)] = i;
            }
            __syncthreads();
            const int w = s_cnt, tasks = (w + 3) >> 2;
            if (w == 0) break;  // (every round takes at least the first contact left)
            if (threadIdx.x < 4 && w + (int)threadIdx.x < 4 * tasks)
                a.tcon[4 * (size_t)(c0 + T) + w + threadIdx.x] = -1;
            if (threadIdx.x == 0) a.tl[c0 + k + l] = T;
            T += tasks;
            total += w;
            l++;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            a.tl[c0 + k + l] = T;
            fl[kFlLevels] = l;
            fl[kFlTasks] = T;
        }
    }
    SYNC();
    int it_n = 0, it_f = 0;
    if (nc > 0) {
        const int levels = fl[kFlLevels], tasks = fl[kFlTasks];
        const int32_t* tl = a.tl + c0 + k;
        __shared__ int32_t s_tl[kWaveCache];
        if (levels < kWaveCache)
            for (int l = threadIdx.x; l <= levels; l += kSolveBlock) s_tl[l] = tl[l];
        const bool cons_in = sizeof(ConS) * 4 * (size_t)((tasks + G - 1) / G) <= rest_bytes;
        ConS* cs = cons_in ? (ConS*)rest : a.cs + 4 * (size_t)c0;
        // place of task gt's first contact: tasks gb, gb + G, ... are this block's
        auto place = [&](int gt) { return cons_in ? 4 * (gt / G) : 4 * gt; };
        const int n_tasks = tasks > gb ? (tasks - gb + G - 1) / G : 0;
        for (int s = threadIdx.x; s < 8 * n_tasks; s += kSolveBlock) {
            const int gt = (s >> 3) * G + gb, q = (s >> 1) & 3, side = s & 1;
            const int i = a.tcon[4 * (size_t)c0 + 4 * (size_t)gt + q];
            ConS& C = cs[place(gt) + q];
            if (side == 0) C.ci = i;
            if (i < 0) continue;
            ConG& g = cg[i];
            const int2 ab = a.ab[c0 + i];
            const int pw = side ? ab.y : ab.x, p = pw & ~kStaticBit;
            const double* R = a.bg[p0 + p].R;
            const double lx = g.local[side][0], ly = g.local[side][1], lz = g.local[side][2];
            for (int r = 0; r < 3; r++) {
                const double v = (R[3 * r] * lx + R[3 * r + 1] * ly) + R[3 * r + 2] * lz;
                C.rl[side][r] = v;
                g.rl[side][r] = v;
            }
            C.body[side] = body(p);
            if (side == 0) {
                for (int r = 0; r < 3; r++) C.n[r] = g.n[r];
                C.imp = g.impulse;
                C.off = 0.0;
                C.outer = g.outer;
                C.m = g.mass_eff;
                C.slop = g.slop;
                C.damp_m = g.damp_m;
                const bool sa = (ab.x & kStaticBit) != 0, sb = (ab.y & kStaticBit) != 0;
                C.sd = sa || sb ? a.sdelta + 3 * (2 * (size_t)c0 + a.lpos[2 * (c0 + i) + (sa ? 0 : 1)]) : nullptr;
                C.sneg = sa ? 0 : 1;
                C.near_ = 0;
            }
        }
        // every iteration compares the moving bodies' impulses with their values
        // at its start (kept in last_imp, refreshed by the convergence test);
        // static bodies keep their running sums
        for (int s = threadIdx.x; s < nloc; s += kSolveBlock) {
            BodyS& B = *own_body(s);
            for (int q = 0; q < 3; q++) B.last_imp[q] = B.imp[q];
        }
        SYNC();
        // ---- normal loop (:230-395).  Warps 0, 1, 4, 5 take velocity halves,
        // 2, 3, 6, 7 position halves: a block's first two tasks put one warp
        // on each sub-partition.
        const bool vel = (warp & 2) == 0;
        const int rank = (warp & 1) | ((warp >> 1) & 2);
        const int grp = lane >> 3, side = (lane >> 2) & 1, c = lane & 3;
        // The block's tasks of wave l: the first, and how many.
        const int32_t* tls = levels < kWaveCache ? s_tl : tl;
        auto wave_tasks = [&](int l, int& first, int& count) {
            const int lo = tls[l], hi = tls[l + 1];
            if (MODE == kSyncBlock) {
                first = lo;
                count = hi - lo;
            } else {
                int d = gb - lo % G;
                if (d < 0) d += G;
                first = lo + d;
                count = first < hi ? (hi - 1 - first) / G + 1 : 0;
            }
        };
        const bool narrow = narrow_waves(a.lanes, n_tasks, levels);
        bool converged = false;
        int p0w = 0, pcw = 0;  // wave 0's tasks
        wave_tasks(0, p0w, pcw);
        auto load16 = [&](int first) {
            return vel ? velocity16_load(cs + place(first), rank) : position16_load(cs + place(first), rank);
        };
        HalfPre pre;
        pre.act = false;
        if (narrow && !vel && pcw == 1 && rank < 2) pre = load16(p0w);
        while (!converged && it_n < 1000) {
            int pf = p0w, pc = pcw, vf = 0, vc = 0;
            for (int j = 0; j <= levels && narrow; j++) {
                // position halves of wave j (tasks pf, pc), velocity halves of
                // wave j - 1 (vf, vc); then the next interval's constants
                const int first = vel ? vf : pf, count = vel ? vc : pc;
                if (count == 1) {
                    if (rank < 2 && __any_sync(0xffffffffu, pre.act)) {
                        if (vel)
                            velocity_half16(pre);
                        else
                            position_half16(pre, t, rt);
                    }
                } else {
                    for (int u = rank; u < count; u += 4) {
                        ConS* C = cs + place(first + u * G);
                        const bool act = C[grp].ci >= 0;
                        ConS& Cg = C[act ? grp : 0];
                        if (vel)
                            velocity_half(Cg, act, side, c);
                        else
                            position_half(Cg, act, side, c, t, rt);
                    }
                }
                vf = pf;
                vc = pc;
                pf = p0w;  // (after the last wave: the next iteration's first)
                pc = pcw;
                if (j + 1 < levels)
                    wave_tasks(j + 1, pf, pc);
                else if (j + 1 == levels)
                    pc = 0;
                if (rank < 2 && (vel ? vc : pc) == 1 && !(vel && j == levels)) pre = load16(vel ? vf : pf);
                SYNC();
            }
            int t0 = 0, t1 = tls[0], t2 = tls[1];
            for (int j = 0; j <= levels && !narrow; j++) {
                // the same with eight lanes for each contact: wave j's tasks
                // [t1, t2), wave j - 1's [t0, t1)
                const int lo = vel ? t0 : t1, hi = vel ? t1 : t2;
                const int t3 = j + 2 <= levels ? tls[j + 2] : t2;
                int gt = lo + (gb - lo % G + G) % G + rank * G;
                for (; gt < hi; gt += 4 * G) {
                    ConS* C = cs + place(gt);
                    const bool act = C[grp].ci >= 0;
                    ConS& Cg = C[act ? grp : 0];
                    if (vel)
                        velocity_half(Cg, act, side, c);
                    else
                        position_half(Cg, act, side, c, t, rt);
                }
                t0 = t1;
                t1 = t2;
                t2 = t3;
                SYNC();
            }
            // convergence over every particle of the cluster (:380-387)
            bool moved = false;
            for (int s = threadIdx.x; s < nloc; s += kSolveBlock) {
                BodyS& B = *own_body(s);
                if (B.is_static) continue;
                const V3 now = ld3(B.imp), d = now - ld3(B.last_imp);
                moved = moved || sq_above(dot(d, d), kSqMax1e6);
                st3(B.last_imp, now);
            }
            for (int q = gb; q < n_static; q += G) {
                const int p = a.statics[p0 + q];
                if (warp != kSolveBlock / 32 - 1) continue;
                double* imp = body(p)->imp;
                const double* sd = a.sdelta + 3 * (2 * (size_t)c0 + a.boff[p0 + p]);
                const double before = lane < 3 ? imp[lane] : 0.0;
                const double s = static_sum(before, a.deg[p0 + p], [&](int j, double* d) {
                    for (int e = 0; e < 3; e++) d[e] = sd[3 * (size_t)j + e];
                });
                const double d = s - before, d2 = d * d;
                const double sq = (shfl_d(d2, 0) + shfl_d(d2, 1)) + shfl_d(d2, 2);
                moved = moved || sq_above(sq, kSqMax1e6);
                if (lane < 3) imp[lane] = s;
            }
            converged = !solve_any<MODE>(S, moved, it_n & 1, gb, &ok);
            if (!ok) {
                if (tid == 0) a.status[k] = 3;
                return;
            }
            it_n++;
        }
        for (int s = threadIdx.x; s < 4 * n_tasks; s += kSolveBlock) {
            const ConS& C = cs[place((s >> 2) * G + gb) + (s & 3)];
            if (C.ci >= 0) cg[C.ci].impulse = C.imp;
        }
        SYNC();
        // ---- friction loop (:397-607): every contact's update reads the state
        // at the iteration's start, then each body adds its own in sorted order
        converged = false;
        while (!converged && it_f < 100) {
            bool big = false;
            const int par = it_f & 1;
            for (int i = tid; i < nc; i += nt) {
                ConG& C = cg[i];
                BodyS &A = *body(C.a), &B = *body(C.b);
                const bool sa = A.is_static != 0, sb = B.is_static != 0;
                const V3 n = ld3(C.n), xA = ld3(A.x), xB = ld3(B.x);
                V3 lA = ld3(C.rl[0]), lB = ld3(C.rl[1]);
                // a lever arm that is not finite makes the body's roff, and so its
                // rotation, NaN from the next iteration on
                const double nan = __longlong_as_double(0x7ff8000000000000ll);
                if (A.rbad && A.rbad <= it_f) lA = mk(nan, nan, nan);
                if (B.rbad && B.rbad <= it_f) lB = mk(nan, nan, nan);
                const V3 rA = (lA + xA) - xA, rB = (lB + xB) - xB;
                auto bad = [](V3 r) {
                    return m_exp_field(r.x) == 2047 || m_exp_field(r.y) == 2047 || m_exp_field(r.z) == 2047;
                };
                if (!sa && bad(rA) && !A.rbad) A.rbad = it_f + 1;
                if (!sb && bad(rB) && !B.rbad) B.rbad = it_f + 1;
                const V3 v1A = sa ? mk(0, 0, 0) : ld3(A.v) + cross(ld3(A.w), rA);
                const V3 v1B = sb ? mk(0, 0, 0) : ld3(B.v) + cross(ld3(B.w), rB);
                const V3 vAB = v1A - v1B;
                const V3 vt = vAB - dot(vAB, n) * n;
                const double max_force = (C.impulse * C.mu) * 10;
                const V3 tan = normalized(vt);
                double kt = 0.0;
                if (!sa) kt += A.rm + quad_form(cross(ld3(C.rF[0]), tan), A.ii);
                if (!sb) kt += B.rm + quad_form(cross(ld3(C.rF[1]), tan), B.ii);
                const double mit = kt < 1e-6 ? 0.0 : 1.0 / kt;
                const V3 dfi = ((-vt) * mit) * 0.9;
                const V3 last = ld3(C.lf);
                V3 total = last + dfi;
                total = normalized(total) * dclamp(norm(total), 0.0, max_force);
                st3(C.lf, total);
                const V3 d = total - last;
                const V3 u = mk(div_by(d.x, C.cnt, C.rcnt), div_by(d.y, C.cnt, C.rcnt), div_by(d.z, C.cnt, C.rcnt));
                st3(C.u, u);
                big = big || sq_above(dot(u, u), kSqMax1e4);
                st3(C.rf[par][0], cross(-total, rA));
                st3(C.rf[par][1], cross(total, rB));
            }
            SYNC();
            accumulate(par, false);
            // (the static bodies' impulse sums are read only by the normal loop's test)
            converged = !solve_any<MODE>(S, big, (it_n + it_f) & 1, gb, &ok);
            if (!ok) {
                if (tid == 0) a.status[k] = 3;
                return;
            }
            it_f++;
        }
    }
    // ---- write back (:622-624) and the contacts' impulses for the warm start
    for (int s = threadIdx.x; s < nloc; s += kSolveBlock) {
        const BodyS& B = *own_body(s);
        if (B.is_static) continue;
        const int p = s * G + gb;
        double* F = a.fut + 14 * (size_t)parts[p];
        const double* q = a.bg[p0 + p].q;
        for (int e = 0; e < 4; e++) F[1 + e] = B.rbad ? __longlong_as_double(0x7ff8000000000000ll) : q[e];
        for (int e = 0; e < 3; e++) {
            F[5 + e] = B.fL[e] + B.rimp[e];
            F[8 + e] = B.x[e];
            F[11 + e] = B.v[e];
        }
    }
    for (int i = tid; i < nc; i += nt) {
        const ConG& C = cg[i];
        a.out_impulse[c0 + i] = C.impulse;
        a.out_ab[2 * (c0 + i)] = parts[C.a];
        a.out_ab[2 * (c0 + i) + 1] = parts[C.b];
        // Warm-start store (sequential_impulses_warm_start.cpp:28-54): each
        // body pair keeps the impulse of its last contact in sorted order;
        // a pair's first contact enters as 0.0 + impulse.
        if (a.pair_warm) {
            const int oi = a.order[c0 + i], pr = a.con_pair[oi];
            const int role = (a.ab[c0 + i].x & kStaticBit) && !(a.ab[c0 + i].y & kStaticBit) ? 1 : 0;
            const int p = role ? C.b : C.a, end = a.boff[p0 + p] + a.deg[p0 + p];
            bool last = true;
            for (int e = a.lpos[2 * (c0 + i) + role] + 1; e < end && last; e++)
                last = a.con_pair[a.order[c0 + (a.blist[2 * c0 + e] >> 1)]] != pr;
            if (last) a.pair_warm[pr] = a.pair_cnt[oi] == 1 ? 0.0 + C.impulse : C.impulse;
        }
    }
    if (tid == 0) {
        a.status[k] = 0;
        a.iters[2 * k] = it_n;
        a.iters[2 * k + 1] = it_f;
    }
    if (MODE == kSyncCluster) cluster_barrier();  // no block leaves while another reads its shared memory
}

#undef SYNC

// One block per cluster (clusters cl_list[b], or b when cl_list is null).
__global__ void __launch_bounds__(kSolveBlock) k_solve(int n_list, const int32_t* __restrict__ cl_list, SolveArgs a) {
    if ((int)blockIdx.x >= n_list) return;
    __shared__ int32_t s_flags[kFlags];
    const SolveSync S{nullptr, nullptr, s_flags, 0u};
    solve_body<kSyncBlock>(cl_list ? cl_list[blockIdx.x] : (int)blockIdx.x, 0, 1, S, a);
}

// Every block of a cooperative grid on cluster k (all blocks resident).
__global__ void __launch_bounds__(kSolveBlock) k_solve_grid(int k, SolveSync S, SolveArgs a) {
    __shared__ unsigned long long s_passed;
    if (threadIdx.x == 0) s_passed = 0;
    __syncthreads();
    S.passed = &s_passed;
    solve_body<kSyncGrid>(k, (int)blockIdx.x, (int)gridDim.x, S, a);
}

// The blocks of thread-block cluster c solve cluster cl_list[c] together
// (every block of a hardware cluster is resident at once); flags: 16 ints
// per hardware cluster, zeroed before the launch.
__global__ void __launch_bounds__(kSolveBlock) k_solve_cl(const int32_t* __restrict__ cl_list,
                                                          int32_t* __restrict__ flags, SolveArgs a) {
    unsigned int rank, nrank, cid;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(nrank));
    asm("mov.u32 %0, %%clusterid.x;" : "=r"(cid));
    const SolveSync S{nullptr, nullptr, flags + 16 * (size_t)cid, 0u};
    solve_body<kSyncCluster>(cl_list[cid], (int)rank, (int)nrank, S, a);
}

// A cluster's contacts in the order of Contact::operator< (contact.h:17-21): by
// |A - B| / (eps_a + eps_b), a non-negative double, ties in input order.
struct OrderArgs {
    const int32_t* off;
    const double* rec;
    u64* keys;  // global working array of the largest clusters
    int32_t *order, *list;
};
__device__ void order_segment(const OrderArgs& f, int k, int n, u64* key, int32_t* id) {
    const int c0 = f.off[k];
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double* h = f.rec + 14 * (size_t)(c0 + i);
        const double prop = norm(mk(h[0] - h[3], h[1] - h[4], h[2] - h[5])) / (h[6] + h[7]);
        key[i] = (u64)__double_as_longlong(prop);
        id[i] = c0 + i;
    }
    sort_segment<false>(n, key, nullptr, id);
    for (int i = threadIdx.x; i < n; i += blockDim.x) f.order[c0 + i] = id[i];
    __syncthreads();
}
__global__ void __launch_bounds__(kSegSmallBlock) k_order(OrderArgs f) {
    __shared__ u64 key[kSegSmall];
    __shared__ int32_t id[kSegSmall];
    const int k = blockIdx.x, n = f.off[k + 1] - f.off[k];
    if (!leave_segment(k, n, f.list)) order_segment(f, k, n, key, id);
}
__global__ void __launch_bounds__(kSegLargeBlock) k_order_large(OrderArgs f) {
    extern __shared__ __align__(16) unsigned char dyn[];
    u64* key = (u64*)dyn;
    for (int q = blockIdx.x; q < f.list[0]; q += gridDim.x) {
        const int k = f.list[1 + q], c0 = f.off[k], n = f.off[k + 1] - c0;
        if (n <= kSegLarge)
            order_segment(f, k, n, key, (int32_t*)(key + kSegLarge));
        else
            order_segment(f, k, n, f.keys + c0, f.order + c0);
    }
}

#define VLAUNCH(kern, n, ...)                                        \
    do {                                                             \
        kern<<<nblocks(n), kBlock, 0, ctx->stream>>>(__VA_ARGS__);   \
        ctx->eng.launches++;                                         \
    } while (0)
#define RC(x)                          \
    do {                               \
        if (int rc_ = (x)) return rc_; \
    } while (0)

}  // namespace

int allow_segment_smem(d2g_ctx* ctx) {
    Engine& E = ctx->eng;
    if (E.seg_smem_set) return D2G_OK;
    D2G_CUDA(cudaFuncSetAttribute((const void*)k_filter_large, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kSegLargeSmem));
    D2G_CUDA(cudaFuncSetAttribute((const void*)k_order_large, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kOrderSmem));
    E.seg_smem_set = true;
    return D2G_OK;
}

// Per-pair filterContacts of contact records grouped by pair (d_rec /
// d_off over n_pairs), into flt (records) / flt_off / flt_cnt (kept per pair).
int run_filter(d2g_ctx* ctx, const int32_t* d_off, const double* d_rec, int n_pairs, int n_rec, double margin,
               int* n_out) {
    Engine& E = ctx->eng;
    cudaStream_t s = ctx->stream;
    const size_t n = (size_t)n_rec;
    RC(E.flt_idx.ensure(n + 1));
    RC(E.flt_cnt.ensure(n_pairs + 1));
    RC(E.flt_off.ensure(n_pairs + 1));
    if (n_rec > 0 && n_pairs > 0) {
        RC(E.flt_list.ensure(n_pairs + 1));
        FilterArgs f{d_off, d_rec, margin, nullptr, nullptr, E.flt_idx.p, E.flt_cnt.p, E.flt_list.p};
        if (n_rec > kSegLarge) {
            RC(E.flt_keys.ensure(n + 1));
            RC(E.flt_keys_s.ensure(n + 1));
            f.ga = E.flt_keys.p;
            f.gb = E.flt_keys_s.p;
        }
        D2G_CUDA(cudaMemsetAsync(E.flt_list.p, 0, sizeof(int32_t), s));
        D2G_CUDA(cudaMemsetAsync(E.flt_cnt.p + n_pairs, 0, sizeof(int32_t), s));
        k_filter<<<n_pairs, kSegSmallBlock, 0, s>>>(f);
        ctx->eng.launches++;
        if (n_rec > kSegSmall) {  // (else no pair has more)
            RC(allow_segment_smem(ctx));
            k_filter_large<<<ctx->n_sms, kSegLargeBlock, kSegLargeSmem, s>>>(f);
            ctx->eng.launches++;
        }
        size_t bytes = 0;
        D2G_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, E.flt_cnt.p, E.flt_off.p, n_pairs + 1, s));
        RC(E.cub_tmp.ensure(bytes + 16));
        D2G_CUDA(cub::DeviceScan::ExclusiveSum(E.cub_tmp.p, bytes, E.flt_cnt.p, E.flt_off.p, n_pairs + 1, s));
    } else {
        if (n_pairs > 0) D2G_CUDA(cudaMemsetAsync(E.flt_cnt.p, 0, sizeof(int32_t) * n_pairs, s));
        D2G_CUDA(cudaMemsetAsync(E.flt_off.p, 0, sizeof(int32_t) * (n_pairs + 1), s));
    }
    D2G_CUDA(cudaMemcpyAsync(ctx->h_pinned, E.flt_off.p + n_pairs, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    D2G_CUDA(cudaStreamSynchronize(s));
    prof_mark_collect(ctx);
    const int kept = ctx->h_pinned[0];
    RC(E.flt.ensure(14 * (size_t)kept + 14));
    if (kept > 0) VLAUNCH(k_filter_write, 32LL * n_pairs, n_pairs, d_off, E.flt_idx.p, E.flt_off.p, d_rec, E.flt.p);
    *n_out = kept;
    D2G_CUDA(cudaGetLastError());
    return D2G_OK;
}

// Dynamic shared memory of a solve block: its share of np bodies and nc
// contacts (a wave's tasks of four leave places empty, hence the factor), at
// most `cap`; a block whose cluster needs more keeps the contacts, then the
// bodies, in global memory.
int solve_smem(int np, int nc, int G, int cap) {
    const long long want = (long long)sizeof(BodyS) * ((np + G - 1) / G) * (np > 0 ? 1 : 0) +
                           std::max(12LL * nc, (long long)sizeof(ConS) * (2LL * nc / G + 64));
    return (int)std::min<long long>((want + 1023) / 1024 * 1024, cap);
}

// The solve kernels' largest dynamic shared memory, allowed once per context.
int allow_solve_smem(d2g_ctx* ctx) {
    Engine& E = ctx->eng;
    if (E.sv_smem_set) return D2G_OK;
    D2G_CUDA(cudaFuncSetAttribute((const void*)k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, kSolveSmemMax));
    D2G_CUDA(cudaFuncSetAttribute((const void*)k_solve_cl, cudaFuncAttributeMaxDynamicSharedMemorySize, kSolveSmemMax));
    D2G_CUDA(cudaFuncSetAttribute((const void*)k_solve_grid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kSolveSmemMax));
    D2G_CUDA(cudaFuncSetAttribute((const void*)k_solve_cl, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    E.sv_smem_set = true;
    return D2G_OK;
}

void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int cs, int n, int smem, cudaStream_t st) {
    cfg = {};
    cfg.gridDim = dim3((unsigned)(n * cs));
    cfg.blockDim = dim3(kSolveBlock);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

// Thread-block clusters of `cs` solve blocks that can be resident at once
// (cached per context).
int max_solve_clusters(d2g_ctx* ctx, int cs, int* out) {
    Engine& E = ctx->eng;
    const int slot = cs == 16 ? 0 : cs == 8 ? 1 : cs == 4 ? 2 : 3;
    if (E.sv_cl_fit[slot] < 0) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        cluster_config(cfg, at, cs, 1, kSolveSmemMax, nullptr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, (const void*)k_solve_cl, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();  // this size is not available: never chosen
            n = 0;
        }
        E.sv_cl_fit[slot] = n;
    }
    *out = E.sv_cl_fit[slot];
    return D2G_OK;
}

// k_solve_cl over n clusters (list d_list), cs blocks each.
int launch_solve_cl(d2g_ctx* ctx, int cs, int n, const int32_t* d_list, int32_t* d_flags, const SolveArgs& a,
                    cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, cs, n, a.smem, st);
    D2G_CUDA(cudaLaunchKernelEx(&cfg, k_solve_cl, d_list, d_flags, a));
    ctx->eng.launches++;
    return D2G_OK;
}

// Solve clusters.  Contacts (14-double records in the reference's hit order,
// clusters contiguous per d_con_off) with per-contact pair counts and warm
// values (NaN = none).  Outputs: status / iteration counts per cluster, the
// final impulse and body pair of each contact in sorted order.
int run_solve(d2g_ctx* ctx, int n_clusters, const int32_t* d_part_off, const int32_t* d_parts, int n_parts,
              const int32_t* d_con_off, int n_con, const double* d_rec, const int32_t* d_pair_cnt,
              const double* d_warm, const double* d_step, double gravity_z, int32_t* d_status, int32_t* d_iters,
              double* d_out_impulse, int32_t* d_out_ab, const int32_t* d_con_pair, double* d_pair_warm,
              const int32_t* h_con_off, const int32_t* h_part_off) {
    Engine& E = ctx->eng;
    cudaStream_t s = ctx->stream;
    const size_t n1 = (size_t)n_con + 1, np1 = (size_t)n_parts + 1;
    RC(E.sv_order.ensure(n1));
    RC(E.sv_long.ensure(n_clusters + 1));
    RC(E.sv_bg_raw.ensure(sizeof(BodyG) * np1));
    RC(E.sv_bs_raw.ensure(sizeof(BodyS) * np1));
    RC(E.sv_cg_raw.ensure(sizeof(ConG) * n1));
    RC(E.sv_cs_raw.ensure(sizeof(ConS) * 4 * n1));
    RC(E.sv_slot.ensure((size_t)ctx->n_bodies + 1));
    RC(E.sv_part_int.ensure(3 * np1));
    RC(E.sv_con_int.ensure(9 * n1 + 1));
    RC(E.sv_tcon.ensure(4 * n1));
    RC(E.sv_tl.ensure(n_con + n_clusters + 2));
    RC(E.sv_sdelta.ensure(6 * n1));
    RC(allow_solve_smem(ctx));
    if (n_con > 0 && n_clusters > 0) {
        OrderArgs f{d_con_off, d_rec, nullptr, E.sv_order.p, E.sv_long.p};
        if (n_con > kSegLarge) {
            RC(E.sv_keys.ensure(n1));
            f.keys = E.sv_keys.p;
        }
        D2G_CUDA(cudaMemsetAsync(E.sv_long.p, 0, sizeof(int32_t), s));
        k_order<<<n_clusters, kSegSmallBlock, 0, s>>>(f);
        ctx->eng.launches++;
        if (n_con > kSegSmall) {
            RC(allow_segment_smem(ctx));
            k_order_large<<<ctx->n_sms, kSegLargeBlock, kOrderSmem, s>>>(f);
            ctx->eng.launches++;
        }
    }
    if (n_clusters > 0) {
        SolveArgs a;
        a.cl_part_off = d_part_off;
        a.cl_parts = d_parts;
        a.cl_con_off = d_con_off;
        a.order = E.sv_order.p;
        a.rec = d_rec;
        a.pair_cnt = d_pair_cnt;
        a.warm = d_warm;
        a.cl_step = d_step;
        a.is_static = ctx->is_static.p;
        a.mass = ctx->mass.p;
        a.ii = ctx->inv_inertia.p;
        a.mu = ctx->mu.p;
        a.fut = ctx->fut.p;
        a.gravity_z = gravity_z;
        a.bg = (BodyG*)E.sv_bg_raw.p;
        a.bs = (BodyS*)E.sv_bs_raw.p;
        a.cg = (ConG*)E.sv_cg_raw.p;
        a.cs = (ConS*)E.sv_cs_raw.p;
        a.slot = E.sv_slot.p;
        a.deg = E.sv_part_int.p;
        a.boff = a.deg + np1;
        a.statics = a.boff + np1;
        a.ab = (int2*)E.sv_con_int.p;
        a.blist = E.sv_con_int.p + 2 * n1;
        a.lpos = a.blist + 2 * n1;
        a.prev = a.lpos + 2 * n1;
        a.level = a.prev + 2 * n1;
        a.tcon = E.sv_tcon.p;
        a.tl = E.sv_tl.p;
        a.sdelta = E.sv_sdelta.p;
        a.status = d_status;
        a.iters = d_iters;
        a.out_impulse = d_out_impulse;
        a.out_ab = d_out_ab;
        a.con_pair = d_con_pair;
        a.pair_warm = d_pair_warm;
        a.lanes = E.tune[D2G_TUNE_SOLVE_LANES];
        // Where each cluster is solved (us per iteration on GB300, normal and
        // friction; one block / thread-block cluster of 4 / 8 / 16 / grid):
        //     8 cubes, 46 waves of 2.2 contacts     60 /   74 /   72 /  74 /    -
        //    27 cubes, 89 waves of 5.0             123 /  141 /  136 / 136 /  214
        //    32 cubes, two layers                  137 /    - /    - / 146 /  240
        //    36 cubes, four layers                 145 /    - /    - / 158 /  253
        //    48 cubes, four layers                 241 /    - /    - / 182 /  297
        //    64 cubes, four layers                 274 /    - /    - / 185 /  308
        //    64 cubes, one layer                   212 /    - /    - / 124 /  187
        //    81 cubes, one layer                   261 /    - /    - / 130 /  196
        //   100 cubes, one layer                   308 /  185 /  152 / 136 /  204
        //   512 hulls, 24 waves of 71              352 /  118 /   79 /  67 /   78
        //   576 hulls                              398 /    - /    - /  68 /   77
        //   704 hulls                              479 /    - /    - /  74 /   74
        //   768 hulls                              529 /    - /    - /  81 /   83
        // 1,024 hulls, 23 waves of 142             666 /  213 /  124 /  87 /   82
        // 2,304 hulls                             1542 /  480 /  289 / 178 /  133
        // (hull piles of 36 to 216 that converge at once: 16 blocks 0.33 to 0.47
        // ms a call, one block 0.33 to 0.87.)
        // (one to four contacts to a warp throughout, eight lanes each: 61 for
        // the 8 cubes, 165 / 164 for the 100 on 8 / 16 blocks, 71 / 85 and 88 /
        // 90 for 512 and 1,024 hulls on 16 blocks / a grid; the halves undivided,
        // a contact on one warp: 331 for the 8 cubes, 257 for the 1,024 hulls.)
        // A block barrier costs ~0.1 us, the cluster barrier with distributed
        // shared memory ~0.5 us more, a grid barrier ~1.5 us: so one block up
        // to kOneBlockParts particles (one block is still 7 to 9% faster at 33 to
        // 37, 16 are 24% faster at 49), then 16, or the most with which all such
        // clusters of the call are resident at once, and a cooperative grid for a
        // cluster with at least kGridMinContacts contacts and more than
        // D2G_TUNE_GRID_MIN_PARTS parts (768 by default, where the table's two
        // columns cross) when at most kGridMaxClusters qualify (grids run one
        // after another).  D2G_TUNE_SOLVE_CLUSTER fixes the cluster's size.
        // Blocks and thread-block clusters run side by side on two streams, the
        // grids after them.
        const int cl_setting = E.tune[D2G_TUNE_SOLVE_CLUSTER];
        std::vector<int32_t> small, mid, big;
        if (h_con_off && h_part_off)
            for (int c = 0; c < n_clusters; c++)
                if (h_con_off[c + 1] - h_con_off[c] >= kGridMinContacts &&
                    h_part_off[c + 1] - h_part_off[c] > E.tune[D2G_TUNE_GRID_MIN_PARTS])
                    big.push_back(c);
        if ((int)big.size() > kGridMaxClusters) big.clear();
        for (int c = 0, b = 0; c < n_clusters; c++) {
            if (b < (int)big.size() && big[b] == c) {
                b++;
                continue;
            }
            const int nck = h_con_off ? h_con_off[c + 1] - h_con_off[c] : 0;
            const int npk = h_con_off && h_part_off ? h_part_off[c + 1] - h_part_off[c] : 0;
            const bool wide = cl_setting > 1 || (cl_setting == 0 && npk > kOneBlockParts);
            if (h_con_off && wide && nck >= kClusterMinContacts)
                mid.push_back(c);
            else
                small.push_back(c);
        }
        int cs = 1;  // blocks per thread-block cluster
        if (!mid.empty()) {
            if (cl_setting > 1) {
                cs = cl_setting;
            } else {
                for (int cand : {16, 8, 4, 2}) {
                    int fit = 0;
                    RC(max_solve_clusters(ctx, cand, &fit));
                    if (fit >= (int)mid.size()) {
                        cs = cand;
                        break;
                    }
                }
            }
            if (cs == 1) {  // too many to be resident at once: one block each
                small.insert(small.end(), mid.begin(), mid.end());
                std::sort(small.begin(), small.end());
                mid.clear();
            }
        }
        auto smem_of = [&](const std::vector<int32_t>& list, int G, int cap) {
            int m = 0;
            for (int c : list)
                m = std::max(m, h_con_off && h_part_off ? solve_smem(h_part_off[c + 1] - h_part_off[c],
                                                                     h_con_off[c + 1] - h_con_off[c], G, cap)
                                                        : cap);
            return m;
        };
        const bool all_small = mid.empty() && big.empty();
        E.sv_layout[0] = (int)small.size();
        E.sv_layout[1] = (int)mid.size();
        E.sv_layout[2] = (int)big.size();
        E.sv_layout[3] = mid.empty() ? 0 : cs;
        const int pf = prof_mark_begin(ctx, PROF_SOLVE, n_con);
        RC(E.sv_list.ensure(small.size() + mid.size() + 2));
        if (!small.empty()) {
            const int32_t* d_list = nullptr;
            if (!all_small) {
                D2G_CUDA(cudaMemcpyAsync(E.sv_list.p, small.data(), small.size() * sizeof(int32_t),
                                         cudaMemcpyHostToDevice, s));
                d_list = E.sv_list.p;
            }
            // one block alone on its SM may take all of its shared memory
            a.smem = smem_of(small, 1, small.size() <= 128 ? kSolveSmemMax : kSolveSmemMax / 2);
            k_solve<<<(int)small.size(), kSolveBlock, a.smem, s>>>((int)small.size(), d_list, a);
            ctx->eng.launches++;
        }
        if (!mid.empty()) {
            // on the second stream, beside the blocks
            int32_t* d_mid = E.sv_list.p + small.size() + 1;
            RC(E.sv_cl_flags.ensure(16 * mid.size() + 16));
            D2G_CUDA(cudaMemcpyAsync(d_mid, mid.data(), mid.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s));
            D2G_CUDA(cudaMemsetAsync(E.sv_cl_flags.p, 0, (16 * mid.size() + 16) * sizeof(int32_t), s));
            D2G_CUDA(cudaEventRecord(ctx->ev_fork, s));
            D2G_CUDA(cudaStreamWaitEvent(ctx->stream2, ctx->ev_fork, 0));
            a.smem = smem_of(mid, cs, kSolveSmemMax);
            RC(launch_solve_cl(ctx, cs, (int)mid.size(), d_mid, E.sv_cl_flags.p, a, ctx->stream2));
            D2G_CUDA(cudaEventRecord(ctx->ev_join, ctx->stream2));
            D2G_CUDA(cudaStreamWaitEvent(s, ctx->ev_join, 0));
        }
        if (!big.empty()) {
            int per_sm = 0;
            a.smem = kSolveSmemMax;
            D2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve_grid, kSolveBlock, a.smem));
            const int G_max = std::max(1, std::min(ctx->n_sms, ctx->n_sms * per_sm));
            RC(E.sv_grid.ensure(16 * big.size() + 16));
            D2G_CUDA(cudaMemsetAsync(E.sv_grid.p, 0, (16 * big.size() + 16) * sizeof(int32_t), s));
            for (size_t b = 0; b < big.size(); b++) {
                SolveSync S;
                S.count = (unsigned long long*)(E.sv_grid.p + 16 * b);  // 8-byte aligned: 16 ints per cluster
                S.passed = nullptr;
                S.flags = E.sv_grid.p + 16 * b + 4;
                S.spin_limit = (unsigned int)E.tune[D2G_TUNE_SPIN_LIMIT];
                int k = big[b];
                // about one warp of contacts per SM and wave: fewer blocks for
                // smaller clusters keep the grid barriers cheap
                const int nck = h_con_off[k + 1] - h_con_off[k];
                const int G = std::max(1, std::min(G_max, std::max(8, nck / E.tune[D2G_TUNE_GRID_CONTACTS])));
                void* args[] = {&k, &S, &a};
                D2G_CUDA(cudaLaunchCooperativeKernel((const void*)k_solve_grid, dim3(G), dim3(kSolveBlock), args,
                                                     (size_t)a.smem, s));
                ctx->eng.launches++;
            }
        }
        prof_mark_end(ctx, pf);
    }
    D2G_CUDA(cudaGetLastError());
    return D2G_OK;
}

}  // namespace d2g
