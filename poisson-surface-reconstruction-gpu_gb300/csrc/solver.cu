// Stage (c): per-depth Laplacian conjugate gradients and the iso-value.
//
// System of depth d (mesh/solver/LaplacianSolver.cu:27-74,120-267): rows are the nodes of
// depth d, columns their same-depth neighbours, entry ff_x ff_y ff_z (d2_x + d2_y + d2_z)
// stored in FP32 and dropped when |value| <= 1e-6.  Same-depth entries depend only on
// the neighbour offset, so the operator is applied matrix-free from a 27-entry stencil
// per depth and the neighbour table.  Right-hand side: the divergence of the depth.
//
// CG (mesh/solver/CGAlgorithm.cu:10-80): x0 = 0, r0 = b, stops when r.r <= tol^2 or after
// max_iter iterations (or after a fixed count).  All depths are independent; they are
// solved together, by thread-block clusters (k_cg_cluster) or, from depth 5 on of trees of
// depth 8 and 9, by the whole GPU in one cooperative launch (k_cg_grid).
// Precision: the operator, the vectors and the updates are FP32; the dot products and
// residual norms are exact products summed as float pairs in a sibling group (k_cg_grid: in a thread)
// and as integers across lanes, warps and CTAs (CgDig, CgSum).  Every res_period iterations and when the
// recursive residual reaches the tolerance, the true residual b - A x of the current x is
// evaluated the same way; it drives iterative refinement:
// the CG restarts from it when it is above both the tolerance and the floor an FP32
// solution can reach (2^-20 ||b||) and the recursive residual has converged or drifted.
//
// Iso-value (:269-305): mean of the implicit function at the sample points, evaluated in
// FP32 per point and averaged in FP64.
#include <cooperative_groups.h>
#include <type_traits>
#include <vector>
#include "workspace.h"
#include "tables.cuh"

PSR_DEFINE_CONST_TABLES(upload_tables_solver)

namespace cg = cooperative_groups;

namespace psr {

// ---- per-depth CG ---------------------------------------------------------------------
// Every depth is an independent system.  Up to depth 7 the two or three finest depths (most rows,
// most iterations) get a thread-block cluster each; the coarser depths get one CTA each (a cluster
// of one, on a second stream, or a CTA of a further cluster of the same launch).  All run the same
// solver body: a cluster of one CTA is a CTA.
//
// Reductions: every product enters exactly (fma: TwoProduct); the 8 products of a sibling group are
// added as float pairs in one order (cg_group_sum), and the groups' sums as integers: four digits of
// 19 bits on a fixed grid of exponents (CgDig), of which the lowest are dropped below the largest
// group's.  What a group contributes depends on the group alone and integers add in any order, so a
// sum is the same however many CTAs, threads or turns its groups are dealt to: a cloud gets the same
// bits from every cluster size, alone, served and in a batch.  It keeps 58 to 76 bits below the largest
// group, more than the reference's float-rounded products summed in double
// (mesh/solver/CGAlgorithm.cu:106-133), and stays off the FP64 pipes (a dependent FP64 add takes 76
// cycles here, an integer warp reduction about 50).  A CTA's
// sum goes to every CTA of the cluster with st.async, whose arrival on an mbarrier is the barrier
// (836 cycles; a cluster barrier and reads of the others' sums 1,442).  The scalars of an iteration
// (alpha, beta, the continue flag) are computed once per CTA, by the thread that finishes the sum,
// and read by every thread from shared memory.  The sums alternate between two slots, so a slot is
// only rewritten after a reduction that follows its reads.
//
// True residual (iterative refinement): every res_period iterations, and when the
// recursive r.r reaches tol^2, each row's b - sum_k st_k x[nb_k] is evaluated with exact
// products and float-pair sums (staged in the A p buffer) and its norm is taken.  With
// the reference's absolute tolerance (1e-5) and right-hand sides of norm ~1e7, the FP32
// recursion ends with a true residual near 1e-7 ||b||, below what an FP32 x can resolve
// (2^-20 ||b||, 16 ulps of b); refinement restarts the CG from the true residual only
// above that floor (and the tolerance), when the recursive residual has converged or has
// drifted below the true one by more than 2x in norm, at most kCgMaxRefine times and while
// each restart cuts the true r.r fourfold.  Replacing r periodically while keeping the
// direction was tried and fails at this scale: beta = r_true.r_true / r_old.r_old mixes a
// true residual at the FP32 floor with a recursive one far below it and the iteration
// stalls (it ran to the 10,000-iteration cap on the depth-3 system of the superquadric).
//
// One iteration costs two reductions: the direction update p = r + beta p is fused into the
// operator application (a row's neighbours rebuild their p values from r and the
// previous p), so the FP32 operations per element are the textbook loop's:
//   p_k = fma(beta, p_{k-1}, r_k)   Ap = sum_k st_k p_k[nb]   alpha = rr / (p.Ap)
//   x = fma(alpha, p, x)            r = fma(-alpha, Ap, r)    beta = rr_new / rr
// Missing neighbours contribute fma(st_k, 0, y) = y, the same as skipping them.
//
// Resident path (depth >= 1 and fewer than kCgGroups sibling groups per CTA): each CTA owns
// a contiguous chunk of sibling groups and keeps (r_k, p_{k-1}), x and A p of their rows in
// shared memory, 16 bytes a row, sibling-major: row `sib` of local group g sits at element
// sib * GP + g, so the lanes of a warp (consecutive groups) read consecutive words.
// The 27-neighbourhoods of a group's 8 rows are one 4x4x4 block of same-depth nodes, made of
// parts of the 27 sibling groups around it (one per neighbour of its parent); which sibling
// of which neighbour group a block position is, is known at compile time.  So one thread
// applies the operator to a whole group: it visits the 64 positions in order, loads each
// (r, p) once (own shared memory, or a peer's through distributed shared memory) and adds
// it to every row it belongs to, which keeps each row's sum in neighbour order.  Nothing is
// staged and nothing is reread: a group costs 64 loads and 216 FMAs, and the neighbour
// groups (CTA rank, local group: 16 bits) are found once per solve and stay packed in 14
// words a group, in shared memory where they fit (up to 1024 groups).
// A chunk of at most kCgRowGroups groups (the coarser depths) gives every row a thread of
// its own instead, 27 loads each, for a shorter chain (the terms of a group then meet in shared memory,
// one block barrier more a reduction).  The first version fetched a group's
// block with 8 lanes through a staging block in shared memory (8 stores and 27 reads a row
// besides the 8 loads) and was bound by the shared-memory queue.  Since p is rebuilt from
// (r, p) after the first barrier, phase B overwrites the one copy of the pair that phase A
// read.
// A chunk of 1792 to 3583 groups keeps the pairs alone in shared memory; x and A p, which an iteration
// reads once and writes once by the thread that owns them, go through L2 (28 us an iteration for 389,000
// rows on 16 CTAs; the path below takes 95 for 278,000).  It is what lets small clusters and single CTAs
// take systems larger than those they are sized for.  Otherwise (the root, or more rows than fit)
// the vectors live in global memory and the neighbour table is read row by row.
constexpr int kCgcBlock = 1024;
constexpr int kCgWarps = kCgcBlock / 32;
constexpr int kCgGroups = 1792;                   // local groups of a CTA's arrays; the last one is the zero group
                                                  //   (absent neighbours: (0, 0), x = 0)
constexpr int kCgPairGroups = 2 * kCgGroups;      // the same of the pairs alone
constexpr int kCgRowGroups = kCgcBlock / 8;       // at most this many groups: a thread per row
constexpr int kCgDescWords = 14;                  // 27 neighbour groups, two per word
constexpr size_t kCgSmemBytes = (size_t)kCgGroups * 8 * (sizeof(float2) + 2 * sizeof(float));   // (r, p), x, A p
constexpr int kCgMaxRefine = 4;

// Workspace pointers of the CG; a multi-cloud launch moves them to the CTA's cloud (a
// copy in registers: the launch parameters below stay where the launch put them).
struct CgcVec {
    const Counters* c;
    Counters* cw;
    const int* neigh;
    const int* parent;
    const int* first_child;
    unsigned* desc;     // [kCgDescWords][dstride]: packed neighbour groups of CTAs with more than one group a thread
    const float* stencil;
    const float* b;
    float* x;
    float2* rp;         // global-memory path: (r_k, p_{k-1}) per row
    float* ap;          //   and A p
    float *xs, *aps;    // x and A p of chunks whose pairs alone fit shared memory: [8][dstride], sibling-major
    __device__ void rebase() { PSR_CLOUD(c, cw, neigh, parent, first_child, desc, stencil, b, x, rp, ap, xs, aps); }
};

// a workspace pointer of cloud 0 moved to cloud k (null stays null)
template <class T>
__device__ __forceinline__ T* at_cloud(T* p, int k) {
    return p ? (T*)((const char*)p + (unsigned long long)k * kCloudStride) : p;
}

struct CgcArgs {
    CgcVec v;
    int depth;
    int first;          // depth of cluster / CTA 0; unit u solves depth first - u
    size_t stride;
    size_t dstride;     // sibling groups of the workspace
    float tol2;
    int max_iter;
    int res_period;     // > 0: true residual every res_period iterations; 0: only at
                        // convergence; < 0: never (the recursive residual alone)
    int clusters;       // units solved by a whole cluster; the CTAs of the clusters behind them
                        // solve a coarser depth each
};

// The resident path holds a depth when the (r, p) pairs of its cluster's chunk of groups fit a CTA's
// shared memory (the last group is the zero group); the root never does.
__device__ __forceinline__ int cg_chunk_groups(int m, int nblk) { return max(1, ((m >> 3) + nblk - 1) / nblk); }
__device__ __forceinline__ bool cg_fits_resident(int d, int m, int nblk) {
    return d >= 1 && cg_chunk_groups(m, nblk) < kCgPairGroups;
}

// A sum in fixed point: m * 2^(e - 183), |m| < 2^62.  k_cg_grid adds the lanes of a warp as 57-bit
// integers aligned to the largest of them, in three integer warp reductions (what falls off a
// smaller term is below 2^-57 of the largest); warps and CTAs the same way.
struct alignas(16) CgSum {
    long long m;
    long long e;      // >= 512: not a number
};

// A sum in digits: (d[0] 2^57 + d[1] 2^38 + d[2] 2^19 + d[3]) 2^(19 (b - 3) - 127).  The digits of the
// bins below the highest, b, are kept apart, so that a sum of a higher bin can drop the lowest ones and
// nothing else.  A digit of a group is below 2^19 and a half: those of up to 4095 groups fit 32 bits.
struct CgDig {
    int4 d;
    int b;            // -1: nothing added yet; above 13: not a number
};

struct CgcShared {
    int4 warp[kCgWarps];           // the warps' sums
    int warp_b[kCgWarps];
    int4 slot[2][16];              // the cluster's CTA sums, written by the CTAs
    int slot_b[2][16];
    unsigned long long bar[2];     // their arrivals
    CgSum rr;           // r.r of the recursive residual
    CgSum pap;
    double floor2;      // (2^-20 ||b||)^2: what the true residual of an FP32 solution can reach
    double rr_true;     // r.r of the last true residual (-1: none yet)
    float rrf;          // r.r rounded to float
    float alpha, beta;
    int go;             // the iteration continues
    int check;          // the true residual is due
    int replace;        // the true residual replaces r (a refinement restart)
    int checks;         // true-residual evaluations
    int restarts;       // refinement restarts
    int until_check;    // iterations until the next periodic true residual
    float st[27];
};
static_assert(kCgWarps == 32, "one lane per warp sum");
static_assert(kCgSmemBytes + sizeof(CgcShared) <= 227 * 1024, "shared memory of one CTA");
static_assert(kCgPairGroups <= 4096, "12 bits of a packed neighbour group, 4 of its CTA");

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// the lanes' sum of m, each |m| <= 2^57, in every lane: three 21-bit pieces, whose sums fit 32 bits
__device__ __forceinline__ long long cgs_add_lanes(long long m) {
    const int p0 = (int)(m & 0x1fffff), p1 = (int)((m >> 21) & 0x1fffff), p2 = (int)(m >> 42);
    const int s0 = __reduce_add_sync(0xffffffffu, p0), s1 = __reduce_add_sync(0xffffffffu, p1),
              s2 = __reduce_add_sync(0xffffffffu, p2);
    return ((long long)s2 << 42) + ((long long)s1 << 21) + (long long)s0;
}

// the sum of the lanes' fixed-point values, in every lane
__device__ __forceinline__ CgSum cgs_warp_sum(CgSum v) {
    const long long mag = v.m < 0 ? -v.m : v.m;
    const int len = 64 - __clzll(mag);   // bits of |m|
    const int top = __reduce_max_sync(0xffffffffu, v.m != 0 ? (int)v.e + len : 0);
    // the largest value takes 57 bits
    const int e = top - 57, d = e - (int)v.e;
    long long m = 0;
    if (d <= 0) m = d > -64 ? v.m << -d : 0;           // to the left: only values of fewer than 57 bits
    else if (d < 63) m = ((v.m >> (d - 1)) + 1) >> 1;  // to the right, to nearest
    return CgSum{cgs_add_lanes(v.m != 0 ? m : 0), e};
}

// 2^x for |x| <= 126
__device__ __forceinline__ float pow2f_exact(int x) { return __int_as_float((127 + x) << 23); }

// The sum of the lanes' float pairs in three pieces (x + y 2^-21 + z 2^-42) 2^(w - 147), in every
// lane.  A piece of a float against 1.5 * 2^23 units of the piece: the addition rounds to the unit
// and leaves the integer in the low bits; what is left over is exact.
__device__ __forceinline__ int4 cgs_warp_sum(FF v) {
    int top = __reduce_max_sync(0xffffffffu, max((__float_as_int(v.hi) >> 23) & 255, (__float_as_int(v.lo) >> 23) & 255));
    if (top == 255) return make_int4(0, 0, 0, 1024);   // infinite or not a number
    int e = top;
    if (top > 200 || top < 64) {   // uniform: keep the units of the pieces normal numbers
        const int sh = top > 200 ? -64 : 64;
        v.hi *= pow2f_exact(sh);
        v.lo *= pow2f_exact(sh);
        top += sh;
    }
    const int c0 = ((top - 20 + 23) << 23) | 0x400000, c1 = c0 - (21 << 23), c2 = c1 - (21 << 23);
    auto take = [](float& r, int c) -> int {
        const float f = __int_as_float(c);
        const float t = __fadd_rn(r, f);
        r = __fsub_rn(r, __fsub_rn(t, f));
        return __float_as_int(t) - c;
    };
    int i0 = take(v.hi, c0), i1 = take(v.hi, c1), i2 = take(v.hi, c2);
    i1 += take(v.lo, c1);
    i2 += take(v.lo, c2);
    i0 = __reduce_add_sync(0xffffffffu, i0);
    i1 = __reduce_add_sync(0xffffffffu, i1);
    i2 = __reduce_add_sync(0xffffffffu, i2);
    return make_int4(i0, i1, i2, e);
}
// the pieces as one number, |m| <= 2^62
__device__ __forceinline__ CgSum cgs_join(int4 q) {
    if (q.w >= 512) return CgSum{1ll << 56, 1024};
    return CgSum{((long long)q.x << 35) + ((long long)q.y << 14) + ((q.z + 64) >> 7), (long long)q.w + 1};
}

__device__ __forceinline__ float cgs_float(const CgSum& s) {
    if (s.e >= 512) return __int_as_float(0x7fc00000);
    // in two steps: the exponent may leave the float's range half way
    const int x = max((int)s.e - 183, -250), h = x / 2;
    return (__ll2float_rn(s.m) * pow2f_exact(h)) * pow2f_exact(x - h);
}
__device__ __forceinline__ double cgs_double(const CgSum& s) {
    if (s.e >= 512) return (double)__int_as_float(0x7fc00000);
    return (double)s.m * __hiloint2double((1023 + max((int)s.e - 183, -1000)) << 20, 0);   // a power of two: exact
}

// The digits of the sum of kLanes lanes' float pairs, kTerms a lane, in every lane: each pair is rounded
// to the lowest unit of the four bins, which start at the largest pair's.  What a pair leaves in the bins
// from any unit upwards is the pair rounded to that unit (to even), whatever bin its digits start at.
template <int kTerms, class Sum, class Max, class Any>
__device__ __forceinline__ CgDig cgd_of(FF (&v)[kTerms], int lanes, Sum sum, Max max_of, Any any) {
    int E = 0;
#pragma unroll
    for (int q = 0; q < kTerms; ++q) E = max(E, __float_as_int(v[q].hi) & 0x7f800000);
    E = max_of(E) >> 23;   // the largest is below 2^(E - 126)
    if (E == 255) return CgDig{make_int4(1, 0, 0, 0), 31};   // infinite or not a number
    const int b = E / 19;
    int at = b;
    if (b < 2 || b > 12) {   // keep the units of the digits normal numbers
        const int up = b < 2 ? 2 : -1;
#pragma unroll
        for (int q = 0; q < kTerms; ++q) {
            v[q].hi *= pow2f_exact(19 * up);
            v[q].lo *= pow2f_exact(19 * up);
        }
        at += up;
    }
    // a digit against 1.5 * 2^23 of its units: the addition rounds to the unit and leaves the integer in
    // the low bits (less those of the constant, taken off the sum); what is left over is exact.  lo is at
    // most 2^-24 hi and has none in the first bin.
    const int c0 = ((19 * at + 23) << 23) | 0x400000, c1 = c0 - (19 << 23), c2 = c1 - (19 << 23), c3 = c2 - (19 << 23);
    auto take = [](float& r, int c) -> int {
        const float f = __int_as_float(c);
        const float t = __fadd_rn(r, f);
        r = __fsub_rn(r, __fsub_rn(t, f));
        return __float_as_int(t);
    };
    unsigned d0 = 0, d1 = 0, d2 = 0, d3 = 0;   // modulo 2^32
    unsigned n = 0;
#pragma unroll
    for (int q = 0; q < kTerms; ++q) {
        if (kTerms > 1 && !any(v[q].hi != 0.0f)) continue;
        n += (unsigned)lanes;
        d0 += take(v[q].hi, c0);
        d1 += take(v[q].hi, c1);
        d2 += take(v[q].hi, c2);
        d3 += take(v[q].hi, c3);
        d1 += take(v[q].lo, c1);
        d2 += take(v[q].lo, c2);
        d3 += take(v[q].lo, c3);
    }
    return CgDig{make_int4((int)(sum(d0) - n * c0), (int)(sum(d1) - 2 * n * c1), (int)(sum(d2) - 2 * n * c2),
                           (int)(sum(d3) - 2 * n * c3)), b};
}
// of a warp's pairs
template <int kTerms>
__device__ __forceinline__ CgDig cgd_warp_sum(FF (&v)[kTerms]) {
    bool some = false;
#pragma unroll
    for (int q = 0; q < kTerms; ++q) some |= v[q].hi != 0.0f;   // not a number differs from 0 too
    if (!__any_sync(0xffffffffu, some)) return CgDig{make_int4(0, 0, 0, 0), -1};
    return cgd_of(v, 32, [](unsigned d) { return __reduce_add_sync(0xffffffffu, d); },
                  [](int e) { return __reduce_max_sync(0xffffffffu, e); },
                  [](bool some) { return __any_sync(0xffffffffu, some) != 0; });
}
// of one lane's pair
__device__ __forceinline__ CgDig cgd_of(FF v) {
    FF t[1] = {v};
    return cgd_of(t, 1, [](unsigned d) { return d; }, [](int e) { return e; }, [](bool some) { return some; });
}
// the digits of a sum whose highest bin is s bins higher (the lowest s are dropped)
template <class D>
__device__ __forceinline__ void cgd_drop(D& d, int s) {
    if (s & 1) { d.w = d.z; d.z = d.y; d.y = d.x; d.x = 0; }
    if (s & 2) { d.w = d.y; d.z = d.x; d.y = d.x = 0; }
    if (s > 3) d.x = d.y = d.z = d.w = 0;
}
__device__ __forceinline__ void cgd_add(CgDig& a, FF v) {
    CgDig t = cgd_of(v);
    const int b = max(a.b, t.b);
    cgd_drop(a.d, b - a.b);
    cgd_drop(t.d, b - t.b);
    a = CgDig{make_int4(a.d.x + t.d.x, a.d.y + t.d.y, a.d.z + t.d.z, a.d.w + t.d.w), b};
}
// the lanes' sum, in every lane
__device__ __forceinline__ CgDig cgd_warp_sum(CgDig v) {
    const int b = __reduce_max_sync(0xffffffffu, v.b);
    cgd_drop(v.d, b - v.b);
    return CgDig{make_int4(__reduce_add_sync(0xffffffffu, v.d.x), __reduce_add_sync(0xffffffffu, v.d.y),
                           __reduce_add_sync(0xffffffffu, v.d.z), __reduce_add_sync(0xffffffffu, v.d.w)), b};
}
// the sum of up to 16 lanes' digits as one number, in every lane (digits of all groups: below 2^38)
template <class D>
__device__ __forceinline__ CgSum cgd_total(D d, int lane_b) {
    const int b = __reduce_max_sync(0xffffffffu, lane_b);
    cgd_drop(d, b - lane_b);
    auto add = [](long long m) -> long long {   // |sum| < 2^57
        const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)m & 0x3ffffffu);
        return ((long long)__reduce_add_sync(0xffffffffu, (int)(m >> 26)) << 26) + (long long)lo;
    };
    const long long hi = add(((long long)d.x << 19) + (long long)d.y), lo = add(((long long)d.z << 19) + (long long)d.w);
    if (b > 13) return CgSum{1ll << 56, 1024};
    const int k = min(38, 61 - (64 - __clzll(hi < 0 ? -hi : hi)));
    return CgSum{(hi << k) + (lo >> (38 - k)), 19 * (b - 3) - 127 + 38 - k + 183};
}

// the sum of a sibling group's 8 terms, in one order: ((0 + 1) + (2 + 3)) + ((4 + 5) + (6 + 7))
template <class Term>
__device__ __forceinline__ FF cg_group_sum(Term term) {
    FF h[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const FF t0 = term(4 * q), t1 = term(4 * q + 1);
        const FF a = ff_add(t0, t1);
        const FF t2 = term(4 * q + 2), t3 = term(4 * q + 3);
        h[q] = ff_add(a, ff_add(t2, t3));
    }
    return ff_add(h[0], h[1]);
}

// a shared-memory address of this CTA in the window of cluster CTA `rank`
__device__ __forceinline__ unsigned cg_map(unsigned sa, unsigned rank) {
    unsigned ra;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(sa), "r"(rank));
    return ra;
}
__device__ __forceinline__ void cgc_barriers_init(CgcShared& sh) {
    if (threadIdx.x < 2) {
        const unsigned b = (unsigned)__cvta_generic_to_shared(&sh.bar[threadIdx.x]);
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// Sum of every thread's `v` over the cluster.  Thread 0 hands the sum to `post`, which sets
// the shared scalars the next step reads; every thread sees them when this returns.
// Identical in every CTA.  It is also the cluster's barrier: when the CTA's threads have met, a
// lane of warp 0 per peer sends the CTA's sum into the peer's slot (st.async, counted by the
// peer's mbarrier), and nobody goes on before its own mbarrier has counted every CTA's.  That
// orders the threads' earlier reads of their peers; with kPublish their earlier writes too (a
// fence before the sends), so that peers may read them next.  Measured in a loop of reductions
// over 16 CTAs of 1024 threads: 836 cycles, 1165 with the fence, against 1442 for
// barrier.cluster and a remote read of the sums and 1574 for remote stores and
// mbarrier arrivals with release.  `n` counts the reductions: they alternate between two
// slots and barriers, and a CTA reuses a slot only after every peer has sent to the other one.
// The wait is bounded; `error` is then flagged and the solve stops.
template <bool kPublish, class Terms, class Post>
__device__ __forceinline__ void cgc_allreduce(unsigned nb, unsigned me, CgcShared& sh, unsigned& n, Terms& terms,
                                              unsigned* error, Post post) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    CgDig v = cgd_warp_sum(terms);
    if (lane == 0) {
        sh.warp[warp] = v.d;
        sh.warp_b[warp] = v.b;
    }
    __syncthreads();
    if (warp == 0) {
        v = cgd_warp_sum(CgDig{sh.warp[lane], sh.warp_b[lane]});
        bool late = false;
        if (nb > 1) {
            const int buf = (int)(n & 1u);
            const unsigned parity = (n >> 1) & 1u;
            const unsigned bar = (unsigned)__cvta_generic_to_shared(&sh.bar[buf]);
            if (kPublish) asm volatile("fence.acq_rel.cluster;" ::: "memory");
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(nb * 20u) : "memory");
            __syncwarp();
            if ((unsigned)lane < nb) {
                const unsigned peer_bar = cg_map(bar, (unsigned)lane);
                const long long d01 = (long long)(unsigned)v.d.x | (long long)v.d.y << 32;
                const long long d23 = (long long)(unsigned)v.d.z | (long long)v.d.w << 32;
                asm volatile(
                    "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(
                        cg_map((unsigned)__cvta_generic_to_shared(&sh.slot[buf][me]), (unsigned)lane)),
                    "l"(d01), "l"(d23), "r"(peer_bar)
                    : "memory");
                asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(
                                 cg_map((unsigned)__cvta_generic_to_shared(&sh.slot_b[buf][me]), (unsigned)lane)),
                             "r"(v.b), "r"(peer_bar)
                             : "memory");
            }
            unsigned done = 0;
            for (int spin = 0; spin < kSpinLimit && !done; ++spin)
                asm volatile(
                    "{\n.reg .pred p;\n"
                    "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                    "selp.u32 %0, 1, 0, p;\n}"
                    : "=r"(done)
                    : "r"(bar), "r"(parity)
                    : "memory");
            late = !done;
            v = CgDig{make_int4(0, 0, 0, 0), -1};
            if ((unsigned)lane < nb) v = CgDig{sh.slot[buf][lane], sh.slot_b[buf][lane]};
        } else if (lane > 0) {
            v = CgDig{make_int4(0, 0, 0, 0), -1};
        }
        const CgSum t = cgd_total(v.d, v.b);
        if (lane == 0) {
            post(t);
            if (late) {
                atomicOr(error, kErrSpinTimeout);
                sh.go = sh.check = sh.replace = 0;
            }
        }
    }
    ++n;
    __syncthreads();
}

// After the r.r reduction of an iteration (thread 0): beta, the continue flag and whether
// the true residual is due.  `it` is the iteration just completed.
// The step scalars are quotients of the sums rounded to float and divided in FP32 (within 1.5 ulp of
// the exact quotient rounded to float): an FP64 division on the one thread that finishes the sums
// would sit on every iteration's critical path, and GB300 divides in FP64 slowly.
template <class St>
__device__ __forceinline__ void cgc_alpha(St& sh, const CgSum& t) {
    sh.pap = t;
    sh.alpha = t.m != 0 ? __fdiv_rn(sh.rrf, cgs_float(t)) : 0.0f;
}
template <class St, class Ar>
__device__ __forceinline__ void cgc_after_rr(St& sh, const Ar& a, const CgSum& t, int it) {
    const float w = cgs_float(t);
    sh.beta = sh.rr.m != 0 ? __fdiv_rn(w, sh.rrf) : 0.0f;
    sh.rr = t;
    sh.rrf = w;
    const bool conv = !(w > a.tol2);
    const bool more = sh.pap.m != 0 && it + 1 <= a.max_iter;
    sh.go = !conv && more;
    const bool due = --sh.until_check == 0;   // every res_period iterations
    if (due) sh.until_check = a.res_period;
    sh.check = a.res_period >= 0 && sh.pap.m != 0 && (conv || (due && more));
}

// After the true-residual reduction (thread 0).  The CG restarts from the true residual
// (beta = 0: one cycle of iterative refinement) when that residual is above both the
// tolerance and the floor an FP32 solution can reach, and either the recursive residual
// has converged or has drifted more than 2x (in norm) below the true one; at most
// kCgMaxRefine restarts, each one reducing the true r.r at least fourfold.  `it` is the
// next iteration's number.
template <class St, class Ar>
__device__ __forceinline__ void cgc_after_true(St& sh, const Ar& a, const CgSum& t, int it) {
    ++sh.checks;
    const double w = cgs_double(t), rr = cgs_double(sh.rr);
    const double target = fmax((double)a.tol2, sh.floor2);
    const bool drift = w > 4.0 * fmax(rr, sh.floor2);
    const bool falling = sh.rr_true < 0.0 || w < 0.25 * sh.rr_true;
    sh.replace = w > target && (!sh.go || drift) && sh.restarts < kCgMaxRefine && it <= a.max_iter && falling;
    if (sh.replace) {
        ++sh.restarts;
        sh.beta = 0.0f;
        sh.go = 1;
        sh.rr = t;
        sh.rrf = cgs_float(t);
    }
    sh.rr_true = w;
}

// Start of a solve (thread 0): r0 = b, so r.r is also ||b||^2.
template <class St, class Ar>
__device__ __forceinline__ void cgc_start(St& sh, const Ar& a, const CgSum& t) {
    sh.rr = t;
    sh.rrf = cgs_float(t);
    sh.beta = 0.0f;
    sh.go = (sh.rrf > a.tol2) && a.max_iter >= 1;
    sh.until_check = a.res_period > 0 ? a.res_period : 0;   // 0: never counts down to 0 again
    sh.floor2 = cgs_double(t) * 0x1p-40;
    sh.rr_true = -1.0;
    sh.checks = 0;
    sh.restarts = 0;
    sh.replace = 0;
}

// Per-depth results of a finished solve (thread 0 of cluster CTA 0).
// The iteration count goes out here and not per iteration: a global store in flight would hold
// up the release at every reduction.
__device__ __forceinline__ void cgc_report(const CgcVec& v, int d, const CgcShared& sh, int iterations) {
    v.cw->cg_iters[d] = iterations;
    v.cw->cg_rr[d] = cgs_double(sh.rr);
    v.cw->cg_rr_true[d] = sh.rr_true;
    v.cw->cg_checks[d] = sh.checks;
    v.cw->cg_restarts[d] = sh.restarts;
}

struct CgUnit {
    int d, row0, row1;
    unsigned me, nb;    // this CTA among those that solve the unit
    unsigned rank0;     // cluster rank of the first of them
};

__device__ __forceinline__ float2 cg_ld2(unsigned a) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float cg_ld1(unsigned a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

// The stencil entry of offset slot k depends only on how many axes the offset is non-zero on
// (0: centre, 1: face, 2: edge, 3: corner): four values per depth (checked at creation).
__host__ __device__ constexpr int cg_class(int k) {
    return (k / 9 != 1) + ((k / 3) % 3 != 1) + (k % 3 != 1);
}
// block position 16 bx + 4 by + bz: the neighbour of the parent it lies in, and its sibling there
__host__ __device__ constexpr int cg_pos_axis(int b) { return b == 0 ? 0 : (b == 3 ? 2 : 1); }
__host__ __device__ constexpr int cg_pos_group(int p) {
    return 9 * cg_pos_axis(p >> 4) + 3 * cg_pos_axis((p >> 2) & 3) + cg_pos_axis(p & 3);
}
__host__ __device__ constexpr int cg_pos_sib(int p) {
    return 4 * (((p >> 4) + 1) & 1) + 2 * ((((p >> 2) & 3) + 1) & 1) + (((p & 3) + 1) & 1);
}

// The sibling group on slot n of group G's parent (global group number), or -1.
__device__ __forceinline__ int cg_neighbour_group(const CgcVec& v, size_t stride, int pa, int n) {
    const int q = v.neigh[(size_t)n * stride + pa];
    const int f = v.first_child[q >= 0 ? q : 0];
    return (q >= 0 && f >= 1) ? (f - 1) >> 3 : -1;
}

// How a CTA's rows are dealt to its threads.
enum CgMode {
    kCgRows,     // a thread per row (thread t: sibling t / kCgRowGroups of group t % kCgRowGroups)
    kCgOne,      // a thread per group, the packed neighbour groups in shared memory
    kCgMany,     // groups in turn, their neighbour groups packed in global memory
    kCgPairs     // the same with x and A p in global memory too
};
// groups of the sibling-major arrays of a mode (the last one is the zero group)
__host__ __device__ constexpr int cg_pitch(int mode) {
    return mode == kCgPairs  ? kCgPairGroups
           : mode == kCgMany ? kCgGroups
           : mode == kCgOne  ? kCgcBlock + 8
                             : kCgRowGroups + 8;
}
static_assert((size_t)cg_pitch(kCgPairs) * 8 * sizeof(float2) <= kCgSmemBytes, "kCgPairs");
static_assert((size_t)cg_pitch(kCgOne) * 8 * 16 + (size_t)kCgDescWords * kCgcBlock * 4 <= kCgSmemBytes, "kCgOne");

// The operator of one group: adds st * val(position) to every row the position neighbours, in
// neighbour order per row.  `val(n, off)` gives the value of neighbour group n's element at
// element offset `off` of the sibling-major arrays.
template <int kPitch, class Val, class Add>
__device__ __forceinline__ void cg_apply_group(Val val, Add add) {
#pragma unroll
    for (int p = 0; p < 64; ++p) {
        const auto x = val(cg_pos_group(p), cg_pos_sib(p) * kPitch);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const int ox = (p >> 4) - (s >> 2), oy = ((p >> 2) & 3) - ((s >> 1) & 1), oz = (p & 3) - (s & 1);
            if (ox >= 0 && ox < 3 && oy >= 0 && oy < 3 && oz >= 0 && oz < 3)
                add(s, cg_class(9 * ox + 3 * oy + oz), x);
        }
    }
}

// Resident path.  CTA k of the cluster owns the unit's groups [k * chunk, (k + 1) * chunk).
template <int kMode>
__device__ __forceinline__ void cgc_resident(cg::cluster_group& cl, CgcShared& sh, const CgcArgs& a,
                                             const CgcVec& v, const CgUnit& u, int chunk, float4* dyn) {
    constexpr int GP = cg_pitch(kMode);
    float2* rp = reinterpret_cast<float2*>(dyn);
    float* sx = reinterpret_cast<float*>(rp + 8 * GP);
    float* sap = sx + 8 * GP;
    constexpr int kDescPitch = kMode == kCgOne ? kCgcBlock : kCgRowGroups;
    unsigned* sdesc = reinterpret_cast<unsigned*>(sap + 8 * GP);   // [kCgDescWords][kDescPitch]
    FF* sterm = reinterpret_cast<FF*>(sdesc + kCgDescWords * kDescPitch);   // kCgRows: [8][kCgRowGroups]
    const unsigned me = u.me, nb = u.nb;
    unsigned* err = &v.cw->error;
    const int tid = threadIdx.x;
    const int ngroups = (u.row1 - u.row0) >> 3;
    const int g0 = (int)me * chunk;                           // the CTA's first group, in the unit
    const int ng = max(0, min(chunk, ngroups - g0));
    const int gbase = ((u.row0 - 1) >> 3) + g0;               // global number of local group 0
    const unsigned rp_sa = (unsigned)__cvta_generic_to_shared(rp);
    const unsigned x_sa = (unsigned)__cvta_generic_to_shared(sx);
    const float w[4] = {sh.st[13], sh.st[14], sh.st[17], sh.st[26]};   // centre, face, edge, corner
    // q / chunk = umulhi(q, ceil(2^32 / chunk)): exact for q < 16 * chunk, chunk <= 2^12
    const unsigned magic = (unsigned)((0x100000000ull + (unsigned)chunk - 1) / (unsigned)chunk);
    // rank << 12 | local group of global group G (absent or outside the unit: the zero group)
    auto locate = [&](int G) -> unsigned {
        const unsigned q = (unsigned)(G - ((u.row0 - 1) >> 3));
        if (G < 0 || q >= (unsigned)ngroups) return ((u.rank0 + me) << 12) | (unsigned)(GP - 1);
        const unsigned own = chunk > 1 ? __umulhi(q, magic) : q;   // q / chunk
        return ((u.rank0 + own) << 12) | (q - own * (unsigned)chunk);
    };
    auto base_of = [&](unsigned d, unsigned sa, unsigned elem) { return cg_map(sa + (d & 4095u) * elem, d >> 12); };

    // kCgRows: this thread's row and the mapped addresses of its 27 neighbours' pairs
    const int rs = tid / kCgRowGroups, rg = tid % kCgRowGroups;
    const bool row_on = kMode == kCgRows && rg < ng;
    // neighbour (kx, ky, kz) of sibling s: its neighbour group slot and sibling there
    auto slot_of = [](int s, int kx, int ky, int kz, int& n, int& sib) {
        const int bx = (s >> 2) + kx, by = ((s >> 1) & 1) + ky, bz = (s & 1) + kz;
        n = 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1);   // cg_pos_axis
        sib = 4 * ((bx + 1) & 1) + 2 * ((by + 1) & 1) + ((bz + 1) & 1);
    };
    // The packed neighbour groups (parent, its neighbour row, first children), in loops of a few
    // steps: long straight-line code that runs once comes from L2
    auto find_word = [&](int g, int pa, int j) {
        const unsigned lo = locate(cg_neighbour_group(v, a.stride, pa, 2 * j));
        const unsigned hi = (2 * j + 1 < 27) ? locate(cg_neighbour_group(v, a.stride, pa, 2 * j + 1)) : 0u;
        const unsigned q = lo | (hi << 16);
        if (kMode >= kCgMany) v.desc[(size_t)j * a.dstride + gbase + g] = q;
        else sdesc[j * kDescPitch + g] = q;
    };
    if (kMode == kCgRows) {   // a word per thread and turn
#pragma unroll 2
        for (int i = tid; i < kCgDescWords * kCgRowGroups; i += kCgcBlock) {
            const int j = i / kCgRowGroups, g = i % kCgRowGroups;
            if (g < ng) find_word(g, v.parent[1 + 8 * (gbase + g)], j);
        }
    } else {
        for (int g = tid; g < ng; g += kCgcBlock) {
            const int pa = v.parent[1 + 8 * (gbase + g)];
#pragma unroll 7
            for (int j = 0; j < kCgDescWords; ++j) find_word(g, pa, j);
        }
    }
    // neighbour group slot n of group g (packed)
    auto desc_of = [&](int g, int n) -> unsigned {
        const unsigned q = kMode >= kCgMany ? v.desc[(size_t)(n >> 1) * a.dstride + gbase + g]
                                            : sdesc[(n >> 1) * kDescPitch + g];
        return (n & 1) ? q >> 16 : q & 0xffffu;
    };
    // kCgRows: the mapped addresses of the row's 27 neighbours' pairs
    unsigned adr[kMode == kCgRows ? 27 : 1];
    if (kMode == kCgRows) {
        __syncthreads();
        if (row_on) {
#pragma unroll
            for (int k = 0; k < 27; ++k) {
                int n, sib;
                slot_of(rs, k / 9, (k / 3) % 3, k % 3, n, sib);
                adr[kMode == kCgRows ? k : 0] = base_of(desc_of(rg, n), rp_sa, 8u) + (unsigned)(sib * GP * 8);
            }
        }
    }
    // x and A p of sibling s of local group g
    const unsigned dpitch = (unsigned)a.dstride;
    auto x_at = [&](int s, int g) -> float& {
        return kMode == kCgPairs ? v.xs[(unsigned)s * dpitch + (unsigned)(gbase + g)] : sx[s * GP + g];
    };
    auto ap_at = [&](int s, int g) -> float& {
        return kMode == kCgPairs ? v.aps[(unsigned)s * dpitch + (unsigned)(gbase + g)] : sap[s * GP + g];
    };
    if (tid < 8) {
        rp[tid * GP + GP - 1] = make_float2(0.0f, 0.0f);
        if (kMode == kCgPairs) v.xs[(unsigned)tid * dpitch + dpitch - 1u] = 0.0f;   // the same in every CTA
        else sx[tid * GP + GP - 1] = 0.0f;
    }
    // A thread's groups' sums of this step's terms.
    constexpr int kTerms = kMode == kCgMany ? 2 : 1;
    std::conditional_t<kMode == kCgPairs, CgDig, FF[kTerms]> acc;
    // body(group) for the thread's groups, its sum to acc
    auto for_groups = [&](auto body) {
        if constexpr (kMode == kCgPairs) {
            acc = CgDig{make_int4(0, 0, 0, 0), -1};
#pragma unroll 1
            for (int g = tid; g < ng; g += kCgcBlock) cgd_add(acc, body(g));
        } else {
            acc[0] = acc[kTerms - 1] = ff_zero();
            if constexpr (kTerms == 1) {
                if (tid < ng) acc[0] = body(tid);
            } else {
#pragma unroll 1
                for (int g = tid; g < ng; g += kCgcBlock) {   // twice at most; one copy of the body
                    const FF t = body(g);
                    if (g == tid) acc[0] = t;
                    else acc[kTerms - 1] = t;
                }
            }
        }
    };
    // The sums of term(sibling, group) over the groups.  Where a row has a thread of its own, the terms of a
    // group meet in shared memory and one thread adds them.
    auto sum_rows = [&](auto term) {
        if constexpr (kMode == kCgRows) {
            sterm[tid] = row_on ? term(rs, rg) : ff_zero();
            __syncthreads();
            acc[0] = ff_zero();
            if (tid < kCgRowGroups) acc[0] = cg_group_sum([&](int s) { return sterm[s * kCgRowGroups + tid]; });
        } else {
            for_groups([&](int g) { return cg_group_sum([&](int s) { return term(s, g); }); });
        }
    };
    // r0 = b, p_{-1} = 0, x0 = 0 (rows in order: coalesced)
    const int mlo = 1 + 8 * gbase;
    for (int l = tid; l < 8 * ng; l += kCgcBlock) {
        rp[(l & 7) * GP + (l >> 3)] = make_float2(v.b[mlo + l], 0.0f);
        if (kMode != kCgPairs) sx[(l & 7) * GP + (l >> 3)] = 0.0f;
    }
    __syncthreads();
    sum_rows([&](int s, int g) {
        if (kMode == kCgPairs) x_at(s, g) = 0.0f;
        const float r = rp[s * GP + g].x;
        return ff_prod(r, r);
    });
    unsigned nred = 0;
    cgc_allreduce<true>(nb, me, sh, nred, acc, err, [&](const CgSum& t) { cgc_start(sh, a, t); });
    bool ran = false;
    int it = 1;
    while (sh.go) {
        const float beta = sh.beta;
        // (A) A p_k from the neighbours' (r_k, p_{k-1}), p.Ap
        if (kMode == kCgRows) {
            sum_rows([&](int s, int g) {
                float y = 0.0f;
#pragma unroll
                for (int k = 0; k < 27; ++k) {
                    const float2 q = cg_ld2(adr[kMode == kCgRows ? k : 0]);
                    y = fmaf(w[cg_class(k)], fmaf(beta, q.y, q.x), y);
                }
                const float2 own = rp[s * GP + g];
                sap[s * GP + g] = y;
                return ff_prod(fmaf(beta, own.y, own.x), y);
            });
        } else {
            for_groups([&](int g) {
                float y[8];
#pragma unroll
                for (int s = 0; s < 8; ++s) y[s] = 0.0f;
                cg_apply_group<GP>(
                    [&](int n, int off) {
                        const float2 q = cg_ld2(base_of(desc_of(g, n), rp_sa, 8u) + (unsigned)(off * 8));
                        return fmaf(beta, q.y, q.x);
                    },
                    [&](int s, int c, float p) { y[s] = fmaf(w[c], p, y[s]); });
                return cg_group_sum([&](int s) {
                    const float2 own = rp[s * GP + g];
                    ap_at(s, g) = y[s];
                    return ff_prod(fmaf(beta, own.y, own.x), y[s]);
                });
            });
        }
        cgc_allreduce<false>(nb, me, sh, nred, acc, err, [&](const CgSum& t) { cgc_alpha(sh, t); });
        const float alpha = sh.alpha;
        // (B) x and r, r.r; every CTA has read the pairs (the barrier of the last reduction)
        auto update = [&](int s, int g, float xo, float y) -> FF {
            const float2 own = rp[s * GP + g];
            const float pi = fmaf(beta, own.y, own.x);
            x_at(s, g) = fmaf(alpha, pi, xo);
            const float ri = fmaf(-alpha, y, own.x);
            rp[s * GP + g] = make_float2(ri, pi);
            return ff_prod(ri, ri);
        };
        if (kMode == kCgPairs) {
            for_groups([&](int g) {
                float xo[8], y[8];   // in flight together
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    xo[s] = x_at(s, g);
                    y[s] = ap_at(s, g);
                }
                return cg_group_sum([&](int s) { return update(s, g, xo[s], y[s]); });
            });
        } else {
            sum_rows([&](int s, int g) { return update(s, g, sx[s * GP + g], sap[s * GP + g]); });
        }
        cgc_allreduce<true>(nb, me, sh, nred, acc, err, [&](const CgSum& t) { cgc_after_rr(sh, a, t, it); });
        ran = true;
        ++it;
        if (sh.check) {
            // (C) true residual b - A x of the current x from the neighbours' x (the barrier
            // of the last reduction published every CTA's x), with exact products and
            // float-pair sums; staged in the A p array, which holds nothing live here
            if (kMode == kCgPairs && nb > 1) cl.sync();   // x is in global memory
            auto x_of = [&](unsigned d, int sib) -> float {   // x of sibling sib of a packed group
                if (kMode != kCgPairs) return cg_ld1(base_of(d, x_sa, 4u) + (unsigned)(sib * GP * 4));
                const unsigned local = d & 4095u, G = (unsigned)(gbase - g0) + ((d >> 12) - u.rank0) * (unsigned)chunk + local;
                return __ldcg(v.xs + (unsigned)sib * dpitch + (local == (unsigned)(GP - 1) ? dpitch - 1u : G));
            };
            // the entry of an offset that moves on `axes` of x and y, and by kz - 1 on z
            auto w_of = [&](int axes, int kz) {
                return kz == 1 ? (axes == 0 ? w[0] : axes == 1 ? w[1] : w[2]) : (axes == 0 ? w[1] : axes == 1 ? w[2] : w[3]);
            };
            auto residual = [&](int g, int s, FF y) -> FF {
                const float ri = ff_to_float(ff_add(FF{v.b[mlo + 8 * g + s], 0.0f}, FF{-y.hi, -y.lo}));
                ap_at(s, g) = ri;
                return ff_prod(ri, ri);
            };
            // rolled over the z-lines of the block: straight-line code that runs twice per solve
            // would come from L2
            if (kMode == kCgRows) {
                sum_rows([&](int, int) {
                    FF y = ff_zero();
#pragma unroll 1
                    for (int q = 0; q < 9; ++q) {
#pragma unroll
                        for (int kz = 0; kz < 3; ++kz) {
                            int n, sib;
                            slot_of(rs, q / 3, q % 3, kz, n, sib);
                            const float wk = w_of((q / 3 != 1) + (q % 3 != 1), kz);
                            y = ff_add(y, ff_prod(wk, x_of(desc_of(rg, n), sib)));
                        }
                    }
                    return residual(rg, rs, y);
                });
            } else {
                for_groups([&](int g) {
                    FF y[8];
#pragma unroll
                    for (int s = 0; s < 8; ++s) y[s] = ff_zero();
#pragma unroll 1
                    for (int q = 0; q < 16; ++q) {
                        const int bx = q >> 2, by = q & 3;
                        const int nxy = 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1);
                        const int sxy = 4 * ((bx + 1) & 1) + 2 * ((by + 1) & 1);
                        float xv[4];
#pragma unroll
                        for (int bz = 0; bz < 4; ++bz) xv[bz] = x_of(desc_of(g, nxy + cg_pos_axis(bz)), sxy + ((bz + 1) & 1));
#pragma unroll
                        for (int sxy2 = 0; sxy2 < 4; ++sxy2) {   // the rows (sx, sy) this line neighbours
                            const int ox = bx - (sxy2 >> 1), oy = by - (sxy2 & 1);
                            if (ox < 0 || ox > 2 || oy < 0 || oy > 2) continue;
                            const int axes = (ox != 1) + (oy != 1);
#pragma unroll
                            for (int sz = 0; sz < 2; ++sz)
#pragma unroll
                                for (int oz = 0; oz < 3; ++oz) {
                                    FF& t = y[2 * sxy2 + sz];
                                    t = ff_add(t, ff_prod(w_of(axes, oz), xv[sz + oz]));
                                }
                        }
                    }
                    return cg_group_sum([&](int s) { return residual(g, s, y[s]); });
                });
            }
            cgc_allreduce<true>(nb, me, sh, nred, acc, err, [&](const CgSum& t) { cgc_after_true(sh, a, t, it); });
            if (sh.replace) {   // refinement restart: CG continues from the true residual
                if (kMode == kCgRows) {
                    if (row_on) rp[rs * GP + rg].x = sap[rs * GP + rg];
                } else {
                    for (int g = tid; g < ng; g += kCgcBlock)
#pragma unroll
                        for (int s = 0; s < 8; ++s) rp[s * GP + g].x = ap_at(s, g);
                }
                // before any CTA reads a neighbour's new r
                if (nb > 1) cl.sync();
                else __syncthreads();
            }
        }
    }
    __syncthreads();
    for (int l = tid; l < 8 * ng; l += kCgcBlock) {
        v.x[mlo + l] = x_at(l & 7, l >> 3);
    }
    if (ran && me == 0 && tid == 0) cgc_report(v, u.d, sh, it - 1);
}

// The same sum for any number of groups a thread (digits of 64 bits), by cluster barriers, which also
// publish the CTAs' vectors in global memory.
struct CgWide {
    long long x, y, z, w;
};
struct CgWideShared {
    CgWide warp[kCgWarps], cta[2];
    int warp_b[kCgWarps], cta_b[2];
    FF term[kCgWarps][32 * 9];   // the terms of 32 groups a warp
};
static_assert(sizeof(CgWideShared) <= kCgSmemBytes, "in the resident path's shared memory");
// the lanes' sum of d, |d| < 2^44
__device__ __forceinline__ long long cgd_add_lanes(long long d) {
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)d & 0xfffffu);
    return ((long long)__reduce_add_sync(0xffffffffu, (int)(d >> 20)) << 20) + (long long)lo;
}
template <class Post>
__device__ __forceinline__ void cgc_allreduce_wide(cg::cluster_group& cl, unsigned nb, CgWideShared& sw, unsigned& n,
                                                   CgDig v, Post post) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, buf = (int)(n & 1u);
    auto lanes_sum = [](CgWide d, int& lane_b) -> CgWide {
        const int b = __reduce_max_sync(0xffffffffu, lane_b);
        cgd_drop(d, b - lane_b);
        lane_b = b;
        return CgWide{cgd_add_lanes(d.x), cgd_add_lanes(d.y), cgd_add_lanes(d.z), cgd_add_lanes(d.w)};
    };
    const CgWide w = lanes_sum(CgWide{v.d.x, v.d.y, v.d.z, v.d.w}, v.b);
    if (lane == 0) {
        sw.warp[warp] = w;
        sw.warp_b[warp] = v.b;
    }
    __syncthreads();
    CgWide t{0, 0, 0, 0};
    int tb = -1;
    if (warp == 0) {
        tb = sw.warp_b[lane];
        t = lanes_sum(sw.warp[lane], tb);
        if (lane == 0) {
            sw.cta[buf] = t;
            sw.cta_b[buf] = tb;
        }
    }
    if (nb > 1) cl.sync();
    if (warp == 0) {
        if (nb > 1 && (unsigned)lane < nb) {
            t = *cl.map_shared_rank(&sw.cta[buf], lane);
            tb = *cl.map_shared_rank(&sw.cta_b[buf], lane);
        } else if (nb > 1 || lane > 0) {
            t = CgWide{0, 0, 0, 0};
            tb = -1;
        }
        const CgSum sum = cgd_total(t, tb);
        if (lane == 0) post(sum);
    }
    ++n;
    __syncthreads();
}

// Global-memory path (any size, any depth).  A row has a lane, so that a warp reads consecutive rows, and
// every eight turns a lane adds the terms of one group.  r and p are one pair, so a neighbour is one
// load (278,000 rows on 16 CTAs: 109 -> 95 us an iteration); the peers' vectors are read through L1, and every reduction passes the cluster
// barrier.
__device__ __forceinline__ void cgc_global(cg::cluster_group& cl, CgcShared& sh, const CgcArgs& a,
                                           const CgcVec& v, const CgUnit& u, float4* dyn) {
    const unsigned me = u.me, nb = u.nb;
    CgWideShared& sw = *reinterpret_cast<CgWideShared*>(dyn);
    const int lane = threadIdx.x & 31;
    const int first = u.row0 + (int)(me * blockDim.x + threadIdx.x), nthr = nb * blockDim.x;
    // the digits of term(row) over the rows of this thread, added group by group in cg_group_sum's order
    auto sum_rows = [&](auto term) -> CgDig {
        CgDig acc{make_int4(0, 0, 0, 0), -1};
        FF* buf = sw.term[threadIdx.x >> 5];
        for (int i0 = first - lane; i0 < u.row1; i0 += 8 * nthr) {
#pragma unroll 1
            for (int q = 0; q < 8; ++q) {
                const int i = i0 + q * nthr + lane;
                buf[9 * (4 * q + (lane >> 3)) + (lane & 7)] = i < u.row1 ? term(i) : ff_zero();
            }
            __syncwarp();
            cgd_add(acc, cg_group_sum([&](int s) { return buf[9 * lane + s]; }));
            __syncwarp();
        }
        return acc;
    };
    unsigned nred = 0;
    CgDig acc = sum_rows([&](int i) {
        const float bi = v.b[i];
        v.rp[i] = make_float2(bi, 0.0f);
        v.x[i] = 0.0f;
        return ff_prod(bi, bi);
    });
    cgc_allreduce_wide(cl, nb, sw, nred, acc, [&](const CgSum& t) { cgc_start(sh, a, t); });
    bool ran = false;
    int it = 1;
    while (sh.go) {
        const float beta = sh.beta;
        acc = sum_rows([&](int i) {
            const float2 own = v.rp[i];
            float y = 0.0f;
#pragma unroll 9
            for (int k = 0; k < 27; ++k) {
                const int nb = __ldg(&v.neigh[(size_t)k * a.stride + i]);
                if (nb >= 0) {
                    const float2 q = v.rp[nb];
                    y = fmaf(sh.st[k], fmaf(beta, q.y, q.x), y);
                }
            }
            v.ap[i] = y;
            return ff_prod(fmaf(beta, own.y, own.x), y);
        });
        cgc_allreduce_wide(cl, nb, sw, nred, acc, [&](const CgSum& t) { cgc_alpha(sh, t); });
        const float alpha = sh.alpha;
        acc = sum_rows([&](int i) {
            const float2 own = v.rp[i];
            const float pi = fmaf(beta, own.y, own.x);
            v.x[i] = fmaf(alpha, pi, v.x[i]);
            const float ri = fmaf(-alpha, v.ap[i], own.x);
            v.rp[i] = make_float2(ri, pi);
            return ff_prod(ri, ri);
        });
        cgc_allreduce_wide(cl, nb, sw, nred, acc, [&](const CgSum& t) { cgc_after_rr(sh, a, t, it); });
        ran = true;
        ++it;
        if (sh.check) {
            // true residual r = b - A x (the barrier of the last reduction published x)
            acc = sum_rows([&](int i) {
                FF y = ff_zero();
                for (int k = 0; k < 27; ++k) {
                    const int nb = __ldg(&v.neigh[(size_t)k * a.stride + i]);
                    if (nb >= 0) y = ff_add(y, ff_prod(sh.st[k], v.x[nb]));
                }
                const float ri = ff_to_float(ff_add(FF{v.b[i], 0.0f}, FF{-y.hi, -y.lo}));
                v.ap[i] = ri;   // staged; A p holds nothing live here
                return ff_prod(ri, ri);
            });
            cgc_allreduce_wide(cl, nb, sw, nred, acc, [&](const CgSum& t) { cgc_after_true(sh, a, t, it); });
            if (sh.replace) {   // refinement restart: CG continues from the true residual
                for (int i = first; i < u.row1; i += nthr) v.rp[i].x = v.ap[i];
                if (nb > 1) cl.sync();
                else __syncthreads();
            }
        }
    }
    if (ran && me == 0 && threadIdx.x == 0) cgc_report(v, u.d, sh, it - 1);
}

// the CTA's shared state, for the kernel and what it calls out of line
__device__ __forceinline__ CgcShared& cgc_shared() {
    __shared__ CgcShared sh;
    return sh;
}

// Out of line: in the kernel their registers would cost the other modes 200 bytes of spills (4% of an
// iteration).
__device__ __noinline__ void cgc_far(const CgcArgs a, const CgUnit u) {
    extern __shared__ float4 cg_dyn[];
    cg::cluster_group cl = cg::this_cluster();
    CgcVec v = a.v;
    v.rebase();
    cgc_global(cl, cgc_shared(), a, v, u, cg_dyn);
}
__device__ __noinline__ void cgc_pairs(const CgcArgs a, const CgUnit u, int chunk) {
    extern __shared__ float4 cg_dyn[];
    cg::cluster_group cl = cg::this_cluster();
    CgcVec v = a.v;
    v.rebase();
    cgc_resident<kCgPairs>(cl, cgc_shared(), a, v, u, chunk, cg_dyn);
}

// One depth per cluster; behind the first a.clusters clusters, one depth per CTA.  Cluster
// barriers are passed by every CTA the same number of times only where a whole cluster solves.
__global__ void __launch_bounds__(kCgcBlock) k_cg_cluster(CgcArgs a) {
    cg::cluster_group cl = cg::this_cluster();
    CgcVec v = a.v;
    v.rebase();
    CgcShared& sh = cgc_shared();
    extern __shared__ float4 cg_dyn[];
    const unsigned long long t_start = global_ns();
    const unsigned size = cl.num_blocks(), rank = cl.block_rank();
    const int cluster = (int)(blockIdx.x / size);
    const bool whole = cluster < a.clusters;
    CgUnit u;
    u.d = whole ? a.first - cluster : a.first - a.clusters - ((cluster - a.clusters) * (int)size + (int)rank);
    u.me = whole ? rank : 0u;
    u.nb = whole ? size : 1u;
    u.rank0 = whole ? 0u : rank;
    cgc_barriers_init(sh);
    if (u.d >= 0) {
        u.row0 = v.c->level_base[u.d];
        u.row1 = (u.d < a.depth) ? v.c->level_base[u.d + 1] : v.c->n_nodes;
        if (threadIdx.x < 27) sh.st[threadIdx.x] = v.stencil[u.d * 27 + threadIdx.x];
    }
    cl.sync();   // the barriers are up before a peer arrives at them
    if (u.d >= 0) {
        const int m = u.row1 - u.row0;
        const int chunk = cg_chunk_groups(m, (int)u.nb);
        const bool fits = cg_fits_resident(u.d, m, (int)u.nb);   // the same in all CTAs of the unit
        if (!fits) cgc_far(a, u);
        else if (chunk <= kCgRowGroups) cgc_resident<kCgRows>(cl, sh, a, v, u, chunk, cg_dyn);
        else if (chunk <= kCgcBlock) cgc_resident<kCgOne>(cl, sh, a, v, u, chunk, cg_dyn);
        else if (chunk < kCgGroups) cgc_resident<kCgMany>(cl, sh, a, v, u, chunk, cg_dyn);
        else cgc_pairs(a, u, chunk);
        if (u.me == 0 && threadIdx.x == 0) v.cw->cg_depth_ns[u.d] = global_ns() - t_start;
    }
    cl.sync();   // no CTA exits while others may still read its shared memory
}

// ---- whole-GPU CG: the depths from 5 on of trees of depth 8 and 9 ------------------------
// One cooperative launch (so all its blocks are resident) solves every unit -- a depth of a cloud
// -- in rounds of two steps: A p with p.Ap, then x and r with r.r.  A unit whose true residual is due
// spends a round on it instead.  The arithmetic, the reductions'
// precision and the decisions are the cluster solver's; the scalars of a unit are kept in the
// shared memory of every block that works on it, each computing them from the same sums.
// Work is dealt in virtual blocks of 256 sibling groups of one unit, a contiguous range of them
// per block; a thread applies the operator to a group (cg_apply_group), from global memory with
// sibling-major vectors (row `sib` of group G at sib * pitch + G), so that a warp's 32 consecutive
// groups read consecutive words for their own rows and runs of them for their neighbours'.  The
// neighbour groups (27 a group, 13.5 bytes a row) are looked up once per solve.  Each virtual
// block's sum goes to global memory and every block adds a unit's sums in one order, which
// depends on the unit's rows alone: a cloud's result is the same alone and in a batch.
// A step ends when a block has the sums of all virtual blocks of its units, which is the only barrier:
// units run at their own pace.  A block's warps go through its passes without waiting for one
// another, and A p, which only the thread that computed it reads, stays in shared memory.  A round of
// 0.28M rows takes 10 us, of 1.2M 19 us and of 3.1M 41 us; with a whole-GPU barrier per step and the
// sums read after it 11, 20 and 49 us, and as kernels in a CUDA-graph while node (7 launches per two
// iterations) 27, 43 and 97 us.  What is left: 4k to 6k cycles per step for records to travel through
// L2, and in A p the gather of 64 (r, p) pairs a group (8k cycles per 512 groups).  Not kept:
// the block's p in shared memory with other blocks' groups read from L2 (5.0 ms a solve against 3.4 of
// 3.1M rows: the scattered reads wait one by one) or copied beside it every round (the gather falls to
// 5.5k cycles, the copies and their block barrier take what it saves); the planes of the gather
// pipelined by hand, 640 threads, virtual blocks of 128 (the same to 8% slower).
constexpr int kGridBlock = 512;    // 128 registers a thread: a group's 27 neighbours and 32 loads in flight
constexpr int kVbGroups = 256;                       // groups of a virtual block
constexpr int kGridSubs = kGridBlock / kVbGroups;    // virtual blocks a block works on at once
constexpr int kGridPasses = 16;                      // passes over its virtual blocks between two block barriers
// passes whose A p stays in shared memory: 96 KB for 3.6M rows on 147 SMs, more of which go to global
// memory; the rest of the SM's 256 KB is L1 for the gather
constexpr int kGridApPasses = 6;
constexpr size_t kGridApBytes = sizeof(float) * 8 * kGridBlock * kGridApPasses;
constexpr int kGridUnits = kMaxBatchClouds * (kMaxDepth - 4);   // most units of a launch
constexpr int kGridDepth = 5;                        // depths below it: at most 4096 rows, one CTA each

struct CgGridArgs {
    CgcVec v;             // cloud 0's workspace
    int depth;
    int first, last;      // depths first .. last (descending) of every cloud
    int clouds;
    size_t stride;
    unsigned pitch;       // groups of the sibling-major arrays; the last one is the zero group (element
                          // numbers up to 8 * pitch fit 32 bits)
    int* nbg;             // [27][pitch]: neighbour groups
    float2* rp;           // [8][pitch]: (r, p)
    float* xs;            // [8][pitch]: x
    float* ap;            // [8][pitch]: A p
    ulonglong2* part;     // [2][part_cap + kGridUnits]: sums of the virtual blocks, of units (cloud 0)
    int part_cap;
    unsigned long long* bar;   // arrivals of the blocks (cloud 0; starts at 0)
    float tol2;
    int max_iter;
    int res_period;
};

// State of one unit in a block's shared memory (the cluster solver's scalars).
struct CgGridUnit {
    CgSum rr, pap;
    double floor2, rr_true;
    float rrf, alpha, beta;
    int go, check, replace, checks, restarts, until_check;
    int it;               // iterations done
    int resid;            // this round evaluated the true residual
    int d, k;             // depth, cloud
    int G0, ng;           // first group (global number), groups
    int vb0, nvb;         // first virtual block of the launch, virtual blocks
    float w[4];           // centre, face, edge, corner
};

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Every block of the launch has arrived.  Thread 0's fences make the block's writes visible to the
// others and theirs to the block.  Bounded: false when the wait ran out.
__device__ __forceinline__ bool grid_barrier(unsigned long long* bar, unsigned target) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1ull);
        unsigned long long v = ld_acquire_u64(bar);
        int spin = 0;
        while (v < target && ++spin < kSpinLimit) v = ld_acquire_u64(bar);
        __threadfence();
        s_ok = v >= target;
    }
    __syncthreads();
    return s_ok != 0;
}

// A virtual block's sum of one step as a 16-byte record that carries the step's number in both
// halves, so that a reader knows from the record alone that the sum is the step's and that what the
// writing block wrote before it is visible (after a fence of the reader's).
__device__ __forceinline__ void cgs_publish(ulonglong2* p, const CgSum& t, unsigned step) {
    const unsigned long long lo = (unsigned)t.m | (unsigned long long)(unsigned short)t.e << 32 |
                                  (unsigned long long)(step & 0xffffu) << 48;
    const unsigned long long hi = (unsigned)(t.m >> 32) | (unsigned long long)step << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
// waits for the record of `step`; false when the wait ran out
__device__ __forceinline__ bool cgs_collect(const ulonglong2* p, unsigned step, CgSum& t) {
    unsigned long long lo, hi;
    int spin = 0;
    do {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
        if ((unsigned)(hi >> 32) == step && (unsigned)(lo >> 48) == (step & 0xffffu)) {
            t.m = (long long)((unsigned long long)(unsigned)hi << 32 | (unsigned)lo);
            t.e = (short)(lo >> 32);
            return true;
        }
    } while (++spin < kSpinLimit);
    t = CgSum{0, 0};
    return false;
}

// a + b, aligned like the lanes of a warp sum
__device__ __forceinline__ CgSum cgs_add(CgSum a, CgSum b) {
    auto top_of = [](const CgSum& v) { return v.m != 0 ? (int)v.e + 64 - __clzll(v.m < 0 ? -v.m : v.m) : 0; };
    const int e = max(top_of(a), top_of(b)) - 57;
    auto to = [&](const CgSum& v) -> long long {
        const int d = e - (int)v.e;
        if (v.m == 0) return 0;
        if (d <= 0) return d > -64 ? v.m << -d : 0;
        return d < 63 ? ((v.m >> (d - 1)) + 1) >> 1 : 0;
    };
    return CgSum{to(a) + to(b), e};
}

__global__ void __launch_bounds__(kGridBlock) k_cg_grid(CgGridArgs a) {
    extern __shared__ float4 cg_dyn[];
    CgGridUnit* U = reinterpret_cast<CgGridUnit*>(cg_dyn);   // one per unit of the launch
    __shared__ int4 s_w[kGridPasses][kGridBlock / 32];   // warp sums of a step's passes
    __shared__ CgSum s_sum[kGridBlock / 32];
    __shared__ int s_total, s_late;   // s_late: a wait ran out
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = tid / kVbGroups, subt = tid % kVbGroups;
    const int per = a.first - a.last + 1, nu = per * a.clouds;
    const unsigned long long t0 = global_ns();
    auto fail = [&](int k, unsigned bits) { atomicOr(&at_cloud(a.v.cw, k)->error, bits); };
    // the units: cloud after cloud, depth after depth
    for (int u = tid; u < nu; u += kGridBlock) {
        CgGridUnit& q = U[u];
        q.k = u / per;
        q.d = a.first - (u - q.k * per);
        const Counters* c = at_cloud(a.v.c, q.k);
        q.G0 = (c->level_base[q.d] - 1) >> 3;
        q.ng = c->level_count[q.d] >> 3;
        q.nvb = (q.ng + kVbGroups - 1) / kVbGroups;
        const float* st = at_cloud(a.v.stencil, q.k) + q.d * 27;
        q.w[0] = st[13]; q.w[1] = st[14]; q.w[2] = st[17]; q.w[3] = st[26];
        q.go = q.check = q.replace = q.resid = q.it = 0;
    }
    __syncthreads();
    if (tid == 0) {
        int v = 0;
        for (int u = 0; u < nu; ++u) {
            U[u].vb0 = v;
            v += U[u].nvb;
        }
        s_total = v;
    }
    __syncthreads();
    const int total = s_total;
    if (total > a.part_cap) {   // uniform over the launch
        if (blockIdx.x == 0)
            for (int k = tid; k < a.clouds; k += kGridBlock) fail(k, kErrCapacity);
        return;
    }
    // this block's virtual blocks, and the units they belong to
    const int v0 = (int)((long long)total * blockIdx.x / gridDim.x);
    const int v1 = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
    const int npass = (v1 - v0 + kGridSubs - 1) / kGridSubs;
    auto unit_of = [&](int v) {
        int lo = 0, hi = nu - 1;   // the last unit with vb0 <= v
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (U[mid].vb0 <= v) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    };
    const int u0 = v0 < v1 ? unit_of(v0) : 0, u1 = v0 < v1 ? unit_of(v1 - 1) + 1 : 0;
    // The records of a step (its number from 1) alternate between two buffers.  A block publishes a
    // step's records after it has read all of the step before, so a record is overwritten (two steps
    // later) only when every block of its unit has read it.
    unsigned nstep = 0;
    if (tid == 0) s_late = 0;
    const size_t part_stride = (size_t)a.part_cap + kGridUnits;   // then a total per unit
    for (int v = v0 + tid; v < v1; v += kGridBlock) a.part[v] = a.part[part_stride + v] = make_ulonglong2(0ull, 0ull);
    for (int u = u0 + tid; u < u1; u += kGridBlock)
        if (U[u].vb0 >= v0) a.part[a.part_cap + u] = a.part[part_stride + a.part_cap + u] = make_ulonglong2(0ull, 0ull);

    // one step over the block's virtual blocks: body(unit, local group, pass) returns the thread's
    // contribution; `skip(unit)`: the unit takes no part.  Publishes the virtual blocks' sums.
    // `writes`: the step leaves vectors for other blocks; only then the records need fences.  (A step
    // that does not only reads what other blocks may overwrite in the next one, and a record depends
    // on every value its block read.)
    bool fenced = true;
    auto step = [&](bool writes, auto skip, auto body) {
        ++nstep;
        fenced = writes;
        for (int p0 = 0; p0 < npass; p0 += kGridPasses) {
            const int np = min(npass - p0, kGridPasses);
            if (p0) __syncthreads();
            for (int p = 0; p < np; ++p) {
                const int vb = v0 + (p0 + p) * kGridSubs + sub;
                FF acc = ff_zero();
                int u = vb < v1 ? unit_of(vb) : -1;
                if (u >= 0 && skip(U[u])) u = -1;
                if (u >= 0) {
                    const int g = (vb - U[u].vb0) * kVbGroups + subt;
                    if (g < U[u].ng) acc = body(U[u], g, p0 + p);
                }
                int4 ws = make_int4(0, 0, 0, 0);
                if (__any_sync(0xffffffffu, acc.hi != 0.0f)) ws = cgs_warp_sum(acc);
                if (lane == 0) s_w[p][warp] = ws;
            }
            __syncthreads();
            for (int q = warp; q < np * kGridSubs; q += kGridBlock / 32) {
                const int p = q / kGridSubs, sb = q % kGridSubs, vb = v0 + (p0 + p) * kGridSubs + sb;
                if (vb >= v1 || skip(U[unit_of(vb)])) continue;
                constexpr int kWarps = kVbGroups / 32;
                const CgSum t = cgs_warp_sum(cgs_join(lane < kWarps ? s_w[p][sb * kWarps + lane] : make_int4(0, 0, 0, 0)));
                if (lane == 0) {
                    if (fenced) fence_gpu();   // the block's writes of the step before its records
                    cgs_publish(a.part + (nstep & 1) * part_stride + vb, t, nstep);
                }
            }
        }
    };
    // Waits for the records of the units that took part in the step, which is also the barrier between
    // the blocks of a unit, and adds them (the order depends on the unit alone); post(unit, sum) by
    // one thread.  Of a unit with up to 32 virtual blocks a warp of every block reads all records; of
    // a larger one the block that holds its first virtual block does and publishes the total (with
    // 106 blocks polling 106 records each the wait took 7k cycles, so 4k).  False when a wait ran out.
    auto sums = [&](auto skip, auto post) -> bool {
        ulonglong2* part = a.part + (nstep & 1) * part_stride;
        bool late = false;
        for (int u = u0; u < u1; ++u) {
            if (U[u].nvb <= 32 || U[u].vb0 < v0 || skip(U[u])) continue;   // the same in all threads
            CgSum t{0, 0}, r;
            for (int v = tid; v < U[u].nvb; v += kGridBlock) {
                late |= !cgs_collect(part + U[u].vb0 + v, nstep, r);
                t = cgs_add(t, r);
            }
            if (fenced && tid < U[u].nvb) fence_gpu();
            t = cgs_warp_sum(t);
            if (lane == 0) s_sum[warp] = t;
            __syncthreads();
            if (warp == 0) {
                t = cgs_warp_sum(lane < kGridBlock / 32 ? s_sum[lane] : CgSum{0, 0});
                if (lane == 0) {
                    if (fenced) fence_gpu();
                    cgs_publish(part + a.part_cap + u, t, nstep);
                }
            }
            __syncthreads();
        }
        for (int u = u0 + warp; u < u1; u += kGridBlock / 32) {
            if (skip(U[u])) continue;
            CgSum t{0, 0};
            if (U[u].nvb <= 32) {
                if (lane < U[u].nvb) late |= !cgs_collect(part + U[u].vb0 + lane, nstep, t);
                if (fenced) fence_gpu();   // what the unit's other blocks wrote before their records
                t = cgs_warp_sum(t);
            } else if (lane == 0) {
                late |= !cgs_collect(part + a.part_cap + u, nstep, t);
                if (fenced) fence_gpu();
            }
            if (lane == 0) post(U[u], t);
        }
        if (late) s_late = 1;
        __syncthreads();
        return s_late == 0;
    };

    // A p of a group, its rows `aps` apart: in shared memory for the first kGridApPasses passes
    float* s_ap = reinterpret_cast<float*>(U + nu);
    auto ap_of = [&](const CgGridUnit& q, int G, int pass, unsigned& aps) -> float* {
        if (pass < kGridApPasses) {
            aps = kGridBlock;
            return s_ap + pass * 8 * kGridBlock + tid;
        }
        aps = a.pitch;
        return at_cloud(a.ap, q.k) + G;
    };

    // neighbour groups; r0 = b, p_{-1} = 0, x0 = 0
    if (blockIdx.x == 0 && tid < 8)
        for (int k = 0; k < a.clouds; ++k) {
            at_cloud(a.rp, k)[tid * a.pitch + a.pitch - 1] = make_float2(0.0f, 0.0f);
            at_cloud(a.xs, k)[tid * a.pitch + a.pitch - 1] = 0.0f;
        }
    bool ok = grid_barrier(a.bar, gridDim.x);   // the cleared records and the zero group
    step(
        true, [](const CgGridUnit&) { return false; },
        [&](const CgGridUnit& q, int g, int) {
            const int G = q.G0 + g;
            CgcVec v = a.v;
            v.neigh = at_cloud(a.v.neigh, q.k);
            v.first_child = at_cloud(a.v.first_child, q.k);
            const int pa = at_cloud(a.v.parent, q.k)[1 + 8 * G];
            int* nbg = at_cloud(a.nbg, q.k);
            int H[27];
#pragma unroll
            for (int n = 0; n < 27; ++n) H[n] = cg_neighbour_group(v, a.stride, pa, n);
#pragma unroll
            for (int n = 0; n < 27; ++n)
                nbg[n * a.pitch + G] = (unsigned)(H[n] - q.G0) < (unsigned)q.ng ? H[n] : (int)a.pitch - 1;
            const float* b = at_cloud(a.v.b, q.k) + 1 + 8 * (size_t)G;
            float2* rp = at_cloud(a.rp, q.k) + G;
            float* xs = at_cloud(a.xs, q.k) + G;
            FF acc = ff_zero();
            float bi[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) bi[s] = b[s];
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                rp[s * a.pitch] = make_float2(bi[s], 0.0f);
                xs[s * a.pitch] = 0.0f;
                acc = ff_add(acc, ff_prod(bi[s], bi[s]));
            }
            return acc;
        });
    ok &= sums([](const CgGridUnit&) { return false; }, [&](CgGridUnit& q, const CgSum& t) { cgc_start(q, a, t); q.check = 0; });
    auto idle = [](const CgGridUnit& q) { return !q.go && !q.check; };
    // a round per iteration and per true residual, until none of the block's units has work
    const long long most = 2LL * a.max_iter + kCgMaxRefine + 8;
    long long round = 0;
    for (; ok && round < most; ++round) {
        bool active = false;
        for (int u = u0; u < u1; ++u) active |= !idle(U[u]);
        if (!active) break;
        // (A) A p_k from the neighbours' (r_k, p_{k-1}), p.Ap; or the true residual b - A x
        step(false, idle, [&](CgGridUnit& q, int g, int pass) {
            const int G = q.G0 + g;
            const int* nbg = at_cloud(a.nbg, q.k) + G;
            unsigned aps;
            float* ap = ap_of(q, G, pass, aps);
            FF acc = ff_zero();
            if (q.check) {
                const float* xs = at_cloud(a.xs, q.k);
                const float* b = at_cloud(a.v.b, q.k) + 1 + 8 * (size_t)G;
                FF y[8];
#pragma unroll
                for (int s = 0; s < 8; ++s) y[s] = ff_zero();
#pragma unroll 1
                for (int z = 0; z < 16; ++z) {   // the z-lines of the block
                    const int bx = z >> 2, by = z & 3;
                    const int nxy = 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1);
                    const int sxy = 4 * ((bx + 1) & 1) + 2 * ((by + 1) & 1);
                    float xv[4];
#pragma unroll
                    for (int bz = 0; bz < 4; ++bz)
                        xv[bz] = xs[(unsigned)(sxy + ((bz + 1) & 1)) * a.pitch +
                                    (unsigned)nbg[(unsigned)(nxy + cg_pos_axis(bz)) * a.pitch]];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int ox = bx - (r >> 1), oy = by - (r & 1);
                        if (ox < 0 || ox > 2 || oy < 0 || oy > 2) continue;
                        const int axes = (ox != 1) + (oy != 1);
#pragma unroll
                        for (int sz = 0; sz < 2; ++sz)
#pragma unroll
                            for (int oz = 0; oz < 3; ++oz) {
                                FF& t = y[2 * r + sz];
                                t = ff_add(t, ff_prod(q.w[axes + (oz != 1)], xv[sz + oz]));
                            }
                    }
                }
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const float ri = ff_to_float(ff_add(FF{b[s], 0.0f}, FF{-y[s].hi, -y[s].lo}));
                    ap[s * aps] = ri;
                    acc = ff_add(acc, ff_prod(ri, ri));
                }
                return acc;
            }
            const float beta = q.beta;
            const float w[4] = {q.w[0], q.w[1], q.w[2], q.w[3]};
            const float2* rp = at_cloud(a.rp, q.k);
            // the table past L1 (read once a round), so that L1 keeps the pairs
            unsigned nb[27];
#pragma unroll
            for (int n = 0; n < 27; ++n) nb[n] = (unsigned)__ldcg(nbg + (unsigned)n * a.pitch);
            float y[8], pi[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) y[s] = 0.0f;
#pragma unroll
            for (int bx = 0; bx < 4; ++bx) {   // a plane's 16 positions are loaded together
                float2 e[16];
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    e[q] = rp[(unsigned)cg_pos_sib(16 * bx + q) * a.pitch + nb[cg_pos_group(16 * bx + q)]];
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const int p = 16 * bx + q;
                    const float v = fmaf(beta, e[q].y, e[q].x);
                    if (cg_pos_group(p) == 13) pi[cg_pos_sib(p)] = v;   // the group itself
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        const int ox = (p >> 4) - (s >> 2), oy = ((p >> 2) & 3) - ((s >> 1) & 1), oz = (p & 3) - (s & 1);
                        if (ox >= 0 && ox < 3 && oy >= 0 && oy < 3 && oz >= 0 && oz < 3)
                            y[s] = fmaf(w[cg_class(9 * ox + 3 * oy + oz)], v, y[s]);
                    }
                }
            }
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                ap[s * aps] = y[s];
                acc = ff_add(acc, ff_prod(pi[s], y[s]));
            }
            // Only a unit's first group can have a table that does not name the group itself (its parent is
            // recorded as the first node of the level above): the operator takes what the table says,
            // the rows' own p their own pairs
            if (g == 0 && nb[13] != (unsigned)G) {
                acc = ff_zero();
#pragma unroll 1
                for (int s = 0; s < 8; ++s) {
                    const float2 o = rp[(unsigned)s * a.pitch + (unsigned)G];
                    acc = ff_add(acc, ff_prod(fmaf(beta, o.y, o.x), ap[s * aps]));
                }
            }
            return acc;
        });
        ok = sums(idle, [&](CgGridUnit& q, const CgSum& t) {
            q.resid = q.check;
            if (q.check) {
                cgc_after_true(q, a, t, q.it + 1);
                q.check = 0;
            } else {
                cgc_alpha(q, t);
            }
        });
        if (!ok) break;
        // (B) x and r, r.r; after a true residual: the restart's r
        auto rest = [](const CgGridUnit& q) { return !q.go && !q.resid; };
        step(true, rest, [&](CgGridUnit& q, int g, int pass) {
            const int G = q.G0 + g;
            float2* rp = at_cloud(a.rp, q.k) + G;
            unsigned aps;
            const float* ap = ap_of(q, G, pass, aps);
            FF acc = ff_zero();
            if (q.resid) {
                if (q.replace)
#pragma unroll
                    for (int s = 0; s < 8; ++s) rp[s * a.pitch].x = ap[s * aps];
                return acc;
            }
            float* xs = at_cloud(a.xs, q.k) + G;
            const float alpha = q.alpha, beta = q.beta;
            float2 own[8];
            float xo[8], y[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) {   // every load before the first store
                own[s] = rp[s * a.pitch];
                xo[s] = xs[s * a.pitch];
                y[s] = ap[s * aps];
            }
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const float pi = fmaf(beta, own[s].y, own[s].x);
                xs[s * a.pitch] = fmaf(alpha, pi, xo[s]);
                const float ri = fmaf(-alpha, y[s], own[s].x);
                rp[s * a.pitch] = make_float2(ri, pi);
                acc = ff_add(acc, ff_prod(ri, ri));
            }
            return acc;
        });
        ok = sums(rest, [&](CgGridUnit& q, const CgSum& t) {
            if (!q.resid) {
                ++q.it;
                cgc_after_rr(q, a, t, q.it);
            }
            q.resid = 0;
        });
    }
    // a wait ran out: the block's units are unfinished, and with them those of every other block that
    // waits for its records, so the clouds of all its units fail
    if (!ok || round >= most)
        for (int u = u0 + tid; u < u1; u += kGridBlock) fail(U[u].k, kErrSpinTimeout);
    // x in row order; the reports by the block that holds a unit's first virtual block
    for (int p = 0; p < npass; ++p) {
        const int vb = v0 + p * kGridSubs + sub;
        if (vb >= v1) continue;
        const CgGridUnit& q = U[unit_of(vb)];
        const int g0 = (vb - q.vb0) * kVbGroups, n = 8 * min(kVbGroups, q.ng - g0);
        const float* xs = at_cloud(a.xs, q.k) + q.G0 + g0;
        float* x = at_cloud(a.v.x, q.k) + 1 + 8 * (size_t)(q.G0 + g0);
        for (int l = subt; l < n; l += kVbGroups) x[l] = xs[(unsigned)(l & 7) * a.pitch + (unsigned)(l >> 3)];
    }
    for (int u = u0 + tid; u < u1; u += kGridBlock) {
        const CgGridUnit& q = U[u];
        if (q.vb0 < v0) continue;
        Counters* c = at_cloud(a.v.cw, q.k);
        if (q.it > 0) {
            c->cg_iters[q.d] = q.it;
            c->cg_rr[q.d] = cgs_double(q.rr);
            c->cg_rr_true[q.d] = q.rr_true;
            c->cg_checks[q.d] = q.checks;
            c->cg_restarts[q.d] = q.restarts;
        }
        c->cg_depth_ns[q.d] = global_ns() - t0;
    }
}

// ---- implicit function at the sample points and the iso-value ----------------------
__device__ __forceinline__ void decode3s(int e, int depth, int& ix, int& iy, int& iz) {
    const int o1 = 1 << (depth + 1);
    ix = e & (o1 - 1);
    iy = (e >> (depth + 1)) & (o1 - 1);
    iz = e >> (2 * (depth + 1));
}

// The value rows of the nodes above the finest depth (ValueRows), one thread per node; the rows go
// out through shared memory, eight lanes a line.  Bound by its 54 reads a node.
constexpr int kRowPitch = 36;   // floats: 16-byte aligned, rows on different banks
__global__ void __launch_bounds__(kBlock) k_value_rows(const Counters* c, int depth, ValueRows R, float4* rows) {
    PSR_CLOUD(c, R, rows);
    __shared__ float s_row[kBlock / 32][32 * kRowPitch];
    const int n = min(c->level_base[depth], R.n);
    const int lane = lane_id();
    float* buf = s_row[threadIdx.x >> 5];
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; b < n; b += gridDim.x * blockDim.x) {
        const int node = b + lane;
        if (node < n) {
            int nb[27];
#pragma unroll
            for (int k = 0; k < 27; ++k) nb[k] = R.neigh[(size_t)k * R.stride + node];
            float* o = buf + lane * kRowPitch;
            o[27] = __int_as_float(R.enc[node]);
            o[28] = __int_as_float(R.parent[node]);
            o[29] = __int_as_float(R.first_child[node]);
            o[30] = o[31] = 0.0f;
            float xv[27];
#pragma unroll
            for (int k = 0; k < 27; ++k) xv[k] = R.x[nb[k]];
#pragma unroll
            for (int k = 0; k < 27; ++k) o[k] = xv[k];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = 4 * j + (lane >> 3);
            if (b + r < n) rows[8 * (size_t)(b + r) + (lane & 7)] = *reinterpret_cast<const float4*>(buf + r * kRowPitch + 4 * (lane & 7));
        }
        __syncwarp();
    }
}

// Implicit value at a sample point: the 27 neighbour terms ((x * Fx) * Fy) * Fz of every
// level of its chain (its depth-D node and that node's ancestors).  The levels up to D-1
// are summed first, as soon as their systems are solved, beside the depth-D CG: on the cell
// of a depth-(D-1) node they form one tensor-product quadratic (k_point_poly: its 27
// Bernstein coefficients, one thread per node), evaluated at each sample of the cell
// (k_point_values_coarse; the partial sum is kept in `out`).  The depth-D terms are added
// after the depth-D CG (k_point_values).  The iso-value is the FP64 mean of these float
// values.
template <bool kRows>
__global__ void __launch_bounds__(kBlock) k_point_poly(const Counters* c, int depth, const float* ctr_x,
                                                       const float* ctr_y, const float* ctr_z, ValueRows R,
                                                       float* coef, size_t cstride) {
    PSR_CLOUD(c, ctr_x, ctr_y, ctr_z, R, coef);
    R.n = kRows ? min(c->level_base[depth], R.n) : 0;
    const int d1 = depth - 1;
    const int n = c->level_count[d1];
    const int b = c->level_base[d1];
    PSR_GRID_STRIDE(a, n) {
        const int node = b + a;
        const float qx = ctr_x[node], qy = ctr_y[node], qz = ctr_z[node];
        float C[27], mag = 0.0f;
#pragma unroll
        for (int k = 0; k < 27; ++k) C[k] = 0.0f;
        for (int now = node; now >= 0;) {
            ValueRow r;
            load_row(R, now, r);
            int ox, oy, oz;
            decode3s(r.enc, depth, ox, oy, oz);
            const int l = ilog2_dev(ox + 1);
            now = r.parent;
            sign_level(r.x, ox, oy, oz, qx, qy, qz, __int_as_float((127 + l - depth) << 23), C, mag);   // h 2^l
        }
#pragma unroll
        for (int k = 0; k < 27; ++k) coef[(size_t)k * cstride + a] = C[k];
    }
}

// the levels up to D-1 at sample i (u in [0, 1] per axis of the sample's depth-(D-1) cell)
struct PointCoarse {
    const int* parent;
    const float *ctr_x, *ctr_y, *ctr_z;
    const float* coef;
    size_t cstride;
    __device__ float operator()(int depth, int bD, int b1, int leaf, float x, float y, float z) const {
        const float inv2h = (float)(1 << (depth - 1));   // 1 / (2 h) of a depth-(D-1) cell
        const int node = parent[bD + leaf];
        const int a = node - b1;
        // cell from centre - h to centre + h
        const float hh = 0.5f / inv2h;
        const float ux = (x - (ctr_x[node] - hh)) * inv2h;
        const float uy = (y - (ctr_y[node] - hh)) * inv2h;
        const float uz = (z - (ctr_z[node] - hh)) * inv2h;
        const float wx[3] = {(1.0f - ux) * (1.0f - ux), 2.0f * ux * (1.0f - ux), ux * ux};
        const float wy[3] = {(1.0f - uy) * (1.0f - uy), 2.0f * uy * (1.0f - uy), uy * uy};
        const float wz[3] = {(1.0f - uz) * (1.0f - uz), 2.0f * uz * (1.0f - uz), uz * uz};
        float val = 0.0f;
#pragma unroll
        for (int k = 0; k < 27; ++k)
            val = fmaf(wx[k / 9] * wy[(k / 3) % 3] * wz[k % 3], coef[(size_t)k * cstride + a], val);
        return val;
    }
    __device__ void rebase() { PSR_CLOUD(parent, ctr_x, ctr_y, ctr_z, coef); }   // to cloud blockIdx.y
};

__global__ void __launch_bounds__(kBlock) k_point_values_coarse(const Counters* c, int depth, const float* px,
                                                                const float* py, const float* pz,
                                                                const int* point2node, PointCoarse coarse, float* out) {
    PSR_CLOUD(c, px, py, pz, point2node, coarse, out);
    const int n = c->n_points;
    const int bD = c->level_base[depth];
    const int b1 = c->level_base[depth - 1];
    PSR_GRID_STRIDE(i, n) out[i] = coarse(depth, bD, b1, point2node[i], px[i], py[i], pz[i]);
}

// The sample values are summed in chunks of kBlock points (chunk_sums[chunk]), then the
// chunks in order: the iso-value's summation order depends only on the point count, not on
// the launch's grid, so a cloud gets the same iso-value alone and in a multi-cloud launch.
// The last block to finish adds the chunks.  kWithCoarse: the levels up to D-1 are evaluated
// here too instead of by a launch beside the depth-D solve.
template <bool kWithCoarse>
__global__ void __launch_bounds__(kBlock) k_point_values(Counters* c, int depth, const float* px, const float* py,
                                                         const float* pz, const int* point2node, const int* neigh,
                                                         size_t stride, const int* enc, const float* x,
                                                         PointCoarse coarse, float* out, double* chunk_sums) {
    PSR_CLOUD(c, px, py, pz, point2node, neigh, enc, x, coarse, out, chunk_sums);
    __shared__ double s_w[kBlock / 32];
    __shared__ int s_last;
    const int n = c->n_points;
    const int bD = c->level_base[depth];
    const int b1 = c->level_base[depth - 1];
    const int nchunks = (n + kBlock - 1) / kBlock;
    for (int ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        const int i = ch * kBlock + threadIdx.x;
        double acc = 0.0;
        if (i < n) {
            const int leaf = point2node[i];
            const float qx = px[i], qy = py[i], qz = pz[i];
            const float v0 = kWithCoarse ? coarse(depth, bD, b1, leaf, qx, qy, qz) : out[i];
            const float v = level_terms(bD + leaf, v0, qx, qy, qz, depth, neigh, stride, enc, x);
            out[i] = v;
            acc = (double)v;
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane_id() == 0) s_w[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double sum = 0.0;
            for (int w = 0; w < kBlock / 32; ++w) sum += s_w[w];
            chunk_sums[ch] = sum;
            __threadfence();
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) s_last = atomicAdd(&c->ticket[2], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double s = 0.0;
    for (int b = threadIdx.x; b < nchunks; b += blockDim.x) s += __ldcg(chunk_sums + b);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane_id() == 0) s_w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_w[w];
        c->iso_sum = t;
        c->iso = (c->n_points > 0) ? (float)(t / (double)c->n_points) : 0.0f;
    }
}

static int g_cg_cluster = 0;

// launch geometry that needs device queries (done once, outside any stream capture):
// the largest cluster (16, else 8) the device can schedule for the CG kernel
void prepare_launch_configs(Workspace& ws) {
    if (g_cg_cluster == 0) {
        int size = 8;
        if (cudaFuncSetAttribute(k_cg_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCgSmemBytes) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_cg_grid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(CgGridUnit) * kMaxBatchClouds * (kMaxDepth - kGridDepth + 1) + kGridApBytes)) !=
                cudaSuccess)
            return;   // left unset: the CG launch reports the error
        if (cudaFuncSetAttribute(k_cg_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(16);
            cfg.blockDim = dim3(kCgcBlock);
            cfg.dynamicSmemBytes = kCgSmemBytes;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 16;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int nclusters = 0;
            if (cudaOccupancyMaxActiveClusters(&nclusters, (void*)k_cg_cluster, &cfg) == cudaSuccess && nclusters >= 2)
                size = 16;
        }
        (void)cudaGetLastError();
        g_cg_cluster = size;
    }
    (void)scan_grid(1 << 20);
}

// one cluster (or CTA) per depth and cloud: x spans the depths, y the clouds of the batch
static cudaError_t launch_cg(void (*kernel)(CgcArgs), CgcArgs& a, int grid, int cluster, int clouds, cudaStream_t s) {
    void* args[] = {&a};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, clouds);
    cfg.blockDim = dim3(kCgcBlock);
    cfg.dynamicSmemBytes = kCgSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, (const void*)kernel, args);
}

// The whole-GPU solver of the depths from kGridDepth on: one block per SM except the SMs that the
// coarser depths' CTAs take (a block and a CTA of theirs each need an SM's registers).
static cudaError_t launch_cg_grid(Workspace& ws, const CgcArgs& a, cudaStream_t s) {
    CgGridArgs L;
    L.v = a.v;
    L.depth = a.depth;
    L.first = a.depth;
    L.last = kGridDepth;
    L.clouds = ws.batch;
    L.stride = a.stride;
    L.pitch = (unsigned)a.dstride;
    L.nbg = ws.cg_nbg;
    L.rp = ws.cg_rp;
    L.xs = ws.cg_q;
    L.ap = ws.cg_ap;
    L.part = ws.cg_part;
    L.part_cap = ws.cg_part_cap;
    L.bar = &ws.cnt->grid_bar;
    L.tol2 = a.tol2;
    L.max_iter = a.max_iter;
    L.res_period = a.res_period;
    void* args[] = {&L};
    cudaLaunchConfig_t cfg = {};
    int grid = ws.num_sms - kGridDepth;
    if (grid < 1) grid = 1;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kGridBlock);
    cfg.dynamicSmemBytes = sizeof(CgGridUnit) * (size_t)(L.first - L.last + 1) * L.clouds + kGridApBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, (const void*)k_cg_grid, args);
}

cudaError_t solve_build(Workspace& ws, int cg_mode, int cg_iters, float cg_tol, int cg_max_iter, int res_period) {
    cudaStream_t s = ws.stream;
    if (g_cg_cluster == 0) prepare_launch_configs(ws);
    const int D = ws.depth;
    CgcArgs a;
    a.v.c = ws.cnt;
    a.v.cw = ws.cnt;
    a.depth = D;
    a.v.neigh = ws.neigh;
    a.v.parent = ws.parent;
    a.v.first_child = ws.first_child;
    a.v.desc = ws.cg_desc;
    a.dstride = (size_t)ws.cap.nodes / 8 + 8;
    a.stride = (size_t)ws.cap.nodes;
    a.v.stencil = ws.stencil;
    a.v.b = ws.divg;
    a.v.x = ws.xsol;
    a.v.rp = ws.cg_p;
    a.v.xs = ws.cg_q;
    a.v.aps = (float*)ws.cg_partial;   // free once the divergence is summed
    a.v.ap = ws.cg_ap;
    a.tol2 = cg_tol * cg_tol;
    // a fixed iteration count replaces the reference's max_iter (10000); the tolerance
    // test of the loop is kept (mesh/solver/CGAlgorithm.cu:36)
    a.max_iter = (cg_mode == 1 && cg_iters > 0) ? cg_iters : cg_max_iter;
    a.res_period = res_period;
    cudaError_t e = cudaSuccess;
    // Trees up to depth 7: the finest depths (D, D-1, and D-2 from depth 5 on; never the root) on
    // clusters -- depth D on the widest cluster, D-1 and D-2 (fewer rows, done well before depth D)
    // on clusters of at most 8 CTAs, on a third stream, so that they hold fewer SMs -- and the rest
    // one CTA each, on the second stream.  Trees of depth 8 and 9, whose finest depths have hundreds
    // of thousands of rows: depths 5 .. D on the whole GPU in one launch (208k + 53k + 14k + 4k rows:
    // 0.61 ms against 0.81 ms with a 16-CTA cluster for the finest), the rest one CTA each.
    const bool whole = D >= 8;
    const int ncl = whole ? 0 : (D < 2 ? D : (D >= 5 ? 3 : 2));
    const int ncta = whole ? kGridDepth : D - ncl + 1;
    // Where the clouds of a launch need more SMs than there are, SM time counts, not the latency of a
    // solve: half the CTAs, which hold 114,624 and 57,312 rows in shared memory (16 clouds of depth 7:
    // 4.55 ms a batch with 16 and 8 CTAs, 4.27 with 16 and 4, 4.39 with 8 and 8, 4.15 with 8 and 4, 4.29
    // with 8 and 2) and the pairs of twice as many.
    const bool crowded = ws.batch * (g_cg_cluster + 2 * 8 + ncta) > ws.num_sms;
    int cl1 = ws.cg_ctas > 0 ? ws.cg_ctas : (crowded && g_cg_cluster > 8 ? 8 : g_cg_cluster);
    if (cl1 > g_cg_cluster) cl1 = g_cg_cluster;
    int cl2 = ws.cg_ctas_fine > 0 ? ws.cg_ctas_fine : (crowded ? 4 : 8);
    if (cl2 > g_cg_cluster) cl2 = g_cg_cluster;
    const size_t cstride = (size_t)ws.cap.dnodes / 8 + 64;
    const PointCoarse coarse{ws.parent, ws.ctr_x, ws.ctr_y, ws.ctr_z, ws.pv_coef, cstride};
    const int nb = ws.num_sms * 4;
    // sample values of all levels and the iso-value, once every depth is solved
    const ValueRows rows = value_rows(ws);
    auto sample_values = [&]() {
        if (whole) {
            k_value_rows<<<PSR_GRID(ws, ws.num_sms * 4), kBlock, 0, s>>>(ws.cnt, D, rows, ws.value_rows);
            k_point_poly<true><<<PSR_GRID(ws, ws.num_sms * 4), kBlock, 0, s>>>(ws.cnt, D, ws.ctr_x, ws.ctr_y, ws.ctr_z,
                                                                               rows, ws.pv_coef, cstride);
        } else {
            k_point_poly<false><<<PSR_GRID(ws, ws.num_sms * 4), kBlock, 0, s>>>(ws.cnt, D, ws.ctr_x, ws.ctr_y, ws.ctr_z,
                                                                                rows, ws.pv_coef, cstride);
        }
        k_point_values<true><<<PSR_GRID(ws, nb), kBlock, 0, s>>>(ws.cnt, ws.depth, ws.px, ws.py, ws.pz, ws.point2node,
                                                                 ws.neigh, (size_t)ws.cap.nodes, ws.enc, ws.xsol, coarse,
                                                                 ws.point_val, ws.iso_partial);
        return cudaGetLastError();
    };
    if (ws.chain && !whole) {
        // One launch for every depth: clusters of at most 8 CTAs for the two finest, a CTA each for
        // the rest in the clusters behind them.  A chain without forks takes one hardware queue,
        // so that the resident slots of a server run side by side (the driver has 8 by default:
        // with three branches a graph, eight depth-5 clouds took 245 us each, 158 with 32 queues).  The
        // one CTA of depth 5 holds the pairs of 28,656 rows; samples throughout the box, which is enlarged 1.25
        // times, make 21,952 (16 served clouds of 200,000 samples, 2% of them scattered in the box: 24.1 ms
        // with all of depth 5 in global memory, 9.4 now).
        const int cs = ws.cg_ctas > 0 ? cl1 : (g_cg_cluster < 8 ? g_cg_cluster : 8);
        CgcArgs b = a;
        b.first = D;
        b.clusters = D < 2 ? D : 2;
        const int singles = D + 1 - b.clusters;
        e = launch_cg(k_cg_cluster, b, (b.clusters + (singles + cs - 1) / cs) * cs, cs, ws.batch, s);
        if (e != cudaSuccess) return e;
        if (ws.ev_cg) {
            e = cudaEventRecordWithFlags(ws.ev_cg, s, ws.ev_flags);
            if (e != cudaSuccess) return e;
        }
        return sample_values();
    }
    e = cudaEventRecord(ws.ev_fork, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ws.aux, ws.ev_fork, 0);
    if (e == cudaSuccess && ncl > 1) e = cudaStreamWaitEvent(ws.aux3, ws.ev_fork, 0);
    if (e == cudaSuccess && ncta > 0) {
        CgcArgs b = a;
        b.first = ncta - 1;
        b.clusters = ncta;
        e = launch_cg(k_cg_cluster, b, ncta, 1, ws.batch, ws.aux);   // clusters of one CTA
    }
    if (e != cudaSuccess) return e;
    if (whole) {
        // every depth is needed before the sample values: both parts join first
        e = launch_cg_grid(ws, a, s);
        if (e == cudaSuccess && ws.ev_cg) e = cudaEventRecordWithFlags(ws.ev_cg, s, ws.ev_flags);
        if (e == cudaSuccess) e = cudaEventRecord(ws.ev_join, ws.aux);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s, ws.ev_join, 0);
        return e == cudaSuccess ? sample_values() : e;
    }
    if (ncl > 1) {
        CgcArgs b = a;
        b.first = D - 1;
        b.clusters = ncl - 1;
        e = launch_cg(k_cg_cluster, b, (ncl - 1) * cl2, cl2, ws.batch, ws.aux3);
        if (e == cudaSuccess) e = cudaEventRecord(ws.ev_join3, ws.aux3);
        if (e != cudaSuccess) return e;
    }
    // the coarser levels' part of the sample values, as soon as every depth below D is
    // solved, beside the depth-D CG
    if (ncl > 1) e = cudaStreamWaitEvent(ws.aux, ws.ev_join3, 0);
    if (e == cudaSuccess) {
        k_point_poly<false><<<PSR_GRID(ws, ws.num_sms * 4), kBlock, 0, ws.aux>>>(ws.cnt, D, ws.ctr_x, ws.ctr_y, ws.ctr_z,
                                                                                 rows, ws.pv_coef, cstride);
        k_point_values_coarse<<<PSR_GRID(ws, nb), kBlock, 0, ws.aux>>>(ws.cnt, D, ws.px, ws.py, ws.pz, ws.point2node, coarse,
                                                                       ws.point_val);
        e = cudaEventRecord(ws.ev_join, ws.aux);
    }
    if (e != cudaSuccess) return e;
    if (ncl > 0) {
        a.first = D;
        a.clusters = 1;
        e = launch_cg(k_cg_cluster, a, cl1, cl1, ws.batch, s);
        if (e != cudaSuccess) return e;
    }
    if (ws.ev_cg) {
        e = cudaEventRecordWithFlags(ws.ev_cg, s, ws.ev_flags);
        if (e != cudaSuccess) return e;
    }
    e = cudaStreamWaitEvent(s, ws.ev_join, 0);
    if (e != cudaSuccess) return e;
    // iso-value: the depth-D terms complete the sample values
    k_point_values<false><<<PSR_GRID(ws, nb), kBlock, 0, s>>>(ws.cnt, ws.depth, ws.px, ws.py, ws.pz, ws.point2node,
                                                              ws.neigh, (size_t)ws.cap.nodes, ws.enc, ws.xsol, coarse,
                                                              ws.point_val, ws.iso_partial);
    return cudaGetLastError();
}

}  // namespace psr
