// Stage (a): normalisation, Morton encoding, radix sort, unique leaves, level-by-level
// octree with full 8-sibling groups, node information and the 27-neighbour table.
//
// Follows mesh/BuildOctree.cu / BuildOctree.cpp:75-194 of the reference (including its
// documented quirks) with a structure-of-arrays layout and device-resident counts.
#include "workspace.h"
#include "tables.cuh"

PSR_DEFINE_CONST_TABLES(upload_tables_octree)

namespace psr {

// ------------------------------------------------------------------------------------
// bounding box (mesh/BuildOctree.cu:51-133) and normalisation parameters (:619-631)
// ------------------------------------------------------------------------------------
// the counters of a call, and the sort's
// The call's input reference is read from the host's pinned memory, a slot per cloud.
__global__ void k_reset_counters(Counters* c, const InputRef* host_in, InputRef* in, unsigned* sort_bins, float* x) {
    PSR_CLOUD(c, in, sort_bins, x);
    static_assert(sizeof(Counters) % 4 == 0, "Counters is cleared word by word");
    unsigned* w = (unsigned*)c;
    for (int i = threadIdx.x; i < (int)(sizeof(Counters) / 4); i += blockDim.x) w[i] = 0u;
    for (int i = threadIdx.x; i < kSortBinWords; i += blockDim.x) sort_bins[i] = 0u;
    __syncthreads();
    if (threadIdx.x == 0) {
        x[-1] = 0.0f;   // the value of absent neighbours
        const InputRef ref = host_in[blockIdx.y];
        *in = ref;
        c->n_points = c->n_input = ref.n;
        for (int a = 0; a < 3; ++a) {
            // The reference seeds its reduction (padding threads, mesh/BuildOctree.cu:66-73)
            // and its host finish (mesh/BuildOctree.cpp:87-88) with -1e6 / 1e6, which gives a
            // wrong box when every coordinate of an axis lies beyond 1e6 in magnitude (a
            // georeferenced scan).  Seeding with -FLT_MAX / FLT_MAX gives the reference's box
            // for every other input and the true box for those.
            ((int*)c->bbox_max)[a] = float_to_ordered(-FLT_MAX);
            ((int*)c->bbox_min)[a] = float_to_ordered(FLT_MAX);
        }
    }
}

// Bounding box; the last block to finish sets the normalisation parameters (a launch of one
// thread of their own would cost as much as the box).
__global__ void __launch_bounds__(kBlock) k_bbox(const InputRef* in, Counters* c, float scale) {
    PSR_CLOUD(in, c);
    const float* xyz = in->xyz;
    const float* nrm = in->nrm;
    const int n = c->n_points;
    float mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX}, mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
    bool bad = false;
    PSR_GRID_STRIDE(i, n) {
        for (int a = 0; a < 3; ++a) {
            float v = xyz[3 * (size_t)i + a];
            float w = nrm[3 * (size_t)i + a];
            if (!isfinite(v) || !isfinite(w)) bad = true;
            mx[a] = mx[a] < v ? v : mx[a];
            mn[a] = mn[a] > v ? v : mn[a];
        }
    }
    for (int a = 0; a < 3; ++a) {
        for (int o = 16; o > 0; o >>= 1) {
            mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
            mn[a] = fminf(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane_id() == 0) atomicOr(&c->error, kErrInvalid);
    // block reduction, then one set of atomics per block
    __shared__ float s_mx[3][kBlock / 32], s_mn[3][kBlock / 32];
    __shared__ int s_last;
    const int w = threadIdx.x >> 5;
    if (lane_id() == 0)
        for (int a = 0; a < 3; ++a) { s_mx[a][w] = mx[a]; s_mn[a][w] = mn[a]; }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int a = threadIdx.x;
        float bmx = s_mx[a][0], bmn = s_mn[a][0];
        for (int q = 1; q < kBlock / 32; ++q) { bmx = fmaxf(bmx, s_mx[a][q]); bmn = fminf(bmn, s_mn[a][q]); }
        atomicMax(&((int*)c->bbox_max)[a], float_to_ordered(bmx));
        atomicMin(&((int*)c->bbox_min)[a], float_to_ordered(bmn));
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&c->ticket[0], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    float bx[3], bn[3];
    for (int a = 0; a < 3; ++a) {
        bx[a] = ordered_to_float(__ldcg(&((int*)c->bbox_max)[a]));
        bn[a] = ordered_to_float(__ldcg(&((int*)c->bbox_min)[a]));
        c->bbox_max[a] = bx[a];
        c->bbox_min[a] = bn[a];
    }
    float edge = 1.0f;
    float ctr[3];
    for (int a = 0; a < 3; ++a) {
        float ext = __fsub_rn(bx[a], bn[a]);
        if (a == 0 || edge < ext) edge = ext;
        ctr[a] = __fdiv_rn(__fadd_rn(bx[a], bn[a]), 2.0f);
    }
    edge = __fmul_rn(edge, __fmul_rn(scale, 1.0f));
    for (int a = 0; a < 3; ++a) ctr[a] = __fsub_rn(ctr[a], __fdiv_rn(edge, 2.0f));
    for (int a = 0; a < 3; ++a) c->center[a] = ctr[a];
    c->max_edge = edge;
    if (!(edge > 0.0f)) atomicOr(&c->error, kErrInvalid);
}

__device__ __forceinline__ float normalise_coord(float v, float ctr, float edge) {
    // (p - c) * 1.0f / maxEdge evaluated left to right (mesh/BuildOctree.cu:149)
    return __fdiv_rn(__fmul_rn(__fsub_rn(v, ctr), 1.0f), edge);
}

// Morton code of a normalised point (mesh/BuildOctree.cu:167-208); bit 3l+2 = x of level
// D-l, so the code equals the reference key's upper 32 bits.  Counts the sort's digits.
__global__ void __launch_bounds__(kBlock) k_encode(const InputRef* in, Counters* c, int depth, unsigned* code,
                                                   SortScratch sc, int passes) {
    PSR_CLOUD(in, c, code, sc);
    __shared__ unsigned s_h[kSortMaxPasses][kRadix];
    const SortCounter count{s_h, passes};
    count.clear();
    const float* xyz = in->xyz;
    const int n = c->n_points;
    const float c0 = c->center[0], c1 = c->center[1], c2 = c->center[2], e = c->max_edge;
    PSR_GRID_STRIDE(i, n) {
        float p[3] = {normalise_coord(xyz[3 * (size_t)i], c0, e), normalise_coord(xyz[3 * (size_t)i + 1], c1, e),
                      normalise_coord(xyz[3 * (size_t)i + 2], c2, e)};
        unsigned k = 0;
        float cc[3] = {0.5f, 0.5f, 0.5f};
        float w = 0.25f;
        for (int l = depth - 1; l >= 0; --l) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (p[a] > cc[a]) { k |= 1u << (3 * l + 2 - a); cc[a] = __fadd_rn(cc[a], w); }
                else cc[a] = __fsub_rn(cc[a], w);
            }
            w = __fmul_rn(w, 0.5f);
        }
        code[i] = k;
        count.count(k);
    }
    count.finish(sc, n, &c->ticket[1], &c->error);
}

// Gathers the sorted points, scales the normals to 2^(D+1) (mesh/BuildOctree.cu:152-164) and
// flags the first point of every unique leaf; the scan over the flags gives point -> unique leaf
// id and unique leaf -> code, first point.
struct GatherLoad {
    const InputRef* in;
    const unsigned* scode;
    const unsigned* sidx;
    const Counters* c;
    int depth;
    float *px, *py, *pz, *nx, *ny, *nz, *cr, *cg, *cb;
    __device__ unsigned operator()(int i) const {
        const float* xyz = in->xyz;
        const float* nrm = in->nrm;
        const uint8_t* rgb = in->rgb;
        const float c0 = c->center[0], c1 = c->center[1], c2 = c->center[2], e = c->max_edge;
        const float nscale = (float)(2 << depth);
        const size_t o = sidx[i];
        // every read of the scattered sample before the first store, which the compiler could not
        // move a read across (106 -> 85 us for 2,000,000 samples)
        const float x = xyz[3 * o], y = xyz[3 * o + 1], z = xyz[3 * o + 2];
        float a = nrm[3 * o], b = nrm[3 * o + 1], d = nrm[3 * o + 2];
        uint8_t r = 0, g = 0, bl = 0;
        if (rgb) { r = rgb[3 * o]; g = rgb[3 * o + 1]; bl = rgb[3 * o + 2]; }
        const unsigned code = scode[i], before = i ? scode[i - 1] : ~code;
        px[i] = normalise_coord(x, c0, e);
        py[i] = normalise_coord(y, c1, e);
        pz[i] = normalise_coord(z, c2, e);
        float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b)), __fmul_rn(d, d)));
        // reference quirk: a normal no longer than 1e-6 is multiplied by its length
        if (len > 1e-6f) len = __fdiv_rn(1.0f, len);
        len = __fmul_rn(len, nscale);
        nx[i] = __fmul_rn(a, len);
        ny[i] = __fmul_rn(b, len);
        nz[i] = __fmul_rn(d, len);
        if (rgb) {
            cr[i] = __fdiv_rn((float)r, 255.0f);
            cg[i] = __fdiv_rn((float)g, 255.0f);
            cb[i] = __fdiv_rn((float)bl, 255.0f);
        } else {
            cr[i] = cg[i] = cb[i] = 0.0f;
        }
        return code != before ? 1u : 0u;
    }
    __device__ void rebase() { PSR_CLOUD(in, scode, sidx, c, px, py, pz, nx, ny, nz, cr, cg, cb); }   // to cloud blockIdx.y
};
struct HeadStore {
    const unsigned* scode;
    Counters* c;
    int* puid;
    unsigned* ucode;
    int* ufirst;
    __device__ void operator()(int i, unsigned pre, unsigned v) const {
        int u = (int)(pre + v) - 1;
        puid[i] = u;
        if (v) { ucode[u] = scode[i]; ufirst[u] = i; }
    }
    __device__ void done(unsigned total) const {
        c->n_unique = (int)total;
        ufirst[total] = c->n_points;
    }
    __device__ void rebase() { PSR_CLOUD(scode, c, puid, ucode, ufirst); }   // to cloud blockIdx.y
};

// Level staging arrays: one record per slot of a level being built.
struct LevelArrays {
    int *key, *pidx, *pnum, *didx, *dnum, *child;
    __device__ void put(int t, int k, int pi, int pn, int di, int dn, int ch) const {
        key[t] = k;
        pidx[t] = pi;
        pnum[t] = pn;
        didx[t] = di;
        dnum[t] = dn;
        child[t] = ch;
    }
    __device__ void rebase() { PSR_CLOUD(key, pidx, pnum, didx, dnum, child); }   // to cloud blockIdx.y
};

// D-level groups: 8 slots for every new parent code (mesh/BuildOctree.cu:267-280)
struct LeafGroupLoad {
    const unsigned* ucode;
    __device__ unsigned operator()(int u) const {
        return (u == 0) ? 0u : (((ucode[u - 1] >> 3) != (ucode[u] >> 3)) ? 8u : 0u);
    }
    __device__ void rebase() { PSR_CLOUD(ucode); }   // to cloud blockIdx.y
};
// Places every unique leaf in its group's slot (:282-292), with the empty slots up to the next
// leaf's (each slot is written once; D level: dnum = 1, didx = slot, :294-300).
struct LeafPlaceStore {
    const unsigned* ucode;
    const int* ufirst;
    Counters* c;
    int depth, cap;
    int* uslot;
    LevelArrays T;
    unsigned* err;
    __device__ void operator()(int u, unsigned pre, unsigned v) const {
        const int n = c->n_unique;
        const unsigned code = ucode[u];
        const int addr = (int)(pre + v), s = addr + (int)(code & 7u);
        uslot[u] = s;
        int end = addr + 8;   // first slot past the empty ones behind this leaf
        if (u + 1 < n) {
            const unsigned nc = ucode[u + 1];
            end = addr + (((nc >> 3) != (code >> 3)) ? 8 : 0) + (int)(nc & 7u);
        }
        if (end > cap) end = cap;   // capacity overflow (flagged by done())
        if (u == 0)
            for (int q = 0; q < s; ++q) T.put(q, 0, 0, 0, q, 1, -1);
        if (s < cap) T.put(s, (int)code, ufirst[u], ufirst[u + 1] - ufirst[u], s, 1, -1);
        for (int q = s + 1; q < end; ++q) T.put(q, 0, 0, 0, q, 1, -1);
    }
    __device__ void done(unsigned total) const {
        int md = (int)total + 8;
        if (c->n_unique == 0) md = 0;
        c->level_tmp_off[depth] = 0;
        if (md > cap) { atomicOr(err, kErrCapacity); md = 0; }
        c->level_count[depth] = md;
        c->level_groups[depth] = md / 8;
    }
    __device__ void rebase() { PSR_CLOUD(ucode, ufirst, c, uslot, T, err); }   // to cloud blockIdx.y
};

// the 8 entries of a group (a group starts on a 32-byte boundary of its array)
__device__ __forceinline__ void load8(const int* p, int (&v)[8]) {
    const int4 a = *reinterpret_cast<const int4*>(p), b = *reinterpret_cast<const int4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// first non-empty slot of group g's 8 (the father's key is its key without the sibling bits)
__device__ __forceinline__ int group_father_key(const LevelArrays& T, int base, int sh) {
    int pn[8];
    load8(T.pnum + base, pn);
    int at = -1;
#pragma unroll
    for (int j = 7; j >= 0; --j)
        if (pn[j] != 0) at = j;
    return at < 0 ? 0 : T.key[base + at] & ~(7 << sh);
}
// One level of the build: the sibling groups of level d aggregate into their fathers
// (mesh/BuildOctree.cu:323-357), a scan over the groups that start a new father group gives the
// father groups' addresses one level up (:359-375, :796-799), and every father goes to its slot
// with the empty slots up to the next father's (:377-390).
struct LevelLoad {
    const Counters* c;
    int d, depth;
    LevelArrays T;
    int *gkey, *gpidx, *gpnum, *gdidx, *gdnum;
    __device__ unsigned operator()(int g) const {
        const int off = c->level_tmp_off[d];
        const int sh = 3 * (depth - d), sh2 = 3 * (depth - d + 2);
        int fk = 0, pn = 0, pi = 0x7fffffff, dn = 0, di = 0x7fffffff;
        const int t = off + 8 * g;
        int pnum[8], dnum[8], didx[8], key[8], pidx[8];
        load8(T.pnum + t, pnum);
        load8(T.dnum + t, dnum);
        load8(T.didx + t, didx);
        load8(T.key + t, key);
        load8(T.pidx + t, pidx);
        const int before = g > 0 ? group_father_key(T, t - 8, sh) : 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (pnum[j] == 0) {
                if (dnum[j] != 0) { dn += dnum[j]; di = min(di, didx[j]); }
            } else {
                fk = key[j] & ~(7 << sh);
                pn += pnum[j];
                pi = min(pi, pidx[j]);
                dn += dnum[j];
                di = min(di, didx[j]);
            }
        }
        gkey[g] = fk;
        gpidx[g] = pi;
        gpnum[g] = pn;
        gdidx[g] = di;
        gdnum[g] = dn;
        if (g == 0) return 0u;
        return ((before >> sh2) != (fk >> sh2)) ? 8u : 0u;
    }
    __device__ void rebase() { PSR_CLOUD(c, T, gkey, gpidx, gpnum, gdidx, gdnum); }   // to cloud blockIdx.y
};
struct LevelStore {
    Counters* c;
    int d, depth, cap;
    LevelArrays T;
    const int *gkey, *gpidx, *gpnum, *gdidx, *gdnum;   // group g's entries: written by the same thread's load
    int* tparent_slot;
    unsigned* err;
    __device__ void operator()(int g, unsigned pre, unsigned v) const {
        const int off = c->level_tmp_off[d], m = c->level_count[d];
        const int sh = 3 * (depth - d), sh2 = 3 * (depth - d + 2), sh3 = 3 * (depth - d + 1);
        const int off1 = off + m;   // first slot of level d - 1
        const int fk = gkey[g];
        const int addr = (int)(pre + v), s = addr + ((fk >> sh3) & 7);
        int end = d > 1 ? addr + 8 : 1;
        if (8 * (g + 1) < m) {
            const int nk = group_father_key(T, off + 8 * (g + 1), sh);
            end = addr + (((nk >> sh2) != (fk >> sh2)) ? 8 : 0) + ((nk >> sh3) & 7);
        }
        if (off1 + end > cap) end = cap - off1;   // capacity overflow (flagged by done())
        if (g == 0)
            for (int q = 0; q < s && off1 + q < cap; ++q) T.put(off1 + q, 0, 0, 0, 0, 0, -1);
        if (off1 + s < cap) T.put(off1 + s, fk, gpidx[g], gpnum[g], gdidx[g], gdnum[g], 8 * g);
        for (int q = s + 1; q < end; ++q) T.put(off1 + q, 0, 0, 0, 0, 0, -1);
        tparent_slot[off / 8 + g] = s;
    }
    __device__ void done(unsigned total) const {
        int m = (d > 1) ? (int)total + 8 : 1;
        const int off = c->level_tmp_off[d] + c->level_count[d];
        c->level_tmp_off[d - 1] = off;
        if (off + m > cap) { atomicOr(err, kErrCapacity); m = 0; }
        c->level_count[d - 1] = m;
        c->level_groups[d - 1] = m / 8;
    }
    __device__ void rebase() { PSR_CLOUD(c, T, gkey, gpidx, gpnum, gdidx, gdnum, tparent_slot, err); }   // to cloud blockIdx.y
};

// ---- coarse levels in one CTA --------------------------------------------------------
// The levels near the root hold few nodes, so their per-level passes (group aggregate,
// father-group scan, level set-up, father placement) run inside one 1024-thread CTA with
// block barriers between steps instead of a scan of their own per level.  Same arithmetic as
// the per-level scans above.
constexpr int kLevelBlock = 1024;
constexpr int kCoarseLevels = 4;   // levels up to this one: at most 4096 nodes, 4 rounds of the CTA

// inclusive block scan of one value per thread (1024 threads); returns the block total
__device__ __forceinline__ unsigned block_inclusive_scan_1024(unsigned v, unsigned* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    if (warp == 0) {
        unsigned w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        s_warp[lane] = w;   // inclusive warp totals
    }
    __syncthreads();
    const unsigned r = v + (warp > 0 ? s_warp[warp - 1] : 0u);
    const unsigned total = s_warp[31];
    __syncthreads();
    s_warp[32] = total;
    return r;
}

// Every level is counted: their places in the node arrays.  A tree that outgrew its arrays is left
// without nodes and points, because its records stop at the capacity and the later stages would follow
// indices into records that were never written.
__device__ __forceinline__ void levels_done(Counters* c, int depth) {
    int b = 0;
    if (atomicOr(&c->error, 0u) & kErrCapacity) {
        c->n_points = 0;
        for (int d = 0; d <= depth; ++d) c->level_count[d] = 0;
    }
    for (int d = 0; d <= depth; ++d) {
        c->level_base[d] = b;
        b += c->level_count[d];
    }
    c->n_nodes = b;
}

__global__ void __launch_bounds__(kLevelBlock) k_levels_block(Counters* c, int dtop, int depth, int* tkey, int* tpidx,
                                                              int* tpnum, int* tdidx, int* tdnum, int* tchild,
                                                              int* tparent_slot, int* gkey, int* gpidx, int* gpnum,
                                                              int* gdidx, int* gdnum, unsigned* gaddr, int node_cap) {
    PSR_CLOUD(c, tkey, tpidx, tpnum, tdidx, tdnum, tchild, tparent_slot, gkey, gpidx, gpnum, gdidx, gdnum, gaddr);
    __shared__ unsigned s_warp[33];
    const int t = threadIdx.x;
    for (int d = dtop; d >= 1; --d) {
        const int m = c->level_count[d];
        const int off = c->level_tmp_off[d];
        const int G = m / 8;
        const int sh = 3 * (depth - d);
        // (1) sibling groups of level d -> father candidates
        for (int g = t; g < G; g += kLevelBlock) {
            int fk = 0, pn = 0, pi = 0x7fffffff, dn = 0, di = 0x7fffffff;
            for (int j = 0; j < 8; ++j) {
                const int q = off + 8 * g + j;
                const int pnum = tpnum[q], dnum = tdnum[q], didx = tdidx[q];
                if (pnum == 0) {
                    if (dnum != 0) { dn += dnum; di = min(di, didx); }
                } else {
                    fk = tkey[q] & ~(7 << sh);
                    pn += pnum;
                    pi = min(pi, tpidx[q]);
                    dn += dnum;
                    di = min(di, didx);
                }
            }
            gkey[g] = fk;
            gpidx[g] = pi;
            gpnum[g] = pn;
            gdidx[g] = di;
            gdnum[g] = dn;
        }
        __syncthreads();
        // (2) inclusive scan of "new father group" flags (8 per new group of level d-1)
        const int sh2 = 3 * (depth - d + 2);
        unsigned carry = 0;
        for (int b = 0; b < G; b += kLevelBlock) {
            const int g = b + t;
            const unsigned f = (g < G && g > 0) ? (((gkey[g - 1] >> sh2) != (gkey[g] >> sh2)) ? 8u : 0u) : 0u;
            const unsigned incl = block_inclusive_scan_1024(f, s_warp);
            if (g < G) gaddr[g] = carry + incl;
            carry += s_warp[32];
            __syncthreads();
        }
        // (3) size and offset of level d-1
        int m1 = (d > 1) ? (int)carry + 8 : 1;
        const int off1 = off + m;
        if (off1 + m1 > node_cap) {
            if (t == 0) atomicOr(&c->error, kErrCapacity);
            m1 = 0;
        }
        if (t == 0) {
            c->level_count[d - 1] = m1;
            c->level_tmp_off[d - 1] = off1;
            c->n_groups = G;
        }
        for (int i = t; i < m1; i += kLevelBlock) {
            tkey[off1 + i] = 0;
            tpidx[off1 + i] = 0;
            tpnum[off1 + i] = 0;
            tdidx[off1 + i] = 0;
            tdnum[off1 + i] = 0;
            tchild[off1 + i] = -1;
        }
        __syncthreads();
        // (4) fathers into their slots of level d-1
        const int off_group = off / 8;
        const int sh3 = 3 * (depth - d + 1);
        for (int g = t; g < G; g += kLevelBlock) {
            const int sl = (int)gaddr[g] + ((gkey[g] >> sh3) & 7);
            if (sl >= m1) continue;   // capacity overflow (flagged)
            const int q = off1 + sl;
            tkey[q] = gkey[g];
            tpidx[q] = gpidx[g];
            tpnum[q] = gpnum[g];
            tdidx[q] = gdidx[g];
            tdnum[q] = gdnum[g];
            tchild[q] = 8 * g;
            tparent_slot[off_group + g] = sl;
        }
        __syncthreads();
    }
    if (t == 0) levels_done(c, depth);
}

// 27-neighbour tables of levels 1..dmax in one CTA (levels in order: a level reads its
// parents' table).  1024 threads leave 64 registers each: 56 bytes of the row spill.
__global__ void __launch_bounds__(kLevelBlock) k_neighbours_block(const Counters* c, int dmax, int depth,
                                                                  const int* key, const int* parent,
                                                                  const int* first_child, int* neigh, size_t stride) {
    PSR_CLOUD(c, key, parent, first_child, neigh);
    for (int d = 1; d <= dmax; ++d) {
        const int m = c->level_count[d];
        const int b = c->level_base[d];
        for (int li = threadIdx.x; li < m; li += kLevelBlock) {
            const int i = b + li;
            const int son = (key[i] >> (3 * (depth - d))) & 7;
            const int pa = parent[i];
            // every read before the first store: the look-ups overlap
            int v[27];
            child_neighbours(son, [&](int j) { return neigh[(size_t)j * stride + pa]; },
                             [&](int n) { return first_child[n]; }, v);
#pragma unroll
            for (int k = 0; k < 27; ++k) neigh[(size_t)k * stride + i] = v[k];
        }
        __syncthreads();
    }
}

__global__ void k_levels_done(Counters* c, int depth) {
    PSR_CLOUD(c);
    if (threadIdx.x == 0 && blockIdx.x == 0) levels_done(c, depth);
}

// Final node records (mesh/BuildOctree.cu:392-488, :552-586, :514-550), the root's neighbour row
// and the points' leaves (:302-313).
__global__ void __launch_bounds__(kBlock) k_finalize_nodes(const Counters* c, int depth, const int* tkey,
                                                           const int* tpidx, const int* tpnum, const int* tdidx,
                                                           const int* tdnum, const int* tchild,
                                                           const int* tparent_slot, int* key, int* pidx, int* pnum,
                                                           int* parent, int* first_child, int* didx, int* dnum,
                                                           int* ndepth, int* enc, float* cx, float* cy, float* cz,
                                                           int* neigh, size_t stride, const int* puid, const int* uslot,
                                                           int* point2node) {
    PSR_CLOUD(c, tkey, tpidx, tpnum, tdidx, tdnum, tchild, tparent_slot, key, pidx, pnum, parent, first_child, didx, dnum, ndepth, enc, cx, cy, cz, neigh, puid, uslot, point2node);
    const int np = c->n_points;
    PSR_GRID_STRIDE(i, np) point2node[i] = uslot[puid[i]];
    if (blockIdx.x == 0 && threadIdx.x < 27) neigh[(size_t)threadIdx.x * stride] = (threadIdx.x == 13) ? 0 : -1;
    const int M = c->n_nodes;
    PSR_GRID_STRIDE(i, M) {
        int d = 0;
        while (d < depth && i >= c->level_base[d + 1]) ++d;
        const int li = i - c->level_base[d];
        const int off = c->level_tmp_off[d];
        const int t = off + li;
        int k, pi, pn, dn, di, par, fc;
        pn = tpnum[t];
        dn = tdnum[t];
        if (d == 0) {
            k = tkey[t];
            pi = tpidx[t];
            di = tdidx[t];
            par = -1;
            fc = 1;   // root children are 1..8 (:403-410)
        } else {
            const int sh = 3 * (depth - d);
            const int g = li >> 3, j = li & 7;
            const int gs = off + 8 * g;
            int gp[8], gd[8];   // the group's counts (a group starts on a 32-byte boundary)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int4 p4 = *reinterpret_cast<const int4*>(tpnum + gs + 4 * q);
                const int4 d4 = *reinterpret_cast<const int4*>(tdnum + gs + 4 * q);
                gp[4 * q] = p4.x; gp[4 * q + 1] = p4.y; gp[4 * q + 2] = p4.z; gp[4 * q + 3] = p4.w;
                gd[4 * q] = d4.x; gd[4 * q + 1] = d4.y; gd[4 * q + 2] = d4.z; gd[4 * q + 3] = d4.w;
            }
            int v = 0;   // the first non-empty node (0: cannot happen, every group holds one)
#pragma unroll
            for (int q = 7; q >= 0; --q)
                if (gp[q] != 0) v = q;
            k = (tkey[gs + v] & ~(7 << sh)) | (j << sh);
            int nowP = tpidx[gs + v], nowD = tdidx[gs + v];
#pragma unroll
            for (int q = 0; q < 7; ++q)
                if (q < j) { nowP += gp[q]; nowD += gd[q]; }
            pi = nowP;
            di = (d == depth) ? tdidx[t] : nowD;
            // reference quirk: the first non-empty node of the group passes its parent to
            // all siblings, and a node at level-local index 0 never had its parent set
            const int lp = (g == 0 && v == 0) ? 0 : tparent_slot[off / 8 + g];
            par = c->level_base[d - 1] + lp;
            fc = (pn != 0 && d < depth) ? c->level_base[d + 1] + tchild[t] : -1;
        }
        key[i] = k;
        pidx[i] = pi;
        pnum[i] = pn;
        parent[i] = par;
        first_child[i] = fc;
        didx[i] = di;
        dnum[i] = dn;
        ndepth[i] = d;
        float cc[3] = {0.5f, 0.5f, 0.5f};
        float w = 0.25f;
        for (int l = depth - 1; l >= depth - d; --l) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if ((k >> (3 * l + 2 - a)) & 1) cc[a] = __fadd_rn(cc[a], w);
                else cc[a] = __fsub_rn(cc[a], w);
            }
            w = __fmul_rn(w, 0.5f);
        }
        cx[i] = cc[0];
        cy[i] = cc[1];
        cz[i] = cc[2];
        int e = ((1 << d) - 1) * (1 + (1 << (depth + 1)) + (1 << (2 * (depth + 1))));
        for (int l = d; l >= 1; --l) {
            int sx = (k >> (3 * (depth - l) + 2)) & 1;
            int sy = (k >> (3 * (depth - l) + 1)) & 1;
            int sz = (k >> (3 * (depth - l))) & 1;
            e += sx * (1 << (d - l)) + sy * (1 << (d - l)) * (1 << (depth + 1)) +
                 sz * (1 << (d - l)) * (1 << (2 * (depth + 1)));
        }
        enc[i] = e;
    }
}

// 27-neighbour table of one depth (mesh/BuildOctree.cu:490-512), stored [27][cap]
__global__ void __launch_bounds__(kBlock) k_neighbours(const Counters* c, int d, int depth, const int* key,
                                                       const int* parent, const int* first_child, int* neigh,
                                                       size_t stride) {
    PSR_CLOUD(c, key, parent, first_child, neigh);
    const int m = c->level_count[d];
    const int b = c->level_base[d];
    PSR_GRID_STRIDE(li, m) {
        const int i = b + li;
        const int son = (key[i] >> (3 * (depth - d))) & 7;
        const int pa = parent[i];
        int v[27];
        child_neighbours(son, [&](int j) { return neigh[(size_t)j * stride + pa]; },
                         [&](int n) { return first_child[n]; }, v);
#pragma unroll
        for (int k = 0; k < 27; ++k) neigh[(size_t)k * stride + i] = v[k];
    }
}

// points -> Morton codes of the reference's normalised coordinates at `depth`, sorted with
// their input indices (the octree's first steps; the normal estimation stage uses them on
// their own).  The input reference, n_points, the bounding-box seeds and the sort's bins must be
// set.
cudaError_t encode_sort_points(Workspace& ws, int depth, const unsigned** scode, const unsigned** sidx) {
    cudaStream_t s = ws.stream;
    Counters* c = ws.cnt;
    const int gp = grid_for(ws, ws.cap.points);
    k_bbox<<<PSR_GRID(ws, gp), kBlock, 0, s>>>(ws.d_params, c, 1.25f);
    k_encode<<<PSR_GRID(ws, gp), kBlock, 0, s>>>(ws.d_params, c, depth, ws.code, ws.sort, sort_passes(3 * depth));
    bool alt = false;
    cudaError_t e = radix_sort_pairs(ws.code, ws.sidx, &c->n_points, 3 * depth, ws.sort, &c->error, s, &alt);
    if (e != cudaSuccess) return e;
    *scode = alt ? ws.sort.keys_alt : ws.code;
    *sidx = alt ? ws.sort.vals_alt : ws.sidx;
    return cudaGetLastError();
}

cudaError_t octree_build(Workspace& ws) {
    cudaStream_t s = ws.stream;
    const int D = ws.depth;
    Counters* c = ws.cnt;
    unsigned* err = &c->error;
    unsigned* total = (unsigned*)&c->scan_total;
    k_reset_counters<<<PSR_GRID(ws, 1), 256, 0, s>>>(c, ws.h_params, ws.d_params, ws.sort.bins, ws.xsol);
    const unsigned *scode = nullptr, *sidx = nullptr;
    cudaError_t e = encode_sort_points(ws, D, &scode, &sidx);
    if (e != cudaSuccess) return e;
    e = launch_scan<2>(GatherLoad{ws.d_params, scode, sidx, c, D, ws.px, ws.py, ws.pz, ws.nx, ws.ny, ws.nz, ws.cr, ws.cg, ws.cb},
                       HeadStore{scode, c, ws.puid, ws.ucode, ws.ufirst}, &c->n_points, 0, ws.scan, total, err, s);
    if (e != cudaSuccess) return e;
    const LevelArrays T{ws.tkey, ws.tpidx, ws.tpnum, ws.tdidx, ws.tdnum, ws.tchild};
    e = launch_scan<2>(LeafGroupLoad{ws.ucode},
                       LeafPlaceStore{ws.ucode, ws.ufirst, c, D, ws.cap.dnodes, ws.uslot, T, err}, &c->n_unique, 0,
                       ws.scan, total, err, s, ScanCount{}, 2);
    if (e != cudaSuccess) return e;
    // levels D .. dfuse+1 level by level across the GPU, the levels near the root (at most 4096
    // nodes each) in one CTA
    const int dfuse = D - 1 < kCoarseLevels ? D - 1 : kCoarseLevels;
    for (int d = D; d > dfuse; --d) {
        e = launch_scan<1>(LevelLoad{c, d, D, T, ws.gkey, ws.gpidx, ws.gpnum, ws.gdidx, ws.gdnum},
                           LevelStore{c, d, D, ws.cap.nodes, T, ws.gkey, ws.gpidx, ws.gpnum, ws.gdidx, ws.gdnum,
                                      ws.tparent_slot, err},
                           &c->level_groups[d], 0, ws.scan, total, err, s, ScanCount{}, 2);
        if (e != cudaSuccess) return e;
    }
    if (dfuse >= 1)
        k_levels_block<<<PSR_GRID(ws, 1), kLevelBlock, 0, s>>>(c, dfuse, D, ws.tkey, ws.tpidx, ws.tpnum, ws.tdidx, ws.tdnum, ws.tchild,
                                                 ws.tparent_slot, ws.gkey, ws.gpidx, ws.gpnum, ws.gdidx, ws.gdnum,
                                                 ws.gaddr, ws.cap.nodes);
    else
        k_levels_done<<<PSR_GRID(ws, 1), 1, 0, s>>>(c, D);
    const int gm = grid_for(ws, ws.cap.nodes);
    const size_t stride = (size_t)ws.cap.nodes;
    k_finalize_nodes<<<PSR_GRID(ws, gm), kBlock, 0, s>>>(c, D, ws.tkey, ws.tpidx, ws.tpnum, ws.tdidx, ws.tdnum, ws.tchild,
                                           ws.tparent_slot, ws.key, ws.pidx, ws.pnum, ws.parent, ws.first_child,
                                           ws.didx, ws.dnum, ws.ndepth, ws.enc, ws.ctr_x, ws.ctr_y, ws.ctr_z, ws.neigh,
                                           stride, ws.puid, ws.uslot, ws.point2node);
    if (dfuse >= 1)
        k_neighbours_block<<<PSR_GRID(ws, 1), kLevelBlock, 0, s>>>(c, dfuse, D, ws.key, ws.parent, ws.first_child, ws.neigh, stride);
    for (int d = (dfuse >= 1 ? dfuse + 1 : 1); d <= D; ++d)
        k_neighbours<<<PSR_GRID(ws, gm), kBlock, 0, s>>>(c, d, D, ws.key, ws.parent, ws.first_child, ws.neigh, stride);
    return cudaGetLastError();
}

}  // namespace psr
