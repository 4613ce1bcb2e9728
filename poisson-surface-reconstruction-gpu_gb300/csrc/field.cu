// Stage (b): B-spline vector-field splat at the finest depth and per-node divergence.
//
// Vector field (mesh/ComputeVectorField.cu:61-100): for every D-level node o
//     V[o] = sum_{27 neighbours nb} sum_{points p in nb} B(p - c_o) n_p,
// B the separable normalised quadratic B-spline of width 2^-D, evaluated in the node's
// local coordinate (the reference expands shifted polynomials in float, which loses
// ~1e-4 relative accuracy at depth 7; the value is the same function).
// Divergence (mesh/ComputeNodesDivergence.cu:25-136): for every node o
//     div[o] = sum_{27 neighbours nb} sum_{D-level l under nb} V[l] . dff(o, l)
// with float terms (table entries rounded to float, as the reference's kernel does)
// accumulated as float pairs (TwoSum, ~44 bits; GB300's FP64 rate is far below FP32), in
// a fixed order.  The
// reference's coarse-depth host loop (one node at a time, :159-207) is replaced by one
// chunked reduction over all coarse nodes.
#include "workspace.h"
#include "tables.cuh"

PSR_DEFINE_CONST_TABLES(upload_tables_field)

namespace psr {

__device__ __forceinline__ float bspline32(float t) {
    const float kF43 = 1.33333337306976318359375f;
    const float kF23 = 0.666666686534881591796875f;
    const float a = fabsf(t), u = __fsub_rn(1.5f, a);
    const float inner = __fmul_rn(__fsub_rn(0.75f, __fmul_rn(t, t)), kF43);
    const float outer = __fmul_rn(__fmul_rn(u, u), kF23);
    return a < 0.5f ? inner : (a < 1.5f ? outer : 0.0f);
}

// 8 lanes per D-level node (4 nodes per warp): the 27 neighbours' sample ranges are
// flattened over the group's lanes (a group scan gives the range offsets), every lane
// accumulates its samples' weighted normals and a butterfly over the group combines the lanes (fixed
// order).  Bound by instruction issue.  Four lanes with two of the eight sums each are 1.7% faster in
// the field stage of 2,000,000 samples at depth 9 (1.67 against 1.70 ms), where a node has about ten
// samples around it, and slower wherever it has more: 200,000 samples at depth 6 84 against 70 us,
// 2,000,000 745 against 367.
constexpr int kVfLanes = 8;
constexpr int kVfGroups = kBlock / kVfLanes;
__global__ void __launch_bounds__(kBlock) k_vector_field(const Counters* c, int depth, const float* px, const float* py,
                                                         const float* pz, const float* nx, const float* ny,
                                                         const float* nz, const int* pidx, const int* pnum,
                                                         const float* cx, const float* cy, const float* cz,
                                                         const int* neigh, size_t stride, const int* enc, float* vx,
                                                         float* vy, float* vz, float4* leaf) {
    PSR_CLOUD(c, px, py, pz, nx, ny, nz, pidx, pnum, cx, cy, cz, neigh, enc, vx, vy, vz, leaf);
    __shared__ int s_off[kVfGroups][28];
    __shared__ int s_base[kVfGroups][27];
    const int md = c->level_count[depth];
    const int b = c->level_base[depth];
    const float s = (float)(1 << depth);
    const int lane = threadIdx.x & (kVfLanes - 1);
    const int gib = threadIdx.x / kVfLanes;
    const unsigned gmask = 0xffu << (threadIdx.x & 24);   // the group's lanes in its warp
    const int group = (blockIdx.x * blockDim.x + threadIdx.x) / kVfLanes;
    const int ngroups = (gridDim.x * blockDim.x) / kVfLanes;
    for (int o = group; o < md; o += ngroups) {
        const int i = b + o;
        const float ox = cx[i], oy = cy[i], oz = cz[i];
        int running = 0, used = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = lane + kVfLanes * r;
            int cnt = 0, base = 0;
            if (k < 27) {
                const int nb = neigh[(size_t)k * stride + i];
                if (nb >= 0) { base = pidx[nb]; cnt = pnum[nb]; }
            }
            list_range<kVfLanes>(gmask, cnt, base, s_off[gib], s_base[gib], used, running);
        }
        if (lane == 0) s_off[gib][used] = 0x7fffffff;
        __syncwarp(gmask);
        float ax = 0.f, ay = 0.f, az = 0.f;
        int k = 0;
        for (int t = lane; t < running; t += kVfLanes) {
            while (s_off[gib][k + 1] <= t) ++k;
            const int p = t + s_base[gib][k];
            const float w = bspline32((px[p] - ox) * s) * bspline32((py[p] - oy) * s) * bspline32((pz[p] - oz) * s);
            ax = fmaf(w, nx[p], ax);
            ay = fmaf(w, ny[p], ay);
            az = fmaf(w, nz[p], az);
        }
#pragma unroll
        for (int q = kVfLanes / 2; q > 0; q >>= 1) {
            ax += __shfl_xor_sync(gmask, ax, q);
            ay += __shfl_xor_sync(gmask, ay, q);
            az += __shfl_xor_sync(gmask, az, q);
        }
        if (lane == 0) {
            vx[o] = ax;
            vy[o] = ay;
            vz[o] = az;
            leaf[o] = make_float4(ax, ay, az, __int_as_float(enc[i]));
        }
        __syncwarp(gmask);
    }
}

__device__ __forceinline__ void decode3(int e, int depth, int& ix, int& iy, int& iz) {
    const int o1 = 1 << (depth + 1);
    ix = e & (o1 - 1);
    iy = (e >> (depth + 1)) & (o1 - 1);
    iz = e >> (2 * (depth + 1));
}

// Term of a leaf (its field and its packed function index, one 16-byte record) for a node whose
// rows of the function table are rx, ry, rz.  The parts below are bound by the latency of these
// dependent loads: with the record one load instead of four separate ones, field and divergence
// of a 2,000,000-sample depth-9 cloud take 2.49 ms instead of 2.62 (2.23 with the
// empty neighbours left out and the chunks in runs, below).
__device__ __forceinline__ float div_term(const float4 leaf, int depth, const float* rx, const float* ry,
                                          const float* rz) {
    int lx, ly, lz;
    decode3(__float_as_int(leaf.w), depth, lx, ly, lz);
    float t = __fmul_rn(leaf.x, rx[lx]);
    t = fmaf(leaf.y, ry[ly], t);
    return fmaf(leaf.z, rz[lz], t);
}

// Divergence arguments of a launch (the three parts below run side by side).
struct DivArgs {
    const Counters* c;
    int depth, dsplit, res;
    const int *enc, *didx, *dnum, *neigh;
    size_t stride;
    const float4* leaf;   // per depth-D node: its field, and its packed function index
    const float* dff;
    const unsigned* item_start;
    FF* partial;
    float* divg;
    __device__ void rebase() { PSR_CLOUD(c, enc, didx, dnum, neigh, leaf, dff, item_start, partial, divg); }
};

// Depth-D nodes: every neighbour holds exactly one depth-D leaf (itself), so a node's
// divergence has at most 27 terms; one thread per node sums them in slot order.
__device__ __forceinline__ void div_leaf(const DivArgs& a) {
    const int bD = a.c->level_base[a.depth];
    const int MD = a.c->level_count[a.depth];
    PSR_GRID_STRIDE(o, MD) {
        const int i = bD + o;
        int ox, oy, oz;
        decode3(a.enc[i], a.depth, ox, oy, oz);
        const float *rx = a.dff + (size_t)a.res * ox, *ry = a.dff + (size_t)a.res * oy, *rz = a.dff + (size_t)a.res * oz;
        int nb[27];
#pragma unroll
        for (int k = 0; k < 27; ++k) nb[k] = a.neigh[(size_t)k * a.stride + i];
        FF acc = ff_zero();
#pragma unroll
        for (int k = 0; k < 27; ++k)
            if (nb[k] >= 0) acc = ff_add_float(acc, div_term(a.leaf[nb[k] - bD], a.depth, rx, ry, rz));
        a.divg[i] = ff_to_float(acc);
    }
}

// One warp per node for depths dsplit .. D-1.  The (neighbour, leaf) pairs of the node are
// flattened over the lanes: lane k < 27 holds neighbour k's leaf range, a warp scan gives
// the range offsets, and term t belongs to the last neighbour whose offset is <= t.  Two thirds of
// the neighbours have no leaves; the list leaves them out, since every lane walks all of it.
__device__ __forceinline__ void div_fine(const DivArgs& a, int (*s_off)[33], int (*s_base)[32]) {
    const int b0 = a.c->level_base[a.dsplit];
    const int bD = a.c->level_base[a.depth];
    const int M = bD;   // depth-D nodes: div_leaf
    const int lane = lane_id();
    const int wib = threadIdx.x >> 5;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int i = b0 + warp; i < M; i += nwarps) {
        int ox, oy, oz;
        decode3(a.enc[i], a.depth, ox, oy, oz);
        const float *rx = a.dff + (size_t)a.res * ox, *ry = a.dff + (size_t)a.res * oy, *rz = a.dff + (size_t)a.res * oz;
        int cnt = 0, base = 0;
        if (lane < 27) {
            const int nb = a.neigh[(size_t)lane * a.stride + i];
            if (nb >= 0) { cnt = a.dnum[nb]; base = a.didx[nb]; }
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        // only neighbours with leaves, in slot order: where their terms start, and the leaf of term t
        // is t + s_base
        const unsigned some = __ballot_sync(0xffffffffu, cnt > 0);
        if (cnt > 0) {
            const int at = __popc(some & ((1u << lane) - 1u));
            s_off[wib][at] = incl - cnt;
            s_base[wib][at] = base - (incl - cnt);
        }
        if (lane == 0) s_off[wib][__popc(some)] = 0x7fffffff;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        __syncwarp();
        FF sum = ff_zero();
        int k = 0;
        for (int t = lane; t < total; t += 32) {
            while (s_off[wib][k + 1] <= t) ++k;   // terms are visited in increasing order
            sum = ff_add_float(sum, div_term(a.leaf[t + s_base[wib][k]], a.depth, rx, ry, rz));
        }
        const FF acc = ff_warp_sum(sum);
        if (lane == 0) a.divg[i] = ff_to_float(acc);
        __syncwarp();
    }
}

// Coarse depths (< dsplit), one warp per chunk: partial sum of up to kDivChunk leaves of one
// neighbour of one node
__device__ __forceinline__ void div_chunks(const DivArgs& a) {
    const int n_nodes = a.c->level_base[a.dsplit];
    const int n_items = a.c->n_div_items;
    const int lane = lane_id();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    // a warp takes consecutive items: it looks for a node once and keeps its neighbours' ranges until
    // the next node's items begin
    const int per = (n_items + nwarps - 1) / nwarps;
    const int it1 = min(n_items, (warp + 1) * per);
    int i = -1, start = 0, next = 0;   // the node and its items
    int dn = 0, di = 0, nc = 0, incl = 0;
    const float *rx = a.dff, *ry = a.dff, *rz = a.dff;
    for (int it = warp * per; it < it1; ++it) {
        if (i < 0 || it >= next) {
            int lo = 0, hi = n_nodes;   // item_start[lo] <= it < item_start[hi]
            if (i >= 0) {   // the next nodes, 32 at once
                while (true) {
                    const int at = i + 1 + lane;
                    const unsigned m = __ballot_sync(0xffffffffu, at < n_nodes && (int)a.item_start[at < n_nodes ? at : i] <= it);
                    lo = i + __popc(m);
                    if (m != 0xffffffffu) break;
                    i += 32;
                }
                hi = lo + 1;
            }
            while (hi - lo > 1) {   // each step the lanes probe 32 places of the range at once
                const int step = (hi - lo + 31) >> 5;
                const int at = lo + lane * step;
                const unsigned m = __ballot_sync(0xffffffffu, at < hi && (int)a.item_start[at < hi ? at : lo] <= it);
                const int last = 31 - __clz(m);   // lane 0 always holds
                lo += last * step;
                hi = min(hi, lo + step);
            }
            i = lo;
            start = (int)a.item_start[i];
            next = i + 1 < n_nodes ? (int)a.item_start[i + 1] : n_items;
            // lane k counts neighbour k's chunks
            int q = -1;
            dn = di = 0;
            if (lane < 27) {
                q = a.neigh[(size_t)lane * a.stride + i];
                if (q >= 0) { dn = a.dnum[q]; di = a.didx[q]; }
            }
            nc = (dn + kDivChunk - 1) / kDivChunk;
            incl = nc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            int ox, oy, oz;
            decode3(a.enc[i], a.depth, ox, oy, oz);
            rx = a.dff + (size_t)a.res * ox;
            ry = a.dff + (size_t)a.res * oy;
            rz = a.dff + (size_t)a.res * oz;
        }
        const int rem = it - start;
        const unsigned own = __ballot_sync(0xffffffffu, rem < incl);
        FF acc = ff_zero();
        if (own) {   // always
            const int k = __ffs(own) - 1;
            const int ch = rem - __shfl_sync(0xffffffffu, incl - nc, k);
            const int d0 = __shfl_sync(0xffffffffu, di, k), d1 = d0 + __shfl_sync(0xffffffffu, dn, k);
            const int l0 = d0 + ch * kDivChunk;
            const int l1 = min(d1, l0 + kDivChunk);
            FF sum = ff_zero();
#pragma unroll 4
            for (int l = l0 + lane; l < l1; l += 32) sum = ff_add_float(sum, div_term(a.leaf[l], a.depth, rx, ry, rz));
            acc = sum;
        }
        acc = ff_warp_sum(acc);
        if (lane == 0) a.partial[it] = acc;
    }
}

// The three parts only read the vector field: one launch, blockIdx.z a part (the longest first).
// Bound by instruction issue (two thirds of the slots) once enough warps hide the table look-ups:
// five blocks per SM, 48 registers with 24 bytes spilled (four: 2% slower at 500,000 samples, depth 9).
__global__ void __launch_bounds__(kBlock, 5) k_divergence(DivArgs a) {
    __shared__ int s_off[kBlock / 32][33];
    __shared__ int s_base[kBlock / 32][32];
    a.rebase();
    const int part = (int)blockIdx.z + (a.dsplit > 0 ? 0 : 1);
    if (part == 0) div_chunks(a);
    else if (part == 1) div_fine(a, s_off, s_base);
    else div_leaf(a);
}

// a warp per coarse node adds its chunks (the root has one per 512 leaves)
__global__ void __launch_bounds__(kBlock) k_div_coarse_reduce(DivArgs a) {
    a.rebase();
    const int n_nodes = a.c->level_base[a.dsplit];
    const int n_items = a.c->n_div_items;
    const int lane = lane_id();
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n_nodes; i += nwarps) {
        const int t0 = (int)a.item_start[i];
        const int t1 = (i + 1 < n_nodes) ? min((int)a.item_start[i + 1], n_items) : n_items;
        FF s = ff_zero();
        for (int t = t0 + lane; t < t1; t += 32) s = ff_add(s, a.partial[t]);
        s = ff_warp_sum(s);
        if (lane == 0) a.divg[i] = ff_to_float(s);
    }
}

cudaError_t field_build(Workspace& ws) {
    cudaStream_t s = ws.stream;
    const int D = ws.depth;
    Counters* c = ws.cnt;
    const size_t stride = (size_t)ws.cap.nodes;
    float* vx = ws.vfield;
    float* vy = ws.vfield + ws.cap.dnodes;
    float* vz = ws.vfield + 2 * (size_t)ws.cap.dnodes;
    k_vector_field<<<PSR_GRID(ws, ws.num_sms * 8), kBlock, 0, s>>>(c, D, ws.px, ws.py, ws.pz, ws.nx, ws.ny, ws.nz,
                                                                    ws.pidx, ws.pnum, ws.ctr_x, ws.ctr_y, ws.ctr_z,
                                                                    ws.neigh, stride, ws.enc, vx, vy, vz, ws.leaf);
    // item_start / partial live in the (otherwise idle) CG scratch; the chunks were counted and
    // numbered beside the mesh records
    const int dsplit = div_split(D);
    const DivArgs a{c, D, dsplit, ws.res, ws.enc, ws.didx, ws.dnum, ws.neigh, stride, ws.leaf, ws.dff,
                    (const unsigned*)ws.cg_p, reinterpret_cast<FF*>(ws.cg_partial), ws.divg};
    if (!ws.chain) {
        const cudaError_t e = cudaStreamWaitEvent(s, ws.ev_geo, 0);
        if (e != cudaSuccess) return e;
    }
    const dim3 g = PSR_GRID(ws, ws.num_sms * 8);
    k_divergence<<<dim3(g.x, g.y, dsplit > 0 ? 3 : 2), kBlock, 0, s>>>(a);
    if (dsplit > 0) k_div_coarse_reduce<<<PSR_GRID(ws, ws.num_sms * 4), kBlock, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace psr
