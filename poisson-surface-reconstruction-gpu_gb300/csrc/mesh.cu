// Stage (d): vertex / edge / face arrays, marching cubes at the finest depth, subdivision
// of coarser leaves that carry surface, and compaction of the output mesh.
//
// Reference: mesh/BuildMeshGeometry.cu:42-546 and mesh/ComputeTriangleIndices.cu:346-2194.
// The reference processes each coarse subdivision root in its own host iteration and the
// finer roots in one host iteration per depth, temporarily redirecting the parent's child
// pointer to the subdivided copy.  Here every root group (one coarse root, or all finer
// roots of one depth) owns a region of one subdivision-space array and an overlay of the
// redirected child pointers that only its own lookups see, so all groups run in one
// batched pass with the same results as the sequential reference.
#include "workspace.h"
#include "tables.cuh"

PSR_DEFINE_CONST_TABLES(upload_tables_mesh)

namespace psr {

// values behind N 1-based vertex pointers, every load issued before any check (a pointer
// <= 0 is a broken record: it reads entry 0, yields 1.0f and flags the error)
template <int N>
__device__ __forceinline__ void ptr_values(const float* vals, const int (&p)[N], float (&v)[N], unsigned* err) {
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = vals[p[q] > 0 ? p[q] - 1 : 0];
    bool bad = false;
#pragma unroll
    for (int q = 0; q < N; ++q)
        if (p[q] <= 0) { v[q] = 1.0f; bad = true; }
    if (bad) atomicOr(err, kErrInvalid);
}

// vertex slot of a neighbour centre relative to a vertex (mesh/BuildMeshGeometry.cu:133-144)
__device__ __forceinline__ int vertex_slot(float ncx, float ncy, float ncz, float vx, float vy, float vz) {
    int idx = 0;
    if (__fsub_rn(ncx, vx) < 0) idx |= 1;
    if (__fsub_rn(ncz, vz) < 0) idx |= 4;
    if (__fsub_rn(ncy, vy) < 0) idx += (idx & 1) ? 1 : 3;
    return idx;
}

// Same-depth cells around a vertex, an edge or a face.  Neighbour slot k of a node is the
// same-depth cell at offset (k/9 - 1, (k/3)%3 - 1, k%3 - 1).  Node centres, corners and
// edge / face midpoints are dyadic, so the reference's test "centre within one cell width
// of the point" is exact, and it holds for precisely these cells: the 8 cells whose offset
// is 0 or the corner's side on every axis, the 4 around an edge, the 2 across a face.
// Ownership (smallest key among those cells) and the back-pointers are evaluated on these
// slots only, with the reference's slot numbering derived from the same offsets.
__device__ __forceinline__ int nslot(int ax, int ay, int az) { return 9 * (ax + 1) + 3 * (ay + 1) + (az + 1); }

// corner q: + side on x if bit 0, y if bit 1, z if bit 2
__device__ __forceinline__ void corner_sides(int q, int& mx, int& my, int& mz) {
    mx = (q & 1) ? 1 : -1;
    my = (q & 2) ? 1 : -1;
    mz = (q & 4) ? 1 : -1;
}
__device__ __forceinline__ unsigned vertex_cells(int q) {
    int mx, my, mz;
    corner_sides(q, mx, my, mz);
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) m |= 1u << nslot((j & 1) ? mx : 0, (j & 2) ? my : 0, (j & 4) ? mz : 0);
    return m;
}
// edge e: axis e >> 2; the two other axes (increasing order) at sides 2 (e & 1) - 1 and
// 2 ((e >> 1) & 1) - 1
__device__ __forceinline__ void edge_offset(int e, int j, int a[3]) {
    const int orient = e >> 2;
    const int m[2] = {2 * (e & 1) - 1, 2 * ((e >> 1) & 1) - 1};
    int dim = 0;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        a[ax] = 0;
        if (ax != orient) { a[ax] = ((j >> dim) & 1) ? m[dim] : 0; dim++; }
    }
}
__device__ __forceinline__ unsigned edge_cells(int e) {
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int a[3];
        edge_offset(e, j, a);
        m |= 1u << nslot(a[0], a[1], a[2]);
    }
    return m;
}
__device__ __forceinline__ unsigned face_cells(int f) {
    int a[3] = {0, 0, 0};
    a[f >> 1] = 2 * (f & 1) - 1;
    return (1u << 13) | (1u << nslot(a[0], a[1], a[2]));
}
// vertex_slot() of the cell at offset a for corner sides m (centre minus corner is
// (2 a - m) half widths on every axis)
__device__ __forceinline__ int vertex_slot_of(int ax, int ay, int az, int mx, int my, int mz) {
    int idx = 0;
    if (2 * ax - mx < 0) idx |= 1;
    if (2 * az - mz < 0) idx |= 4;
    if (2 * ay - my < 0) idx += (idx & 1) ? 1 : 3;
    return idx;
}
// edge slot of the cell at offset a around edge e (mesh/BuildMeshGeometry.cu:255-268)
__device__ __forceinline__ int edge_slot_of(int e, const int a[3]) {
    const int orient = e >> 2;
    const int m[2] = {2 * (e & 1) - 1, 2 * ((e >> 1) & 1) - 1};
    int idx = orient << 2, dim = 0;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax)
        if (ax != orient) { if (2 * a[ax] - m[dim] < 0) idx |= 1 << dim; dim++; }
    return idx;
}

// ------------------------------------------------------------------------------------
// octree vertex / edge / face records
// ------------------------------------------------------------------------------------
// Ownership of a node's corners, edges (depth D) and faces from its neighbours' keys
// (initVertexOwner, initEdgeArray, initFaceArray, mesh/BuildMeshGeometry.cu:42-101, :149-220,
// :282-354): a node owns an element when no other cell around it has a smaller key.  Also clears
// the back-pointers and overlays of the node; blockIdx.z = 1 clears the colour cell table.
__global__ void __launch_bounds__(kBlock) k_mesh_owners(const Counters* c, int depth, const int* key, const int* neigh,
                                                        size_t stride, unsigned char* vmask, unsigned short* emask,
                                                        unsigned char* fmask, int* node_vtx, int* node_edge,
                                                        int* node_face, int* ov_group, int* ov_sub, int* cell_table,
                                                        int cells) {
    PSR_CLOUD(c, key, neigh, vmask, emask, fmask, node_vtx, node_edge, node_face, ov_group, ov_sub, cell_table);
    if (blockIdx.z == 1) {
        PSR_GRID_STRIDE(i, cells) cell_table[i] = 0;
        return;
    }
    const int M = c->n_nodes;
    const int bD = c->level_base[depth], mD = c->level_count[depth];
    PSR_GRID_STRIDE(i, M) {
        const int myk = key[i];
        unsigned smaller = 0;
        int nb[27];
#pragma unroll
        for (int k = 0; k < 27; ++k) nb[k] = neigh[(size_t)k * stride + i];
#pragma unroll
        for (int k = 0; k < 27; ++k)   // an absent neighbour is never smaller
            if (k != 13 && key[nb[k] != -1 ? nb[k] : i] < myk) smaller |= 1u << k;
        unsigned m = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) if (!(smaller & vertex_cells(q))) m |= 1u << q;
        vmask[i] = (unsigned char)m;
        m = 0;
#pragma unroll
        for (int f = 0; f < 6; ++f) if (!(smaller & face_cells(f))) m |= 1u << f;
        fmask[i] = (unsigned char)m;
        if ((unsigned)(i - bD) < (unsigned)mD) {
            m = 0;
#pragma unroll
            for (int e = 0; e < 12; ++e) if (!(smaller & edge_cells(e))) m |= 1u << e;
            emask[i - bD] = (unsigned short)m;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) node_vtx[(size_t)k * stride + i] = 0;
#pragma unroll
        for (int k = 0; k < 12; ++k) node_edge[(size_t)k * stride + i] = 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) node_face[(size_t)k * stride + i] = 0;
        if (i < bD)   // only nodes with children are looked up there
#pragma unroll
            for (int k = 0; k < 8; ++k) { ov_group[(size_t)k * stride + i] = -1; ov_sub[(size_t)k * stride + i] = -1; }
    }
}

struct PopcLoad8 {
    const unsigned char* m;
    __device__ unsigned operator()(int i) const { return __popc((unsigned)m[i]); }
    __device__ void rebase() { PSR_CLOUD(m); }   // to cloud blockIdx.y
};

struct VertexStore {
    const unsigned char* vmask;
    const int* ndepth;
    const float *cx, *cy, *cz;
    float *vx, *vy, *vz;
    int *vowner, *vkind, *vdepth;
    int cap;
    unsigned* err;
    __device__ void operator()(int i, unsigned pre, unsigned cnt) const {
        if (!cnt) return;
        if ((int)(pre + cnt) > cap) { atomicOr(err, kErrCapacity); return; }
        const unsigned m = vmask[i];
        const int d = ndepth[i];
        const float hw = 1.0f / (float)(1 << (d + 1));
        const float x = cx[i], y = cy[i], z = cz[i];
        int o = (int)pre;
        for (int q = 0; q < 8; ++q) {
            if (!((m >> q) & 1)) continue;
            vx[o] = __fadd_rn(x, (float)(2 * (q & 1) - 1) * hw);
            vy[o] = __fadd_rn(y, (float)(2 * ((q >> 1) & 1) - 1) * hw);
            vz[o] = __fadd_rn(z, (float)(2 * ((q >> 2) & 1) - 1) * hw);
            vowner[o] = i;
            vkind[o] = q;
            vdepth[o] = d;
            ++o;
        }
    }
    __device__ void rebase() { PSR_CLOUD(vmask, ndepth, cx, cy, cz, vx, vy, vz, vowner, vkind, vdepth, err); }   // to cloud blockIdx.y
};

struct PopcLoad16 {
    const unsigned short* m;
    __device__ unsigned operator()(int i) const { return __popc((unsigned)m[i]); }
    __device__ void rebase() { PSR_CLOUD(m); }   // to cloud blockIdx.y
};

struct EdgeStore {
    const unsigned short* emask;
    const int* base_ptr;   // first D-level node
    int *eowner, *ekind;
    int cap;
    unsigned* err;
    __device__ void operator()(int o, unsigned pre, unsigned cnt) const {
        if (!cnt) return;
        if ((int)(pre + cnt) > cap) { atomicOr(err, kErrCapacity); return; }
        const unsigned m = emask[o];
        const int i = *base_ptr + o;
        int q = (int)pre;
        for (int e = 0; e < 12; ++e)
            if ((m >> e) & 1) { eowner[q] = i; ekind[q] = e; ++q; }
    }
    __device__ void rebase() { PSR_CLOUD(emask, base_ptr, eowner, ekind, err); }   // to cloud blockIdx.y
};

struct FaceStore {
    const unsigned char* fmask;
    const int* key;
    const int* ndepth;
    const int* parent;
    int depth;
    int *fowner, *fkind, *fhas;
    int* face_hit;   // starts cleared
    int cap;
    unsigned* err;
    __device__ void operator()(int i, unsigned pre, unsigned cnt) const {
        if (!cnt) return;
        if ((int)(pre + cnt) > cap) { atomicOr(err, kErrCapacity); return; }
        const unsigned m = fmask[i];
        const int d = ndepth[i];
        const int son = (key[i] >> (3 * (depth - d))) & 7, pa = parent[i];
        int q = (int)pre;
        for (int f = 0; f < 6; ++f) {
            if (!((m >> f) & 1)) continue;
            fowner[q] = i;
            fkind[q] = f;
            face_hit[q] = 0;
            fhas[q] = (pa == -1) ? -1 : ((__ldg(&g_tab.parent_face_kind[son][f]) != -1) ? 1 : -1);
            ++q;
        }
    }
    __device__ void rebase() { PSR_CLOUD(fmask, key, ndepth, parent, fowner, fkind, fhas, face_hit, err); }   // to cloud blockIdx.y
};

// chunk count of every coarse node (depth < dsplit) of the divergence
struct DivChunkLoad {
    const int* neigh;
    size_t stride;
    const int* dnum;
    __device__ unsigned operator()(int i) const {
        int nb[27], dn[27];
#pragma unroll
        for (int k = 0; k < 27; ++k) nb[k] = neigh[(size_t)k * stride + i];
#pragma unroll
        for (int k = 0; k < 27; ++k) dn[k] = dnum[nb[k] >= 0 ? nb[k] : 0];
        unsigned n = 0;
#pragma unroll
        for (int k = 0; k < 27; ++k)
            if (nb[k] >= 0) n += (unsigned)((dn[k] + kDivChunk - 1) / kDivChunk);
        return n;
    }
    __device__ void rebase() { PSR_CLOUD(neigh, dnum); }   // to cloud blockIdx.y
};
struct DivChunkStore {
    unsigned* item_start;
    Counters* c;
    int cap;
    __device__ void operator()(int i, unsigned pre, unsigned) const { item_start[i] = pre; }
    __device__ void done(unsigned total) const {
        int n = (int)total;
        if (n > cap) { atomicOr(&c->error, kErrCapacity); n = 0; }
        c->n_div_items = n;
    }
    __device__ void rebase() { PSR_CLOUD(item_start, c); }   // to cloud blockIdx.y
};

// Back-pointers of the nodes around every vertex, edge and face (maintainVertexNodePointer,
// maintainEdgeNodePointer, maintainFaceNodePointer, mesh/BuildMeshGeometry.cu:108-147, :222-280,
// :356-400), blockIdx.z an element kind each; blockIdx.z = 3 counts the samples of the colour cells.
__global__ void __launch_bounds__(kBlock) k_mesh_maintain(Counters* c, int depth, const int* neigh, size_t stride,
                                                          const int* vowner, const int* vkind, int* node_vtx,
                                                          const int* eowner, const int* ekind, int* node_edge,
                                                          const int* fowner, const int* fkind, int* node_face, int g,
                                                          const int* key, const int* point2node, int* cell_table) {
    PSR_CLOUD(c, neigh, vowner, vkind, node_vtx, eowner, ekind, node_edge, fowner, fkind, node_face, key, point2node, cell_table);
    if (blockIdx.z == 0) {
        const int V = c->n_vertices;
        PSR_GRID_STRIDE(v, V) {
            const int ow = vowner[v];
            int mx, my, mz, nb[8];
            corner_sides(vkind[v], mx, my, mz);
#pragma unroll
            for (int j = 0; j < 8; ++j)   // all reads before the first store
                nb[j] = neigh[(size_t)nslot((j & 1) ? mx : 0, (j & 2) ? my : 0, (j & 4) ? mz : 0) * stride + ow];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int ax = (j & 1) ? mx : 0, ay = (j & 2) ? my : 0, az = (j & 4) ? mz : 0;
                if (nb[j] != -1) node_vtx[(size_t)vertex_slot_of(ax, ay, az, mx, my, mz) * stride + nb[j]] = v + 1;
            }
        }
    } else if (blockIdx.z == 1) {
        const int E = c->n_edges;
        PSR_GRID_STRIDE(ei, E) {
            const int ow = eowner[ei], kind = ekind[ei];
            int nb[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int a[3];
                edge_offset(kind, j, a);
                nb[j] = neigh[(size_t)nslot(a[0], a[1], a[2]) * stride + ow];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int a[3];
                edge_offset(kind, j, a);
                if (nb[j] != -1) node_edge[(size_t)edge_slot_of(kind, a) * stride + nb[j]] = ei + 1;
            }
        }
    } else if (blockIdx.z == 2) {
        const int F = c->n_faces;
        PSR_GRID_STRIDE(fi, F) {
            const int ow = fowner[fi], kind = fkind[fi];
            const int orient = kind >> 1, m = 2 * (kind & 1) - 1;
            const int step = orient == 0 ? 9 : (orient == 1 ? 3 : 1);
            const int nb0 = neigh[(size_t)13 * stride + ow], nb1 = neigh[(size_t)(13 + m * step) * stride + ow];
            if (nb0 != -1) node_face[(size_t)((orient << 1) + (m > 0 ? 1 : 0)) * stride + nb0] = fi + 1;
            if (nb1 != -1) node_face[(size_t)((orient << 1) + (m < 0 ? 1 : 0)) * stride + nb1] = fi + 1;
        }
    } else {
        // run length of every occupied cell of level g at the last sample of its run (the samples are
        // Morton-sorted)
        const int n = c->n_points;
        const int bD = c->level_base[depth];
        const int sh = 3 * (depth - g);
        auto cell = [&](int i) { return (unsigned)key[bD + point2node[i]] >> sh; };
        if (blockIdx.x == 0 && threadIdx.x == 0) c->n_colour_cells = (1 << (3 * g)) + 1;
        PSR_GRID_STRIDE(i, n) {
            const unsigned m = cell(i);
            if (i + 1 < n && cell(i + 1) == m) continue;
            int lo = 0, hi = i;   // first sample of the run ending at i
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (cell(mid) < m) lo = mid + 1;
                else hi = mid;
            }
            cell_table[m] = i + 1 - lo;
        }
    }
}

// ------------------------------------------------------------------------------------
// implicit values at the octree vertices (mesh/ComputeTriangleIndices.cu:346-399)
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) k_vertex_values(const Counters* c, int depth, const float* vx,
                                                          const float* vy, const float* vz, const int* vowner,
                                                          const int* vkind, const int* vdepth, const int* neigh,
                                                          size_t stride, const int* parent, const int* first_child,
                                                          const int* enc, const float* x, float* vvalue) {
    PSR_CLOUD(c, vx, vy, vz, vowner, vkind, vdepth, neigh, parent, first_child, enc, x, vvalue);
    const int V = c->n_vertices;
    const float iso = c->iso;
    PSR_GRID_STRIDE(v, V) {
        float val = 0.0f;
        const int ow = vowner[v];
        if (ow > 0) {
            // The chain: the owner, its ancestors up to the root, then the owner's
            // descendants of child kind ec down to depth D.  Software-pipelined: the next
            // node's neighbour row, code, parent and first child are read while the current
            // node's values are in flight; terms are added in chain order as before.
            const float qx = vx[v], qy = vy[v], qz = vz[v];
            const int ec = __ldg(&g_tab.children_vertex_kind[vkind[v]]);
            int d = vdepth[v];
            const int fc_ow = first_child[ow];
            bool up = true;
            int nbs[27];
#pragma unroll
            for (int k = 0; k < 27; ++k) nbs[k] = neigh[(size_t)k * stride + ow];
            int e = enc[ow], par = parent[ow], fcn = fc_ow;
            while (true) {
                float xv[27];
#pragma unroll
                for (int k = 0; k < 27; ++k) xv[k] = x[nbs[k]];
                int nx;
                if (up && par != -1) {
                    nx = par;
                } else {
                    const int f = up ? fc_ow : fcn;
                    up = false;
                    nx = (d < depth && f != -1) ? f + ec : -1;
                    if (nx != -1) ++d;
                }
                int nb2[27];
                int e2 = 0, par2 = -1, fc2 = -1;
                const int n0 = (nx != -1) ? nx : 0;
#pragma unroll
                for (int k = 0; k < 27; ++k) nb2[k] = neigh[(size_t)k * stride + n0];
                e2 = enc[n0];
                par2 = parent[n0];
                fc2 = first_child[n0];
                val = terms_from(e, xv, val, qx, qy, qz, depth);
                if (nx == -1) break;
#pragma unroll
                for (int k = 0; k < 27; ++k) nbs[k] = nb2[k];
                e = e2;
                par = par2;
                fcn = fc2;
            }
        }
        vvalue[v] = __fsub_rn(val, iso);
    }
}

// The same for trees of depth 8 and 9, where the kernel is bound by instruction issue: the chain's
// nodes above depth D come from their value rows.  Three blocks per SM, 80 registers (36 bytes spilled).
__global__ void __launch_bounds__(kBlock, 3) k_vertex_values_rows(const Counters* c, int depth, const float* vx,
                                                                  const float* vy, const float* vz, const int* vowner,
                                                                  const int* vkind, const int* vdepth, ValueRows R,
                                                                  float* vvalue) {
    PSR_CLOUD(c, vx, vy, vz, vowner, vkind, vdepth, R, vvalue);
    R.n = min(c->level_base[depth], R.n);
    const int V = c->n_vertices;
    const float iso = c->iso;
    PSR_GRID_STRIDE(v, V) {
        float val = 0.0f;
        const int ow = vowner[v];
        if (ow > 0) {
            const float qx = vx[v], qy = vy[v], qz = vz[v];
            const int ec = __ldg(&g_tab.children_vertex_kind[vkind[v]]);
            int d = vdepth[v];
            bool up = true;
            ValueRow cur, nxt;
            load_row(R, ow, cur);
            const int fc_ow = cur.first_child;
            while (true) {
                int nx;
                if (up && cur.parent != -1) {
                    nx = cur.parent;
                } else {
                    const int f = up ? fc_ow : cur.first_child;
                    up = false;
                    nx = (d < depth && f != -1) ? f + ec : -1;
                    if (nx != -1) ++d;
                }
                load_row(R, nx != -1 ? nx : 0, nxt);   // in flight during the terms
                val = terms_from(cur.enc, cur.x, val, qx, qy, qz, depth);
                if (nx == -1) break;
                cur = nxt;
            }
        }
        vvalue[v] = __fsub_rn(val, iso);
    }
}

// ------------------------------------------------------------------------------------
// marching cubes at depth D (mesh/ComputeTriangleIndices.cu:401-526)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void interp_point(float p1x, float p1y, float p1z, float p2x, float p2y, float p2z, int dim,
                                             float v1, float v2, float* out) {
    out[0] = p1x; out[1] = p1y; out[2] = p1z;
    const float a1 = (dim == 0) ? p1x : (dim == 1) ? p1y : p1z;   // selects: no local array
    const float a2 = (dim == 0) ? p2x : (dim == 1) ? p2y : p2z;
    float pivot = __fdiv_rn(v1, __fsub_rn(v1, v2));
    float other = __fsub_rn(1.0f, pivot);
    out[dim] = __fadd_rn(__fmul_rn(a2, pivot), __fmul_rn(a1, other));
}

// the two vertex pointers of K edges, then their values, each step's loads in flight together
template <int K, class EdgeAt>
__device__ __forceinline__ void edge_values(const int* vtx, size_t stride, const float* vals, EdgeAt at, float (&v)[2 * K],
                                            unsigned* err) {
    int owner[K], kind[K], p[2 * K];
#pragma unroll
    for (int k = 0; k < K; ++k) at(k, owner[k], kind[k]);
#pragma unroll
    for (int k = 0; k < 2 * K; ++k)
        p[k] = vtx[(size_t)__ldg(&g_tab.edge_vertex[kind[k >> 1]][k & 1]) * stride + owner[k >> 1]];
    ptr_values(vals, p, v, err);
}

struct CrossLoad {
    const int* eowner;
    const int* ekind;
    const int* node_vtx;
    size_t stride;
    const float* vvalue;
    unsigned* err;
    __device__ unsigned operator()(int e) const {
        float ab[2];
        edge_values<1>(node_vtx, stride, vvalue, [&](int, int& ow, int& kind) { ow = eowner[e]; kind = ekind[e]; }, ab, err);
        return (__fmul_rn(ab[0], ab[1]) <= 0.0f) ? 1u : 0u;
    }
    template <int K>
    __device__ bool all(int base, unsigned (&v)[K]) const {
        float ab[2 * K];
        edge_values<K>(node_vtx, stride, vvalue, [&](int k, int& ow, int& kind) { ow = eowner[base + k]; kind = ekind[base + k]; }, ab, err);
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = (__fmul_rn(ab[2 * k], ab[2 * k + 1]) <= 0.0f) ? 1u : 0u;
        return true;
    }
    __device__ void rebase() { PSR_CLOUD(eowner, ekind, node_vtx, vvalue, err); }   // to cloud blockIdx.y
};

struct CrossStore {
    const int* eowner;
    const int* ekind;
    const int* node_vtx;
    size_t stride;
    const float* vvalue;
    const float *vx, *vy, *vz;
    unsigned* ecross;   // per edge: staged vertex index (valid when the edge crosses)
    float* part_v;      // staged vertices (3 floats each)
    int voff;
    int cap;
    unsigned* err;
    __device__ void operator()(int e, unsigned pre, unsigned flag) const {
        ecross[e] = pre;
        if (!flag) return;
        const int at = voff + (int)pre;
        if (at >= cap) { atomicOr(err, kErrCapacity); return; }
        const int ow = eowner[e], kind = ekind[e];
        const int v1 = node_vtx[(size_t)__ldg(&g_tab.edge_vertex[kind][0]) * stride + ow] - 1;
        const int v2 = node_vtx[(size_t)__ldg(&g_tab.edge_vertex[kind][1]) * stride + ow] - 1;
        if (v1 < 0 || v2 < 0) return;   // only reachable for a malformed tree (flagged in the load)
        interp_point(vx[v1], vy[v1], vz[v1], vx[v2], vy[v2], vz[v2], kind >> 2, vvalue[v1], vvalue[v2],
                     &part_v[3 * (size_t)at]);
    }
    __device__ void rebase() { PSR_CLOUD(eowner, ekind, node_vtx, vvalue, vx, vy, vz, ecross, part_v, err); }   // to cloud blockIdx.y
};

struct CubeLoad {
    const int* node_vtx;
    size_t stride;
    const int* base_ptr;
    const float* vvalue;
    int* cube_class;
    unsigned* err;
    __device__ unsigned operator()(int o) const {
        const int i = *base_ptr + o;
        int p[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) p[q] = node_vtx[(size_t)q * stride + i];
        float vq[8];
        ptr_values(vvalue, p, vq, err);
        int cls = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (vq[q] < 0.0f) cls |= 1 << q;
        cube_class[o] = cls;
        return (unsigned)__ldg(&g_tab.mc_count[cls]);
    }
    __device__ void rebase() { PSR_CLOUD(node_vtx, base_ptr, vvalue, cube_class, err); }   // to cloud blockIdx.y
};

// The cnt triangles (edge numbers in `tri`) of a cell, whose edge pointers are `edges` with stride
// `stride`: crossing numbers relative to `base`, from triangle `at` on.  Returns the edges used.  All
// pointers are read before any crossing and all crossings before any store: triangle by triangle the
// up to 15 pairs of loads waited for one another (27 -> 17 us for the cubes of 200,000 samples, depth 7).
__device__ __forceinline__ unsigned store_triangles(unsigned long long tri, int cnt, const int* edges, size_t stride,
                                                    const unsigned* ecross, unsigned base, int* out, int at, int cap,
                                                    unsigned* err) {
    int p[15];
    unsigned used = 0;
#pragma unroll
    for (int q = 0; q < 15; ++q) {
        const int e = (int)((tri >> (4 * q)) & 0xF);
        p[q] = q < 3 * cnt ? edges[(size_t)e * stride] - 1 : -1;
        if (q < 3 * cnt) used |= 1u << e;
    }
#pragma unroll
    for (int q = 0; q < 15; ++q)
        if (p[q] >= 0) p[q] = (int)(ecross[p[q]] - base);
#pragma unroll
    for (int q = 0; q < 15; ++q)
        if (q < 3 * cnt && at + q / 3 < cap) out[3 * (size_t)at + q] = p[q];
    if (at + cnt > cap) atomicOr(err, kErrCapacity);
    return used;
}

// emits the triangles of a D-level cube and marks surface-edge intersections on faces,
// propagating them to the parent faces (generateTrianglePos, :476-526)
struct CubeStore {
    const int* cube_class;
    const int* base_ptr;
    const int* node_edge;
    const int* node_face;
    size_t stride;
    const unsigned* ecross;
    const int* parent;
    const int* fhas;
    int* face_hit;
    int* part_t;
    int toff;
    int cap;
    unsigned* err;
    __device__ void operator()(int o, unsigned pre, unsigned cnt) const {
        if (!cnt) return;
        const int i = *base_ptr + o;
        const int cls = cube_class[o];
        const unsigned long long tri = __ldg(&g_tab.mc_tri[cls]);
        const unsigned used = store_triangles(tri, (int)cnt, node_edge + i, stride, ecross, 0u, part_t, toff + (int)pre, cap, err);
        // the faces with an intersected edge, and the parents' faces they lie on: the six walks
        // side by side
        int cf[6], pn[6];
        const int pa = parent[i];
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            unsigned mark = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) mark |= (used >> c_tab.face_edges[f][j]) & 1u;
            cf[f] = mark ? node_face[(size_t)f * stride + i] - 1 : -1;
            pn[f] = pa;
        }
        for (int guard = 0; guard <= 32; ++guard) {
            bool more = false;
            int has[6], up[6], next[6];
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                const bool on = cf[f] >= 0;
                has[f] = on ? fhas[cf[f]] : -1;
                const bool go = on && pn[f] >= 0 && guard < 32;
                up[f] = go ? node_face[(size_t)f * stride + pn[f]] - 1 : -1;
                next[f] = go ? parent[pn[f]] : -1;
            }
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                if (cf[f] >= 0) face_hit[cf[f]] = 1;
                cf[f] = has[f] != -1 ? up[f] : -1;
                pn[f] = next[f];
                more |= cf[f] >= 0;
            }
            if (!more) break;
        }
    }
    __device__ void rebase() { PSR_CLOUD(cube_class, base_ptr, node_edge, node_face, ecross, parent, fhas, face_hit, part_t, err); }   // to cloud blockIdx.y
};

// ------------------------------------------------------------------------------------
// subdivision roots (ProcessLeafNodesAtOtherDepth :555-587, selection :1284-1346)
// ------------------------------------------------------------------------------------
struct RootLoad {
    const int* node_vtx;
    const int* node_face;
    size_t stride;
    const float* vvalue;
    const int* face_hit;
    const int* first_child;
    unsigned* err;
    __device__ unsigned operator()(int i) const {
        // all reads first (the cell's 8 corner values, 6 faces and their flags), then the tests
        int p[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) p[q] = node_vtx[(size_t)q * stride + i];
        int fp[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) fp[f] = node_face[(size_t)f * stride + i] - 1;
        int fh[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) fh[f] = face_hit[fp[f] >= 0 ? fp[f] : 0];
        const int fc = first_child[i];
        float vq[8];
        ptr_values(vvalue, p, vq, err);
        const float s = (vq[0] < 0.0f) ? -1.0f : 1.0f;
        int ht = 0;
#pragma unroll
        for (int q = 1; q < 8; ++q)
            if (__fmul_rn(s, vq[q]) < 0.0f) ht = 1;
        int hi = 0;
#pragma unroll
        for (int f = 0; f < 6; ++f)
            if (fp[f] >= 0 && fh[f]) hi = 1;
        return (fc == -1 && (ht || hi)) ? 1u : 0u;
    }
    __device__ void rebase() { PSR_CLOUD(node_vtx, node_face, vvalue, face_hit, first_child, err); }   // to cloud blockIdx.y
};
struct RootStore {
    Counters* c;
    int depth;
    int* sub_root;
    int cap;
    unsigned* err;
    __device__ void operator()(int i, unsigned pre, unsigned f) const {
        // the roots are in depth order: the count before a level's first node (1 + a multiple of 8) is
        // where the roots of its depth start
        if ((i & 7) == 1)
            for (int d = 1; d < depth; ++d)
                if (c->level_base[d] == i) c->sub_rstart[d] = min((int)pre, cap);
        if (!f) return;
        if ((int)pre >= cap) { atomicOr(err, kErrCapacity); return; }
        sub_root[pre] = i;
    }
    __device__ void rebase() { PSR_CLOUD(c, sub_root, err); }   // to cloud blockIdx.y
};

// Group table.  Group record (ints): 0 root depth, 1 first root, 2 root count,
// 3 virtual node offset, 4 virtual node count.  Coarse roots (depth < D - 4) are one group each; the finer roots
// of one depth form one group (mesh/ComputeTriangleIndices.cu:1475-1799, :1801-2194).
constexpr int kGroupRec = 8;

// ---- subdivision, breadth-first over live nodes ----------------------------------------
// Virtual numbering (singleRebuildArray :599-635 / wholeRebuildArray :1110-1168): group g
// owns the virtual sub nodes G[3] .. G[3] + G[4] - 1, level by level from its root depth rd
// (its n roots) to D; node (q, rel) of level d sits at G[3] + off_d + q 8^(d-rd) + rel (rel:
// the Morton code below root q).  Only live nodes are stored, in one list, depth after depth:
// of depth d's candidates (the 8 children of every live node of depth d-1, in order, then the
// roots of depth d) those that stay live.  Both parts are in virtual order (groups are ordered
// by root depth), so the live depth-D cells, which carry all records from here on, come out in
// the reference's order.  Neighbour rows hold octree nodes (< na), na + list entry for live sub
// nodes, or -1 (nothing there, or a sub node that is not live: it carries no value, and neither
// it nor anything below it is referred to again).
__device__ __forceinline__ int sub_level_off(int rd, int n, int d) {
    int off = 0, cnt = n;
    for (int e = rd; e < d; ++e) { off += cnt; cnt *= 8; }
    return off;
}

// The groups of a depth's roots.  The roots are in depth order, so with the first root of every depth
// known the groups follow without a scan: a coarse root is group number its own, a finer depth is the
// group after those of the depths before it, and a root of depth d brings (8^(D-d+1) - 1) / 7 virtual
// nodes (two scans of up to 12 us each before).  In shared memory of every block; block 0 also sets up the
// per-depth bookkeeping (Counters::sub_*).
struct DepthGroups {
    int start[kMaxDepth + 2];     // first root of the depth
    int count[kMaxDepth + 2];
    int group[kMaxDepth + 2];     // first group
    long long per[kMaxDepth + 2];    // virtual nodes of a root
    long long first[kMaxDepth + 2];  // first virtual node
    int n_groups;
};
__device__ __forceinline__ void sub_setup(Counters* c, int depth, int max_groups, int na, int cap_nodes, DepthGroups& t) {
    if (threadIdx.x == 0) {
        const int R = c->n_subroots;
        int start[kMaxDepth + 2];
#pragma unroll
        for (int d = 0; d <= kMaxDepth + 1; ++d)   // a level without nodes has no roots
            start[d] = d == 0 ? 0 : (d < depth && c->level_count[min(d, kMaxDepth)] > 0 ? c->sub_rstart[d] : -1);
        int next = R, ng = 0;
#pragma unroll
        for (int d = kMaxDepth + 1; d >= 0; --d) {
            if (start[d] < 0) start[d] = next;
            t.start[d] = start[d];
            t.count[d] = next - start[d];
            next = start[d];
        }
        long long virt = 0;
        unsigned bad = 0;
        for (int d = 0; d <= depth; ++d) {
            const bool coarse = d < depth - 4;
            long long per = 0, n = 1;
            for (int e = d; e <= depth; ++e) { per += n; n *= 8; }
            t.per[d] = per;
            t.group[d] = ng;
            t.first[d] = virt;
            ng += coarse ? t.count[d] : (t.count[d] > 0 ? 1 : 0);
            if (t.count[d] > 0 && per * (coarse ? 1 : t.count[d]) > 0x3fffffffLL) bad = 1;
            virt += per * t.count[d];
        }
        // the numbering of the groups must fit the table, and their virtual nodes beside the octree's
        if (ng > max_groups || virt > 0x7fffffffLL - na) { bad = 1; ng = 0; }
        t.n_groups = ng;
        if (blockIdx.x == 0) {
            if (bad) atomicOr(&c->error, kErrCapacity);
            c->n_groups = ng;
            c->n_sub_nodes = 0;
            c->n_sub_dnodes = 0;
        }
    }
    __syncthreads();
    const int d = threadIdx.x;
    if (blockIdx.x == 0 && d <= depth + 1) {
        const int n = t.n_groups > 0 ? t.count[d] : 0;
        c->sub_nroots[d] = n;
        c->sub_cbase[d] = 0;
        c->sub_lbase[d] = 0;
        c->sub_nlive[d] = 0;
        if (d == 1 && n > cap_nodes) atomicOr(&c->error, kErrCapacity);
        c->sub_cand[d] = d == 1 && n <= cap_nodes ? n : 0;
    }
}

struct SubArrays {
    int4* rec;      // per live entry: parent (entry, or -2 - octree parent), group, key, virtual index
    float4* pos;    // centre, depth (as bits)
    int* jump;      // nearest contributing entry on the path to the root (itself when it contributes)
    int2* kids;     // its live children: first entry, octant bits
    int* neigh;     // [27][cap_live]: same-depth neighbours
    float* poly;    // [28][cap_live]: Bernstein coefficients of its levels, sum |y|
    int* lv_vnode;  // virtual index of each live depth-D cell
    int cap_nodes, cap_live, cap_live_d;
    __device__ void rebase() { PSR_CLOUD(rec, pos, jump, kids, neigh, poly, lv_vnode); }   // to cloud blockIdx.y
};

// ---- certain-sign cells -------------------------------------------------------------
// Subdivision replaces a coarse leaf that carries surface by all of its depth-D cells, but
// the surface crosses few of them.  A cell where F - iso provably keeps one sign has no
// crossing edge and no triangle, so it needs no vertex, edge or cube record, and its
// subtree is never built.  The test below is conservative, so the mesh is unchanged.
//
// On the closed cell of a sub node s at depth d, F is the sum over the levels l <= d of the
// 27 neighbour terms y_k B_k of s's ancestor at l (y = 0 for absent nodes and for sub nodes
// that are not roots), provided no octree node deeper than d reaches the cell: that holds
// when none of s's 27 neighbours is an octree node with children.  B_k = b(x) b(y) b(z) with
// b(t) = 4/3 (3/4 - t^2) for |t| < 1/2 and 2/3 (3/2 - |t|)^2 for |t| < 3/2 (t in level
// widths from the translate's centre).  The knots of a level-l translate lie on level-l cell
// boundaries and the cell of s lies inside one level-l cell, so on it every translate is a
// single quadratic and F is a tensor-product quadratic.  Written in the Bernstein basis of
// the cell, F's 27 coefficients bound its values there (convex hull), so all coefficients
// above iso (below iso) make the sign certain.  With s in [-1, 1] across the cell, a
// translate is q(s) = b + g s + k/2 s^2 (b, g = h b', k = h^2 b'' at the centre, h the half
// width), whose Bernstein coefficients are b - g + k/2, b - k/2, b + g + k/2.
// Float vertex values are sums of the same nonzero terms (at most 27 (D+1)), within
// ~1.7e-5 sum |y| of the exact value; the float coefficients here are as close; the test
// keeps a margin of 1e-4 (sum |y| + |iso|).

// Levels up to a root's depth are the same for every cell below that root: their sum is one
// tensor-product quadratic on the root's cell, kept as its 27 Bernstein coefficients
// (k_root_setup: root_poly[k][r], k < 27; [27][r]: sum |y| of those levels).  A cell inside it takes
// them by Bernstein subdivision: with the cell at [a, b] of the root's unit interval, the
// new coefficients are the blossom values P(a, a), P(a, b), P(b, b) -- convex weights, exact
// for these dyadic a, b.
// Per root: its group's record, the octree node it stands for, the redirected child slot of its parent (overlay) and
// its polynomial; block 0 also sets up the per-depth bookkeeping.
__global__ void __launch_bounds__(kBlock) k_root_setup(Counters* c, int depth, const int* sub_root, const int* ndepth,
                                                       const int* key, int* root_group, int* groups, int max_groups,
                                                       int na, int* root_self, int* ov_group, int* ov_sub, const float* ctr_x,
                                                       const float* ctr_y, const float* ctr_z, const int* neigh,
                                                       size_t stride, const int* parent, const int* enc, const float* x,
                                                       float* root_poly, int cap_poly, int cap_nodes) {
    PSR_CLOUD(c, sub_root, ndepth, key, root_group, groups, root_self, ov_group, ov_sub, ctr_x, ctr_y, ctr_z, neigh, parent, enc, x, root_poly);
    __shared__ DepthGroups T;
    sub_setup(c, depth, max_groups, na, cap_nodes, T);
    const int R = c->n_subroots;
    const int ng = T.n_groups;
    PSR_GRID_STRIDE(r, R) {
        const int node = sub_root[r];
        const int rd = ndepth[node];
        const int self = neigh[(size_t)13 * stride + node];   // its neighs[13] in the reference
        root_self[r] = (self == -1) ? node : self;
        const int q = r - T.start[rd];
        const bool coarse = rd < depth - 4;
        const int g = T.group[rd] + (coarse ? q : 0), head = coarse ? r : T.start[rd];
        const int pa = parent[node];
        root_group[r] = g;
        if (g < ng) {
            if (r == head) {
                int* G = groups + (size_t)g * kGroupRec;
                const int n = coarse ? 1 : T.count[rd];
                G[0] = rd;
                G[1] = r;
                G[2] = n;
                G[3] = (int)(T.first[rd] + (coarse ? q * T.per[rd] : 0));
                G[4] = (int)min(n * T.per[rd], 0x3fffffffLL);
            }
            if (pa >= 0) {
                const int son = (key[node] >> (3 * (depth - rd))) & 7;
                ov_group[(size_t)son * stride + pa] = g;
                ov_sub[(size_t)son * stride + pa] = r - head;
            }
        }
        if (r >= cap_poly) continue;
        const float qx = ctr_x[node], qy = ctr_y[node], qz = ctr_z[node];
        float C[27];
#pragma unroll
        for (int k = 0; k < 27; ++k) C[k] = 0.0f;
        float mag = 0.0f, y[27];
        for (int now = node; now >= 0; now = parent[now]) {
            int ox, oy, oz;
            decode_fn_index(enc[now], depth, ox, oy, oz);
            const int l = ilog2_dev(ox + 1);
#pragma unroll
            for (int k = 0; k < 27; ++k) {
                const int v = neigh[(size_t)k * stride + now];
                y[k] = (v >= 0) ? x[v] : 0.0f;
            }
            sign_level(y, ox, oy, oz, qx, qy, qz, __int_as_float((126 + l - rd) << 23), C, mag);
        }
#pragma unroll
        for (int k = 0; k < 27; ++k) root_poly[(size_t)k * cap_poly + r] = C[k];
        root_poly[(size_t)27 * cap_poly + r] = mag;
    }
}

// blossom matrix of [a, b] (rows: new coefficients, columns: old)
__device__ __forceinline__ void blossom3(float a, float b, float (&M)[3][3]) {
    const float a1 = 1.0f - a, b1 = 1.0f - b;
    M[0][0] = a1 * a1; M[0][1] = 2.0f * a * a1;     M[0][2] = a * a;
    M[1][0] = a1 * b1; M[1][1] = a1 * b + a * b1;   M[1][2] = a * b;
    M[2][0] = b1 * b1; M[2][1] = 2.0f * b * b1;     M[2][2] = b * b;
}

// polynomial P (27 coefficients, pstride apart) restricted to octant ch of its cell
__device__ __forceinline__ void sub_octant(const float* P, size_t pstride, int ch, float (&C)[27]) {
    float Mx[3][3], My[3][3], Mz[3][3];
    const float ax = 0.5f * (float)((ch >> 2) & 1), ay = 0.5f * (float)((ch >> 1) & 1), az = 0.5f * (float)(ch & 1);
    blossom3(ax, ax + 0.5f, Mx);
    blossom3(ay, ay + 0.5f, My);
    blossom3(az, az + 0.5f, Mz);
    float p[27];
#pragma unroll
    for (int k = 0; k < 27; ++k) p[k] = P[(size_t)k * pstride];
    float T1[27], T2[27];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int jk = 0; jk < 9; ++jk)
            T1[a * 9 + jk] = fmaf(Mx[a][0], p[jk], fmaf(Mx[a][1], p[9 + jk], Mx[a][2] * p[18 + jk]));
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int bb = 0; bb < 3; ++bb)
#pragma unroll
            for (int k = 0; k < 3; ++k)
                T2[a * 9 + bb * 3 + k] = fmaf(My[bb][0], T1[a * 9 + k],
                                              fmaf(My[bb][1], T1[a * 9 + 3 + k], My[bb][2] * T1[a * 9 + 6 + k]));
#pragma unroll
    for (int ab3 = 0; ab3 < 9; ++ab3)
#pragma unroll
        for (int gg = 0; gg < 3; ++gg)
            C[ab3 * 3 + gg] = fmaf(Mz[gg][0], T2[ab3 * 3], fmaf(Mz[gg][1], T2[ab3 * 3 + 1], Mz[gg][2] * T2[ab3 * 3 + 2]));
}

// centre and depth of child ch (depth d) of the cell at `p`
__device__ __forceinline__ float4 sub_child_pos(const float4 p, int ch, int d) {
    const float w = __int_as_float((126 - d) << 23);   // 2^-(d+1)
    return make_float4((ch & 4) ? __fadd_rn(p.x, w) : __fsub_rn(p.x, w), (ch & 2) ? __fadd_rn(p.y, w) : __fsub_rn(p.y, w),
                       (ch & 1) ? __fadd_rn(p.z, w) : __fsub_rn(p.z, w), __int_as_float(d));
}

// Coefficients of a live node are kept (per live entry): a child's levels above its own are
// its parent's polynomial restricted to the child's octant (Bernstein subdivision, convex
// weights: the float error grows by a few ulp of the coefficients per level, inside the
// margin), so a candidate adds at most its own level.  A root starts from root_poly, or,
// beyond its capacity, from the walk over its octree chain.
__device__ __forceinline__ void root_coefficients(int r, int root_node, int rd, float qx, float qy, float qz,
                                                  int depth, const int* neigh, size_t stride, const int* parent,
                                                  const int* enc, const float* x, const float* root_poly,
                                                  int cap_poly, float (&C)[27], float& mag) {
    if (r < cap_poly) {
#pragma unroll
        for (int k = 0; k < 27; ++k) C[k] = root_poly[(size_t)k * cap_poly + r];
        mag = root_poly[(size_t)27 * cap_poly + r];
        return;
    }
#pragma unroll
    for (int k = 0; k < 27; ++k) C[k] = 0.0f;
    mag = 0.0f;
    float y[27];
    for (int now = root_node; now >= 0; now = parent[now]) {
        int ox, oy, oz;
        decode_fn_index(enc[now], depth, ox, oy, oz);
        const int l = ilog2_dev(ox + 1);
#pragma unroll
        for (int k = 0; k < 27; ++k) {
            const int v = neigh[(size_t)k * stride + now];
            y[k] = (v >= 0) ? x[v] : 0.0f;
        }
        sign_level(y, ox, oy, oz, qx, qy, qz, __int_as_float((126 + l - rd) << 23), C, mag);
    }
}

// per-thread hand-over of a candidate's coefficients (28) from the scan's load to its store
__device__ __forceinline__ float* sub_poly_stash() {
    __shared__ float s_stash[28 * kBlock];
    return s_stash;
}

// The octree's part of the subdivision's look-ups: written by earlier launches only.
struct SubTree {
    const int* groups;
    const int* sub_root;
    const int* root_group;
    const int* key;
    const int* neigh;
    size_t stride;
    const int* first_child;
    const int* parent;
    const int* ov_group;
    const int* ov_sub;
    const int* enc;
    const float* x;
    const float* root_poly;
    int cap_poly;
    int na;
    __device__ void rebase() { PSR_CLOUD(groups, sub_root, root_group, key, neigh, first_child, parent, ov_group, ov_sub, enc, x, root_poly); }   // to cloud blockIdx.y
};

// first live entry of the roots of depth d (they follow the depth's live children)
__device__ __forceinline__ int sub_first_root(const Counters* c, int d) {
    return c->sub_lbase[d] + c->sub_nlive[d] - c->sub_nroots[d];
}

// a root's number less this is its index among the roots of depth d
__device__ __forceinline__ int sub_root_shift(const Counters* c, int d) { return c->sub_rstart[d] - sub_first_root(c, d); }

// Slots k0, k0 + kstep, .. of the neighbour row of live entry e of depth d, whose depth is complete
// (computeRebuildNeighbor :669-696); found(slot, record, neighbour) gets each.  A neighbour is a child
// of one of the parent's neighbours: of an octree node its octree child (or, for a root, the root of the
// same group that replaces it), of a live entry its child entry if that is live.  The chain of a slot
// is four dependent loads (record, parent's row, children, what `found` reads), and all rows of a
// depth are in flight at once.
template <class Found>
__device__ __forceinline__ void sub_rows(const Counters* c, const SubTree& o, const SubArrays& A, int d, int depth,
                                         int e, int k0, int kstep, Found found) {
    const int4 me = A.rec[e];
    const int son = (me.z >> (3 * (depth - d))) & 7;
    const bool root = me.x < 0;
    const int pa = root ? -2 - me.x : me.x;
    const int* row = root ? o.neigh + (pa >= 0 ? pa : 0) : A.neigh + pa;
    const size_t rstride = root ? o.stride : (size_t)A.cap_live;
    for (int k = k0; k < 27; k += kstep) {
        int lp, lc;
        nb_lut(son, k, lp, lc);
        int v = -1;
        if (k == 13) {
            v = o.na + e;
        } else if (pa >= 0) {
            const int nb = row[(size_t)lp * rstride];
            if (nb >= o.na) {
                const int2 kd = A.kids[nb - o.na];
                if ((kd.y >> lc) & 1) v = o.na + kd.x + __popc(kd.y & ((1 << lc) - 1));
            } else if (nb >= 0) {
                const int fc = __ldg(o.first_child + nb);
                v = fc < 0 ? -1 : fc + lc;
                if (root && __ldg(o.ov_group + (size_t)lc * o.stride + nb) == me.y) {
                    const int r = __ldg(o.groups + (size_t)me.y * kGroupRec + 1) +
                                  __ldg(o.ov_sub + (size_t)lc * o.stride + nb);
                    v = o.na + sub_first_root(c, d) + r - c->sub_rstart[d];
                }
            }
        }
        A.neigh[(size_t)k * A.cap_live + e] = v;
        found(k, me, v);
    }
}

// Sign test of one depth's candidates: the 8 children of every live entry of the depth above, then
// the roots of this depth (always live).  A tile starts with the neighbour rows of its parents
// (begin), which name the octree nodes whose values a child's own level can read: a child's
// neighbours are children of its parent's, subdivision nodes below a root carry nothing, so a child
// none of whose parent's outer neighbours has octree children takes its parent's polynomial as it
// is.  Nothing else is built before the test; only live candidates get a record.
// Latency-bound at depth 7 (a few thousand candidates a launch), bound by the polynomials' arithmetic
// at depth 9 (3.1 million).  With a record of 27 neighbours built for every candidate the launches of
// depths 4 to D took 131 us (200,000 samples, depth 7), 533 us (500,000, depth 9) and 1.22 ms
// (2,000,000, depth 9); now 90, 327 and 768 us.  Two blocks per SM: 128 registers, nothing spilled.
struct SubLevelLoad {
    static constexpr int kMinBlocks = 2;
    const Counters* c;
    int d, depth;
    SubTree o;
    SubArrays A;
    static __device__ int* first_children() {   // [32 parents][27]: first child of an octree neighbour, or -1
        __shared__ int s_fc[32 * 27];
        return s_fc;
    }
    static __device__ unsigned char* contributes() {   // per parent: an octree neighbour, or a root
        __shared__ unsigned char s_con[32];
        return s_con;
    }
    // rows of the tile's parents, a warp for the four of its candidates; called by every thread of the
    // block before the tile's loads
    __device__ void begin(int base) const {
        const int p = threadIdx.x >> 3, f = (base >> 3) + p;
        bool con = false;
        if (f < c->sub_nlive[d - 1]) {
            int* s_fc = first_children() + p * 27;
            sub_rows(c, o, A, d - 1, depth, c->sub_lbase[d - 1] + f, threadIdx.x & 7, 8, [&](int k, const int4& me, int v) {
                const bool oct = v >= 0 && v < o.na;
                s_fc[k] = oct ? __ldg(o.first_child + v) : -1;
                con |= oct || me.x < 0;
            });
        }
        con = (__ballot_sync(0xffffffffu, con) >> (threadIdx.x & 24) & 0xffu) != 0;
        if ((threadIdx.x & 7) == 0) contributes()[p] = con;
        __syncwarp();
    }
    __device__ unsigned operator()(int i) const {
        if (i >= 8 * c->sub_nlive[d - 1]) return 1u;   // a root
        const int ch = i & 7, p = threadIdx.x >> 3;
        const int pl = c->sub_lbase[d - 1] + (i >> 3);
        float C[27];
        sub_octant(A.poly + pl, (size_t)A.cap_live, ch, C);
        float mag = A.poly[(size_t)27 * A.cap_live + pl];
        const int* s_fc = first_children() + p * 27;
        // the eight of its parent's neighbours that a child's neighbours are children of
        const int sx = (ch >> 2) & 1, sy = (ch >> 1) & 1, sz = ch & 1;
        int most = -1;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            most = max(most, s_fc[9 * (sx + (j >> 2)) + 3 * (sy + ((j >> 1) & 1)) + sz + (j & 1)]);
        const bool contrib = most >= 0;
        bool deeper = false;   // an octree neighbour with children
        if (contrib) {   // its own level
            float y[27];
            int v[27];
            child_neighbours(ch, [](int j) { return j; }, [&](int j) { return s_fc[j]; }, v);
#pragma unroll
            for (int k = 0; k < 27; ++k) {
                y[k] = __ldg(o.x + v[k]);   // x[-1] = 0
                if (v[k] >= 0 && d < depth) deeper |= __ldg(o.first_child + v[k]) != -1;
            }
            const float4 q = sub_child_pos(A.pos[pl], ch, d);
            const float sc = (float)(1 << d);
            const int b = (1 << d) - 1;
            sign_level(y, b + (int)__fmul_rn(q.x, sc), b + (int)__fmul_rn(q.y, sc), b + (int)__fmul_rn(q.z, sc), q.x,
                       q.y, q.z, 0.5f, C, mag);
        }
        if (!deeper) {
            float lo = C[0], hi = C[0];
#pragma unroll
            for (int kk = 1; kk < 27; ++kk) { lo = fminf(lo, C[kk]); hi = fmaxf(hi, C[kk]); }
            const float iso = c->iso;
            const float margin = 1e-4f * (mag + fabsf(iso));
            if (lo - iso > margin || hi - iso < -margin) return 0u;   // certain sign
        }
        float* stash = sub_poly_stash();
#pragma unroll
        for (int kk = 0; kk < 27; ++kk) stash[kk * kBlock + threadIdx.x] = C[kk];
        stash[27 * kBlock + threadIdx.x] = mag;
        return 1u;
    }
    __device__ void rebase() { PSR_CLOUD(c, o, A); }   // to cloud blockIdx.y
};
// Records of the live candidates, at their place in the live list.
struct SubLevelStore {
    Counters* c;
    int d, depth;
    SubTree o;
    SubArrays A;
    unsigned* err;
    __device__ void operator()(int i, unsigned pre, unsigned live) const {
        const int nchild = 8 * c->sub_nlive[d - 1];
        const int at = c->sub_lbase[d] + (int)pre;
        const bool keep = live && at < A.cap_live && (d < depth || (int)pre < A.cap_live_d);
        if (live && !keep) atomicOr(err, kErrCapacity);
        const bool child = i < nchild;
        const int pl = c->sub_lbase[d - 1] + (i >> 3);
        if (child) {   // the family's eight lanes are all here
            const unsigned fam = __ballot_sync(0xffu << (threadIdx.x & 24), keep) >> (threadIdx.x & 24);
            if ((i & 7) == 0) {
                A.kids[pl] = make_int2(at, (int)(fam & 0xffu));
                A.jump[pl] = SubLevelLoad::contributes()[threadIdx.x >> 3] ? pl : A.jump[A.rec[pl].x];
            }
        }
        if (!keep) return;
        int4 me;
        if (child) {
            const int ch = i & 7;
            const int4 pr = A.rec[pl];
            const int* G = o.groups + (size_t)pr.y * kGroupRec;
            const int rd = __ldg(G), n = __ldg(G + 2), first = __ldg(G + 3);
            me.x = pl;
            me.y = pr.y;
            me.z = pr.z | (ch << (3 * (depth - d)));
            me.w = first + sub_level_off(rd, n, d) + 8 * (pr.w - first - sub_level_off(rd, n, d - 1)) + ch;
            A.pos[at] = sub_child_pos(A.pos[pl], ch, d);
            const float* stash = sub_poly_stash();
#pragma unroll
            for (int k = 0; k < 28; ++k) A.poly[(size_t)k * A.cap_live + at] = stash[k * kBlock + threadIdx.x];
        } else {
            const int r = c->sub_rstart[d] + (i - nchild);
            const int node = __ldg(o.sub_root + r);
            me.y = __ldg(o.root_group + r);
            const int* G = o.groups + (size_t)me.y * kGroupRec;
            me.x = -2 - __ldg(o.parent + node);
            me.z = __ldg(o.key + node);
            me.w = __ldg(G + 3) + (r - __ldg(G + 1));
            float q[3] = {0.5f, 0.5f, 0.5f}, w = 0.25f;
            for (int l = depth - 1; l >= depth - d; --l) {
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    q[a] = ((me.z >> (3 * l + 2 - a)) & 1) ? __fadd_rn(q[a], w) : __fsub_rn(q[a], w);
                w = __fmul_rn(w, 0.5f);
            }
            A.pos[at] = make_float4(q[0], q[1], q[2], __int_as_float(d));
            float C[27], mag;
            root_coefficients(r, node, d, q[0], q[1], q[2], depth, o.neigh, o.stride, o.parent, o.enc, o.x,
                              o.root_poly, o.cap_poly, C, mag);
#pragma unroll
            for (int k = 0; k < 27; ++k) A.poly[(size_t)k * A.cap_live + at] = C[k];
            A.poly[(size_t)27 * A.cap_live + at] = mag;
        }
        A.rec[at] = me;
        if (d == depth) A.lv_vnode[pre] = me.w;
    }
    // chains the counts: candidates of depth d + 1 = 8 x live of depth d + roots of d + 1
    __device__ void done(unsigned total) const {
        const int nl = (int)total;
        c->sub_nlive[d] = nl;
        const int cend = c->sub_cbase[d] + c->sub_cand[d];
        if (d < depth) {
            const long long nc = 8LL * nl + c->sub_nroots[d + 1];
            c->sub_cbase[d + 1] = cend;
            c->sub_lbase[d + 1] = c->sub_lbase[d] + nl;
            if (cend + nc > (long long)A.cap_nodes || c->sub_lbase[d] + nl > A.cap_live) {
                atomicOr(err, kErrCapacity);
                c->sub_cand[d + 1] = 0;
            } else {
                c->sub_cand[d + 1] = (int)nc;
            }
        } else {
            // live cells beyond either capacity were not stored (and flagged)
            int n = nl;
            if (n > A.cap_live_d) n = A.cap_live_d;
            if (n > A.cap_live - c->sub_lbase[d]) n = A.cap_live - c->sub_lbase[d];
            c->n_sub_nodes = cend;
            c->n_sub_dnodes = n;
        }
    }
    __device__ void rebase() { PSR_CLOUD(c, o, A, err); }   // to cloud blockIdx.y
};

// The depths 1 .. dmax (at most 8 + 64 + 512 candidates) in one CTA: the scans of so few elements
// cost a launch each otherwise.
__global__ void __launch_bounds__(kBlock) k_sub_coarse(SubLevelLoad load, SubLevelStore store, int dmax) {
    PSR_CLOUD(load, store);
    __shared__ unsigned s_warp[kBlock / 32 + 1];
    for (int d = 1; d <= dmax; ++d) {
        load.d = d;
        store.d = d;
        const int n = *(volatile const int*)&load.c->sub_cand[d];
        unsigned run = 0;
        for (int base = 0; base < n; base += kBlock) {
            load.begin(base);
            const int i = base + (int)threadIdx.x;
            const unsigned v = i < n ? load(i) : 0u;
            unsigned excl;
            const unsigned sum = block_exclusive_scan(v, excl, s_warp);
            if (i < n) store(i, run + excl, v);
            run += sum;
            __syncthreads();
        }
        if (threadIdx.x == 0) store.done(run);
        __syncthreads();   // the depth's records and counts before the next depth reads them
    }
}

// Per live depth-D cell: its neighbour row and jump link, and which vertices and edges it owns.
// A corner is owned by the smallest-key live cell around it (initSubdivideVertexOwner :698-763).
// Cells with a certain sign take no part:
// every corner of a live cell still gets exactly one record, the records of crossing edges
// keep their owners (every cell around a crossing edge has a sign change, so is live), and a
// vertex value does not depend on the cell that evaluates it (the same nonzero terms in the
// same order), so the mesh is unchanged.
// Edges likewise (initSubdivideEdgeArray :812-886).  32 cells per block, as in the level scans.  A
// search of every neighbour's number in the live list took 585 us for 757,000 cells (2,000,000
// samples, depth 9) and the owners another 31 us in a launch of their own; now 197 us.
__global__ void __launch_bounds__(kBlock) k_sub_owners(const Counters* c, int depth, SubTree o, SubArrays A,
                                                       int* group_live, unsigned char* s_vmask,
                                                       unsigned short* s_emask) {
    PSR_CLOUD(c, o, A, group_live, s_vmask, s_emask);
    __shared__ unsigned s_con[32], s_smaller[32];
    const int nl = c->n_sub_dnodes;
    const int lb = c->sub_lbase[depth];
    const int q = threadIdx.x & 7, p = threadIdx.x >> 3;
    for (int L0 = 32 * blockIdx.x; L0 < nl; L0 += 32 * gridDim.x) {
        const int n = min(nl - L0, 32);
        if (threadIdx.x < 32) s_con[threadIdx.x] = s_smaller[threadIdx.x] = 0u;
        __syncthreads();
        const int pp = (int)lane_id();   // a lane a cell, the block's warps share its slots
        if (pp < n) sub_rows(c, o, A, depth, depth, lb + L0 + pp, threadIdx.x >> 5, kBlock / 32, [&](int k, const int4& me, int v) {
            if (v >= o.na) {
                if (k != 13 && A.rec[v - o.na].z < me.z) atomicOr(&s_smaller[pp], 1u << k);
            } else if (v >= 0) {
                s_con[pp] = 1u;
            }
            if (k == 13) {   // a group's live cells are consecutive
                if (L0 + pp == 0 || A.rec[lb + L0 + pp - 1].y != me.y) group_live[me.y] = L0 + pp;
            }
        });
        __syncthreads();
        // eight lanes per cell: a vertex each, then edges q and 8 + q
        const unsigned smaller = s_smaller[p];
        const int sh = threadIdx.x & 24;
        const unsigned mv = __ballot_sync(0xffffffffu, !(smaller & vertex_cells(q))) >> sh;
        const unsigned m0 = __ballot_sync(0xffffffffu, !(smaller & edge_cells(q))) >> sh;
        const unsigned m1 = __ballot_sync(0xffffffffu, q < 4 && !(smaller & edge_cells(8 + (q & 3)))) >> sh;
        if (p < n && q == 0) {
            const int e = lb + L0 + p;
            s_vmask[L0 + p] = (unsigned char)(mv & 0xffu);
            s_emask[L0 + p] = (unsigned short)((m0 & 0xffu) | ((m1 & 0xfu) << 8));
            A.jump[e] = s_con[p] ? e : A.jump[A.rec[e].x];
        }
        __syncthreads();
    }
}

struct SubVertexStore {
    const unsigned char* vmask;
    const Counters* c;
    int depth;
    SubArrays A;
    float *vx, *vy, *vz;
    int *vowner, *vkind;
    int cap;
    unsigned* err;
    __device__ void operator()(int L, unsigned pre, unsigned cnt) const {
        if (!cnt) return;
        if ((int)(pre + cnt) > cap) { atomicOr(err, kErrCapacity); return; }
        const float4 p = A.pos[c->sub_lbase[depth] + L];
        const unsigned m = vmask[L];
        const float hw = 1.0f / (float)(1 << (depth + 1));
        int q = (int)pre;
        for (int k = 0; k < 8; ++k) {
            if (!((m >> k) & 1)) continue;
            vx[q] = __fadd_rn(p.x, (float)(2 * (k & 1) - 1) * hw);
            vy[q] = __fadd_rn(p.y, (float)(2 * ((k >> 1) & 1) - 1) * hw);
            vz[q] = __fadd_rn(p.z, (float)(2 * ((k >> 2) & 1) - 1) * hw);
            vowner[q] = L;
            vkind[q] = k;
            ++q;
        }
    }
    __device__ void rebase() { PSR_CLOUD(vmask, c, A, vx, vy, vz, vowner, vkind, err); }   // to cloud blockIdx.y
};

struct SubEdgeStore {
    const unsigned short* emask;
    int *eowner, *ekind;
    unsigned* edge_of_live;   // sub-edge prefix per live cell (for the part table)
    int cap;
    unsigned* err;
    __device__ void operator()(int L, unsigned pre, unsigned cnt) const {
        edge_of_live[L] = pre;
        if (!cnt) return;
        if ((int)(pre + cnt) > cap) { atomicOr(err, kErrCapacity); return; }
        const unsigned m = emask[L];
        int q = (int)pre;
        for (int e = 0; e < 12; ++e)
            if ((m >> e) & 1) { eowner[q] = L; ekind[q] = e; ++q; }
    }
    __device__ void rebase() { PSR_CLOUD(emask, eowner, ekind, edge_of_live, err); }   // to cloud blockIdx.y
};

// maintainSubdivideVertexNodePointer (:765-810) and maintainSubdivideEdgeNodePointer (:888-949), an
// element kind per blockIdx.z: s_vtx, s_edge indexed by live cell.  They need no clearing: every
// slot of a live cell is written by the owner of that vertex / edge.
__global__ void __launch_bounds__(kBlock) k_sub_maintain(const Counters* c, int depth, SubArrays A, int na, size_t dstride,
                                                         const int* vowner, const int* vkind, int* s_vtx,
                                                         const int* eowner, const int* ekind, int* s_edge) {
    PSR_CLOUD(c, A, vowner, vkind, s_vtx, eowner, ekind, s_edge);
    const int lb = c->sub_lbase[depth];   // a live neighbour's entry is lb + its live index
    if (blockIdx.z == 0) {
        const int V = c->n_sub_vertices;
        PSR_GRID_STRIDE(v, V) {
            const int ow = vowner[v];
            int mx, my, mz, nb[8];
            corner_sides(vkind[v], mx, my, mz);
#pragma unroll
            for (int j = 0; j < 8; ++j)   // all reads before the first store
                nb[j] = A.neigh[(size_t)nslot((j & 1) ? mx : 0, (j & 2) ? my : 0, (j & 4) ? mz : 0) * A.cap_live + lb + ow] - na - lb;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int ax = (j & 1) ? mx : 0, ay = (j & 2) ? my : 0, az = (j & 4) ? mz : 0;
                if (nb[j] >= 0) s_vtx[(size_t)vertex_slot_of(ax, ay, az, mx, my, mz) * dstride + nb[j]] = v + 1;
            }
        }
    } else {
        const int E = c->n_sub_edges;
        PSR_GRID_STRIDE(ei, E) {
            const int ow = eowner[ei], kind = ekind[ei];
            int nb[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int a[3];
                edge_offset(kind, j, a);
                nb[j] = A.neigh[(size_t)nslot(a[0], a[1], a[2]) * A.cap_live + lb + ow] - na - lb;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int a[3];
                edge_offset(kind, j, a);
                if (nb[j] >= 0) s_edge[(size_t)edge_slot_of(kind, a) * dstride + nb[j]] = ei + 1;
            }
        }
    }
}

// implicit values of subdivision vertices (:956-1038): x = 0 inside subdivision space,
// a root stands for the octree node it replaces (same depth and position).  Every
// neighbour of a level is a same-depth cell, so its function index is the level node's
// own plus the slot offset.  A subdivision node's own index comes from its centre
// ((off + 1/2) / 2^d exactly).  The value is the sum, level after level from the owner's
// nearest contributing node up to the root and then 27 neighbour terms in slot order, of
// ((x Fx) Fy) Fz (levels whose 27 neighbours are all zero-valued subdivision nodes add nothing:
// the jump links skip them).  One thread per vertex: its 27 loads of a level are in flight together
// and the next octree row is read during the terms.  Eight lanes per vertex, which form the terms in
// parallel and leave seven idle while one adds them, took 115 us where this takes 25 (60,000 samples
// with clutter, depth 7), and 28 against 17 for the few thousand vertices of 200,000 samples.
__global__ void __launch_bounds__(kBlock) k_sub_vertex_values(const Counters* c, int depth, const float* vx,
                                                              const float* vy, const float* vz, const int* vowner,
                                                              const int* root_self, SubArrays A, ValueRows R,
                                                              float* vvalue, int na) {
    PSR_CLOUD(c, vx, vy, vz, vowner, root_self, A, R, vvalue);
    R.n = min(c->level_base[depth], R.n);
    const int V = c->n_sub_vertices;
    const float iso = c->iso;
    const int lb = c->sub_lbase[depth];
    PSR_GRID_STRIDE(v, V) {
        const float qx = vx[v], qy = vy[v], qz = vz[v];
        // subdivision nodes through the jump links
        float val = 0.0f;
        int node = A.jump[lb + vowner[v]], now;
        while (true) {
            int nbs[27];
#pragma unroll
            for (int k = 0; k < 27; ++k) nbs[k] = A.neigh[(size_t)k * A.cap_live + node];
            const float4 q = A.pos[node];
            const int p = A.rec[node].x;
            const int next = p >= 0 ? A.jump[p] : 0;
            const int d = __float_as_int(q.w);
            const float sc = (float)(1 << d);
            const int base = (1 << d) - 1;
            const int shift = p < 0 ? sub_root_shift(c, d) - na : 0;
#pragma unroll
            for (int k = 0; k < 27; ++k)
                if (nbs[k] >= na) nbs[k] = p < 0 ? root_self[nbs[k] + shift] : -1;
            float xv[27];
#pragma unroll
            for (int k = 0; k < 27; ++k) xv[k] = R.x[nbs[k]];
            val = terms_at(base + (int)__fmul_rn(q.x, sc), base + (int)__fmul_rn(q.y, sc), base + (int)__fmul_rn(q.z, sc),
                           d, xv, val, qx, qy, qz);
            now = -2 - p;
            if (p < 0) break;
            node = next;
        }
        // then the octree ancestors
        if (now >= 0) {
            ValueRow cur, nxt;
            load_row(R, now, cur);
            while (true) {
                load_row(R, cur.parent >= 0 ? cur.parent : 0, nxt);
                val = terms_from(cur.enc, cur.x, val, qx, qy, qz, depth);
                if (cur.parent < 0) break;
                cur = nxt;
            }
        }
        vvalue[v] = __fsub_rn(val, iso);
    }
}

struct SubCrossLoad {
    const int* eowner;   // live cell owning the edge
    const int* ekind;
    const int* s_vtx;
    size_t dstride;
    const float* vvalue;
    unsigned* err;
    __device__ unsigned operator()(int e) const {
        float ab[2];
        edge_values<1>(s_vtx, dstride, vvalue, [&](int, int& dn, int& kind) { dn = eowner[e]; kind = ekind[e]; }, ab, err);
        return (__fmul_rn(ab[0], ab[1]) <= 0.0f) ? 1u : 0u;
    }
    template <int K>
    __device__ bool all(int base, unsigned (&v)[K]) const {
        float ab[2 * K];
        edge_values<K>(s_vtx, dstride, vvalue, [&](int k, int& dn, int& kind) { dn = eowner[base + k]; kind = ekind[base + k]; }, ab, err);
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = (__fmul_rn(ab[2 * k], ab[2 * k + 1]) <= 0.0f) ? 1u : 0u;
        return true;
    }
    __device__ void rebase() { PSR_CLOUD(eowner, ekind, s_vtx, vvalue, err); }   // to cloud blockIdx.y
};
struct SubCrossStore {
    const int* eowner;
    const int* ekind;
    const int* s_vtx;
    size_t dstride;
    const float* vvalue;
    const float *vx, *vy, *vz;
    unsigned* ecross;
    float* part_v;
    const int* voff_ptr;
    int cap;
    unsigned* err;
    __device__ void operator()(int e, unsigned pre, unsigned flag) const {
        ecross[e] = pre;
        if (!flag) return;
        const int at = *voff_ptr + (int)pre;
        if (at >= cap) { atomicOr(err, kErrCapacity); return; }
        const int dn = eowner[e];
        const int kind = ekind[e];
        const int v1 = s_vtx[(size_t)__ldg(&g_tab.edge_vertex[kind][0]) * dstride + dn] - 1;
        const int v2 = s_vtx[(size_t)__ldg(&g_tab.edge_vertex[kind][1]) * dstride + dn] - 1;
        if (v1 < 0 || v2 < 0) return;
        interp_point(vx[v1], vy[v1], vz[v1], vx[v2], vy[v2], vz[v2], kind >> 2, vvalue[v1], vvalue[v2],
                     &part_v[3 * (size_t)at]);
    }
    __device__ void rebase() { PSR_CLOUD(eowner, ekind, s_vtx, vvalue, vx, vy, vz, ecross, part_v, voff_ptr, err); }   // to cloud blockIdx.y
};

struct SubCubeLoad {
    const int* s_vtx;
    size_t dstride;
    const float* vvalue;
    int* cube_class;
    unsigned* err;
    __device__ unsigned operator()(int L) const {
        int p[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) p[q] = s_vtx[(size_t)q * dstride + L];
        float vq[8];
        ptr_values(vvalue, p, vq, err);
        int cls = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (vq[q] < 0.0f) cls |= 1 << q;
        cube_class[L] = cls;
        return (unsigned)__ldg(&g_tab.mc_count[cls]);
    }
    __device__ void rebase() { PSR_CLOUD(s_vtx, vvalue, cube_class, err); }   // to cloud blockIdx.y
};

// triangles of a live cell; indices relative to its group's first crossing (the crossing prefix at
// the first edge of the group's first live cell).  The last element fixes the staged counts.
struct SubCubeStore {
    const int* cube_class;
    const int* s_edge;
    size_t dstride;
    const unsigned* ecross;
    const unsigned* edge_of_live;
    const int* group_live;
    unsigned* tri_of_live;   // sub-triangle prefix per live cell (for the part table)
    Counters* c;
    int depth;
    SubArrays A;
    int* part_t;
    const int* toff_ptr;
    int cap, cap_v;
    int *n_parts, *n_staged_v, *n_staged_t;
    unsigned* err;
    __device__ void operator()(int L, unsigned pre, unsigned cnt) const {
        tri_of_live[L] = pre;
        if (!cnt) return;
        const int g = A.rec[c->sub_lbase[depth] + L].y;
        const unsigned e0 = edge_of_live[group_live[g]];
        const unsigned base = ((int)e0 < c->n_sub_edges) ? ecross[e0] : (unsigned)c->n_sub_cross;
        const int cls = cube_class[L];
        const unsigned long long tri = __ldg(&g_tab.mc_tri[cls]);
        store_triangles(tri, (int)cnt, s_edge + L, dstride, ecross, base, part_t, *toff_ptr + (int)pre, cap, err);
    }
    __device__ void done(unsigned total) const {
        *n_parts = 1 + c->n_groups;
        const int nv = c->n_cross + c->n_sub_cross;
        const int nt = c->n_tri + ((int)total < cap ? (int)total : cap);
        if (nv > cap_v || nt > cap) atomicOr(&c->error, kErrCapacity);
        *n_staged_v = nv < cap_v ? nv : cap_v;
        *n_staged_t = nt < cap ? nt : cap;
    }
    __device__ void rebase() { PSR_CLOUD(cube_class, s_edge, ecross, edge_of_live, group_live, tri_of_live, c, A, part_t, toff_ptr, n_parts, n_staged_v, n_staged_t, err); }   // to cloud blockIdx.y
};

// first live index at or after virtual node v
__device__ __forceinline__ int live_lower_bound(const int* lv_vnode, int n, int v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (lv_vnode[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// per-group first sub edge / first crossing / first triangle -> part table
// parts: [0] main, [1 + g] group g.  part record: vstart, vcount, tstart, tcount.
// A job of the launch that scans the staged vertices.
struct PartTableJob {
    const Counters* c;
    int depth;
    const int* groups;
    const int* lv_vnode;
    const unsigned *edge_of_live, *ecross_sub, *tri_of_live;
    int* parts;
    static constexpr bool kUsed = true;
    __device__ void run(unsigned*) {
        PSR_CLOUD(c, groups, lv_vnode, edge_of_live, ecross_sub, tri_of_live, parts);
        const int ng = c->n_groups;
        const int nE = c->n_sub_edges;
        const int nl = c->n_sub_dnodes;
        if (threadIdx.x == 0 && blockIdx.x == 0) {
            parts[0] = 0;
            parts[1] = c->n_cross;
            parts[2] = 0;
            parts[3] = c->n_tri;
        }
        PSR_GRID_STRIDE(g, ng) {   // one thread per group (independent entries)
            const int* G = groups + (size_t)g * kGroupRec;
            const int v0 = G[3] + sub_level_off(G[0], G[2], depth);
            const int v1 = G[3] + G[4];
            // first sub edge of the group = edge prefix at its first live cell
            const int L0 = live_lower_bound(lv_vnode, nl, v0);
            const int L1 = live_lower_bound(lv_vnode, nl, v1);
            const int e0 = (L0 < nl) ? (int)edge_of_live[L0] : nE;
            const int e1 = (L1 < nl) ? (int)edge_of_live[L1] : nE;
            const unsigned x0 = (e0 < nE) ? ecross_sub[e0] : (unsigned)c->n_sub_cross;
            const unsigned x1 = (e1 < nE) ? ecross_sub[e1] : (unsigned)c->n_sub_cross;
            const unsigned t0 = (L0 < nl) ? tri_of_live[L0] : (unsigned)c->n_sub_tri;
            const unsigned t1 = (L1 < nl) ? tri_of_live[L1] : (unsigned)c->n_sub_tri;
            int* P = parts + 4 * (size_t)(g + 1);
            P[0] = c->n_cross + (int)x0;
            P[1] = (int)(x1 - x0);
            P[2] = c->n_tri + (int)t0;
            P[3] = (int)(t1 - t0);
        }
    }
};

// ------------------------------------------------------------------------------------
// insertion (insertTriangle :1247-1282): drop vertices with |x| < 1e-6, offset triangle
// indices by the vertices kept before the part, drop triangles out of the part's range
// ------------------------------------------------------------------------------------
struct KeepVertexLoad {
    const float* part_v;
    __device__ unsigned operator()(int v) const { return (fabsf(part_v[3 * (size_t)v]) < 1e-6f) ? 0u : 1u; }
    __device__ void rebase() { PSR_CLOUD(part_v); }   // to cloud blockIdx.y
};
struct KeepVertexStore {
    const float* part_v;
    float* mesh_v;
    unsigned* kept_prefix;
    double* nacc;   // normal accumulators, cleared for the transfer (null: no normals)
    int* vcount;
    int cap;
    unsigned* err;
    __device__ void operator()(int v, unsigned pre, unsigned keep) const {
        kept_prefix[v] = pre;
        if (!keep) return;
        if ((int)pre >= cap) { atomicOr(err, kErrCapacity); return; }
        if (nacc) {
            nacc[3 * (size_t)pre] = nacc[3 * (size_t)pre + 1] = nacc[3 * (size_t)pre + 2] = 0.0;
            vcount[pre] = 0;
        }
        mesh_v[3 * (size_t)pre] = part_v[3 * (size_t)v];
        mesh_v[3 * (size_t)pre + 1] = part_v[3 * (size_t)v + 1];
        mesh_v[3 * (size_t)pre + 2] = part_v[3 * (size_t)v + 2];
    }
    __device__ void rebase() { PSR_CLOUD(part_v, mesh_v, kept_prefix, nacc, vcount, err); }   // to cloud blockIdx.y
};

__device__ __forceinline__ int find_part(const int* parts, int np, int t) {
    int lo = 0, hi = np - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (parts[4 * mid + 2] <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// four triangles in three 16-byte loads (the staged triangles start on a 16-byte boundary)
__device__ __forceinline__ void load_tris4(const int* part_t, int base, int (&l)[12]) {
    const int4* p = reinterpret_cast<const int4*>(part_t + 3 * (size_t)base);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const int4 q = p[j];
        l[4 * j] = q.x; l[4 * j + 1] = q.y; l[4 * j + 2] = q.z; l[4 * j + 3] = q.w;
    }
}

// A part is found by bisection, which four consecutive triangles share (one each took 109 us for the
// 1.7 million of 2,000,000 samples, depth 9, now 68; most of the parts may be
// empty, so the next one is bisected too).
struct KeepTriLoad {
    const int* part_t;
    const int* parts;
    const int* np_ptr;
    __device__ unsigned operator()(int t) const {
        const int p = find_part(parts, *np_ptr, t);
        const int vc = parts[4 * p + 1];
        for (int a = 0; a < 3; ++a) {
            int l = part_t[3 * (size_t)t + a];
            if (l < 0 || l >= vc) return 0u;
        }
        return 1u;
    }
    __device__ bool all(int base, unsigned (&v)[4]) const {
        const int np = *np_ptr;
        int l[12];
        load_tris4(part_t, base, l);
        int p = find_part(parts, np, base);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (p + 1 < np && parts[4 * (p + 1) + 2] <= base + k) p = find_part(parts, np, base + k);
            const int vc = parts[4 * p + 1];
            v[k] = 1u;
#pragma unroll
            for (int a = 0; a < 3; ++a)
                if (l[3 * k + a] < 0 || l[3 * k + a] >= vc) v[k] = 0u;
        }
        return true;
    }
    __device__ void rebase() { PSR_CLOUD(part_t, parts, np_ptr); }   // to cloud blockIdx.y
};
struct KeepTriStore {
    const int* part_t;
    const int* parts;
    const int* np_ptr;
    const unsigned* kept_prefix;
    const int* n_staged_v;
    const int* n_kept_v;
    int* mesh_t;
    int cap;
    unsigned* err;
    __device__ int kept_before(int p) const {   // vertices kept before part p
        const int vs = parts[4 * p];
        return (vs < *n_staged_v) ? (int)kept_prefix[vs] : *n_kept_v;
    }
    __device__ void operator()(int t, unsigned pre, unsigned keep) const {
        if (!keep) return;
        if ((int)pre >= cap) { atomicOr(err, kErrCapacity); return; }
        const int prev = kept_before(find_part(parts, *np_ptr, t));
        for (int a = 0; a < 3; ++a) mesh_t[3 * (size_t)pre + a] = part_t[3 * (size_t)t + a] + prev;
    }
    __device__ bool all(int base, unsigned pre, const unsigned (&keep)[4]) const {
        const int np = *np_ptr;
        int l[12];
        load_tris4(part_t, base, l);
        int p = find_part(parts, np, base), prev = kept_before(p);
        bool over = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (p + 1 < np && parts[4 * (p + 1) + 2] <= base + k) {
                p = find_part(parts, np, base + k);
                prev = kept_before(p);
            }
            if (keep[k]) {
                if ((int)pre < cap)
#pragma unroll
                    for (int a = 0; a < 3; ++a) mesh_t[3 * (size_t)pre + a] = l[3 * k + a] + prev;
                else
                    over = true;
                ++pre;
            }
        }
        if (over) atomicOr(err, kErrCapacity);
        return true;
    }
    __device__ void rebase() { PSR_CLOUD(part_t, parts, np_ptr, kept_prefix, n_staged_v, n_kept_v, mesh_t, err); }   // to cloud blockIdx.y
};

// Vertex, edge and face records of the octree: they need only the octree, so they are
// issued on their own stream beside the divergence and the solve (ws.stream, ws.scan and
// the scan total are the caller's for that stream).  The chunks of the coarse divergence and the
// colour cells are counted in the same launches.
cudaError_t mesh_geometry_impl(Workspace& ws, const MeshBufs& mb, unsigned* total, int with_colour) {
    cudaStream_t s = ws.stream;
    const int D = ws.depth;
    Counters* c = ws.cnt;
    unsigned* err = &c->error;
    unsigned* side = (unsigned*)c->scan_total_side;
    const size_t stride = (size_t)ws.cap.nodes;
    const dim3 gm = PSR_GRID(ws, grid_for(ws, ws.cap.nodes));
    const int g = D < kColourGridLevel ? D : kColourGridLevel;
    const int dsplit = div_split(D);
    k_mesh_owners<<<dim3(gm.x, gm.y, with_colour ? 2 : 1), kBlock, 0, s>>>(
        c, D, ws.key, ws.neigh, stride, ws.vmask, ws.emask16, ws.fmask, ws.node_vtx, ws.node_edge, ws.node_face,
        mb.ov_group, mb.ov_sub, ws.cell_start, (1 << (3 * g)) + 1);
    auto vertices = scan_job<1>(PopcLoad8{ws.vmask},
                                VertexStore{ws.vmask, ws.ndepth, ws.ctr_x, ws.ctr_y, ws.ctr_z, ws.v_x, ws.v_y, ws.v_z,
                                            ws.v_owner, ws.v_kind, ws.v_depth, ws.cap.vertices, err},
                                &c->n_nodes, ws.scan, total, ScanCount{&c->n_vertices, ws.cap.vertices});
    auto faces = scan_job<1>(PopcLoad8{ws.fmask},
                             FaceStore{ws.fmask, ws.key, ws.ndepth, ws.parent, D, ws.f_owner, ws.f_kind, ws.f_hasparent,
                                       ws.face_hit, ws.cap.faces, err},
                             &c->n_nodes, ws.scan_side[0], side, ScanCount{&c->n_faces, ws.cap.faces});
    auto edges = scan_job<1>(PopcLoad16{ws.emask16},
                             EdgeStore{ws.emask16, &c->level_base[D], ws.e_owner, ws.e_kind, ws.cap.edges, err},
                             &c->level_count[D], ws.scan_side[1], side + 1, ScanCount{&c->n_edges, ws.cap.edges});
    cudaError_t e;
    if (dsplit > 0)
        e = launch_scans(scan_job<1>(DivChunkLoad{ws.neigh, stride, ws.dnum},
                                     DivChunkStore{(unsigned*)ws.cg_p, c, ws.cap.nodes},   // as many float pairs
                                     &c->level_base[dsplit], ws.scan_side[2], side + 2),
                         vertices, faces, edges, err, s);
    else
        e = launch_scans(vertices, faces, edges, NoScan{}, err, s);
    if (e == cudaSuccess && !ws.chain) e = cudaEventRecord(ws.ev_geo, s);
    if (e != cudaSuccess) return e;
    k_mesh_maintain<<<dim3(gm.x, gm.y, with_colour ? 4 : 3), kBlock, 0, s>>>(
        c, D, ws.neigh, stride, ws.v_owner, ws.v_kind, ws.node_vtx, ws.e_owner, ws.e_kind, ws.node_edge, ws.f_owner,
        ws.f_kind, ws.node_face, g, ws.key, ws.point2node, ws.cell_start);
    return cudaGetLastError();
}

cudaError_t mesh_build_impl(Workspace& ws, const MeshBufs& mb) {
    cudaStream_t s = ws.stream;
    const int D = ws.depth;
    Counters* c = ws.cnt;
    unsigned* err = &c->error;
    unsigned* total = (unsigned*)&c->scan_total;
    const size_t stride = (size_t)ws.cap.nodes;
    const int gm = grid_for(ws, ws.cap.nodes);
    cudaError_t e;
    // implicit values
    if (D >= 8)
        k_vertex_values_rows<<<PSR_GRID(ws, gm), kBlock, 0, s>>>(c, D, ws.v_x, ws.v_y, ws.v_z, ws.v_owner, ws.v_kind,
                                                                 ws.v_depth, value_rows(ws), ws.vvalue);
    else
        k_vertex_values<<<PSR_GRID(ws, gm), kBlock, 0, s>>>(c, D, ws.v_x, ws.v_y, ws.v_z, ws.v_owner, ws.v_kind, ws.v_depth, ws.neigh,
                                              stride, ws.parent, ws.first_child, ws.enc, ws.xsol, ws.vvalue);
    // crossings -> staged vertices of the main part
    e = launch_scan<4>(CrossLoad{ws.e_owner, ws.e_kind, ws.node_vtx, stride, ws.vvalue, err},
                    CrossStore{ws.e_owner, ws.e_kind, ws.node_vtx, stride, ws.vvalue, ws.v_x, ws.v_y, ws.v_z,
                               ws.e_cross, ws.part_v, 0, ws.part_cap_v, err},
                    &c->n_edges, 0, ws.scan, total, err, s, ScanCount{&c->n_cross, ws.part_cap_v});
    if (e != cudaSuccess) return e;
    e = launch_scan<1>(CubeLoad{ws.node_vtx, stride, &c->level_base[D], ws.vvalue, ws.cube_class, err},
                    CubeStore{ws.cube_class, &c->level_base[D], ws.node_edge, ws.node_face, stride, ws.e_cross,
                              ws.parent, ws.f_hasparent, ws.face_hit, ws.part_t, 0, ws.part_cap_t, err},
                    &c->level_count[D], 0, ws.scan, total, err, s, ScanCount{&c->n_tri, ws.part_cap_t});
    if (e != cudaSuccess) return e;
    // subdivision roots among nodes of depth < D
    e = launch_scan<1>(RootLoad{ws.node_vtx, ws.node_face, stride, ws.vvalue, ws.face_hit, ws.first_child, err},
                    RootStore{c, D, ws.sub_root, ws.cap.nodes, err}, &c->level_base[D], 0, ws.scan, total, err, s, ScanCount{&c->n_subroots, ws.cap.nodes});
    if (e != cudaSuccess) return e;
    k_root_setup<<<PSR_GRID(ws, 4 * ws.num_sms), kBlock, 0, s>>>(
        c, D, ws.sub_root, ws.ndepth, ws.key, ws.root_group, mb.groups, mb.max_groups, ws.cap.nodes, ws.root_self, mb.ov_group, mb.ov_sub, ws.ctr_x,
        ws.ctr_y, ws.ctr_z, ws.neigh, stride, ws.parent, ws.enc, ws.xsol, ws.root_poly, ws.cap_poly, ws.cap.sub_nodes);
    return cudaGetLastError();
}

// Subdivision nodes appear in neighbour tables as cap.nodes + virtual index: every such
// number is larger than any octree index, which is all the kernels compare against.
cudaError_t mesh_build_sub(Workspace& ws, const MeshBufs& mb) {
    cudaStream_t s = ws.stream;
    const int D = ws.depth;
    Counters* c = ws.cnt;
    unsigned* err = &c->error;
    unsigned* total = (unsigned*)&c->scan_total;
    unsigned* side = (unsigned*)c->scan_total_side;
    const size_t stride = (size_t)ws.cap.nodes;
    const size_t dstride = (size_t)ws.cap.sub_dnodes;
    const int na = ws.cap.nodes;
    // kernels over live depth-D cells and the scans of the subdivision: sized for a few
    // thousand live cells (one block per SM, grid-stride beyond) up to depth 7; the trees of
    // depth 8 and 9 have hundreds of thousands to millions, four blocks per SM
    const int gl = D >= 8 ? 4 * ws.num_sms : ws.num_sms;
    const int sbps = D >= 8 ? 4 : 1;
    cudaError_t e;
    const SubTree o{mb.groups, ws.sub_root, ws.root_group, ws.key, ws.neigh, stride, ws.first_child, ws.parent,
                    mb.ov_group, mb.ov_sub, ws.enc, ws.xsol, ws.root_poly, ws.cap_poly, na};
    const SubArrays A{ws.c_rec, ws.c_pos, ws.c_jump, ws.c_kids, ws.c_neigh, ws.c_poly, ws.lv_vnode,
                      ws.cap.sub_nodes, ws.cap.sub_live, ws.cap.sub_dnodes};
    // depth after depth: candidates (children of the live nodes above, then the roots of this
    // depth) and their sign tests; the live ones are compacted in order
    const int dcoarse = D < 3 ? D : 3;
    k_sub_coarse<<<PSR_GRID(ws, 1), kBlock, 0, s>>>(SubLevelLoad{c, 1, D, o, A}, SubLevelStore{c, 1, D, o, A, err}, dcoarse);
    for (int d = dcoarse + 1; d <= D; ++d) {
        e = launch_scan<1>(SubLevelLoad{c, d, D, o, A}, SubLevelStore{c, d, D, o, A, err}, &c->sub_cand[d], 0, ws.scan,
                           total, err, s, ScanCount{}, sbps);
        if (e != cudaSuccess) return e;
    }
    // the live depth-D cells carry every record from here on, indexed by their live index
    k_sub_owners<<<PSR_GRID(ws, 2 * gl), kBlock, 0, s>>>(c, D, o, A, mb.group_live, ws.s_vmask, ws.s_emask);
    e = launch_scans(scan_job<2>(PopcLoad8{ws.s_vmask},
                                 SubVertexStore{ws.s_vmask, c, D, A, ws.sv_x, ws.sv_y, ws.sv_z, ws.sv_owner, ws.sv_kind,
                                                8 * ws.cap.sub_dnodes, err},
                                 &c->n_sub_dnodes, ws.scan, total, ScanCount{&c->n_sub_vertices, 8 * ws.cap.sub_dnodes}),
                     scan_job<2>(PopcLoad16{ws.s_emask},
                                 SubEdgeStore{ws.s_emask, ws.se_owner, ws.se_kind, mb.edge_of_dnode,
                                              12 * ws.cap.sub_dnodes, err},
                                 &c->n_sub_dnodes, ws.scan_side[0], side,
                                 ScanCount{&c->n_sub_edges, 12 * ws.cap.sub_dnodes}),
                     NoScan{}, NoScan{}, err, s, sbps);
    if (e != cudaSuccess) return e;
    const dim3 g2 = PSR_GRID(ws, gl);
    k_sub_maintain<<<dim3(g2.x, g2.y, 2), kBlock, 0, s>>>(c, D, A, na, dstride, ws.sv_owner, ws.sv_kind, ws.s_vtx,
                                                          ws.se_owner, ws.se_kind, ws.s_edge);
    k_sub_vertex_values<<<PSR_GRID(ws, 8 * ws.num_sms), kBlock, 0, s>>>(
        c, D, ws.sv_x, ws.sv_y, ws.sv_z, ws.sv_owner, ws.root_self, A, value_rows(ws), ws.sv_value, na);
    // crossings: staged after the main part's vertices
    e = launch_scan<4>(SubCrossLoad{ws.se_owner, ws.se_kind, ws.s_vtx, dstride, ws.sv_value, err},
                       SubCrossStore{ws.se_owner, ws.se_kind, ws.s_vtx, dstride, ws.sv_value, ws.sv_x, ws.sv_y,
                                     ws.sv_z, ws.se_cross, ws.part_v, &c->n_cross, ws.part_cap_v, err},
                       &c->n_sub_edges, 0, ws.scan, total, err, s, ScanCount{&c->n_sub_cross, ws.part_cap_v}, sbps);
    if (e != cudaSuccess) return e;
    int* n_parts = mb.misc;
    int* n_staged_v = mb.misc + 1;
    int* n_staged_t = mb.misc + 2;
    e = launch_scan<2>(SubCubeLoad{ws.s_vtx, dstride, ws.sv_value, ws.s_cube_class, err},
                       SubCubeStore{ws.s_cube_class, ws.s_edge, dstride, ws.se_cross, mb.edge_of_dnode, mb.group_live,
                                    mb.tri_of_dnode, c, D, A, ws.part_t, &c->n_tri, ws.part_cap_t, ws.part_cap_v, n_parts,
                                    n_staged_v, n_staged_t, err},
                       &c->n_sub_dnodes, 0, ws.scan, total, err, s, ScanCount{&c->n_sub_tri, ws.part_cap_t}, sbps);
    if (e != cudaSuccess) return e;
    // insertion of all parts
    e = launch_scans(scan_job<2>(KeepVertexLoad{ws.part_v},
                                 KeepVertexStore{ws.part_v, ws.mesh_v, mb.kept_prefix,
                                                 ws.want_normals ? ws.nacc : nullptr, ws.vcount, ws.cap.mesh_vertices, err},
                                 n_staged_v, ws.scan, total, ScanCount{&c->n_mesh_vertices, ws.cap.mesh_vertices}),
                     PartTableJob{c, D, mb.groups, ws.lv_vnode, mb.edge_of_dnode, ws.se_cross, mb.tri_of_dnode, mb.parts},
                     NoScan{}, NoScan{}, err, s, sbps);
    if (e != cudaSuccess) return e;
    e = launch_scan<4>(KeepTriLoad{ws.part_t, mb.parts, n_parts},
                    KeepTriStore{ws.part_t, mb.parts, n_parts, mb.kept_prefix, n_staged_v, &c->n_mesh_vertices,
                                 ws.mesh_t, ws.cap.mesh_tris, err},
                    n_staged_t, 0, ws.scan, total, err, s, ScanCount{&c->n_mesh_triangles, ws.cap.mesh_tris}, sbps);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace psr

namespace psr {
cudaError_t mesh_geometry(Workspace& ws, int with_colour) {
    return mesh_geometry_impl(ws, ws.mb, (unsigned*)&ws.cnt->scan_total_aux, with_colour);
}

cudaError_t mesh_build(Workspace& ws) {
    cudaError_t e = mesh_build_impl(ws, ws.mb);
    if (e != cudaSuccess) return e;
    return mesh_build_sub(ws, ws.mb);
}
}  // namespace psr
