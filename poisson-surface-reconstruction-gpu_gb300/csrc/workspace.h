// Device workspace of one reconstruction handle.  Every buffer is allocated once at
// handle creation from the configured capacities; a reconstruction never allocates.
//
// HBM layout (structure of arrays, one array per field):
//   points   : sorted positions / scaled normals / colours, 3 x N floats each
//   nodes    : key, pidx, pnum, parent, first_child, didx, dnum, depth, enc (int32 x M),
//              centre (3 x M floats), neighbour table [27][M] int32,
//              vertex / edge / face back-pointers [8|12|6][M] int32
//   build    : level-by-level staging arrays used while the octree is assembled
//   mesh     : vertex / edge / face records, implicit values, output vertices/triangles
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include "primitives.cuh"

namespace psr {

struct Caps {
    int points;        // N cap
    int nodes;         // M cap (all depths)
    int dnodes;        // D-level node cap
    int vertices;      // octree vertex records
    int edges;         // D-level edge records
    int faces;         // face records
    int sub_nodes;     // subdivision-space nodes (all groups of one reconstruction)
    int sub_dnodes;    // live D-level subdivision cells
    int sub_live;      // live subdivision nodes of all depths
    int mesh_vertices; // output vertex cap
    int mesh_tris;     // output triangle cap
    int scan_tiles;    // tiles of the largest scan
};

// mesh-stage scratch
struct MeshBufs {
    int* ov_group;             // [8][cap.nodes]: group whose root redirects this child slot
    int* ov_sub;               // [8][cap.nodes]: root slot inside that group
    int* groups;               // group records (see mesh.cu)
    int max_groups;
    unsigned* edge_of_dnode;   // sub-edge prefix per live depth-D cell
    unsigned* tri_of_dnode;    // sub-triangle prefix per live depth-D cell
    int* group_live;           // per group: its first live depth-D cell
    int* parts;                // per output part: vertex start / count, triangle start / count
    unsigned* kept_prefix;     // per staged vertex: kept vertices before it
    int* misc;                 // [0] parts, [1] staged vertices, [2] staged triangles
};

struct Workspace {
    int batch = 1;          // clouds of the launches being issued (the grids' y extent)
    bool want_normals = false;   // the call's mesh gets vertex normals
    bool chain = false;     // the pipeline is issued as one chain, without forks (depths up to 7)
    int cg_ctas = 0;        // CTAs of the depth-D CG cluster (0: the largest the device runs, 16)
    int cg_ctas_fine = 0;   // CTAs of each depth-(D-1), (D-2) CG cluster (0: 8)
    MeshBufs mb;
    Caps cap;
    int depth;
    Counters* cnt;          // device
    Counters* cnt_host;     // pinned mirror for the final read-back
    ScanScratch scan;
    ScanScratch scan_aux;   // scans issued on the geometry stream (aux2) while `scan` is in use
    ScanScratch scan_side[3];   // scans that run beside another one in its launch
    SortScratch sort;
    unsigned* scan_total;   // device scratch (points into cnt)

    // input staging (device copies of host inputs, or caller's device pointers)
    float* in_xyz;
    float* in_nrm;
    uint8_t* in_rgb;

    // sort
    unsigned *code, *sidx;

    // sorted points (SoA)
    float *px, *py, *pz, *nx, *ny, *nz, *cr, *cg, *cb;
    int* point2node;        // D-level local index of each sorted point
    int* puid;              // unique-leaf id of each sorted point
    unsigned* ucode;        // unique leaf codes
    int* ufirst;            // first sorted point of each unique leaf (+ sentinel)
    int* uslot;             // D-level slot of each unique leaf

    // level build staging (levels D, D-1, ..., 0 appended in that order)
    int *tkey, *tpidx, *tpnum, *tdidx, *tdnum, *tchild;
    int* tparent_slot;      // per group of 8: slot of its father one level up
    int *gkey, *gpidx, *gpnum, *gdidx, *gdnum;   // per-group aggregates of the current level
    unsigned* gaddr;

    // final node arrays
    int *key, *pidx, *pnum, *parent, *first_child, *didx, *dnum, *ndepth, *enc;
    float *ctr_x, *ctr_y, *ctr_z;
    int* neigh;             // [27][cap.nodes]
    int* node_vtx;          // [8][cap.nodes]
    int* node_edge;         // [12][cap.nodes]
    int* node_face;         // [6][cap.nodes]

    // function tables (FP64, res x res) and per-depth stencil coefficients
    int res;
    float* dff;             // d/dx F_i . F_j rounded to float (index res * i + j)
    float* stencil;         // [D+1][27] Laplacian coefficients (0 where dropped)

    // field / solve
    float* vfield;          // 3 x dnodes (SoA: x block, y block, z block)
    float4* leaf;           // dnodes: the field and the packed function index of each depth-D node
    float* divg;            // M
    float* xsol;            // M, with xsol[-1] = 0
    cudaEvent_t ev_cg = nullptr;   // recorded right after the CG kernel (stage timing)
    unsigned ev_flags = 0;         // flags of the stage-timing event records (external in a capture)
    float2* cg_p;           // M: (r, p) of the cluster CG's global-memory path; before the solve, where the
                            //   coarse divergence's chunks start
    float *cg_q, *cg_ap;    // x (sibling-major) and A p of the whole-GPU CG; A p of the global-memory path
    int* cg_nbg;            // [27][cap.nodes / 8 + 8]: neighbour groups of every sibling group (whole-GPU CG)
    float2* cg_rp;          // [8][cap.nodes / 8 + 8]: (r, p), sibling-major
    float4* value_rows;     // after the CG of a tree of depth 8 or 9, in its vectors: [8] per node (ValueRows)
    int cap_rows;
    ulonglong2* cg_part;    // [2][cg_part_cap]: sums of its virtual blocks
    int cg_part_cap;
    unsigned* cg_desc;      // [14][cap.nodes / 8 + 8]: packed neighbour groups (solver.cu)
    double* cg_partial;     // scratch: divergence chunk sums (float pairs, 8 bytes each)
    float* point_val;       // N
    float* pv_coef;         // [27][cap.dnodes / 8 + 64]: per depth-(D-1) node, Bernstein coefficients
    double* iso_partial;

    // mesh geometry
    unsigned char* vmask;   // per node: owned corner mask (8 bits)
    unsigned short* emask16;   // per D node: owned edge mask (12 bits)
    unsigned char* fmask;   // per node: owned face mask (6 bits)
    float *v_x, *v_y, *v_z; // vertex positions
    int *v_owner, *v_kind, *v_depth;
    int *e_owner, *e_kind;
    int *f_owner, *f_kind, *f_hasparent;
    float* vvalue;          // implicit value - iso at every vertex
    unsigned* e_cross;      // per edge: staged vertex index of its crossing (exclusive scan)
    int* cube_class;        // per D node
    int* face_hit;          // per face: surface-edge intersection

    // subdivision
    int* sub_root;          // node index of each root (node order)
    int* root_group;        // per subdivision root: its group
    int* root_self;         // per root: the octree node it stands for
    float* root_poly;       // [28][cap_poly]: per root, Bernstein coefficients of the levels up to it
    int cap_poly;
    // live subdivision nodes, depth after depth (capacity cap.sub_live)
    int4* c_rec;            // parent, group, key, virtual index
    float4* c_pos;          // centre, depth
    int* c_jump;            // nearest contributing node on the path to the root
    int2* c_kids;           // live children: first entry, octant bits
    int* c_neigh;           // [27][cap.sub_live]
    float* c_poly;          // [28][cap.sub_live]: Bernstein coefficients, sum |y|
    // live depth-D cells (capacity cap.sub_dnodes)
    int* lv_vnode;          // virtual index, ascending
    int *s_vtx, *s_edge;    // [8|12][cap.sub_dnodes]
    unsigned char* s_vmask;
    unsigned short* s_emask;
    float *sv_x, *sv_y, *sv_z;
    int *sv_owner, *sv_kind;
    float* sv_value;
    int *se_owner, *se_kind;
    unsigned* se_cross;
    int* s_cube_class;

    // output (device)
    float* mesh_v;          // 3 x mesh_vertices
    int* mesh_t;            // 3 x mesh_tris
    float* mesh_c;          // colours
    float* mesh_n;          // normals
    double* nacc;           // per output vertex normal accumulator (3 doubles)
    int* vcount;            // per output vertex triangle count
    int* cell_start;        // sample grid for the colour search
    int* colour_far;        // (vertex, bound) pairs the near colour search left
    // vertex welding (allocated only when the handle welds)
    int* weld_table = nullptr;   // hash slots: a vertex of the class, then its smallest index
    unsigned weld_mask = 0;      // slots - 1 (a power of two >= 2 x mesh vertex capacity)
    int* weld_slot = nullptr;    // slot of every vertex's class
    int* weld_newid = nullptr;   // welded number of every representative
    float* weld_v = nullptr;     // compacted positions

    // staging for the two-phase insertion of each mesh part
    float* part_v;          // 3 x cap
    int* part_t;
    int part_cap_v, part_cap_t;

    InputRef* d_params;     // the current call's input (written by its first kernel)
    const InputRef* h_params;   // and where that reads it: pinned host memory, one per cloud slot

    cudaStream_t stream;
    cudaStream_t aux = nullptr;         // second stream for work forked off `stream`
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    cudaStream_t aux2 = nullptr;        // third stream: octree-only mesh records beside the solve
    cudaEvent_t ev_fork2 = nullptr, ev_join2 = nullptr;
    cudaEvent_t ev_geo = nullptr;       // the mesh records' scans (and the divergence chunks') are done
    cudaStream_t aux3 = nullptr;        // fourth stream: the CG of depths D-1 and D-2
    cudaEvent_t ev_join3 = nullptr;
    int num_sms;
};

// sample grid of the colour search: 2^g cells per axis (128^3: a few samples per surface
// cell at 200k points)
constexpr int kColourGridLevel = 7;

// launch grid for the clouds of the batch being issued (gx blocks for one cloud)
#define PSR_GRID(ws, gx) dim3(::psr::cloud_blocks((ws).batch, (gx)), (ws).batch)

// the clouds of the next launches (every scan scratch copy carries the count too)
inline void set_batch(Workspace& ws, int clouds) {
    ws.batch = clouds;
    ws.scan.batch = clouds;
    ws.scan_aux.batch = clouds;
    for (auto& sc : ws.scan_side) sc.batch = clouds;
    ws.sort.batch = clouds;
}

// grid of a grid-stride kernel over `work` items: enough blocks, at most 8 per SM
inline int grid_for(const Workspace& ws, long long work) {
    long long g = (work + kBlock - 1) / kBlock;
    long long cap = (long long)ws.num_sms * 8;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

// coarse divergence: depths below div_split(D) are summed in chunks of kDivChunk leaves, the others a
// warp per node.  A chunk ends with its neighbour, so at depth 9 those of depth 6 hold 77 leaves each
// (2,000,000 samples) and cost more to find than to add: from depth 8 on the line is at depth 5 (field
// and divergence 2.45 ms; with it at D - 2 = 7 2.55 ms, at 4 2.64 ms, where a node's 12,000 terms take a
// warp too long).  Trees of depth 7 keep D - 2 = 5 by the same measure.
constexpr int kDivChunk = 512;
inline int div_split(int D) { return D >= 8 ? 5 : (D >= 2 ? D - 2 : 0); }

inline ValueRows value_rows(const Workspace& ws) {   // none below depth 8
    return ValueRows{ws.value_rows, ws.depth >= 8 ? ws.cap_rows : 0, ws.neigh, (size_t)ws.cap.nodes, ws.parent, ws.first_child, ws.enc, ws.xsol};
}

// stage entry points (each issues kernels on ws.stream; no host synchronisation)
cudaError_t octree_build(Workspace& ws);
void prepare_launch_configs(Workspace& ws);
cudaError_t field_build(Workspace& ws);
// res_period: true residual every res_period CG iterations and at convergence (0: only at
// convergence, < 0: never)
cudaError_t solve_build(Workspace& ws, int cg_mode, int cg_iters, float cg_tol, int cg_max_iter, int res_period);
// vertex / edge / face records, divergence chunks, and the colour search's sample grid (octree and
// points only)
cudaError_t mesh_geometry(Workspace& ws, int with_colour);
cudaError_t mesh_build(Workspace& ws);      // values, marching cubes, subdivision, compaction
cudaError_t transfer_prepare(Workspace& ws, int with_colour);   // last step of the sample grid
cudaError_t transfer_build(Workspace& ws, int with_colour, int with_normals);

}  // namespace psr
