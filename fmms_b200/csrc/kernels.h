// Kernel declarations and the device-side structures shared between the
// kernel files and the host orchestration (engine.cu).
#pragma once

#include <vector>

#include "common.cuh"

namespace fmmx {

// first position of each level in the level lists
struct LevelStarts {
    int start[FMMX_NLEVELS];
};

struct CellsMut {
    uint32_t* first;
    uint32_t* count;
    int32_t* child;
    int32_t* parent;
    uint8_t* leaf;
    uint8_t* level;
    double* cx;
    double* cy;
    double* cz;
    double* mass;
    double* rho;
};

struct MacParams {
    int p;
    double eps;
    double theta;
    double gap;  // minimum separation of the bodies of an M2L pair (soft_gap * softening); 0: none
};

// Pool of list chunks of the walk: 32 entries each, each of one list.
struct WalkPool {
    uint32_t* entry;  // 32 cap
    uint32_t* next;   // cap: the following chunk of a list passed down
    uint2* owner;     // cap: whose entries the chunk of an M2L or P2P list holds (x: all bits set, nobody's); set by the
                      // walk for every chunk reserved, so nothing is cleared before it
    uint32_t cap;     // chunks
    unsigned* used;   // chunks reserved; above cap after an overflow, but also where only the unused tails of the
                      // last reservations (up to 16 chunks per block) lie beyond the pool
    int* overflow;    // set when a chunk was refused: the lists are incomplete
};

// Per-cell results of the walk: the list passed down to the children (entries
// and first chunk), whether the cell was walked a second time (as a heavy one),
// and the lists' sizes with the near field's work units and partial sums (m2l,
// p2p, units, scratch).
struct WalkLists {
    uint32_t* down_n;
    uint32_t* down_head;
    uint8_t* redone;
    uint4* sizes;                // ncells + 1
    // pairs examined, body interactions, directed M2L and P2P entries; k_near_sizes: work units, partial sums
    unsigned long long* totals;
};

// Directed interaction list: for destination cell c, the sources src[seg_begin[c]
// .. seg_end[c]), in the walk's order.
struct DirList {
    const uint32_t* src;
    const uint32_t* seg_begin;
    const uint32_t* seg_end;
};

// tree_exact.cu
void upload_tables_exact(const OrderTables& t, cudaStream_t s);
__global__ void k_bbox_partial(const double* pos, size_t n, double* part, int* bad);
__global__ void k_bbox_final(const double* part, int nparts, double* box);
__global__ void k_keys(const double* pos, size_t n, const double* box, uint64_t* keys, uint32_t* idx);
__global__ void k_gather(const double* pos, const double* mass, const uint32_t* order, size_t n, double* x,
                         double* y, double* z, double* m);
__global__ void k_bbox_seg(const double* pos, size_t n, const uint64_t* off, int nsys, unsigned long long* enc,
                           int* bad);
__global__ void k_bbox_seg_final(const unsigned long long* enc, int nsys, double* box);
#define BBOX_CHUNK 2048  // bodies per block of k_bbox_seg
__global__ void k_keys_seg(const double* pos, size_t n, const uint64_t* off, int nsys, const double* box,
                           uint64_t* keys, uint32_t* idx);
__global__ void k_entry_system(const uint32_t* order, size_t n, const uint64_t* off, int nsys, uint32_t* sys,
                               uint32_t* at);
__global__ void k_permute_entries(const uint32_t* at, size_t n, const uint64_t* keys_in, const uint32_t* order_in,
                                  uint64_t* keys, uint32_t* order);
#define TREE_BLOCK 256
#define TREE_PER_THREAD 4  // slots per thread of the two tree kernels
__global__ void k_cell_count(const uint64_t* keys, uint32_t n, const uint64_t* off, int nsys, uint32_t n_leaf,
                             uint32_t* count, int* lvl);
__global__ void k_cell_emit(const uint64_t* keys, uint32_t n, const uint64_t* off, int nsys, uint32_t n_leaf,
                            const uint32_t* id0, LevelStarts ls, int* cursor, const double* box, CellsMut cells,
                            int32_t* level_cells, int32_t* body_leaf, double* h);
#define GEO_WARPS 4
__global__ void k_geometry_com(int nc, CellsMut cells, const double* x, const double* y, const double* z,
                               const double* m, unsigned* arrive, double4* geo);
__global__ void k_geometry_ritter(const int32_t* level_cells, int lstart, int lcnt, CellsMut cells, const double* x,
                                  const double* y, const double* z, const double* m);
// bodies per round of the exact P2M (the lanes of a warp build that many Υ tables at once)
__host__ __device__ inline int p2m_round(int p) { return p <= 12 ? 32 : (p <= 16 ? 16 : 8); }
__host__ __device__ size_t upward_exact_smem_per_warp(int p);
__global__ void k_upward_exact(const int32_t* level_cells, int lstart, int lcnt, CellsView cells, const double* x,
                               const double* y, const double* z, const double* m, int p, zd* moments, double* pows);
#define M2M_EXACT_WIDE 512  // threads where a level has few cells
__global__ void k_m2m_exact_block(const int32_t* level_cells, int lstart, int lcnt, CellsView cells, int p,
                                  zd* moments, double* pows);
__global__ void k_fmin(int nc, CellsView cv, const int32_t* parent, const double* f, double* fmin_out,
                       unsigned* arrive);
#define FPRE_WARPS 2
void launch_fprepass(cudaStream_t s, CellsView cells, const double* x, const double* y, const double* z,
                     const double* m, size_t n, const uint64_t* off, int nsys, const int32_t* roots, double* f,
                     int* err);
__global__ void k_pack_geo(int nc, CellsMut cells, double4* geo);

// Cells whose walk is left to many warps: their ids, and a queue of ring_cap
// sources for each of `blocks` blocks.
struct WalkHeavy {
    int32_t* list;
    int* count;  // of the level, zero at its start
    uint32_t* ring;
    uint32_t ring_cap;
    unsigned blocks;
};

// walk.cu
void upload_tables_walk(const OrderTables& t, cudaStream_t s);
// rows of p + 2 per cell for Dehnen's MAC
__global__ void k_mac_rows(int nc, CellsView cv, int p, const double* pows, const double* fminv, double2* rows);
// The cells of one level (Dehnen's error-estimate MAC, else theta and soft_gap); work, heavy_work: zero
// counters. Returns the launches.
int launch_walk_level(bool dehnen, cudaStream_t s, const int32_t* level_cells, int lcnt, int nleaves, CellsView cv,
                      const int32_t* parent, MacParams mp, const double2* rows, WalkPool P, WalkLists Ls, WalkHeavy heavy,
                      int* work, int* heavy_work);
bool walk_needs_heavy(const int* lvl_count, int nlevels, int nleaves);
unsigned walk_heavy_blocks(int nleaves);
// contiguous lists from the first nchunks chunks (at most P.cap); off: the exclusive sums of W.sizes
void launch_lists_gather(cudaStream_t s, int nc, uint32_t nchunks, WalkPool P, WalkLists W, const uint4* off, uint32_t* m2l_off,
                         uint32_t* p2p_off, uint32_t* uoff, uint32_t* soff, uint32_t* m2l, uint32_t* p2p,
                         int32_t* ucell);

// lists.cu
// exclusive prefix sums of n values, and of four at once
size_t scan_u32_temp(int n);
cudaError_t scan_u32(void* tmp, size_t tmp_bytes, const uint32_t* in, uint32_t* out, int n, cudaStream_t s);
size_t scan_u32x4_temp(int n);
cudaError_t scan_u32x4(void* tmp, size_t tmp_bytes, const uint4* in, uint4* out, int n, cudaStream_t s);

// m2l.cu
void upload_tables_m2l(const OrderTables& t, cudaStream_t s);
size_t m2l_rot_smem_bytes(int p);
__global__ void k_m2l_naive_f64(DirList L, int ncells, CellsView cv, int p, const zd* moments, zd* locals);
__global__ void k_m2l_rot_f64(DirList L, int ncells, CellsView cv, int p, const zd* moments, zd* locals,
                              const double* swap_g);

// sweeps.cu
void upload_tables_sweeps(const OrderTables& t, cudaStream_t s);
__global__ void k_l2l_f64(const int32_t* level_cells, int lstart, int lcnt, CellsView cv, const int32_t* parent,
                          int p, zd* locals);
__global__ void k_l2p_f64(size_t n, const int32_t* body_leaf, const uint32_t* order, CellsView cv, int p,
                          const zd* locals, const double* x, const double* y, const double* z, const double* nax,
                          const double* nay, const double* naz, const double* npot, double* acc, double* pot);

// p2p.cu
// Near-field work units (both forms): up to P2P_NT targets of a leaf against a
// share of its source leaves, a warp each. Units of cell c: uoff[c] ..
// uoff[c+1], ucell[u] the cell of unit u; the partial sums of a leaf with
// several shares at part[soff[c] + share * count + i].
#define P2P_NT 32
struct P2pUnits {
    const uint32_t* uoff;  // ncells + 1
    const int32_t* ucell;  // nunits
    const uint32_t* soff;  // ncells + 1
    double4* part;
    unsigned* next;  // work counter, zero at launch
    uint32_t nunits;  // below 2^31: the counter passes it by one per warp
};

// Work units of the near field, a warp each: up to P2P_NT targets of a leaf
// against an equal share of its source leaves, p2p_shares(targets, sources, grain)
// of them. The share depends on the leaf alone -- about the same work per unit,
// `grain` target-source-leaf products -- so a leaf in a dense core with thousands
// of neighbours, or one of few leaves of a small system, spreads over many warps
// (the load-balancing aim of the reference's split_fat, crates/visual/src/
// gpufmm.rs:1350-1414). A leaf with one share writes its bodies' sums directly;
// the shares of the others write partial sums, which k_p2p_combine adds per
// body in share order (a fixed order: the results do not depend on which warp
// ran which unit). The grain is P2P_GRAIN unless the partial sums (32 bytes for
// every body and share of a split leaf; leaves of 250 bodies with 10^3 sources each:
// 600 bytes a body) are more than 2^32 - 1 or than the memory holds; the walk
// then takes a coarser one, in the end P2P_WHOLE: one share a leaf, no partial sums.
#define P2P_GRAIN 2048u
#define P2P_WHOLE 0xffffffffu
__host__ __device__ __forceinline__ uint32_t p2p_shares(uint32_t nt, uint32_t len, uint32_t grain) {
    if (grain == P2P_WHOLE) return len ? 1u : 0u;
    const uint32_t t = nt < P2P_NT ? nt : P2P_NT;
    uint32_t per = grain / (t > 0 ? t : 1u);
    per = per > grain / 4 ? grain / 4 : per;
    uint32_t s = (len + per - 1) / per;
    const uint32_t most = (1u << 22) / (nt > 0 ? nt : 1u) + 1u;  // bounds the partial sums of a very large leaf
    return s < most ? s : most;
}

// a cell's list sizes with its near-field units and partial sums
__host__ __device__ __forceinline__ uint4 near_sizes(uint32_t m2l, uint32_t p2p, uint32_t count, uint32_t grain) {
    const uint32_t sh = p2p ? p2p_shares(count, p2p, grain) : 0u;
    uint4 v;
    v.x = m2l;
    v.y = p2p;
    v.z = sh * ((count + P2P_NT - 1) / P2P_NT);
    v.w = sh > 1 ? sh * count : 0u;
    return v;
}
// units and partial sums of the leaves for another grain: sizes[c].z, .w and their sums totals[4], [5]
// (both zero before)
void launch_near_sizes(cudaStream_t s, int ncells, const uint32_t* count, uint32_t grain, WalkLists Ls);
// shares of leaf c of nt bodies
__device__ __forceinline__ uint32_t p2p_shares_of(const P2pUnits& U, int c, uint32_t nt) {
    return (U.uoff[c + 1] - U.uoff[c]) / ((nt + P2P_NT - 1) / P2P_NT);
}
void launch_p2p_combine(cudaStream_t s, int ncells, DirList L, CellsView cv, P2pUnits U, double* ax, double* ay,
                        double* az, double* pot);
void launch_p2p_f64(int nsm, cudaStream_t s, DirList L, int ncells, CellsView cv, P2pUnits U, const double* x,
                    const double* y, const double* z, const double* m, double soft2, double* ax, double* ay,
                    double* az, double* pot);

// mixed.cu
void upload_tables_mixed(const OrderTables& t, cudaStream_t s);
__global__ void k_cell_scale(int nc, const double* rho, const double* h, double* ell, float* ellf);
__global__ void k_rho_now(int nc, CellsView cv, const int32_t* parent, const double* x, const double* y,
                          const double* z, double* rho, unsigned* arrive);
__global__ void k_moments_to_mixed(int nc, int p, const zd* full, const double* ell, zf* half);
// top: cells of the top three levels, ntop of them; arrive: nc zeros
void launch_upward_mixed(cudaStream_t s, const int32_t* top, int ntop, int nc, CellsView cv, const int32_t* parent,
                         const double* ell, const double* x, const double* y, const double* z, const double* m, int p,
                         zf* mom, unsigned* arrive);
void l2l_schedule(int p, std::vector<uint32_t>& out);  // the product list k_l2l_mixed works through
void launch_l2l_mixed(bool fp64, unsigned grid, cudaStream_t s, const int32_t* level_cells, int lstart, int lcnt,
                      CellsView cv, const int32_t* parent, const double* ell, int p, const uint32_t* sched, zf* loc);
__global__ void k_l2p_mixed(size_t n, const int32_t* body_leaf, const uint32_t* order, CellsView cv,
                            const double* ell, int p, const zf* loc, const double* x, const double* y,
                            const double* z, const double* nax, const double* nay, const double* naz,
                            const double* npot, double* acc, double* pot);
// pairs: p2p_pairs_floats4 float4 of scratch (the bodies relative to their leaf's centre, with the mass, in pairs)
size_t p2p_pairs_floats4(size_t n, int ncells);
void launch_p2p_mixed(int tile, int nsm, cudaStream_t s, DirList L, int ncells, CellsView cv, P2pUnits U, size_t n,
                      const int32_t* body_leaf, const double* x, const double* y, const double* z, const double* m,
                      float4* pairs, float soft2, double* ax, double* ay, double* az, double* pot);

// integrate.cu
__global__ void k_kick(size_t n3, double* v, const double* a, double h);
__global__ void k_drift(size_t n3, double* x, const double* v, double h);
__global__ void k_kick_rows(size_t n3, double* v, const double* a, const double* dt, double c);
__global__ void k_drift_rows(size_t n3, double* x, const double* v, const double* dt);

// direct.cu
int direct_splits(size_t n, size_t nt);  // splits of the sources
__global__ void k_direct_targets(const double* pos, const double* mass, size_t n, const uint32_t* tgt, size_t nt,
                                 double soft2, double* part);
__global__ void k_direct_reduce(const double* part, int nsplit, size_t nt, double* acc, double* pot, double* fsc);

}  // namespace fmmx
