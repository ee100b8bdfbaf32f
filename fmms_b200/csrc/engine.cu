// Host orchestration of the engine behind the C ABI (include/fmmx.h).
//
// fmmx_build   = Fmm::new / refresh (fmm.rs:26-56): bounding box, Morton keys,
//                key sort, body gather, cells, cell geometry.
// fmmx_evaluate = Fmm::run (fmm.rs:60-142): gather, f pre-pass, P2M/M2M and
//                multipole power, dual walk with the lists, M2L, L2L, P2P,
//                L2P + scatter.
//
// Work runs on two streams; the host waits only where a size must be known
// (the cells of a tree, the lists after the walk) and at the end of a build or evaluation.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "rotw.h"
#include "sort.h"

using namespace fmmx;

namespace {

// Device-memory budget of a context (fmmx_config.device_budget_bytes): every
// engine buffer is charged to it, and the allocation that would take the
// context above it fails with FMMX_OVER_BUDGET, naming the buffer, the bytes
// it needs and the limit (the reference's GPU OverBudget error,
// crates/visual/src/gpufmm.rs:1653-1672, after which its callers fall back).
struct Budget {
    uint64_t limit = 0;  // bytes; 0: no limit
    uint64_t used = 0;
    bool over = false;   // the last refusal, until reported
    uint64_t asked = 0;
};
// the budget of the context whose API call runs on this thread
thread_local Budget* tl_budget = nullptr;

// Every device buffer of a context registers itself while the context is
// constructed, so that the context can drop all of them (a cache: the next
// call reallocates) after a call fails over its budget.
struct DBufBase {
    DBufBase();
    virtual ~DBufBase() = default;
    virtual void release() = 0;
};
thread_local std::vector<DBufBase*>* tl_registry = nullptr;
DBufBase::DBufBase() {
    if (tl_registry) tl_registry->push_back(this);
}

template <class T>
struct DBuf : DBufBase {
    T* p = nullptr;
    size_t cap = 0;
    Budget* bud = nullptr;  // charged for this buffer
    ~DBuf() override { release(); }
    void release() override {
        if (p) {
            cudaFree(p);
            if (bud) bud->used -= cap * sizeof(T);
        }
        p = nullptr;
        cap = 0;
        bud = nullptr;
    }
    void swap(DBuf& o) {
        std::swap(p, o.p);
        std::swap(cap, o.cap);
        std::swap(bud, o.bud);
    }
    // Grows by at least half of the current capacity, so a context that sees
    // slowly growing inputs (a serving loop's forests) reallocates -- and
    // cudaFree synchronises the device -- only a logarithmic number of times;
    // a first allocation carries 1/8 slack, so that sizes which drift up a
    // little between calls (a leapfrog's interaction lists) do not reallocate
    // at the first step (cudaMalloc of a large buffer took over a second at
    // times on a busy device).
    cudaError_t ensure(size_t n) {
        if (n <= cap && p) return cudaSuccess;
        const size_t grown = cap + cap / 2;
        size_t want = std::max<size_t>(std::max<size_t>(n + n / 8, grown), 1);
        Budget* b = tl_budget;
        if (b && b->limit) {
            const uint64_t base = b->used - (p && bud == b ? cap * sizeof(T) : 0);
            if (base + want * sizeof(T) > b->limit) want = std::max<size_t>(n, 1);  // no slack
            if (base + want * sizeof(T) > b->limit) {
                b->over = true;
                b->asked = want * sizeof(T);
                return cudaErrorMemoryAllocation;
            }
        }
        release();
        cudaError_t e = cudaMalloc((void**)&p, want * sizeof(T));
        if (e != cudaSuccess && want > n) {  // no room for the slack: exactly n
            cudaGetLastError();
            want = std::max<size_t>(n, 1);
            e = cudaMalloc((void**)&p, want * sizeof(T));
        }
        if (e != cudaSuccess) {
            p = nullptr;
            cudaGetLastError();
            return e;
        }
        cap = want;
        bud = b;
        if (bud) bud->used += cap * sizeof(T);
        return cudaSuccess;
    }
};

// charges the allocations of one API call to its context's budget
struct BudgetScope {
    Budget* prev;
    explicit BudgetScope(Budget* b) : prev(tl_budget) { tl_budget = b; }
    ~BudgetScope() { tl_budget = prev; }
};

int bits_for(uint64_t v) {
    int b = 0;
    while (b < 64 && (v >> b) != 0) ++b;
    return std::max(b, 1);
}

struct Status {
    fmmx_status code = FMMX_OK;
    std::string msg;
};

// device flags and counters of the build: non-finite input, f pre-pass stack
// overflow, cells per level and leaves, level-list cursors
enum { TF_BAD = 0, TF_STACK = 1, TF_LEVELS = 2, TF_CURSOR = TF_LEVELS + FMMX_NLEVELS + 1,
       TF_SIZE = TF_CURSOR + FMMX_NLEVELS };
// 64-bit words of the walk's state: chunks used, overflow flag, totals (WalkLists), and per level the work
// counters of the level and of its heavy cells and the number of those
enum { WS_USED = 0, WS_OVERFLOW = 1, WS_TOTALS = 2, WS_WORK = WS_TOTALS + 6, WS_HWORK = WS_WORK + FMMX_NLEVELS,
       WS_HEAVY = WS_HWORK + FMMX_NLEVELS, WS_SIZE = WS_HEAVY + FMMX_NLEVELS };

}  // namespace

struct fmmx_ctx {
    Budget budget;  // first: outlives every buffer charged to it
    fmmx_config cfg;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    std::string err;

    OrderTables tab;
    std::vector<double> swap_host;
    DBuf<double> swap_dev;
    DBuf<uint32_t> l2l_sched;  // product list of the mixed L2L

    // sizes of the current tree; a forest of nsys independent systems
    size_t n = 0;
    int nsys = 1;
    DBuf<uint64_t> sys_off;  // nsys + 1 offsets into the inputs
    std::vector<uint64_t> sys_off_host;
    int steps_since_build = 0;
    DBuf<double> c_h;        // box size of every cell
    int nc = 0, nleaves = 0, nlevels = 0;
    int lvl_start[FMMX_NLEVELS + 1] = {0}, lvl_count[FMMX_NLEVELS + 1] = {0};
    bool built = false, evaluated = false, lists_valid = false;
    // leapfrog steps on a reused tree, recorded once per tree as a CUDA graph
    cudaGraphExec_t step_graph = nullptr;
    const void* graph_key[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    double graph_dt = 0.0;
    int graph_scheme = -1;
    void drop_graph() {
        if (step_graph) cudaGraphExecDestroy(step_graph);
        step_graph = nullptr;
    }
    std::vector<DBufBase*> cache;  // every buffer but the constant tables
    int n_m2l = 0, n_p2p = 0;
    unsigned long long pops = 0, p2p_inter = 0;

    // inputs (host API copies) and outputs
    DBuf<double> pos_in, mass_in, acc_out, pot_out;
    const double* build_pos = nullptr;  // device pointers of the last build's inputs
    const double* build_mass = nullptr;

    DBuf<double> box, bbox_part;
    DBuf<int> flags;
    DBuf<uint64_t> keys, keys_sorted;
    DBuf<uint32_t> idx, order;
    DBuf<double> x, y, z, m, nax, nay, naz, npot;
    DBuf<char> cub_tmp;

    DBuf<uint32_t> cell_id0;  // n + 1: cells that start before each slot
    DBuf<unsigned> geo_arrive, up_arrive;  // children of a cell whose geometry (moments) are done
    DBuf<unsigned long long> bbox_enc;
    DBuf<uint32_t> sort_sys, sort_sys_alt;  // a forest's second sort (by system)

    // cells (depth-first pre-order)
    DBuf<uint32_t> c_first, c_count;
    DBuf<int32_t> c_child, c_parent, level_cells, body_leaf;
    DBuf<uint8_t> c_leaf, c_level;
    DBuf<double> c_cx, c_cy, c_cz, c_mass, c_rho;
    DBuf<double4> c_geo;  // (cx, cy, cz, rho) per cell

    // expansions
    DBuf<zd> moments, locals;
    DBuf<double> pows, f, fmin;
    // mixed form: normalised FP32 half-layout expansions and the per-cell length
    DBuf<zf> mom_f, loc_f;
    DBuf<double> ell;
    DBuf<double> rho_now;  // radii about the build's centres on a reused tree
    DBuf<float> ellf;

    // walk: the pool of list chunks, per-cell results, counters (WS_*)
    DBuf<uint32_t> pool_entry, pool_next, down_n, down_head;
    DBuf<uint2> pool_owner;
    DBuf<uint8_t> list_redone;
    DBuf<uint4> list_sizes, list_off;
    DBuf<unsigned long long> walk_state;
    uint32_t cap_pool = 0;   // chunks
    bool pool_short = false; // the memory did not hold the expected capacity
    DBuf<double2> mac_rows;  // per cell for Dehnen's MAC
    DBuf<int32_t> heavy_list;
    DBuf<uint32_t> heavy_ring;
    uint64_t walk_cap0 = 0;  // FMMX_TEST_WALK_CAPACITY (entries; tests of the overflow retry); 0: sized by the tree
    uint64_t p2p_parts_max = 0xffffffffull;  // partial sums (FMMX_TEST_P2P_PARTIALS: a smaller bound, for tests)
    int walk_retries = 0;

    // directed lists: per destination cell c the sources src[off[c] .. off[c+1])
    DBuf<uint32_t> m2l_src, p2p_src;
    DBuf<uint32_t> m2l_off, p2p_off;  // nc + 1 each
    // near-field work units (per leaf: first unit, first partial sum)
    DBuf<uint32_t> p2p_uoff, p2p_soff;
    DBuf<int32_t> p2p_ucell;
    uint32_t p2p_nunits = 0;
    DBuf<double4> p2p_part;
    DBuf<float4> body_pairs;  // mixed near field: bodies relative to their leaf's centre, FP32, with the mass, in pairs
    DBuf<unsigned> p2p_next;

    DBuf<int> work;  // persistent-kernel work counter
    int nsm = 148;
    uint64_t launches = 0, launches_build = 0;

    fmmx_stats st;
    cudaEvent_t ev[16];
    // second stream: the walk and the lists run beside the upward pass, the
    // P2P beside the M2L and L2L; fork/join events order the two
    cudaStream_t stream2 = nullptr;
    cudaEvent_t fork[3] = {nullptr, nullptr, nullptr};
    bool events = false;
};

namespace {

fmmx_status fail(fmmx_ctx* c, fmmx_status s, const std::string& msg) {
    c->err = msg;
    return s;
}

fmmx_status cuda_fail(fmmx_ctx* c, cudaError_t e, const char* where) {
    if (e == cudaErrorMemoryAllocation && c->budget.over) {
        c->budget.over = false;
        char buf[256];
        std::snprintf(buf, sizeof(buf), "%s needs %.1f MiB, device budget %.1f MiB (%.1f MiB in use)", where,
                      c->budget.asked / 1048576.0, c->budget.limit / 1048576.0, c->budget.used / 1048576.0);
        return fail(c, FMMX_OVER_BUDGET, buf);
    }
    std::string m = std::string(where) + ": " + cudaGetErrorString(e);
    cudaGetLastError();
    if (e == cudaErrorMemoryAllocation) return fail(c, FMMX_OUT_OF_MEMORY, m);
    return fail(c, FMMX_DEVICE_ERROR, m);
}

// A call that failed over the budget leaves the context with whatever its
// buffers had grown to: drop them all (the next call reallocates what it
// needs), so that a smaller system fits again.
fmmx_status finish(fmmx_ctx* ctx, fmmx_status st) {
    if (st != FMMX_OVER_BUDGET) return st;
    cudaStreamSynchronize(ctx->stream);
    if (ctx->stream2) cudaStreamSynchronize(ctx->stream2);
    cudaGetLastError();
    ctx->drop_graph();
    for (DBufBase* b : ctx->cache) b->release();
    ctx->built = ctx->evaluated = ctx->lists_valid = false;
    ctx->cap_pool = 0;
    ctx->pool_short = false;
    return st;
}

#define CK(expr, where)                                   \
    do {                                                  \
        cudaError_t e__ = (expr);                         \
        if (e__ != cudaSuccess) return cuda_fail(ctx, e__, where); \
    } while (0)

#define CKL(where) CK(cudaGetLastError(), where)
// kernel launches of the current build/evaluate (reported in fmmx_stats)
#define LCOUNT(k) (ctx->launches += (k))

CellsView view(fmmx_ctx* c) {
    CellsView v;
    v.first = c->c_first.p;
    v.count = c->c_count.p;
    v.child = c->c_child.p;
    v.leaf = c->c_leaf.p;
    v.level = c->c_level.p;
    v.cx = c->c_cx.p;
    v.cy = c->c_cy.p;
    v.cz = c->c_cz.p;
    v.mass = c->c_mass.p;
    v.rho = c->c_rho.p;
    v.geo = c->c_geo.p;
    return v;
}

CellsMut view_mut(fmmx_ctx* c) {
    CellsMut v;
    v.first = c->c_first.p;
    v.count = c->c_count.p;
    v.child = c->c_child.p;
    v.parent = c->c_parent.p;
    v.leaf = c->c_leaf.p;
    v.level = c->c_level.p;
    v.cx = c->c_cx.p;
    v.cy = c->c_cy.p;
    v.cz = c->c_cz.p;
    v.mass = c->c_mass.p;
    v.rho = c->c_rho.p;
    return v;
}

// Swap matrices B_n in block layout, Dehnen 2014 eq 63 (rotation.rs:136-211).
void build_swap(int p, std::vector<double>& sw) {
    auto boff = [](int j) { return j == 0 ? 0 : j * (4 * j * j - 1) / 3; };
    const int bs = (p + 1) * (4 * p * p + 8 * p + 3) / 3;
    sw.assign(bs, 0.0);
    sw[0] = 1.0;
    for (int n = 1; n <= p; ++n) {
        const int nb = 2 * n + 1, off = boff(n), nbp = 2 * n - 1, offp = boff(n - 1);
        auto prev = [&](int row_base, int l) -> double {
            return (std::abs(l) <= n - 1) ? sw[row_base + l + (n - 1)] : 0.0;
        };
        for (int mr = 0; mr < nb; ++mr) {
            const int mm = mr - n;
            for (int lc = 0; lc < nb; ++lc) {
                const int l = lc - n;
                double v;
                if (std::abs(mm) <= n - 1) {
                    const int rp = offp + (mr - 1) * nbp;
                    v = (prev(rp, l - 1) - prev(rp, l + 1)) * 0.5;
                } else if (mm == n) {
                    const int src = offp + (2 * n - 2) * nbp;
                    v = (prev(src, l - 1) + prev(src, l + 1) + 2.0 * prev(src, l)) * 0.5;
                } else {
                    const int src = offp;
                    v = (prev(src, l - 1) + prev(src, l + 1) - 2.0 * prev(src, l)) * 0.5;
                }
                sw[off + mr * nb + lc] = v;
            }
        }
    }
}

}  // namespace

namespace {

void make_tables(OrderTables& t) {
    const int P = FMMX_MAXP;
    std::memset(&t, 0, sizeof(t));
    t.fact[0] = 1.0;
    for (int i = 1; i <= 2 * P; ++i) t.fact[i] = t.fact[i - 1] * (double)i;  // moments.rs:11-17
    for (int p = 0; p <= P; ++p)
        for (int k = 0; k <= p; ++k) t.binom[p][k] = t.fact[p] / (t.fact[k] * t.fact[p - k]);  // :20-27
    for (int m = 1; m <= P; ++m) t.inv2m[m] = 1.0 / (double)(2 * m);
    for (int n = 0; n <= P; ++n)
        for (int m = 0; m < n; ++m) t.invc[n][m] = 1.0 / (double)(n * n - m * m);
}

enum M2lChoice { M2L_NAIVE_BLOCK, M2L_ROT_BLOCK, M2L_ROT_WARP };

// AUTO and ROTATION take the warp rotation kernel where its constant tables
// reach (p <= 16), else the block rotation kernel; NAIVE keeps the reference's
// O(p^4) convolution.
M2lChoice m2l_choice(const fmmx_config& c) {
    if (c.m2l_kernel == FMMX_M2L_NAIVE) return M2L_NAIVE_BLOCK;
    return c.p <= kRotwMaxP ? M2L_ROT_WARP : M2L_ROT_BLOCK;
}


// ---------------------------------------------------------------- build
// nsys > 1 builds a forest: system s is inputs [off[s], off[s+1]) (host
// offsets), each with its own bounding box, keys, key sort and root.
fmmx_status build_impl(fmmx_ctx* ctx, size_t n, const double* d_pos, const double* d_mass, int nsys = 1,
                       const uint64_t* h_off = nullptr) {
    cudaStream_t s = ctx->stream;
    if (n == 0) return fail(ctx, FMMX_INVALID_ARG, "empty input (the reference asserts !parts.is_empty(), tree.rs:95)");
    if (n >= (1ull << 31)) return fail(ctx, FMMX_INVALID_ARG, "n must be below 2^31");
    if (nsys < 1) return fail(ctx, FMMX_INVALID_ARG, "no systems");
    if (nsys > 1) {
        if (h_off[0] != 0 || h_off[nsys] != n) return fail(ctx, FMMX_INVALID_ARG, "offsets must run from 0 to n");
        for (int q = 0; q < nsys; ++q)
            if (h_off[q + 1] <= h_off[q]) return fail(ctx, FMMX_INVALID_ARG, "every system needs at least one body");
    }
    ctx->built = false;
    ctx->evaluated = false;
    ctx->lists_valid = false;
    ctx->drop_graph();  // its kernels address the buffers and sizes of the old tree
    ctx->n = n;
    ctx->nsys = nsys;
    if (ctx->events) CK(cudaEventRecord(ctx->ev[0], s), "event");
    CK(ctx->keys.ensure(n), "alloc keys");
    CK(ctx->keys_sorted.ensure(n), "alloc keys");
    CK(ctx->idx.ensure(n + 1), "alloc idx");
    CK(ctx->order.ensure(n + 1), "alloc order");  // (it may change places with idx)
    for (DBuf<double>* b : {&ctx->x, &ctx->y, &ctx->z, &ctx->m, &ctx->nax, &ctx->nay, &ctx->naz, &ctx->npot})
        CK(b->ensure(n), "alloc bodies");
    CK(ctx->box.ensure(8 * (size_t)nsys), "alloc box");
    ctx->steps_since_build = 0;
    if (nsys > 1) {
        ctx->sys_off_host.assign(h_off, h_off + nsys + 1);
        CK(ctx->sys_off.ensure(nsys + 1), "alloc offsets");
        CK(cudaMemcpyAsync(ctx->sys_off.p, h_off, (nsys + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, s), "copy");
    }
    const unsigned gb = std::min<unsigned>(grid_for(n, 256), 1024u);
    CK(ctx->bbox_part.ensure(gb * 6), "alloc box");
    CK(ctx->flags.ensure(TF_SIZE), "alloc flags");
    CK(cudaMemsetAsync(ctx->flags.p, 0, TF_SIZE * sizeof(int), s), "memset");

    ctx->launches = 0;
    const int nbits = 3 * FMMX_BITS;
    size_t tb;
    LCOUNT(5);  // bbox (2), keys, key sort (onesweep passes counted as 1), gather
    int* bad = ctx->flags.p + TF_BAD;
    uint64_t longest = n;  // the longest system
    if (nsys == 1) {
        k_bbox_partial<<<gb, 256, 0, s>>>(d_pos, n, ctx->bbox_part.p, bad);
        k_bbox_final<<<1, 32, 0, s>>>(ctx->bbox_part.p, (int)gb, ctx->box.p);
        k_keys<<<grid_for(n, 256), 256, 0, s>>>(d_pos, n, ctx->box.p, ctx->keys.p, ctx->idx.p);
    } else {
        longest = 0;
        for (int q = 0; q < nsys; ++q) longest = std::max(longest, h_off[q + 1] - h_off[q]);
        CK(ctx->bbox_enc.ensure(6 * (size_t)nsys), "alloc box");
        CK(cudaMemsetAsync(ctx->bbox_enc.p, 0xff, 6 * (size_t)nsys * sizeof(unsigned long long), s), "memset");
        k_bbox_seg<<<(unsigned)((n + BBOX_CHUNK - 1) / BBOX_CHUNK), 256, 0, s>>>(d_pos, n, ctx->sys_off.p, nsys,
                                                                                 ctx->bbox_enc.p, bad);
        k_bbox_seg_final<<<grid_for(nsys, 128), 128, 0, s>>>(ctx->bbox_enc.p, nsys, ctx->box.p);
        k_keys_seg<<<grid_for(n, 256), 256, 0, s>>>(d_pos, n, ctx->sys_off.p, nsys, ctx->box.p, ctx->keys.p,
                                                    ctx->idx.p);
    }
    CKL("keys");
    // A forest of short systems is sorted a block per system. Where a system
    // is longer than what a block sorts in a few steps, that block would run on
    // alone (48 systems of together 10^6 bodies: 1.8 ms): one sort of all
    // entries by key, then a stable one by system.
    if (nsys > 1 && longest <= 4096) {
        tb = sort_pairs_seg_temp((int)n, nsys, ctx->sys_off.p, nbits);
        CK(ctx->cub_tmp.ensure(tb), "alloc sort");
        CK(sort_pairs_seg(ctx->cub_tmp.p, tb, ctx->keys.p, ctx->keys_sorted.p, ctx->idx.p, ctx->order.p, (int)n, nsys,
                          ctx->sys_off.p, nbits, s),
           "key sort");
    } else {
        tb = sort_pairs_u64_u32_temp((int)n, nbits);
        CK(ctx->cub_tmp.ensure(tb), "alloc sort");
        CK(sort_pairs_u64_u32(ctx->cub_tmp.p, tb, ctx->keys.p, ctx->keys_sorted.p, ctx->idx.p, ctx->order.p, (int)n,
                              nbits, s),
           "key sort");
        if (nsys > 1) {
            // positions before and after the sort in buffers that are free until the cells are made
            CK(ctx->sort_sys.ensure(n), "alloc sort");
            CK(ctx->sort_sys_alt.ensure(n), "alloc sort");
            CK(ctx->cell_id0.ensure(n + 1), "alloc cells");
            CK(ctx->body_leaf.ensure(n), "alloc cells");
            uint32_t* at = reinterpret_cast<uint32_t*>(ctx->body_leaf.p);
            const int sbits = bits_for((uint64_t)(nsys - 1));
            tb = sort_by_system_temp((int)n, sbits);
            CK(ctx->cub_tmp.ensure(tb), "alloc sort");
            k_entry_system<<<grid_for(n, 256), 256, 0, s>>>(ctx->order.p, n, ctx->sys_off.p, nsys, ctx->sort_sys.p,
                                                            ctx->cell_id0.p);
            CK(sort_by_system(ctx->cub_tmp.p, tb, ctx->sort_sys.p, ctx->sort_sys_alt.p, ctx->cell_id0.p, at, (int)n,
                              sbits, s),
               "key sort");
            k_permute_entries<<<grid_for(n, 256), 256, 0, s>>>(at, n, ctx->keys_sorted.p, ctx->order.p, ctx->keys.p,
                                                               ctx->idx.p);
            ctx->keys.swap(ctx->keys_sorted);
            ctx->idx.swap(ctx->order);
            LCOUNT(3);
        }
    }
    k_gather<<<grid_for(n, 256), 256, 0, s>>>(d_pos, d_mass, ctx->order.p, n, ctx->x.p, ctx->y.p, ctx->z.p, ctx->m.p);
    CKL("gather");

    // the cells that start at each slot, and their numbers
    const uint32_t n32 = (uint32_t)n, n_leaf = (uint32_t)ctx->cfg.n_leaf;
    const unsigned gt = (unsigned)((n + 1 + TREE_BLOCK * TREE_PER_THREAD - 1) / (TREE_BLOCK * TREE_PER_THREAD));
    CK(ctx->cell_id0.ensure(n + 1), "alloc cells");
    tb = scan_u32_temp((int)(n + 1));
    CK(ctx->cub_tmp.ensure(tb), "alloc scan");
    k_cell_count<<<gt, TREE_BLOCK, 0, s>>>(ctx->keys_sorted.p, n32, ctx->sys_off.p, nsys, n_leaf, ctx->idx.p,
                                           ctx->flags.p + TF_LEVELS);
    CKL("tree cells");
    CK(scan_u32(ctx->cub_tmp.p, ctx->cub_tmp.cap, ctx->idx.p, ctx->cell_id0.p, (int)(n + 1), s), "tree cells");
    LCOUNT(3);
    int hf[TF_SIZE];
    CK(cudaMemcpyAsync(hf, ctx->flags.p, sizeof(hf), cudaMemcpyDeviceToHost, s), "copy");
    CK(cudaStreamSynchronize(s), "tree build");
    if (hf[TF_BAD]) return fail(ctx, FMMX_INVALID_ARG, "non-finite position");
    uint64_t total = 0;
    int nlev = 0;
    LevelStarts ls;
    for (int L = 0; L < FMMX_NLEVELS; ++L) {
        ctx->lvl_start[L] = ls.start[L] = (int)std::min<uint64_t>(total, 0x7fffffffull);
        ctx->lvl_count[L] = hf[TF_LEVELS + L];
        total += (uint64_t)hf[TF_LEVELS + L];
        if (hf[TF_LEVELS + L] > 0) nlev = L + 1;
    }
    if (total > 0x7fffffffull) return fail(ctx, FMMX_OUT_OF_MEMORY, "node capacity");
    const int nc = (int)total;
    ctx->nc = nc;
    ctx->nlevels = nlev;
    ctx->nleaves = hf[TF_LEVELS + FMMX_NLEVELS];

    for (DBuf<uint32_t>* b : {&ctx->c_first, &ctx->c_count}) CK(b->ensure(nc), "alloc cells");
    CK(ctx->c_child.ensure(8 * (size_t)nc), "alloc cells");
    CK(ctx->c_parent.ensure(nc), "alloc cells");
    CK(ctx->level_cells.ensure(nc), "alloc cells");
    CK(ctx->body_leaf.ensure(n), "alloc cells");
    CK(ctx->c_leaf.ensure(nc), "alloc cells");
    CK(ctx->c_level.ensure(nc), "alloc cells");
    for (DBuf<double>* b : {&ctx->c_cx, &ctx->c_cy, &ctx->c_cz, &ctx->c_mass, &ctx->c_rho, &ctx->c_h})
        CK(b->ensure(nc), "alloc cells");
    CK(ctx->c_geo.ensure(nc), "alloc cells");
    CK(cudaMemsetAsync(ctx->c_child.p, 0xff, 8 * (size_t)nc * sizeof(int32_t), s), "memset");
    k_cell_emit<<<gt, TREE_BLOCK, 0, s>>>(ctx->keys_sorted.p, n32, ctx->sys_off.p, nsys, n_leaf, ctx->cell_id0.p, ls,
                                          ctx->flags.p + TF_CURSOR, ctx->box.p, view_mut(ctx), ctx->level_cells.p,
                                          ctx->body_leaf.p, ctx->c_h.p);
    CKL("tree cells");
    LCOUNT(2);  // cells, geometry
    if (ctx->cfg.center_mode == FMMX_CENTER_COM) {
        CK(ctx->geo_arrive.ensure(nc), "alloc cells");
        CK(cudaMemsetAsync(ctx->geo_arrive.p, 0, (size_t)nc * sizeof(unsigned), s), "memset");
        k_geometry_com<<<grid_for(nc, GEO_WARPS), 32 * GEO_WARPS, 0, s>>>(nc, view_mut(ctx), ctx->x.p, ctx->y.p,
                                                                         ctx->z.p, ctx->m.p, ctx->geo_arrive.p,
                                                                         ctx->c_geo.p);
    } else {
        for (int L = nlev - 1; L >= 0; --L) {
            const int cnt = ctx->lvl_count[L];
            k_geometry_ritter<<<grid_for(cnt, 128), 128, 0, s>>>(ctx->level_cells.p, ctx->lvl_start[L], cnt,
                                                                 view_mut(ctx), ctx->x.p, ctx->y.p, ctx->z.p,
                                                                 ctx->m.p);
        }
        k_pack_geo<<<grid_for(nc, 256), 256, 0, s>>>(nc, view_mut(ctx), ctx->c_geo.p);
        LCOUNT(nlev);
    }
    CKL("geometry");
    if (ctx->events) CK(cudaEventRecord(ctx->ev[1], s), "event");
    CK(cudaStreamSynchronize(s), "build");
    if (ctx->events) {
        float ms = 0;
        cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
        ctx->st.ms_build = ms;
    }
    ctx->build_pos = d_pos;
    ctx->build_mass = d_mass;
    ctx->launches_build = ctx->launches;
    ctx->built = true;
    return FMMX_OK;
}

// ---------------------------------------------------------------- evaluate
// Room for `want` list chunks or, where the memory or the budget does not hold
// them, for as many as it holds, more than `least` (which were too few).
cudaError_t pool_room(fmmx_ctx* ctx, uint64_t least, uint64_t want) {
    for (;;) {
        cudaError_t e = ctx->pool_entry.ensure(32 * (size_t)want);
        if (e == cudaSuccess) e = ctx->pool_next.ensure(want);
        if (e == cudaSuccess) e = ctx->pool_owner.ensure(want);
        if (e == cudaSuccess) ctx->cap_pool = (uint32_t)want;
        const uint64_t next = least + (want - least) / 2;
        if (e != cudaErrorMemoryAllocation || next <= least + least / 32) return e;
        ctx->budget.over = false;
        ctx->pool_entry.release();
        ctx->pool_next.release();
        ctx->pool_owner.release();
        ctx->pool_short = true;
        want = next;
    }
}

// The walk and the interaction lists on stream s, with the lists' sizes read
// back once in between; returns with the lists queued.
fmmx_status walk_impl(fmmx_ctx* ctx, cudaStream_t s) {
    const int nc = ctx->nc;
    // the pool: at least what the current tree is expected to take, more after
    // an overflow, never less than it has had; no walk's work grows with it
    const uint64_t most = 1ull << 28;
    // chunks per cell at the first attempt (uniform systems take about 40); a context with a budget starts small
    const uint64_t per = ctx->budget.limit || nc < 4096 ? 24 : 44;
    const uint64_t spare = 16ull * std::min<uint64_t>((uint64_t)nc, 512);  // what the blocks of a small level reserve
    const uint64_t want = ctx->walk_cap0 > 0 ? std::max<uint64_t>(ctx->walk_cap0 / 32, 1) : per * nc + spare + 256;
    uint64_t cap = std::min(std::max<uint64_t>(ctx->cap_pool, want), most), least = 0;
    if (ctx->pool_short && ctx->cap_pool > 0) cap = ctx->cap_pool;  // (what an earlier walk ended with)
    ctx->walk_retries = 0;
    CK(ctx->walk_state.ensure(WS_SIZE), "alloc walk");
    CK(ctx->down_n.ensure(nc), "alloc walk");
    CK(ctx->down_head.ensure(nc), "alloc walk");
    CK(ctx->list_redone.ensure(nc), "alloc walk");
    CK(ctx->list_sizes.ensure(nc + 1), "alloc walk");
    CK(ctx->list_off.ensure(nc + 1), "alloc walk");
    for (DBuf<uint32_t>* b : {&ctx->m2l_off, &ctx->p2p_off, &ctx->p2p_uoff, &ctx->p2p_soff})
        CK(b->ensure(nc + 1), "alloc lists");
    const size_t tb = scan_u32x4_temp(nc + 1);
    CK(ctx->cub_tmp.ensure(tb), "alloc scan");
    MacParams mp;
    mp.p = ctx->cfg.p;
    mp.eps = ctx->cfg.mac_eps;
    mp.theta = ctx->cfg.theta;
    mp.gap = ctx->cfg.soft_gap * ctx->cfg.softening;
    const CellsView cv = view(ctx);
    const bool dehnen = ctx->cfg.mac_mode == FMMX_MAC_DEHNEN;
    if (dehnen) {
        CK(ctx->mac_rows.ensure((size_t)nc * (mp.p + 2)), "alloc walk");
        k_mac_rows<<<grid_for(nc, 128), 128, 0, s>>>(nc, cv, mp.p, ctx->pows.p, ctx->fmin.p, ctx->mac_rows.p);
        LCOUNT(1);
    }
    WalkHeavy heavy{nullptr, nullptr, nullptr, (uint32_t)ctx->nleaves, 0};
    if (walk_needs_heavy(ctx->lvl_count, ctx->nlevels, ctx->nleaves)) {
        heavy.blocks = walk_heavy_blocks(ctx->nleaves);
        CK(ctx->heavy_list.ensure(nc), "alloc walk");
        for (;;) {  // fewer queues where the memory does not hold them
            const cudaError_t e = ctx->heavy_ring.ensure((size_t)heavy.blocks * (size_t)ctx->nleaves);
            if (e == cudaSuccess) break;
            if (e != cudaErrorMemoryAllocation || heavy.blocks == 1) return cuda_fail(ctx, e, "alloc walk");
            ctx->budget.over = false;
            heavy.blocks = (heavy.blocks + 1) / 2;
        }
        heavy.list = ctx->heavy_list.p;
        heavy.ring = ctx->heavy_ring.p;
    }
    unsigned long long hs[WS_SIZE];
    uint64_t dm = 0, dp = 0;  // directed entries
    uint4 sizes;
    WalkPool pool;
    const WalkLists lists{ctx->down_n.p, ctx->down_head.p, ctx->list_redone.p, ctx->list_sizes.p,
                          ctx->walk_state.p + WS_TOTALS};
    for (int attempt = 0;; ++attempt) {
        CK(pool_room(ctx, least, cap), "alloc walk");
        pool = WalkPool{ctx->pool_entry.p, ctx->pool_next.p, ctx->pool_owner.p, ctx->cap_pool,
                        reinterpret_cast<unsigned*>(ctx->walk_state.p + WS_USED),
                        reinterpret_cast<int*>(ctx->walk_state.p + WS_OVERFLOW)};
        CK(cudaMemsetAsync(ctx->walk_state.p, 0, WS_SIZE * sizeof(unsigned long long), s), "memset");
        CK(cudaMemsetAsync(ctx->list_sizes.p + nc, 0, sizeof(uint4), s), "memset");
        for (int L = 0; L < ctx->nlevels; ++L) {
            unsigned long long* ws = ctx->walk_state.p + L;
            heavy.count = reinterpret_cast<int*>(ws + WS_HEAVY);
            LCOUNT(launch_walk_level(dehnen, s, ctx->level_cells.p + ctx->lvl_start[L], ctx->lvl_count[L], ctx->nleaves,
                                     cv, ctx->c_parent.p, mp, ctx->mac_rows.p, pool, lists, heavy,
                                     reinterpret_cast<int*>(ws + WS_WORK), reinterpret_cast<int*>(ws + WS_HWORK)));
        }
        CKL("walk");
        CK(scan_u32x4(ctx->cub_tmp.p, ctx->cub_tmp.cap, ctx->list_sizes.p, ctx->list_off.p, nc + 1, s), "list offsets");
        LCOUNT(2);
        int stack_overflow = 0;
        CK(cudaMemcpyAsync(hs, ctx->walk_state.p, sizeof(hs), cudaMemcpyDeviceToHost, s), "copy");
        CK(cudaMemcpyAsync(&sizes, ctx->list_off.p + nc, sizeof(sizes), cudaMemcpyDeviceToHost, s), "copy");
        if (dehnen)
            CK(cudaMemcpyAsync(&stack_overflow, ctx->flags.p + TF_STACK, sizeof(int), cudaMemcpyDeviceToHost, s), "copy");
        CK(cudaStreamSynchronize(s), "walk");
        if (stack_overflow) return fail(ctx, FMMX_DEVICE_ERROR, "f pre-pass stack overflow");
        const uint64_t used = (uint32_t)hs[WS_USED];
        if (hs[WS_OVERFLOW]) {
            if (attempt > 48 || ctx->cap_pool >= most) return fail(ctx, FMMX_OUT_OF_MEMORY, "walk capacity");
            least = ctx->cap_pool;
            cap = std::min(std::max<uint64_t>(2 * least, used + used / 4 + 64), most);
        } else {
            dm = hs[WS_TOTALS + 2];
            dp = hs[WS_TOTALS + 3];
            if (dm > 0x7fffffffull || dp > 0x7fffffffull)
                return fail(ctx, FMMX_OUT_OF_MEMORY, "interaction lists above 2^31 entries");
            cudaError_t e = ctx->m2l_src.ensure(std::max<size_t>(dm, 1));
            if (e == cudaSuccess) e = ctx->p2p_src.ensure(std::max<size_t>(dp, 1));
            if (e == cudaSuccess) break;
            // the lists did not fit beside the pool: once more with what this walk used of it
            cap = used + used / 16 + 64;
            if (e != cudaErrorMemoryAllocation || attempt > 48 || cap >= ctx->cap_pool) return cuda_fail(ctx, e, "alloc lists");
            ctx->budget.over = false;
            ctx->pool_entry.release();
            ctx->pool_next.release();
            ctx->pool_owner.release();
            ctx->pool_short = true;
        }
        ctx->walk_retries++;
    }
    ctx->pops = hs[WS_TOTALS];
    ctx->p2p_inter = hs[WS_TOTALS + 1];
    ctx->n_m2l = (int)(dm / 2);
    ctx->n_p2p = (int)((dp + (uint64_t)ctx->nleaves) / 2);  // a leaf's self pair is one entry
    CK(ctx->p2p_next.ensure(1), "alloc lists");
    // the near field's units and partial sums, coarser where they are too many for the 32-bit sums or the
    // memory. W targets times source leaves are at most the body pairs; a share has 64 source leaves or more, a unit 32
    // targets, so W bounds both, and the 32-bit sums are right unless it is 1.4e11 and more: then they are counted anew.
    const uint64_t W = ctx->p2p_inter + ctx->n;
    const bool bounded = W / 32 <= 0xffffffffull && W / 2048 + ctx->n / 32 + dp / 64 + ctx->nleaves <= 0x7fffffffull &&
                         ctx->p2p_parts_max == 0xffffffffull;
    uint64_t units = sizes.z, parts = sizes.w;
    for (uint32_t grain = bounded ? P2P_GRAIN : 0;;) {  // (0: not counted yet)
        cudaError_t e = cudaErrorMemoryAllocation;
        if (grain && units <= 0x7fffffffull && parts <= ctx->p2p_parts_max) {
            e = ctx->p2p_ucell.ensure(std::max<size_t>(units, 1));
            if (e == cudaSuccess) e = ctx->p2p_part.ensure(std::max<size_t>(parts, 1));
        }
        ctx->p2p_nunits = (uint32_t)units;
        if (e == cudaSuccess) break;
        if (grain == P2P_WHOLE || (grain && e != cudaErrorMemoryAllocation)) return cuda_fail(ctx, e, "alloc p2p scratch");
        ctx->budget.over = false;
        grain = !grain ? P2P_GRAIN : grain < (1u << 20) ? 8 * grain : P2P_WHOLE;
        unsigned long long* t = lists.totals + 4;
        CK(cudaMemsetAsync(t, 0, 2 * sizeof(*t), s), "memset");
        launch_near_sizes(s, nc, ctx->c_count.p, grain, lists);
        CKL("list offsets");
        CK(scan_u32x4(ctx->cub_tmp.p, ctx->cub_tmp.cap, ctx->list_sizes.p, ctx->list_off.p, nc + 1, s), "list offsets");
        LCOUNT(2);
        unsigned long long ht[2];
        CK(cudaMemcpyAsync(ht, t, sizeof(ht), cudaMemcpyDeviceToHost, s), "copy");
        CK(cudaStreamSynchronize(s), "list offsets");
        units = ht[0];
        parts = ht[1];
    }
    if (ctx->events) CK(cudaEventRecord(ctx->ev[4], s), "event");
    // chunks reserved but not used may lie beyond the pool: no entry is there
    const uint32_t nchunks = std::min((uint32_t)hs[WS_USED], pool.cap);
    launch_lists_gather(s, nc, nchunks, pool, lists, ctx->list_off.p, ctx->m2l_off.p, ctx->p2p_off.p, ctx->p2p_uoff.p,
                        ctx->p2p_soff.p, ctx->m2l_src.p, ctx->p2p_src.p, ctx->p2p_ucell.p);
    CKL("lists");
    LCOUNT(1);
    return FMMX_OK;
}

// the near field's work units, as walk_impl left them
P2pUnits near_units(fmmx_ctx* ctx) {
    return P2pUnits{ctx->p2p_uoff.p, ctx->p2p_ucell.p, ctx->p2p_soff.p, ctx->p2p_part.p, ctx->p2p_next.p,
                    ctx->p2p_nunits};
}

// Mixed form, near field: FP32 P2P with FP64 sums on the second stream.
fmmx_status near_mixed(fmmx_ctx* ctx, const DirList& lp, bool tm) {
    cudaStream_t s2 = ctx->cfg.overlap ? ctx->stream2 : ctx->stream;
    const int nc = ctx->nc;
    const size_t n = ctx->n;
    const CellsView cv = view(ctx);
    cudaEvent_t* ev = ctx->ev;
    if (tm) CK(cudaEventRecord(ev[12], s2), "event");
    const float soft2 = (float)(ctx->cfg.softening * ctx->cfg.softening);
    CK(cudaMemsetAsync(ctx->p2p_next.p, 0, sizeof(unsigned), s2), "memset");
    launch_p2p_mixed(ctx->cfg.p2p_tile > 0 ? ctx->cfg.p2p_tile : 512, ctx->nsm, s2, lp, nc, cv, near_units(ctx), n,
                     ctx->body_leaf.p, ctx->x.p, ctx->y.p, ctx->z.p, ctx->m.p, ctx->body_pairs.p, soft2, ctx->nax.p,
                     ctx->nay.p, ctx->naz.p, ctx->npot.p);
    CKL("p2p (mixed)");
    if (tm) CK(cudaEventRecord(ev[8], s2), "event");
    CK(cudaEventRecord(ctx->fork[2], s2), "event");
    return FMMX_OK;
}

// Mixed form, far field: FP32 M2L/L2L on normalised expansions, then the L2P,
// which adds the near field.
fmmx_status far_mixed(fmmx_ctx* ctx, const DirList& lm, double* d_acc, double* d_pot, bool tm) {
    cudaStream_t s = ctx->stream;
    const int p = ctx->cfg.p, nc = ctx->nc;
    const size_t n = ctx->n;
    const CellsView cv = view(ctx);
    cudaEvent_t* ev = ctx->ev;
    if (tm) CK(cudaEventRecord(ev[11], s), "event");  // far field from here
    CK(cudaMemsetAsync(ctx->loc_f.p, 0, (size_t)nc * half_stride(p) * sizeof(zf), s), "memset");
    if (ctx->n_m2l > 0) {
        if (p > kRotwMaxP) return fail(ctx, FMMX_INVALID_ARG, "mixed precision supports p <= 16");
        int* work = nullptr;  // preemptible: short blocks instead of persistent ones
        if (!ctx->cfg.preemptible) {
            CK(ctx->work.ensure(1), "alloc");
            CK(cudaMemsetAsync(ctx->work.p, 0, sizeof(int), s), "memset");
            work = ctx->work.p;
        }
        CK(launch_rotw_f32(p, lm, nc, cv, ctx->ellf.p, ctx->mom_f.p, ctx->loc_f.p, work, ctx->nsm, s), "m2l");
    }
    if (tm) CK(cudaEventRecord(ev[6], s), "event");
    LCOUNT((ctx->n_m2l > 0 ? 1 : 0) + (ctx->nlevels - 1) + 4);  // m2l, l2l per level, pairs + p2p + combine, l2p
    for (int L = 1; L < ctx->nlevels; ++L) {
        const int cnt = ctx->lvl_count[L];
        const unsigned g = std::min<unsigned>(cnt, 16u * (unsigned)ctx->nsm);
        launch_l2l_mixed(L <= 3, g, s, ctx->level_cells.p, ctx->lvl_start[L], cnt, cv, ctx->c_parent.p, ctx->ell.p,
                         p, ctx->l2l_sched.p, ctx->loc_f.p);
    }
    CKL("l2l (mixed)");
    if (tm) CK(cudaEventRecord(ev[7], s), "event");
    CK(cudaStreamWaitEvent(s, ctx->fork[2], 0), "join");  // L2P adds the near field
    if (tm) CK(cudaEventRecord(ev[13], s), "event");
    k_l2p_mixed<<<grid_for(n, 128), 128, 0, s>>>(n, ctx->body_leaf.p, ctx->order.p, cv, ctx->ell.p, p,
                                                 ctx->loc_f.p, ctx->x.p, ctx->y.p, ctx->z.p, ctx->nax.p,
                                                 ctx->nay.p, ctx->naz.p, ctx->npot.p, d_acc, d_pot);
    CKL("l2p (mixed)");
    return FMMX_OK;
}

// reuse: keep the interaction lists of the last evaluation of this tree (no
// f pre-pass, walk or list build); moments and locals are recomputed from the
// given positions about the cell centres of the last build. This is the
// tree reuse of the reference's GPU backend (crates/visual/src/gpufmm.rs:9-20).
// capture: the calls are being recorded into a CUDA graph (reuse only): no
// timing events and no read-back at the end.
fmmx_status evaluate_impl(fmmx_ctx* ctx, const double* d_pos, const double* d_mass, double* d_acc, double* d_pot,
                          bool reuse = false, bool capture = false) {
    cudaStream_t s = ctx->stream, s2 = ctx->cfg.overlap ? ctx->stream2 : ctx->stream;
    if (!ctx->built) return fail(ctx, FMMX_NOT_BUILT, "evaluate before build");
    const int p = ctx->cfg.p, dim = dimp(p), nc = ctx->nc;
    const size_t n = ctx->n;
    cudaEvent_t* ev = ctx->ev;
    const bool tm = ctx->events && !capture;
    if (tm) CK(cudaEventRecord(ev[2], s), "event");
    ctx->launches = ctx->launches_build;
    if (d_pos == nullptr) d_pos = ctx->build_pos;
    if (d_mass == nullptr) d_mass = ctx->build_mass;
    k_gather<<<grid_for(n, 256), 256, 0, s>>>(d_pos, d_mass, ctx->order.p, n, ctx->x.p, ctx->y.p, ctx->z.p, ctx->m.p);
    CKL("gather");
    LCOUNT(4 + (ctx->cfg.mac_mode == FMMX_MAC_DEHNEN ? 2 : 0));  // gather, upward (mixed; plain counts its own), f pre-pass
    CK(ctx->moments.ensure((size_t)nc * dim), "alloc expansions");
    CK(ctx->locals.ensure((size_t)nc * dim), "alloc expansions");
    CK(ctx->pows.ensure((size_t)nc * (p + 1)), "alloc expansions");
    CK(ctx->fmin.ensure(nc), "alloc expansions");
    CK(ctx->f.ensure(n), "alloc expansions");
    if (reuse && !ctx->lists_valid) reuse = false;
    const bool dehnen = ctx->cfg.mac_mode == FMMX_MAC_DEHNEN && !reuse;  // f pre-pass and power needed
    const bool mixed = ctx->cfg.precision == FMMX_MIXED;
    const int H = (p + 1) * (p + 2) / 2;
    const CellsView cv = view(ctx);
    if (mixed) {
        CK(ctx->body_pairs.ensure(p2p_pairs_floats4(n, nc)), "alloc expansions");
        CK(ctx->mom_f.ensure((size_t)nc * half_stride(p)), "alloc expansions");
        CK(ctx->loc_f.ensure((size_t)nc * half_stride(p)), "alloc expansions");
        CK(ctx->ell.ensure(nc), "alloc expansions");
        CK(ctx->ellf.ensure(nc), "alloc expansions");
        const double* rho = ctx->c_rho.p;
        // sized on every mixed evaluation, so that a reuse step recorded into
        // a CUDA graph never allocates while capturing
        CK(ctx->rho_now.ensure(nc), "alloc expansions");
        CK(ctx->up_arrive.ensure(nc), "alloc expansions");
        if (reuse) {  // the bodies moved since the build: radii about the same centres
            CK(cudaMemsetAsync(ctx->up_arrive.p, 0, (size_t)nc * sizeof(unsigned), s), "memset");
            k_rho_now<<<grid_for(nc, 4), 128, 0, s>>>(nc, cv, ctx->c_parent.p, ctx->x.p, ctx->y.p, ctx->z.p,
                                                      ctx->rho_now.p, ctx->up_arrive.p);
            LCOUNT(1);
            rho = ctx->rho_now.p;
        }
        k_cell_scale<<<grid_for(nc, 256), 256, 0, s>>>(nc, rho, ctx->c_h.p, ctx->ell.p, ctx->ellf.p);
        LCOUNT(1);
    }
    // the second stream starts once the bodies are gathered: the walk, or for
    // the Dehnen MAC the f pre-pass and fmin (its walk reads the multipole power
    // too and waits for the upward pass)
    CK(cudaEventRecord(ctx->fork[0], s), "event");
    CK(cudaStreamWaitEvent(s2, ctx->fork[0], 0), "fork");
    if (dehnen) {
        CK(ctx->up_arrive.ensure(nc), "alloc expansions");
        CK(cudaMemsetAsync(ctx->flags.p + TF_STACK, 0, sizeof(int), s2), "memset");
        CK(cudaMemsetAsync(ctx->up_arrive.p, 0, (size_t)nc * sizeof(unsigned), s2), "memset");
        launch_fprepass(s2, cv, ctx->x.p, ctx->y.p, ctx->z.p, ctx->m.p, n, ctx->sys_off.p, ctx->nsys,
                        ctx->level_cells.p, ctx->f.p, ctx->flags.p + TF_STACK);
        k_fmin<<<grid_for(nc, 4), 128, 0, s2>>>(nc, cv, ctx->c_parent.p, ctx->f.p, ctx->fmin.p, ctx->up_arrive.p);
        CKL("f pre-pass");
    }
    if (mixed && !dehnen) {
        // normalised FP32 upward pass; FP64 accumulation on the top three levels
        CK(cudaMemsetAsync(ctx->up_arrive.p, 0, (size_t)nc * sizeof(unsigned), s), "memset");
        const int ntop = ctx->nlevels > 3 ? ctx->lvl_start[3] : nc;
        launch_upward_mixed(s, ctx->level_cells.p, ntop, nc, cv, ctx->c_parent.p, ctx->ell.p, ctx->x.p, ctx->y.p,
                            ctx->z.p, ctx->m.p, p, ctx->mom_f.p, ctx->up_arrive.p);
        CKL("upward (mixed)");
    } else {
        const int warps = 2;  // the P2M tables take 35 KB of shared memory per warp at p = 10
        const size_t smem = (size_t)warps * upward_exact_smem_per_warp(p);
        const size_t smem_b = 16 * (size_t)dim * sizeof(zd);
        CK(allow_smem(k_upward_exact, smem), "attr");
        CK(allow_smem(k_m2m_exact_block, smem_b), "attr");
        // the leaves' P2M (a warp per leaf), then level by level the internal
        // cells' M2M (a block per cell, a wide one where a level has few)
        k_upward_exact<<<std::min<unsigned>((nc + warps - 1) / warps, 16u * (unsigned)ctx->nsm), 32 * warps, smem, s>>>(
            ctx->level_cells.p, 0, nc, cv, ctx->x.p, ctx->y.p, ctx->z.p, ctx->m.p, p, ctx->moments.p, ctx->pows.p);
        for (int L = ctx->nlevels - 2; L >= 0; --L) {
            const int cnt = ctx->lvl_count[L];
            k_m2m_exact_block<<<std::min<unsigned>(cnt, 16u * (unsigned)ctx->nsm),
                                cnt <= 8 * ctx->nsm ? M2M_EXACT_WIDE : 256, smem_b, s>>>(
                ctx->level_cells.p, ctx->lvl_start[L], cnt, cv, p, ctx->moments.p, ctx->pows.p);
        }
        LCOUNT(ctx->nlevels);
        CKL("upward");
        if (mixed) {  // the MAC saw exact FP64 moments; the translations use FP32
            k_moments_to_mixed<<<grid_for((size_t)nc * H, 256), 256, 0, s>>>(nc, p, ctx->moments.p, ctx->ell.p,
                                                                            ctx->mom_f.p);
            LCOUNT(1);
            CKL("moments to mixed");
        }
    }
    if (tm) CK(cudaEventRecord(ev[3], s), "event");
    if (dehnen) {
        CK(cudaEventRecord(ctx->fork[0], s), "event");
        CK(cudaStreamWaitEvent(s2, ctx->fork[0], 0), "fork");
    }
    if (tm) CK(cudaEventRecord(ev[10], s2), "event");
    if (!reuse) {
        // a recorded leapfrog step addresses the list buffers and list sizes of
        // the last walk; this walk and its lists may reallocate or resize them
        ctx->drop_graph();
        ctx->lists_valid = false;
        fmmx_status st = walk_impl(ctx, s2);
        if (st != FMMX_OK) return st;
        ctx->lists_valid = true;
    } else if (tm) {
        CK(cudaEventRecord(ev[4], s2), "event");
    }
    if (!reuse) CK(cudaEventRecord(ctx->fork[1], s2), "event");  // the lists are in place
    if (tm) CK(cudaEventRecord(ev[5], s2), "event");

    // (the lists' pointers are taken after the walk, which may reallocate them)
    const DirList lp{ctx->p2p_src.p, ctx->p2p_off.p, ctx->p2p_off.p + 1};
    if (mixed) {
        fmmx_status ms = near_mixed(ctx, lp, tm);
        if (ms != FMMX_OK) return ms;
    } else {
        if (tm) CK(cudaEventRecord(ev[12], s2), "event");
        const double soft2 = ctx->cfg.softening * ctx->cfg.softening;
        CK(cudaMemsetAsync(ctx->p2p_next.p, 0, sizeof(unsigned), s2), "memset");
        launch_p2p_f64(ctx->nsm, s2, lp, nc, cv, near_units(ctx), ctx->x.p, ctx->y.p, ctx->z.p, ctx->m.p, soft2,
                       ctx->nax.p, ctx->nay.p, ctx->naz.p, ctx->npot.p);
        CKL("p2p");
        if (tm) CK(cudaEventRecord(ev[8], s2), "event");
        CK(cudaEventRecord(ctx->fork[2], s2), "event");
    }
    if (!reuse) CK(cudaStreamWaitEvent(s, ctx->fork[1], 0), "join");  // the M2L reads its list
    const DirList lm{ctx->m2l_src.p, ctx->m2l_off.p, ctx->m2l_off.p + 1};
    if (mixed) {
        fmmx_status ms = far_mixed(ctx, lm, d_acc, d_pot, tm);
        if (ms != FMMX_OK) return ms;
    } else {
    if (tm) CK(cudaEventRecord(ev[11], s), "event");  // far field from here
    CK(cudaMemsetAsync(ctx->locals.p, 0, (size_t)nc * dim * sizeof(zd), s), "memset");
    if (ctx->n_m2l > 0) {
        const unsigned g = std::min<unsigned>(nc, 16u * (unsigned)ctx->nsm);
        const M2lChoice ch = m2l_choice(ctx->cfg);
        if (ch == M2L_ROT_WARP) {
            int* work = nullptr;  // preemptible: short blocks instead of persistent ones
            if (!ctx->cfg.preemptible) {
                CK(ctx->work.ensure(1), "alloc");
                CK(cudaMemsetAsync(ctx->work.p, 0, sizeof(int), s), "memset");
                work = ctx->work.p;
            }
            CK(launch_rotw_f64(p, lm, nc, cv, ctx->moments.p, ctx->locals.p, work, ctx->nsm, s), "m2l");
        } else if (ch == M2L_ROT_BLOCK) {
            const size_t smem = m2l_rot_smem_bytes(p);
            CK(allow_smem(k_m2l_rot_f64, smem), "attr");
            k_m2l_rot_f64<<<g, 128, smem, s>>>(lm, nc, cv, p, ctx->moments.p, ctx->locals.p, ctx->swap_dev.p);
        } else {
            const size_t smem = 2 * (size_t)dim * sizeof(zd);
            k_m2l_naive_f64<<<g, 128, smem, s>>>(lm, nc, cv, p, ctx->moments.p, ctx->locals.p);
        }
        CKL("m2l");
    }
    if (tm) CK(cudaEventRecord(ev[6], s), "event");
    LCOUNT((ctx->n_m2l > 0 ? 1 : 0) + (ctx->nlevels - 1) + 3);  // m2l, l2l per level, p2p + combine, l2p
    {
        const size_t smem = 2 * (size_t)dim * sizeof(zd);
        for (int L = 1; L < ctx->nlevels; ++L) {
            const int cnt = ctx->lvl_count[L];
            k_l2l_f64<<<std::min<unsigned>(cnt, 16u * (unsigned)ctx->nsm), 128, smem, s>>>(ctx->level_cells.p, ctx->lvl_start[L],
                                                                            cnt, cv, ctx->c_parent.p, p,
                                                                            ctx->locals.p);
        }
        CKL("l2l");
    }
    if (tm) CK(cudaEventRecord(ev[7], s), "event");
    CK(cudaStreamWaitEvent(s, ctx->fork[2], 0), "join");  // L2P adds the near field
    if (tm) CK(cudaEventRecord(ev[13], s), "event");
    k_l2p_f64<<<grid_for(n, 128), 128, 0, s>>>(n, ctx->body_leaf.p, ctx->order.p, cv, p, ctx->locals.p, ctx->x.p,
                                               ctx->y.p, ctx->z.p, ctx->nax.p, ctx->nay.p, ctx->naz.p, ctx->npot.p,
                                               d_acc, d_pot);
    CKL("l2p");
    }
    if (tm) CK(cudaEventRecord(ev[9], s), "event");
    if (capture) return FMMX_OK;
    CK(cudaStreamSynchronize(s), "evaluate");
    if (tm) {
        auto el = [&](int a, int b) {
            float ms = 0;
            cudaEventElapsedTime(&ms, ev[a], ev[b]);
            return (double)ms;
        };
        // stages on the two streams overlap: each is timed on its own stream
        ctx->st.ms_upward = el(2, 3);
        ctx->st.ms_walk = el(10, 4);
        ctx->st.ms_lists = el(4, 5);
        ctx->st.ms_m2l = el(11, 6);
        ctx->st.ms_l2l = el(6, 7);
        ctx->st.ms_p2p = el(12, 8);
        ctx->st.ms_l2p = el(13, 9);
        ctx->st.ms_evaluate = el(2, 9);
    }
    ctx->evaluated = true;
    return FMMX_OK;
}

}  // namespace

// ================================================================== C ABI
extern "C" {

void fmmx_config_default(fmmx_config* c) {
    if (!c) return;
    c->p = 8;
    c->mac_mode = FMMX_MAC_DEHNEN;
    c->mac_eps = 1e-5;
    c->theta = 0.5;
    c->softening = 0.0;
    c->n_leaf = 16;
    c->center_mode = FMMX_CENTER_COM;
    c->precision = FMMX_PLAIN_FP64;
    c->m2l_kernel = FMMX_M2L_AUTO;
    c->device = 0;
    c->stream = nullptr;
    c->p2p_tile = 0;
    c->preemptible = 0;
    c->soft_gap = 0.0;
    c->use_graphs = 1;
    c->overlap = 1;
    c->device_budget_bytes = 0;
}

const char* fmmx_status_string(fmmx_status s) {
    switch (s) {
        case FMMX_OK: return "ok";
        case FMMX_INVALID_ARG: return "invalid argument";
        case FMMX_OUT_OF_MEMORY: return "out of memory";
        case FMMX_OVER_BUDGET: return "over budget";
        case FMMX_LEAF_OVERFLOW: return "leaf overflow";
        case FMMX_DEVICE_ERROR: return "device error";
        case FMMX_TIMEOUT: return "timeout";
        case FMMX_NOT_BUILT: return "not built";
        case FMMX_NO_DEVICE: return "no CUDA device";
    }
    return "unknown";
}

fmmx_status fmmx_create(const fmmx_config* cfg, fmmx_ctx** out) {
    if (!out) return FMMX_INVALID_ARG;
    *out = nullptr;
    fmmx_config c;
    if (cfg) c = *cfg;
    else fmmx_config_default(&c);
    if (c.p < 1 || c.p > FMMX_MAXP) return FMMX_INVALID_ARG;
    if (c.n_leaf < 0) return FMMX_INVALID_ARG;
    if (c.mac_mode != FMMX_MAC_DEHNEN && c.mac_mode != FMMX_MAC_THETA) return FMMX_INVALID_ARG;
    if (c.mac_mode == FMMX_MAC_THETA && !(c.theta > 0.0)) return FMMX_INVALID_ARG;
    if (!(c.softening >= 0.0)) return FMMX_INVALID_ARG;
    if (c.center_mode != FMMX_CENTER_COM && c.center_mode != FMMX_CENTER_SPHERE) return FMMX_INVALID_ARG;
    if (c.precision != FMMX_PLAIN_FP64 && c.precision != FMMX_MIXED) return FMMX_INVALID_ARG;
    if (c.p2p_tile < 0 || c.p2p_tile > 1024) return FMMX_INVALID_ARG;
    if (c.preemptible != 0 && c.preemptible != 1) return FMMX_INVALID_ARG;
    if (!(c.soft_gap >= 0.0) || !std::isfinite(c.soft_gap)) return FMMX_INVALID_ARG;
    if (c.use_graphs != 0 && c.use_graphs != 1) return FMMX_INVALID_ARG;
    if (c.overlap != 0 && c.overlap != 1) return FMMX_INVALID_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return FMMX_NO_DEVICE;
    }
    if (c.device < 0 || c.device >= ndev) return FMMX_INVALID_ARG;
    if (cudaSetDevice(c.device) != cudaSuccess) return FMMX_DEVICE_ERROR;
    std::vector<DBufBase*> reg;
    tl_registry = &reg;
    fmmx_ctx* ctx = new fmmx_ctx();
    tl_registry = nullptr;
    for (DBufBase* b : reg)
        if (b != &ctx->swap_dev && b != &ctx->l2l_sched) ctx->cache.push_back(b);
    ctx->cfg = c;
    ctx->budget.limit = c.device_budget_bytes;
    BudgetScope bscope(&ctx->budget);
    if (const char* wc = std::getenv("FMMX_TEST_WALK_CAPACITY")) ctx->walk_cap0 = std::strtoull(wc, nullptr, 10);
    if (const char* pm = std::getenv("FMMX_TEST_P2P_PARTIALS"))
        ctx->p2p_parts_max = std::min<uint64_t>(std::strtoull(pm, nullptr, 10), ctx->p2p_parts_max);
    std::memset(&ctx->st, 0, sizeof(ctx->st));
    if (c.stream) {
        ctx->stream = (cudaStream_t)c.stream;
    } else {
        if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) {
            delete ctx;
            return FMMX_DEVICE_ERROR;
        }
        ctx->own_stream = true;
    }
    ctx->events = true;
    for (int i = 0; i < 16; ++i) cudaEventCreate(&ctx->ev[i]);
    {
        int prio = 0;
        cudaStreamGetPriority(ctx->stream, &prio);
        if (cudaStreamCreateWithPriority(&ctx->stream2, cudaStreamNonBlocking, prio) != cudaSuccess) {
            cudaGetLastError();
            fmmx_destroy(ctx);
            return FMMX_DEVICE_ERROR;
        }
        for (int i = 0; i < 3; ++i)
            if (cudaEventCreateWithFlags(&ctx->fork[i], cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                fmmx_destroy(ctx);
                return FMMX_DEVICE_ERROR;
            }
    }
    cudaDeviceGetAttribute(&ctx->nsm, cudaDevAttrMultiProcessorCount, c.device);
    if (ctx->nsm < 1) ctx->nsm = 1;
    g_nsm = ctx->nsm;
    make_tables(ctx->tab);
    upload_tables_exact(ctx->tab, ctx->stream);
    upload_tables_walk(ctx->tab, ctx->stream);
    upload_tables_m2l(ctx->tab, ctx->stream);
    upload_tables_sweeps(ctx->tab, ctx->stream);
    upload_tables_mixed(ctx->tab, ctx->stream);
    build_swap(c.p, ctx->swap_host);
    std::vector<uint32_t> sched;
    l2l_schedule(c.p, sched);
    if (ctx->l2l_sched.ensure(sched.size()) != cudaSuccess ||
        cudaMemcpyAsync(ctx->l2l_sched.p, sched.data(), sched.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                        ctx->stream) != cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        fmmx_destroy(ctx);
        return FMMX_DEVICE_ERROR;
    }
    if (ctx->swap_dev.ensure(ctx->swap_host.size()) != cudaSuccess ||
        cudaMemcpyAsync(ctx->swap_dev.p, ctx->swap_host.data(), ctx->swap_host.size() * sizeof(double),
                        cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        fmmx_destroy(ctx);
        return FMMX_DEVICE_ERROR;
    }
    *out = ctx;
    return FMMX_OK;
}

void fmmx_destroy(fmmx_ctx* ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->cfg.device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    if (ctx->stream2) cudaStreamSynchronize(ctx->stream2);
    ctx->drop_graph();
    for (int i = 0; i < 16; ++i)
        if (ctx->ev[i]) cudaEventDestroy(ctx->ev[i]);
    for (int i = 0; i < 3; ++i)
        if (ctx->fork[i]) cudaEventDestroy(ctx->fork[i]);
    if (ctx->stream2) cudaStreamDestroy(ctx->stream2);
    if (ctx->own_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

const char* fmmx_last_error(const fmmx_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

fmmx_status fmmx_build_device(fmmx_ctx* ctx, size_t n, const double* d_pos, const double* d_mass) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!d_pos || !d_mass) return fail(ctx, FMMX_INVALID_ARG, "null input");
    cudaSetDevice(ctx->cfg.device);
    return finish(ctx, build_impl(ctx, n, d_pos, d_mass));
}

fmmx_status fmmx_build(fmmx_ctx* ctx, size_t n, const double* pos, const double* mass) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!pos || !mass) return fail(ctx, FMMX_INVALID_ARG, "null input");
    if (n == 0) return fail(ctx, FMMX_INVALID_ARG, "empty input (the reference asserts !parts.is_empty(), tree.rs:95)");
    cudaSetDevice(ctx->cfg.device);
    if (ctx->pos_in.ensure(3 * n) != cudaSuccess || ctx->mass_in.ensure(n) != cudaSuccess)
        return fail(ctx, FMMX_OUT_OF_MEMORY, "input buffers");
    cudaStream_t s = ctx->stream;
    if (cudaMemcpyAsync(ctx->pos_in.p, pos, 3 * n * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemcpyAsync(ctx->mass_in.p, mass, n * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess)
        return cuda_fail(ctx, cudaGetLastError(), "copy inputs");
    return finish(ctx, build_impl(ctx, n, ctx->pos_in.p, ctx->mass_in.p));
}

fmmx_status fmmx_build_ensemble_device(fmmx_ctx* ctx, size_t nsys, const uint64_t* offsets, const double* d_pos,
                                       const double* d_mass) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!d_pos || !d_mass || !offsets || nsys == 0 || nsys > (1u << 24)) return fail(ctx, FMMX_INVALID_ARG, "bad input");
    cudaSetDevice(ctx->cfg.device);
    return finish(ctx, build_impl(ctx, (size_t)offsets[nsys], d_pos, d_mass, (int)nsys, offsets));
}

fmmx_status fmmx_build_ensemble(fmmx_ctx* ctx, size_t nsys, const uint64_t* offsets, const double* pos,
                                const double* mass) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!pos || !mass || !offsets || nsys == 0 || nsys > (1u << 24)) return fail(ctx, FMMX_INVALID_ARG, "bad input");
    const size_t n = (size_t)offsets[nsys];
    if (n == 0) return fail(ctx, FMMX_INVALID_ARG, "empty input");
    cudaSetDevice(ctx->cfg.device);
    if (ctx->pos_in.ensure(3 * n) != cudaSuccess || ctx->mass_in.ensure(n) != cudaSuccess)
        return fail(ctx, FMMX_OUT_OF_MEMORY, "input buffers");
    cudaStream_t s = ctx->stream;
    if (cudaMemcpyAsync(ctx->pos_in.p, pos, 3 * n * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemcpyAsync(ctx->mass_in.p, mass, n * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess)
        return cuda_fail(ctx, cudaGetLastError(), "copy inputs");
    return finish(ctx, build_impl(ctx, n, ctx->pos_in.p, ctx->mass_in.p, (int)nsys, offsets));
}

fmmx_status fmmx_evaluate_device(fmmx_ctx* ctx, const double* d_pos, const double* d_mass, double* d_acc,
                                 double* d_pot) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!d_acc) return fail(ctx, FMMX_INVALID_ARG, "null output");
    cudaSetDevice(ctx->cfg.device);
    if (!d_pot) {
        if (ctx->pot_out.ensure(ctx->n) != cudaSuccess) return fail(ctx, FMMX_OUT_OF_MEMORY, "pot buffer");
        d_pot = ctx->pot_out.p;
    }
    return finish(ctx, evaluate_impl(ctx, d_pos, d_mass, d_acc, d_pot));
}

static constexpr int kGraphMinUses = 2;

fmmx_status fmmx_leapfrog_device(fmmx_ctx* ctx, double* d_pos, double* d_vel, const double* d_mass, double* d_acc,
                                 double* d_pot, double dt, int nsteps, int scheme, int refresh_every) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!d_pos || !d_vel || !d_mass || !d_acc || nsteps < 0 || refresh_every < 1 || (scheme != 0 && scheme != 1))
        return fail(ctx, FMMX_INVALID_ARG, "bad leapfrog arguments");
    if (!ctx->built) return fail(ctx, FMMX_NOT_BUILT, "leapfrog needs a built tree (build + evaluate first)");
    cudaSetDevice(ctx->cfg.device);
    cudaStream_t s = ctx->stream;
    const size_t n = ctx->n;
    if (!d_pot) {
        if (ctx->pot_out.ensure(n) != cudaSuccess) return fail(ctx, FMMX_OUT_OF_MEMORY, "pot buffer");
        d_pot = ctx->pot_out.p;
    }
    const unsigned g = grid_for(3 * n, 256);
    const void* key[5] = {d_pos, d_vel, d_mass, d_acc, d_pot};
    for (int step = 0; step < nsteps; ++step) {
        const bool rebuild = (ctx->steps_since_build + 1) >= refresh_every;
        // A step on a reused tree is the same sequence of launches every time:
        // record it once as a CUDA graph and replay it (one launch instead of
        // about 30). Not on the legacy default stream, which cannot be captured.
        // A recording costs more than a launched step, so a tree is recorded
        // only when the refresh cadence will replay it at least
        // kGraphMinUses times (steps_since_build counts the reuse steps done).
        const bool same = ctx->step_graph && ctx->graph_dt == dt && ctx->graph_scheme == scheme &&
                          std::equal(key, key + 5, ctx->graph_key);
        const int reuse_left = refresh_every - 1 - ctx->steps_since_build;
        if (!rebuild && ctx->cfg.use_graphs && s != nullptr && ctx->lists_valid &&
            (same || reuse_left >= kGraphMinUses)) {
            if (!same) {
                ctx->drop_graph();
                const bool ev_saved = ctx->events;
                ctx->events = false;
                cudaGraph_t graph = nullptr;
                fmmx_status st = FMMX_OK;
                if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
                    st = cuda_fail(ctx, cudaGetLastError(), "graph capture");
                if (st == FMMX_OK) {
                    if (scheme == 0) {
                        k_kick<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, 0.5 * dt);
                        k_drift<<<g, 256, 0, s>>>(3 * n, d_pos, d_vel, dt);
                    } else {
                        k_drift<<<g, 256, 0, s>>>(3 * n, d_pos, d_vel, 0.5 * dt);
                    }
                    st = evaluate_impl(ctx, d_pos, d_mass, d_acc, d_pot, true, true);
                    if (scheme == 0) {
                        k_kick<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, 0.5 * dt);
                    } else {
                        k_kick<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, dt);
                        k_drift<<<g, 256, 0, s>>>(3 * n, d_pos, d_vel, 0.5 * dt);
                    }
                    const cudaError_t ec = cudaStreamEndCapture(s, &graph);
                    if (st == FMMX_OK && ec != cudaSuccess) st = cuda_fail(ctx, ec, "graph capture");
                }
                ctx->events = ev_saved;
                if (st == FMMX_OK && cudaGraphInstantiate(&ctx->step_graph, graph, 0) != cudaSuccess) {
                    ctx->step_graph = nullptr;
                    st = cuda_fail(ctx, cudaGetLastError(), "graph instantiate");
                }
                if (graph) cudaGraphDestroy(graph);
                if (st != FMMX_OK) return st;
                std::copy(key, key + 5, ctx->graph_key);
                ctx->graph_dt = dt;
                ctx->graph_scheme = scheme;
            }
            if (cudaGraphLaunch(ctx->step_graph, s) != cudaSuccess) return cuda_fail(ctx, cudaGetLastError(), "graph");
            ctx->steps_since_build++;
            continue;
        }
        if (scheme == 0) {  // kick-drift-kick; d_acc holds the forces at d_pos
            k_kick<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, 0.5 * dt);
            k_drift<<<g, 256, 0, s>>>(3 * n, d_pos, d_vel, dt);
        } else {  // drift-kick-drift (crates/fmm/tests/energy_gate.rs:156-177)
            k_drift<<<g, 256, 0, s>>>(3 * n, d_pos, d_vel, 0.5 * dt);
        }
        if (cudaGetLastError() != cudaSuccess) return fail(ctx, FMMX_DEVICE_ERROR, "leapfrog update");
        fmmx_status st;
        if (rebuild) {
            if (ctx->nsys == 1) {
                st = build_impl(ctx, n, d_pos, d_mass);
            } else {
                std::vector<uint64_t> off(ctx->sys_off_host);
                st = build_impl(ctx, n, d_pos, d_mass, ctx->nsys, off.data());
            }
            if (st != FMMX_OK) return finish(ctx, st);
            ctx->steps_since_build = 0;
            st = evaluate_impl(ctx, d_pos, d_mass, d_acc, d_pot, false);
        } else {
            ctx->steps_since_build++;
            st = evaluate_impl(ctx, d_pos, d_mass, d_acc, d_pot, true);
        }
        if (st != FMMX_OK) return finish(ctx, st);
        if (scheme == 0) {
            k_kick<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, 0.5 * dt);
        } else {
            k_kick<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, dt);
            k_drift<<<g, 256, 0, s>>>(3 * n, d_pos, d_vel, 0.5 * dt);
        }
        if (cudaGetLastError() != cudaSuccess) return fail(ctx, FMMX_DEVICE_ERROR, "leapfrog update");
    }
    if (cudaStreamSynchronize(s) != cudaSuccess) return cuda_fail(ctx, cudaGetLastError(), "leapfrog");
    return FMMX_OK;
}

fmmx_status fmmx_kdk_step_device(fmmx_ctx* ctx, double* d_pos, double* d_vel, const double* d_mass, double* d_acc,
                                 double* d_pot, const double* d_dt, size_t nsys, const uint64_t* offsets,
                                 int rebuild) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!d_pos || !d_vel || !d_mass || !d_acc || !d_dt) return fail(ctx, FMMX_INVALID_ARG, "null pointer");
    if (!offsets && !ctx->built) return fail(ctx, FMMX_NOT_BUILT, "no tree to step on: give offsets");
    if (offsets && (nsys == 0 || nsys > (1u << 24))) return fail(ctx, FMMX_INVALID_ARG, "bad system count");
    cudaSetDevice(ctx->cfg.device);
    cudaStream_t s = ctx->stream;
    const size_t n = offsets ? (size_t)offsets[nsys] : ctx->n;
    if (n == 0) return fail(ctx, FMMX_INVALID_ARG, "empty input");
    if (!d_pot) {
        if (ctx->pot_out.ensure(n) != cudaSuccess) return fail(ctx, FMMX_OUT_OF_MEMORY, "pot buffer");
        d_pot = ctx->pot_out.p;
    }
    const unsigned g = grid_for(3 * n, 256);
    k_kick_rows<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, d_dt, 0.5);
    k_drift_rows<<<g, 256, 0, s>>>(3 * n, d_pos, d_vel, d_dt);
    if (cudaGetLastError() != cudaSuccess) return fail(ctx, FMMX_DEVICE_ERROR, "kick/drift");
    fmmx_status st = FMMX_OK;
    const bool build = offsets != nullptr || rebuild || !ctx->lists_valid;
    if (build) {
        if (offsets) {
            st = nsys == 1 ? build_impl(ctx, n, d_pos, d_mass) : build_impl(ctx, n, d_pos, d_mass, (int)nsys, offsets);
        } else if (ctx->nsys == 1) {
            st = build_impl(ctx, n, d_pos, d_mass);
        } else {
            std::vector<uint64_t> off(ctx->sys_off_host);
            st = build_impl(ctx, n, d_pos, d_mass, ctx->nsys, off.data());
        }
        if (st != FMMX_OK) return finish(ctx, st);
        ctx->steps_since_build = 0;
        st = evaluate_impl(ctx, d_pos, d_mass, d_acc, d_pot, false);
    } else {
        ctx->steps_since_build++;
        st = evaluate_impl(ctx, d_pos, d_mass, d_acc, d_pot, true);
    }
    if (st != FMMX_OK) return finish(ctx, st);
    k_kick_rows<<<g, 256, 0, s>>>(3 * n, d_vel, d_acc, d_dt, 0.5);
    if (cudaGetLastError() != cudaSuccess) return fail(ctx, FMMX_DEVICE_ERROR, "kick");
    return FMMX_OK;
}

fmmx_status fmmx_evaluate(fmmx_ctx* ctx, const double* pos, const double* mass, double* acc, double* pot) {
    if (!ctx) return FMMX_INVALID_ARG;
    BudgetScope bscope(&ctx->budget);
    if (!acc) return fail(ctx, FMMX_INVALID_ARG, "null output");
    if (!ctx->built) return fail(ctx, FMMX_NOT_BUILT, "evaluate before build");
    cudaSetDevice(ctx->cfg.device);
    const size_t n = ctx->n;
    cudaStream_t s = ctx->stream;
    const double* dp = nullptr;
    const double* dm = nullptr;
    if (pos || mass) {
        if (ctx->pos_in.ensure(3 * n) != cudaSuccess || ctx->mass_in.ensure(n) != cudaSuccess)
            return fail(ctx, FMMX_OUT_OF_MEMORY, "input buffers");
        if (pos) {
            if (cudaMemcpyAsync(ctx->pos_in.p, pos, 3 * n * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess)
                return cuda_fail(ctx, cudaGetLastError(), "copy inputs");
            dp = ctx->pos_in.p;
        }
        if (mass) {
            if (cudaMemcpyAsync(ctx->mass_in.p, mass, n * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess)
                return cuda_fail(ctx, cudaGetLastError(), "copy inputs");
            dm = ctx->mass_in.p;
        }
    }
    if (ctx->acc_out.ensure(3 * n) != cudaSuccess || ctx->pot_out.ensure(n) != cudaSuccess)
        return fail(ctx, FMMX_OUT_OF_MEMORY, "output buffers");
    fmmx_status st = evaluate_impl(ctx, dp, dm, ctx->acc_out.p, ctx->pot_out.p);
    if (st != FMMX_OK) return finish(ctx, st);
    if (cudaMemcpyAsync(acc, ctx->acc_out.p, 3 * n * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return cuda_fail(ctx, cudaGetLastError(), "copy outputs");
    if (pot && cudaMemcpyAsync(pot, ctx->pot_out.p, n * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return cuda_fail(ctx, cudaGetLastError(), "copy outputs");
    if (cudaStreamSynchronize(s) != cudaSuccess) return cuda_fail(ctx, cudaGetLastError(), "evaluate");
    return FMMX_OK;
}

fmmx_status fmmx_synchronize(fmmx_ctx* ctx) {
    if (!ctx) return FMMX_INVALID_ARG;
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "synchronize");
    return FMMX_OK;
}

fmmx_status fmmx_get_stats(const fmmx_ctx* ctx, fmmx_stats* out) {
    if (!ctx || !out) return FMMX_INVALID_ARG;
    *out = ctx->st;
    out->n = ctx->n;
    out->n_cells = ctx->nc;
    out->n_leaves = ctx->nleaves;
    out->n_levels = ctx->nlevels;
    out->n_m2l = ctx->n_m2l;
    out->n_p2p = ctx->n_p2p;
    out->walk_pops = ctx->pops;
    out->p2p_interactions = ctx->p2p_inter;
    out->m2l_directed = 2ull * (uint64_t)ctx->n_m2l;
    out->kernel_launches = ctx->launches;
    out->walk_retries = (uint64_t)ctx->walk_retries;
    out->device_bytes = ctx->budget.used;
    return FMMX_OK;
}

fmmx_status fmmx_export_tree(const fmmx_ctx* cctx, uint32_t* order, uint64_t* keys_sorted, uint32_t* cell_info,
                             int32_t* children, double* cen, double* mass, double* rho) {
    fmmx_ctx* ctx = const_cast<fmmx_ctx*>(cctx);
    if (!ctx) return FMMX_INVALID_ARG;
    if (!ctx->built) return fail(ctx, FMMX_NOT_BUILT, "export before build");
    cudaSetDevice(ctx->cfg.device);
    CK(cudaStreamSynchronize(ctx->stream), "sync");
    const size_t n = ctx->n, nc = ctx->nc;
    if (order) CK(cudaMemcpy(order, ctx->order.p, n * 4, cudaMemcpyDeviceToHost), "copy");
    if (keys_sorted) CK(cudaMemcpy(keys_sorted, ctx->keys_sorted.p, n * 8, cudaMemcpyDeviceToHost), "copy");
    if (cell_info) {
        std::vector<uint32_t> f(nc), c(nc);
        std::vector<uint8_t> lv(nc), lf(nc);
        CK(cudaMemcpy(f.data(), ctx->c_first.p, nc * 4, cudaMemcpyDeviceToHost), "copy");
        CK(cudaMemcpy(c.data(), ctx->c_count.p, nc * 4, cudaMemcpyDeviceToHost), "copy");
        CK(cudaMemcpy(lv.data(), ctx->c_level.p, nc, cudaMemcpyDeviceToHost), "copy");
        CK(cudaMemcpy(lf.data(), ctx->c_leaf.p, nc, cudaMemcpyDeviceToHost), "copy");
        for (size_t i = 0; i < nc; ++i) {
            cell_info[4 * i] = f[i];
            cell_info[4 * i + 1] = c[i];
            cell_info[4 * i + 2] = lv[i];
            cell_info[4 * i + 3] = lf[i];
        }
    }
    if (children) CK(cudaMemcpy(children, ctx->c_child.p, nc * 8 * 4, cudaMemcpyDeviceToHost), "copy");
    if (cen) {
        std::vector<double> a(nc), b(nc), c(nc);
        CK(cudaMemcpy(a.data(), ctx->c_cx.p, nc * 8, cudaMemcpyDeviceToHost), "copy");
        CK(cudaMemcpy(b.data(), ctx->c_cy.p, nc * 8, cudaMemcpyDeviceToHost), "copy");
        CK(cudaMemcpy(c.data(), ctx->c_cz.p, nc * 8, cudaMemcpyDeviceToHost), "copy");
        for (size_t i = 0; i < nc; ++i) {
            cen[3 * i] = a[i];
            cen[3 * i + 1] = b[i];
            cen[3 * i + 2] = c[i];
        }
    }
    if (mass) CK(cudaMemcpy(mass, ctx->c_mass.p, nc * 8, cudaMemcpyDeviceToHost), "copy");
    if (rho) CK(cudaMemcpy(rho, ctx->c_rho.p, nc * 8, cudaMemcpyDeviceToHost), "copy");
    return FMMX_OK;
}

fmmx_status fmmx_export_lists(const fmmx_ctx* cctx, uint32_t* m2l, uint32_t* p2p) {
    fmmx_ctx* ctx = const_cast<fmmx_ctx*>(cctx);
    if (!ctx) return FMMX_INVALID_ARG;
    if (!ctx->evaluated) return fail(ctx, FMMX_NOT_BUILT, "export before evaluate");
    cudaSetDevice(ctx->cfg.device);
    CK(cudaStreamSynchronize(ctx->stream), "sync");
    // the mutual pairs (a, b), a before b in depth-first order, from the directed lists
    auto pairs = [&](const DBuf<uint32_t>& off, const DBuf<uint32_t>& src, uint32_t* out) -> fmmx_status {
        std::vector<uint32_t> o(ctx->nc + 1);
        CK(cudaMemcpy(o.data(), off.p, o.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost), "copy");
        std::vector<uint32_t> v(o.back());
        if (!v.empty()) CK(cudaMemcpy(v.data(), src.p, v.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost), "copy");
        for (uint32_t c = 0; c < (uint32_t)ctx->nc; ++c)
            for (uint32_t i = o[c]; i < o[c + 1]; ++i)
                if (v[i] >= c) {
                    *out++ = c;
                    *out++ = v[i];
                }
        return FMMX_OK;
    };
    if (m2l) {
        const fmmx_status st = pairs(ctx->m2l_off, ctx->m2l_src, m2l);
        if (st != FMMX_OK) return st;
    }
    return p2p ? pairs(ctx->p2p_off, ctx->p2p_src, p2p) : FMMX_OK;
}

fmmx_status fmmx_export_expansions(const fmmx_ctx* cctx, double* moments, double* locals, double* pows, double* f,
                                   double* fmin) {
    fmmx_ctx* ctx = const_cast<fmmx_ctx*>(cctx);
    if (!ctx) return FMMX_INVALID_ARG;
    if (!ctx->evaluated) return fail(ctx, FMMX_NOT_BUILT, "export before evaluate");
    cudaSetDevice(ctx->cfg.device);
    CK(cudaStreamSynchronize(ctx->stream), "sync");
    const size_t nc = ctx->nc, dim = dimp(ctx->cfg.p);
    if (moments) CK(cudaMemcpy(moments, ctx->moments.p, nc * dim * 16, cudaMemcpyDeviceToHost), "copy");
    if (locals) CK(cudaMemcpy(locals, ctx->locals.p, nc * dim * 16, cudaMemcpyDeviceToHost), "copy");
    if (pows) CK(cudaMemcpy(pows, ctx->pows.p, nc * (ctx->cfg.p + 1) * 8, cudaMemcpyDeviceToHost), "copy");
    if (f && ctx->cfg.mac_mode == FMMX_MAC_DEHNEN) CK(cudaMemcpy(f, ctx->f.p, ctx->n * 8, cudaMemcpyDeviceToHost), "copy");
    if (fmin && ctx->cfg.mac_mode == FMMX_MAC_DEHNEN)
        CK(cudaMemcpy(fmin, ctx->fmin.p, nc * 8, cudaMemcpyDeviceToHost), "copy");
    return FMMX_OK;
}

fmmx_status fmmx_direct_targets(int device, size_t n, const double* pos, const double* mass, double softening,
                                size_t nt, const uint32_t* targets, double* acc, double* pot, double* fscale) {
    if (!pos || !mass || !targets || !acc || n == 0) return FMMX_INVALID_ARG;
    if (nt == 0) return FMMX_OK;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return FMMX_NO_DEVICE;
    }
    if (device < 0 || device >= ndev) return FMMX_INVALID_ARG;
    for (size_t q = 0; q < nt; ++q)
        if (targets[q] >= n) return FMMX_INVALID_ARG;
    cudaSetDevice(device);
    const int nsplit = direct_splits(n, nt);
    // one allocation for everything (seven cost more than the kernel for 10^5 bodies), in 256-byte steps
    size_t bytes = 0;
    auto room = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    const size_t opos = room(3 * n * 8), omass = room(n * 8), ot = room(nt * 4), opart = room(nsplit * nt * 5 * 8),
                 oacc = room(nt * 3 * 8), opot = room(nt * 8), of = room(nt * 8);
    char* d = nullptr;
    fmmx_status st = FMMX_OK;
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc((void**)&d, bytes) != cudaSuccess) {
        cudaGetLastError();
        st = FMMX_OUT_OF_MEMORY;
    } else {
        double *dpos = (double*)(d + opos), *dmass = (double*)(d + omass), *part = (double*)(d + opart),
               *dacc = (double*)(d + oacc), *dpot = (double*)(d + opot), *df = (double*)(d + of);
        uint32_t* dt = (uint32_t*)(d + ot);
        cudaMemcpyAsync(dpos, pos, 3 * n * 8, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(dmass, mass, n * 8, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(dt, targets, nt * 4, cudaMemcpyHostToDevice, s);
        dim3 g((unsigned)((nt + 127) / 128), (unsigned)nsplit);
        k_direct_targets<<<g, 128, 0, s>>>(dpos, dmass, n, dt, nt, softening * softening, part);
        k_direct_reduce<<<grid_for(nt, 128), 128, 0, s>>>(part, nsplit, nt, dacc, dpot, df);
        cudaMemcpyAsync(acc, dacc, nt * 3 * 8, cudaMemcpyDeviceToHost, s);
        if (pot) cudaMemcpyAsync(pot, dpot, nt * 8, cudaMemcpyDeviceToHost, s);
        if (fscale) cudaMemcpyAsync(fscale, df, nt * 8, cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess) st = FMMX_DEVICE_ERROR;
    }
    if (d) cudaFree(d);
    if (s) cudaStreamDestroy(s);
    return st;
}

}  // extern "C"
