// Solver handle of libvbd_b200: device state, launch sequencing, CUDA-graph replay and the
// solver half of the C ABI declared in include/vbd_b200.h.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "vbd_b200.h"
#include "vbd_internal.h"
#include "vbd_cluster.cuh"
#include "vbd_kernels.cuh"
#include "vbd_tile.cuh"

namespace vbd {

#define CUDA_TRY(call)                                                                                 \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess)                                                                         \
            VBD_FAIL(VBD_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)

#define VBD_TRY(expr)            \
    do {                         \
        int rc_ = (expr);        \
        if (rc_) return rc_;     \
    } while (0)

template <class T> struct DBuf {
    T* p = nullptr;
    size_t n = 0;
    int alloc(size_t count) {
        release();
        if (count == 0) return VBD_OK;
        cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&p), count * sizeof(T));
        if (e != cudaSuccess) {
            p = nullptr;
            VBD_FAIL(VBD_ERR_ALLOC, "cudaMalloc of %zu bytes failed: %s", count * sizeof(T), cudaGetErrorString(e));
        }
        n = count;
        return VBD_OK;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    ~DBuf() { release(); }
};

static inline unsigned nblk(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// getAcceleratorOmega (VBD.cpp:302-311): double literals, float result.
static float omega_of(int order, float rho, float prev) {
    if (order == 1) return 1.0f;
    if (order == 2) return (float)(2.0 / (2.0 - (double)(rho * rho)));
    return (float)(4.0 / (4.0 - (double)(rho * rho * prev)));
}

// getAcceleratorOmega of the GPU wrapper (VBD_GPU_Wrapper.cu:240-244): float arithmetic.
static float omega_of_wrapper(int order, float rho, float prev) {
    if (order == 1) return 1.0f;
    if (order == 2) return 2.0f / (2.0f - (rho * rho));
    return 4.0f / (4.0f - (rho * rho) * prev);
}

using SweepFn = void (*)(SweepParams);

// prefetch 0 / 1 / 2 / 3 = k_sweep's PREFETCH 0 / 1 / 3 and k_sweep_capped's PREFETCH 2 (the deep
// forms for the factored layouts only; the others run PREFETCH 1 for options 2 and 3).  The
// factored layouts' PREFETCH 1 runs as k_sweep_capped (56 registers).  `cache` selects the
// record loads with an L2 policy (factored layouts; k_sweep's CACHE).
template <int L, int LAYOUT, bool CACHE> static SweepFn pick_depth(int prefetch) {
    if (prefetch == 0) return &k_sweep<L, LAYOUT, 0, CACHE>;
    if constexpr (LAYOUT >= 3 && L > 1) {
        if (prefetch == 1) return &k_sweep_capped<L, LAYOUT, 1, CACHE>;
        if (prefetch == 3) return &k_sweep_capped<L, LAYOUT, 2, CACHE>;
        return &k_sweep<L, LAYOUT, 3, CACHE>;
    } else if constexpr (LAYOUT >= 3) {
        return prefetch == 1 ? &k_sweep<L, LAYOUT, 1, CACHE> : &k_sweep<L, LAYOUT, 3, CACHE>;
    } else {
        return &k_sweep<L, LAYOUT, 1, CACHE>;
    }
}

template <int L> static SweepFn pick_sweep(int layout, int prefetch, bool cache) {
    switch (layout) {
        case 0: return pick_depth<L, 0, false>(prefetch);
        case 1: return pick_depth<L, 1, false>(prefetch);
        case 2: return pick_depth<L, 2, false>(prefetch);
        case 3: return cache ? pick_depth<L, 3, true>(prefetch) : pick_depth<L, 3, false>(prefetch);
        default: return cache ? pick_depth<L, 4, true>(prefetch) : pick_depth<L, 4, false>(prefetch);
    }
}

static SweepFn pick_sweep(int lanes, int layout, int prefetch, bool cache) {
    switch (lanes) {
        case 1: return pick_sweep<1>(layout, prefetch, cache);
        case 2: return pick_sweep<2>(layout, prefetch, cache);
        case 4: return pick_sweep<4>(layout, prefetch, cache);
        case 8: return pick_sweep<8>(layout, prefetch, cache);
        case 16: return pick_sweep<16>(layout, prefetch, cache);
        default: return pick_sweep<32>(layout, prefetch, cache);
    }
}

// The cluster walk with whole-mesh copies reads the factored records (layouts 3 and 4) from L2.
template <int L> static void (*pick_cluster(int layout))(PersistParams) {
    return layout == 3 ? &k_cluster_walk<L, 3> : &k_cluster_walk<L, 4>;
}

template <int L> static void (*pick_cluster_adjoint(int layout))(AdjWalkParams) {
    return layout == 3 ? &k_cluster_adjoint<L, 3> : &k_cluster_adjoint<L, 4>;
}

// The tile walk runs lanes / 2 threads per vertex; it reads its own record chunks, packed from the
// factored records of either layout.  With `cluster` the tiles are the CTAs of one cluster.
template <TileKind KIND, int W, bool CL> static void (*pick_tile_form(int lanes, bool stack))(TileParams) {
    if constexpr (W == 8)  // group_tiles stacks for 8 warps only
        if (stack)
            return lanes == 8    ? &k_tile_walk<4, KIND, W, CL, true>
                   : lanes == 16 ? &k_tile_walk<8, KIND, W, CL, true>
                                 : &k_tile_walk<16, KIND, W, CL, true>;
    if (CL && lanes == 32) return &k_tile_walk<16, KIND, 8, true>;
    return lanes == 4 ? &k_tile_walk<2, KIND, W, CL> : lanes == 8 ? &k_tile_walk<4, KIND, W, CL> : &k_tile_walk<8, KIND, W, CL>;
}
template <TileKind KIND> static void (*pick_tile(const TilePlan& p, bool cluster))(TileParams) {  // adjoint: 8 warps
    if (cluster) return pick_tile_form<KIND, 8, true>(p.lanes, p.stack);
    if (KIND == kTileAdjoint || p.warps == 8) return pick_tile_form<KIND, 8, false>(p.lanes, p.stack);
    return pick_tile_form<kTileForward, 16, false>(p.lanes, p.stack);
}
static void (*pick_tile_wrapper(int warps))(TileParams) {
    return warps == 8 ? &k_tile_walk<16, kTileWrapper, 8> : &k_tile_walk<16, kTileWrapper, 16>;
}

// What launch_tile and tile_launch return where the device refuses a cooperative launch of as many CTAs
// (nothing of the walk has run then).
constexpr int kWalkRefused = -1;

// A tile plan on the device.
struct TileSet {
    TilePlan plan;
    bool cluster = false;     // the tiles are the CTAs of one cluster
    bool wrapper = false;     // VBD_GPU_Solver semantics
    int chunk_bytes() const { return wrapper ? kWrapperChunkBytes : kTileChunkBytes; }
    bool dirty = true;        // the chunks must be packed again (new records)
    int layout = 0;           // layout they were packed from
    int sums = 0;             // the solver's lanes the plan's groups are for
    int lanes = 0, warps = 0; // the plan's lanes and warps the device lists are for
    // One allocation: the exchanged words and the start counter, the record chunks, the plan's lists.
    DBuf<float4> mem;
    float4 *words = nullptr, *chunk = nullptr;
    int* lists = nullptr;
    size_t nwords = 0;
    enum { HEAD, GROUPS, WCOL, WSTREAM, TABLE, LID, GHOST, VTILE, VLOCAL, TARGET_OFF, TARGET, COUNT };
    size_t at[COUNT + 1] = {};
    const int* ints(int which) const { return lists + at[which]; }
    // after the words: the count of started CTAs, the limit of a wait
    unsigned long long* arrived() const { return reinterpret_cast<unsigned long long*>(words + nwords - 1); }
    unsigned long long started = 0;  // CTAs of all launches so far
    unsigned tag = 1;                // next unused word tag
    int stride = 1;                  // of the exchanged words
    bool no_room = false;            // its memory could not be had, or its launch was refused
    bool captured = false;           // launches that the caller captured read this set: it is never laid out again
    // cluster form: the forward and adjoint launches checked to fit the device, and the answers
    const void* checked[2] = {nullptr, nullptr};
    bool resident[2] = {false, false};
    void reset(TilePlan&& p) {
        plan = std::move(p);
        dirty = true;
        sums = lanes = 0;
        no_room = false;
        checked[0] = checked[1] = nullptr;
    }
};

template <int L> static void (*pick_persistent(int layout))(PersistParams) {
    switch (layout) {
        case 0: return &k_persistent<L, 0>;
        case 1: return &k_persistent<L, 1>;
        case 2: return &k_persistent<L, 2>;
        case 3: return &k_persistent<L, 3>;
        default: return &k_persistent<L, 4>;
    }
}

// The adjoint reads tet records (layouts 0 and 1) or the forward's streamed incidence records.
template <int L> static void (*pick_adj_sweep(int layout))(AdjParams) {
    switch (layout) {
        case 2: return &k_adj_sweep<L, 2>;
        case 3: return &k_adj_sweep<L, 3>;
        case 4: return &k_adj_sweep<L, 4>;
        default: return &k_adj_sweep<L, 0>;
    }
}

// Key of a captured step / solve graph: everything baked into its kernel parameters.
struct GraphKey {
    int kind;  // 0 = step, 1 = solve, 2 = single sweep
    int iters, accel, init, lanes, layout, prefetch, pdl, block, semantics, l2_prefetch, src;
    int record_cache, persist_mb, energy_every, walk;  // walk: 2 = the adjoint sweeps as a cluster walk
    unsigned long long colour_shape;  // hash of the per-colour lanes (0 = uniform) and the mesh
    float h, dtsr, hg[3], rho;
    bool operator==(const GraphKey& o) const { return std::memcmp(this, &o, sizeof(GraphKey)) == 0; }
};

struct GraphEntry {
    GraphKey key;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    size_t nodes = 0;
};

}  // namespace vbd

struct vbd_solver {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int N = 0, T = 0, C = 0, nfree = 0;
    long long ninc = 0;
    bool ready = false, have_materials = false;
    std::vector<int> cstart;  // colour c = internal ids [cstart[c], cstart[c+1])
    std::vector<int32_t> h_inc_off;  // incidence offsets of the internal vertices (host copy)
    vbd::DBuf<float4> x0, x1, pp, y, v, xprev;
    vbd::DBuf<int> perm, inc_off, inc_tet;
    vbd::DBuf<vbd::TetRec> rec, irec;
    vbd::DBuf<int4> crec;                           // compact (layout 2) or factored (layout 3) records
    vbd::DBuf<float2> cmat;
    vbd::DBuf<int> inc_vertex;                      // internal vertex of each incidence
    vbd::DBuf<float> stage, mat_stage;
    vbd::DBuf<unsigned long long> status;
    std::chrono::steady_clock::time_point looked_at{};  // when finish() last read the record of waits that gave up
    vbd::DBuf<double> partials, scalar;
    // defaults: 64-thread blocks, programmatic dependent launch and graphs; lanes, layout and
    // record prefetch are chosen at init from the mesh (below) until their options are set
    int lanes = 8, layout = 3, use_graph = 1, timing = 0, prefetch = 1, pdl = 1, block = 64;
    // Until VBD_OPT_LANES is set, init picks the lane count: 8 lanes when the free vertices average
    // at least 21 incident tets (the 64^3 cube: 22.9, 5.04 vs 5.49 ms/step with 4), else 4 (the
    // 512-block batch: 19.5, 9.06 vs 10.2 ms/step with 8); then doubled, up to 16, while the
    // largest colour would still fill less than half of the GPU's resident threads (taken as 1024
    // per SM, the sweep's occupancy at 60-64 registers): a small mesh leaves SMs idle, and more lanes per vertex shorten
    // each vertex's dependent chain (the 2,673-vertex beam: 24.7 / 19.3 / 17.2 ms per 30 steps
    // with 4 / 8 / 16 lanes).
    bool lanes_auto = true;
    bool layout_auto = true;  // layout 4 when the ids fit its 21-bit fields, else 3 (at init)
    bool prefetch_auto = true;  // see eff_prefetch
    int max_valence = 0;        // most incident tets of any free vertex
    // VBD_OPT_L2_PREFETCH: each colour sweep prefetches the next colour's streamed records into L2.
    // Off by default: on the 64^3 cube it measured 5.48 against 4.78 ms/step (the extra DRAM
    // traffic competes with the running colour's own stream).
    int l2_prefetch = 0;
    // VBD_OPT_RECORD_CACHE: the factored records are loaded with an L2 policy, evict-first except
    // the first persist_mb megabytes of the record stream (VBD_OPT_RECORD_PERSIST_MB), which are
    // loaded evict-last so that they stay in L2 from one sweep to the next.
    // Until they are set, vbd_solver_init turns the evict-first stream on (64^3 cube: 4.12 against
    // 4.46 ms/step) with a 32 MB evict-last prefix when the vertex state (four float4 arrays) fits
    // in 32 MB (cube: 4.08 ms; 64 MB: 4.21, 96 MB: 4.45 -- the prefix then competes with the state).
    int record_cache = 1, persist_mb = 32;
    bool record_cache_auto = true, persist_auto = true;
    // Per-colour threads per vertex (vbd_solver_set_colour_lanes); empty = `lanes` for every colour.
    // Graph keys carry a hash of the per-colour lanes and of the mesh generation (shape_gen, bumped
    // by every vbd_solver_init), so a shape set again reuses its captured graph.
    std::vector<int> colour_lanes;
    std::vector<int> colour_maxval;     // most incident tets of a free vertex, per colour
    int shape_gen = 0;
    // VBD_OPT_ENERGY_EVERY: vbd_solver_step appends VBDsolver::computeTotalEnergy after iterations
    // 0, k, 2k, ... of every sub-step (VBD.cpp:93-95 with k = 10) to a device-side history, read by
    // vbd_solver_energy_history.  ehist_queued counts the values enqueued since the last reset.
    int energy_every = 0;
    vbd::DBuf<double> ehist;
    vbd::DBuf<int> ecount;
    long long ehist_queued = 0;
    std::vector<long long> colour_inc;  // first incidence of each colour (C + 1 entries)
    // VBD_OPT_SEMANTICS: 0 = VBDsolver (VBD.cpp), 1 = VBD_GPU_Solver (VBD_GPU_Wrapper.cu)
    int semantics = 0;
    float omega_next(int k, float rho, float prev) const {
        return semantics ? vbd::omega_of_wrapper(k, rho, prev) : vbd::omega_of(k, rho, prev);
    }
    // whole step in one launch: 1 = cooperative kernel with grid barriers, 2 = one thread-block
    // cluster holding the positions in shared memory (meshes of up to about 7,000 vertices)
    int persistent = 0;
    int cluster_ctas_opt = 0;                       // CTAs of the cluster walk (0 = from the colour sizes)
    int cluster_resident = 1;  // the cluster's CTAs hold a tile each and its records, not the whole mesh
    // launch shape resolved for the mesh, the kernel and the requested CTAs (the kernel's shared-memory
    // and cluster-size attributes are set per kernel)
    int cl_ctas = 0, cl_block = 0, cl_gen = -1, cl_req = 0;
    const void* cl_fn = nullptr;
    int ca_ctas = 0, ca_gen = -1, ca_req = 0;  // the same for the adjoint walk
    const void* ca_fn = nullptr;
    vbd::DBuf<float> d_adj_omega;
    std::vector<float> adj_omega_cache;
    long long spin_limit = 1LL << 22;               // barrier polls before a persistent launch gives up
    vbd::DBuf<int> d_cstart;
    // Chebyshev schedules on the device, the last used last: a step with another schedule than the step before
    // uploads nothing and waits for nothing
    struct Schedule {
        std::vector<float> w;
        vbd::DBuf<float> d;
        bool captured = false;  // launches that the caller captured read it: it is never overwritten
    };
    std::vector<std::unique_ptr<Schedule>> schedules;
    const float* omega_at = nullptr;  // of the last upload_schedule
    vbd::DBuf<vbd::GridBarrier> barrier;
    int adj_alternate = 0;  // adjoint sweeps alternate the colour order (symmetric Gauss-Seidel pairs)
    // adjoint tape: sub-steps taken since vbd_solver_record, (x, v) every ckpt_every sub-steps
    struct TapeStep {
        float h, dtsr, hg[3], rho;
        int iters, accel;
    };
    std::vector<TapeStep> tape;
    int ckpt_every = 0;
    // 2N each: x then v.  A new recording takes the buffers of the last one (ckpt_pool) before it allocates:
    // cudaMalloc and cudaFree in every pass of a fit cost 1.5 ms, and now and then 100 ms to a second.
    std::vector<std::unique_ptr<vbd::DBuf<float4>>> ckpts, ckpt_pool;
    int add_ckpt() {
        if (ckpt_pool.empty()) {
            ckpts.emplace_back(new vbd::DBuf<float4>());
        } else {
            ckpts.push_back(std::move(ckpt_pool.back()));
            ckpt_pool.pop_back();
        }
        if (ckpts.back()->n != 2 * (size_t)N) VBD_TRY(tape_alloc(*ckpts.back(), 2 * (size_t)N));
        return snapshot(*ckpts.back());
    }
    // Memory of a recording or a backward pass; buffers kept from earlier recordings give way where there is none left.
    template <class T> int tape_alloc(vbd::DBuf<T>& b, size_t n) {
        int rc = b.alloc(n);
        if (rc == VBD_ERR_ALLOC && !ckpt_pool.empty()) {
            vbd::clear_error();
            (void)cudaGetLastError();
            ckpt_pool.clear();
            rc = b.alloc(n);
        }
        return rc;
    }
    vbd::DBuf<float4> adj_lam, adj_lam2, adj_lpp, adj_G, adj_ax, adj_av, adj_seg, adj_save;
    // converged positions of the recorded sub-steps of the newest segment, kept as the forward runs
    // so that the backward starts without recomputing that segment
    vbd::DBuf<float4> live_seg;
    vbd::DBuf<float> adj_gmu, adj_glam;
    int adj_cur = 0;  // which of adj_lam / adj_lam2 holds lam
    // the tile walk (vbd_tile.cuh): its plan for the mesh, whether it runs in place of the captured
    // graph (chosen at init or by the autotuner, off once VBD_OPT_PERSISTENT is set), and its device data
    vbd::TileSet tset;   // one tile per SM, exchanging words through L2
    vbd::TileSet aset;   // tset's tiles as the adjoint sweeps them, where tset has 16 warps or would not stay resident
    vbd::TileSet wset;   // tset's tiles for VBD_GPU_Solver semantics
    // one tile per CTA of a cluster, its plan merged from tset's tiles; and the sets for other lanes or CTA counts
    // that launches captured by the caller read
    std::unique_ptr<vbd::TileSet> cset{new vbd::TileSet()};
    std::vector<std::unique_ptr<vbd::TileSet>> held;
    int tile_walk = 0;
    bool persistent_set = false;
    std::vector<int32_t> batch_mesh;  // mesh of each vertex, set by vbd_solver_init_batch for its init
    int sm_count = 0, smem_optin = 0;
    long long launches = 0;
    std::vector<vbd::GraphEntry> graphs;
    std::vector<double> colour_bytes;               // algorithmic bytes of one sweep of colour c
    std::vector<cudaEvent_t> ev_pool;               // event pairs of timed sweeps
    std::vector<double> ev_bytes;                   // bytes of each timed sweep
    size_t ev_used = 0;                             // pairs in use
    double timed_ms = 0.0, timed_bytes = 0.0;
    long long timed_launches = 0;

    ~vbd_solver() {
        drop_graphs();
        for (cudaEvent_t e : ev_pool) cudaEventDestroy(e);
        if (own_stream && stream) cudaStreamDestroy(stream);
    }

    // Waits for the work queued so far, and reports a wait of a walk or a grid barrier that gave up since the
    // last report: positions, velocities and gradients computed since then are not to be used.  The record is read
    // where kLookAfter has passed since it was last read with the stream drained: a wait that gave up since then
    // lasted longer (1 s in a cluster, 2 s for words, 2^22 loads from L2 at a barrier).  A read takes 10 us, which
    // the reads after each 240 us step would pay twice; a word in pinned host memory that the kernel sets took
    // 0.5 to 10 ms a handle.
    static constexpr std::chrono::milliseconds kLookAfter{250};
    int finish() {
        CUDA_TRY(cudaStreamSynchronize(stream));
        const auto now = std::chrono::steady_clock::now();
        if (now - looked_at < kLookAfter) return VBD_OK;
        unsigned long long t[2] = {0, 0};  // ST_TIMEOUT, ST_WALK_TIMEOUT
        CUDA_TRY(cudaMemcpyAsync(t, status.p + vbd::ST_TIMEOUT, sizeof(t), cudaMemcpyDeviceToHost, stream));
        CUDA_TRY(cudaStreamSynchronize(stream));
        looked_at = now;
        if (!t[0] && !t[1]) return VBD_OK;
        CUDA_TRY(cudaMemsetAsync(status.p + vbd::ST_TIMEOUT, 0, sizeof(t), stream));
        CUDA_TRY(cudaStreamSynchronize(stream));
        if (t[0]) VBD_FAIL(VBD_ERR_TIMEOUT, "a grid barrier of the persistent kernel gave up waiting");
        VBD_FAIL(VBD_ERR_TIMEOUT, "a wait of the cluster or tile walk gave up");
    }

    // Folds the recorded event pairs into the running totals (synchronises on the last one).
    int collect_timing() {
        if (ev_used == 0) return VBD_OK;
        CUDA_TRY(cudaEventSynchronize(ev_pool[2 * ev_used - 1]));
        for (size_t k = 0; k < ev_used; ++k) {
            float ms = 0.f;
            CUDA_TRY(cudaEventElapsedTime(&ms, ev_pool[2 * k], ev_pool[2 * k + 1]));
            timed_ms += ms;
            timed_bytes += ev_bytes[k];
        }
        timed_launches += (long long)ev_used;
        ev_used = 0;
        ev_bytes.clear();
        return VBD_OK;
    }

    int timing_event(cudaEvent_t* out) {
        if (ev_pool.size() < 2 * (ev_used + 1)) {
            if (ev_used >= 4096) VBD_TRY(collect_timing());
            while (ev_pool.size() < 2 * (ev_used + 1)) {
                cudaEvent_t e;
                CUDA_TRY(cudaEventCreate(&e));
                ev_pool.push_back(e);
            }
        }
        out[0] = ev_pool[2 * ev_used];
        out[1] = ev_pool[2 * ev_used + 1];
        return VBD_OK;
    }

    void drop_graphs() {
        for (auto& g : graphs) {
            if (g.exec) cudaGraphExecDestroy(g.exec);
            if (g.graph) cudaGraphDestroy(g.graph);
        }
        graphs.clear();
    }

    // The record prefetch the sweeps run.  Until VBD_OPT_PREFETCH is set: 2 (the lane's first three
    // records before the dependency wait) with the packed records when no lane holds more than
    // three records, else 1.  Measured on the 64^3 cube (8 lanes, at most 3 records a lane): 4.46
    // against 4.55 ms/step; on the 512-mesh batch (4 lanes, up to 6): 7.72 against 7.44 (both
    // before PREFETCH 1 was held to 56 registers, which brought the cube to 4.48 and the batch to
    // 7.10).
    int eff_prefetch() const { return prefetch_for(lanes, max_valence); }
    int prefetch_for(int L, int maxval) const {
        if (!prefetch_auto) return prefetch;
        return (layout == 4 && L > 0 && (maxval + L - 1) / L <= 3) ? 2 : 1;
    }
    int lanes_of(int c) const { return colour_lanes.empty() ? lanes : colour_lanes[c]; }
    int prefetch_of(int c) const {
        return colour_lanes.empty() ? eff_prefetch() : prefetch_for(colour_lanes[c], colour_maxval[c]);
    }
    // First incidence whose record is loaded evict-first (records before it evict-last).
    int persist_end() const {
        if (!record_cache || persist_mb <= 0) return 0;
        const double rec_bytes = layout == 4 ? 40.0 : 48.0;
        const double n = (double)persist_mb * 1048576.0 / rec_bytes;
        return (int)std::min<double>(n, (double)ninc);
    }
    // The launch-shape fields of a graph key.
    void shape_key(vbd::GraphKey& key) const {
        key.lanes = lanes;
        key.layout = layout;
        key.prefetch = eff_prefetch();
        key.pdl = pdl;
        key.block = block;
        key.semantics = semantics;
        key.l2_prefetch = l2_prefetch;
        key.record_cache = record_cache;
        key.persist_mb = persist_mb;
        unsigned long long h = 1469598103934665603ull ^ (unsigned long long)shape_gen;  // FNV-1a
        for (int L : colour_lanes) h = (h ^ (unsigned long long)L) * 1099511628211ull;
        key.colour_shape = colour_lanes.empty() ? (unsigned long long)shape_gen : h;
        key.energy_every = energy_every;
    }

    // Energies a step of `substeps` x `iters` appends to the history.
    long long energies_per_step(int substeps, int iters) const {
        if (energy_every <= 0 || iters <= 0) return 0;
        return (long long)substeps * ((iters + energy_every - 1) / energy_every);
    }

    // Room in the history for `more` values after those already queued; a larger buffer keeps the
    // queued values (captured graphs bake the buffer's address, so they are dropped).
    int reserve_energies(long long more) {
        if (!ecount.p) {
            VBD_TRY(ecount.alloc(1));
            CUDA_TRY(cudaMemsetAsync(ecount.p, 0, sizeof(int), stream));
        }
        const long long need = ehist_queued + more;
        if (need <= (long long)ehist.n) return VBD_OK;
        if (need > 0x7fffffffLL) VBD_FAIL(VBD_ERR_INVALID_ARG, "energy history is full: read it with reset");
        vbd::DBuf<double> bigger;
        VBD_TRY(bigger.alloc((size_t)std::max<long long>(2 * need, 64)));
        if (ehist_queued > 0 && ehist.p)
            CUDA_TRY(cudaMemcpyAsync(bigger.p, ehist.p, sizeof(double) * (size_t)std::min<long long>(ehist_queued, ehist.n),
                                     cudaMemcpyDeviceToDevice, stream));
        CUDA_TRY(cudaStreamSynchronize(stream));
        drop_graphs();
        std::swap(ehist.p, bigger.p);
        std::swap(ehist.n, bigger.n);
        return VBD_OK;
    }

    // VBDsolver::computeTotalEnergy (log-J elastic energy, FP64 sums) of positions X, appended to
    // the history.
    int emit_energy_append(const float4* X) {
        const unsigned blocks = std::max(1u, std::min<unsigned>(vbd::nblk(T, 256), 4096u));
        vbd::k_energy<<<blocks, 256, 0, stream>>>(X, y.p, rec.p, 0, T, 1, 0.0, partials.p);
        VBD_TRY(check_launch());
        vbd::k_sum_partials_append<<<1, 1024, 0, stream>>>(partials.p, (int)blocks, ehist.p, ecount.p, (int)ehist.n);
        return check_launch();
    }

    int check_launch() {
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) VBD_FAIL(VBD_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(e));
        ++launches;
        return VBD_OK;
    }

    int launch_sweep(int c, float4* xr, float4* xn, bool accel, bool keep_pp, float dtsr, float omega) {
        const int vb = cstart[c], ve = cstart[c + 1];
        if (ve <= vb) return VBD_OK;
        vbd::SweepParams p{xr,     xn,     pp.p,     y.p, inc_off.p, inc_tet.p, rec.p,          irec.p,
                           crec.p, cmat.p, status.p, vb,  ve,        dtsr,      omega, accel ? 1 : 0,
                           keep_pp ? 1 : 0, persist_end(), 0};
        if (l2_prefetch && layout >= 2 && crec.p && C > 0) {
            // the colour swept after this one (colour 0 of the next iteration after the last)
            const int cn = (c + 1) % C;
            const long long j0 = colour_inc[cn], j1 = colour_inc[cn + 1];
            const int words = layout == 4 ? 2 : 3;  // int4 per incidence in crec
            p.l2_next = reinterpret_cast<const char*>(crec.p + words * j0);
            p.l2_bytes = (unsigned long long)(j1 - j0) * 16ull * words;
        }
        const int L = lanes_of(c);
        long long threads = (long long)(ve - vb) * L;
        vbd::SweepFn fn = vbd::pick_sweep(L, layout, prefetch_of(c), record_cache != 0);
        int threads_per_block = block;
        if (semantics) threads = (long long)(ve - vb) * vbd::kWrapperLanes;
        cudaEvent_t ev[2] = {nullptr, nullptr};
        if (timing) {
            VBD_TRY(timing_event(ev));
            CUDA_TRY(cudaEventRecord(ev[0], stream));
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(vbd::nblk(threads, threads_per_block));
        cfg.blockDim = dim3(threads_per_block);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = (pdl && !timing) ? 1 : 0;
        if (semantics) {
            const vbd::WrapperParams w{p.x,    p.xnext,  p.pp,    p.y,    p.inc_off, p.inc_tet, p.rec,   p.irec,  p.crec,
                                       p.cmat, p.status, p.v_begin, p.v_end, p.dtsr, p.omega, p.accel, p.keep_pp, nullptr};
            cfg.gridDim = dim3(vbd::nblk(threads, vbd::kWrapperBlock));
            cfg.blockDim = dim3(vbd::kWrapperBlock);
            CUDA_TRY(cudaLaunchKernelEx(&cfg, &vbd::k_sweep_wrapper, w));
        } else {
            CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, p));
        }
        VBD_TRY(check_launch());
        if (timing) {
            CUDA_TRY(cudaEventRecord(ev[1], stream));
            ev_bytes.push_back(colour_bytes[c]);
            ++ev_used;
        }
        return VBD_OK;
    }

    // `iters` sweeps with the Chebyshev schedule; `cur` tracks which buffer holds x.  With
    // record_energy, the log-J energy of the blended positions is appended after iterations 0, k,
    // 2k, ... (k = energy_every), where VBDsolver::step evaluates it (VBD.cpp:93-95).
    int emit_iterations(int iters, float dtsr, bool accel, float rho, int& cur, bool record_energy = false) {
        float omega = 1.0f;
        for (int k = 1; k <= iters; ++k) {
            bool blend = false;
            if (accel) {
                omega = omega_next(k, rho, omega);
                blend = omega > 1.0f;
            }
            float4* xr = cur ? x1.p : x0.p;
            float4* xo = cur ? x0.p : x1.p;
            for (int c = 0; c < C; ++c) VBD_TRY(launch_sweep(c, xr, xo, blend, accel, dtsr, omega));
            if (blend) cur ^= 1;
            if (record_energy && energy_every > 0 && (k - 1) % energy_every == 0)
                VBD_TRY(emit_energy_append(cur ? x1.p : x0.p));
        }
        return VBD_OK;
    }

    int emit_substep(float h, float dtsr, const float* hg, int iters, bool accel, float rho,
                     bool record_energy = false, bool predicted = false) {
        if (!predicted) {
            vbd::k_predict<<<vbd::nblk(N, 256), 256, 0, stream>>>(x0.p, v.p, xprev.p, y.p, nfree, N, h, hg[0], hg[1],
                                                                  hg[2]);
            VBD_TRY(check_launch());
        }
        if (semantics) {
            // main.cpp's GPU loop: solveVBD starts every substep from the inertial target
            // (VBD_GPU_Wrapper.cu:334)
            vbd::k_copy_xyz<<<vbd::nblk(N, 256), 256, 0, stream>>>(y.p, x0.p, x1.p, N);
            VBD_TRY(check_launch());
        }
        int cur = 0;
        VBD_TRY(emit_iterations(iters, dtsr, accel, rho, cur, record_energy));
        if (nfree > 0) {
            vbd::k_finish<<<vbd::nblk(nfree, 256), 256, 0, stream>>>(cur ? x1.p : x0.p, x0.p, xprev.p, v.p, nfree, h,
                                                                     cur, 1);
            VBD_TRY(check_launch());
        }
        return VBD_OK;
    }

    int emit_solve(int iters, float dtsr, bool accel, float rho, int init) {
        if (init == VBD_INIT_FROM_INERTIA) {
            vbd::k_copy_xyz<<<vbd::nblk(N, 256), 256, 0, stream>>>(y.p, x0.p, x1.p, N);
            VBD_TRY(check_launch());
        }
        int cur = 0;
        VBD_TRY(emit_iterations(iters, dtsr, accel, rho, cur));
        if (cur && nfree > 0) {
            vbd::k_finish<<<vbd::nblk(nfree, 256), 256, 0, stream>>>(x1.p, x0.p, nullptr, nullptr, nfree, 1.0f, 1, 0);
            VBD_TRY(check_launch());
        }
        return VBD_OK;
    }

    // Chebyshev weights of `iters` iterations (1 where no blend happens).
    std::vector<float> omega_schedule(int iters, bool accel, float rho) const {
        std::vector<float> w(std::max(iters, 1), 1.0f);
        float omega = 1.0f;
        for (int k = 1; k <= iters; ++k) {
            if (accel) omega = omega_next(k, rho, omega);
            w[k - 1] = accel ? omega : 1.0f;
        }
        return w;
    }

    // The colour starts and the Chebyshev schedule (omega_at) on the device, for the single-launch walks.
    int upload_schedule(int iters, bool accel, float rho) {
        if (d_cstart.n != cstart.size()) {
            VBD_TRY(d_cstart.alloc(cstart.size()));
            CUDA_TRY(cudaMemcpy(d_cstart.p, cstart.data(), sizeof(int) * cstart.size(), cudaMemcpyHostToDevice));
            CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));  // landed before any kernel of `stream`
        }
        std::vector<float> w = omega_schedule(iters, accel, rho);
        const bool captured = persistent && capturing();
        size_t at = schedules.size();
        while (at > 0 && !(schedules[at - 1]->w.size() >= w.size() && std::equal(w.begin(), w.end(), schedules[at - 1]->w.begin())))
            --at;
        std::unique_ptr<Schedule> s;
        if (at > 0) {  // it, or one that starts with it
            s = std::move(schedules[at - 1]);
            schedules.erase(schedules.begin() + (at - 1));
        } else {
            if (captured) VBD_FAIL(VBD_ERR_STATE, "run a step with these iterations and weights before capturing one");
            if (schedules.size() >= 8)
                for (auto i = schedules.begin(); i != schedules.end() && !s; ++i)
                    if (!(*i)->captured) {
                        s = std::move(*i);
                        schedules.erase(i);
                        break;
                    }
            if (!s) s.reset(new Schedule());
            s->w.clear();
            if (s->d.n < w.size()) VBD_TRY(s->d.alloc(std::max<size_t>(w.size(), 64)));
            // pageable memory: read before the call returns
            CUDA_TRY(cudaMemcpyAsync(s->d.p, w.data(), sizeof(float) * w.size(), cudaMemcpyHostToDevice, stream));
            s->w = std::move(w);
        }
        s->captured = s->captured || captured;
        omega_at = s->d.p;
        schedules.push_back(std::move(s));
        return VBD_OK;
    }

    // The parameters of a single-launch walk (the persistent kernel or the cluster walk).
    vbd::PersistParams walk_params(int iters, float dtsr, bool accel, bool predict, bool finish, bool from_inertia,
                                   float h, const float* hg) const {
        vbd::PersistParams w{};
        w.sw = vbd::SweepParams{x0.p, x1.p, pp.p, y.p,  inc_off.p, inc_tet.p, rec.p, irec.p, crec.p, cmat.p,
                                status.p, 0,  0,    dtsr, 1.0f,      0,         accel ? 1 : 0, 0, 0};
        w.xa = x0.p;
        w.xb = x1.p;
        w.v = v.p;
        w.xprev = xprev.p;
        w.cstart = d_cstart.p;
        w.omega = omega_at;
        w.ncol = C;
        w.iters = iters;
        w.nfree = nfree;
        w.n = N;
        w.predict = predict ? 1 : 0;
        w.finish = finish ? 1 : 0;
        w.init_from_inertia = from_inertia ? 1 : 0;
        w.h = h;
        w.hgx = hg ? hg[0] : 0.f;
        w.hgy = hg ? hg[1] : 0.f;
        w.hgz = hg ? hg[2] : 0.f;
        return w;
    }

    int launch_persistent(int iters, float dtsr, bool accel, float rho, bool predict, bool finish, bool from_inertia,
                          float h, const float* hg, int expected_extra = 0) {
        if (!barrier.p) VBD_TRY(barrier.alloc(1));
        VBD_TRY(upload_schedule(iters, accel, rho));
        const int L = lanes < 4 ? 4 : lanes;
        const int threads = 256;
        void (*fn)(vbd::PersistParams) = nullptr;
        switch (L) {
            case 4: fn = vbd::pick_persistent<4>(layout); break;
            case 8: fn = vbd::pick_persistent<8>(layout); break;
            case 16: fn = vbd::pick_persistent<16>(layout); break;
            default: fn = vbd::pick_persistent<32>(layout); break;
        }
        int per_sm = 0, sms = 0;
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0));
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        if (per_sm < 1) VBD_FAIL(VBD_ERR_CUDA, "persistent kernel cannot be resident");
        const int grid = per_sm * sms;
        vbd::PersistParams pp_ = walk_params(iters, dtsr, accel, predict, finish, from_inertia, h, hg);
        pp_.bar = barrier.p;
        pp_.spin_limit = spin_limit;
        pp_.expected_blocks = grid + expected_extra;
        CUDA_TRY(cudaMemsetAsync(barrier.p, 0, sizeof(vbd::GridBarrier), stream));
        void* args[] = {&pp_};
        CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(fn), dim3(grid), dim3(threads), args, 0, stream));
        return check_launch();
    }

    // The cluster walk holds both position buffers of the mesh and the pre-sweep positions in each
    // CTA's shared memory.
    size_t cluster_smem() const { return 3 * sizeof(float4) * (size_t)N; }
    bool cluster_fit(const char** why) const {
        if (semantics) {
            *why = "the cluster walk runs the VBDsolver semantics only";
            return false;
        }
        if (layout != 3 && layout != 4) {
            *why = "the cluster walk reads the factored records (VBD_OPT_LAYOUT 3 or 4)";
            return false;
        }
        int optin = 0;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess ||
            cluster_smem() + 64 > (size_t)optin) {  // + the walk's two mbarriers
            *why = "the mesh's positions (48 B per vertex) do not fit in one CTA's shared memory";
            return false;
        }
        return true;
    }

    // CTAs of the cluster walk: enough 256-thread CTAs for the largest colour in one round, at most
    // 16, fewer when the device cannot hold a cluster of that size.
    // Enough CTAs of the cluster walk to sweep the largest colour at L lanes in one round, at most 16.
    int cluster_auto_ctas(int L) const {
        int maxcol = 1;
        for (int c = 0; c < C; ++c) maxcol = std::max(maxcol, cstart[c + 1] - cstart[c]);
        const long long need = (long long)maxcol * L;
        const int block = vbd::kClusterMaxBlock;
        return (int)std::max<long long>(1, std::min<long long>(16, (need + block - 1) / block));
    }

    // Lets a kernel be launched with all the shared memory of a CTA.  The attribute belongs to the kernel, not to
    // the handle: every handle sets the same value, so that threads cannot undo each other's.
    cudaError_t allow_shared(const void* fn, bool cluster) const {
        cudaFuncAttributes fa;
        cudaError_t e = cudaFuncGetAttributes(&fa, fn);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     smem_optin - (int)fa.sharedSizeBytes);
        if (e == cudaSuccess && cluster) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return e;
    }

    template <class Params>
    int cluster_ctas_for(void (*fn)(Params), int L, size_t smem, int* out) {
        const int block = vbd::kClusterMaxBlock;
        int ctas = cluster_ctas_opt > 0 ? cluster_ctas_opt : cluster_auto_ctas(L);
        CUDA_TRY(allow_shared(reinterpret_cast<const void*>(fn), true));
        for (; ctas >= 1; --ctas) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(ctas);
            cfg.blockDim = dim3(block);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = ctas;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg);
            if (e == cudaSuccess && clusters >= 1) break;
            (void)cudaGetLastError();
            if (cluster_ctas_opt > 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "a cluster of %d CTAs cannot be resident", ctas);
        }
        if (ctas < 1) VBD_FAIL(VBD_ERR_CUDA, "the cluster walk cannot be resident");
        *out = ctas;
        return VBD_OK;
    }

    int resolve_cluster(void (*fn)(vbd::PersistParams), int L) {
        const void* f = reinterpret_cast<const void*>(fn);
        if (cl_gen == shape_gen && cl_fn == f && cl_req == cluster_ctas_opt && cl_ctas > 0) return VBD_OK;
        cl_ctas = 0;
        VBD_TRY(cluster_ctas_for(fn, L, cluster_smem(), &cl_ctas));
        cl_block = vbd::kClusterMaxBlock;
        cl_fn = f;
        cl_gen = shape_gen;
        cl_req = cluster_ctas_opt;
        return VBD_OK;
    }

    // The adjoint walk holds X, both adjoint buffers and the pre-sweep adjoint: 64 B per vertex.
    size_t cluster_adj_smem() const { return 4 * sizeof(float4) * (size_t)N; }
    bool cluster_adj_fit() const {
        int optin = 0;
        return semantics == 0 && (layout == 3 || layout == 4) &&
               cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) == cudaSuccess &&
               cluster_adj_smem() + 64 <= (size_t)optin;
    }
    // With the cluster walk selected, the adjoint sweeps of a sub-step run as one cluster launch
    // too where the mesh fits.
    bool adj_walk() const { return persistent == 2 && !timing && cluster_adj_fit(); }

    // Set-up of the adjoint walk outside any graph capture: the sweep schedule on the device and
    // the cluster shape.
    int upload_adj_schedule(int sweeps, float rho) {
        std::vector<float> w(std::max(sweeps, 1), 1.0f);
        float omega = 1.0f;
        for (int it = 1; it <= sweeps; ++it) {
            if (rho > 0.0f) omega = vbd::omega_of(it, rho, omega);
            w[it - 1] = rho > 0.0f ? omega : 1.0f;
        }
        if (w != adj_omega_cache) {
            if (d_adj_omega.n < w.size()) {
                drop_graphs();  // the cluster adjoint's captured launches hold the address
                VBD_TRY(d_adj_omega.alloc(w.size()));
            }
            CUDA_TRY(cudaMemcpyAsync(d_adj_omega.p, w.data(), sizeof(float) * w.size(), cudaMemcpyHostToDevice, stream));
            CUDA_TRY(cudaStreamSynchronize(stream));
            adj_omega_cache = w;
        }
        return VBD_OK;
    }

    int prepare_adj_walk(int sweeps, float rho, void (**fn_out)(vbd::AdjWalkParams)) {
        VBD_TRY(upload_adj_schedule(sweeps, rho));
        if (d_cstart.n != cstart.size()) {
            VBD_TRY(d_cstart.alloc(cstart.size()));
            CUDA_TRY(cudaMemcpy(d_cstart.p, cstart.data(), sizeof(int) * cstart.size(), cudaMemcpyHostToDevice));
            CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));  // landed before any kernel of `stream`
        }
        const int L = lanes < 4 ? 4 : lanes;
        void (*fn)(vbd::AdjWalkParams) = nullptr;
        switch (L) {
            case 4: fn = vbd::pick_cluster_adjoint<4>(layout); break;
            case 8: fn = vbd::pick_cluster_adjoint<8>(layout); break;
            case 16: fn = vbd::pick_cluster_adjoint<16>(layout); break;
            default: fn = vbd::pick_cluster_adjoint<32>(layout); break;
        }
        const void* f = reinterpret_cast<const void*>(fn);
        if (!(ca_gen == shape_gen && ca_fn == f && ca_req == cluster_ctas_opt && ca_ctas > 0)) {
            ca_ctas = 0;
            VBD_TRY(cluster_ctas_for(fn, L, cluster_adj_smem(), &ca_ctas));
            ca_fn = f;
            ca_gen = shape_gen;
            ca_req = cluster_ctas_opt;
        }
        *fn_out = fn;
        return VBD_OK;
    }

    // The adjoint sweeps of one sub-step as one cluster launch, from the live buffer adj_cur.
    int launch_cluster_adjoint(void (*fn)(vbd::AdjWalkParams), const TapeStep& t, const float4* X, int sweeps,
                               float rho) {
        vbd::AdjWalkParams w{};
        w.a = vbd::AdjParams{X,      nullptr, adj_G.p, y.p,  inc_off.p, inc_tet.p, rec.p,
                             crec.p, cmat.p,  t.dtsr,  0,    0,         nullptr,   nullptr,
                             1.0f,   0,       0};
        w.lam0 = adj_cur ? adj_lam2.p : adj_lam.p;
        w.lam1 = adj_cur ? adj_lam.p : adj_lam2.p;
        w.cstart = d_cstart.p;
        w.omega = d_adj_omega.p;
        w.status = status.p;
        w.ncol = C;
        w.sweeps = sweeps;
        w.n = N;
        w.nfree = nfree;
        w.keep_pp = rho > 0.0f ? 1 : 0;
        w.alternate = adj_alternate;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ca_ctas);
        cfg.blockDim = dim3(vbd::kClusterMaxBlock);
        cfg.dynamicSmemBytes = cluster_adj_smem();
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ca_ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, w));
        return check_launch();
    }

    // A sub-step (predict and finish) or a solve as one cluster launch: the tile walk of one cluster where it
    // fits, its memory can be had and VBD_OPT_CLUSTER_RESIDENT allows it, else vbd::k_cluster_walk.
    int launch_cluster(int iters, float dtsr, bool accel, float rho, bool predict, bool finish, bool from_inertia,
                       float h, const float* hg) {
        const char* why = nullptr;
        if (!cluster_fit(&why)) VBD_FAIL(VBD_ERR_INVALID_ARG, "%s", why);
        VBD_TRY(upload_schedule(iters, accel, rho));
        const int L = lanes < 4 ? 4 : lanes;
        if (cluster_resident && cluster_tiles(L, false) && cluster_ready())
            return launch_tile(*cset, iters, dtsr, accel, rho, from_inertia, h, predict ? hg : nullptr, false);
        void (*fn)(vbd::PersistParams) = nullptr;
        switch (L) {
            case 4: fn = vbd::pick_cluster<4>(layout); break;
            case 8: fn = vbd::pick_cluster<8>(layout); break;
            case 16: fn = vbd::pick_cluster<16>(layout); break;
            default: fn = vbd::pick_cluster<32>(layout); break;
        }
        VBD_TRY(resolve_cluster(fn, L));
        vbd::PersistParams w = walk_params(iters, dtsr, accel, predict, finish, from_inertia, h, hg);
        const size_t smem = cluster_smem();
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cl_ctas);
        cfg.blockDim = dim3(cl_block);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cl_ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, w));
        return check_launch();
    }

    // A sub-step or solve through the single-launch walk VBD_OPT_PERSISTENT selects.
    int launch_walk(int iters, float dtsr, bool accel, float rho, bool predict, bool finish, bool from_inertia,
                    float h, const float* hg) {
        if (persistent == 2) return launch_cluster(iters, dtsr, accel, rho, predict, finish, from_inertia, h, hg);
        return launch_persistent(iters, dtsr, accel, rho, predict, finish, from_inertia, h, hg);
    }

    // Shared memory a tile launch whose CTAs hold `vectors` local vectors leaves for record chunks.
    int tile_chunk_room(const vbd::TileSet& s, int vectors) const {
        const long long fixed = (long long)vbd::tile_smem(s.plan.warps, 0, 0, s.plan, C, vectors, s.cluster) + 10240 +
                                (s.wrapper ? 32 * 13 * 4 * s.plan.warps : 0);
        return (int)std::max<long long>(0, (smem_optin - fixed) / s.chunk_bytes());
    }
    // Chunks per warp ring.
    int tile_ring(const vbd::TileSet& s, int vectors) const {
        return std::min(vbd::kTileMaxRing, tile_chunk_room(s, vectors) / s.plan.warps);
    }
    // Whether every chunk of every tile stays in shared memory (the kernel of 8 warps).
    bool tile_resident(const vbd::TileSet& s, int vectors) const {
        return s.plan.warps == 8 && s.plan.max_chunks <= tile_chunk_room(s, vectors);
    }
    int tile_ring_chunks(const vbd::TileSet& s, int vectors) const {
        return tile_resident(s, vectors) ? s.plan.max_chunks : s.plan.warps * tile_ring(s, vectors);
    }
    // The kernel of 8 warps holds a group's chunks at once, that of 16 warps two chunks at least.
    bool tile_fits(const vbd::TileSet& s, int vectors) const {
        return s.plan.max_local <= (s.wrapper ? vbd::kWrapperMaxLocal : vbd::kTileMaxLocal) &&
               (tile_resident(s, vectors) || tile_ring(s, vectors) >= (s.plan.warps == 8 ? s.plan.max_rounds : 2));
    }
    // Cuts a set's tiles into groups for L lanes and CTAs of `warps` warps (0: chosen here).  A thread's two
    // incidences are those of two lanes, or (stack) of one lane in turn: half the rounds, and twice the
    // threads, shuffles and solves per vertex.  Stacked where the SM's four schedulers then have about one
    // group of a colour each, so that a colour lasts one vertex's chain: microseconds a colour stacked / not,
    // 16x4x4 beam 1.30 / 1.39, 16^3 cube 1.45 / 1.51, 32x8x8 beam 1.37 / 1.48 (its adjoint 1.52 / 1.80); with
    // more groups 8 beams 1.62 / 1.50, 24^3 2.16 / 1.84, and with 16 warps 32^3 3.22 / 2.74, 64^3 10.5 / 8.4.
    void group_tiles(vbd::TileSet& s, int L, int warps, int vectors) {
        const double groups = (double)nfree / std::max(1, C) / std::max(1, s.plan.P) * L / vbd::kTileChunk;
        const int rounds = (max_valence + L - 1) / L;
        const bool few = groups <= vbd::kTileFewGroups && rounds <= vbd::kTileMaxRing / 2;
        const int w = warps ? warps : few ? 8 : 16;
        s.sums = L;
        s.no_room = false;
        s.plan.stack = L <= 16 && rounds > 1 && w == 8;
        vbd::tile_groups(&s.plan, s.plan.stack ? 2 * L : L, w, h_inc_off.data());
        if (s.plan.stack && (s.plan.max_colour_groups > vbd::kTileStackGroups || !tile_resident(s, vectors))) {
            s.plan.stack = false;
            vbd::tile_groups(&s.plan, L, w, h_inc_off.data());
        }
    }
    // Whether the caller is capturing the stream (or that cannot be asked).
    bool capturing() const {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &cs) == cudaSuccess) return cs != cudaStreamCaptureStatusNone;
        (void)cudaGetLastError();
        return true;
    }
    // Whether steps and solves run as tile walks.  Under a caller's stream capture they do not: each
    // launch needs tags of its own, which a replayed launch would repeat.
    bool use_tile() {
        if (!tile_walk || tset.plan.P == 0 || timing || !use_graph || persistent || ninc == 0) return false;
        // VBD_GPU_Solver semantics read the tet records, with lanes of their own
        if (!semantics && (!colour_lanes.empty() || layout < 3 || (lanes != 4 && lanes != 8 && lanes != 16))) return false;
        if (capturing()) return false;
        if (semantics) {
            if (wset.plan.P == 0) {
                vbd::TilePlan q = tset.plan;
                vbd::tile_groups(&q, vbd::kWrapperTileLanes, wrapper_warps(), h_inc_off.data());
                wset.reset(std::move(q));
                wset.wrapper = true;
            }
        } else if (tset.sums != lanes) {
            group_tiles(tset, lanes, 0, 2);
        }
        return tile_fits(walk_tiles(), 1) && tile_room(walk_tiles());
    }
    // Whether the device has (or just gave) the memory of a set's records and words, and has not refused its
    // launch; else the per-colour launches run, or the cluster walk with whole-mesh copies.
    bool tile_room(vbd::TileSet& s) {
        if (!s.no_room && ensure_tile(s) == VBD_ERR_ALLOC) {
            vbd::clear_error();
            (void)cudaGetLastError();
            s.no_room = true;
        }
        return !s.no_room;
    }
    vbd::TileSet& walk_tiles() { return semantics ? wset : tset; }
    // Warps of VBD_GPU_Solver semantics: microseconds per colour with 8 / 16, 16^3 cube (2 groups a colour and
    // tile) 2.56 / 2.91, 24^3 (6) 4.5 / 3.8, 32^3 7.5 / 6.4.
    int wrapper_warps() const {
        const double groups = (double)nfree / std::max(1, C) / std::max(1, tset.plan.P) * vbd::kWrapperTileLanes / vbd::kTileChunk;
        return groups <= vbd::kWrapperFewGroups && max_valence <= vbd::kWrapperTileLanes * (vbd::kTileMaxRing / 2) ? 8 : 16;
    }
    // The adjoint's tiles: its kernel takes more than the 128 registers of 16 warps (with them it spills: 5.2 us
    // a colour against 4.2 with 8 warps for the adjoint of 64 beams).
    vbd::TileSet& adjoint_tiles() {
        if (tset.plan.warps == 8 && (!tset.plan.stack || tile_resident(tset, 3))) return tset;
        if (aset.sums != lanes) {
            vbd::TilePlan q = tset.plan;
            aset.reset(std::move(q));
            group_tiles(aset, lanes, 8, 3);
        }
        return aset;
    }

    // Plans the tiles of one cluster for L lanes and checks that a launch of the walk (or of its adjoint) can
    // be resident.
    bool cluster_tiles(int L, bool adjoint) {
        if (tset.plan.P == 0 || C > vbd::kTileMaxColours || layout < 3) return false;
        const int P = std::min({16, tset.plan.P, cluster_ctas_opt > 0 ? cluster_ctas_opt : std::max(1, nfree / vbd::kClusterTileMin)});
        if ((cset->plan.P != P || cset->sums != L) && !cluster_plan(P, L)) return false;
        vbd::TileSet& s = *cset;
        const int which = adjoint ? 1 : 0, vectors = adjoint ? 3 : 2;
        if (!tile_fits(s, vectors)) return false;
        const void* f = reinterpret_cast<const void*>(adjoint ? vbd::pick_tile<vbd::kTileAdjoint>(s.plan, true)
                                                              : vbd::pick_tile<vbd::kTileForward>(s.plan, true));
        if (s.checked[which] != f) {
            s.checked[which] = f;
            s.resident[which] = false;
            const size_t smem = vbd::tile_smem(8, tile_ring_chunks(s, vectors), s.chunk_bytes(), s.plan, C, vectors, true);
            if (allow_shared(f, true) == cudaSuccess) {
                cudaLaunchConfig_t cfg = {};
                cudaLaunchAttribute attr[1];
                cluster_config(&cfg, attr, P, 256, smem);
                int clusters = 0;
                s.resident[which] = cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) == cudaSuccess && clusters >= 1;
            }
            (void)cudaGetLastError();
        }
        return s.resident[which];
    }
    // Makes cset the set of P tiles and L lanes.  One that a caller's captured launches read is put by, and is
    // taken back when it is wanted again.
    bool cluster_plan(int P, int L) {
        if (capturing()) return false;
        if (cset->captured) {
            held.push_back(std::move(cset));
            cset.reset(new vbd::TileSet());
        }
        for (auto& h : held)
            if (h->plan.P == P && h->sums == L) {
                drop_graphs();  // the adjoint's captured launches hold the addresses of the set that goes
                std::swap(cset, h);
                std::swap(h, held.back());
                held.pop_back();
                return true;
            }
        vbd::TilePlan q;
        vbd::tile_merge(tset.plan, P, cstart, &q);
        cset->reset(std::move(q));
        cset->cluster = true;
        group_tiles(*cset, L, 8, 3);
        return true;
    }
    // Whether cset is on the device, packed from the present records.  While the caller captures the stream
    // nothing can be packed (a pack that is only captured packs nothing now, and memory cannot be had): a
    // set that needs it is not used, and one that is used keeps its place and is packed with every new material.
    bool cluster_ready() {
        vbd::TileSet& s = *cset;
        if (!capturing()) return tile_room(s);
        if (s.dirty || s.layout != layout || s.lanes != s.plan.lanes || s.warps != s.plan.warps) return false;
        return s.captured = true;
    }
    // Readies the cluster's tiles when an option or a mesh calls for them, so that the next step may be one that
    // the caller captures.
    int prepare_cluster() {
        const char* why = nullptr;
        if (!ready || persistent != 2 || !cluster_resident || capturing() || !cluster_fit(&why)) return VBD_OK;
        if (cluster_tiles(lanes < 4 ? 4 : lanes, false) && tile_room(*cset)) CUDA_TRY(cudaStreamSynchronize(stream));
        return VBD_OK;
    }
    // The automatic CTA count of VBD_OPT_CLUSTER_CTAS.
    int cluster_auto(int L) { return cluster_resident && cluster_tiles(L, false) ? cset->plan.P : cluster_auto_ctas(L); }
    void cluster_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int ctas, int threads, size_t smem) const {
        cfg->gridDim = dim3(ctas);
        cfg->blockDim = dim3(threads);
        cfg->dynamicSmemBytes = smem;
        cfg->stream = stream;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg->attrs = attr;
        cfg->numAttrs = 1;
    }

    // Gives the memory of a set that no step will use back; it is made again if one does.
    void give_back(vbd::TileSet& s) {
        if (!s.mem.p || capturing()) return;
        s.mem.release();
        s.lanes = s.warps = 0;
        s.dirty = true;
    }

    // After how many nanoseconds a wait of the set's walks gives up.
    int set_wait_limit(vbd::TileSet& s, unsigned long long ns) {
        CUDA_TRY(cudaMemcpyAsync(s.arrived() + 1, &ns, sizeof(ns), cudaMemcpyHostToDevice, stream));
        CUDA_TRY(cudaStreamSynchronize(stream));
        return VBD_OK;
    }

    // The plan's lists and the record chunks on the device, made when first needed for the current lanes, layout
    // and materials.
    int ensure_tile(vbd::TileSet& s) {
        vbd::TilePlan& q = s.plan;
        if (s.lanes != q.lanes || s.warps != q.warps) {
            s.lanes = 0;  // until the new lists are there
            const struct {
                const void* p;
                size_t ints;
            } lists[vbd::TileSet::COUNT] = {
                {q.head.data(), q.head.size() * sizeof(vbd::TileHead) / 4},
                {q.groups.data(), q.groups.size() * sizeof(vbd::TileGroup) / 4},
                {q.wcol.data(), q.wcol.size()},
                {q.wstream.data(), q.wstream.size()},
                {q.chunk.data(), q.chunk.size()},
                {q.lid.data(), q.lid.size()},
                {q.ghost.data(), q.ghost.size()},
                {q.vtile.data(), q.vtile.size()},
                {q.vlocal.data(), q.vlocal.size()},
                {q.target_off.data(), q.target_off.size()},
                {q.target.data(), q.target.size()},
            };
            for (int k = 0; k < vbd::TileSet::COUNT; ++k) s.at[k + 1] = s.at[k] + (lists[k].ints + 3) / 4 * 4;
            std::vector<int> all(s.at[vbd::TileSet::COUNT]);
            for (int k = 0; k < vbd::TileSet::COUNT; ++k)
                if (lists[k].ints) std::memcpy(all.data() + s.at[k], lists[k].p, 4 * lists[k].ints);
            s.stride = nfree <= (long long)vbd::kTileSpreadWords * q.P ? 8 : 1;
            s.nwords = s.cluster ? 0 : 4 * (size_t)s.stride * N + 1;
            const size_t nchunk = q.chunk.size() / 3 * (size_t)(s.chunk_bytes() / 16);
            const size_t need = s.nwords + nchunk + all.size() / 4;
            if (s.mem.n < need) {
                if (s.cluster) drop_graphs();  // the adjoint's captured launches hold the addresses
                VBD_TRY(s.mem.alloc(need));
            }
            s.words = s.mem.p;
            s.chunk = s.words + s.nwords;
            s.lists = reinterpret_cast<int*>(s.chunk + nchunk);
            CUDA_TRY(cudaMemcpyAsync(s.lists, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice, stream));
            if (s.nwords) {
                CUDA_TRY(cudaMemsetAsync(s.words, 0, sizeof(float4) * s.nwords, stream));
                VBD_TRY(set_wait_limit(s, vbd::kTileWaitNs));
            }
            s.started = 0;
            s.tag = 1;
            CUDA_TRY(cudaStreamSynchronize(stream));  // the host lists may change after this
            s.dirty = true;
            s.lanes = q.lanes;
            s.warps = q.warps;
        }
        if (s.wrapper && s.dirty) {
            const int nch = (int)(q.chunk.size() / 3);
            if (nch > 0) {
                vbd::k_pack_wrapper<<<vbd::nblk((long long)nch * 32, 256), 256, 0, stream>>>(
                    inc_off.p, inc_tet.p, rec.p, s.ints(vbd::TileSet::TABLE), nch,
                    reinterpret_cast<const vbd::TileGroup*>(s.ints(vbd::TileSet::GROUPS)),
                    reinterpret_cast<const vbd::TileHead*>(s.ints(vbd::TileSet::HEAD)), s.ints(vbd::TileSet::LID),
                    s.ints(vbd::TileSet::VTILE), s.ints(vbd::TileSet::VLOCAL), nfree, s.chunk);
                VBD_TRY(check_launch());
            }
            s.dirty = false;
        } else if (!s.wrapper && (s.dirty || s.layout != layout)) {
            const int nch = (int)(q.chunk.size() / 3);
            vbd::SweepParams p{};
            p.inc_off = inc_off.p;
            p.crec = crec.p;
            p.cmat = cmat.p;
            if (nch > 0) {
                const unsigned grid = vbd::nblk((long long)nch * 32, 256);
                auto fn = layout == 3 ? &vbd::k_pack_tile<3> : &vbd::k_pack_tile<4>;
                fn<<<grid, 256, 0, stream>>>(p, s.ints(vbd::TileSet::TABLE), nch, q.lanes,
                                             reinterpret_cast<const vbd::TileGroup*>(s.ints(vbd::TileSet::GROUPS)),
                                             reinterpret_cast<const vbd::TileHead*>(s.ints(vbd::TileSet::HEAD)),
                                             s.ints(vbd::TileSet::LID), s.ints(vbd::TileSet::VTILE),
                                             s.ints(vbd::TileSet::VLOCAL), nfree, s.chunk);
                VBD_TRY(check_launch());
            }
            s.dirty = false;
            s.layout = layout;
        }
        return VBD_OK;
    }

    // The share of the chunk stream that stays in L2 from one iteration to the next.  A stream larger than L2
    // read in order finds nothing of the last iteration there; 48 MB of it held with evict-last, and the rest
    // evict-first, leave the words and vertex state their place.  Microseconds per colour with 0 / 24 / 48 /
    // 72 / 96 MB held, and plain loads: 48^3 cube 4.61 / 4.60 / 4.57 / 4.62 / 5.02, 5.05; 64^3 8.24 / 8.09 / 8.09 / 8.30 /
    // 8.36, 8.40; 128 meshes 8.75 / 8.79 / 8.90 / 9.09 / 9.18, 9.24.  A stream that fits stays by itself (32
    // meshes 3.31 with 48 MB held, 3.26 plain).
    float tile_keep(const vbd::TileSet& s) const {
        const double bytes = (double)(s.plan.chunk.size() / 3) * s.chunk_bytes();
        return !record_cache || bytes <= vbd::kTileStreamFits ? 1.0f : (float)(vbd::kTileStreamKept / bytes);
    }
    int tile_params(vbd::TileSet& s, int k0, int k1, float dtsr, const float* omega, bool accel, int vectors,
                    vbd::TileParams* out) {
        using S = vbd::TileSet;
        const vbd::TilePlan& q = s.plan;
        vbd::TileParams w{};
        if (!s.cluster) {
            if ((unsigned long long)s.tag + (unsigned)(k1 - k0) > 0xfffffff0ull) {  // the tags start over
                CUDA_TRY(cudaMemsetAsync(s.words, 0, sizeof(float4) * (s.nwords - 1), stream));
                s.tag = 1;
            }
            w.words = s.words;
            w.word_stride = s.stride;
            w.arrived = s.arrived();
            w.arrived_target = s.started + (unsigned)q.P;
            w.tag = s.tag - (unsigned)k0;
        }
        w.chunk = s.chunk;
        w.head = reinterpret_cast<const vbd::TileHead*>(s.ints(S::HEAD));
        w.lid = s.ints(S::LID);
        w.groups = reinterpret_cast<const vbd::TileGroup*>(s.ints(S::GROUPS));
        w.wcol = s.ints(S::WCOL);
        w.ghost = s.ints(S::GHOST);
        w.wstream = reinterpret_cast<const int2*>(s.ints(S::WSTREAM));
        w.target_off = s.ints(S::TARGET_OFF);
        w.target = s.ints(S::TARGET);
        w.max_own = q.max_own;
        w.max_target = q.max_target;
        w.status = status.p;
        w.omega = omega;
        w.n = N;
        w.nfree = nfree;
        w.ncol = C;
        w.k0 = k0;
        w.k1 = k1;
        w.ring = tile_ring(s, vectors);
        w.keep = tile_keep(s);
        w.resident = tile_resident(s, vectors);
        w.ring_chunks = tile_ring_chunks(s, vectors);
        w.max_local = q.max_local;
        w.max_ids = q.max_ids;
        w.max_groups = q.max_groups;
        w.max_rounds = q.max_rounds;
        w.dtsr = dtsr;
        w.keep_pp = accel ? 1 : 0;
        w.y = y.p;
        *out = w;
        return VBD_OK;
    }

    int tile_launch(vbd::TileSet& s, void (*fn)(vbd::TileParams), vbd::TileParams& w, int vectors) {
        const size_t smem = vbd::tile_smem(s.plan.warps, w.ring_chunks, s.chunk_bytes(), s.plan, C, vectors, s.cluster);
        CUDA_TRY(allow_shared(reinterpret_cast<const void*>(fn), s.cluster));
        if (s.cluster) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            cluster_config(&cfg, attr, s.plan.P, 32 * s.plan.warps, smem);
            CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, w));
            return check_launch();
        }
        void* args[] = {&w};
        const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<void*>(fn), dim3(s.plan.P),
                                                          dim3(32 * s.plan.warps), args, smem, stream);
        if (e == cudaErrorCooperativeLaunchTooLarge) {
            (void)cudaGetLastError();
            s.no_room = true;
            return vbd::kWalkRefused;
        }
        CUDA_TRY(e);
        s.started += (unsigned)s.plan.P;
        s.tag += (unsigned)(w.k1 - w.k0);
        return check_launch();
    }

    // A sub-step (hg given: predictor and velocity update) or a solve as tile walks: one launch, or one
    // per energy evaluation with an energy history (emit_iterations' schedule).  kWalkRefused: nothing has run but,
    // with VBD_GPU_Solver semantics, the predictor.
    int launch_tile(vbd::TileSet& s, int iters, float dtsr, bool accel, float rho, bool from_inertia, float h,
                    const float* hg, bool record_energy) {
        if (!s.cluster) VBD_TRY(upload_schedule(iters, accel, rho));  // launch_cluster has
        VBD_TRY(ensure_tile(s));
        if (s.wrapper && hg) {
            // every vertex starts from its inertial target, which a tile's ghosts need before the walk
            vbd::k_predict<<<vbd::nblk(N, 256), 256, 0, stream>>>(x0.p, v.p, xprev.p, y.p, nfree, N, h, hg[0], hg[1], hg[2]);
            VBD_TRY(check_launch());
            from_inertia = true;
        }
        int k0 = 0;
        do {
            int k1 = iters;
            if (record_energy) k1 = std::min(iters, k0 == 0 ? 1 : k0 + energy_every);
            // both position buffers in shared memory where that leaves the rings their depth
            const int two = s.cluster || (accel && (tile_resident(s, 2) || (!tile_resident(s, 1) && tile_ring(s, 2) >= vbd::kTileTwoRing)));
            vbd::TileParams w;
            VBD_TRY(tile_params(s, k0, k1, dtsr, omega_at, accel, 1 + two, &w));
            w.two = two;
            w.x0 = x0.p;
            w.x1 = x1.p;
            w.pp = pp.p;
            w.v = v.p;
            w.xprev = xprev.p;
            w.predict = hg && k0 == 0 && !s.wrapper;
            w.finish = hg && k1 == iters;
            w.from_inertia = from_inertia && k0 == 0;
            w.h = h;
            if (hg) {
                w.hgx = hg[0];
                w.hgy = hg[1];
                w.hgz = hg[2];
            }
            VBD_TRY(tile_launch(s, s.wrapper ? vbd::pick_tile_wrapper(s.plan.warps)
                                         : vbd::pick_tile<vbd::kTileForward>(s.plan, s.cluster),
                                w, 1 + two));
            if (record_energy && k1 > k0 && (k1 - 1) % energy_every == 0) VBD_TRY(emit_energy_append(x0.p));
            k0 = k1;
        } while (k0 < iters);
        return VBD_OK;
    }

    // Three iterations of the walk in which the first tile that others read from publishes nothing, so that
    // their waits run out after wait_us.  The result goes nowhere.
    int walk_selftest(long long wait_us, int32_t* timed_out) {
        if (!use_tile()) VBD_FAIL(VBD_ERR_STATE, "with this mesh and these options steps do not run as tile walks");
        vbd::TileSet& s = walk_tiles();
        std::vector<vbd::TileGroup> groups = s.plan.groups;
        bool muted = false;
        for (const vbd::TileHead& h : s.plan.head) {
            for (int i = h.group; i < h.group + h.ngroups; ++i) {
                muted = muted || groups[i].publish > 0;
                groups[i].publish = 0;
            }
            if (muted) break;
        }
        if (!muted) VBD_FAIL(VBD_ERR_STATE, "no tile of this mesh reads from another");
        VBD_TRY(upload_schedule(3, false, 0.0f));
        VBD_TRY(ensure_tile(s));
        vbd::DBuf<vbd::TileGroup> list;
        vbd::DBuf<float4> x;
        VBD_TRY(list.alloc(groups.size()));
        VBD_TRY(x.alloc(N));
        CUDA_TRY(cudaMemcpyAsync(list.p, groups.data(), sizeof(vbd::TileGroup) * groups.size(), cudaMemcpyHostToDevice, stream));
        CUDA_TRY(cudaMemcpyAsync(x.p, x0.p, sizeof(float4) * (size_t)N, cudaMemcpyDeviceToDevice, stream));
        if (std::chrono::microseconds(wait_us) <= kLookAfter) looked_at = {};  // shorter than a real wait that gives up
        vbd::TileParams w;
        VBD_TRY(tile_params(s, 0, 3, 3600.0f, omega_at, false, 1, &w));
        w.groups = list.p;
        w.x0 = x.p;
        w.pp = pp.p;
        VBD_TRY(set_wait_limit(s, 1000ull * (unsigned long long)wait_us));
        const int rc = tile_launch(
            s, s.wrapper ? vbd::pick_tile_wrapper(s.plan.warps) : vbd::pick_tile<vbd::kTileForward>(s.plan, false), w, 1);
        VBD_TRY(set_wait_limit(s, vbd::kTileWaitNs));
        if (rc == vbd::kWalkRefused) VBD_FAIL(VBD_ERR_STATE, "the device refuses the walk's launch");
        VBD_TRY(rc);
        unsigned long long t = 0;
        CUDA_TRY(cudaMemcpyAsync(&t, status.p + vbd::ST_WALK_TIMEOUT, sizeof(t), cudaMemcpyDeviceToHost, stream));
        CUDA_TRY(cudaStreamSynchronize(stream));
        *timed_out = t ? 1 : 0;
        return VBD_OK;
    }

    int snapshot(vbd::DBuf<float4>& dst) {
        const size_t b4 = sizeof(float4) * (size_t)N;
        CUDA_TRY(cudaMemcpyAsync(dst.p, x0.p, b4, cudaMemcpyDeviceToDevice, stream));
        CUDA_TRY(cudaMemcpyAsync(dst.p + N, v.p, b4, cudaMemcpyDeviceToDevice, stream));
        return VBD_OK;
    }

    int record_substep(float h, float dtsr, const float* hg, int iters, bool accel, float rho) {
        if (!ckpt_every) return VBD_OK;
        TapeStep t{h, dtsr, {hg[0], hg[1], hg[2]}, rho, iters, accel ? 1 : 0};
        tape.push_back(t);
        const size_t slot = (tape.size() - 1) % (size_t)ckpt_every;
        CUDA_TRY(cudaMemcpyAsync(live_seg.p + slot * (size_t)N, x0.p, sizeof(float4) * (size_t)N,
                                 cudaMemcpyDeviceToDevice, stream));
        if (tape.size() % (size_t)ckpt_every == 0) {
            VBD_TRY(add_ckpt());
        }
        return VBD_OK;
    }

    // One recorded sub-step again, exactly as it ran (same launch sequence, hence same bits).
    int replay_substep(const TapeStep& t) {
        vbd::GraphKey key{};
        key.kind = 0;
        key.iters = t.iters;
        key.accel = t.accel;
        shape_key(key);
        key.energy_every = 0;  // the recompute appends no energies (the sweeps, hence the bits, are the same)
        key.h = t.h;
        key.dtsr = t.dtsr;
        key.hg[0] = t.hg[0];
        key.hg[1] = t.hg[1];
        key.hg[2] = t.hg[2];
        key.rho = t.rho;
        if (persistent && !timing)
            return launch_walk(t.iters, t.dtsr, t.accel != 0, t.rho, true, true, false, t.h, t.hg);
        if (use_tile()) {
            const int rc = launch_tile(tset, t.iters, t.dtsr, t.accel != 0, t.rho, false, t.h, t.hg, false);
            if (rc != vbd::kWalkRefused) return rc;
        }
        return run(key, [&] { return emit_substep(t.h, t.dtsr, t.hg, t.iters, t.accel != 0, t.rho); });
    }

    // Adjoint of one recorded sub-step whose converged positions are X: `sweeps` Gauss-Seidel
    // sweeps on (M/h^2 + H) lam = x~ + c v~ with the Chebyshev blend of weight schedule
    // getAcceleratorOmega(k, rho) (rho = 0: plain Gauss-Seidel), then the parameter gradients, the
    // pinned-vertex coupling and the step's adjoint update.
    int emit_adjoint_substep(const TapeStep& t, const float4* X, int sweeps, float rho,
                             void (*walk)(vbd::AdjWalkParams) = nullptr, vbd::TileSet* tile = nullptr) {
        const float c = 0.999f / t.h;
        const int L = lanes < 4 ? 4 : lanes;
        vbd::k_adj_rhs<<<vbd::nblk(std::max(nfree, 1), 256), 256, 0, stream>>>(adj_ax.p, adj_av.p, adj_G.p, c, nfree);
        VBD_TRY(check_launch());
        int cur = adj_cur;
        float omega = 1.0f;
        const bool accel = rho > 0.0f;
        if (walk) {
            // all sweeps in one cluster launch; the live buffer afterwards follows the same flips
            VBD_TRY(launch_cluster_adjoint(walk, t, X, sweeps, rho));
            for (int it = 1; it <= sweeps && accel; ++it) {
                omega = vbd::omega_of(it, rho, omega);
                if (omega > 1.0f) cur ^= 1;
            }
        }
        if (tile) {
            const int vectors = tile->cluster ? 3 : 2;
            vbd::TileParams w;
            VBD_TRY(tile_params(*tile, 0, sweeps, t.dtsr, d_adj_omega.p, accel, vectors, &w));
            w.X = X;
            w.G = adj_G.p;
            w.pp = adj_lpp.p;
            w.lam_in = cur ? adj_lam2.p : adj_lam.p;
            for (int it = 1; it <= sweeps && accel; ++it) {
                omega = vbd::omega_of(it, rho, omega);
                if (omega > 1.0f) cur ^= 1;
            }
            w.lam_out = cur ? adj_lam2.p : adj_lam.p;
            VBD_TRY(tile_launch(*tile, vbd::pick_tile<vbd::kTileAdjoint>(tile->plan, tile->cluster), w, vectors));
        }
        for (int it = 1; it <= sweeps && !walk && !tile; ++it) {
            bool blend = false;
            if (accel) {
                omega = vbd::omega_of(it, rho, omega);
                blend = omega > 1.0f;
            }
            float4* lr = cur ? adj_lam2.p : adj_lam.p;
            float4* lo = cur ? adj_lam.p : adj_lam2.p;
            vbd::AdjParams ap{X,         lr,      adj_G.p, y.p,   inc_off.p,     inc_tet.p,     rec.p,
                              crec.p,    cmat.p,  t.dtsr,  0,     0,             lo,            adj_lpp.p,
                              omega,     blend ? 1 : 0,    accel ? 1 : 0};
            const int alay = layout >= 2 ? layout : 0;
            for (int k = 0; k < C; ++k) {
                const int col = (adj_alternate && (it % 2 == 0)) ? C - 1 - k : k;
                ap.v_begin = cstart[col];
                ap.v_end = cstart[col + 1];
                if (ap.v_end <= ap.v_begin) continue;
                void (*fn)(vbd::AdjParams) = nullptr;
                switch (L) {
                    case 4: fn = vbd::pick_adj_sweep<4>(alay); break;
                    case 8: fn = vbd::pick_adj_sweep<8>(alay); break;
                    case 16: fn = vbd::pick_adj_sweep<16>(alay); break;
                    default: fn = vbd::pick_adj_sweep<32>(alay); break;
                }
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(vbd::nblk((long long)(ap.v_end - ap.v_begin) * L, 128));
                cfg.blockDim = dim3(128);
                cfg.stream = stream;
                cudaLaunchAttribute attr[1];
                attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
                attr[0].val.programmaticStreamSerializationAllowed = 1;
                cfg.attrs = attr;
                cfg.numAttrs = pdl ? 1 : 0;
                CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, ap));
                VBD_TRY(check_launch());
            }
            if (blend) cur ^= 1;
        }
        float4* lam = cur ? adj_lam2.p : adj_lam.p;
        if (T > 0) {
            vbd::k_adj_params<<<vbd::nblk(T, 256), 256, 0, stream>>>(rec.p, X, lam, adj_gmu.p, adj_glam.p, T);
            VBD_TRY(check_launch());
        }
        if (N > nfree) {
            vbd::AdjParams ap{X,      lam,     adj_G.p, y.p,  inc_off.p, inc_tet.p, rec.p,
                              crec.p, cmat.p,  t.dtsr,  nfree, N,        nullptr,   nullptr,
                              1.0f,   0,       0};
            const unsigned grid = vbd::nblk((long long)(N - nfree) * 8, 256);
            vbd::k_adj_pinned<8><<<grid, 256, 0, stream>>>(ap, adj_ax.p);
            VBD_TRY(check_launch());
        }
        if (nfree > 0) {
            vbd::k_adj_update<<<vbd::nblk(nfree, 256), 256, 0, stream>>>(lam, y.p, adj_ax.p, adj_av.p, t.dtsr, c, t.h,
                                                                      nfree);
            VBD_TRY(check_launch());
        }
        return VBD_OK;
    }

    // The adjoint sequence of a sub-step is replayed as a graph keyed by its parameters, the
    // positions slot it reads and which adjoint buffer is live.
    // `src` tells the state buffers apart (0 = recomputed segment, 1 = kept newest segment): the
    // captured graph bakes X's address.
    int adjoint_substep(const TapeStep& t, int slot, const float4* X, int sweeps, float rho, int src) {
        vbd::GraphKey key{};
        key.kind = 3 + slot;
        key.src = src;
        key.iters = sweeps;
        key.init = adj_cur;
        key.lanes = lanes;
        key.layout = layout;
        key.pdl = pdl;
        key.accel = adj_alternate;
        key.h = t.h;
        key.dtsr = t.dtsr;
        key.rho = rho;
        void (*walk)(vbd::AdjWalkParams) = nullptr;
        vbd::TileSet* tile = nullptr;
        if (!adj_alternate) {
            const bool walk_tiles = adj_walk() && cluster_resident && cluster_tiles(lanes < 4 ? 4 : lanes, true) && cluster_ready();
            if (walk_tiles) {
                tile = cset.get();
            } else if (use_tile()) {
                tile = &adjoint_tiles();
                if (!tile_fits(*tile, 2) || !tile_room(*tile)) tile = nullptr;
            }
        }
        if (tile) {
            VBD_TRY(upload_adj_schedule(sweeps, rho));
            VBD_TRY(ensure_tile(*tile));
        } else if (adj_walk()) {
            VBD_TRY(prepare_adj_walk(sweeps, rho, &walk));
            key.walk = 2;
            key.block = ca_ctas;
        }
        // a launch that exchanges words needs tags of its own each time: no graph
        int rc = vbd::kWalkRefused;
        if (tile && !tile->cluster) rc = emit_adjoint_substep(t, X, sweeps, rho, nullptr, tile);
        if (rc == vbd::kWalkRefused) {
            if (tile && !tile->cluster) tile = nullptr;
            if (tile) {
                key.walk = 3;
                key.block = tile->plan.P;
            }
            rc = run(key, [&] { return emit_adjoint_substep(t, X, sweeps, rho, walk, tile); });
        }
        VBD_TRY(rc);
        float omega = 1.0f;
        for (int it = 1; it <= sweeps && rho > 0.0f; ++it) {
            omega = vbd::omega_of(it, rho, omega);
            if (omega > 1.0f) adj_cur ^= 1;
        }
        return VBD_OK;
    }

    template <class Emit> int run(const vbd::GraphKey& key, Emit emit) {
        if (!use_graph || timing) return emit();
        vbd::GraphEntry* hit = nullptr;
        for (auto& g : graphs)
            if (g.key == key) hit = &g;
        // the caller is capturing the stream: the launches go straight into that capture
        if (!hit && capturing()) return emit();
        if (!hit) {
            vbd::GraphEntry e;
            e.key = key;
            const long long saved = launches;
            CUDA_TRY(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
            int rc = emit();
            cudaGraph_t g = nullptr;
            cudaError_t ce = cudaStreamEndCapture(stream, &g);
            launches = saved;
            if (rc) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            if (ce != cudaSuccess) VBD_FAIL(VBD_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(ce));
            e.graph = g;
            CUDA_TRY(cudaGraphGetNodes(g, nullptr, &e.nodes));
            cudaError_t ie = cudaGraphInstantiate(&e.exec, g, 0);
            if (ie != cudaSuccess) {
                cudaGraphDestroy(g);
                VBD_FAIL(VBD_ERR_CUDA, "graph instantiation failed: %s", cudaGetErrorString(ie));
            }
            if (graphs.size() >= 64) {
                cudaGraphExecDestroy(graphs.front().exec);
                cudaGraphDestroy(graphs.front().graph);
                graphs.erase(graphs.begin());
            }
            graphs.push_back(e);
            hit = &graphs.back();
        }
        CUDA_TRY(cudaGraphLaunch(hit->exec, stream));
        launches += (long long)hit->nodes;
        return VBD_OK;
    }

    int upload3(const float* src, float4* d0, float4* d1) {
        CUDA_TRY(cudaMemcpyAsync(stage.p, src, sizeof(float) * 3 * (size_t)N, cudaMemcpyDefault, stream));
        vbd::k_scatter3<<<vbd::nblk(N, 256), 256, 0, stream>>>(stage.p, perm.p, d0, d1, N);
        VBD_TRY(check_launch());
        CUDA_TRY(cudaStreamSynchronize(stream));
        return VBD_OK;
    }

    int download3(const float4* src, float* dst) {
        vbd::k_gather3<<<vbd::nblk(N, 256), 256, 0, stream>>>(src, perm.p, stage.p, N);
        VBD_TRY(check_launch());
        CUDA_TRY(cudaMemcpyAsync(dst, stage.p, sizeof(float) * 3 * (size_t)N, cudaMemcpyDefault, stream));
        return finish();
    }

    // Captured graphs bake in buffer addresses: every (re)allocation or release of the streamed
    // record copies invalidates them.
    int repack_stream() {
        tset.dirty = aset.dirty = cset->dirty = wset.dirty = true;
        for (auto& h : held) h->dirty = true;
        if (layout != 1 && irec.p) {
            drop_graphs();
            irec.release();
        }
        if (layout != 2 && layout != 4 && cmat.p) {
            drop_graphs();
            cmat.release();
        }
        if (layout < 2 && crec.p) {
            drop_graphs();
            crec.release();
        }
        if (layout == 1) {
            if (irec.n != (size_t)ninc) {
                drop_graphs();
                VBD_TRY(irec.alloc(ninc));
            }
            if (ninc > 0) {
                vbd::k_pack_stream<<<vbd::nblk(ninc, 256), 256, 0, stream>>>(rec.p, inc_tet.p, irec.p, (int)ninc);
                VBD_TRY(check_launch());
            }
        } else if (layout >= 2) {
            const size_t words = layout == 4 ? 2 : 3;
            if (crec.n != words * (size_t)ninc) {
                drop_graphs();
                VBD_TRY(crec.alloc(words * (size_t)ninc));
            }
            if (layout != 3 && cmat.n != (size_t)ninc) {
                drop_graphs();
                VBD_TRY(cmat.alloc(ninc));
            }
            if (ninc > 0 && layout == 2) {
                vbd::k_pack_compact<<<vbd::nblk(ninc, 256), 256, 0, stream>>>(rec.p, inc_tet.p, inc_vertex.p, crec.p,
                                                                             cmat.p, (int)ninc);
                VBD_TRY(check_launch());
            } else if (ninc > 0 && layout == 3) {
                vbd::k_pack_factored<false><<<vbd::nblk(ninc, 256), 256, 0, stream>>>(
                    rec.p, inc_tet.p, inc_vertex.p, crec.p, nullptr, (int)ninc);
                VBD_TRY(check_launch());
            } else if (ninc > 0) {
                vbd::k_pack_factored<true><<<vbd::nblk(ninc, 256), 256, 0, stream>>>(
                    rec.p, inc_tet.p, inc_vertex.p, crec.p, cmat.p, (int)ninc);
                VBD_TRY(check_launch());
            }
        }
        // what the caller's captured launches read, as they read the records themselves
        if (layout >= 3) {
            for (auto& h : held) VBD_TRY(ensure_tile(*h));
            if (cset->captured) VBD_TRY(ensure_tile(*cset));
            else if (persistent == 2 && cset->lanes) (void)tile_room(*cset);
        }
        return VBD_OK;
    }

    int reduce_scalar(unsigned blocks, double* out) {
        vbd::k_sum_partials<<<1, 1024, 0, stream>>>(partials.p, (int)blocks, scalar.p);
        VBD_TRY(check_launch());
        CUDA_TRY(cudaMemcpyAsync(out, scalar.p, sizeof(double), cudaMemcpyDeviceToHost, stream));
        return finish();
    }
};

namespace {

struct DeviceScope {
    int prev = -1;
    explicit DeviceScope(int d) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != d) cudaSetDevice(d);
    }
    ~DeviceScope() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

// The SMs that launches on `stream` may use: fewer than the device's where the stream belongs to a green context.
int stream_sms(cudaStream_t stream, int device_sms) {
    void *of_stream = nullptr, *resource = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuStreamGetGreenCtx", &of_stream, 12040, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess ||
        cudaGetDriverEntryPointByVersion("cuGreenCtxGetDevResource", &resource, 12040, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
        (void)cudaGetLastError();
        return device_sms;
    }
    CUgreenCtx ctx = nullptr;
    CUdevResource r{};
    if (reinterpret_cast<decltype(&cuStreamGetGreenCtx)>(of_stream)(stream, &ctx) != CUDA_SUCCESS || !ctx ||
        reinterpret_cast<decltype(&cuGreenCtxGetDevResource)>(resource)(ctx, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
        return device_sms;
    return std::max(1, std::min<int>(device_sms, (int)r.sm.smCount));
}

int need_ready(vbd_solver* s) {
    if (!s) VBD_FAIL(VBD_ERR_INVALID_ARG, "null solver handle");
    if (!s->ready) VBD_FAIL(VBD_ERR_STATE, "solver has no mesh: call vbd_solver_init first");
    return VBD_OK;
}

}  // namespace

extern "C" {

int vbd_solver_create(vbd_solver** out, int device, void* cuda_stream) {
    vbd::clear_error();
    if (!out) VBD_FAIL(VBD_ERR_INVALID_ARG, "out is null");
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        cudaGetLastError();
        VBD_FAIL(VBD_ERR_NO_DEVICE, "no CUDA device available");
    }
    if (device < 0 || device >= count) VBD_FAIL(VBD_ERR_NO_DEVICE, "device %d out of range (%d devices)", device, count);
    // single attributes: cudaGetDeviceProperties takes 2.5 ms
    int major = 0, minor = 0, sms = 0, smem = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    CUDA_TRY(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    CUDA_TRY(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    if (major != 10 || minor != 0)
        VBD_FAIL(VBD_ERR_NO_DEVICE, "device %d is sm_%d%d; this library is built for sm_100a only", device, major, minor);
    DeviceScope scope(device);
    std::unique_ptr<vbd_solver> s(new vbd_solver());
    s->device = device;
    if (cuda_stream) {
        s->stream = static_cast<cudaStream_t>(cuda_stream);
    } else {
        CUDA_TRY(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
        s->own_stream = true;
    }
    s->sm_count = stream_sms(s->stream, sms);
    s->smem_optin = smem;
    VBD_TRY(s->status.alloc(vbd::ST_SLOTS));
    CUDA_TRY(cudaMemsetAsync(s->status.p, 0, sizeof(unsigned long long) * vbd::ST_SLOTS, s->stream));
    VBD_TRY(s->scalar.alloc(1));
    *out = s.release();
    return VBD_OK;
}

int vbd_solver_destroy(vbd_solver* s) {
    vbd::clear_error();
    if (!s) return VBD_OK;
    DeviceScope scope(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    delete s;
    return VBD_OK;
}

int vbd_solver_init(vbd_solver* s, int32_t N, int32_t T, const float* positions, const float* velocities,
                    const float* inertia, const float* vertex_mass, const uint8_t* fixed, const int32_t* tets,
                    int32_t num_colours, const int32_t* group_offsets, const int32_t* group_vertices,
                    const float* dm_inv, const float* rest_vol, const float* tet_mu, const float* tet_lambda) {
    vbd::clear_error();
    if (!s) VBD_FAIL(VBD_ERR_INVALID_ARG, "null solver handle");
    if (N <= 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "num_verts must be positive (got %d)", N);
    if (T < 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "num_tets is negative");
    if (!positions || !vertex_mass || !fixed) VBD_FAIL(VBD_ERR_INVALID_ARG, "positions, vertex_mass, fixed are required");
    if (T > 0 && (!dm_inv || !rest_vol)) VBD_FAIL(VBD_ERR_INVALID_ARG, "dm_inv and rest_vol are required");
    if (num_colours < 0 || (num_colours > 0 && (!group_offsets || !group_vertices)))
        VBD_FAIL(VBD_ERR_INVALID_ARG, "colour groups missing");
    if ((tet_mu == nullptr) != (tet_lambda == nullptr))
        VBD_FAIL(VBD_ERR_INVALID_ARG, "give both tet_mu and tet_lambda, or neither");
    if ((long long)T * 4 > 0x7fffffffLL) VBD_FAIL(VBD_ERR_INVALID_ARG, "too many tets for 32-bit incidence ids");
    if (!s->layout_auto && s->layout == 4 && N > vbd::kPackedMaxVertices)
        VBD_FAIL(VBD_ERR_INVALID_ARG, "layout 4 holds vertex ids below 2^21; this mesh has %d vertices", N);
    VBD_TRY(vbd::check_tets(N, T, tets));
    // colour groups: a partition of the vertices into independent sets
    if (num_colours == 0 || group_offsets[0] != 0 || group_offsets[num_colours] != N)
        VBD_FAIL(VBD_ERR_INVALID_ARG, "colour groups must cover all %d vertices", N);
    std::vector<int32_t> colour(N, -1);
    for (int c = 0; c < num_colours; ++c) {
        if (group_offsets[c + 1] < group_offsets[c]) VBD_FAIL(VBD_ERR_INVALID_ARG, "colour offsets decrease at %d", c);
        for (int k = group_offsets[c]; k < group_offsets[c + 1]; ++k) {
            int vtx = group_vertices[k];
            if (vtx < 0 || vtx >= N) VBD_FAIL(VBD_ERR_INVALID_ARG, "colour group %d holds vertex %d out of range", c, vtx);
            if (colour[vtx] != -1) VBD_FAIL(VBD_ERR_INVALID_ARG, "vertex %d appears in two colour groups", vtx);
            colour[vtx] = c;
        }
    }
    for (int t = 0; t < T; ++t) {
        const int32_t* q = tets + 4LL * t;
        for (int a = 0; a < 4; ++a)
            for (int b = 0; b < a; ++b)
                if (colour[q[a]] == colour[q[b]])
                    VBD_FAIL(VBD_ERR_INVALID_ARG,
                             "colour groups are not independent: vertices %d and %d of tet %d share colour %d", q[a],
                             q[b], t, colour[q[a]]);
    }
    for (int i = 0; i < N; ++i)
        if (!(vertex_mass[i] >= 0.0f) || !std::isfinite(vertex_mass[i]))
            VBD_FAIL(VBD_ERR_INVALID_ARG, "vertex_mass[%d] is negative or not finite", i);

    DeviceScope scope(s->device);
    CUDA_TRY(cudaStreamSynchronize(s->stream));
    s->ckpt_pool.clear();
    s->ready = false;
    s->drop_graphs();
    s->irec.release();
    s->crec.release();
    s->cmat.release();

    // Incident tets of each vertex, ascending tet id (TetMesh::vertAdjacentTets).
    std::vector<int32_t> voff(N + 1), vtets(4LL * T);
    vbd::build_vertex_tets(N, T, tets, voff.data(), vtets.data());

    // Tiles of the tile walk.
    vbd::TilePlan plan;
    std::vector<int32_t> tile;
    std::vector<uint8_t> boundary;
    {
        int free_count = 0;
        for (int i = 0; i < N; ++i) free_count += fixed[i] ? 0 : 1;
        if (free_count > 0 && T > 0) {
            // one per SM, kTileVertices at least; for small meshes a multiple of 16, which the cluster's CTAs
            // share evenly
            plan.P = std::min(s->sm_count, free_count / vbd::kTileVertices);
            if (free_count <= vbd::kClusterMeshVertices) plan.P = std::max(16, plan.P / 16 * 16);
            plan.P = std::max(1, std::min(plan.P, free_count));
            plan.n = N;
            plan.nfree = free_count;
            const int32_t* mesh = (int)s->batch_mesh.size() == N ? s->batch_mesh.data() : nullptr;
            vbd::tile_partition(N, positions, fixed, mesh, plan.P, &tile);
            vbd::tile_boundary(N, T, tets, tile, &boundary);
        }
    }

    // Internal order: free vertices colour by colour, then the pinned ones.  Inside a colour: group
    // order, or with tiles tile by tile, in a tile the vertices other tiles read first, then by falling
    // valence (the vertices a warp of the tile walk sweeps together then have about as many tets).
    std::vector<int32_t> perm;
    perm.reserve(N);
    std::vector<int> cstart(num_colours + 1, 0);
    std::vector<std::pair<unsigned long long, int32_t>> order, keys;
    std::vector<std::pair<int, int>> sorted_at;
    for (int c = 0; c < num_colours; ++c) {
        cstart[c] = (int)perm.size();
        if (!plan.P) {
            for (int k = group_offsets[c]; k < group_offsets[c + 1]; ++k)
                if (!fixed[group_vertices[k]]) perm.push_back(group_vertices[k]);
            continue;
        }
        order.clear();
        for (int k = group_offsets[c]; k < group_offsets[c + 1]; ++k) {
            const int32_t i = group_vertices[k];
            if (fixed[i]) continue;
            const unsigned long long val = (unsigned)std::min(voff[i + 1] - voff[i], 0xffff);
            order.emplace_back(((unsigned long long)tile[i] << 17) | ((boundary[i] ? 0ull : 1ull) << 16) | (0xffffull - val), i);
        }
        for (const auto& o : order) perm.push_back(o.second);
        sorted_at.emplace_back(cstart[c], (int)perm.size());
        keys.insert(keys.end(), order.begin(), order.end());
    }
    if (plan.P)  // each colour in its own order
        vbd::each_item((int)sorted_at.size(), N > 4000, [&](int, int c) {
            const auto r = sorted_at[c];
            std::sort(keys.begin() + r.first, keys.begin() + r.second);
            for (int i = r.first; i < r.second; ++i) perm[i] = keys[i].second;
        });
    cstart[num_colours] = (int)perm.size();
    const int nfree = (int)perm.size();
    for (int i = 0; i < N; ++i)
        if (fixed[i]) perm.push_back(i);
    std::vector<int32_t> iperm(N);
    for (int i = 0; i < N; ++i) iperm[perm[i]] = i;

    // Incident tets of every vertex (free ones first, so the sweeps' incidences are [0, ninc); the
    // pinned vertices' lists serve the adjoint's coupling term).
    std::vector<int32_t> inc_off(N + 1, 0);
    for (int i = 0; i < N; ++i) inc_off[i + 1] = inc_off[i] + (voff[perm[i] + 1] - voff[perm[i]]);
    const long long ninc = inc_off[nfree];
    const long long ninc_all = inc_off[N];
    std::vector<int32_t> inc_tet(std::max<long long>(ninc_all, 1)), inc_vertex(std::max<long long>(ninc_all, 1));
    const bool large = N > 4000;
    vbd::each_range(N, large, [&](int, long long b, long long e) {
        for (long long i = b; i < e; ++i) {
            std::copy(vtets.begin() + voff[perm[i]], vtets.begin() + voff[perm[i] + 1], inc_tet.begin() + inc_off[i]);
            std::fill(inc_vertex.begin() + inc_off[i], inc_vertex.begin() + inc_off[i + 1], (int32_t)i);
        }
    });

    std::vector<vbd::TetRec> rec(std::max(T, 1));
    vbd::each_range(T, large, [&](int, long long b, long long e) {
        for (long long t = b; t < e; ++t) {
            const int32_t* q = tets + 4LL * t;
            const float* d = dm_inv + 9LL * t;
            vbd::TetRec& r = rec[t];
            r.ids = make_int4(iperm[q[0]], iperm[q[1]], iperm[q[2]], iperm[q[3]]);
            r.a = make_float4(d[0], d[1], d[2], d[3]);
            r.b = make_float4(d[4], d[5], d[6], d[7]);
            r.c = make_float4(d[8], rest_vol[t], tet_mu ? tet_mu[t] : 0.0f, tet_lambda ? tet_lambda[t] : 0.0f);
        }
    });

    if (plan.P) {
        std::vector<int32_t> tile_in(N, -1);
        std::vector<uint8_t> bnd_in(N, 0);
        for (int i = 0; i < nfree; ++i) {
            tile_in[i] = tile[perm[i]];
            bnd_in[i] = boundary[perm[i]];
        }
        vbd::tile_lists(&plan, cstart, tile_in, bnd_in, inc_off.data(), inc_tet.data(), &rec[0].ids.x,
                        (int)(sizeof(vbd::TetRec) / sizeof(int)));
    }
    s->tset.reset(std::move(plan));
    s->aset.reset(vbd::TilePlan());
    s->cset.reset(new vbd::TileSet());
    s->held.clear();
    s->wset.reset(vbd::TilePlan());
    s->tile_walk = !s->persistent_set && nfree >= vbd::kTileMinVertices;

    std::vector<float4> hx(N), hv(N), hy(N);
    for (int i = 0; i < N; ++i) {
        const int o = perm[i];
        hx[i] = make_float4(positions[3LL * o], positions[3LL * o + 1], positions[3LL * o + 2], 0.0f);
        hv[i] = velocities ? make_float4(velocities[3LL * o], velocities[3LL * o + 1], velocities[3LL * o + 2], 0.0f)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
        const float* yy = inertia ? inertia + 3LL * o : positions + 3LL * o;
        hy[i] = make_float4(yy[0], yy[1], yy[2], vertex_mass[o]);
    }

    VBD_TRY(s->x0.alloc(N));
    VBD_TRY(s->x1.alloc(N));
    VBD_TRY(s->pp.alloc(N));
    VBD_TRY(s->y.alloc(N));
    VBD_TRY(s->v.alloc(N));
    VBD_TRY(s->xprev.alloc(N));
    VBD_TRY(s->perm.alloc(N));
    VBD_TRY(s->inc_off.alloc(N + 1));
    VBD_TRY(s->inc_tet.alloc(inc_tet.size()));
    VBD_TRY(s->inc_vertex.alloc(inc_vertex.size()));
    VBD_TRY(s->rec.alloc(rec.size()));
    VBD_TRY(s->stage.alloc(3LL * N));
    VBD_TRY(s->mat_stage.alloc(2LL * std::max(T, 1)));
    const long long max_blocks = std::max<long long>(4096, vbd::nblk((long long)N * 32, 256));
    VBD_TRY(s->partials.alloc(max_blocks));
    const size_t b4 = sizeof(float4) * (size_t)N;
    // on the solver's own stream: a copy from pageable memory may return before it has landed, and a
    // non-blocking stream's kernels do not wait for the legacy stream's copies
    CUDA_TRY(cudaMemcpyAsync(s->x0.p, hx.data(), b4, cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->x1.p, hx.data(), b4, cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->xprev.p, hx.data(), b4, cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->pp.p, hx.data(), b4, cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->v.p, hv.data(), b4, cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->y.p, hy.data(), b4, cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->perm.p, perm.data(), sizeof(int) * N, cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->inc_off.p, inc_off.data(), sizeof(int) * (N + 1), cudaMemcpyHostToDevice, s->stream));
    s->h_inc_off = inc_off;  // the tile plans read it on the host
    CUDA_TRY(cudaMemcpyAsync(s->inc_tet.p, inc_tet.data(), sizeof(int) * inc_tet.size(), cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->inc_vertex.p, inc_vertex.data(), sizeof(int) * inc_vertex.size(), cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->rec.p, rec.data(), sizeof(vbd::TetRec) * rec.size(), cudaMemcpyHostToDevice, s->stream));
    CUDA_TRY(cudaMemsetAsync(s->status.p, 0, sizeof(unsigned long long) * vbd::ST_SLOTS, s->stream));
    // the energy history belongs to the previous mesh
    s->ehist_queued = 0;
    if (s->ecount.p) CUDA_TRY(cudaMemsetAsync(s->ecount.p, 0, sizeof(int), s->stream));

    if (s->lanes_auto) {
        int L = (nfree > 0 && (double)ninc >= 21.0 * nfree) ? 8 : 4;
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
        long long largest = 0;
        for (int c = 0; c < num_colours; ++c) largest = std::max<long long>(largest, cstart[c + 1] - cstart[c]);
        while (L < 16 && largest * L * 2 <= (long long)sms * 1024) L *= 2;
        s->lanes = L;
    }
    if (s->layout_auto) {
        // Layout 4 derives det M from s and w, which cancels on anisotropic tets (a vertex whose row
        // of Ps Dm^-1 is small next to the others); layout 3 stores det M.  On sliver tets both carry
        // the FP32 conditioning error of Dm^-1 itself, which the reference's own F = Ds Dm^-1 shares.
        // So layout 4 is kept unless it loses accuracy on more than a small fraction of the
        // incidences.
        double e3 = 0.0, e4 = 0.0, f4 = 0.0;
        vbd::factored_detm_error(T, dm_inv, &e3, &e4, &f4);
        s->layout = (N <= vbd::kPackedMaxVertices && f4 <= vbd::kFactoredLossFraction) ? 4 : 3;
    }
    if (s->record_cache_auto) s->record_cache = 1;
    if (s->persist_auto) s->persist_mb = 64.0 * N <= 32.0 * 1048576.0 ? 32 : 0;
    s->max_valence = 0;
    for (int i = 0; i < nfree; ++i) s->max_valence = std::max(s->max_valence, inc_off[i + 1] - inc_off[i]);
    s->colour_maxval.assign(num_colours, 0);
    for (int c = 0; c < num_colours; ++c)
        for (int i = cstart[c]; i < cstart[c + 1]; ++i)
            s->colour_maxval[c] = std::max(s->colour_maxval[c], inc_off[i + 1] - inc_off[i]);
    // a per-colour launch shape belongs to the previous mesh's colours
    s->colour_lanes.clear();
    ++s->shape_gen;
    s->colour_inc.assign(num_colours + 1, 0);
    for (int c = 0; c <= num_colours; ++c) s->colour_inc[c] = inc_off[cstart[c]];
    s->colour_bytes.assign(num_colours, 0.0);
    for (int c = 0; c < num_colours; ++c)
        for (int i = cstart[c]; i < cstart[c + 1]; ++i)
            s->colour_bytes[c] += 60.0 * (inc_off[i + 1] - inc_off[i]) + 96.0;
    s->N = N;
    s->T = T;
    s->C = num_colours;
    s->nfree = nfree;
    s->ninc = ninc;
    s->cstart = cstart;
    s->d_cstart.release();
    s->schedules.clear();
    s->have_materials = tet_mu != nullptr;
    VBD_TRY(s->repack_stream());
    if (s->use_tile()) VBD_TRY(s->ensure_tile(s->walk_tiles()));
    CUDA_TRY(cudaStreamSynchronize(s->stream));
    s->looked_at = std::chrono::steady_clock::now();  // the record was cleared above
    s->ready = true;
    return s->prepare_cluster();
}

int vbd_solver_init_batch(vbd_solver* s, int32_t M, const int32_t* voff, const int32_t* toff, const float* positions,
                          const float* velocities, const float* vertex_mass, const uint8_t* fixed,
                          const int32_t* tets_local, const float* dm_inv, const float* rest_vol, const float* tet_mu,
                          const float* tet_lambda) {
    vbd::clear_error();
    if (!s) VBD_FAIL(VBD_ERR_INVALID_ARG, "null solver handle");
    if (M <= 0 || !voff || !toff) VBD_FAIL(VBD_ERR_INVALID_ARG, "need num_meshes > 0 and the offset arrays");
    if (voff[0] != 0 || toff[0] != 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "offsets must start at 0");
    for (int m = 0; m < M; ++m)
        if (voff[m + 1] < voff[m] || toff[m + 1] < toff[m])
            VBD_FAIL(VBD_ERR_INVALID_ARG, "offsets of mesh %d decrease", m);
    const int32_t N = voff[M], T = toff[M];
    if (T > 0 && !tets_local) VBD_FAIL(VBD_ERR_INVALID_ARG, "tets_local is null");
    // global ids; each mesh's ids must stay inside its own vertex range
    std::vector<int32_t> tets(4LL * T);
    for (int m = 0; m < M; ++m) {
        const int32_t nv = voff[m + 1] - voff[m];
        for (int64_t k = 4LL * toff[m]; k < 4LL * toff[m + 1]; ++k) {
            const int32_t id = tets_local[k];
            if (id < 0 || id >= nv)
                VBD_FAIL(VBD_ERR_INVALID_ARG, "mesh %d: tet %lld holds local vertex id %d outside [0, %d)", m,
                         (long long)(k / 4), id, nv);
            tets[k] = id + voff[m];
        }
    }
    // Greedy colouring of the union: a vertex's neighbours all lie in its own mesh, so every mesh
    // receives exactly its own GraphColoring::colorVertices assignment.
    std::vector<int32_t> colour_of(N);
    int32_t nc = 0;
    VBD_TRY(vbd_color_vertices(N, T, tets.data(), colour_of.data(), &nc, 0, nullptr, nullptr));
    std::vector<int32_t> offs(nc + 1), verts(N);
    VBD_TRY(vbd_color_vertices(N, T, tets.data(), colour_of.data(), &nc, nc, offs.data(), verts.data()));
    s->batch_mesh.resize(N);
    for (int m = 0; m < M; ++m) std::fill(s->batch_mesh.begin() + voff[m], s->batch_mesh.begin() + voff[m + 1], m);
    const int rc = vbd_solver_init(s, N, T, positions, velocities, nullptr, vertex_mass, fixed, tets.data(), nc, offs.data(),
                                   verts.data(), dm_inv, rest_vol, tet_mu, tet_lambda);
    s->batch_mesh.clear();
    return rc;
}

int vbd_solver_set_materials(vbd_solver* s, const float* tet_mu, const float* tet_lambda) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!tet_mu && !tet_lambda) return VBD_OK;
    if (!s->have_materials && !(tet_mu && tet_lambda))
        VBD_FAIL(VBD_ERR_STATE, "materials were never set: give both tet_mu and tet_lambda");
    DeviceScope scope(s->device);
    if (s->T == 0) {
        s->have_materials = true;
        return VBD_OK;
    }
    float* dmu = nullptr;
    float* dlam = nullptr;
    if (tet_mu) {
        dmu = s->mat_stage.p;
        CUDA_TRY(cudaMemcpyAsync(dmu, tet_mu, sizeof(float) * s->T, cudaMemcpyDefault, s->stream));
    }
    if (tet_lambda) {
        dlam = s->mat_stage.p + s->T;
        CUDA_TRY(cudaMemcpyAsync(dlam, tet_lambda, sizeof(float) * s->T, cudaMemcpyDefault, s->stream));
    }
    vbd::k_set_materials<<<vbd::nblk(s->T, 256), 256, 0, s->stream>>>(s->rec.p, dmu, dlam, -1.f, -1.f, s->T);
    VBD_TRY(s->check_launch());
    VBD_TRY(s->repack_stream());
    CUDA_TRY(cudaStreamSynchronize(s->stream));
    s->have_materials = true;
    return VBD_OK;
}

int vbd_solver_set_uniform_material(vbd_solver* s, float mu, float lambda) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!(mu >= 0.f) || !(lambda >= 0.f) || !std::isfinite(mu) || !std::isfinite(lambda))
        VBD_FAIL(VBD_ERR_INVALID_ARG, "mu and lambda must be finite and non-negative");
    DeviceScope scope(s->device);
    if (s->T > 0) {
        vbd::k_set_materials<<<vbd::nblk(s->T, 256), 256, 0, s->stream>>>(s->rec.p, nullptr, nullptr, mu, lambda,
                                                                          s->T);
        VBD_TRY(s->check_launch());
        VBD_TRY(s->repack_stream());
        CUDA_TRY(cudaStreamSynchronize(s->stream));
    }
    s->have_materials = true;
    return VBD_OK;
}

int vbd_solver_set_positions(vbd_solver* s, const float* xyz) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!xyz) VBD_FAIL(VBD_ERR_INVALID_ARG, "xyz is null");
    DeviceScope scope(s->device);
    return s->upload3(xyz, s->x0.p, s->x1.p);
}

int vbd_solver_get_positions(vbd_solver* s, float* xyz) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!xyz) VBD_FAIL(VBD_ERR_INVALID_ARG, "xyz is null");
    DeviceScope scope(s->device);
    return s->download3(s->x0.p, xyz);
}

int vbd_solver_set_velocities(vbd_solver* s, const float* xyz) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!xyz) VBD_FAIL(VBD_ERR_INVALID_ARG, "xyz is null");
    DeviceScope scope(s->device);
    return s->upload3(xyz, s->v.p, nullptr);
}

int vbd_solver_get_velocities(vbd_solver* s, float* xyz) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!xyz) VBD_FAIL(VBD_ERR_INVALID_ARG, "xyz is null");
    DeviceScope scope(s->device);
    return s->download3(s->v.p, xyz);
}

int vbd_solver_set_inertia(vbd_solver* s, const float* xyz) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!xyz) VBD_FAIL(VBD_ERR_INVALID_ARG, "xyz is null");
    DeviceScope scope(s->device);
    return s->upload3(xyz, s->y.p, nullptr);
}

int vbd_solver_get_inertia(vbd_solver* s, float* xyz) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!xyz) VBD_FAIL(VBD_ERR_INVALID_ARG, "xyz is null");
    DeviceScope scope(s->device);
    return s->download3(s->y.p, xyz);
}

int vbd_solver_solve(vbd_solver* s, int32_t iterations, float dt_sqr_reciprocal, int32_t use_acceleration, float rho,
                     int32_t init_mode) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!s->have_materials) VBD_FAIL(VBD_ERR_STATE, "materials not set");
    if (iterations < 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "iterations must be >= 0");
    if (!(dt_sqr_reciprocal > 0.f) || !std::isfinite(dt_sqr_reciprocal))
        VBD_FAIL(VBD_ERR_INVALID_ARG, "dt_sqr_reciprocal must be positive and finite");
    if (init_mode != VBD_INIT_FROM_POSITIONS && init_mode != VBD_INIT_FROM_INERTIA)
        VBD_FAIL(VBD_ERR_INVALID_ARG, "unknown init_mode %d", init_mode);
    DeviceScope scope(s->device);
    vbd::GraphKey key{};
    key.kind = 1;
    key.iters = iterations;
    key.accel = use_acceleration ? 1 : 0;
    key.init = init_mode;
    s->shape_key(key);
    key.dtsr = dt_sqr_reciprocal;
    key.rho = rho;
    if (s->persistent && !s->timing)
        return s->launch_walk(iterations, dt_sqr_reciprocal, use_acceleration != 0, rho, false, false,
                              init_mode == VBD_INIT_FROM_INERTIA, 1.0f, nullptr);
    if (s->use_tile()) {
        const int rc = s->launch_tile(s->walk_tiles(), iterations, dt_sqr_reciprocal, use_acceleration != 0, rho,
                                      init_mode == VBD_INIT_FROM_INERTIA, 1.0f, nullptr, false);
        if (rc != vbd::kWalkRefused) return rc;
    }
    return s->run(key, [&] { return s->emit_solve(iterations, dt_sqr_reciprocal, use_acceleration != 0, rho, init_mode); });
}

int vbd_solver_solve_iteration(vbd_solver* s, float dt_sqr_reciprocal) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!s->have_materials) VBD_FAIL(VBD_ERR_STATE, "materials not set");
    if (!(dt_sqr_reciprocal > 0.f) || !std::isfinite(dt_sqr_reciprocal))
        VBD_FAIL(VBD_ERR_INVALID_ARG, "dt_sqr_reciprocal must be positive and finite");
    DeviceScope scope(s->device);
    int cur = 0;
    return s->emit_iterations(1, dt_sqr_reciprocal, false, 0.f, cur);
}

int vbd_solver_step(vbd_solver* s, float dt, int32_t substeps, int32_t iterations, const float* gravity,
                    int32_t use_acceleration, float rho) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!s->have_materials) VBD_FAIL(VBD_ERR_STATE, "materials not set");
    if (!(dt > 0.f) || !std::isfinite(dt)) VBD_FAIL(VBD_ERR_INVALID_ARG, "dt must be positive and finite");
    if (substeps < 1) VBD_FAIL(VBD_ERR_INVALID_ARG, "substeps must be >= 1");
    if (iterations < 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "iterations must be >= 0");
    if (!gravity) VBD_FAIL(VBD_ERR_INVALID_ARG, "gravity is null");
    DeviceScope scope(s->device);
    const float h = dt / (float)substeps;
    // 1/h^2: VBD.cpp computes it through double, main.cpp's GPU loop in float (main.cpp:211)
    const float dtsr = s->semantics ? 1.0f / (h * h) : (float)(1.0 / (double)(h * h));
    const float hg[3] = {h * gravity[0], h * gravity[1], h * gravity[2]};
    vbd::GraphKey key{};
    key.kind = 0;
    key.iters = iterations;
    key.accel = use_acceleration ? 1 : 0;
    s->shape_key(key);
    key.h = h;
    key.dtsr = dtsr;
    key.hg[0] = hg[0];
    key.hg[1] = hg[1];
    key.hg[2] = hg[2];
    key.rho = rho;
    const long long nenergy = s->energies_per_step(substeps, iterations);
    if (nenergy > 0) VBD_TRY(s->reserve_energies(nenergy));
    for (int k = 0; k < substeps; ++k) {
        // the persistent kernel evaluates no energies: with an energy history the step runs as
        // separate launches
        int rc = vbd::kWalkRefused;
        bool predicted = false;
        if (s->persistent && !s->timing && nenergy == 0) {
            rc = s->launch_walk(iterations, dtsr, use_acceleration != 0, rho, true, true, false, h, hg);
        } else if (s->use_tile()) {
            rc = s->launch_tile(s->walk_tiles(), iterations, dtsr, use_acceleration != 0, rho, false, h, hg, nenergy > 0);
            predicted = s->semantics != 0;
        }
        const auto emit = [&] {
            return s->emit_substep(h, dtsr, hg, iterations, use_acceleration != 0, rho, nenergy > 0, predicted);
        };
        if (rc == vbd::kWalkRefused) rc = predicted ? emit() : s->run(key, emit);
        VBD_TRY(rc);
        VBD_TRY(s->record_substep(h, dtsr, hg, iterations, use_acceleration != 0, rho));
    }
    s->ehist_queued += nenergy;
    return VBD_OK;
}

int vbd_solver_energy_history(vbd_solver* s, double* energies, int32_t capacity, int32_t* count, int32_t reset) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!count) VBD_FAIL(VBD_ERR_INVALID_ARG, "count is null");
    if (capacity < 0 || (capacity > 0 && !energies)) VBD_FAIL(VBD_ERR_INVALID_ARG, "need energies[capacity]");
    DeviceScope scope(s->device);
    int n = 0;
    if (s->ecount.p) {
        CUDA_TRY(cudaMemcpyAsync(&n, s->ecount.p, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
        VBD_TRY(s->finish());
    }
    const int avail = (int)std::min<long long>(n, (long long)s->ehist.n);
    const int copy = std::min(avail, capacity);
    if (copy > 0) {
        CUDA_TRY(cudaMemcpyAsync(energies, s->ehist.p, sizeof(double) * copy, cudaMemcpyDefault, s->stream));
        CUDA_TRY(cudaStreamSynchronize(s->stream));
    }
    *count = n;
    if (reset && s->ecount.p) {
        CUDA_TRY(cudaMemsetAsync(s->ecount.p, 0, sizeof(int), s->stream));
        CUDA_TRY(cudaStreamSynchronize(s->stream));
        s->ehist_queued = 0;
    }
    return VBD_OK;
}

int vbd_solver_record(vbd_solver* s, int32_t checkpoint_every) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (checkpoint_every < 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "checkpoint_every must be >= 0");
    if (checkpoint_every > 0 && s->semantics)
        VBD_FAIL(VBD_ERR_STATE, "the adjoint differentiates the VBDsolver semantics; set VBD_OPT_SEMANTICS to 0");
    DeviceScope scope(s->device);
    if (checkpoint_every > 0) VBD_TRY(s->finish());  // of a state to start from
    s->tape.clear();
    // a new recording reuses the last one's buffers; stopping, and a new mesh, give them back
    if (checkpoint_every == 0) s->ckpt_pool.clear();
    else for (auto& c : s->ckpts) s->ckpt_pool.push_back(std::move(c));
    s->ckpts.clear();
    s->ckpt_every = checkpoint_every;
    if (checkpoint_every > 0) {
        if (s->live_seg.n != (size_t)checkpoint_every * s->N) {
            s->drop_graphs();
            VBD_TRY(s->tape_alloc(s->live_seg, (size_t)checkpoint_every * s->N));
        }
        VBD_TRY(s->add_ckpt());
        CUDA_TRY(cudaStreamSynchronize(s->stream));
    }
    return VBD_OK;
}

int vbd_solver_backward(vbd_solver* s, const float* dl_dx, const float* dl_dv, int32_t adjoint_iterations,
                        float adjoint_rho, float* dl_dx0, float* dl_dv0, float* dl_dmu, float* dl_dlambda) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (s->ckpt_every <= 0 || s->ckpts.empty()) VBD_FAIL(VBD_ERR_STATE, "nothing recorded: call vbd_solver_record first");
    if (!dl_dx) VBD_FAIL(VBD_ERR_INVALID_ARG, "dl_dx is null");
    if (adjoint_iterations < 1) VBD_FAIL(VBD_ERR_INVALID_ARG, "adjoint_iterations must be >= 1");
    if (!(adjoint_rho >= 0.0f) || !(adjoint_rho < 1.0f)) VBD_FAIL(VBD_ERR_INVALID_ARG, "adjoint_rho must be in [0, 1)");
    DeviceScope scope(s->device);
    const int N = s->N, T = s->T, K = s->ckpt_every;
    const size_t b4 = sizeof(float4) * (size_t)N;
    // adjoint buffers; captured graphs bake their addresses, so any reallocation drops them
    for (auto* b : {&s->adj_lam, &s->adj_lam2, &s->adj_lpp, &s->adj_G, &s->adj_ax, &s->adj_av})
        if (b->n != (size_t)N) {
            s->drop_graphs();
            VBD_TRY(s->tape_alloc(*b, N));
        }
    if (s->adj_seg.n != (size_t)K * N) {
        s->drop_graphs();
        VBD_TRY(s->tape_alloc(s->adj_seg, (size_t)K * N));
    }
    if (s->adj_save.n != 6 * (size_t)N) VBD_TRY(s->tape_alloc(s->adj_save, 6 * (size_t)N));
    if (s->adj_gmu.n != (size_t)std::max(T, 1)) {
        s->drop_graphs();
        VBD_TRY(s->tape_alloc(s->adj_gmu, std::max(T, 1)));
        VBD_TRY(s->tape_alloc(s->adj_glam, std::max(T, 1)));
    }
    // keep the caller's state; the recompute overwrites it
    float4* live[6] = {s->x0.p, s->x1.p, s->pp.p, s->y.p, s->v.p, s->xprev.p};
    for (int k = 0; k < 6; ++k)
        CUDA_TRY(cudaMemcpyAsync(s->adj_save.p + (size_t)k * N, live[k], b4, cudaMemcpyDeviceToDevice, s->stream));
    CUDA_TRY(cudaMemsetAsync(s->adj_lam.p, 0, b4, s->stream));
    CUDA_TRY(cudaMemsetAsync(s->adj_lam2.p, 0, b4, s->stream));
    CUDA_TRY(cudaMemsetAsync(s->adj_lpp.p, 0, b4, s->stream));
    CUDA_TRY(cudaMemsetAsync(s->adj_gmu.p, 0, sizeof(float) * s->adj_gmu.n, s->stream));
    CUDA_TRY(cudaMemsetAsync(s->adj_glam.p, 0, sizeof(float) * s->adj_glam.n, s->stream));
    s->adj_cur = 0;
    VBD_TRY(s->upload3(dl_dx, s->adj_ax.p, nullptr));
    if (dl_dv)
        VBD_TRY(s->upload3(dl_dv, s->adj_av.p, nullptr));
    else
        CUDA_TRY(cudaMemsetAsync(s->adj_av.p, 0, b4, s->stream));
    const int nsteps = (int)s->tape.size();
    const int nseg = (nsteps + K - 1) / K;
    int rc = VBD_OK;
    for (int seg = nseg - 1; seg >= 0 && !rc; --seg) {
        const int t0 = seg * K, t1 = std::min(nsteps, t0 + K);
        // the newest segment's converged states were kept during the forward; older segments are
        // recomputed from their checkpoint (same graphs, hence the same bits)
        const bool live = seg == nseg - 1;
        float4* states = live ? s->live_seg.p : s->adj_seg.p;
        if (!live) {
            vbd::DBuf<float4>& ck = *s->ckpts[seg];
            CUDA_TRY(cudaMemcpyAsync(s->x0.p, ck.p, b4, cudaMemcpyDeviceToDevice, s->stream));
            CUDA_TRY(cudaMemcpyAsync(s->x1.p, ck.p, b4, cudaMemcpyDeviceToDevice, s->stream));
            CUDA_TRY(cudaMemcpyAsync(s->v.p, ck.p + N, b4, cudaMemcpyDeviceToDevice, s->stream));
            for (int t = t0; t < t1 && !rc; ++t) {
                rc = s->replay_substep(s->tape[t]);
                if (!rc && cudaMemcpyAsync(s->adj_seg.p + (size_t)(t - t0) * N, s->x0.p, b4,
                                           cudaMemcpyDeviceToDevice, s->stream) != cudaSuccess)
                    VBD_FAIL(VBD_ERR_CUDA, "segment copy failed");
            }
        }
        for (int t = t1 - 1; t >= t0 && !rc; --t)
            rc = s->adjoint_substep(s->tape[t], t - t0, states + (size_t)(t - t0) * N, adjoint_iterations,
                                    adjoint_rho, live ? 1 : 0);
    }
    if (!rc) {
        if (dl_dx0) rc = s->download3(s->adj_ax.p, dl_dx0);
        if (!rc && dl_dv0) rc = s->download3(s->adj_av.p, dl_dv0);
        if (!rc && dl_dmu && T > 0 &&
            cudaMemcpyAsync(dl_dmu, s->adj_gmu.p, sizeof(float) * T, cudaMemcpyDefault, s->stream) != cudaSuccess)
            rc = VBD_ERR_CUDA;
        if (!rc && dl_dlambda && T > 0 &&
            cudaMemcpyAsync(dl_dlambda, s->adj_glam.p, sizeof(float) * T, cudaMemcpyDefault, s->stream) != cudaSuccess)
            rc = VBD_ERR_CUDA;
    }
    for (int k = 0; k < 6; ++k)
        CUDA_TRY(cudaMemcpyAsync(live[k], s->adj_save.p + (size_t)k * N, b4, cudaMemcpyDeviceToDevice, s->stream));
    const int waits = s->finish();
    return rc ? rc : waits;
}

int vbd_solver_sync(vbd_solver* s) {
    vbd::clear_error();
    if (!s) VBD_FAIL(VBD_ERR_INVALID_ARG, "null solver handle");
    DeviceScope scope(s->device);
    return s->finish();
}

int vbd_solver_barrier_selftest(vbd_solver* s, int64_t spin_limit, int32_t* timed_out) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!timed_out || spin_limit < 1) VBD_FAIL(VBD_ERR_INVALID_ARG, "need timed_out and spin_limit >= 1");
    DeviceScope scope(s->device);
    const long long saved = s->spin_limit;
    s->spin_limit = spin_limit;
    // one arrival more than the grid has: the first barrier can never complete
    int rc = s->launch_persistent(0, 1.0f, false, 0.0f, false, false, false, 1.0f, nullptr, 1);
    s->spin_limit = saved;
    if (rc) return rc;
    CUDA_TRY(cudaStreamSynchronize(s->stream));
    unsigned long long t = 0;
    CUDA_TRY(cudaMemcpy(&t, s->status.p + vbd::ST_TIMEOUT, sizeof(t), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemsetAsync(s->status.p + vbd::ST_TIMEOUT, 0, sizeof(t), s->stream));
    *timed_out = t ? 1 : 0;
    return VBD_OK;
}

int vbd_solver_walk_selftest(vbd_solver* s, int64_t wait_us, int32_t* timed_out) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!timed_out || wait_us < 1 || wait_us > 1000000) VBD_FAIL(VBD_ERR_INVALID_ARG, "need timed_out and wait_us in 1..1000000");
    DeviceScope scope(s->device);
    return s->walk_selftest(wait_us, timed_out);
}

int vbd_solver_energy(vbd_solver* s, int32_t kind, float h, double* out) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!out) VBD_FAIL(VBD_ERR_INVALID_ARG, "out is null");
    if (kind < 0 || kind > 2) VBD_FAIL(VBD_ERR_INVALID_ARG, "unknown energy kind %d", kind);
    if (kind != VBD_ENERGY_ELASTIC_LOGJ && (!(h > 0.f) || !std::isfinite(h)))
        VBD_FAIL(VBD_ERR_INVALID_ARG, "h must be positive and finite");
    DeviceScope scope(s->device);
    if (kind == VBD_ENERGY_RESIDUAL) {
        if (s->nfree == 0) {
            *out = 0.0;
            return VBD_OK;
        }
        vbd::SweepParams p{s->x0.p,     nullptr, s->pp.p,    s->y.p, s->inc_off.p, s->inc_tet.p,
                           s->rec.p,    s->irec.p, s->crec.p, s->cmat.p, s->status.p, 0,
                           s->nfree,    (float)(1.0 / ((double)h * h)), 1.0f, 0, 0, 0, 0};
        const int L = std::max(4, s->lanes);
        const unsigned blocks = vbd::nblk((long long)s->nfree * L, 256);
        switch (L) {
            case 4: vbd::k_residual<4><<<blocks, 256, 0, s->stream>>>(p, s->partials.p); break;
            case 8: vbd::k_residual<8><<<blocks, 256, 0, s->stream>>>(p, s->partials.p); break;
            case 16: vbd::k_residual<16><<<blocks, 256, 0, s->stream>>>(p, s->partials.p); break;
            default: vbd::k_residual<32><<<blocks, 256, 0, s->stream>>>(p, s->partials.p); break;
        }
        VBD_TRY(s->check_launch());
        double r2 = 0.0;
        VBD_TRY(s->reduce_scalar(blocks, &r2));
        *out = std::sqrt(r2);
        return VBD_OK;
    }
    const long long work = std::max<long long>(kind == VBD_ENERGY_IP ? s->N : 0, s->T);
    const unsigned blocks = std::max(1u, std::min<unsigned>(vbd::nblk(work, 256), 4096u));
    const double inv_h2 = kind == VBD_ENERGY_IP ? 1.0 / ((double)h * h) : 0.0;
    vbd::k_energy<<<blocks, 256, 0, s->stream>>>(s->x0.p, s->y.p, s->rec.p, kind == VBD_ENERGY_IP ? s->N : 0, s->T,
                                                 kind, inv_h2, s->partials.p);
    VBD_TRY(s->check_launch());
    return s->reduce_scalar(blocks, out);
}

int vbd_solver_status(vbd_solver* s, int64_t* singular_skips, int32_t* nonfinite, int32_t reset) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    DeviceScope scope(s->device);
    const int waits = s->finish();
    unsigned long long h[vbd::ST_SLOTS];
    CUDA_TRY(cudaMemcpyAsync(h, s->status.p, sizeof(h), cudaMemcpyDeviceToHost, s->stream));
    CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (singular_skips) *singular_skips = (int64_t)h[vbd::ST_SINGULAR];
    if (nonfinite) *nonfinite = h[vbd::ST_NONFINITE] ? 1 : 0;
    if (reset) {
        CUDA_TRY(cudaMemsetAsync(s->status.p, 0, sizeof(h), s->stream));
        CUDA_TRY(cudaStreamSynchronize(s->stream));
    }
    return waits;
}

int vbd_solver_set_option(vbd_solver* s, int32_t option, int32_t value) {
    vbd::clear_error();
    if (!s) VBD_FAIL(VBD_ERR_INVALID_ARG, "null solver handle");
    DeviceScope scope(s->device);
    switch (option) {
        case VBD_OPT_LANES:
            if (value != 1 && value != 2 && value != 4 && value != 8 && value != 16 && value != 32)
                VBD_FAIL(VBD_ERR_INVALID_ARG, "lanes must be 1, 2, 4, 8, 16 or 32");
            s->lanes = value;
            s->lanes_auto = false;
            return s->prepare_cluster();
        case VBD_OPT_PREFETCH:
            if (value < 0 || value > 3) VBD_FAIL(VBD_ERR_INVALID_ARG, "prefetch must be 0, 1, 2 or 3");
            s->prefetch = value;
            s->prefetch_auto = false;
            return VBD_OK;
        case VBD_OPT_RECORD_CACHE:
            s->record_cache = value ? 1 : 0;
            s->record_cache_auto = false;
            return VBD_OK;
        case VBD_OPT_RECORD_PERSIST_MB:
            if (value < 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "persist megabytes must be >= 0");
            s->persist_mb = value;
            s->persist_auto = false;
            return VBD_OK;
        case VBD_OPT_ENERGY_EVERY:
            if (value < 0) VBD_FAIL(VBD_ERR_INVALID_ARG, "energy interval must be >= 0");
            s->energy_every = value;
            return VBD_OK;
        case VBD_OPT_PDL:
            s->pdl = value ? 1 : 0;
            return VBD_OK;
        case VBD_OPT_PERSISTENT:
            if (value < 0 || value > 2) VBD_FAIL(VBD_ERR_INVALID_ARG, "persistent must be 0, 1 or 2");
            if (value && s->semantics)
                VBD_FAIL(VBD_ERR_INVALID_ARG, "the persistent kernel runs the VBDsolver semantics only");
            if (value == 2 && s->ready) {
                const char* why = nullptr;
                if (!s->cluster_fit(&why)) VBD_FAIL(VBD_ERR_INVALID_ARG, "%s", why);
            }
            s->persistent = value;
            s->persistent_set = true;
            s->tile_walk = 0;
            for (auto* t : {&s->tset, &s->aset, &s->wset}) s->give_back(*t);
            return s->prepare_cluster();
        case VBD_OPT_CLUSTER_CTAS:
            if (value < 0 || value > 16) VBD_FAIL(VBD_ERR_INVALID_ARG, "cluster CTAs must be 0 (automatic) to 16");
            s->cluster_ctas_opt = value;
            return s->prepare_cluster();
        case VBD_OPT_CLUSTER_RESIDENT:
            s->cluster_resident = value ? 1 : 0;
            return s->prepare_cluster();
        case VBD_OPT_L2_PREFETCH:
            s->l2_prefetch = value ? 1 : 0;
            return VBD_OK;
        case VBD_OPT_SEMANTICS:
            if (value != 0 && value != 1) VBD_FAIL(VBD_ERR_INVALID_ARG, "semantics must be 0 (VBDsolver) or 1 (VBD_GPU_Solver)");
            if (value && s->persistent)
                VBD_FAIL(VBD_ERR_INVALID_ARG, "the persistent kernel runs the VBDsolver semantics only");
            if (value && s->ckpt_every > 0)
                VBD_FAIL(VBD_ERR_STATE, "recording for the adjoint is on; the adjoint needs the VBDsolver semantics");
            s->semantics = value;
            if (value && s->tset.started == 0) s->give_back(s->tset);  // made at init, and no step has run it
            if (value && s->ready && s->use_tile()) {
                VBD_TRY(s->ensure_tile(s->wset));
                CUDA_TRY(cudaStreamSynchronize(s->stream));
            }
            return VBD_OK;
        case VBD_OPT_ADJOINT_ALTERNATE:
            s->adj_alternate = value ? 1 : 0;
            return VBD_OK;
        case VBD_OPT_BLOCK:
            if (value != 64 && value != 128 && value != 256)
                VBD_FAIL(VBD_ERR_INVALID_ARG, "block must be 64, 128 or 256");
            s->block = value;
            return VBD_OK;
        case VBD_OPT_LAYOUT:
            if (value < 0 || value > 4) VBD_FAIL(VBD_ERR_INVALID_ARG, "layout must be 0, 1, 2, 3 or 4");
            if (value == 4 && s->ready && s->N > vbd::kPackedMaxVertices)
                VBD_FAIL(VBD_ERR_INVALID_ARG, "layout 4 holds vertex ids below 2^21; this mesh has %d vertices", s->N);
            s->layout = value;
            s->layout_auto = false;
            if (s->ready) {
                VBD_TRY(s->repack_stream());
                CUDA_TRY(cudaStreamSynchronize(s->stream));
            }
            return s->prepare_cluster();
        case VBD_OPT_GRAPH:
            s->use_graph = value ? 1 : 0;
            return VBD_OK;
        case VBD_OPT_KERNEL_TIMING:
            s->timing = value ? 1 : 0;
            return VBD_OK;
        default:
            VBD_FAIL(VBD_ERR_INVALID_ARG, "unknown option %d", option);
    }
}

int vbd_solver_get_option(vbd_solver* s, int32_t option, int32_t* value) {
    vbd::clear_error();
    if (!s || !value) VBD_FAIL(VBD_ERR_INVALID_ARG, "null argument");
    DeviceScope scope(s->device);
    switch (option) {
        case VBD_OPT_LANES: *value = s->lanes; return VBD_OK;
        case VBD_OPT_LAYOUT: *value = s->layout; return VBD_OK;
        case VBD_OPT_GRAPH: *value = s->use_graph; return VBD_OK;
        case VBD_OPT_KERNEL_TIMING: *value = s->timing; return VBD_OK;
        case VBD_OPT_PREFETCH: *value = s->eff_prefetch(); return VBD_OK;
        case VBD_OPT_PDL: *value = s->pdl; return VBD_OK;
        case VBD_OPT_BLOCK: *value = s->block; return VBD_OK;
        case VBD_OPT_PERSISTENT: *value = s->persistent; return VBD_OK;
        case VBD_OPT_CLUSTER_RESIDENT: *value = s->cluster_resident; return VBD_OK;
        case VBD_OPT_CLUSTER_CTAS:
            *value = s->cluster_ctas_opt > 0 || !s->ready ? s->cluster_ctas_opt
                                                           : s->cluster_auto(s->lanes < 4 ? 4 : s->lanes);
            return VBD_OK;
        case VBD_OPT_SEMANTICS: *value = s->semantics; return VBD_OK;
        case VBD_OPT_L2_PREFETCH: *value = s->l2_prefetch; return VBD_OK;
        case VBD_OPT_ADJOINT_ALTERNATE: *value = s->adj_alternate; return VBD_OK;
        case VBD_OPT_RECORD_CACHE: *value = s->record_cache; return VBD_OK;
        case VBD_OPT_RECORD_PERSIST_MB: *value = s->persist_mb; return VBD_OK;
        case VBD_OPT_ENERGY_EVERY: *value = s->energy_every; return VBD_OK;
        default: VBD_FAIL(VBD_ERR_INVALID_ARG, "unknown option %d", option);
    }
}

int vbd_solver_set_colour_lanes(vbd_solver* s, int32_t num_colours, const int32_t* lanes) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!lanes) {
        s->colour_lanes.clear();
        return VBD_OK;
    }
    if (num_colours != s->C) VBD_FAIL(VBD_ERR_INVALID_ARG, "need one lane count per colour (%d), got %d", s->C, num_colours);
    for (int c = 0; c < num_colours; ++c) {
        const int v = lanes[c];
        if (v != 1 && v != 2 && v != 4 && v != 8 && v != 16 && v != 32)
            VBD_FAIL(VBD_ERR_INVALID_ARG, "colour %d: lanes must be 1, 2, 4, 8, 16 or 32 (got %d)", c, v);
    }
    s->colour_lanes.assign(lanes, lanes + num_colours);
    return VBD_OK;
}

int vbd_solver_get_colour_lanes(vbd_solver* s, int32_t num_colours, int32_t* lanes) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!lanes || num_colours != s->C)
        VBD_FAIL(VBD_ERR_INVALID_ARG, "need an array of one entry per colour (%d)", s->C);
    for (int c = 0; c < num_colours; ++c) lanes[c] = s->lanes_of(c);
    return VBD_OK;
}

int vbd_solver_info(vbd_solver* s, int32_t* num_verts, int32_t* num_tets, int32_t* num_colours) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (num_verts) *num_verts = s->N;
    if (num_tets) *num_tets = s->T;
    if (num_colours) *num_colours = s->C;
    return VBD_OK;
}

int vbd_solver_kernel_time(vbd_solver* s, double* sweep_ms, int64_t* sweep_launches, double* sweep_bytes,
                           int32_t reset) {
    vbd::clear_error();
    if (!s) VBD_FAIL(VBD_ERR_INVALID_ARG, "null solver handle");
    DeviceScope scope(s->device);
    VBD_TRY(s->collect_timing());
    if (sweep_ms) *sweep_ms = s->timed_ms;
    if (sweep_launches) *sweep_launches = s->timed_launches;
    if (sweep_bytes) *sweep_bytes = s->timed_bytes;
    if (reset) {
        s->timed_ms = 0.0;
        s->timed_bytes = 0.0;
        s->timed_launches = 0;
    }
    return VBD_OK;
}

int vbd_solver_autotune(vbd_solver* s, float dt, int32_t iterations, int32_t repeats, int32_t* chosen) {
    vbd::clear_error();
    VBD_TRY(need_ready(s));
    if (!s->have_materials) VBD_FAIL(VBD_ERR_STATE, "materials not set");
    if (!(dt > 0.f) || iterations < 1 || repeats < 1) VBD_FAIL(VBD_ERR_INVALID_ARG, "need dt > 0, iterations >= 1, repeats >= 1");
    DeviceScope scope(s->device);
    // Save the state the candidate steps overwrite.
    const size_t b4 = sizeof(float4) * (size_t)s->N;
    vbd::DBuf<float4> save;
    VBD_TRY(save.alloc(6 * (size_t)s->N));
    float4* bufs[6] = {s->x0.p, s->x1.p, s->pp.p, s->y.p, s->v.p, s->xprev.p};
    for (int k = 0; k < 6; ++k)
        CUDA_TRY(cudaMemcpyAsync(save.p + (size_t)k * s->N, bufs[k], b4, cudaMemcpyDeviceToDevice, s->stream));
    unsigned long long st[vbd::ST_SLOTS];
    CUDA_TRY(cudaMemcpyAsync(st, s->status.p, sizeof(st), cudaMemcpyDeviceToHost, s->stream));
    VBD_TRY(s->finish());
    const int saved_timing = s->timing;
    const int saved_energy = s->energy_every;
    s->timing = 0;
    s->energy_every = 0;  // the candidate steps append no energies
    // The whole launch configuration a candidate sets.
    struct Cand {
        int lanes, layout, prefetch, pdl, block, persistent, cache, persist;
        std::vector<int> colour_lanes;  // empty = `lanes` for every colour
        int ctas = 0;                   // CTAs of the cluster walk (0 = automatic)
        int tile = 0;                   // the tile walk instead of the captured graph
    };
    const float g[3] = {0.f, 0.f, 0.f};
    cudaEvent_t e0, e1;
    CUDA_TRY(cudaEventCreate(&e0));
    CUDA_TRY(cudaEventCreate(&e1));
    auto apply = [&](const Cand& c) -> int {
        s->lanes = c.lanes;
        s->prefetch = c.prefetch;
        s->pdl = c.pdl;
        s->block = c.block;
        s->persistent = c.persistent;
        s->record_cache = c.cache;
        s->persist_mb = c.persist;
        s->colour_lanes = c.colour_lanes;
        s->cluster_ctas_opt = c.ctas;
        s->tile_walk = c.tile;
        if (s->layout != c.layout) {
            s->layout = c.layout;
            return s->repack_stream();
        }
        return VBD_OK;
    };
    // device time of `repeats` steps after one warm-up step (which captures the graph); the
    // simulation state is restored afterwards
    int reps = repeats;  // timed steps per candidate
    auto time_of = [&](const Cand& c, float* ms) -> int {
        VBD_TRY(apply(c));
        VBD_TRY(vbd_solver_step(s, dt, 1, iterations, g, 1, 0.9f));
        CUDA_TRY(cudaEventRecord(e0, s->stream));
        for (int r = 0; r < reps; ++r) VBD_TRY(vbd_solver_step(s, dt, 1, iterations, g, 1, 0.9f));
        CUDA_TRY(cudaEventRecord(e1, s->stream));
        CUDA_TRY(cudaEventSynchronize(e1));
        VBD_TRY(vbd_solver_sync(s));  // a persistent barrier that gave up makes the candidate fail
        CUDA_TRY(cudaEventElapsedTime(ms, e0, e1));
        for (int k = 0; k < 6; ++k)
            CUDA_TRY(cudaMemcpyAsync(bufs[k], save.p + (size_t)k * s->N, b4, cudaMemcpyDeviceToDevice, s->stream));
        return VBD_OK;
    };
    // Phase 1: uniform launch shapes (threads per vertex, record layout, prefetch, PDL, block).
    static const int uniform[][5] = {
        {8, 4, 2, 1, 64}, {8, 4, 3, 1, 64}, {8, 4, 1, 1, 64}, {8, 4, 1, 1, 128}, {4, 4, 1, 1, 128},
        {16, 4, 2, 1, 64}, {16, 4, 1, 1, 64}, {8, 4, 0, 1, 64},
        {8, 3, 1, 1, 64}, {8, 3, 1, 1, 128}, {4, 3, 1, 1, 128}, {16, 3, 1, 1, 64}, {8, 3, 0, 1, 64},
        {8, 3, 1, 0, 64}, {4, 2, 1, 1, 128}, {8, 2, 1, 1, 64},  {2, 2, 1, 1, 128}, {8, 1, 1, 1, 128},
        {8, 0, 1, 1, 128}, {4, 0, 1, 1, 128},
    };
    Cand best{s->lanes,      s->layout,       s->eff_prefetch(), s->pdl,          s->block,
              s->persistent, s->record_cache, s->persist_mb,     s->colour_lanes, s->cluster_ctas_opt, s->tile_walk};
    float best_ms = 1e30f;
    const int init_persist = s->persist_mb;  // the init-time record policy, for the factored candidates
    s->prefetch_auto = false;
    int rc = VBD_OK;
    for (const auto& u : uniform) {
        if (u[1] == 4 && s->N > vbd::kPackedMaxVertices) continue;
        Cand c{u[0], u[1], u[2], u[3], u[4], 0, u[1] >= 3 ? 1 : 0, u[1] >= 3 ? init_persist : 0, {}};
        float ms = 0.f;
        if ((rc = time_of(c, &ms))) break;
        if (ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    }
    // A later phase replaces the choice only when it is faster by more than 1% (timing noise).
    auto try_cand = [&](const Cand& c) -> int {
        float ms = 0.f;
        VBD_TRY(time_of(c, &ms));
        if (ms < 0.99f * best_ms) {
            best_ms = ms;
            best = c;
        }
        return VBD_OK;
    };
    // Phase 2: the factored records' L2 policy: plain loads, or the evict-first stream with an
    // evict-last prefix of 0, 32 or 64 MB.  (The 64^3 cube is fastest with the stream and 32 MB;
    // the 512-mesh batch, whose vertex state alone outgrows L2, with plain loads.)
    if (!rc && best.layout >= 3) {
        const Cand base = best;
        for (int pm : {-1, 0, 32, 64}) {
            Cand c = base;
            c.cache = pm < 0 ? 0 : 1;
            c.persist = pm < 0 ? 0 : pm;
            if (c.cache == base.cache && c.persist == base.persist) continue;
            if ((rc = try_cand(c))) break;
        }
    }
    // Phase 3: per-colour threads per vertex.  A colour's lane count moves the step by 1-3%, about
    // as much as the drift between timings taken a few seconds apart, so each candidate is timed
    // alternately with the incumbent, twice each over 2 x repeats steps, and replaces it when the
    // sums differ by more than 1%.  Greedy over the colours (lane counts 2, 4, 8, 16), two passes,
    // restarted from uniform lanes under each factored prefetch depth (which interacts with the
    // lane count: the 64^3 cube is fastest with the three-deep prefetch and lanes 4,8,4,8,4,4,8,8).
    auto beats = [&](const Cand& c, const Cand& inc, bool* better) -> int {
        float a = 0.f, b = 0.f, t = 0.f;
        for (int r = 0; r < 2; ++r) {
            VBD_TRY(time_of(inc, &t));
            a += t;
            VBD_TRY(time_of(c, &t));
            b += t;
        }
        *better = b < 0.99f * a;
        return VBD_OK;
    };
    if (!rc && s->semantics == 0 && s->C > 1) {
        reps = 2 * repeats;
        std::vector<int> depths{best.prefetch};
        if (best.layout >= 3)
            for (int pf : {1, 2, 3})
                if (pf != best.prefetch) depths.push_back(pf);
        Cand overall = best;
        float overall_ms = 1e30f;
        for (size_t d = 0; d < depths.size() && !rc; ++d) {
            Cand inc = best;
            inc.prefetch = depths[d];
            inc.colour_lanes.assign(s->C, inc.lanes);
            for (int pass = 0; pass < 2 && !rc; ++pass)
                for (int col = 0; col < s->C && !rc; ++col)
                    for (int L : {2, 4, 8, 16}) {
                        if (L == inc.colour_lanes[col]) continue;
                        Cand c = inc;
                        c.colour_lanes[col] = L;
                        bool better = false;
                        if ((rc = beats(c, inc, &better))) break;
                        if (better) inc = c;
                    }
            float ms = 0.f;
            if (!rc && !(rc = time_of(inc, &ms)) && ms < overall_ms) {
                overall_ms = ms;
                overall = inc;
            }
        }
        if (!rc) {
            bool better = false;
            if (!(rc = beats(overall, best, &better)) && better) best = overall;
        }
        if (!rc) rc = time_of(best, &best_ms);  // the incumbent at this phase's length, for phase 4
    }
    // VBD_GPU_Solver semantics: the tile walk against the captured graph
    if (!rc && s->semantics && s->tset.plan.P > 0) {
        Cand k = best;
        k.tile = 1;
        rc = try_cand(k);
    }
    // Phase 4: the whole step as one persistent colour-walking launch (uniform lanes, no per-colour
    // shape) against the captured graph.
    if (!rc && s->semantics == 0) {
        const Cand base = best;
        Cand c = base;
        c.persistent = 1;
        c.colour_lanes.clear();
        rc = try_cand(c);
        // the tile walk at each lane count it runs
        if (s->tset.plan.P > 0 && base.layout >= 3)
            for (int L : {4, 8, 16}) {
                if (rc) break;
                Cand k = base;
                k.persistent = 0;
                k.lanes = L;
                k.colour_lanes.clear();
                k.tile = 1;
                rc = try_cand(k);
            }
        // the cluster walk, for a mesh whose positions fit in one CTA's shared memory: each lane count
        // with either factored layout (the stored det M of layout 3 saves a division per record,
        // which counts where the records stay in L2)
        const char* why = nullptr;
        if (!rc && base.layout >= 3 && s->cluster_fit(&why)) {
            for (int lay : {3, 4}) {
                if (lay == 4 && s->N > vbd::kPackedMaxVertices) continue;
                for (int L : {4, 8, 16, 32}) {
                    Cand k = base;
                    k.persistent = 2;
                    k.tile = 0;
                    k.lanes = L;
                    k.layout = lay;
                    k.colour_lanes.clear();
                    if ((rc = try_cand(k))) break;
                }
                if (rc) break;
            }
            // the chosen walk's CTA count around the automatic one (fewer CTAs send fewer copies of
            // each update; more take fewer rounds)
            if (!rc && best.persistent == 2 && best.ctas == 0) {
                const int a = s->cluster_auto(best.lanes < 4 ? 4 : best.lanes);
                const Cand walk = best;
                for (int n : {a / 2, (3 * a) / 4, a + (a + 1) / 2, 16}) {
                    n = std::min(16, std::max(1, n));
                    if (n == a) continue;
                    Cand k = walk;
                    k.ctas = n;
                    if ((rc = try_cand(k))) break;
                }
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    for (int k = 0; k < 6; ++k)
        CUDA_TRY(cudaMemcpyAsync(bufs[k], save.p + (size_t)k * s->N, b4, cudaMemcpyDeviceToDevice, s->stream));
    CUDA_TRY(cudaMemcpyAsync(s->status.p, st, sizeof(st), cudaMemcpyHostToDevice, s->stream));
    s->timing = saved_timing;
    s->energy_every = saved_energy;
    s->record_cache_auto = s->persist_auto = false;  // the tuned policy stays for this mesh
    const int arc = apply(best);
    CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (rc) return rc;
    if (arc) return arc;
    if (chosen) {
        chosen[0] = best.lanes;
        chosen[1] = best.layout;
        chosen[2] = best.prefetch;
        chosen[3] = best.pdl;
        chosen[4] = best.block;
    }
    return VBD_OK;
}

int vbd_solver_kernel_launches(vbd_solver* s, int64_t* launches) {
    vbd::clear_error();
    if (!s || !launches) VBD_FAIL(VBD_ERR_INVALID_ARG, "null argument");
    *launches = s->launches;
    return VBD_OK;
}

}  // extern "C"
