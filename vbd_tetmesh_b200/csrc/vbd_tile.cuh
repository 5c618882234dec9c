// The tile walk: all iterations of a sub-step (or of its adjoint solve) in ONE launch: a cooperative one, the
// default from kTileMinVertices free vertices until a tile no longer fits in an SM's shared memory, or one cluster
// (VBD_OPT_PERSISTENT 2).
//
// Per-colour launches pay a kernel boundary per colour (2.3 us and up) and start each colour's
// record stream only then.  Here the free vertices are cut into one spatial tile per CTA (one CTA per
// SM; vbd_tile_plan.cpp) and the colours are separated by data instead of by launches:
//   * a tile keeps the positions of its own vertices and of the neighbours it reads (its ghosts) in
//     shared memory, so every neighbour gather is a shared-memory load;
//   * a vertex that other tiles read is published as ONE 16-byte word, {x~, tag}, with a relaxed
//     128-bit store (single-copy atomic); after sweeping colour c a tile polls the words of its
//     colour-c ghosts until they carry the iteration's tag.  Data and flag travel together, so there
//     are no fences, no flags and no grid barrier: a tile waits for its neighbours only.  One
//     __syncthreads per colour separates the colours inside the tile;
//   * the element records are re-ordered into the exact order each warp reads them (chunks of 64
//     incidences, two per thread, field by field), and each warp streams its own chunks through a
//     private shared-memory ring with asynchronous copies.  Records never change during the
//     sweeps, so the ring runs ahead across colours and iterations: the stream does not stop while
//     a tile waits for its neighbours.
// Why overwriting a published word is safe: words alternate by tag parity, and the owner of v can be
// two iterations ahead of a reader of v only if it has received, from that reader, a value computed
// after the reader took v's word (every reader of v owns a free neighbour of v, and v's own sweep
// gathers that neighbour).
//
// What bounds it (one B200): small tiles by one exchange through L2 (a word takes 480 to 1,050 cycles from
// one SM to another's poll, 885 on average) plus one vertex's chain per colour (about 1,000 cycles from
// the barrier to its publication): 1.3 to 1.8 us a colour against 2.3 to 3.3 us a launch.  Large tiles by
// issue and the chunk stream: 64^3 cube 3.15 against 4.17 ms a step of 400 colours, 4.1 TB/s of DRAM
// traffic.  VBD_GPU_Solver semantics: 425-vertex beam 2.6 against 4.6 us a colour, 32^3 cube 6.6 against 9.6.
// Same bits as the per-colour launches at the same lane count L: the partial sum of lane l takes
// records l, l + L, ... in order, and lanes are added in the order of group_reduce.  A thread holds
// the sums of lanes t and t + L/2 (group_reduce's first addition), so a vertex takes L/2 threads:
// half the warps' shuffles and idle solve lanes of the per-colour kernel.  Or (STACK, and always with
// VBD_GPU_Solver semantics) it takes records t and t + L of one lane, one after the other: L threads, half
// the rounds.
#pragma once

#include <type_traits>

#include "vbd_cluster.cuh"
#include "vbd_tile_plan.h"

namespace vbd {

struct TileParams {
    const float4* chunk;        // record chunks, kTileChunkBytes each
    const TileHead* head;
    const int* lid;
    const TileGroup* groups;
    const int* wcol;            // [P][warps][C + 1]: first group of each warp and colour
    const int* ghost;           // [P][C + 1]
    const int2* wstream;        // [P][warps]
    float4* words;              // exchanged words: [parity][n] x~, then [parity][n] blended, word_stride apart
    int word_stride;
    unsigned long long* arrived;        // and after it the nanoseconds after which a wait gives up (kTileWaitNs)
    unsigned long long arrived_target;  // *arrived once every CTA of this launch has started
    unsigned long long* status;
    const float* omega;         // Chebyshev weight of each iteration (1 = no blend)
    unsigned tag;               // iteration k publishes tag + k; unused by any earlier launch
    int n, nfree, ncol, k0, k1; // iterations [k0, k1) of the schedule
    int ring, max_local, max_ids, max_groups, max_rounds;
    int two;                    // both position buffers in shared memory
    float keep;                 // W = 16: share of the chunk stream kept in L2 (evict-last; the rest evict-first); 1 = plain
    int ring_chunks;            // chunks of all the CTA's rings
    int resident;               // W = 8: the rings hold every chunk of the tile, copied once
    // cluster exchange: where each own vertex's results go, [own vertex] first target, then the targets
    // (CTA rank << 16 | local id there)
    const int* target_off;      // [P][max_own + 1]
    const int* target;          // [P][max_target]
    int max_own, max_target;
    float dtsr;
    int keep_pp;
    // forward: positions start and end in x0
    float4* x0;
    float4* x1;
    float4* pp;
    float4* y;
    float4* v;
    float4* xprev;
    int predict, finish, from_inertia;
    float h, hgx, hgy, hgz;
    // adjoint: converged positions X, right-hand side G, adjoint in / out, pre-sweep adjoint in pp
    const float4* X;
    const float4* G;
    const float4* lam_in;
    float4* lam_out;
};

// Dynamic shared memory of a CTA: the rings, the local vectors (`vectors` of them, one entry more each),
// the groups, the internal ids of the own vertices and ghosts, the first ghost of each colour, the first
// group of each warp and colour, and (cluster exchange) the own vertices' targets.
inline size_t tile_smem(int warps, int ring_chunks, int chunk_bytes, const TilePlan& p, int ncol, int vectors, bool cluster) {
    return (size_t)ring_chunks * chunk_bytes + 16u * (size_t)(p.max_local + 1) * vectors +
           sizeof(TileGroup) * (size_t)p.max_groups + 4u * (size_t)p.max_ids + 4u * (size_t)(warps + 1) * (ncol + 1) +
           (cluster ? 4u * (size_t)(p.max_own + 1 + p.max_target) : 0u);
}
constexpr int kTileMaxColours = 64;  // of a cluster exchange: one mbarrier per colour

// The 128-bit words: one relaxed, single-copy-atomic access each.
__device__ __forceinline__ void word_store(float4* p, float x, float y, float z, unsigned tag) {
    const unsigned long long a = ((unsigned long long)__float_as_uint(y) << 32) | __float_as_uint(x);
    const unsigned long long b = ((unsigned long long)tag << 32) | __float_as_uint(z);
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(a),
                 "l"(b)
                 : "memory");
}
__device__ __forceinline__ float4 word_load(const float4* p) {
    unsigned long long a, b;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
    return make_float4(__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)), __uint_as_float((unsigned)b),
                       __uint_as_float((unsigned)(b >> 32)));
}

// Gives up a wait: another wait already gave up, or this one has lasted arrived[1] nanoseconds with every CTA of
// the launch running (a CTA that cannot start while another program's kernel holds its SM is
// waited for up to kTileStartNs).  The walk then sweeps on to the end of the iteration with what it has, so
// that no thread leaves a barrier, a shuffle or a copy that the others wait for.
constexpr unsigned long long kTileWaitNs = 2000000000ull;
constexpr unsigned long long kTileStartNs = 60000000000ull;
constexpr unsigned long long kTileDrainNs = 20000000ull;  // for the copies under way of a walk that gave up
struct TileClock {
    unsigned long long first = 0, last = 0;
};
__device__ __noinline__ bool tile_give_up(unsigned long long* status, unsigned long long* arrived,
                                          unsigned long long target, TileClock& c) {
    if (*reinterpret_cast<volatile unsigned long long*>(status + ST_WALK_TIMEOUT) != 0ull) return true;
    const unsigned long long now = global_ns();
    if (c.first == 0) c.first = c.last = now;
    if (now - c.last <= arrived[1]) return false;
    if (*reinterpret_cast<volatile unsigned long long*>(arrived) < target && now - c.first <= kTileStartNs) {
        c.last = now;
        return false;
    }
    atomicOr(reinterpret_cast<unsigned int*>(status + ST_WALK_TIMEOUT), 1u);
    return true;
}

// Waits for word w to carry `tag` and stores its vector to *dst.
__device__ __forceinline__ bool tile_spin(const TileParams& p, const float4* w, unsigned tag, float4* dst) {
    TileClock clk;
    for (unsigned i = 1;; ++i) {
        const float4 v = word_load(w);
        if (__float_as_uint(v.w) == tag) {
            *dst = make_float4(v.x, v.y, v.z, 0.f);
            return true;
        }
        if ((i & 255u) == 0u && tile_give_up(p.status, p.arrived, p.arrived_target, clk)) return false;
    }
}
// The same with a first look already taken.
__device__ __forceinline__ bool tile_take(const TileParams& p, float4 v, const float4* w, unsigned tag, float4* dst) {
    if (__float_as_uint(v.w) != tag) return tile_spin(p, w, tag, dst);
    *dst = make_float4(v.x, v.y, v.z, 0.f);
    return true;
}

// A warp's ring of record chunks.  W = 8 fills it by its own lanes with 16-byte asynchronous copies, one
// commit group per chunk (empty ones once the walk's chunks are all under way).
struct TileRing {
    int first, end, next;  // the warp's chunks [first, end), read cyclically; next one to copy
    int left;              // chunks still to copy
    int slot;              // slot of the next chunk to sweep
};

template <int kBytes>
__device__ __forceinline__ void ring_issue(const TileParams& p, TileRing& r, unsigned buf, int slot, int lane) {
    constexpr int kFull = kBytes / 512;
    static_assert(kBytes == kFull * 512 + 256, "16-byte pieces, the last of half the lanes");
    if (r.left > 0) {
        const char* src = reinterpret_cast<const char*>(p.chunk) + (size_t)r.next * kBytes + 16 * lane;
        const unsigned dst = buf + (unsigned)(slot * kBytes + 16 * lane);
#pragma unroll
        for (int i = 0; i < kFull; ++i)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512 * i), "l"(src + 512 * i) : "memory");
        if (lane < 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512 * kFull), "l"(src + 512 * kFull) : "memory");
        --r.left;
        if (++r.next == r.end) r.next = r.first;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// The same as one bulk copy, completing on the slot's mbarrier (W = 16).
template <unsigned kBytes, bool HINT>
__device__ __forceinline__ void ring_issue_bulk(const TileParams& p, TileRing& r, unsigned buf, unsigned bar, int slot,
                                                int lane, unsigned long long policy) {
    if (r.left <= 0) return;
    if (lane == 0) {
        mbar_expect(bar + 8u * slot, kBytes);
        const char* src = reinterpret_cast<const char*>(p.chunk) + (size_t)r.next * kBytes;
        const unsigned dst = buf + (unsigned)(slot * kBytes);
        if constexpr (HINT)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
                "l"(src), "r"(kBytes), "r"(bar + 8u * slot), "l"(policy)
                : "memory");
        else
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                         "r"(kBytes), "r"(bar + 8u * slot)
                         : "memory");
    }
    --r.left;
    if (++r.next == r.end) r.next = r.first;
}
__device__ __forceinline__ bool ring_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// The same without a wait of its own.
__device__ __forceinline__ bool ring_test(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Waits for a slot's chunk; the same answer for the whole warp.  The repeated tries stand in a function of their
// own: inlined they cost the sweep loop registers (a step of 50 iterations of the 64^3 cube 2.98 ms against 3.17 with 4
// lanes, 3.10 against 3.27 with 8; 128 meshes 1.36 against 1.44, 32^3 1.12 against 1.14, VBD_GPU_Solver semantics 32^3
// 2.56 against 2.66).
__device__ __noinline__ bool ring_wait_again(unsigned bar, unsigned parity, unsigned long long* status,
                                             unsigned long long* arrived, unsigned long long target) {
    TileClock clk;
    for (unsigned i = 1;; ++i) {
        if (ring_try(bar, parity)) return true;
        if ((i & 255u) == 0u && tile_give_up(status, arrived, target, clk)) return false;
    }
}
__device__ __forceinline__ bool ring_wait_bulk(const TileParams& p, unsigned bar, unsigned parity) {
    bool done = ring_try(bar, parity);
    if (!done) done = ring_wait_again(bar, parity, p.status, p.arrived, p.arrived_target);
    return __all_sync(0xffffffffu, done);
}
// Waits until at most `pending` of the newest commit groups are outstanding.
template <int N> __device__ __forceinline__ void ring_wait_for() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ring_wait(int pending) {
    switch (pending) {
        case 0: ring_wait_for<0>(); break;
        case 1: ring_wait_for<1>(); break;
        case 2: ring_wait_for<2>(); break;
        case 3: ring_wait_for<3>(); break;
        default: ring_wait_for<4>(); break;
    }
    __syncwarp();
}

// Two FP32 values in one 64-bit register pair, for the two-wide FP32 instructions (each half rounds as
// the scalar instruction does).
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float f2_lo(F2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float f2_hi(F2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 neg2(F2 a) { return mul2(a, f2(-1.f, -1.f)); }
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(b, f2(-1.f, -1.f), a); }
// a0 b0 + a1 b1 + a2 b2, rounded as nvcc contracts that expression.
__device__ __forceinline__ F2 dot2(F2 a0, F2 b0, F2 a1, F2 b1, F2 a2, F2 b2) {
    return fma2(a2, b2, fma2(a0, b0, mul2(a1, b1)));
}
// a b - c d, rounded as nvcc contracts it; given nc = -c it is one instruction shorter.
__device__ __forceinline__ F2 cross2(F2 a, F2 b, F2 c, F2 d) { return fma2(a, b, neg2(mul2(c, d))); }
__device__ __forceinline__ F2 cross2n(F2 a, F2 b, F2 nc, F2 d) { return fma2(a, b, mul2(nc, d)); }

__device__ __forceinline__ void load_if(bool pred, const float4* p, float4& v) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %5, 0;\n @q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
                 : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
                 : "l"(p), "r"((int)pred)
                 : "memory");
}
__device__ __forceinline__ void load_if(bool pred, const float* p, float& v) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.global.f32 %0, [%1];\n}"
                 : "+f"(v)
                 : "l"(p), "r"((int)pred)
                 : "memory");
}

// One thread's two records of a chunk: lanes t (first half of each pair) and t + L/2 of its vertex.  The
// fields are read where they are used (they would hold 18 registers).
struct TilePair {
    const char* buf;
    int lane;
    __device__ __forceinline__ ulonglong2 two(int k) const { return reinterpret_cast<const ulonglong2*>(buf)[32 * k + lane]; }
    __device__ __forceinline__ ulonglong2 s01() const { return two(0); }
    __device__ __forceinline__ ulonglong2 s2w0() const { return two(1); }
    __device__ __forceinline__ ulonglong2 w12() const { return two(2); }
    __device__ __forceinline__ ulonglong2 ab() const { return two(3); }
    // neighbours: {nb0 | nb1 << 16, nb2 | valid << 16} of the first record, then of the second
    __device__ __forceinline__ int4 ids() const { return reinterpret_cast<const int4*>(buf)[128 + lane]; }
    __device__ __forceinline__ F2 detm() const { return reinterpret_cast<const F2*>(buf + 160 * 16)[lane]; }
};

// What a thread's two records add up to: the sums of two lanes of one vertex (Acc2), or of one lane that takes
// the first record, then the second (Acc1).
struct Acc2 {
    F2 h00, h01, h02, h11, h12, h22, g0, g1, g2;
    __device__ __forceinline__ void zero() { h00 = h01 = h02 = h11 = h12 = h22 = g0 = g1 = g2 = 0ull; }
    __device__ __forceinline__ void grad(int i, F2 x) {
        F2& g = i == 0 ? g0 : i == 1 ? g1 : g2;
        g = add2(g, x);
    }
    __device__ __forceinline__ void diag(int i, F2 x) {
        F2& h = i == 0 ? h00 : i == 1 ? h11 : h22;
        h = add2(h, x);
    }
    __device__ __forceinline__ void off(int i, F2 x, F2 y) {
        F2& h = i == 0 ? h01 : i == 1 ? h02 : h12;
        h = fma2(x, y, h);
    }
    __device__ __forceinline__ Acc sum() const {
        Acc r;
        r.h00 = f2_lo(h00) + f2_hi(h00);
        r.h01 = f2_lo(h01) + f2_hi(h01);
        r.h02 = f2_lo(h02) + f2_hi(h02);
        r.h11 = f2_lo(h11) + f2_hi(h11);
        r.h12 = f2_lo(h12) + f2_hi(h12);
        r.h22 = f2_lo(h22) + f2_hi(h22);
        r.g0 = f2_lo(g0) + f2_hi(g0);
        r.g1 = f2_lo(g1) + f2_hi(g1);
        r.g2 = f2_lo(g2) + f2_hi(g2);
        return r;
    }
};
struct Acc1 {
    float d[3], o[3], g[3];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 3; ++i) d[i] = o[i] = g[i] = 0.f;
    }
    __device__ __forceinline__ void grad(int i, F2 x) { g[i] = __fadd_rn(__fadd_rn(g[i], f2_lo(x)), f2_hi(x)); }
    __device__ __forceinline__ void diag(int i, F2 x) { d[i] = __fadd_rn(__fadd_rn(d[i], f2_lo(x)), f2_hi(x)); }
    __device__ __forceinline__ void off(int i, F2 x, F2 y) {
        o[i] = fmaf(f2_hi(x), f2_hi(y), fmaf(f2_lo(x), f2_lo(y), o[i]));
    }
    __device__ __forceinline__ Acc sum() const {
        Acc r;
        r.h00 = d[0], r.h11 = d[1], r.h22 = d[2];
        r.h01 = o[0], r.h02 = o[1], r.h12 = o[2];
        r.g0 = g[0], r.g1 = g[1], r.g2 = g[2];
        return r;
    }
};

// The geometry of two records: edge vectors d_k and the columns c_k of cof(D) (c_0 = d_1 x d_2, ...).
struct Geom2 {
    F2 d[3][3], c[3][3];
};
__device__ __forceinline__ void tile_edges(const int4 id, float4 xi, const float4* X, Geom2& q) {
    const unsigned a0 = id.x, a1 = id.y, b0 = id.z, b1 = id.w;
    const float4 pa[3] = {X[a0 & 0xffffu], X[a0 >> 16], X[a1 & 0xffffu]};
    const float4 pb[3] = {X[b0 & 0xffffu], X[b0 >> 16], X[b1 & 0xffffu]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        q.d[k][0] = f2(pa[k].x - xi.x, pb[k].x - xi.x);
        q.d[k][1] = f2(pa[k].y - xi.y, pb[k].y - xi.y);
        q.d[k][2] = f2(pa[k].z - xi.z, pb[k].z - xi.z);
    }
    // the negated d_1 and d_2 serve all three columns
    const F2 n1[3] = {neg2(q.d[1][0]), neg2(q.d[1][1]), neg2(q.d[1][2])};
    const F2 n2[3] = {neg2(q.d[2][0]), neg2(q.d[2][1]), neg2(q.d[2][2])};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
        q.c[0][i] = cross2n(q.d[1][i1], q.d[2][i2], n1[i2], q.d[2][i1]);
        q.c[1][i] = cross2n(q.d[2][i1], q.d[0][i2], n2[i2], q.d[0][i1]);
        q.c[2][i] = cross2n(q.d[0][i1], q.d[1][i2], q.d[0][i2], n1[i1]);
    }
}

// fact_contrib for two records at once, operation for operation as nvcc contracts it, so that each
// half has fact_contrib's bits.  A record that is only padding has zero fields and the vertex itself
// as its neighbours: d = 0, and it adds zero to every sum.
template <class Sums>
__device__ __forceinline__ void tile_contrib(const TilePair& r, const int4 id, float4 xi, const float4* X, Sums& acc) {
    Geom2 q;
    tile_edges(id, xi, X, q);
    const ulonglong2 ab = r.ab();
    const F2 bj = mul2(ab.y, fma2(dot2(q.d[0][0], q.c[0][0], q.d[0][1], q.c[0][1], q.d[0][2], q.c[0][2]), r.detm(),
                                  f2(-1.f, -1.f)));
    const ulonglong2 sw = r.s2w0(), w12 = r.w12(), s01 = r.s01();
    F2 C[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        C[i] = dot2(q.c[0][i], sw.y, q.c[1][i], w12.x, q.c[2][i], w12.y);
        const F2 Fq = dot2(q.d[0][i], s01.x, q.d[1][i], s01.y, q.d[2][i], sw.x);
        acc.grad(i, fma2(ab.x, sub2(Fq, C[i]), mul2(bj, C[i])));
    }
    const F2 am = mul2(ab.x, neg2(add2(add2(s01.x, s01.y), sw.x)));
    const F2 b0 = mul2(ab.y, C[0]), b1 = mul2(ab.y, C[1]), b2 = mul2(ab.y, C[2]);
    acc.diag(0, fma2(b0, C[0], am));
    acc.off(0, b0, C[1]);
    acc.off(1, b0, C[2]);
    acc.diag(1, fma2(b1, C[1], am));
    acc.off(2, b1, C[2]);
    acc.diag(2, fma2(b2, C[2], am));
}

// fact_adjoint for two records at once.  A padding record reads the zero entry `zero` of L.
__device__ __forceinline__ void tile_lambdas(const int4 id, const float4* L, int zero, F2 m[3][3]) {
    const unsigned a0 = id.x, a1 = id.y, b0 = id.z, b1 = id.w;
    const bool va = a1 >> 16, vb = b1 >> 16;
    const float4 la[3] = {L[va ? a0 & 0xffffu : zero], L[va ? a0 >> 16 : zero], L[va ? a1 & 0xffffu : zero]};
    const float4 lb[3] = {L[vb ? b0 & 0xffffu : zero], L[vb ? b0 >> 16 : zero], L[vb ? b1 & 0xffffu : zero]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        m[k][0] = f2(la[k].x, lb[k].x);
        m[k][1] = f2(la[k].y, lb[k].y);
        m[k][2] = f2(la[k].z, lb[k].z);
    }
}

template <class Sums>
__device__ __forceinline__ void tile_adjoint(const TilePair& r, const int4 id, float4 xi, const float4* X,
                                             const float4* L, int zero, Sums& acc) {
    Geom2 q;
    tile_edges(id, xi, X, q);
    F2 m[3][3];
    tile_lambdas(id, L, zero, m);
    const F2 detm = r.detm();
    const F2 jm1 = fma2(dot2(q.d[0][0], q.c[0][0], q.d[0][1], q.c[0][1], q.d[0][2], q.c[0][2]), detm, f2(-1.f, -1.f));
    F2 dJ;
    {
        const F2 t0 = dot2(q.c[0][0], m[0][0], q.c[0][1], m[0][1], q.c[0][2], m[0][2]);
        const F2 t1 = dot2(q.c[1][0], m[1][0], q.c[1][1], m[1][1], q.c[1][2], m[1][2]);
        const F2 t2 = dot2(q.c[2][0], m[2][0], q.c[2][1], m[2][1], q.c[2][2], m[2][2]);
        dJ = mul2(detm, add2(add2(t0, t1), t2));
    }
    ulonglong2 sw = r.s2w0(), w12 = r.w12();
    F2 C[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) C[i] = dot2(q.c[0][i], sw.y, q.c[1][i], w12.x, q.c[2][i], w12.y);
    const ulonglong2 ab = r.ab(), s01 = r.s01();
    {
        const F2 am = mul2(ab.x, neg2(add2(add2(s01.x, s01.y), sw.x)));
        const F2 b0 = mul2(ab.y, C[0]), b1 = mul2(ab.y, C[1]), b2 = mul2(ab.y, C[2]);
        acc.diag(0, fma2(b0, C[0], am));
        acc.off(0, b0, C[1]);
        acc.off(1, b0, C[2]);
        acc.diag(1, fma2(b1, C[1], am));
        acc.off(2, b1, C[2]);
        acc.diag(2, fma2(b2, C[2], am));
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
        // lam_1 x d_2 + d_1 x lam_2 and cyclic
        const F2 e0 = add2(cross2(m[1][i1], q.d[2][i2], m[1][i2], q.d[2][i1]), cross2(q.d[1][i1], m[2][i2], q.d[1][i2], m[2][i1]));
        const F2 e1 = add2(cross2(m[2][i1], q.d[0][i2], m[2][i2], q.d[0][i1]), cross2(q.d[2][i1], m[0][i2], q.d[2][i2], m[0][i1]));
        const F2 e2 = add2(cross2(m[0][i1], q.d[1][i2], m[0][i2], q.d[1][i1]), cross2(q.d[0][i1], m[1][i2], q.d[0][i2], m[1][i1]));
        const F2 dF = dot2(m[0][i], s01.x, m[1][i], s01.y, m[2][i], sw.x);
        const F2 dC = dot2(e0, sw.y, e1, w12.x, e2, w12.y);
        acc.grad(i, fma2(ab.x, sub2(dF, dC), mul2(ab.y, fma2(dJ, C[i], mul2(jm1, dC)))));
    }
}

// The corotated element of VBD_GPU_Solver semantics (corot_block) for two records at once: every
// operation rounds as nvcc contracts corot_block, so that the sums have k_sweep_wrapper's bits.  The
// minors of the row-0 determinant are the cofactors of row 0 (the middle one negated); the middle one,
// which appears with both signs, is a difference of two rounded products.
// Padding repeats a record of its vertex and is not added.
__device__ __forceinline__ float cross1(float a, float b, float c, float d) { return fmaf(a, b, -__fmul_rn(c, d)); }
__device__ __forceinline__ float dot1(float a0, float b0, float a1, float b1, float a2, float b2) {
    return fmaf(a2, b2, fmaf(a0, b0, __fmul_rn(a1, b1)));
}
// The difference of two products, each rounded: ptxas contracts mul.rn.f32x2 into add.rn.f32x2, which the scalar
// instruction prevents.
__device__ __forceinline__ F2 sub_rn(F2 a, F2 b) {
    return f2(__fsub_rn(f2_lo(a), f2_lo(b)), __fsub_rn(f2_hi(a), f2_hi(b)));
}
struct CorotSums {
    float h[9], f[3];
};
__device__ __forceinline__ void tile_corot(const char* buf, int lane, const float4* X, CorotSums& acc) {
    auto two = [&](int k) { return reinterpret_cast<const ulonglong2*>(buf)[32 * k + lane]; };
    const int4 id = reinterpret_cast<const int4*>(buf)[224 + lane];
    F2 F[3][3];
    {
        const unsigned a0 = id.x, a1 = id.y, b0 = id.z, b1 = id.w;
        const float4 pa = X[a0 & 0xffffu], pb = X[b0 & 0xffffu];
        const float4 qa[3] = {X[a0 >> 16], X[a1 & 0xffffu], X[(a1 >> 16) & 0x7fffu]};
        const float4 qb[3] = {X[b0 >> 16], X[b1 & 0xffffu], X[(b1 >> 16) & 0x7fffu]};
        F2 d[3][3];  // [axis][column]
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d[0][k] = f2(qa[k].x - pa.x, qb[k].x - pb.x);
            d[1][k] = f2(qa[k].y - pa.y, qb[k].y - pb.y);
            d[2][k] = f2(qa[k].z - pa.z, qb[k].z - pb.z);
        }
        const ulonglong2 m01 = two(0), m23 = two(1), m45 = two(2), m67 = two(3);
        const F2 m8 = two(4).x;
        const F2 M[3][3] = {{m01.x, m01.y, m23.x}, {m23.y, m45.x, m45.y}, {m67.x, m67.y, m8}};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) F[a][b] = dot2(d[a][0], M[0][b], d[a][1], M[1][b], d[a][2], M[2][b]);
    }
    F2 R[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) R[a][b] = F[a][b];
    const F2 half = f2(0.5f, 0.5f);
#pragma unroll 1
    for (int it = 0; it < 5; ++it) {
        F2 C[3][3];
        const F2 n1[3] = {neg2(R[1][0]), neg2(R[1][1]), neg2(R[1][2])};
        const F2 n2[3] = {neg2(R[2][0]), neg2(R[2][1]), neg2(R[2][2])};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
            C[0][i] = i == 1 ? sub_rn(mul2(R[1][2], R[2][0]), mul2(R[1][0], R[2][2]))
                             : cross2n(R[1][i1], R[2][i2], n1[i2], R[2][i1]);
            C[1][i] = cross2n(R[2][i1], R[0][i2], n2[i2], R[0][i1]);
            C[2][i] = cross2n(R[0][i1], R[1][i2], R[0][i2], n1[i1]);
        }
        const F2 det = dot2(R[0][0], C[0][0], R[0][1], C[0][1], R[0][2], C[0][2]);
        const float da = f2_lo(det), db = f2_hi(det);
        const bool stop_a = fabsf(da) < 1e-8f, stop_b = fabsf(db) < 1e-8f;
        const F2 inv = f2(__frcp_rn(da), __frcp_rn(db));
        if (!stop_a && !stop_b) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) R[a][b] = mul2(half, fma2(C[a][b], inv, R[a][b]));
        } else {  // a record whose steps have ended keeps its R (and ends here again next time)
            if (stop_a && stop_b) break;
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const F2 n = mul2(half, fma2(C[a][b], inv, R[a][b]));
                    R[a][b] = f2(stop_a ? f2_lo(R[a][b]) : f2_lo(n), stop_b ? f2_hi(R[a][b]) : f2_hi(n));
                }
        }
    }
    F2 tr = 0ull;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) tr = fma2(R[a][b], F[a][b], tr);
    tr = add2(tr, f2(-3.f, -3.f));
    const ulonglong2 q01 = two(5), qv = two(6);
    const F2 q0 = two(4).y, q1 = q01.x, q2 = q01.y, vol = qv.x, m2 = qv.y;  // m2 = 2 mu
    const F2 lam = reinterpret_cast<const F2*>(buf + 256 * 16)[lane];
    const F2 lt = mul2(lam, tr), nvol = neg2(vol), diag = dot2(q0, q0, q1, q1, q2, q2);
    F2 RQ[3], lr[3];
    const bool va = (id.y >= 0), vb = (id.w >= 0);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        F2 P[3];
#pragma unroll
        for (int b = 0; b < 3; ++b) P[b] = fma2(lt, R[a][b], mul2(m2, sub2(F[a][b], R[a][b])));
        const F2 s = dot2(P[0], q0, P[1], q1, P[2], q2);
        if (va) acc.f[a] = fmaf(f2_lo(nvol), f2_lo(s), acc.f[a]);
        if (vb) acc.f[a] = fmaf(f2_hi(nvol), f2_hi(s), acc.f[a]);
        RQ[a] = dot2(R[a][0], q0, R[a][1], q1, R[a][2], q2);
        lr[a] = mul2(lam, RQ[a]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const F2 in = a == b ? fma2(m2, diag, mul2(lr[a], RQ[a])) : fma2(lr[a], RQ[b], 0ull);
            if (va) acc.h[3 * a + b] = fmaf(f2_lo(vol), f2_lo(in), acc.h[3 * a + b]);
            if (vb) acc.h[3 * a + b] = fmaf(f2_hi(vol), f2_hi(in), acc.h[3 * a + b]);
        }
}

// k_sweep_wrapper's update of a vertex from its 16 threads' sums: thread t < 12 adds component t in lane order,
// then every thread solves.  `red` holds 32 x 13 floats of the warp.
__device__ __forceinline__ float4 wrapper_update(const CorotSums& acc, float* red, int lane, float4 xi, float4 y,
                                                 float dtsr, unsigned long long* status, bool count) {
    const int slot = lane >> 4, t = lane & 15;
    __syncwarp();  // the last group's sums have been read
#pragma unroll
    for (int k = 0; k < 9; ++k) red[13 * lane + k] = acc.h[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) red[13 * lane + 9 + k] = acc.f[k];
    __syncwarp();
    const float coeff = __fmul_rn(y.w, dtsr);
    float s = t == 9    ? __fmul_rn(coeff, __fsub_rn(y.x, xi.x))
              : t == 10 ? __fmul_rn(coeff, __fsub_rn(y.y, xi.y))
              : t >= 11 ? __fmul_rn(coeff, __fsub_rn(y.z, xi.z))
              : t % 4 == 0 ? __fmul_rn(coeff, 1.000001f)
                           : 0.0f;
    const float* col = red + 13 * 16 * slot + min(t, 11);
#pragma unroll
    for (int src = 0; src < 16; ++src) s = __fadd_rn(s, col[13 * src]);
    float A[3][3], f[3], C[3][3];
#pragma unroll
    for (int k = 0; k < 9; ++k) A[k / 3][k % 3] = __shfl_sync(0xffffffffu, s, k, 16);
#pragma unroll
    for (int k = 0; k < 3; ++k) f[k] = __shfl_sync(0xffffffffu, s, 9 + k, 16);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
        C[0][i] = i == 1 ? __fsub_rn(__fmul_rn(A[1][2], A[2][0]), __fmul_rn(A[1][0], A[2][2]))
                         : cross1(A[1][i1], A[2][i2], A[1][i2], A[2][i1]);
        C[1][i] = cross1(A[2][i1], A[0][i2], A[2][i2], A[0][i1]);
        C[2][i] = cross1(A[0][i1], A[1][i2], A[0][i2], A[1][i1]);
    }
    const float det = dot1(A[0][0], C[0][0], A[0][1], C[0][1], A[0][2], C[0][2]);
    float4 xn = xi;
    if (fabsf(det) < 1.0e-8f) {
        if (count) atomicAdd(status + ST_SINGULAR, 1ull);
    } else {
        const float inv = __frcp_rn(det);
        xn.x = fmaf(inv, dot1(C[0][0], f[0], C[1][0], f[1], C[2][0], f[2]), xi.x);
        xn.y = fmaf(inv, dot1(C[0][1], f[0], C[1][1], f[1], C[2][1], f[2]), xi.y);
        xn.z = fmaf(inv, dot1(C[0][2], f[0], C[1][2], f[1], C[2][2], f[2]), xi.z);
    }
    return xn;
}

// Local id of vertex v in a tile: an own vertex's, or by its place among the tile's ghosts and pinned neighbours
// (ascending ids).
__device__ __forceinline__ int tile_local(int v, int tile, const TileHead& h, const int* lid, const int* vtile,
                                          const int* vlocal, int nfree) {
    if (v < nfree && vtile[v] == tile) return vlocal[v];
    const int* e = lid + h.lid + h.nown;
    int lo = 0, hi = h.nghost + h.npinned;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (e[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return h.nown + lo;
}

// Record chunks from the packed incidence records (layout 3 or 4): a chunk holds one round of a group;
// vertex slot k's threads t take incidences r L + t and r L + t + L/2.  Neighbour ids become local.
template <int LAYOUT>
__global__ void __launch_bounds__(256) k_pack_tile(SweepParams p, const int* __restrict__ table, int nchunks, int lanes,
                                                   const TileGroup* __restrict__ groups,
                                                   const TileHead* __restrict__ head, const int* __restrict__ lid,
                                                   const int* __restrict__ vtile, const int* __restrict__ vlocal,
                                                   int nfree, float4* __restrict__ out) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nchunks) return;
    const int tile = table[3 * i], round = table[3 * i + 2];
    const TileGroup g = groups[table[3 * i + 1]];
    const TileHead h = head[tile];
    const int T = lanes / 2;
    const int slot = lane / T, t = lane % T;
    auto local = [&](int v) { return tile_local(v, tile, h, lid, vtile, vlocal, nfree); };
    FactRec r[2];
    int id0[2], id1[2];
    const int self = g.lv + min(slot, g.count - 1);  // padding: the vertex itself
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        r[b] = FactRec{};
        id0[b] = self | (self << 16);
        id1[b] = self;
        if (slot >= g.count) continue;
        const int j = p.inc_off[g.gv + slot] + round * lanes + t + b * T;
        if (j >= p.inc_off[g.gv + slot + 1]) continue;
        r[b] = decode_fact(Elem<LAYOUT>::fetch(p, j));
        id0[b] = local(r[b].nb0) | (local(r[b].nb1) << 16);
        id1[b] = local(r[b].nb2) | (1 << 16);
    }
    float4* o = out + (size_t)i * (kTileChunkBytes / 16);
    o[lane] = make_float4(r[0].s0, r[1].s0, r[0].s1, r[1].s1);
    o[32 + lane] = make_float4(r[0].s2, r[1].s2, r[0].w0, r[1].w0);
    o[64 + lane] = make_float4(r[0].w1, r[1].w1, r[0].w2, r[1].w2);
    o[96 + lane] = make_float4(r[0].a, r[1].a, r[0].b, r[1].b);
    reinterpret_cast<int4*>(o)[128 + lane] = make_int4(id0[0], id1[0], id0[1], id1[1]);
    reinterpret_cast<float2*>(o + 160)[lane] = make_float2(r[0].detm, r[1].detm);
}

// The chunks of VBD_GPU_Solver semantics, from the tet records: slot k's threads t take incidences 32 r + t and
// 32 r + t + 16.  A pair of fields per thread: Dm^-1 (9), Dm^-1's row of the vertex q (3), V0, 2 mu, then the
// tets' local ids (bit 31 of the second word: padding, a repeated record), then lambda.
__global__ void __launch_bounds__(256) k_pack_wrapper(const int* __restrict__ inc_off, const int* __restrict__ inc_tet,
                                                      const TetRec* __restrict__ rec, const int* __restrict__ table,
                                                      int nchunks, const TileGroup* __restrict__ groups,
                                                      const TileHead* __restrict__ head, const int* __restrict__ lid,
                                                      const int* __restrict__ vtile, const int* __restrict__ vlocal,
                                                      int nfree, float4* __restrict__ out) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nchunks) return;
    const int tile = table[3 * i], round = table[3 * i + 2];
    const TileGroup g = groups[table[3 * i + 1]];
    const TileHead h = head[tile];
    const int slot = lane >> 4, t = lane & 15;
    const int v = g.gv + min(slot, g.count - 1), self = g.lv + min(slot, g.count - 1);
    const int j0 = inc_off[v], j1 = inc_off[v + 1];
    float fld[15][2];
    int ids[2][2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        const int j = j0 + kWrapperTileLanes * round + t + 16 * b;
        const bool valid = slot < g.count && j < j1;
        for (int k = 0; k < 15; ++k) fld[k][b] = 0.f;
        int l[4] = {self, self, self, self};
        if (j1 > j0) {
            const TetRec r = rec[inc_tet[valid ? j : j0]];
            const int q[4] = {r.ids.x, r.ids.y, r.ids.z, r.ids.w};
            const float D[9] = {r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y, r.b.z, r.b.w, r.c.x};
            const int n = q[0] == v ? 0 : q[1] == v ? 1 : q[2] == v ? 2 : 3;
            for (int k = 0; k < 9; ++k) fld[k][b] = D[k];
            for (int k = 0; k < 3; ++k)
                fld[9 + k][b] = n == 0 ? -D[k] - D[3 + k] - D[6 + k] : D[3 * (n - 1) + k];
            fld[12][b] = r.c.y;
            fld[13][b] = 2.0f * r.c.z;
            fld[14][b] = r.c.w;
            for (int k = 0; k < 4; ++k) l[k] = tile_local(q[k], tile, h, lid, vtile, vlocal, nfree);
        }
        ids[b][0] = l[0] | (l[1] << 16);
        ids[b][1] = l[2] | (l[3] << 16) | (valid ? 0 : (int)0x80000000u);
    }
    float4* o = out + (size_t)i * (kWrapperChunkBytes / 16);
#pragma unroll
    for (int k = 0; k < 7; ++k)
        o[32 * k + lane] = make_float4(fld[2 * k][0], fld[2 * k][1], fld[2 * k + 1][0], fld[2 * k + 1][1]);
    reinterpret_cast<int4*>(o)[224 + lane] = make_int4(ids[0][0], ids[0][1], ids[1][0], ids[1][1]);
    reinterpret_cast<float2*>(o + 256)[lane] = make_float2(fld[14][0], fld[14][1]);
}

// T threads per vertex (2 T lanes' partial sums, two per thread in the two-wide FP32 instructions), W warps.
// W = 8 is the form for tiles with little work per colour, where a colour lasts as long as one vertex's
// dependency chain: everything that does not depend on the neighbours is fetched before the barrier, and
// the chunks stay in shared memory where they fit, else are refilled only after the group's results are
// out.  (One lane per thread and round in plain FP32 measured 1.32 against 1.41 us a colour on the beam, but 1.75
// against 1.68 on the 16^3 cube and 2.16 against 1.86 on the 24^3.)  W = 16 is the form for tiles that keep
// an SM's issue slots and memory streams busy, held to 128 registers.
//
// CL: the tiles are the CTAs of one thread-block cluster, and a vertex's results go straight into its
// neighbours' ghost entries with st.async, completing on the receiver's mbarrier of that colour, instead
// of through words in L2.  A receiver knows the bytes each colour brings.  A sender's colour c of
// iteration k + 1 cannot reach a receiver still waiting for colour c of iteration k: it holds a value
// that receiver computed after that wait (the argument for the words, above), so one barrier per colour
// is enough, armed for the next iteration when its wait ends; bytes that arrive before that are held
// against the same phase.
enum TileKind { kTileForward, kTileAdjoint, kTileWrapper };
template <int T, TileKind KIND, int W, bool CL = false, bool STACK = false>
__global__ void __launch_bounds__(W * 32, 1) k_tile_walk(TileParams p) {
    extern __shared__ __align__(16) unsigned char tsm[];
    constexpr bool ADJ = KIND == kTileAdjoint, WRAP = KIND == kTileWrapper;
    constexpr int kBytes = WRAP ? kWrapperChunkBytes : kTileChunkBytes;
    static_assert(!WRAP || (T == 16 && !CL), "two vertices a warp");
    constexpr int NT = W * 32;
    constexpr bool LAT = W <= 8;
    static_assert(LAT || !CL, "the cluster exchange is the W = 8 form's");
    __shared__ __align__(8) unsigned long long bars[LAT ? 1 : W * kTileMaxRing];
    __shared__ __align__(8) unsigned long long cbars[CL ? kTileMaxColours : 1];
    __shared__ float red[WRAP ? W * 32 * 13 : 1];
    __shared__ float4 stage[LAT ? 1 : W * 64 / T];  // W = 16: own data of each warp's next group
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x;
    const bool two = CL || p.two;
    const TileHead h = p.head[tile];
    const bool resident = LAT && p.resident;
    const int2 ws = p.wstream[tile * W + warp];
    const int slots = resident ? ws.y : p.ring;  // of this warp's ring
    char* ring_buf = reinterpret_cast<char*>(tsm) +
                     (size_t)(resident ? ws.x - p.wstream[tile * W].x : warp * p.ring) * kBytes;
    float4* sx = reinterpret_cast<float4*>(tsm + (size_t)p.ring_chunks * kBytes);  // x (or lambda)
    float4* sb = sx + (two ? p.max_local + 1 : 0);                  // the blended buffer
    float4* sX = sb + (ADJ ? p.max_local + 1 : 0);                  // adjoint: X
    TileGroup* sg = reinterpret_cast<TileGroup*>(sX + p.max_local + 1);
    int* gid = reinterpret_cast<int*>(sg + p.max_groups);  // internal ids of own vertices and ghosts
    int* ghost = gid + p.max_ids;
    int* wcols = ghost + p.ncol + 1;
    int* toff = wcols + W * (p.ncol + 1);
    int* targets = toff + p.max_own + 1;

    const unsigned ring_smem = (unsigned)__cvta_generic_to_shared(ring_buf);
    TileRing ring;
    ring.first = ring.next = ws.x;
    ring.end = ws.x + ws.y;
    ring.left = ws.y * (p.k1 - p.k0);
    ring.slot = 0;
    const unsigned bar = LAT ? 0u : (unsigned)__cvta_generic_to_shared(bars + warp * kTileMaxRing);
    // VBD_GPU_Solver semantics have no registers left for the policy (32^3 cube 2.72 to 2.75 ms with it, 2.64 to 2.69 without)
    constexpr bool HINT = !LAT && !WRAP;
    unsigned long long policy = 0;
    if (HINT) {
        if (p.keep < 1.f)
            asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_first.b64 %0, %1;" : "=l"(policy) : "f"(p.keep));
        else
            asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(policy));
    }
    unsigned parity = 0;  // W = 16: of the ring's current round
    if (!LAT) {
        if (lane == 0) {
            for (int i = 0; i < p.ring; ++i) mbar_init(bar + 8u * i);
            fence_mbar_init();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
    }
    for (int i = 0; i < slots; ++i) {
        if (LAT) ring_issue<kBytes>(p, ring, ring_smem, i, lane);
        else ring_issue_bulk<kBytes, HINT>(p, ring, ring_smem, bar, i, lane, policy);
    }
    if (!CL && tid == 0) atomicAdd(p.arrived, 1ull);

    for (int i = tid; i < h.ngroups; i += NT) sg[i] = p.groups[h.group + i];
    for (int i = tid; i <= p.ncol; i += NT) ghost[i] = p.ghost[tile * (p.ncol + 1) + i];
    for (int i = tid; i < W * (p.ncol + 1); i += NT) wcols[i] = p.wcol[tile * W * (p.ncol + 1) + i];
    const int* lid = p.lid + h.lid;
    const int nloc = h.nown + h.nghost + h.npinned;
    for (int i = tid; i < h.nown + h.nghost; i += NT) gid[i] = lid[i];
    // Cluster exchange: the bytes colour c of iteration k brings this CTA; nobody reads x~ of the last
    // colour when the iteration blends, and nothing of the last iteration's last colour.
    const unsigned cbar0 = (unsigned)__cvta_generic_to_shared(cbars);
    auto colour_bytes = [&](int k, int c, bool blend) {
        const bool last = c == p.ncol - 1, more = k < p.k1 - 1;
        const unsigned words = ((last ? !blend && more : true) ? 1u : 0u) + (blend && more ? 1u : 0u);
        return 16u * words * (unsigned)(ghost[c + 1] - ghost[c]);
    };
    if constexpr (CL) {
        for (int i = tid; i <= h.nown; i += NT) toff[i] = p.target_off[tile * (p.max_own + 1) + i];
        __syncthreads();
        for (int i = tid; i < toff[h.nown]; i += NT) targets[i] = p.target[tile * p.max_target + i];
        if (tid == 0) {
            for (int c = 0; c < p.ncol; ++c) {
                mbar_init(cbar0 + 8u * c);
                const unsigned b = p.k1 > p.k0 ? colour_bytes(p.k0, c, __ldg(p.omega + p.k0) > 1.0f) : 0u;
                if (b) mbar_expect(cbar0 + 8u * c, b);
            }
            fence_mbar_init();
        }
    }
    if constexpr (ADJ) {
        for (int i = tid; i < nloc; i += NT) {
            const int g = lid[i];
            sX[i] = __ldg(p.X + g);
            const float4 l = p.lam_in[g];
            sx[i] = l;
            if (CL) sb[i] = l;
        }
        if (tid == 0) sx[p.max_local] = sb[p.max_local] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        // own vertices, and this CTA's share of the pinned ones
        const int gp = p.nfree + tile * NT + tid, step = gridDim.x * NT;
        if (p.predict) {
            for (int i = tid; i < h.nown; i += NT)
                predict_vertex(lid[i], p.x0, p.v, p.xprev, p.y, p.nfree, p.h, p.hgx, p.hgy, p.hgz);
            for (int g = gp; g < p.n; g += step)
                predict_vertex(g, p.x0, p.v, p.xprev, p.y, p.nfree, p.h, p.hgx, p.hgy, p.hgz);
        }
        for (int i = tid; i < nloc; i += NT) {
            const int g = lid[i];
            const float4 a = p.from_inertia ? p.y[g] : p.x0[g];
            sx[i] = make_float4(a.x, a.y, a.z, 0.f);
            if (two) sb[i] = make_float4(a.x, a.y, a.z, 0.f);
        }
        if (p.from_inertia)  // x = y for the pinned vertices too (k_copy_xyz)
            for (int g = gp; g < p.n; g += step) {
                const float4 a = p.y[g];
                p.x0[g] = p.x1[g] = make_float4(a.x, a.y, a.z, 0.f);
            }
    }
    if (CL) {  // every CTA's barriers and vectors are ready before any CTA sends
        cluster_arrive();
        cluster_wait();
    }
    __syncthreads();

    // Which ghost a thread polls first: W = 8 spreads them over the last warps (a warp's poll takes as long as
    // its slowest lane, and the first warps sweep): 1.66 us a colour on the 16^3 cube, 1.72 over all warps.
    // Two or four polls of a word in flight, spaced over the round trip, made stores land later: 1.87.
    constexpr int kPollWarps = W / 2;
    const int poll_at = !LAT               ? NT - 1 - tid
                        : warp >= kPollWarps ? lane * kPollWarps + (W - 1 - warp)
                                             : (32 + lane) * kPollWarps + (kPollWarps - 1 - warp);
    const int slot = lane / T, t = lane & (T - 1);
    const int* wcol = wcols + warp * (p.ncol + 1);
    const int wfirst = wcol[0], wlast = wcol[p.ncol];
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    // The warp's next group and its vertices' own data, fetched before the barrier that precedes its
    // sweep: y (adjoint: G) and the position before the last sweep.  W = 8 holds them in registers of every
    // thread of the vertex; W = 16 has none to spare and stages them in shared memory.
    TileGroup next_g{};
    float4 own = zero4, prev = zero4;
    float mass = 0.f;
    int send_to = -1, send_more = 0, send_end = 0;  // CL: this thread's first target and the further ones
    float4* my_stage = stage + (LAT ? 0 : warp * (64 / T) + 2 * slot);
    auto load_group = [&](int gi) {
        const TileGroup g = sg[gi];
        const int gv = g.gv + slot;
        if (LAT) {
            next_g = g;
            // predicated loads into the same registers: no instruction waits for them before the solve
            load_if(slot < g.count, (ADJ ? p.G : p.y) + gv, own);
            load_if(slot < g.count, p.pp + gv, prev);
            if constexpr (ADJ) load_if(slot < g.count, &p.y[gv].w, mass);
            if constexpr (CL) {
                send_to = -1;
                send_more = send_end = 0;
                if (slot < g.count) {
                    send_more = toff[g.lv + slot] + t;
                    send_end = toff[g.lv + slot + 1];
                    if (send_more < send_end) send_to = targets[send_more];
                }
            }
        } else {
            if (slot < g.count && t < 2)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(my_stage + t)),
                             "l"((t == 0 ? (ADJ ? p.G : p.y) : p.pp) + gv)
                             : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    bool ok = true;  // of this thread, not of its warp: no shuffle or vote may depend on it
    // Chunk i is commit group i.  W = 8: a group's chunks (at most p.max_rounds) have all landed before the
    // barrier that precedes its sweep, and its slots are refilled after its results are out.  W = 16: a
    // chunk is waited for when it is swept and refilled right after.
    const int pending = resident ? 0 : p.ring - p.max_rounds;
    auto chunk_at = [&](int s) { return TilePair{ring_buf + s * kBytes, lane}; };
    auto next_slot = [&](int s) { return s + 1 == slots ? 0 : s + 1; };
    if (p.k1 > p.k0 && wlast > wfirst) {
        load_group(wfirst);
        if (LAT) ring_wait(pending);
    }
    bool alive = true;
    float4* xs = sx;  // x (adjoint: lambda) of this iteration
    float4* xb = sb;  // two: receives the blended positions
    float om_next = p.k1 > p.k0 ? __ldg(p.omega + p.k0) : 1.0f;
    for (int k = p.k0; k < p.k1 && alive; ++k) {
        const float om = om_next;
        om_next = __ldg(p.omega + min(k + 1, p.k1 - 1));  // known a whole iteration ahead
        const bool blend = om > 1.0f, more = k < p.k1 - 1;
        const unsigned tag = p.tag + (unsigned)k;
        // the words of x~ and of the blended positions; W = 16 forms the addresses where it uses them
        auto words = [&](unsigned which) {
            unsigned at = which + (tag & 1u);
            if (!LAT) asm volatile("" : "+r"(at));
            return p.words + (size_t)at * p.n * p.word_stride;
        };
        int gi = wfirst;
        for (int c = 0; c < p.ncol; ++c) {
            const int gend = wcol[c + 1];
            const bool last = c == p.ncol - 1;
            const bool need_x = last ? !blend && more : true, need_b = blend && more;  // by other tiles
            int p0 = 0, p1 = 0;  // the ghosts of colour c
            if (LAT) p0 = ghost[c] + poll_at, p1 = ghost[c + 1];
            __syncthreads();  // everything colour c reads is in shared memory
            while (gi < gend) {
                float4 xi = zero4;
                int rounds;
                {
                    const TileGroup g = LAT ? next_g : sg[gi];
                    if (slot < g.count) xi = (ADJ ? sX : xs)[g.lv + slot];
                    rounds = g.rounds;
                }
                std::conditional_t<STACK, Acc1, Acc2> acc2;
                CorotSums sums;
                if constexpr (WRAP) {
#pragma unroll
                    for (int i = 0; i < 9; ++i) sums.h[i] = 0.f;
                    sums.f[0] = sums.f[1] = sums.f[2] = 0.f;
                } else {
                    acc2.zero();
                }
                if constexpr (LAT && WRAP) {
                    for (int at = ring.slot, left = rounds; left > 0; --left, at = next_slot(at))
                        tile_corot(ring_buf + at * kBytes, lane, xs, sums);
                } else if constexpr (LAT) {
                    // two chunks at a time: their gathers and products are independent, the sums in order
                    int at = ring.slot, left = rounds;
                    for (; left > 1; left -= 2) {
                        const TilePair r0 = chunk_at(at), r1 = chunk_at(next_slot(at));
                        at = next_slot(next_slot(at));
                        if constexpr (ADJ) {
                            tile_adjoint(r0, r0.ids(), xi, sX, xs, p.max_local, acc2);
                            tile_adjoint(r1, r1.ids(), xi, sX, xs, p.max_local, acc2);
                        } else {
                            tile_contrib(r0, r0.ids(), xi, xs, acc2);
                            tile_contrib(r1, r1.ids(), xi, xs, acc2);
                        }
                    }
                    if (left > 0) {
                        const TilePair r0 = chunk_at(at);
                        if constexpr (ADJ) tile_adjoint(r0, r0.ids(), xi, sX, xs, p.max_local, acc2);
                        else tile_contrib(r0, r0.ids(), xi, xs, acc2);
                    }
                } else {
                    for (; rounds > 0; --rounds) {
                        const int used = ring.slot;
                        if (!ring_wait_bulk(p, bar + 8u * used, parity)) {  // the whole warp; nothing to read there
                            ok = false;
                            break;
                        }
                        ring.slot = next_slot(used);
                        if (ring.slot == 0) parity ^= 1u;
                        const TilePair rec = chunk_at(used);
                        if constexpr (WRAP) tile_corot(rec.buf, lane, xs, sums);
                        else if constexpr (ADJ) tile_adjoint(rec, rec.ids(), xi, sX, xs, p.max_local, acc2);
                        else tile_contrib(rec, rec.ids(), xi, xs, acc2);
                        __syncwarp();  // every lane has read slot `used`
                        ring_issue_bulk<kBytes, HINT>(p, ring, ring_smem, bar, used, lane, policy);
                    }
                }
                // W = 16 reads the group again instead of holding it
                const TileGroup g = LAT ? next_g : sg[gi];
                const bool active = slot < g.count;
                const int lv = g.lv + slot, gv = g.gv + slot;
                // lanes t and t + T, then the T threads: group_reduce's order for 2 T lanes.  Every thread of the
                // vertex ends with the same sums.
                Acc acc;
                if constexpr (!WRAP) {
                    acc = acc2.sum();
                    group_reduce<T>(acc);
                }
                float4 y = own, q = prev;
                if (!LAT) {
                    ring_wait_for<0>();
                    __syncwarp();
                    if (active && (WRAP || t == 0)) {
                        y = my_stage[0];
                        q = my_stage[1];
                        if constexpr (ADJ) mass = __ldg(&p.y[gv].w);
                    }
                }
                float4 xw;
                if constexpr (WRAP)
                    xw = wrapper_update(sums, red + warp * 32 * 13, lane, xi, y, p.dtsr, p.status, active && t == 0);
                if (active && (CL || t == 0)) {
                    float4 xn, xa = zero4, old;
                    if constexpr (ADJ) {
                        old = xs[lv];
                        xn = adj_block_solve(acc, mass, p.dtsr, y);
                    } else {
                        old = xi;
                        if constexpr (WRAP) xn = xw;
                        else xn = block_update(acc, xi, y, p.dtsr, p.status, t == 0);
                    }
                    if (CL) {
                        if (blend) xa = ADJ ? adj_blend(xn, q, om) : cheb_blend(xn, q, om);
                        for (int to = send_to; to >= 0;) {
                            const unsigned r = (unsigned)to >> 16, at = (unsigned)to & 0xffffu;
                            const unsigned rb = cluster_map(cbar0 + 8u * c, r);
                            if (need_x) st_async(cluster_map((unsigned)__cvta_generic_to_shared(xs + at), r), xn, rb);
                            if (need_b) st_async(cluster_map((unsigned)__cvta_generic_to_shared(xb + at), r), xa, rb);
                            send_more += T;
                            to = send_more < send_end ? targets[send_more] : -1;
                        }
                        if (t == 0 && blend) xb[lv] = xa;
                    } else {
                        if (slot < g.publish) word_store(words(0u) + (size_t)gv * p.word_stride, xn.x, xn.y, xn.z, tag);
                        if (blend) {
                            xa = ADJ ? adj_blend(xn, q, om) : cheb_blend(xn, q, om);
                            if (!two || slot < g.publish) word_store(words(2u) + (size_t)gv * p.word_stride, xa.x, xa.y, xa.z, tag);
                            if (two) xb[lv] = xa;
                        }
                    }
                    if (t == 0) {
                        xs[lv] = xn;
                        if (p.keep_pp) p.pp[gv] = old;
                        if (!ADJ) flag_nonfinite(xn, p.status);
                    }
                }
                __syncwarp();  // the other threads may read p.pp of the same vertex next
                ++gi;
                load_group(gi < wlast ? gi : wfirst);
                if (LAT && resident) {
                    ring.slot += rounds;
                    if (ring.slot >= slots) ring.slot = 0;
                } else if (LAT) {
                    for (; rounds > 0; --rounds) {
                        ring_issue<kBytes>(p, ring, ring_smem, ring.slot, lane);
                        ring.slot = next_slot(ring.slot);
                    }
                    ring_wait(pending);
                }
            }
            if constexpr (CL) {
                if ((need_x || need_b) && p1 > ghost[c]) {
                    ok = ok && mbar_wait(cbar0 + 8u * c, (unsigned)(k - p.k0) & 1u, p.status);
                    if (tid == 0 && more) {
                        const unsigned b = colour_bytes(k + 1, c, om_next > 1.0f);
                        if (b) mbar_expect(cbar0 + 8u * c, b);
                    }
                }
            } else {
                // Colour c of the neighbouring tiles: x~, which the next colour reads.  Nobody reads x~ of the last
                // colour when the iteration blends.  With both buffers here the blended words are taken as
                // well, one colour late (they have landed by then and are needed only next iteration).
                if (!LAT) p0 = ghost[c] + poll_at, p1 = ghost[c + 1];
                if (need_b && two) {
                    const int e = last ? ghost[c + 1] : ghost[c];
                    for (int i = (c ? ghost[c - 1] : ghost[0]) + poll_at; ok && i < e; i += NT) {
                        const float4* w = words(2u) + (size_t)gid[i] * p.word_stride;
                        ok = tile_take(p, word_load(w), w, tag, xb + i);
                    }
                }
                if (need_x)
                    for (int i = p0; ok && i < p1; i += NT) {
                        const float4* w = words(0u) + (size_t)gid[i] * p.word_stride;
                        ok = LAT ? tile_spin(p, w, tag, xs + i) : tile_take(p, word_load(w), w, tag, xs + i);
                    }
            }
        }
        // one wait that gave up ends the walk
        alive = __syncthreads_and(ok) != 0;
        if (!alive || !blend) continue;
        if (two) {
            float4* s = xs;
            xs = xb;
            xb = s;
            continue;
        }
        // the blended positions replace x~: own ones and ghosts
        const int e = more ? h.nown + h.nghost : h.nown;
        constexpr int kBatch = 6;
        const float4* wb = words(2u);
        for (int i0 = tid; ok && i0 < e; i0 += kBatch * NT) {
            float4 w[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (i0 + u * NT < e) w[u] = word_load(wb + (size_t)gid[i0 + u * NT] * p.word_stride);
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int i = i0 + u * NT;
                if (i >= e) continue;
                if (__float_as_uint(w[u].w) == tag) xs[i] = make_float4(w[u].x, w[u].y, w[u].z, 0.f);
                else ok = ok && tile_spin(p, wb + (size_t)gid[i] * p.word_stride, tag, xs + i);
            }
        }
    }
    ok = __syncthreads_and(alive && ok) != 0;
    if (CL) {  // no CTA leaves while another may still send to it
        cluster_arrive();
        cluster_wait();
    }
    // no copy outlives the walk (one that gave up has bulk copies under way; the waits are bounded)
    ring_wait_for<0>();
    if (!LAT && !ok) {
        const unsigned long long t0 = global_ns();
        for (int i = 0; i < p.ring; ++i) {
            while (!ring_test(bar + 8u * ring.slot, parity) && global_ns() - t0 < kTileDrainNs) __nanosleep(100);
            ring.slot = next_slot(ring.slot);
            if (ring.slot == 0) parity ^= 1u;
        }
    }
    if (!ok) return;
    for (int i = tid; i < h.nown; i += NT) {
        const int gv = gid[i];
        const float4 xf = xs[i];
        if constexpr (ADJ) {
            p.lam_out[gv] = xf;
        } else {
            p.x0[gv] = xf;
            if (p.from_inertia) p.x1[gv] = xf;
            if (p.finish) p.v[gv] = damped_velocity(xf, p.xprev[gv], p.v[gv], p.h);
        }
    }
}

}  // namespace vbd
