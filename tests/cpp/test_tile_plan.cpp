// The tile walk's host plan (vbd_tile_plan.h) on Kuhn grids: every list the kernels index, and the
// exchange of published words replayed on the CPU with tiles advancing in random order.
//   test_tile_plan LX LY LZ MESHES TILES LANES PIN SEED   (PIN: 1 = the x = 0 face is pinned)
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>
#include <vector>

#include "vbd_tile_plan.h"

#define REQUIRE(c)                                             \
    do {                                                       \
        if (!(c)) {                                            \
            std::printf("line %d: %s\n", __LINE__, #c);        \
            return 1;                                          \
        }                                                      \
    } while (0)

int main(int argc, char** argv) {
    if (argc < 9) return 2;
    const int lx = atoi(argv[1]), ly = atoi(argv[2]), lz = atoi(argv[3]), M = atoi(argv[4]), P = atoi(argv[5]);
    const int L = atoi(argv[6]), W = argc > 9 ? atoi(argv[9]) : 16, pin = atoi(argv[7]);
    std::mt19937 rng(atoi(argv[8]));
    const int per = (lx + 1) * (ly + 1) * (lz + 1), N = per * M;
    std::vector<int32_t> tets, mesh(N);
    std::vector<float> pos(3 * N);
    std::vector<uint8_t> fixed(N, 0);
    static const int ord[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
    const int step[3] = {1, lx + 1, (lx + 1) * (ly + 1)};
    for (int m = 0; m < M; ++m) {
        for (int k = 0; k <= lz; ++k)
            for (int j = 0; j <= ly; ++j)
                for (int i = 0; i <= lx; ++i) {
                    const int v = m * per + i + (lx + 1) * (j + (ly + 1) * k);
                    pos[3 * v] = (float)i, pos[3 * v + 1] = (float)j, pos[3 * v + 2] = (float)k;
                    mesh[v] = m;
                    fixed[v] = pin && i == 0;
                    if (i < lx && j < ly && k < lz)
                        for (auto& o : ord) {
                            int q = v;
                            tets.push_back(q);
                            for (int a : o) tets.push_back(q += step[a]);
                        }
                }
    }
    pos[0] = 0.0f / 0.0f;  // a non-finite position must not upset the ordering
    const int T = (int)tets.size() / 4;
    // greedy colours
    std::vector<std::set<int>> nb(N);
    for (int t = 0; t < T; ++t)
        for (int a = 0; a < 4; ++a)
            for (int b = 0; b < 4; ++b)
                if (a != b) nb[tets[4 * t + a]].insert(tets[4 * t + b]);
    std::vector<int> colour(N, -1);
    int C = 0;
    for (int v = 0; v < N; ++v) {
        std::set<int> used;
        for (int u : nb[v]) used.insert(colour[u]);
        int c = 0;
        while (used.count(c)) ++c;
        colour[v] = c;
        C = std::max(C, c + 1);
    }
    std::vector<int32_t> tile;
    std::vector<uint8_t> boundary;
    vbd::tile_partition(N, pos.data(), fixed.data(), M > 1 ? mesh.data() : nullptr, P, &tile);
    vbd::tile_boundary(N, T, tets.data(), tile, &boundary);
    // internal order as vbd_solver_init makes it
    std::vector<int32_t> perm, iperm(N);
    std::vector<int> cstart(C + 1);
    std::vector<std::vector<int>> vt(N);
    for (int t = 0; t < T; ++t)
        for (int a = 0; a < 4; ++a) vt[tets[4 * t + a]].push_back(t);
    for (int c = 0; c < C; ++c) {
        cstart[c] = (int)perm.size();
        std::vector<std::vector<long long>> o;
        for (int v = 0; v < N; ++v)
            if (colour[v] == c && !fixed[v]) o.push_back({tile[v], !boundary[v], -(long long)vt[v].size(), v});
        std::sort(o.begin(), o.end());
        for (auto& q : o) perm.push_back((int)q[3]);
    }
    cstart[C] = (int)perm.size();
    const int nfree = (int)perm.size();
    for (int v = 0; v < N; ++v)
        if (fixed[v]) perm.push_back(v);
    for (int i = 0; i < N; ++i) iperm[perm[i]] = i;
    std::vector<int32_t> off(N + 1, 0), inc, tin(tets.size()), til(N, -1);
    std::vector<uint8_t> bin(N, 0);
    for (size_t k = 0; k < tets.size(); ++k) tin[k] = iperm[tets[k]];
    for (int i = 0; i < N; ++i) {
        for (int t : vt[perm[i]]) inc.push_back(t);
        off[i + 1] = (int)inc.size();
        if (i < nfree) til[i] = tile[perm[i]], bin[i] = boundary[perm[i]];
        REQUIRE(i >= nfree || (til[i] >= 0 && til[i] < P));
    }
    vbd::TilePlan p;
    p.P = P;
    p.n = N;
    p.nfree = nfree;
    vbd::tile_lists(&p, cstart, til, bin, off.data(), inc.data(), tin.data(), 4);
    // merged plans (the CTAs of a cluster): the lists of the merged tiles made directly, and each ghost
    // entry the target of its vertex exactly once
    for (int parts : {1, std::min(P, 3), std::min(P, 16)}) {
        vbd::TilePlan m, d;
        vbd::tile_merge(p, parts, cstart, &m);
        std::vector<int32_t> mt(N, -1);
        for (int v = 0; v < nfree; ++v) mt[v] = m.vtile[v];
        d.P = parts;
        d.n = N;
        d.nfree = nfree;
        vbd::tile_lists(&d, cstart, mt, bin, off.data(), inc.data(), tin.data(), 4);
        REQUIRE(m.vlocal == d.vlocal && m.lid == d.lid && m.ghost == d.ghost && m.cb == d.cb);
        REQUIRE(m.max_local == d.max_local && m.max_ids == d.max_ids);
        std::set<int> targets;
        size_t ghosts = 0;
        for (int t = 0; t < parts; ++t) {
            const vbd::TileHead& h = m.head[t];
            REQUIRE(h.nown == d.head[t].nown && h.nghost == d.head[t].nghost && h.npinned == d.head[t].npinned);
            ghosts += h.nghost;
            const int32_t* at = &m.target_off[(size_t)t * (m.max_own + 1)];
            REQUIRE(h.nown <= m.max_own && at[0] == 0 && at[h.nown] <= m.max_target);
            for (int i = 0; i < h.nown; ++i)
                for (int k = at[i]; k < at[i + 1]; ++k) {
                    const int to = m.target[(size_t)t * m.max_target + k], r = to >> 16, l = to & 0xffff;
                    REQUIRE(r < parts && r != t && l >= m.head[r].nown && l < m.head[r].nown + m.head[r].nghost);
                    REQUIRE(m.lid[m.head[r].lid + l] == m.lid[h.lid + i] && targets.insert(to).second);
                }
        }
        REQUIRE(targets.size() == ghosts);
    }
    vbd::tile_groups(&p, L, W, off.data());
    REQUIRE((int)p.head.size() == P && p.max_local <= vbd::kTileMaxLocal);
    // local ids
    auto local = [&](int t, int v) {
        const vbd::TileHead& h = p.head[t];
        if (v < nfree && p.vtile[v] == t) return p.vlocal[v];
        const int32_t* b = p.lid.data() + h.lid + h.nown;
        return h.nown + (int)(std::lower_bound(b, b + h.nghost + h.npinned, v) - b);
    };
    std::vector<int> seen(nfree, 0), covered(off[nfree], 0);
    std::vector<char> published(nfree, 0);
    for (int t = 0; t < P; ++t) {
        const vbd::TileHead& h = p.head[t];
        REQUIRE(h.lid + h.nown + h.nghost + h.npinned <= (int)p.lid.size());
        REQUIRE(h.nown + h.nghost + h.npinned <= p.max_local && h.ngroups <= p.max_groups);
        REQUIRE(h.group + h.ngroups <= (int)p.groups.size());
        for (int i = 0; i < h.nown; ++i) REQUIRE(p.lid[h.lid + i] < nfree && p.vlocal[p.lid[h.lid + i]] == i);
        for (int c = 0; c < C; ++c) {
            const int32_t* g = &p.ghost[(size_t)t * (C + 1)];
            REQUIRE(g[c] >= h.nown && g[c + 1] >= g[c] && g[c + 1] <= h.nown + h.nghost);
            for (int i = g[c]; i < g[c + 1]; ++i)
                REQUIRE(p.lid[h.lid + i] >= cstart[c] && p.lid[h.lid + i] < cstart[c + 1]);
            for (int w = 0; w < W; ++w)
            for (int k = p.wcol[((size_t)t * W + w) * (C + 1) + c];
                 k < p.wcol[((size_t)t * W + w) * (C + 1) + c + 1]; ++k) {
                const vbd::TileGroup& gr = p.groups[h.group + k];
                REQUIRE(h.group + k < (int)p.groups.size());
                REQUIRE(gr.count >= 1 && gr.count <= vbd::kTileChunk / L && gr.publish <= gr.count);
                for (int s = 0; s < gr.count; ++s) {
                    const int v = gr.gv + s;
                    REQUIRE(v >= cstart[c] && v < cstart[c + 1] && p.vtile[v] == t && p.vlocal[v] == gr.lv + s);
                    ++seen[v];
                    published[v] = s < gr.publish;
                    for (int j = off[v]; j < off[v + 1]; ++j)
                        for (int a = 0; a < 4; ++a) {
                            const int u = tin[4 * inc[j] + a], l = local(t, u);
                            REQUIRE(l < h.nown + h.nghost + h.npinned && p.lid[h.lid + l] == u);
                        }
                }
            }
        }
        REQUIRE(p.ghost[(size_t)t * (C + 1) + C] == h.nown + h.nghost);
    }
    for (int v = 0; v < nfree; ++v) REQUIRE(seen[v] == 1);
    for (int t = 0; t < P; ++t)
        for (int i = 0; i < p.head[t].nghost; ++i) {
            const int u = p.lid[p.head[t].lid + p.head[t].nown + i];
            REQUIRE(p.vtile[u] != t && published[u]);
        }
    // chunks: every incidence once, in the order each warp sweeps its groups
    const int nch = (int)p.chunk.size() / 3, T2 = L / 2;
    int at = 0;
    for (int t = 0; t < P; ++t)
        for (int w = 0; w < W; ++w) {
            const int32_t* ws = &p.wstream[((size_t)t * W + w) * 2];
            REQUIRE(ws[0] == at);
            int i = at;
            for (int c = 0; c < C; ++c) {
                const int32_t* gc = &p.wcol[((size_t)t * W + w) * (C + 1)];
                for (int g = gc[c]; g < gc[c + 1]; ++g)
                    for (int r = 0; r < p.groups[p.head[t].group + g].rounds; ++r, ++i) {
                        REQUIRE(i < nch && p.chunk[3 * i] == t && p.chunk[3 * i + 1] == p.head[t].group + g &&
                                p.chunk[3 * i + 2] == r);
                        const vbd::TileGroup& gr = p.groups[p.chunk[3 * i + 1]];
                        for (int lane = 0; lane < 32; ++lane)
                            for (int b = 0; b < 2; ++b) {
                                const int s = lane / T2;
                                if (s >= gr.count) continue;
                                const int j = off[gr.gv + s] + r * L + lane % T2 + b * T2;
                                if (j < off[gr.gv + s + 1]) ++covered[j];
                            }
                    }
            }
            at += ws[1];
            REQUIRE(i == at);
        }
    REQUIRE(at == nch);
    for (int j = 0; j < off[nfree]; ++j) REQUIRE(covered[j] == 1);
    // the exchange: tiles advance phase by phase in random order; a tile's phase ends by taking its ghosts'
    // words.  A word must never be overwritten before all its readers took it, and every tile finishes.
    const int iters = 6;
    for (int blend_from : {99, 1}) {  // no blend; blend from the second iteration on
        std::vector<int> wx(2 * N, 0), wb(2 * N, 0);
        struct State {
            int k = 1, c = 0;
            bool swept = false;  // published, now taking ghosts
        };
        std::vector<State> st(P);
        int done = 0, idle = 0;
        while (done < P) {
            REQUIRE(++idle < 200 * P * iters * C);
            State& s = st[rng() % P];
            const int t = (int)(&s - st.data());
            if (s.k > iters) continue;
            const bool blend = s.k > blend_from;
            const int32_t* lid = p.lid.data() + p.head[t].lid;
            if (!s.swept) {
                for (int v = p.cb[(size_t)s.c * (P + 1) + t]; v < p.cb[(size_t)s.c * (P + 1) + t + 1]; ++v) {
                    if (published[v]) wx[(s.k & 1) * N + v] = s.k;
                    if (blend) wb[(s.k & 1) * N + v] = s.k;
                }
                s.swept = true;
            }
            bool ready = true;
            const bool last = s.c == C - 1;
            if (!(blend && last) && !(s.k == iters && last)) {
                const int32_t* g = &p.ghost[(size_t)t * (C + 1)];
                for (int i = g[s.c]; i < g[s.c + 1]; ++i) {
                    REQUIRE(wx[(s.k & 1) * N + lid[i]] <= s.k);  // a newer tag would never match
                    ready = ready && wx[(s.k & 1) * N + lid[i]] == s.k;
                }
            }
            if (last && blend)
                for (int i = 0; i < p.head[t].nown + (s.k == iters ? 0 : p.head[t].nghost); ++i) {
                    REQUIRE(wb[(s.k & 1) * N + lid[i]] <= s.k);
                    ready = ready && wb[(s.k & 1) * N + lid[i]] == s.k;
                }
            if (!ready) continue;
            idle = 0;
            s.swept = false;
            if (++s.c == C) {
                s.c = 0;
                if (++s.k > iters) ++done;
            }
        }
    }
    std::printf("ok %d vertices %d tiles max_local %d chunks %d (%.2f of the records)\n", N, P, p.max_local, nch,
                nch * (double)vbd::kTileChunk / std::max(1, off[nfree]));
    return 0;
}
