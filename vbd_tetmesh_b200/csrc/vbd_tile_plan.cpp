// Host plan of the tile walk: see vbd_tile_plan.h.
#include "vbd_tile_plan.h"

#include <algorithm>
#include <cmath>
#include <thread>

#include "vbd_internal.h"

namespace vbd {
namespace {

// A vertex as the bisection compares it.
struct Point {
    float x[3];
    int32_t mesh, id;
};

void bisect(Point* b, Point* e, int first, int parts, std::vector<int32_t>* tile, int spawn) {
    if (parts <= 1 || e - b <= 1) {
        for (Point* p = b; p < e; ++p) (*tile)[p->id] = first;
        return;
    }
    float lo[3], hi[3];
    int32_t mlo = b->mesh, mhi = b->mesh;
    for (int a = 0; a < 3; ++a) lo[a] = hi[a] = b->x[a];
    for (const Point* p = b; p < e; ++p) {
        for (int a = 0; a < 3; ++a) {
            lo[a] = std::min(lo[a], p->x[a]);
            hi[a] = std::max(hi[a], p->x[a]);
        }
        mlo = std::min(mlo, p->mesh);
        mhi = std::max(mhi, p->mesh);
    }
    int a0 = 0;
    for (int a = 1; a < 3; ++a)
        if (hi[a] - lo[a] > hi[a0] - lo[a0]) a0 = a;
    const int a1 = (a0 + 1) % 3, a2 = (a0 + 2) % 3;
    const bool by_mesh = mlo != mhi;
    const int left = parts / 2;
    Point* mid = b + (long long)(e - b) * left / parts;
    // ties (planes of a regular grid) are split by the other axes, then by id
    std::nth_element(b, mid, e, [=](const Point& p, const Point& q) {
        if (by_mesh && p.mesh != q.mesh) return p.mesh < q.mesh;
        if (p.x[a0] != q.x[a0]) return p.x[a0] < q.x[a0];
        if (p.x[a1] != q.x[a1]) return p.x[a1] < q.x[a1];
        if (p.x[a2] != q.x[a2]) return p.x[a2] < q.x[a2];
        return p.id < q.id;
    });
    each_item(2, spawn > 0 && e - b > 10000, [=](int, int half) {
        if (half == 0) bisect(b, mid, first, left, tile, spawn - 1);
        else bisect(mid, e, first + left, parts - left, tile, spawn - 1);
    });
}

}  // namespace

void tile_partition(int n, const float* positions, const uint8_t* fixed, const int32_t* mesh_of, int parts,
                    std::vector<int32_t>* tile) {
    tile->assign(n, -1);
    std::vector<Point> pts;
    pts.reserve(n);
    for (int i = 0; i < n; ++i) {
        if (fixed[i]) continue;
        Point p;
        for (int a = 0; a < 3; ++a) {
            const float v = positions[3LL * i + a];
            p.x[a] = std::isfinite(v) ? v : 0.0f;  // an ordering needs comparable values
        }
        p.mesh = mesh_of ? mesh_of[i] : 0;
        p.id = i;
        pts.push_back(p);
    }
    if (!pts.empty()) bisect(pts.data(), pts.data() + pts.size(), 0, parts, tile, 4);
}

void tile_boundary(int n, int ntet, const int32_t* tets, const std::vector<int32_t>& tile,
                   std::vector<uint8_t>* boundary) {
    boundary->assign(n, 0);
    for (int t = 0; t < ntet; ++t) {
        const int32_t* q = tets + 4LL * t;
        int lo = 0x7fffffff, hi = -1;
        for (int k = 0; k < 4; ++k) {
            const int v = tile[q[k]];
            if (v < 0) continue;
            lo = std::min(lo, v);
            hi = std::max(hi, v);
        }
        if (hi > lo)  // with two tiles among them, each free vertex has a neighbour of another tile
            for (int k = 0; k < 4; ++k)
                if (tile[q[k]] >= 0) (*boundary)[q[k]] = 1;
    }
}

void tile_lists(TilePlan* plan, const std::vector<int>& cstart, const std::vector<int32_t>& tile_internal,
                const std::vector<uint8_t>& boundary_internal, const int32_t* inc_off, const int32_t* inc_tet,
                const int32_t* tets_internal, int tet_stride) {
    TilePlan& p = *plan;
    const int C = (int)cstart.size() - 1, P = p.P, nfree = p.nfree;
    p.C = C;
    p.vtile.assign(tile_internal.begin(), tile_internal.begin() + nfree);
    p.vlocal.assign(nfree, 0);
    p.cb.assign((size_t)C * (P + 1), 0);
    p.bnd.assign((size_t)C * P, 0);
    p.head.assign(P, TileHead{});
    for (int c = 0; c < C; ++c) {
        int32_t* cb = &p.cb[(size_t)c * (P + 1)];
        int v = cstart[c];
        for (int t = 0; t < P; ++t) {
            cb[t] = v;
            while (v < cstart[c + 1] && tile_internal[v] == t && boundary_internal[v]) ++v;
            p.bnd[(size_t)c * P + t] = v;
            while (v < cstart[c + 1] && tile_internal[v] == t) ++v;
        }
        cb[P] = v;
    }
    for (int t = 0; t < P; ++t) {
        int l = 0;
        for (int c = 0; c < C; ++c) {
            const int32_t* cb = &p.cb[(size_t)c * (P + 1)];
            for (int v = cb[t]; v < cb[t + 1]; ++v) p.vlocal[v] = l++;
        }
        p.head[t].nown = l;
    }
    // ghosts: the other tiles' and the pinned vertices that share a tet with an own vertex, by id (hence
    // by colour, the pinned ones last)
    std::vector<std::vector<int32_t>> ext(P);
    std::vector<std::vector<int32_t>> stamp(kMaxWorkers);
    each_item(P, nfree > 4000, [&](int w, int t) {
        std::vector<int32_t>& st = stamp[w];
        if (st.empty()) st.assign(p.n, -1);
        std::vector<int32_t>& out = ext[t];
        for (int c = 0; c < C; ++c) {
            const int32_t* cb = &p.cb[(size_t)c * (P + 1)];
            for (int v = cb[t]; v < cb[t + 1]; ++v)
                for (int j = inc_off[v]; j < inc_off[v + 1]; ++j) {
                    const int32_t* q = tets_internal + (long long)tet_stride * inc_tet[j];
                    for (int k = 0; k < 4; ++k) {
                        const int u = q[k];
                        if ((u < nfree && tile_internal[u] == t) || st[u] == t) continue;
                        st[u] = t;
                        out.push_back(u);
                    }
                }
        }
        std::sort(out.begin(), out.end());
    });
    p.ghost.assign((size_t)P * (C + 1), 0);
    p.lid.clear();
    p.max_local = p.max_ids = 0;
    for (int t = 0; t < P; ++t) {
        TileHead& h = p.head[t];
        h.lid = (int)p.lid.size();
        for (int c = 0; c < C; ++c) {
            const int32_t* cb = &p.cb[(size_t)c * (P + 1)];
            for (int v = cb[t]; v < cb[t + 1]; ++v) p.lid.push_back(v);
        }
        p.lid.insert(p.lid.end(), ext[t].begin(), ext[t].end());
        h.nghost = (int)(std::lower_bound(ext[t].begin(), ext[t].end(), nfree) - ext[t].begin());
        h.npinned = (int)ext[t].size() - h.nghost;
        for (int c = 0; c <= C; ++c)
            p.ghost[(size_t)t * (C + 1) + c] =
                h.nown + (int)(std::lower_bound(ext[t].begin(), ext[t].end(), cstart[c]) - ext[t].begin());
        p.max_ids = std::max(p.max_ids, h.nown + h.nghost);
        p.max_local = std::max(p.max_local, h.nown + h.nghost + h.npinned);
    }
}

void tile_merge(const TilePlan& fine, int parts, const std::vector<int>& cstart, TilePlan* out) {
    TilePlan& p = *out;
    const int C = fine.C, F = fine.P;
    p.P = parts;
    p.C = C;
    p.n = fine.n;
    p.nfree = fine.nfree;
    p.vtile.resize(fine.nfree);
    p.vlocal.assign(fine.nfree, 0);
    for (int v = 0; v < fine.nfree; ++v) p.vtile[v] = (int)((long long)fine.vtile[v] * parts / F);
    p.cb.assign((size_t)C * (parts + 1), 0);
    p.bnd.assign((size_t)C * parts, 0);  // no words are published
    for (int c = 0; c < C; ++c) {
        int32_t* cb = &p.cb[(size_t)c * (parts + 1)];
        int v = cstart[c];
        for (int t = 0; t < parts; ++t) {
            cb[t] = v;
            while (v < cstart[c + 1] && p.vtile[v] == t) ++v;
        }
        cb[parts] = v;
    }
    p.head.assign(parts, TileHead{});
    p.ghost.assign((size_t)parts * (C + 1), 0);
    std::vector<std::vector<int32_t>> ext(parts);
    for (int f = 0; f < F; ++f) {
        const TileHead& h = fine.head[f];
        const int t = (int)((long long)f * parts / F);
        for (int i = h.lid + h.nown; i < h.lid + h.nown + h.nghost + h.npinned; ++i) {
            const int u = fine.lid[i];
            if (u >= fine.nfree || p.vtile[u] != t) ext[t].push_back(u);
        }
    }
    for (int t = 0; t < parts; ++t) {
        TileHead& h = p.head[t];
        std::sort(ext[t].begin(), ext[t].end());
        ext[t].erase(std::unique(ext[t].begin(), ext[t].end()), ext[t].end());
        h.lid = (int)p.lid.size();
        for (int c = 0; c < C; ++c)
            for (int v = p.cb[(size_t)c * (parts + 1) + t]; v < p.cb[(size_t)c * (parts + 1) + t + 1]; ++v) {
                p.vlocal[v] = h.nown++;
                p.lid.push_back(v);
            }
        p.lid.insert(p.lid.end(), ext[t].begin(), ext[t].end());
        h.nghost = (int)(std::lower_bound(ext[t].begin(), ext[t].end(), p.nfree) - ext[t].begin());
        h.npinned = (int)ext[t].size() - h.nghost;
        for (int c = 0; c <= C; ++c)
            p.ghost[(size_t)t * (C + 1) + c] =
                h.nown + (int)(std::lower_bound(ext[t].begin(), ext[t].end(), cstart[c]) - ext[t].begin());
        p.max_own = std::max(p.max_own, h.nown);
        p.max_ids = std::max(p.max_ids, h.nown + h.nghost);
        p.max_local = std::max(p.max_local, h.nown + h.nghost + h.npinned);
    }
    std::vector<std::vector<std::vector<int32_t>>> to(parts);
    for (int t = 0; t < parts; ++t) to[t].resize(p.head[t].nown);
    for (int t = 0; t < parts; ++t)
        for (int i = 0; i < p.head[t].nghost; ++i) {
            const int u = ext[t][i];
            to[p.vtile[u]][p.vlocal[u]].push_back((t << 16) | (p.head[t].nown + i));
        }
    for (int t = 0; t < parts; ++t) {
        int n = 0;
        for (const auto& l : to[t]) n += (int)l.size();
        p.max_target = std::max(p.max_target, n);
    }
    p.target_off.assign((size_t)parts * (p.max_own + 1), 0);
    p.target.assign((size_t)parts * std::max(1, p.max_target), 0);
    for (int t = 0; t < parts; ++t) {
        int n = 0;
        int32_t* off = &p.target_off[(size_t)t * (p.max_own + 1)];
        for (int i = 0; i < p.max_own; ++i) {
            off[i] = n;
            if (i < p.head[t].nown)
                for (int x : to[t][i]) p.target[(size_t)t * p.max_target + n++] = x;
        }
        off[p.max_own] = n;
    }
}

void tile_groups(TilePlan* plan, int lanes, int warps, const int32_t* inc_off) {
    TilePlan& p = *plan;
    p.lanes = lanes;
    p.warps = warps;
    p.groups.clear();
    p.chunk.clear();
    p.wcol.assign((size_t)p.P * warps * (p.C + 1), 0);
    p.wstream.assign((size_t)p.P * warps * 2, 0);
    p.max_groups = p.max_rounds = p.max_chunks = p.max_colour_groups = 0;
    const int per = kTileChunk / lanes;  // vertices per group
    for (int c = 0; c < p.C; ++c)
        for (int t = 0; t < p.P; ++t) {
            const int32_t* cb = &p.cb[(size_t)c * (p.P + 1) + t];
            p.max_colour_groups = std::max(p.max_colour_groups, (cb[1] - cb[0] + per - 1) / per);
        }
    for (int t = 0; t < p.P; ++t) {
        TileHead& h = p.head[t];
        h.group = (int)p.groups.size();
        const int first = (int)(p.chunk.size() / 3);
        // colour c's groups go round the warps; each warp's groups and chunks lie in the order it sweeps them
        for (int w = 0; w < warps; ++w) {
            int32_t* ws = &p.wstream[((size_t)t * warps + w) * 2];
            int32_t* wc = &p.wcol[((size_t)t * warps + w) * (p.C + 1)];
            ws[0] = (int)(p.chunk.size() / 3);
            for (int c = 0; c < p.C; ++c) {
                wc[c] = (int)p.groups.size() - h.group;
                const int ve = p.cb[(size_t)c * (p.P + 1) + t + 1], bnd = p.bnd[(size_t)c * p.P + t];
                for (int v = p.cb[(size_t)c * (p.P + 1) + t] + w * per; v < ve; v += warps * per) {
                    TileGroup g;
                    g.gv = v;
                    g.lv = p.vlocal[v];
                    g.count = (short)std::min(per, ve - v);
                    g.publish = (short)std::max(0, std::min<int>(g.count, bnd - v));
                    g.rounds = 0;
                    for (int k = 0; k < g.count; ++k)
                        g.rounds = std::max(g.rounds, (inc_off[v + k + 1] - inc_off[v + k] + lanes - 1) / lanes);
                    for (int r = 0; r < g.rounds; ++r) {
                        p.chunk.push_back(t);
                        p.chunk.push_back((int)p.groups.size());
                        p.chunk.push_back(r);
                    }
                    p.max_rounds = std::max(p.max_rounds, g.rounds);
                    p.groups.push_back(g);
                }
            }
            wc[p.C] = (int)p.groups.size() - h.group;
            ws[1] = (int)(p.chunk.size() / 3) - ws[0];
        }
        h.ngroups = (int)p.groups.size() - h.group;
        p.max_groups = std::max(p.max_groups, h.ngroups);
        p.max_chunks = std::max(p.max_chunks, (int)(p.chunk.size() / 3) - first);
    }
}

}  // namespace vbd
