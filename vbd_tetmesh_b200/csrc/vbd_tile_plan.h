// Host plan of the tile walk (vbd_tile.cuh): which free vertices each CTA ("tile") owns, the
// vertices it reads from other tiles, and the order its warps sweep them in.
#pragma once

#include <cstdint>
#include <vector>

namespace vbd {

constexpr int kTileMaxWarps = 16;           // warps of a tile's CTA: 8 or 16 (TilePlan::warps)
constexpr int kTileChunk = 64;              // incidences per record chunk: two per thread of a warp
constexpr int kTileChunkBytes = kTileChunk * 44;
// VBD_GPU_Solver semantics: a chunk holds two vertices' incidences (16 threads each, two incidences per thread)
constexpr int kWrapperTileLanes = 32;
constexpr int kWrapperChunkBytes = kTileChunk * 68;
constexpr int kWrapperFewGroups = 4;
constexpr int kWrapperMaxLocal = 32767;     // the 16th bit of an id marks padding
constexpr int kTileMaxRing = 6;             // chunks a warp's ring holds at most
constexpr int kTileMaxLocal = 65535;        // local vertex ids are 16 bits
// A mesh gets a plan from this many free vertices.  Microseconds per colour of a step, tile walk against
// captured graph (cubes of n^3 cells, one B200): n = 6 (294 free vertices) 1.29 / 2.33, 12 1.51 / 2.50, 16
// 1.51 / 2.57, 24 1.84 / 3.31, 32 2.73 / 3.53, 48 4.57 / 5.5, 64 7.9 / 10.2.  Smaller meshes were not
// measured: the line lies below the smallest that was, not where the gain ends.
constexpr int kTileMinVertices = 256;
// Free vertices per tile at least, up to one tile per SM.  32, 64 and 128 measured 0.81, 0.81 and 0.86 ms a
// step on the 12^3 to 16^3 cubes: a colour lasts one exchange and one vertex's chain either way.
constexpr int kTileVertices = 32;
// Groups per colour and tile up to which 8 warps sweep them; 16 above.  Microseconds per colour with 8 / 16
// warps: 28^3 cube (4.6 groups) 2.36 / 2.46, 32^3 (7.2) 2.99 / 2.76, 64 beams (7.7) 3.06 / 2.81, 64^3 (29)
// 10.8 / 8.4.
constexpr int kTileFewGroups = 6;
// Groups of a colour in a tile up to which a thread's two incidences belong to one lane (TilePlan::stack): at
// 5 the 14^3 cube takes 1.43 us a colour against 1.51, at 6 the 12^3 1.51 / 1.51 and the 18^3 1.57 / 1.55.
constexpr int kTileStackGroups = 5;
// Up to this many free vertices per tile each exchanged word has a 128-byte line of its own: polls of the
// words beside it delay a store's arrival.  Microseconds per colour with words 16 / 32 / 128 bytes apart:
// 12^3 cube 1.59 / 1.53 / 1.47, 16^3 1.66 / 1.57 / 1.50, 24^3 (100 vertices a tile) 1.83 / 1.79 / 1.82, 28^3
// 2.26 / 2.30 / 2.31, 64^3 8.41 / 8.62 / -.
constexpr int kTileSpreadWords = 80;
// Up to this many free vertices the number of tiles is a multiple of 16, so that a cluster's CTAs share them
// evenly (VBD_OPT_PERSISTENT 2), with this many vertices per CTA at least.
constexpr int kClusterMeshVertices = 5000;
constexpr int kClusterTileMin = 16;
// Bytes of a chunk stream that L2 (126 MB) holds beside the rest, and those held of a larger one (the 44^3
// cube's 92 MB: 3.95 us a colour with 48 MB held, 4.40 plain).
constexpr double kTileStreamFits = 90e6;
constexpr double kTileStreamKept = 48e6;
// Ring depth that holding both position buffers must leave.
constexpr int kTileTwoRing = 4;

// One group of vertices a warp sweeps together: internal ids [gv, gv + count), local ids from lv;
// `rounds` chunks hold its incidences.  The first `publish` of them are read by other tiles.
struct alignas(16) TileGroup {
    int gv, lv;
    short count, publish;
    int rounds;
};

struct TileHead {
    int nown, nghost, npinned;  // local ids: own by colour, then ghosts by colour, then pinned vertices
    int lid;                    // first entry in the local-to-internal id list
    int group;                  // first group
    int ngroups;
};

struct TilePlan {
    int P = 0, C = 0, n = 0, nfree = 0;
    std::vector<int32_t> vtile;    // tile of each internal free vertex
    std::vector<int32_t> vlocal;   // its local id in that tile
    std::vector<int32_t> cb;       // [C][P + 1]: colour c's vertices of tile t are [cb[t], cb[t + 1])
    std::vector<int32_t> bnd;      // [C][P]: the first of them up to this id are read by other tiles
    std::vector<TileHead> head;    // [P]
    std::vector<int32_t> lid;      // local-to-internal ids of all tiles
    std::vector<int32_t> ghost;    // [P][C + 1]: first ghost of each colour (local id)
    int max_local = 0, max_ids = 0, max_groups = 0, max_rounds = 0, max_chunks = 0;
    // for `lanes` threads' worth of partial sums per vertex:
    int lanes = 0, warps = 0;
    int max_colour_groups = 0;     // of one colour and tile
    bool stack = false;            // a thread's two incidences belong to one lane (lanes = 2 x threads' sums)
    std::vector<TileGroup> groups;
    std::vector<int32_t> wcol;     // [P][warps][C + 1]: first group of each warp and colour, from the tile's first
    std::vector<int32_t> wstream;  // [P][warps][2]: first chunk and chunks of each warp
    std::vector<int32_t> chunk;    // [chunks][3]: tile, group, round
    // of a merged plan: where each own vertex is a ghost, as tile << 16 | local id there
    int max_own = 0, max_target = 0;
    std::vector<int32_t> target_off;  // [P][max_own + 1], from the tile's first
    std::vector<int32_t> target;      // [P][max_target]
};

// The tile of each vertex (-1 for pinned ones): recursive bisection of the free vertices, first by
// mesh (mesh_of may be null: one mesh), then along the longest axis of their positions.
void tile_partition(int n, const float* positions, const uint8_t* fixed, const int32_t* mesh_of, int parts,
                    std::vector<int32_t>* tile);

// Marks the free vertices that a free vertex of another tile shares a tet with.
void tile_boundary(int n, int ntet, const int32_t* tets, const std::vector<int32_t>& tile, std::vector<uint8_t>* boundary);

// The plan's lists that do not depend on the lane count, from the internal numbering.  tets_internal[4 T]
// holds internal ids; inc_off / inc_tet the incidences of internal vertices.
void tile_lists(TilePlan* plan, const std::vector<int>& cstart, const std::vector<int32_t>& tile_internal,
                const std::vector<uint8_t>& boundary_internal, const int32_t* inc_off, const int32_t* inc_tet,
                const int32_t* tets_internal, int tet_stride);

// The plan with runs of consecutive tiles of `fine` merged into `parts` tiles, and its targets.
void tile_merge(const TilePlan& fine, int parts, const std::vector<int>& cstart, TilePlan* out);

// The groups and record chunks for `lanes` partial sums per vertex (two per thread) and CTAs of `warps` warps.
void tile_groups(TilePlan* plan, int lanes, int warps, const int32_t* inc_off);

}  // namespace vbd
