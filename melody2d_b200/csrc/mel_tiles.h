// Tiles: the Gauss points of a deformable body of at most MEL_MAX_BODY_NODES nodes, in the layout the
// body kernel's Gauss-point pass reads (larger bodies keep the chunk images of mel_chunks.h).
//
// A tile is up to MEL_TILE_GP consecutive points, sorted by (support count descending, index) into
// groups of up to 32, one warp each.  The pass keeps a point's first derivative pairs in registers,
// loaded straight from global memory, and holds in shared memory the points' contributions, one slot
// an entry, and what bulk copies bring: the other pairs (about half of them in FP64, a quarter in the
// mixed form) and the indices.  Sections of a tile (byte offsets from mel_tile::base, each 16-byte aligned):
//   head    pairs dN/dx, dN/dy of the rows k < MEL_TILE_HEAD, read straight into registers: entry k of
//           lane l of a group at h0 + k w + l, h0 the pairs of the groups before and w the group's
//           width (its points rounded up to the slots of one shared-memory wavefront).  FP64 pairs;
//           FP32 in the mixed form, two rows side by side (entry (k, l) at h0 + (k / 2) 2 w + 2 l +
//           k % 2, a group's rows padded to an even count)
//   rec     mel_point per point
//   tail    the other rows the same way, row k at t0 + (k - MEL_TILE_HEAD) w
//   idx     per group, four rows a 64-bit word: word i0 + (k / 4) w + l holds the entries k .. k+3 of
//           lane l, 16 bits each: body-local node (12 bits) | place << 12.  Padding names the node
//           after the body's last, a zero displacement
//   slot    mel_pull per touched node, sorted by entry count (descending), groups of 32
//   pos     per pull group, four entries a 64-bit word: word p0 + (j / 4) 32 + l holds the slots of
//           contributions j .. j+3 of lane l's node, in ascending point order.  Padding names the
//           slot after the cap, a zero contribution
// An entry's slot is s0 + k w + (l with its low bits replaced by `place`), s0 = h0 + t0: entries written together
// by one wavefront keep their row of slots but may take any place in it.  The places are a colouring
// of the bipartite graph whose edges are the entries and whose vertices are the wavefronts that
// write them and the wavefronts that read them: both have at most MEL_PLACES entries, so (Konig)
// MEL_PLACES colours suffice and neither the writes nor the reads meet a bank twice.
#pragma once
#include <cstdint>
#include <vector>
#include "mel_internal.h"

struct mel_tile_set {
    bool mixed = false;
    int cap = 0;
    std::vector<mel_tile> tiles;
    std::vector<int> b_tile0;        // [n_bodies+1] first tile of each body
    std::vector<int> gp0;            // first point of each tile
    uint8_t* data = nullptr;         // all tiles (malloc), each base a multiple of 128 bytes
    size_t bytes = 0;
    int max_idx = 16, max_pull = 16; // largest index and pull sections (bytes)
    long long n_entries = 0;         // support entries of the tiled points
    long long n_points = 0, n_pull = 0;
    mel_tile_set() = default;
    mel_tile_set(const mel_tile_set&) = delete;
    mel_tile_set& operator=(const mel_tile_set&) = delete;
    ~mel_tile_set();
};

// Cuts the points of every deformable body of at most MEL_MAX_BODY_NODES nodes into tiles of at most
// `cap` slots (at least 256 x MEL_PLACES, so that any one point fits) and lays them out; the second call
// writes them.  Both return MEL_OK or an error code with the message set.
mel_status mel_plan_tiles(const mel_model_desc* d, int cap, bool mixed, mel_tile_set& out);
mel_status mel_fill_tiles(const mel_model_desc* d, mel_tile_set& out);
