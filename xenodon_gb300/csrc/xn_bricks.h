// Shared types of the octree build, and the interface of its brick form
// (svo_bricks.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace xn {

struct LevelGeom {
    uint32_t bx, by, bz;  // box of stored cells
    uint64_t n;           // bx*by*bz
    uint64_t e;           // cell extent in voxels
};

struct CDStats {  // ChannelDiff: sums, per-channel min and max (packed RGBA)
    unsigned long long sum[4];
    uint32_t mn, mx;
};

struct SDStats {  // StdDev: first moments, and second moments (whose sum over the channels is what is used)
    unsigned long long s1[4];
    unsigned long long s2[4];
};

struct GridDev {
    const uint32_t* vox;  // packed RGBA8, x fastest
    uint32_t dx, dy, dz;
};

constexpr int MAX_LEVELS = 40;

// The cells of depth d that are stored, for every depth below L
// (svo_build.cu's header).
void level_boxes(LevelGeom* geo, int L, uint64_t side, uint32_t dx, uint32_t dy, uint32_t dz);

// What the build has to write: the reference's node array, the device layout
// of svo_layout.cu, or of that only the internal nodes (the lean build).
enum BrickMode { BRICK_NODES = 0, BRICK_LAYOUT = 1, BRICK_LEAN = 2 };

struct BrickOut {
    uint32_t* nodes;       // BRICK_NODES: n x 10 words
    uint64_t capacity;     // BRICK_NODES: room in nodes; a larger tree writes nothing
    uint32_t* inner;       // BRICK_LAYOUT, BRICK_LEAN
    uint32_t* inner_depth;
    uint32_t* rinner;      // BRICK_LAYOUT
    uint32_t* leaves;
};

// One build over 16^3-voxel bricks: grids of at least 16 voxels on their
// longest side (L >= BRICK_LEVELS).
constexpr int BRICK_LEVELS = 4;
struct BrickBuild {
    GridDev g;
    int L, Lb;  // depth of single voxels; depth of the bricks, L - BRICK_LEVELS
    int heuristic;
    uint32_t chan_diff;
    double stddev;
    int equality;    // ChannelDiff with threshold 0, and only the leaves' colours are wanted (not BRICK_NODES)
    int sequential;  // StdDev: every decision through the reference's loop (a check mode)
    LevelGeom geo[MAX_LEVELS];     // depths 0 .. Lb
    uint64_t off[MAX_LEVELS + 1];  // first cell of each depth in the arrays below
    // scratch
    void* stats;                 // per cell: CDStats or SDStats
    unsigned long long* size;    // internal nodes of the subtree
    unsigned long long* start;   // internal nodes before it in post-order, NONE: no such node
    uint32_t* color;
    uint8_t* flags;
    void* rec;                   // per brick: BrickRec
    unsigned long long* info;    // [0] internal nodes of the tree, [1] depth of the deepest of them
};

// Fills b's geometry and returns the scratch it needs; with base != nullptr
// lays the arrays out there.
uint64_t brick_plan(BrickBuild& b, uint64_t side, unsigned char* base);
// Bottom-up pass and starts; b.info is valid once it is done.
cudaError_t brick_scan(const BrickBuild& b, cudaStream_t s);
// Writes the tree.  ropes: leaves get their rope links.
cudaError_t brick_write(const BrickBuild& b, BrickMode mode, bool ropes, int depth_offset, const BrickOut& out,
                        cudaStream_t s);

}  // namespace xn
