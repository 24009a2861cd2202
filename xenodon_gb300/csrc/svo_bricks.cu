// The octree build over 16^3-voxel bricks: the four deepest levels of the
// tree (cells of 2, 4, 8 and 16 voxels) handled inside one block, from the
// voxels, with nothing per cell in memory but bits.
//
// Both counts that place a node follow from internal nodes alone.  Every
// internal node has eight children, so a subtree with Si internal nodes has
// 8 Si + 1 nodes; and the nodes that come before a cell in post-order are
// whole subtrees, the earlier siblings of the cell and of its ancestors, so a
// cell with si internal nodes before it has 8 si + P nodes before it, where P
// is the sum of the child digits on its path: 4 popc(x) + 2 popc(y) + popc(z)
// of its coordinates at its depth.  With Ni internal nodes in the tree and
// R = Ni - si - Si, a node's place in the reference's array (the reversed
// post-order, src/model/OctreeConstruction.h:92-112) is 8 R - P; R is an
// internal node's rank among the internal nodes, and 7 R - P a leaf's rank
// among the leaves.
//
// So a brick keeps one bit per cell (internal or not, in child order): within
// a brick, si is a count of the bits before a cell.  A 128-byte record per
// 4096 voxels holds them; sizes, starts, colours and statistics exist per
// brick and above only.
//
//  brick_scan   reads the grid once: decisions of the four levels, the record
//               and the brick's statistics; then the levels above, one launch
//               per level of more than TOP_CELLS cells and one block for the
//               rest, and the starts back down the same way.
//  brick_write  reads the grid once more and writes the tree; a rope looks its
//               neighbour up in the records.
//
// Both passes stream the grid; what they cannot do without is two reads of it
// and one write of the tree.  Against one launch per level over per-cell arrays
// (53 bytes for every cell of every level, the node array converted into the
// device layout afterwards), kernel times: 1024^3 gas field, lean, 15.8 ms -> 2.8
// ms (4.3 GB of grid, 4.5 GB of tree: 1.3 ms at copy rate); 509x361x487 CT shell
// with ropes into the layout, 4.2 -> 0.5 ms.
#include <algorithm>
#include <cstring>

#include "../../include/xenodon.h"
#include "xn_bricks.h"
#include "xn_ctx.h"
#include "xn_heuristics.cuh"
#include "xn_internal.h"

namespace xn {
namespace {

using namespace heur;

constexpr uint32_t LEAF = 0x80000000u;
constexpr unsigned long long NONE = ~0ull;
constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr uint8_t F_LEAF = 1, F_INSIDE = 2;
constexpr int BT = 128;          // a scan block: 4 warps, each two octants (8^3 voxels) of the brick that are neighbours in x
constexpr uint32_t ROOT_BIT = 256;
constexpr uint64_t TOP_CELLS = 1024;
// Levels whose cells' std-dev decisions may take the reference's loop over the
// cell's voxels, a thread each, are spread over the GPU from here, in blocks of
// as many: with all 512 cells of 32^3 voxels of a 256^3 grid at the threshold
// the build takes 19 ms; in one block their loops alone took 76.
constexpr uint64_t TOP_LOOPS = 64;

// Octants o, groups g (4^3 voxels, eight an octant) and cells m (2^3 voxels,
// 64 an octant, m = 8 g + child) are in child order: x is the high digit.
struct alignas(16) BrickRec {
    unsigned long long l1[8];  // per octant: internal cells of 2^3 voxels
    unsigned long long l2;     // byte o: internal groups of octant o
    uint16_t pre[8];           // internal nodes of the brick before octant o in post-order
    uint32_t top;              // bit o: octant o is internal; ROOT_BIT: the brick is; from bit 16: its internal levels
    uint32_t pad;
    uint32_t ocol[8];          // average colour of each octant
};
static_assert(sizeof(BrickRec) == 128, "a record is one 128-byte line");

struct Levels {  // a BrickBuild as the kernels take it
    GridDev g;
    int L, Lb;
    uint32_t chan_diff;
    int sequential;
    int equality;  // BrickBuild::equality
    double stddev;
    LevelGeom geo[MAX_LEVELS];
    uint64_t off[MAX_LEVELS + 1];
    void* stats;
    unsigned long long* size;
    unsigned long long* start;
    uint32_t* color;
    uint8_t* flags;
    BrickRec* rec;
    unsigned long long* info;
};

Levels levels_of(const BrickBuild& b) {
    Levels a{};
    a.g = b.g;
    a.L = b.L;
    a.Lb = b.Lb;
    a.chan_diff = b.chan_diff;
    a.sequential = b.sequential;
    a.equality = b.equality;
    a.stddev = b.stddev;
    std::memcpy(a.geo, b.geo, sizeof a.geo);
    std::memcpy(a.off, b.off, sizeof a.off);
    a.stats = b.stats;
    a.size = b.size;
    a.start = b.start;
    a.color = b.color;
    a.flags = b.flags;
    a.rec = static_cast<BrickRec*>(b.rec);
    a.info = b.info;
    return a;
}

__device__ __forceinline__ void coords_of(uint64_t i, const LevelGeom& L, uint32_t& x, uint32_t& y, uint32_t& z) {
    if (L.n <= 0xFFFFFFFFull) {
        const uint32_t j = (uint32_t)i, r = j / L.bx;
        x = j - r * L.bx;
        z = r / L.by;
        y = r - z * L.by;
        return;
    }
    x = (uint32_t)(i % L.bx);
    const uint64_t r = i / L.bx;
    y = (uint32_t)(r % L.by);
    z = (uint32_t)(r / L.by);
}

__device__ __forceinline__ uint64_t index_of(const LevelGeom& L, uint32_t x, uint32_t y, uint32_t z) {
    return (uint64_t)x + (uint64_t)L.bx * ((uint64_t)y + (uint64_t)L.by * z);
}

__device__ __forceinline__ uint32_t digit_sum(uint32_t x, uint32_t y, uint32_t z) {
    return 4u * __popc(x) + 2u * __popc(y) + __popc(z);
}

// Statistics of a cell inside a brick.  Channels 0 and 2, and 1 and 3, share a
// word as 16-bit halves: a sum over up to 4 groups of 4^3 voxels fits (4 * 64
// * 255 < 2^16), so only the last step to an octant widens.
struct Part {
    uint32_t s02, s13;                 // sums
    uint32_t mn02, mn13, mx02, mx13;   // ChannelDiff
    uint32_t q;                        // StdDev: sum of squares over the four channels (4096 voxels fit)
};

template <int HEUR>
__device__ __forceinline__ void part_add(Part& p, uint32_t v, bool valid) {
    const uint32_t a = v & 0x00FF00FFu, b = (v >> 8) & 0x00FF00FFu;
    p.s02 += a;  // a voxel outside the grid is loaded as 0
    p.s13 += b;
    if (HEUR == XN_HEUR_CHANNEL_DIFF) {
        p.mx02 = __vmaxu2(p.mx02, a);
        p.mx13 = __vmaxu2(p.mx13, b);
        p.mn02 = __vminu2(p.mn02, valid ? a : 0x00FF00FFu);
        p.mn13 = __vminu2(p.mn13, valid ? b : 0x00FF00FFu);
    } else {
        p.q = __dp4a(v, v, p.q);
    }
}

__device__ __forceinline__ Part part_empty() {
    return Part{0, 0, 0x00FF00FFu, 0x00FF00FFu, 0, 0, 0};
}

template <int HEUR>
__device__ __forceinline__ void part_merge(Part& p, const Part& o) {
    p.s02 += o.s02;
    p.s13 += o.s13;
    if (HEUR == XN_HEUR_CHANNEL_DIFF) {
        p.mx02 = __vmaxu2(p.mx02, o.mx02);
        p.mx13 = __vmaxu2(p.mx13, o.mx13);
        p.mn02 = __vminu2(p.mn02, o.mn02);
        p.mn13 = __vminu2(p.mn13, o.mn13);
    } else {
        p.q += o.q;
    }
}

template <int HEUR>
__device__ __forceinline__ Part part_shfl(const Part& p, int mask) {
    Part o;
    o.s02 = __shfl_xor_sync(FULL, p.s02, mask);
    o.s13 = __shfl_xor_sync(FULL, p.s13, mask);
    if (HEUR == XN_HEUR_CHANNEL_DIFF) {
        o.mx02 = __shfl_xor_sync(FULL, p.mx02, mask);
        o.mx13 = __shfl_xor_sync(FULL, p.mx13, mask);
        o.mn02 = __shfl_xor_sync(FULL, p.mn02, mask);
        o.mn13 = __shfl_xor_sync(FULL, p.mn13, mask);
    } else {
        o.q = __shfl_xor_sync(FULL, p.q, mask);
    }
    return o;
}

// construct()'s decision (OctreeConstruction.h:141-171) for a cell inside a
// brick: internal unless it is a leaf or outside the grid.  Cells of a brick
// that lies inside the grid as a whole (WHOLE) skip the geometry.
template <int HEUR, bool WHOLE>
__device__ __forceinline__ bool cell_internal(const Levels& a, uint32_t x, uint32_t y, uint32_t z,
                                              uint32_t e, const Part& p, uint32_t s0, uint32_t s1, uint32_t s2,
                                              uint32_t s3) {
    if (!WHOLE) {
        if (x >= a.g.dx || y >= a.g.dy || z >= a.g.dz) return false;
        if (x + e > a.g.dx || y + e > a.g.dy || z + e > a.g.dz) return true;  // partly inside: always split
    }
    if (HEUR == XN_HEUR_CHANNEL_DIFF) {
        // _mm_subs_epu8(max, min), then the largest channel (Grid.cpp:124,135)
        const uint32_t d = __vmaxu2(p.mx02 - p.mn02, p.mx13 - p.mn13);
        return max(d & 0xFFFFu, d >> 16) > a.chan_diff;
    }
    const uint32_t n = e * e * e;  // at most 4096: E < 2^43
    const unsigned long long E = (unsigned long long)n * p.q -
                                 ((unsigned long long)s0 * s0 + (unsigned long long)s1 * s1 +
                                  (unsigned long long)s2 * s2 + (unsigned long long)s3 * s3);
    bool split, seq;  // seq: never needed, e <= EXACT_CELL
    if (E == 0) {
        split = 0.0 > a.stddev;  // every voxel equals the mean: the double sum is exactly 0
    } else {
        // far from the threshold (single precision is off by less than 1e-6
        // here) the decision is plain; near it, in double precision
        const float ef = (float)E, tf = (float)a.stddev * (float)n, lim = tf * tf;
        if (ef > lim * 1.001f && lim < 1e30f) split = true;
        else if (ef < lim * 0.999f && lim < 1e30f) split = false;
        else split = stddev_split((double)E, n, a.stddev, seq);
    }
    if (a.sequential) {
        const unsigned long long s[4] = {s0, s1, s2, s3};
        split = sequential_split(a.g, x, y, z, e, s, a.stddev);
    }
    return split;
}

// ------------------------------------------------------------ brick loads ---

// A lane's place: cells of 2^3 voxels at (2 gx, 2 gy + y0, 2 gz + z0) and the
// next one in x of its octant; its group is g = lane >> 2.
struct Place {
    uint32_t g, sub;     // group of the octant; y0 << 1 | z0
    uint32_t cx, cy, cz; // cell coordinates of the first cell within the octant
};

__device__ __forceinline__ Place place_of(uint32_t lane) {
    Place p;
    p.g = lane >> 2;
    p.sub = lane & 3u;
    p.cx = (lane >> 4) * 2u;
    p.cy = ((lane >> 3) & 1u) * 2u + ((lane >> 1) & 1u);
    p.cz = ((lane >> 2) & 1u) * 2u + (lane & 1u);
    return p;
}

// The 4x2x2 voxels of a lane's two cells: row r = (y << 1 | z), as the
// words of four 16-byte loads, 0 outside the grid.  VEC: rows start on a
// 16-byte boundary (dx a multiple of 4, an aligned grid), so four voxels of a
// row are one load and lie inside the grid together.
template <bool VEC>
__device__ __forceinline__ void load_cells(const GridDev& g, bool whole, uint32_t x, uint32_t y, uint32_t z,
                                           uint4 q[4]) {
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t yy = y + (r >> 1), zz = z + (r & 1u);
        const bool in = whole || (yy < g.dy && zz < g.dz);
        const uint32_t* p = g.vox + (uint64_t)x + (uint64_t)g.dx * ((uint64_t)yy + (uint64_t)g.dy * zz);
        if (VEC) {
            q[r] = in && (whole || x < g.dx) ? __ldg(reinterpret_cast<const uint4*>(p)) : make_uint4(0, 0, 0, 0);
        } else {
            q[r].x = in && (whole || x < g.dx) ? __ldg(p) : 0u;
            q[r].y = in && (whole || x + 1 < g.dx) ? __ldg(p + 1) : 0u;
            q[r].z = in && (whole || x + 2 < g.dx) ? __ldg(p + 2) : 0u;
            q[r].w = in && (whole || x + 3 < g.dx) ? __ldg(p + 3) : 0u;
        }
    }
}

__device__ __forceinline__ uint32_t cell_voxel(const uint4 q[4], uint32_t c, uint32_t k) {
    const uint4& r = q[k & 3u];
    return c == 0 ? ((k & 4u) ? r.y : r.x) : ((k & 4u) ? r.w : r.z);
}

// The eight 4-bit nibbles of w, each in the low (high: shift 4) half of a byte.
__device__ __forceinline__ unsigned long long nibbles_to_bytes(uint32_t w) {
    unsigned long long x = w;
    x = (x | (x << 16)) & 0x0000FFFF0000FFFFull;
    x = (x | (x << 8)) & 0x00FF00FF00FF00FFull;
    return (x | (x << 4)) & 0x0F0F0F0F0F0F0F0Full;
}

// Each bit of a byte as a whole byte.
__device__ __forceinline__ unsigned long long bits_to_bytes(uint32_t b) {
    unsigned long long x = b;
    x = (x | (x << 28)) & 0x0000000F0000000Full;
    x = (x | (x << 14)) & 0x0003000300030003ull;
    x = (x | (x << 7)) & 0x0101010101010101ull;
    return x * 255ull;
}

__device__ __forceinline__ uint32_t average4(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, uint32_t n) {
    return (s0 / n) | ((s1 / n) << 8) | ((s2 / n) << 16) | ((s3 / n) << 24);  // Grid.cpp:126-131
}

// The part of the grid in [x, x + e) x ... as a voxel count (e <= 16).
__device__ __forceinline__ uint32_t count_in(const GridDev& g, uint32_t x, uint32_t y, uint32_t z, uint32_t e) {
    if (x >= g.dx || y >= g.dy || z >= g.dz) return 0;
    return min(e, g.dx - x) * min(e, g.dy - y) * min(e, g.dz - z);
}

struct OctantSums {
    uint32_t s[4];
    uint32_t mn, mx;  // ChannelDiff, packed RGBA
    uint32_t q;
};

// One octant of a brick by one warp: the lane's 16 voxels are q, h is the
// octant's place in x.
template <int HEUR, bool WHOLE>
__device__ __forceinline__ void scan_octant(const Levels& a, const uint4 q[4], const Place& pl, uint32_t lane, uint32_t OX,
                                            uint32_t OY, uint32_t OZ, OctantSums& os, unsigned long long& l1,
                                            uint32_t& l2, uint32_t& l3) {
    if (WHOLE) {
        // an octant of one value, as most of a sparse volume is: a leaf
        uint32_t dif = (q[0].y ^ q[0].x) | (q[0].z ^ q[0].x) | (q[0].w ^ q[0].x);
#pragma unroll
        for (int r = 1; r < 4; ++r)
            dif |= (q[r].x ^ q[0].x) | (q[r].y ^ q[0].x) | (q[r].z ^ q[0].x) | (q[r].w ^ q[0].x);
        dif |= __shfl_sync(FULL, q[0].x, 0) ^ q[0].x;
        if (!__any_sync(FULL, dif != 0)) {
            if (lane == 0) {
                const uint32_t v = q[0].x;
#pragma unroll
                for (int c = 0; c < 4; ++c) os.s[c] = 512u * ((v >> (8 * c)) & 0xFFu);
                os.mn = os.mx = v;
                os.q = 512u * __dp4a(v, v, 0u);
                l1 = 0;
                l2 = l3 = 0;
            }
            return;
        }
    }
    const uint32_t x = OX + pl.cx * 2, y = OY + pl.cy * 2, z = OZ + pl.cz * 2;
    Part group = part_empty();
    uint32_t in[2];
#pragma unroll
    for (uint32_t c = 0; c < 2; ++c) {
        Part p = part_empty();
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const bool valid = WHOLE || (x + 2 * c + (k >> 2) < a.g.dx && y + ((k >> 1) & 1u) < a.g.dy &&
                                         z + (k & 1u) < a.g.dz);
            part_add<HEUR>(p, cell_voxel(q, c, k), valid);
        }
        const bool internal = cell_internal<HEUR, WHOLE>(a, x + 2 * c, y, z, 2, p, p.s02 & 0xFFFFu, p.s13 & 0xFFFFu,
                                                         p.s02 >> 16, p.s13 >> 16);
        in[c] = __ballot_sync(FULL, internal);
        if (c == 0) group = p;
        else part_merge<HEUR>(group, p);
    }
    // groups: the four lanes of one
    part_merge<HEUR>(group, part_shfl<HEUR>(group, 1));
    part_merge<HEUR>(group, part_shfl<HEUR>(group, 2));
    const bool ginternal =
        pl.sub == 0 && cell_internal<HEUR, WHOLE>(a, OX + (pl.g >> 2) * 4, OY + ((pl.g >> 1) & 1u) * 4, OZ + (pl.g & 1u) * 4, 4,
                                                  group, group.s02 & 0xFFFFu, group.s13 & 0xFFFFu, group.s02 >> 16,
                                                  group.s13 >> 16);
    uint32_t gbits = __ballot_sync(FULL, ginternal);  // bit 4 g
    gbits = (gbits | (gbits >> 3)) & 0x03030303u;
    gbits = (gbits | (gbits >> 6)) & 0x000F000Fu;
    gbits = (gbits | (gbits >> 12)) & 0xFFu;
    part_merge<HEUR>(group, part_shfl<HEUR>(group, 4));
    part_merge<HEUR>(group, part_shfl<HEUR>(group, 8));
    uint32_t s0 = group.s02 & 0xFFFFu, s2 = group.s02 >> 16, s1 = group.s13 & 0xFFFFu, s3 = group.s13 >> 16;
    const Part other = part_shfl<HEUR>(group, 16);
    s0 += other.s02 & 0xFFFFu;
    s2 += other.s02 >> 16;
    s1 += other.s13 & 0xFFFFu;
    s3 += other.s13 >> 16;
    part_merge<HEUR>(group, other);  // its sums may have wrapped, s0..s3 hold them
    if (lane == 0) {
        l3 = cell_internal<HEUR, WHOLE>(a, OX, OY, OZ, 8, group, s0, s1, s2, s3);
        os.s[0] = s0;
        os.s[1] = s1;
        os.s[2] = s2;
        os.s[3] = s3;
        if (HEUR == XN_HEUR_CHANNEL_DIFF) {
            os.mn = group.mn02 | (group.mn13 << 8);
            os.mx = group.mx02 | (group.mx13 << 8);
        }
        os.q = group.q;
        l1 = nibbles_to_bytes(in[0]) | (nibbles_to_bytes(in[1]) << 4);
        l2 = gbits;
    }
}

// scan_octant where a cell is a leaf exactly when its voxels are equal
// (ChannelDiff with threshold 0) and no colour but a leaf's is wanted: an OR of
// differences a level instead of sums, minima and maxima (about a third of the
// instructions).  A cell of unequal voxels has minimum 0 and maximum ~0.
__device__ __forceinline__ void scan_octant_equality(const uint4 q[4], uint32_t lane, OctantSums& os,
                                                     unsigned long long& l1, uint32_t& l2, uint32_t& l3) {
    const uint32_t v = q[0].x, v1 = q[0].z;  // the first voxels of the lane's two cells
    uint32_t d0 = q[0].y ^ v, d1 = q[0].w ^ v1;
#pragma unroll
    for (int r = 1; r < 4; ++r) {
        d0 |= (q[r].x ^ v) | (q[r].y ^ v);
        d1 |= (q[r].z ^ v1) | (q[r].w ^ v1);
    }
    const uint32_t in0 = __ballot_sync(FULL, d0 != 0), in1 = __ballot_sync(FULL, d1 != 0);
    // the four lanes of a group against the first of them
    const uint32_t dg = d0 | d1 | (v1 ^ v) | (__shfl_sync(FULL, v, lane & ~3u) ^ v);
    uint32_t gbits = __ballot_sync(FULL, dg != 0);
    gbits |= gbits >> 1;
    gbits = (gbits | (gbits >> 2)) & 0x11111111u;  // bit 4 g
    gbits = (gbits | (gbits >> 3)) & 0x03030303u;
    gbits = (gbits | (gbits >> 6)) & 0x000F000Fu;
    gbits = (gbits | (gbits >> 12)) & 0xFFu;
    const bool octant = gbits || __any_sync(FULL, __shfl_sync(FULL, v, 0) != v);
    if (lane == 0) {
        os.s[0] = os.s[1] = os.s[2] = os.s[3] = 0;
        os.mn = octant ? 0u : v;
        os.mx = octant ? ~0u : v;
        os.q = 0;
        l1 = nibbles_to_bytes(in0) | (nibbles_to_bytes(in1) << 4);
        l2 = gbits;
        l3 = octant;
    }
}

// One block per brick: the record, and the brick's size, colour, flags and
// statistics.
template <int HEUR, bool VEC>
__global__ void __launch_bounds__(BT) brick_scan_kernel(const __grid_constant__ Levels a) {
    const LevelGeom& G = a.geo[a.Lb];
    const uint64_t b = blockIdx.x;
    const uint64_t cell = a.off[a.Lb] + b;
    uint32_t bx, by, bz;
    coords_of(b, G, bx, by, bz);
    const uint32_t X = bx << BRICK_LEVELS, Y = by << BRICK_LEVELS, Z = bz << BRICK_LEVELS;
    BrickRec& rec = a.rec[b];
    if (X >= a.g.dx || Y >= a.g.dy || Z >= a.g.dz) {  // OctreeConstruction.h:146-154
        if (threadIdx.x == 0) {
            a.size[cell] = 0;
            a.color[cell] = 0;
            a.flags[cell] = F_LEAF;
            rec.top = 0;
        }
        return;
    }
    const bool whole = X + 16 <= a.g.dx && Y + 16 <= a.g.dy && Z + 16 <= a.g.dz;
    __shared__ OctantSums s_oct[8];
    __shared__ unsigned long long s_l1[8];
    __shared__ uint32_t s_l2[8], s_l3[8];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const Place pl = place_of(lane);
    const uint32_t OY = Y + (warp >> 1) * 8, OZ = Z + (warp & 1u) * 8;
    uint4 q[2][4];
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h)
        load_cells<VEC>(a.g, whole, X + h * 8 + pl.cx * 2, OY + pl.cy * 2, OZ + pl.cz * 2, q[h]);
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t o = h * 4 + warp;
        if (HEUR == XN_HEUR_CHANNEL_DIFF && whole && a.equality)
            scan_octant_equality(q[h], lane, s_oct[o], s_l1[o], s_l2[o], s_l3[o]);
        else if (whole) scan_octant<HEUR, true>(a, q[h], pl, lane, X + h * 8, OY, OZ, s_oct[o], s_l1[o], s_l2[o], s_l3[o]);
        else scan_octant<HEUR, false>(a, q[h], pl, lane, X + h * 8, OY, OZ, s_oct[o], s_l1[o], s_l2[o], s_l3[o]);
    }
    __syncthreads();
    if (warp != 0) return;
    const uint32_t o = lane & 7u;  // lanes 8.. repeat lanes 0..7
    OctantSums os = s_oct[o];
    const uint32_t on = count_in(a.g, X + (o >> 2) * 8, Y + ((o >> 1) & 1u) * 8, Z + (o & 1u) * 8, 8);
    const bool by_value = HEUR == XN_HEUR_CHANNEL_DIFF && a.equality;  // only leaves' colours: their one value
    const uint32_t ocol = by_value ? (on ? os.mn : 0u) : on ? average4(os.s[0], os.s[1], os.s[2], os.s[3], on) : 0u;
    Part p{};
    p.mn02 = os.mn & 0x00FF00FFu;
    p.mn13 = (os.mn >> 8) & 0x00FF00FFu;
    p.mx02 = os.mx & 0x00FF00FFu;
    p.mx13 = (os.mx >> 8) & 0x00FF00FFu;
    p.q = os.q;
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) {
        part_merge<HEUR>(p, part_shfl<HEUR>(p, m));
#pragma unroll
        for (int c = 0; c < 4; ++c) os.s[c] += __shfl_xor_sync(FULL, os.s[c], m);
    }
    bool internal = false;
    if (lane == 0)
        internal = whole ? cell_internal<HEUR, true>(a, X, Y, Z, 16, p, os.s[0], os.s[1], os.s[2], os.s[3])
                         : cell_internal<HEUR, false>(a, X, Y, Z, 16, p, os.s[0], os.s[1], os.s[2], os.s[3]);
    internal = __shfl_sync(FULL, internal, 0);
    // cells below a leaf do not exist
    const uint32_t l3 = internal ? s_l3[o] : 0u;
    const uint32_t l2 = l3 ? s_l2[o] : 0u;
    const unsigned long long l1 = s_l1[o] & bits_to_bytes(l2);
    const uint32_t count = __popcll(l1) + __popc(l2) + l3;
    uint32_t before = count;
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, before, m);
        if (o >= (uint32_t)m) before += v;
    }
    const uint32_t l3bits = __ballot_sync(FULL, l3 != 0) & 0xFFu;
    const bool any2 = __any_sync(FULL, l2 != 0), any1 = __any_sync(FULL, l1 != 0);
    if (lane < 8) {
        rec.l1[o] = l1;
        reinterpret_cast<uint8_t*>(&rec.l2)[o] = (uint8_t)l2;
        rec.pre[o] = (uint16_t)(before - count);
        rec.ocol[o] = ocol;
    }
    if (lane == 7) a.size[cell] = before + (internal ? 1u : 0u);
    if (lane == 0) {
        const uint32_t deep = !internal ? 0u : any1 ? 4u : any2 ? 3u : l3bits ? 2u : 1u;
        rec.top = l3bits | (internal ? ROOT_BIT : 0u) | (deep << 16);
        const uint32_t n = count_in(a.g, X, Y, Z, 16);
        a.color[cell] = by_value ? p.mn02 | (p.mn13 << 8) : average4(os.s[0], os.s[1], os.s[2], os.s[3], n);
        a.flags[cell] = (internal ? 0 : F_LEAF) | F_INSIDE;
        if (HEUR == XN_HEUR_CHANNEL_DIFF) {
            CDStats& st = static_cast<CDStats*>(a.stats)[cell];
            for (int c = 0; c < 4; ++c) st.sum[c] = os.s[c];
            st.mn = p.mn02 | (p.mn13 << 8);
            st.mx = p.mx02 | (p.mx13 << 8);
        } else {
            SDStats& st = static_cast<SDStats*>(a.stats)[cell];
            for (int c = 0; c < 4; ++c) {
                st.s1[c] = os.s[c];
                st.s2[c] = 0;
            }
            st.s2[0] = p.q;
        }
    }
}

// ------------------------------------------------------ levels above bricks ---

// s / n for a quotient of at most 255, without a 64-bit division: the rounded
// quotient of the rounded operands is off by less than 2^-14, so its integer
// part is off by one at most.
__device__ __forceinline__ uint32_t byte_quotient(unsigned long long s, unsigned long long n) {
    uint32_t q = (uint32_t)__fdiv_rn((float)s, (float)n);
    if (q * n > s) --q;
    else if (s - q * n >= n) ++q;
    return q & 0xFFu;
}

// One cell of depth d < Lb: statistics, decision and size from its children.
template <int HEUR>
__device__ void up_cell(const Levels& a, int d, uint64_t i) {
    const LevelGeom& G = a.geo[d];
    const LevelGeom& C = a.geo[d + 1];
    const uint64_t cell = a.off[d] + i;
    uint32_t x, y, z;
    coords_of(i, G, x, y, z);
    const uint64_t e = G.e, ox = x * e, oy = y * e, oz = z * e;
    if (ox >= a.g.dx || oy >= a.g.dy || oz >= a.g.dz) {  // OctreeConstruction.h:146-154
        a.size[cell] = 0;
        a.color[cell] = 0;
        a.flags[cell] = F_LEAF;
        return;
    }
    // the reference names this "partly_in_grid"; it means fully inside
    const bool fully = ox + e <= a.g.dx && oy + e <= a.g.dy && oz + e <= a.g.dz;
    const uint64_t half = e >> 1;
    unsigned long long s[4] = {0, 0, 0, 0}, q = 0, sz = 1;
    uint32_t mn = 0xFFFFFFFFu, mx = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t cx = 2 * x + (k >> 2), cy = 2 * y + ((k >> 1) & 1u), cz = 2 * z + (k & 1u);
        const uint64_t ci = a.off[d + 1] + index_of(C, cx, cy, cz);
        sz += a.size[ci];
        if ((uint64_t)cx * half >= a.g.dx || (uint64_t)cy * half >= a.g.dy || (uint64_t)cz * half >= a.g.dz) continue;
        if (HEUR == XN_HEUR_CHANNEL_DIFF) {
            const CDStats& cs = static_cast<const CDStats*>(a.stats)[ci];
            mn = __vminu4(mn, cs.mn);
            mx = __vmaxu4(mx, cs.mx);
#pragma unroll
            for (int c = 0; c < 4; ++c) s[c] += cs.sum[c];
        } else {
            const SDStats& cs = static_cast<const SDStats*>(a.stats)[ci];
#pragma unroll
            for (int c = 0; c < 4; ++c) s[c] += cs.s1[c];
            q += cs.s2[0];
        }
    }
    const uint64_t n = clamped_count(a.g, ox, oy, oz, e);
    uint32_t avg = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) avg |= byte_quotient(s[c], n) << (8 * c);  // Grid.cpp:126-131,180-186
    bool split;
    if (HEUR == XN_HEUR_CHANNEL_DIFF) {
        CDStats& out = static_cast<CDStats*>(a.stats)[cell];
        for (int c = 0; c < 4; ++c) out.sum[c] = s[c];
        out.mn = mn;
        out.mx = mx;
        // _mm_subs_epu8(max, min), then the largest channel (Grid.cpp:124,135)
        const uint32_t dif = __vsubus4(mx, mn);
        split = max(max(dif & 0xFFu, (dif >> 8) & 0xFFu), max((dif >> 16) & 0xFFu, dif >> 24)) > a.chan_diff;
        if (a.equality) avg = mn;
    } else {
        SDStats& out = static_cast<SDStats*>(a.stats)[cell];
        unsigned __int128 E = (unsigned __int128)n * q;  // n * sum((x - mean)^2), exact
        for (int c = 0; c < 4; ++c) {
            out.s1[c] = s[c];
            out.s2[c] = 0;
            E -= (unsigned __int128)s[c] * s[c];
        }
        out.s2[0] = q;
        bool seq = false;
        split = E == 0 ? 0.0 > a.stddev : stddev_split((double)E, n, a.stddev, seq);
        // (a cell partly outside is split whatever its deviation)
        if ((seq && fully) || a.sequential) split = sequential_split(a.g, ox, oy, oz, e, s, a.stddev);
    }
    const bool leaf = !split && fully;
    a.color[cell] = avg;
    a.flags[cell] = (leaf ? F_LEAF : 0) | F_INSIDE;
    a.size[cell] = leaf ? 0 : sz;
}

// One cell of depth d < Lb hands its children their starts, and reports the
// depth of the deepest internal node it knows of.
__device__ uint32_t start_cell(const Levels& a, int d, uint64_t i) {
    const uint64_t cell = a.off[d] + i;
    if (!(a.flags[cell] & F_INSIDE)) return 0;  // no stored children
    const LevelGeom& C = a.geo[d + 1];
    uint32_t x, y, z;
    coords_of(i, a.geo[d], x, y, z);
    unsigned long long run = a.start[cell];
    const bool has = run != NONE && !(a.flags[cell] & F_LEAF);
    uint32_t deep = has ? (uint32_t)d : 0u;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint64_t ci = index_of(C, 2 * x + (k >> 2), 2 * y + ((k >> 1) & 1u), 2 * z + (k & 1u));
        const uint64_t cc = a.off[d + 1] + ci;
        a.start[cc] = has ? run : NONE;
        if (has) {
            run += a.size[cc];
            if (d + 1 == a.Lb) {
                const uint32_t levels = a.rec[ci].top >> 16;
                if (levels) deep = max(deep, (uint32_t)a.Lb + levels - 1u);
            }
        }
    }
    return deep;
}

__device__ __forceinline__ void report_depth(const Levels& a, uint32_t deep) {
    deep = __reduce_max_sync(FULL, deep);
    if ((threadIdx.x & 31u) == 0 && deep > *reinterpret_cast<volatile unsigned long long*>(a.info + 1))
        atomicMax(a.info + 1, (unsigned long long)deep);
}

template <int HEUR>
__global__ void __launch_bounds__(256) up_kernel(const __grid_constant__ Levels a, int d) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.geo[d].n) up_cell<HEUR>(a, d, i);
}

__global__ void __launch_bounds__(256) start_kernel(const __grid_constant__ Levels a, int d) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    report_depth(a, i < a.geo[d].n ? start_cell(a, d, i) : 0u);
}

// Depths dup .. 0 up, and of depths 0 .. dtop the children's starts down, in one
// block.
template <int HEUR>
__global__ void __launch_bounds__(1024) top_kernel(const __grid_constant__ Levels a, int dup, int dtop) {
    for (int d = dup; d >= 0; --d) {
        for (uint64_t i = threadIdx.x; i < a.geo[d].n; i += blockDim.x) up_cell<HEUR>(a, d, i);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        a.start[0] = 0;
        a.info[0] = a.size[0];
        a.info[1] = a.Lb == 0 ? max(1u, a.rec[0].top >> 16) - 1u : 0u;
    }
    __syncthreads();
    for (int d = 0; d <= dtop; ++d) {
        const uint64_t n = a.geo[d].n;
        for (uint64_t i0 = 0; i0 < n; i0 += blockDim.x) {
            const uint64_t i = i0 + threadIdx.x;
            report_depth(a, i < n ? start_cell(a, d, i) : 0u);
        }
        __syncthreads();
    }
}

// ----------------------------------------------------------------- writing ---

struct WriteArgs {
    Levels a;
    BrickOut out;
    int depth_off;
};

// The word that names a leaf: its index in the node array, or bit 31 | its
// record's index.
template <int MODE>
__device__ __forceinline__ uint32_t leaf_word(uint32_t Ni, uint32_t si, uint32_t P) {
    return MODE == BRICK_NODES ? 8u * (Ni - si) - P : LEAF | (7u * (Ni - si) - P);
}
template <int MODE>
__device__ __forceinline__ uint32_t inner_word(uint32_t rank, uint32_t P) {
    return MODE == BRICK_NODES ? 8u * rank - P : rank;
}

struct Found {
    uint32_t word;   // of the deepest existing node on the way to the cell
    uint32_t inner;  // it is the cell itself, and internal
    uint32_t base;   // then, with 2^3 voxels: the index of its voxel child k is base - k
};

template <int MODE>
__device__ Found climb(const Levels& a, uint32_t Ni, int d, uint32_t x, uint32_t y, uint32_t z) {
    // the deepest existing cell on the root path of cell (x, y, z) of depth d
    // <= Lb, which is what Octree::find returns (Octree.cpp:116-201)
    for (;; --d, x >>= 1, y >>= 1, z >>= 1) {
        const LevelGeom& G = a.geo[d];
        if (x < G.bx && y < G.by && z < G.bz) {
            const uint64_t cell = a.off[d] + index_of(G, x, y, z);
            const unsigned long long st = a.start[cell];
            if (st != NONE) {
                const uint32_t si = (uint32_t)st, Si = (uint32_t)a.size[cell], P = digit_sum(x, y, z);
                if (Si == 0) return Found{leaf_word<MODE>(Ni, si, P), 0, 0};
                return Found{inner_word<MODE>(Ni - si - Si, P), 1, 0};
            }
        }
        if (d == 0) return Found{0, 0, 0};  // the root always exists
    }
}

__device__ __forceinline__ unsigned long long below64(uint32_t n) { return (1ull << n) - 1ull; }  // n < 64

// A brick and its six neighbours (across face f: 1 + f) as a block holds them.
struct Near {
    BrickRec rec[7];
    unsigned long long start[7];
};

// The same for a cell of extent 2^j, j = 1, 2 or 3 (depth L - j), in the
// block's brick (bx, by, bz) or, a step across face f, in its neighbour.
template <int MODE>
__device__ Found find_cell(const Levels& a, const Near& near, uint32_t bx0, uint32_t by0, uint32_t bz0, uint32_t Ni,
                           int j, uint32_t f, uint32_t cx, uint32_t cy, uint32_t cz) {
    const int up = BRICK_LEVELS - j;
    const uint32_t bx = cx >> up, by = cy >> up, bz = cz >> up;
    const uint32_t slot = bx == bx0 && by == by0 && bz == bz0 ? 0u : 1u + f;
    const unsigned long long st = near.start[slot];
    if (st == NONE) return climb<MODE>(a, Ni, a.Lb - 1, bx >> 1, by >> 1, bz >> 1);
    const BrickRec& r = near.rec[slot];
    const uint32_t top = r.top;
    if (!(top & ROOT_BIT)) return Found{leaf_word<MODE>(Ni, (uint32_t)st, digit_sum(bx, by, bz)), 0, 0};
    const uint32_t ox = cx >> (3 - j), oy = cy >> (3 - j), oz = cz >> (3 - j);
    const uint32_t o = (ox & 1u) << 2 | (oy & 1u) << 1 | (oz & 1u);
    const uint32_t so = (uint32_t)st + r.pre[o];
    if (!(top >> o & 1u)) return Found{leaf_word<MODE>(Ni, so, digit_sum(ox, oy, oz)), 0, 0};
    const unsigned long long l1 = r.l1[o];
    const uint32_t l2 = (uint32_t)(r.l2 >> (8 * o)) & 0xFFu;
    if (j == 3)
        return Found{inner_word<MODE>(Ni - so - (__popcll(l1) + __popc(l2) + 1u), digit_sum(ox, oy, oz)), 1, 0};
    const uint32_t gx = cx >> (2 - j), gy = cy >> (2 - j), gz = cz >> (2 - j);
    const uint32_t g = (gx & 1u) << 2 | (gy & 1u) << 1 | (gz & 1u);
    const uint32_t sg = so + __popcll(l1 & below64(8 * g)) + __popc(l2 & ((1u << g) - 1u));
    if (!(l2 >> g & 1u)) return Found{leaf_word<MODE>(Ni, sg, digit_sum(gx, gy, gz)), 0, 0};
    if (j == 2) return Found{inner_word<MODE>(Ni - sg - (__popc((uint32_t)(l1 >> (8 * g)) & 0xFFu) + 1u), digit_sum(gx, gy, gz)), 1, 0};
    const uint32_t k = (cx & 1u) << 2 | (cy & 1u) << 1 | (cz & 1u);
    const uint32_t sc = sg + __popc((uint32_t)(l1 >> (8 * g)) & ((1u << k) - 1u));
    const uint32_t P = digit_sum(cx, cy, cz);
    if (!(l1 >> (8 * g + k) & 1ull)) return Found{leaf_word<MODE>(Ni, sc, P), 0, 0};
    return Found{0, 1, (MODE == BRICK_NODES ? 8u : 7u) * (Ni - sc) - P};
}

// Rope f (Octree.cpp:181-201: +x, -x, +y, -y, +z, -z) of a leaf cell of
// extent 2^j at (x, y, z) of its depth.  A rope to nothing is 0 in a node
// and ROPE_EXIT in a record; bricks and larger cells: j >= BRICK_LEVELS.
template <int MODE>
__device__ uint32_t rope_of(const Levels& a, const Near* near, uint32_t bx, uint32_t by, uint32_t bz, uint32_t Ni, int j,
                            uint32_t f, uint32_t x, uint32_t y, uint32_t z) {
    const uint32_t step = (f & 1u) ? ~0u : 1u, lim = 1u << (a.L - j);
    const uint32_t nx = x + (f < 2 ? step : 0u), ny = y + ((f >> 1) == 1 ? step : 0u), nz = z + (f >= 4 ? step : 0u);
    if (nx >= lim || ny >= lim || nz >= lim) return MODE == BRICK_NODES ? 0u : ROPE_EXIT;  // outside the octree
    const Found r = j < BRICK_LEVELS ? find_cell<MODE>(a, *near, bx, by, bz, Ni, j, f, nx, ny, nz)
                                     : climb<MODE>(a, Ni, a.L - j, nx, ny, nz);
    if (j != 1 || !r.inner) return r.word;
    // an internal cell of 2^3 voxels as the target itself
    return MODE == BRICK_NODES ? r.base - 8u : (r.base - 7u + digit_sum(nx, ny, nz)) / 7u;
}

__device__ __forceinline__ void put_node(uint32_t* nodes, uint64_t idx, const uint32_t ch[8], uint32_t color, uint32_t leaf_depth) {
    uint2* p = reinterpret_cast<uint2*>(nodes + idx * 10);  // 40-byte nodes are 8-byte aligned
    p[0] = make_uint2(ch[0], ch[1]);
    p[1] = make_uint2(ch[2], ch[3]);
    p[2] = make_uint2(ch[4], ch[5]);
    p[3] = make_uint2(ch[6], ch[7]);
    p[4] = make_uint2(color, leaf_depth);
}

// A leaf's node or record; `word` is its leaf_word.
template <int MODE, bool ROPES>
__device__ void put_leaf(const WriteArgs& w, const Near* near, uint32_t bx, uint32_t by, uint32_t bz, uint32_t Ni,
                         uint32_t word, int j, uint32_t x, uint32_t y, uint32_t z, uint32_t color) {
    if (MODE == BRICK_LEAN) return;
#pragma unroll 1
    for (uint32_t f = 0; f < 6; ++f) {
        const uint32_t v = ROPES ? rope_of<MODE>(w.a, near, bx, by, bz, Ni, j, f, x, y, z) : MODE == BRICK_NODES ? 0u : ROPE_EXIT;
        if (MODE == BRICK_NODES) w.out.nodes[(uint64_t)word * 10 + f] = v;
        else w.out.leaves[(uint64_t)(word & ~LEAF) * 8 + 1 + f] = v;
    }
    const uint32_t depth = LEAF | (uint32_t)(w.a.L - j + w.depth_off);
    if (MODE == BRICK_NODES) {
        uint2* p = reinterpret_cast<uint2*>(w.out.nodes + (uint64_t)word * 10);
        p[3] = make_uint2(0, 0);
        p[4] = make_uint2(color, depth);
    } else {
        w.out.leaves[(uint64_t)(word & ~LEAF) * 8] = color;
        w.out.leaves[(uint64_t)(word & ~LEAF) * 8 + 7] = depth;
    }
}

// Child word k of an internal node: `rank` is the parent's; of the child, the
// rank if it is internal, or its leaf word and colour.
template <int MODE>
__device__ __forceinline__ void put_child(const WriteArgs& w, uint32_t rank, uint32_t Pparent, uint32_t k, bool internal,
                                          uint32_t word, uint32_t color) {
    if (MODE == BRICK_NODES) {
        w.out.nodes[(uint64_t)(8u * rank - Pparent) * 10 + k] = word;
    } else {
        w.out.inner[(uint64_t)rank * 8 + k] = internal ? word : LEAF | (color & 0xFFFFFFu);
        if (MODE == BRICK_LAYOUT) w.out.rinner[(uint64_t)rank * 8 + k] = word;
    }
}

// Colour and depth of an internal node.
template <int MODE>
__device__ __forceinline__ void put_inner(const WriteArgs& w, uint32_t rank, uint32_t P, uint32_t color, int depth) {
    if (MODE == BRICK_NODES)
        reinterpret_cast<uint2*>(w.out.nodes + (uint64_t)(8u * rank - P) * 10)[4] =
            make_uint2(color, (uint32_t)(depth + w.depth_off));
    else w.out.inner_depth[rank] = (uint32_t)depth;
}

// The cells of depth Lb and above: leaves, and internal nodes above the bricks.
template <int MODE, bool ROPES>
__device__ void write_coarse(const WriteArgs& w, uint64_t c) {
    const Levels& a = w.a;
    if (c >= a.off[a.Lb + 1]) return;
    const unsigned long long st = a.start[c];
    if (st == NONE) return;
    if (MODE == BRICK_NODES && 8ull * a.info[0] + 1ull > w.out.capacity) return;
    const uint32_t Ni = (uint32_t)a.info[0];
    int d = a.Lb;
    while (c < a.off[d]) --d;
    const uint8_t fl = a.flags[c];
    if (!(fl & F_LEAF) && d == a.Lb) return;  // the brick's own block writes it
    uint32_t x, y, z;
    coords_of(c - a.off[d], a.geo[d], x, y, z);
    const uint32_t P = digit_sum(x, y, z);
    if (fl & F_LEAF) {
        put_leaf<MODE, ROPES>(w, nullptr, 0, 0, 0, Ni, leaf_word<MODE>(Ni, (uint32_t)st, P), a.L - d, x, y, z, a.color[c]);
        return;
    }
    const uint32_t rank = Ni - (uint32_t)st - (uint32_t)a.size[c];
#pragma unroll 1
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t cx = 2 * x + (k >> 2), cy = 2 * y + ((k >> 1) & 1u), cz = 2 * z + (k & 1u);
        const uint64_t cc = a.off[d + 1] + index_of(a.geo[d + 1], cx, cy, cz);
        const uint32_t cs = (uint32_t)a.start[cc], cS = (uint32_t)a.size[cc], cP = P + k;
        const bool internal = cS != 0;
        put_child<MODE>(w, rank, P, k, internal, internal ? inner_word<MODE>(Ni - cs - cS, cP) : leaf_word<MODE>(Ni, cs, cP),
                        a.color[cc]);
    }
    put_inner<MODE>(w, rank, P, a.color[c], d);
}

// What a warp keeps per internal cell of 2^3 voxels of its octant while the
// lanes write one voxel leaf each.
struct VoxelStage {
    uint32_t vox[64][8];
    uint32_t base[64];     // index of voxel child k: base - k
    uint32_t face[64][6];  // neighbour across face f: the base of its voxels, or the rope word
    uint8_t fine[64];      // bit f: face f's neighbour has voxels
    uint8_t list[64];      // internal cells in child order
};
struct NoStage {};

template <bool NEEDED>
struct StageOf { using T = VoxelStage; };
template <>
struct StageOf<false> { using T = NoStage; };

// One block per brick that is internal, a warp per octant: its internal nodes
// and their leaves.  The blocks after the bricks' write the cells above, a
// thread each.
constexpr int WT = 256;
template <int MODE, bool ROPES, bool VEC>
__global__ void __launch_bounds__(WT) brick_write_kernel(const __grid_constant__ WriteArgs w) {
    const Levels& a = w.a;
    const uint64_t b = blockIdx.x;
    if (b >= a.geo[a.Lb].n) {
        write_coarse<MODE, ROPES>(w, (b - a.geo[a.Lb].n) * WT + threadIdx.x);
        return;
    }
    const unsigned long long st = a.start[a.off[a.Lb] + b];
    const BrickRec& rec = a.rec[b];
    const uint32_t top = rec.top;
    if (st == NONE || !(top & ROOT_BIT)) return;
    if (MODE == BRICK_NODES && 8ull * a.info[0] + 1ull > w.out.capacity) return;
    const uint32_t Ni = (uint32_t)a.info[0];
    const LevelGeom& G = a.geo[a.Lb];
    uint32_t bx, by, bz;
    coords_of(b, G, bx, by, bz);
    const uint32_t X = bx << 4, Y = by << 4, Z = bz << 4;
    const bool whole = X + 16 <= a.g.dx && Y + 16 <= a.g.dy && Z + 16 <= a.g.dz;
    const uint32_t bsi = (uint32_t)st;
    const uint32_t brank = Ni - bsi - (uint32_t)a.size[a.off[a.Lb] + b];
    const uint32_t Pb = digit_sum(bx, by, bz);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const Place pl = place_of(lane);
    const uint32_t o = warp, h = o >> 2, oy = (o >> 1) & 1u, oz = o & 1u;
    constexpr bool STAGED = MODE != BRICK_LEAN;
    __shared__ typename StageOf<STAGED>::T s_stage[STAGED ? WT / 32 : 1];
    __shared__ __align__(16) uint32_t s_nodes[MODE == BRICK_NODES ? WT / 32 : 1][MODE == BRICK_NODES ? 320 : 1];
    if (threadIdx.x == 0) put_inner<MODE>(w, brank, Pb, a.color[a.off[a.Lb] + b], a.Lb);
    __shared__ Near s_near;
    if (ROPES) {  // the records that ropes can reach
        if (threadIdx.x < 7) {
            const uint32_t f = threadIdx.x - 1u, step = (f & 1u) ? ~0u : 1u;
            const uint32_t nx = bx + (threadIdx.x && f < 2 ? step : 0u), ny = by + (threadIdx.x && (f >> 1) == 1 ? step : 0u),
                           nz = bz + (threadIdx.x && f >= 4 ? step : 0u);
            s_near.start[threadIdx.x] =
                nx < G.bx && ny < G.by && nz < G.bz ? a.start[a.off[a.Lb] + index_of(G, nx, ny, nz)] : NONE;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < 7 * sizeof(BrickRec) / 16; i += WT) {
            const uint32_t slot = i / (sizeof(BrickRec) / 16), f = slot - 1u, step = (f & 1u) ? ~0u : 1u;
            if (s_near.start[slot] == NONE) continue;
            const uint64_t bi = index_of(G, bx + (slot && f < 2 ? step : 0u), by + (slot && (f >> 1) == 1 ? step : 0u),
                                         bz + (slot && f >= 4 ? step : 0u));
            reinterpret_cast<uint4*>(s_near.rec)[i] = reinterpret_cast<const uint4*>(a.rec + bi)[i % (sizeof(BrickRec) / 16)];
        }
        __syncthreads();
    }
    const uint32_t so = bsi + rec.pre[o];
    const uint32_t Ox = bx * 2 + h, Oy = by * 2 + oy, Oz = bz * 2 + oz;  // octant coordinates (depth L - 3)
    const uint32_t Po = Pb + o;
    if (!(top >> o & 1u)) {
        if (lane == 0) {
            const uint32_t word = leaf_word<MODE>(Ni, so, Po);
            put_child<MODE>(w, brank, Pb, o, false, word, rec.ocol[o]);
            put_leaf<MODE, ROPES>(w, &s_near, bx, by, bz, Ni, word, 3, Ox, Oy, Oz, rec.ocol[o]);
        }
        return;
    }
    const unsigned long long l1 = rec.l1[o];
    const uint32_t l2 = (uint32_t)(rec.l2 >> (8 * o)) & 0xFFu;
    uint4 q[4];
    load_cells<VEC>(a.g, whole, X + h * 8 + pl.cx * 2, Y + oy * 8 + pl.cy * 2, Z + oz * 8 + pl.cz * 2, q);
    const uint32_t orank = Ni - so - (__popcll(l1) + __popc(l2) + 1u);
    const uint32_t g = pl.g;
    const uint32_t cells = (uint32_t)(l1 >> (8 * g)) & 0xFFu;  // the group's internal cells
    const bool ginternal = l2 >> g & 1u;
    const uint32_t sg = so + __popcll(l1 & below64(8 * g)) + __popc(l2 & ((1u << g) - 1u));
    const uint32_t Gx = Ox * 2 + (g >> 2), Gy = Oy * 2 + ((g >> 1) & 1u), Gz = Oz * 2 + (g & 1u);
    const uint32_t Pg = Po + g;
    const uint32_t grank = Ni - sg - (__popc(cells) + 1u);
    // sums: of the lane's two cells, its group and the octant
    uint32_t c02[2], c13[2];
#pragma unroll
    for (uint32_t c = 0; c < 2; ++c) {
        c02[c] = c13[c] = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t v = cell_voxel(q, c, k);
            c02[c] += v & 0x00FF00FFu;
            c13[c] += (v >> 8) & 0x00FF00FFu;
        }
    }
    uint32_t g02 = c02[0] + c02[1], g13 = c13[0] + c13[1];
    g02 += __shfl_xor_sync(FULL, g02, 1);
    g13 += __shfl_xor_sync(FULL, g13, 1);
    g02 += __shfl_xor_sync(FULL, g02, 2);
    g13 += __shfl_xor_sync(FULL, g13, 2);
    // a leaf cell is whole or outside the grid (all zeros), so its average
    // is a shift; only a partly covered internal node divides
    uint32_t gcol = ((g02 >> 6) & 0x00FF00FFu) | (((g13 >> 6) & 0x00FF00FFu) << 8);
    if (MODE == BRICK_NODES && !whole && ginternal) {
        const uint32_t n = count_in(a.g, Gx * 4, Gy * 4, Gz * 4, 4);
        gcol = average4(g02 & 0xFFFFu, g13 & 0xFFFFu, g02 >> 16, g13 >> 16, n);
    }
    if (lane == 0) {
        put_child<MODE>(w, brank, Pb, o, true, inner_word<MODE>(orank, Po), 0);
        put_inner<MODE>(w, orank, Po, MODE == BRICK_NODES ? rec.ocol[o] : 0u, a.L - 3);
    }
    if (pl.sub == 0) {
        const uint32_t word = ginternal ? inner_word<MODE>(grank, Pg) : leaf_word<MODE>(Ni, sg, Pg);
        put_child<MODE>(w, orank, Po, g, ginternal, word, gcol);
        if (ginternal) put_inner<MODE>(w, grank, Pg, gcol, a.L - 2);
        else put_leaf<MODE, ROPES>(w, &s_near, bx, by, bz, Ni, word, 2, Gx, Gy, Gz, gcol);
    }
    if (ginternal) {
#pragma unroll
        for (uint32_t c = 0; c < 2; ++c) {
            const uint32_t k = c * 4 + pl.sub;
            const uint32_t m = g * 8 + k;
            const bool internal = cells >> k & 1u;
            const uint32_t sc = sg + __popc(cells & ((1u << k) - 1u));
            const uint32_t Pc = Pg + k;
            const uint32_t Cx = Gx * 2 + c, Cy = Gy * 2 + (pl.sub >> 1), Cz = Gz * 2 + (pl.sub & 1u);
            uint32_t col = ((c02[c] >> 3) & 0x00FF00FFu) | (((c13[c] >> 3) & 0x00FF00FFu) << 8);
            const uint32_t rank = Ni - sc - 1u;
            const uint32_t word = internal ? inner_word<MODE>(rank, Pc) : leaf_word<MODE>(Ni, sc, Pc);
            put_child<MODE>(w, grank, Pg, k, internal, word, col);
            if (!internal) {
                put_leaf<MODE, ROPES>(w, &s_near, bx, by, bz, Ni, word, 1, Cx, Cy, Cz, col);
                continue;
            }
            uint32_t v[8];
#pragma unroll
            for (uint32_t t = 0; t < 8; ++t) v[t] = cell_voxel(q, c, t);
            const uint32_t base = (MODE == BRICK_NODES ? 8u : 7u) * (Ni - sc) - Pc;
            if constexpr (MODE == BRICK_NODES) {
                if (!whole) {
                    const uint32_t n = count_in(a.g, Cx * 2, Cy * 2, Cz * 2, 2);
                    col = average4(c02[c] & 0xFFFFu, c13[c] & 0xFFFFu, c02[c] >> 16, c13[c] >> 16, n);
                }
                uint32_t ch[8];
#pragma unroll
                for (uint32_t t = 0; t < 8; ++t) ch[t] = base - t;
                put_node(w.out.nodes, 8u * rank - Pc, ch, col, (uint32_t)(a.L - 1 + w.depth_off));
            } else {
                uint4* p = reinterpret_cast<uint4*>(w.out.inner + (uint64_t)rank * 8);
                p[0] = make_uint4(LEAF | (v[0] & 0xFFFFFFu), LEAF | (v[1] & 0xFFFFFFu), LEAF | (v[2] & 0xFFFFFFu),
                                  LEAF | (v[3] & 0xFFFFFFu));
                p[1] = make_uint4(LEAF | (v[4] & 0xFFFFFFu), LEAF | (v[5] & 0xFFFFFFu), LEAF | (v[6] & 0xFFFFFFu),
                                  LEAF | (v[7] & 0xFFFFFFu));
                w.out.inner_depth[rank] = (uint32_t)(a.L - 1);
                if constexpr (MODE == BRICK_LAYOUT) {
                    uint4* p2 = reinterpret_cast<uint4*>(w.out.rinner + (uint64_t)rank * 8);
                    p2[0] = make_uint4(LEAF | base, LEAF | (base - 1), LEAF | (base - 2), LEAF | (base - 3));
                    p2[1] = make_uint4(LEAF | (base - 4), LEAF | (base - 5), LEAF | (base - 6), LEAF | (base - 7));
                }
            }
            if constexpr (STAGED) {
                VoxelStage& sg_ = s_stage[warp];
#pragma unroll
                for (uint32_t t = 0; t < 8; ++t) sg_.vox[m][t] = v[t];
                sg_.base[m] = base;
                sg_.list[__popcll(l1 & below64(m))] = (uint8_t)m;
                if constexpr (ROPES) {
                    uint32_t fine = 0;
                    const uint32_t lim = 1u << (a.L - 1);
#pragma unroll 1
                    for (uint32_t f = 0; f < 6; ++f) {
                        const uint32_t step = (f & 1u) ? ~0u : 1u;
                        const uint32_t nx = Cx + (f < 2 ? step : 0u), ny = Cy + ((f >> 1) == 1 ? step : 0u),
                                       nz = Cz + (f >= 4 ? step : 0u);
                        uint32_t word2 = MODE == BRICK_NODES ? 0u : ROPE_EXIT;
                        if (nx < lim && ny < lim && nz < lim) {
                            const Found r = find_cell<MODE>(a, s_near, bx, by, bz, Ni, 1, f, nx, ny, nz);
                            word2 = r.inner ? r.base : r.word;
                            fine |= r.inner << f;
                        }
                        sg_.face[m][f] = word2;
                    }
                    sg_.fine[m] = (uint8_t)fine;
                }
            }
        }
    }
    if constexpr (STAGED) {
        VoxelStage& sg_ = s_stage[warp];
        __syncwarp();
        const uint32_t total = 8u * __popcll(l1);
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {
            const uint32_t t = t0 + lane;
            const bool on = t < total;
            const uint32_t m = on ? sg_.list[t >> 3] : 0u, k = t & 7u;
            uint32_t r[6];
            uint32_t idx = 0, color = 0;
            if (on) {
                idx = sg_.base[m] - k;
                color = sg_.vox[m][k];
                if (ROPES) {
                    const uint32_t fine = sg_.fine[m];
#pragma unroll
                    for (uint32_t f = 0; f < 6; ++f) {
                        const uint32_t bit = 4u >> (f >> 1);
                        // towards +axis the sibling is the child with the
                        // axis bit set, towards -axis the one without
                        const bool sibling = ((k & bit) != 0) == ((f & 1u) != 0);
                        const uint32_t kn = k ^ bit;
                        const uint32_t face = sg_.face[m][f];
                        const uint32_t target = (sibling ? sg_.base[m] : face) - kn;
                        r[f] = sibling || (fine >> f & 1u) ? (MODE == BRICK_NODES ? target : LEAF | target) : face;
                    }
                } else {
#pragma unroll
                    for (uint32_t f = 0; f < 6; ++f) r[f] = MODE == BRICK_NODES ? 0u : ROPE_EXIT;
                }
            }
            const uint32_t depth = LEAF | (uint32_t)(a.L + w.depth_off);
            if constexpr (MODE == BRICK_LAYOUT) {
                if (on) {
                    uint4* p = reinterpret_cast<uint4*>(w.out.leaves + (uint64_t)idx * 8);
                    p[0] = make_uint4(color, r[0], r[1], r[2]);
                    p[1] = make_uint4(r[3], r[4], r[5], depth);
                }
            } else {
                // through shared memory, so that neighbouring lanes write
                // neighbouring words of the 40-byte nodes
                uint32_t* sn = s_nodes[warp];
                if (on) {
                    uint2* p = reinterpret_cast<uint2*>(sn + lane * 10);
                    p[0] = make_uint2(r[0], r[1]);
                    p[1] = make_uint2(r[2], r[3]);
                    p[2] = make_uint2(r[4], r[5]);
                    p[3] = make_uint2(0, 0);
                    p[4] = make_uint2(color, depth);
                }
                __syncwarp();
                const uint32_t words = min(32u, total - t0) * 10u;
#pragma unroll
                for (uint32_t i = 0; i < 10; ++i) {
                    const uint32_t wd = i * 32 + lane;
                    const uint32_t node = wd / 10u;
                    const uint32_t at = __shfl_sync(FULL, idx, node & 31u);
                    if (wd < words) w.out.nodes[(uint64_t)at * 10 + (wd - node * 10u)] = sn[wd];
                }
                __syncwarp();
            }
        }
    }
}

inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

bool vector_rows(const GridDev& g) { return g.dx % 4 == 0 && (reinterpret_cast<uintptr_t>(g.vox) & 15) == 0; }

template <int MODE, bool ROPES>
void launch_write(const WriteArgs& w, cudaStream_t s) {
    const unsigned nb = (unsigned)w.a.geo[w.a.Lb].n + blocks_for(w.a.off[w.a.Lb + 1], WT);
    if (vector_rows(w.a.g)) brick_write_kernel<MODE, ROPES, true><<<nb, WT, 0, s>>>(w);
    else brick_write_kernel<MODE, ROPES, false><<<nb, WT, 0, s>>>(w);
}

}  // namespace

void level_boxes(LevelGeom* geo, int L, uint64_t side, uint32_t dx, uint32_t dy, uint32_t dz) {
    for (int d = 0; d < L; ++d) {
        const uint64_t e = side >> d;
        auto box = [&](uint64_t dim) -> uint32_t {
            if (d == 0) return 1;
            const uint64_t pe = e * 2;  // parent extent
            return (uint32_t)std::min<uint64_t>(1ull << d, 2 * ((dim + pe - 1) / pe));
        };
        geo[d].bx = box(dx);
        geo[d].by = box(dy);
        geo[d].bz = box(dz);
        geo[d].n = (uint64_t)geo[d].bx * geo[d].by * geo[d].bz;
        geo[d].e = e;
    }
}

uint64_t brick_plan(BrickBuild& b, uint64_t side, unsigned char* base) {
    b.Lb = b.L - BRICK_LEVELS;
    level_boxes(b.geo, b.Lb + 1, side, b.g.dx, b.g.dy, b.g.dz);
    b.off[0] = 0;
    for (int d = 0; d <= b.Lb; ++d) b.off[d + 1] = b.off[d] + b.geo[d].n;
    const uint64_t cells = b.off[b.Lb + 1];
    uint64_t used = 0;
    auto take = [&](uint64_t bytes) -> unsigned char* {
        unsigned char* p = base ? base + used : nullptr;
        used += (bytes + 255) & ~255ull;
        return p;
    };
    b.rec = take(b.geo[b.Lb].n * sizeof(BrickRec));
    b.stats = take(cells * (b.heuristic == XN_HEUR_STD_DEV ? sizeof(SDStats) : sizeof(CDStats)));
    b.size = reinterpret_cast<unsigned long long*>(take(cells * 8));
    b.start = reinterpret_cast<unsigned long long*>(take(cells * 8));
    b.color = reinterpret_cast<uint32_t*>(take(cells * 4));
    b.flags = take(cells);
    b.info = reinterpret_cast<unsigned long long*>(take(16));
    return used;
}

cudaError_t brick_scan(const BrickBuild& b, cudaStream_t s) {
    const Levels a = levels_of(b);
    const unsigned nb = (unsigned)b.geo[b.Lb].n;
    const bool vec = vector_rows(b.g), cd = b.heuristic == XN_HEUR_CHANNEL_DIFF;
    if (cd && vec) brick_scan_kernel<XN_HEUR_CHANNEL_DIFF, true><<<nb, BT, 0, s>>>(a);
    else if (cd) brick_scan_kernel<XN_HEUR_CHANNEL_DIFF, false><<<nb, BT, 0, s>>>(a);
    else if (vec) brick_scan_kernel<XN_HEUR_STD_DEV, true><<<nb, BT, 0, s>>>(a);
    else brick_scan_kernel<XN_HEUR_STD_DEV, false><<<nb, BT, 0, s>>>(a);
    int up = b.Lb - 1;
    for (; up >= 0 && b.geo[up].n > (cd ? TOP_CELLS : TOP_LOOPS); --up) {
        if (cd) up_kernel<XN_HEUR_CHANNEL_DIFF><<<blocks_for(b.geo[up].n, 256), 256, 0, s>>>(a, up);
        else up_kernel<XN_HEUR_STD_DEV><<<blocks_for(b.geo[up].n, TOP_LOOPS), TOP_LOOPS, 0, s>>>(a, up);
    }
    int d = up;
    while (d + 1 < b.Lb && b.geo[d + 1].n <= TOP_CELLS) ++d;
    if (cd) top_kernel<XN_HEUR_CHANNEL_DIFF><<<1, 1024, 0, s>>>(a, up, d);
    else top_kernel<XN_HEUR_STD_DEV><<<1, 1024, 0, s>>>(a, up, d);
    for (++d; d < b.Lb; ++d) start_kernel<<<blocks_for(b.geo[d].n, 256), 256, 0, s>>>(a, d);
    return cudaGetLastError();
}

cudaError_t brick_write(const BrickBuild& b, BrickMode mode, bool ropes, int depth_offset, const BrickOut& out,
                        cudaStream_t s) {
    WriteArgs w{levels_of(b), out, depth_offset};
    if (mode == BRICK_NODES) {
        if (ropes) launch_write<BRICK_NODES, true>(w, s);
        else launch_write<BRICK_NODES, false>(w, s);
    } else if (mode == BRICK_LAYOUT) {
        if (ropes) launch_write<BRICK_LAYOUT, true>(w, s);
        else launch_write<BRICK_LAYOUT, false>(w, s);
    } else {
        launch_write<BRICK_LEAN, false>(w, s);
    }
    return cudaGetLastError();
}

}  // namespace xn
