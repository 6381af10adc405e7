// Production walkers. The Cartesian and octree walkers follow the reference generators' FP64
// operation order exactly (every wall distance, position update and containment test), so their
// cell sequences and segment lengths equal the reference's bit for bit; what makes them fast is the
// data layout and the division: a wall distance is the correctly rounded quotient from the ray's
// precomputed reciprocal direction (qdiv, three FP64 operations), and the octree walker reads
// 64-byte leaf records with exact FP64 walls from small per-axis lattice tables. Both serve either
// precision: at production precision optical depth, path length and radiation-field factors accumulate
// in FP32 (Acc); in the FP64 life cycle everything does. Tallies are always FP64. The Voronoi and
// tetrahedral walkers below keep FP32 face distances with FP64 re-decisions.
//
// Both were bound by instruction issue (64 % of the peel-off rays' issue slots busy, 205 instructions
// per octree crossing), a good part of them choices by the direction's sign; mirrored coordinates take
// those out (175 per crossing). Galaxy on 5.1e5 leaves, 2e7 packets at production precision: 319 ->
// 304 ms. In FP64 the octree walker used to follow the node arrays with six-wall neighbour scans: 1.5e6
// packets on 8.6e4 leaves 42 -> 26 ms. The Cartesian walker gains 10 % in FP64 and nothing in FP32.
#pragma once

#include <type_traits>

#include "grids.cuh"

namespace skg {

// 1 / k rounded to nearest for |k| > 1e-15 (the reference's threshold for a usable direction
// component), 0 otherwise
SKG_D double recipDir(double k) { return fabs(k) > 1e-15 ? 1.0 / k : 0.0; }

// Sign-flips v where the word d has its top bit set. The Cartesian and octree walkers mirror every
// axis along which the ray moves downwards, so that a ray always moves towards the upper walls: a
// wall distance, a position update and a containment test then need no choice by the direction's
// sign. Negation is exact and rounding to nearest is symmetric, so a mirrored walk takes the same
// steps bit for bit.
SKG_D double mirror(double v, unsigned d)
{
    return __hiloint2double(__double2hiint(v) ^ static_cast<int>(d & 0x80000000u), __double2loint(v));
}

// state shared by the walkers over axis-aligned cells, in mirrored coordinates once inside
struct BoxWalker : GenBase
{
    double xE, yE, zE;  // exit walls of the current cell

    // the ray's reciprocal direction lives in a per-thread shared-memory slot (blocks of at most
    // 256 threads): six registers less per thread. Of the FP32 kernels at four blocks per SM (64 registers)
    // the Cartesian ones then spill nothing, the octree's 20 (peel-off rays) to 64 bytes (forced paths).
    static constexpr size_t kSharedBytes = 3 * 256 * sizeof(double);
    SKG_D static double* recip()
    {
        __shared__ double slots[kSharedBytes / (256 * sizeof(double))][256];
        return &slots[0][threadIdx.x];
    }

    SKG_D void startBox(double x, double y, double z, double ux, double uy, double uz)
    {
        startRay(x, y, z, ux, uy, uz);
        double* ik = recip();
        ik[0] = recipDir(fabs(ux));
        ik[256] = recipDir(fabs(uy));
        ik[512] = recipDir(fabs(uz));
    }

    // the reference's wall distance (wall - r) / k, or DBL_MAX for a direction component that is
    // not usable (ik = 0)
    SKG_D static double exitDist(double wall, double r, double k, double ik)
    {
        double d = qdiv(xsub(wall, r), k, ik);
        return __double2hiint(ik) != 0 ? d : DBL_MAX;
    }

    // the nearest exit wall: its distance, whether it is not the z wall, and if so whether it is the
    // x wall (the reference's order on ties: x before y before z)
    SKG_D void nearest(double& d, bool& xy, bool& x) const
    {
        const double* ik = recip();
        double dsx = exitDist(xE, rx, kx, ik[0]);
        double dsy = exitDist(yE, ry, ky, ik[256]);
        double dsz = exitDist(zE, rz, kz, ik[512]);
        x = dsx <= dsy;
        d = x ? dsx : dsy;
        xy = d <= dsz;
        d = xy ? d : dsz;
    }
};

// ---------------------------------------------------------------------------------------------
// Cartesian grid (CartesianSpatialGrid::MySegmentGenerator::next, CartesianSpatialGrid.cpp:77-155):
// the reference's steps with the quotient from the reciprocal direction, in mirrored coordinates. The
// exit walls stay in registers; a crossing reads the next wall of its own axis only, which for either
// direction is the next entry of one table (GridDev::cWall), and takes no branch by axis.
// ---------------------------------------------------------------------------------------------
template<class A>
struct CartesianT : BoxWalker
{
    using Acc = A;
    static constexpr int kMinBlocks = std::is_same<A, float>::value ? 4 : 3;
    static constexpr int kRefillMin = 16;  // waiting lanes before a warp takes new tasks
    int ix, iy, iz;  // table index of the exit wall of each axis
    int cx, cy, cz;  // what a crossing of each axis adds to the cell index
    int cell;

    SKG_D void start(const GridDev&, double x, double y, double z, double ux, double uy, double uz, int = -1)
    {
        startBox(x, y, z, ux, uy, uz);
    }

    // mirrors one axis of n cells and finds its exit wall: i the current cell, table the axis's upward
    // walls (n + 2 entries), after which its downward ones follow
    SKG_D static void turn(const GridDev& g, int table, int n, int i, double& r, double& k, double& wall, int& index, int& step)
    {
        const bool down = k < 0.0;
        index = table + (down ? 2 * n + 2 - i : i + 1);
        wall = __ldg(g.cWall + index);
        step = down ? -step : step;
        r = down ? -r : r;
        k = fabs(k);
    }

    SKG_D bool next(const GridDev& g)
    {
        if (state != GS_INSIDE)
        {
            if (state == GS_OUTSIDE) return false;
            if (!moveInside(g.ext, g.eps)) return false;
            int i = locateClip(g.xb, g.nx + 1, rx);
            int j = locateClip(g.yb, g.ny + 1, ry);
            int k = locateClip(g.zb, g.nz + 1, rz);
            cx = g.nz * g.ny;
            cy = g.nz;
            cz = 1;
            cell = k * cz + j * cy + i * cx;
            turn(g, 0, g.nx, i, rx, kx, xE, ix, cx);
            turn(g, 2 * g.nx + 4, g.ny, j, ry, ky, yE, iy, cy);
            turn(g, 2 * (g.nx + g.ny) + 8, g.nz, k, rz, kz, zE, iz, cz);
            if (ds > 0.) return true;
        }
        double d;
        bool xy, x;
        nearest(d, xy, x);
        m = cell;
        ds = d;
        const bool ax = xy && x, ay = xy && !x;
        rx = ax ? xE : xadd(rx, xmul(kx, d));
        ry = ay ? yE : xadd(ry, xmul(ky, d));
        rz = xy ? xadd(rz, xmul(kz, d)) : zE;
        const int index = (ax ? ix : (ay ? iy : iz)) + 1;
        const double wall = __ldg(g.cWall + index);
        cell += ax ? cx : (ay ? cy : cz);
        xE = ax ? wall : xE;
        yE = ay ? wall : yE;
        zE = xy ? zE : wall;
        ix = ax ? index : ix;
        iy = ay ? index : iy;
        iz = xy ? iz : index;
        if (isnan(wall)) state = GS_OUTSIDE;  // past the last wall
        return true;
    }
};

// ---------------------------------------------------------------------------------------------
// Octree (TreeSpatialGrid::MySegmentGenerator::next, TreeSpatialGrid.cpp:143-228,
// TreeNode::neighbor, TreeNode.cpp:103-112), in mirrored coordinates. The reference takes the first
// neighbour across the exit wall, in overlap order, whose closed box contains the new position
// (Box::contains). Here:
//  - a wall with a single positive-overlap neighbour: that neighbour's face covers the whole wall,
//    and since entering the current cell (whose closed box held the position) the position has only
//    moved towards the cell's exit walls; so the neighbour contains it exactly when it lies at or
//    beyond the crossed wall and not beyond the other two exit walls: comparisons with the FP64
//    exit walls held in registers (on the crossed axis the neighbour's far wall is at least one
//    finest cell away, far beyond the eps step);
//  - a wall with several neighbours, or a position past a corner: each candidate's six FP64 walls
//    from the FP64 lattice tables, indexed by its record's 16-bit wall indices;
//  - otherwise the reference's complete procedure on the FP64 node arrays: the wall's full neighbour
//    list, the top-down search, the nextafter escape.
// Entering a cell reads its exit walls from the lattice tables. A start in a known cell (a
// scattering event's interaction cell) skips the top-down search when the top-down search would
// return that cell (half-open bounds).
// ---------------------------------------------------------------------------------------------
#ifndef SKG_OCTREE_MIN_BLOCKS
#define SKG_OCTREE_MIN_BLOCKS 4
#endif

template<class A>
struct OctreeT : BoxWalker
{
    using Acc = A;
    static constexpr bool kSingle = std::is_same<A, float>::value;
    static constexpr int kMinBlocks = kSingle ? SKG_OCTREE_MIN_BLOCKS : 3;
    static constexpr int kRefillMin = 16;  // waiting lanes before a warp takes new tasks
    // Per axis: in the low half the byte selector that picks the exit wall's 16-bit index out of a
    // record word (upper half of the word for an upward axis, lower half for a downward one), in the
    // top bit whether the axis is mirrored.
    static constexpr unsigned kUp = 0x4432u, kDown = 0x80004410u, kOther = 0x22u;
    unsigned wx, wy, wz;
    int cell;             // the current cell; before the first step the start cell when
                          // the caller knows it (an interaction cell), else -1
    A cellDens, segDens;  // density of the current cell / of the segment just returned

    SKG_D void start(const GridDev&, double x, double y, double z, double ux, double uy, double uz, int h = -1)
    {
        startBox(x, y, z, ux, uy, uz);
        cell = h;
    }

    SKG_D double density(const double*) const { return static_cast<double>(segDens); }

    static constexpr bool kLocates = true;
    SKG_D static int locate(const GridDev& g, double x, double y, double z)
    {
        int n = octreeLeafChild(g, x, y, z);
        return n < 0 ? -1 : g.tCell[n];
    }

    // the wall of a record word that the selector picks, mirrored with its axis
    SKG_D static double wall(const GridDev& g, int axis, int word, unsigned sel)
    {
        return mirror(__ldg(g.tWall + axis * g.tWallN + __byte_perm(word, 0, sel)), sel);
    }

    SKG_D static double wallAt(const GridDev& g, int axis, unsigned idx) { return __ldg(g.tWall + axis * g.tWallN + idx); }

    // makes c, whose record starts with w0, the current cell
    SKG_D void become(const GridDev& g, int c, int4 w0)
    {
        cell = c;
        if constexpr (kSingle)
            cellDens = __int_as_float(w0.w);
        else
            cellDens = __ldg(reinterpret_cast<const double*>(g.tRec + 4 * static_cast<size_t>(c) + 3) + 1);
        xE = wall(g, 0, w0.x, wx);
        yE = wall(g, 1, w0.y, wy);
        zE = wall(g, 2, w0.z, wz);
    }

    // enters c, whose closed box is known to hold the position
    SKG_D void enter(const GridDev& g, int c) { become(g, c, __ldg(g.tRec + 4 * static_cast<size_t>(c))); }

    // Box::contains (closed bounds) of cell c; on success c becomes the current cell
    SKG_D bool tryEnter(const GridDev& g, int c)
    {
        int4 w0 = __ldg(g.tRec + 4 * static_cast<size_t>(c));
        bool in = rx <= wall(g, 0, w0.x, wx) && rx >= wall(g, 0, w0.x, wx ^ kOther) && ry <= wall(g, 1, w0.y, wy)
                  && ry >= wall(g, 1, w0.y, wy ^ kOther) && rz <= wall(g, 2, w0.z, wz) && rz >= wall(g, 2, w0.z, wz ^ kOther);
        if (in) become(g, c, w0);
        return in;
    }

    // whether the top-down search (TreeNode::leafChild with OctTreeNode::child: lower half for
    // coordinates below the centre) would return cell c: lo <= r < hi per axis, or r on the domain's
    // upper wall (unmirrored position)
    SKG_D bool holds(const GridDev& g, int c) const
    {
        int4 w0 = __ldg(g.tRec + 4 * static_cast<size_t>(c));
        auto axis = [&](int a, int w, double r) {
            double lo = wallAt(g, a, static_cast<unsigned>(w) & 0xFFFFu), hi = wallAt(g, a, static_cast<unsigned>(w) >> 16);
            return r >= lo && (r < hi || (r == hi && hi == g.ext[3 + a]));
        };
        return axis(0, w0.x, rx) && axis(1, w0.y, ry) && axis(2, w0.z, rz);
    }

    SKG_D static unsigned turn(double& r, double& k)
    {
        const unsigned w = k < 0.0 ? kDown : kUp;
        r = mirror(r, w);
        k = fabs(k);
        return w;
    }

    SKG_D int leafAt(const GridDev& g) const { return octreeLeafChild(g, mirror(rx, wx), mirror(ry, wy), mirror(rz, wz)); }

    SKG_D bool next(const GridDev& g)
    {
        if (state != GS_INSIDE)
        {
            if (state == GS_OUTSIDE) return false;
            if (!moveInside(g.ext, g.eps)) return false;
            if (!(cell >= 0 && ds == 0. && holds(g, cell)))
            {
                cell = locate(g, rx, ry, rz);
                if (cell < 0)
                {
                    state = GS_OUTSIDE;
                    return false;
                }
            }
            wx = turn(rx, kx);
            wy = turn(ry, ky);
            wz = turn(rz, kz);
            enter(g, cell);
            if (ds > 0.) return true;
        }
        double d;
        bool xy, x;
        nearest(d, xy, x);
        propagater(xadd(d, g.eps));
        m = cell;
        ds = d;
        segDens = cellDens;
        const int old = cell;
        // exit wall index: 2 * axis, +1 when the ray moves towards the upper wall
        const int wl = (xy ? (x ? 1 : 3) : 5) - static_cast<int>((xy ? (x ? wx : wy) : wz) >> 31);
        const int* R = reinterpret_cast<const int*>(g.tRec + 4 * static_cast<size_t>(old));
        int one = __ldg(R + 8 + wl);
        // single neighbour: at or beyond the crossed exit wall, within the other two
        const bool ox = rx <= xE, oy = ry <= yE, oz = rz <= zE;
        const bool inOne = xy ? (x ? rx >= xE && oy && oz : ox && ry >= yE && oz) : ox && oy && rz >= zE;
        bool found = false;
        if (one >= 0 && inOne)
        {
            enter(g, one);
            found = true;
        }
        else if (one >= 0)
        {
            found = tryEnter(g, one);
        }
        else if (one == -2)
        {
            unsigned long long cnt = (static_cast<unsigned long long>(static_cast<unsigned>(__ldg(R + 6))) << 32)
                                     | static_cast<unsigned>(__ldg(R + 5));
            if (cnt != ~0ULL)
            {
                int base = __ldg(R + 4);
                int e0 = base + static_cast<int>((cnt >> (9 * wl)) & 511);
                int e1 = base + static_cast<int>((cnt >> (9 * (wl + 1))) & 511);
                for (int e = e0; e < e1 && !found; ++e) found = tryEnter(g, __ldg(g.tLeafNb + e));
            }
        }
        if (!found)
        {
            // the reference's complete procedure on the FP64 node arrays: the wall's full neighbour
            // list in overlap order, the top-down search, the nextafter escape
            int node = __ldg(R + 7);
            int nb = -1;
            int e1 = g.tNbBegin[6 * node + wl + 1];
            for (int e = g.tNbBegin[6 * node + wl]; e < e1; ++e)
            {
                int cand = g.tNb[e];
                if (boxContains(g.tBounds + 6 * static_cast<size_t>(cand), mirror(rx, wx), mirror(ry, wy), mirror(rz, wz)))
                {
                    nb = cand;
                    break;
                }
            }
            if (nb < 0) nb = leafAt(g);
            if (nb == node)
            {
                rx = nextafter(rx, DBL_MAX);
                ry = nextafter(ry, DBL_MAX);
                rz = nextafter(rz, DBL_MAX);
                nb = leafAt(g);
            }
            if (nb < 0 || nb == node)
                state = GS_OUTSIDE;
            else
                enter(g, g.tCell[nb]);
        }
        return true;
    }
};

// Octree, production precision for trees that are not a lattice of depth <= 15 (no leaf records):
// the FP64 node walker with FP32 accumulators
struct OctreeNodeFast : OctreeExact
{
    using Acc = float;
};

// Adaptive mesh, production: the reference-order FP64 walk (single neighbour per wall, top-down
// fallback) with FP32 accumulators
struct AdaptiveMeshFast : AdaptiveMeshExact
{
    using Acc = float;
};

// Nearest site of a point by a greedy walk on the neighbour graph (the Delaunay graph of the sites,
// on which the walk towards ever nearer sites ends at the nearest one), starting from the
// representative site of the point's block in the site-search grid. -1 outside the domain.
SKG_D int voronoiLocate(const GridDev& g, double x, double y, double z)
{
    if (!GenBase::boxContains(g.ext, x, y, z)) return -1;
    const int n = g.vGridN;
    auto blk = [&](double v, double lo, double hi) {
        return min(n - 1, max(0, static_cast<int>((v - lo) / ((hi - lo) / n))));
    };
    int c = g.vBlkRep[(blk(x, g.ext[0], g.ext[3]) * n + blk(y, g.ext[1], g.ext[4])) * n + blk(z, g.ext[2], g.ext[5])];
    for (int guard = 0; guard < 100000; ++guard)
    {
        const double* p = g.vSites + 3 * static_cast<size_t>(c);
        double best = (p[0] - x) * (p[0] - x) + (p[1] - y) * (p[1] - y) + (p[2] - z) * (p[2] - z);
        int next = -1;
        for (int e = g.vNbBegin[c]; e < g.vNbBegin[c + 1]; ++e)
        {
            int j = __ldg(g.vNb + e);
            if (j < 0) continue;
            const double* q = g.vSites + 3 * static_cast<size_t>(j);
            double d = (q[0] - x) * (q[0] - x) + (q[1] - y) * (q[1] - y) + (q[2] - z) * (q[2] - z);
            if (d < best)
            {
                best = d;
                next = j;
            }
        }
        if (next < 0) return c;
        c = next;
    }
    return c;
}

// ---------------------------------------------------------------------------------------------
// Voronoi mesh, production walker (VoronoiMeshSnapshot::MySegmentGenerator::next,
// VoronoiMeshSnapshot.cpp:1089-1222). Each cell is one contiguous record in 16-byte units:
//   [0] site x, y (FP64)   [1] site z (FP64), cell index, face count n
//   then per group of four faces five units: for each face the outward unit normal n and the
//   distance d of the face's plane from the site (half the site distance, or the distance to a domain
//   wall), and the four neighbours' record offsets (16-byte units), or the wall id -1..-6, or kPad
// (padding faces have n = 0 and are never ahead). A crossing reads one record and takes the next cell's offset from it: no index arrays between
// cells. On entering a cell the FP64 position is rebased to FP32 coordinates l relative to the
// site; the exit through a face is s = (d - n . l) / (n . k). The two smallest exits are
// re-decided in FP64 from the exact sites when they lie within a near-tie tolerance (FP32 would
// misorder near-degenerate faces). The face just crossed is skipped (a ray cannot re-enter a convex
// cell), and a cell without a positive exit falls back to the reference's eps step and an FP64
// nearest-site search. A start in a known cell (a scattering event's interaction cell) needs no
// search; other starts walk greedily over the Delaunay neighbours from a site of the search block.
// ---------------------------------------------------------------------------------------------
struct VoronoiRec32 : GenBase
{
    using Acc = float;
    // Two blocks per SM and 128 registers for the two groups of faces in flight: the walk waits on
    // loads, not on warps (galaxy on 1e5 sites, 2e6 packets: 150 ms; three blocks 166 ms, four 199 ms)
    static constexpr int kMinBlocks = 2;
    static constexpr int kRefillMin = 8;  // waiting lanes before a warp takes new tasks
    static constexpr int kNone = -99;     // no previous cell, no exit (the wall ids -1..-6 are taken)
    static constexpr int kPad = -100;     // padding face
    int rec, prev;                        // record offsets of the current and the previous cell
    float kxf, kyf, kzf;
    int hint;                             // the start cell when the caller knows it, else -1

    SKG_D void start(const GridDev&, double x, double y, double z, double ux, double uy, double uz, int h = -1)
    {
        startRay(x, y, z, ux, uy, uz);
        hint = h;
        rec = -1;
        prev = kNone;
        kxf = static_cast<float>(ux);
        kyf = static_cast<float>(uy);
        kzf = static_cast<float>(uz);
    }

    SKG_D static void site(const GridDev& g, int r, double& x, double& y, double& z)
    {
        const double* h = reinterpret_cast<const double*>(g.vRec + r);
        x = __ldg(h);
        y = __ldg(h + 1);
        z = __ldg(h + 2);
    }

    // FP64 exit distance from the current position through the face towards `to` (a record offset
    // or a wall id) of the cell with site p (0 when the face is not ahead)
    SKG_D double exit64(const GridDev& g, double px, double py, double pz, int to) const
    {
        if (to >= 0)
        {
            double qx, qy, qz;
            site(g, to, qx, qy, qz);
            double nx = qx - px, ny = qy - py, nz = qz - pz;
            double nk = nx * kx + ny * ky + nz * kz;
            if (!(nk > 0)) return 0.;
            return (nx * (0.5 * (qx + px) - rx) + ny * (0.5 * (qy + py) - ry) + nz * (0.5 * (qz + pz) - rz)) / nk;
        }
        switch (to)
        {
            case -1: return (g.ext[0] - rx) / kx;
            case -2: return (g.ext[3] - rx) / kx;
            case -3: return (g.ext[1] - ry) / ky;
            case -4: return (g.ext[4] - ry) / ky;
            case -5: return (g.ext[2] - rz) / kz;
            case -6: return (g.ext[5] - rz) / kz;
        }
        return 0.;
    }

    static constexpr bool kLocates = true;
    SKG_D static int locate(const GridDev& g, double x, double y, double z) { return voronoiLocate(g, x, y, z); }

    SKG_D bool locateRec(const GridDev& g, int cellHint)
    {
        int c = cellHint >= 0 ? cellHint : voronoiLocate(g, rx, ry, rz);
        rec = c >= 0 ? __ldg(g.vRecOff + c) : -1;
        prev = kNone;
        return rec >= 0;
    }

    SKG_D bool next(const GridDev& g)
    {
        if (state != GS_INSIDE)
        {
            if (state == GS_OUTSIDE) return false;
            if (!moveInside(g.ext, g.eps)) return false;
            if (!locateRec(g, (hint >= 0 && ds == 0.) ? hint : -1))
            {
                state = GS_OUTSIDE;
                return false;
            }
            if (ds > 0.) return true;
        }
        for (int guard = 0; guard < 64; ++guard)
        {
            // the loads of a group of faces are issued together, and those of the next group before the
            // present one is worked on: the walk waits on record loads that miss L1 more than on anything
            // else
            const float4* R = g.vRec + rec;
            float4 h0 = __ldg(R), h1 = __ldg(R + 1);
            const float4* E = R + 2;
            float4 q[4] = {__ldg(E), __ldg(E + 1), __ldg(E + 2), __ldg(E + 3)};
            float4 ids = __ldg(E + 4);
            // the FP64 site only rebases the position here (the near-tie branch reloads it)
            float lx = static_cast<float>(rx - __hiloint2double(__float_as_int(h0.y), __float_as_int(h0.x)));
            float ly = static_cast<float>(ry - __hiloint2double(__float_as_int(h0.w), __float_as_int(h0.z)));
            float lz = static_cast<float>(rz - __hiloint2double(__float_as_int(h1.y), __float_as_int(h1.x)));
            int cell = __float_as_int(h1.z);
            const int n = __float_as_int(h1.w);
            // the two nearest exits me / nk, compared by cross-multiplication so that only those two
            // distances take a division, without branches (a face is ahead or not as good as at random, so
            // that a branch leaves half the lanes idle); none yet is the fraction inf / 1
            float meB = INFINITY, nkB = 1.f, meS = INFINITY, nkS = 1.f, scale = 0.f;
            int ib = kNone, is = kNone;
            for (int c = n;;)
            {
                float4 qn[4], idn;
                c -= 4;
                E += 5;
                if (c > 0)
                {
                    qn[0] = __ldg(E);
                    qn[1] = __ldg(E + 1);
                    qn[2] = __ldg(E + 2);
                    qn[3] = __ldg(E + 3);
                    idn = __ldg(E + 4);
                }
                const int id[4] = {__float_as_int(ids.x), __float_as_int(ids.y), __float_as_int(ids.z), __float_as_int(ids.w)};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    const float nk = q[j].x * kxf + q[j].y * kyf + q[j].z * kzf;
                    const float me = q[j].w - (q[j].x * lx + q[j].y * ly + q[j].z * lz);
                    const bool ahead = (nk > 0.f) & (me > 0.f) & (id[j] != prev);
                    const bool b = ahead & (me * nkB < meB * nk);
                    const bool s = ahead & (me * nkS < meS * nk);
                    meS = b ? meB : (s ? me : meS);
                    nkS = b ? nkB : (s ? nk : nkS);
                    is = b ? ib : (s ? id[j] : is);
                    meB = b ? me : meB;
                    nkB = b ? nk : nkB;
                    ib = b ? id[j] : ib;
                    scale = b ? q[j].w : scale;
                }
                if (c <= 0) break;
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] = qn[j];
                ids = idn;
            }
            if (ib == kNone)
            {
                // no exit ahead (the point sits on an edge or slightly outside the cell): the
                // reference's eps step and a fresh nearest-site search
                propagater(g.eps);
                if (!locateRec(g, -1))
                {
                    state = GS_OUTSIDE;
                    return false;
                }
                continue;
            }
            const float best = meB / nkB, second = is != kNone ? meS / nkS : FLT_MAX;
            double sq = best;
            if (is != kNone && second - best <= 2e-5f * (best + scale))
            {
                // near tie: decide with the exact FP64 sites
                double px, py, pz;
                site(g, rec, px, py, pz);
                double s1 = exit64(g, px, py, pz, ib), s2 = exit64(g, px, py, pz, is);
                if (s2 > 0. && (s2 < s1 || !(s1 > 0.)))
                {
                    ib = is;
                    sq = s2;
                }
                else if (s1 > 0.)
                {
                    sq = s1;
                }
            }
            m = cell;
            ds = sq;
            propagater(sq);
            prev = rec;
            rec = ib;
            if (rec < 0) state = GS_OUTSIDE;
            return true;
        }
        state = GS_OUTSIDE;
        return false;
    }
};


// 32 bytes of read-only memory in one load. A gather of records costs the L1 a wavefront per lane and
// load, whatever the load's size: half as many loads of twice the size.
SKG_D void load32(const void* p, unsigned (&v)[8])
{
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// ---------------------------------------------------------------------------------------------
// Tetrahedral mesh, production walker (TetraMeshSpatialGrid::MySegmentGenerator::next,
// TetraMeshSpatialGrid.cpp:688-831). Every step reads one 128-byte record (TetRec) of the current
// tetrahedron: the exit is the nearest face plane ahead, s_f = (c_f - n_f . r) / (n_f . k) over the
// faces with n_f . k > 0 other than the face just entered (a ray cannot re-enter a convex cell),
// with the plane offset difference in FP64 and the division in FP32. Shared faces are one plane
// seen from both sides, so the walk stays watertight. The float planes are tilted from the exact
// ones by up to ~1e-7 of a tetrahedron's size; a decision within that bound of an edge, a vertex or
// a tie between two faces is re-taken in FP64 by the reference's Plucker decision (teLeavingFace),
// so that the cell sequence is the reference's.
// As the reference, the last in-mesh segment is dropped when the path leaves the hull. A start at a
// known cell (a scattering event's interaction cell) needs no point location; otherwise a walk over
// the face planes from the search block's representative finds the containing tetrahedron.
// ---------------------------------------------------------------------------------------------
// a record in registers (the fields are picked with selects, never by a dynamic index, so that the
// record stays out of local memory)
struct TetRegs
{
    double c[4];
    float n[12];
    int to[4];

    SKG_D static TetRegs load(const TetRec* rec)
    {
        unsigned v[8], u[8], t8[8];
        load32(rec->c, v);
        load32(rec->n, u);
        load32(rec->n + 8, t8);
        TetRegs t;
#pragma unroll
        for (int f = 0; f < 4; ++f)
        {
            t.c[f] = __hiloint2double(v[2 * f + 1], v[2 * f]);
            t.n[8 + f] = __uint_as_float(t8[f]);
            t.to[f] = static_cast<int>(t8[4 + f]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) t.n[i] = __uint_as_float(u[i]);
        return t;
    }

    // TetRec::to of face f
    SKG_D int across(int f) const { return f == 0 ? to[0] : f == 1 ? to[1] : f == 2 ? to[2] : to[3]; }

    // positive when (x, y, z) lies outside face F's plane
    template<int F>
    SKG_D double excess(double x, double y, double z) const
    {
        return static_cast<double>(n[3 * F]) * x + static_cast<double>(n[3 * F + 1]) * y + static_cast<double>(n[3 * F + 2]) * z - c[F];
    }
};

SKG_D int tetraLocate(const GridDev& g, double x, double y, double z)
{
    if (!GenBase::boxContains(g.ext, x, y, z)) return -1;
    const int n = g.teGridN;
    auto blk = [&](double v, double lo, double hi) {
        return min(n - 1, max(0, static_cast<int>(n * (v - lo) / (hi - lo))));
    };
    int t = g.teBlkRep[(blk(x, g.ext[0], g.ext[3]) * n + blk(y, g.ext[1], g.ext[4])) * n + blk(z, g.ext[2], g.ext[5])];
    // visibility walk: cross the face whose plane the point is farthest outside of
    for (int guard = 0; guard < 4096 && t >= 0; ++guard)
    {
        TetRegs r = TetRegs::load(g.teRec + t);
        int f = -1;
        double worst = 0., e;
        if ((e = r.excess<0>(x, y, z)) > worst) { worst = e; f = 0; }
        if ((e = r.excess<1>(x, y, z)) > worst) { worst = e; f = 1; }
        if ((e = r.excess<2>(x, y, z)) > worst) { worst = e; f = 2; }
        if ((e = r.excess<3>(x, y, z)) > worst) { worst = e; f = 3; }
        if (f < 0) return t;
        t = r.across(f) >> 2;
    }
    return tetraCellIndex(g, x, y, z);  // walk left the hull or did not settle: the reference's block scan
}

#ifndef SKG_TETRA32_MIN_BLOCKS
#define SKG_TETRA32_MIN_BLOCKS 3
#endif
struct TetraPlane32 : GenBase
{
    using Acc = float;
    static constexpr int kMinBlocks = SKG_TETRA32_MIN_BLOCKS;
    static constexpr bool kEndsOutside = true;
    static constexpr int kRefillMin = 8;  // waiting lanes before a warp takes new tasks
    // bound on the displacement of a float plane from its exact one, in units of eps (1e-12 of the
    // domain diagonal): 2^-24 per normal component over at most the diagonal, with margin
    static constexpr double kTilt = 1.6e5;
    static constexpr float kNk = 1e-6f;  // |n.k| below this may have either sign in exact arithmetic
    int mr, ef;  // current tetrahedron, face it was entered through (-1: none)
    int hint;
    float kxf, kyf, kzf;

    SKG_D void start(const GridDev&, double x, double y, double z, double ux, double uy, double uz, int h = -1)
    {
        startRay(x, y, z, ux, uy, uz);
        hint = h;
        mr = -1;
        ef = -1;
        kxf = static_cast<float>(ux);
        kyf = static_cast<float>(uy);
        kzf = static_cast<float>(uz);
    }

    static constexpr bool kLocates = true;
    SKG_D static int locate(const GridDev& g, double x, double y, double z) { return tetraLocate(g, x, y, z); }

    // whether the float exit decision in tetrahedron r may differ from the exact one: the point lies
    // within tol of the exit plane, the two nearest exits lie within the planes' error of each other
    // (an edge or a vertex), or a face almost parallel to the path lies within tol of the point
    SKG_D bool ambiguous(const TetRegs& r, double x, double y, double z, float tol) const
    {
        float best = FLT_MAX, second = FLT_MAX, nkBest = 1.f, nkSecond = 1.f;
        float inside = FLT_MAX, graze = FLT_MAX;
        auto face = [&](auto F) {
            constexpr int f = decltype(F)::value;
            if (f == ef) return;
            float nk = r.n[3 * f] * kxf + r.n[3 * f + 1] * kyf + r.n[3 * f + 2] * kzf;
            float me = static_cast<float>(-r.template excess<f>(x, y, z));
            if (!(nk > 0.f))
            {
                if (nk > -kNk) graze = fminf(graze, me);  // may be a face ahead in exact arithmetic
                return;
            }
            float s = me / nk;
            if (s < best)
            {
                second = best;
                nkSecond = nkBest;
                best = s;
                nkBest = nk;
                inside = me;
            }
            else if (s < second)
            {
                second = s;
                nkSecond = nk;
            }
        };
        face(std::integral_constant<int, 0>());
        face(std::integral_constant<int, 1>());
        face(std::integral_constant<int, 2>());
        face(std::integral_constant<int, 3>());
        // second - best < tol (1/nkBest + 1/nkSecond) + 1e-6 second, multiplied through by the
        // positive nkBest nkSecond (the bound is far coarser than the rounding of the test)
        return inside < tol || graze < tol + 1e-6f * best ||
               (second < FLT_MAX &&
                (second - best) * nkBest * nkSecond < tol * (nkBest + nkSecond) + 1e-6f * second * nkBest * nkSecond);
    }

    SKG_D bool next(const GridDev& g)
    {
        if (state != GS_INSIDE)
        {
            if (state == GS_OUTSIDE) return false;
            if (!moveInside(g.ext, g.eps)) return false;
            mr = (hint >= 0 && ds == 0.) ? hint : tetraLocate(g, rx, ry, rz);
            ef = -1;
            if (mr < 0)
            {
                state = GS_OUTSIDE;
                return false;
            }
            if (ds > 0.) return true;
        }
        // the float planes (normals rounded to FP32, offsets through a shared vertex, so neighbours
        // agree) lie within kTilt * eps = 1.6e-7 of the domain diagonal of the exact ones
        const float tol = static_cast<float>(kTilt * g.eps);
        for (int guard = 0; guard < 256; ++guard)
        {
            TetRegs r = TetRegs::load(g.teRec + mr);
            // the nearest exit me / nk over the faces ahead (nk > 0), compared by cross-multiplication
            // so that only the chosen face's distance takes a division
            float meBest = 0.f, nkBest = 1.f;
            int lf = -1;
            auto face = [&](auto F) {
                constexpr int f = decltype(F)::value;
                float nk = r.n[3 * f] * kxf + r.n[3 * f + 1] * kyf + r.n[3 * f + 2] * kzf;
                if (f == ef || !(nk > 0.f)) return;
                float me = static_cast<float>(-r.template excess<f>(rx, ry, rz));
                if (lf < 0 || me * nkBest < meBest * nk)
                {
                    meBest = me;
                    nkBest = nk;
                    lf = f;
                }
            };
            face(std::integral_constant<int, 0>());
            face(std::integral_constant<int, 1>());
            face(std::integral_constant<int, 2>());
            face(std::integral_constant<int, 3>());
            const float best = lf >= 0 ? meBest / nkBest : FLT_MAX;
            // Between two interior faces either choice continues the walk from the same point; only
            // in a tetrahedron on the hull can a float decision end the path where the reference's
            // goes on (or the reverse), so only there is the decision tested, in a second pass.
            if (lf >= 0 && ((r.to[0] | r.to[1] | r.to[2] | r.to[3]) >= 0 || !ambiguous(r, rx, ry, rz, tol)))
            {
                const int to = r.across(lf);
                if (best > 0.f)
                {
                    m = mr;
                    ds = best;
                    propagater(ds);
                }
                mr = to >> 2;
                ef = to & 3;
                if (mr < 0)
                {
                    // the reference drops the final in-mesh segment when the path leaves the hull
                    state = GS_OUTSIDE;
                    return false;
                }
                if (best > 0.f) return true;
                continue;
            }
            // no face ahead, or a decision within the float planes' error of an edge, a vertex or a
            // tie: re-taken in FP64 the reference's way
            double d;
            int xf = teLeavingFace(g, mr, ef, rx, ry, rz, kx, ky, kz, d);
            if (xf == -1 || d < g.eps)
            {
                // no exit point: the reference's eps step and its own point location
                propagater(g.eps);
                mr = tetraCellIndex(g, rx, ry, rz);
                ef = -1;
                if (mr < 0)
                {
                    state = GS_OUTSIDE;
                    return false;
                }
                continue;
            }
            m = mr;
            ds = d;
            propagater(d);
            ef = g.teNFace[4 * static_cast<size_t>(mr) + xf];
            mr = g.teNTet[4 * static_cast<size_t>(mr) + xf];
            if (mr < 0)
            {
                state = GS_OUTSIDE;
                return false;
            }
            return true;
        }
        state = GS_OUTSIDE;
        return false;
    }
};

// ---------------------------------------------------------------------------------------------
// 1D spherical grid, production: the reference-order FP64 shell crossings (a handful of square
// roots per ray over a border table that stays in L1) with FP32 accumulators like the other
// production walkers.
// ---------------------------------------------------------------------------------------------
struct Sphere1DFast : Sphere1DExact
{
    using Acc = float;
};

// 2D cylindrical grid, production: the reference-order FP64 crossings with FP32 accumulators
struct Cylinder2DFast : Cylinder2DExact
{
    using Acc = float;
};

// 2D spherical grid, production: the reference-order FP64 crossings with FP32 accumulators
struct Sphere2DFast : Sphere2DExact
{
    using Acc = float;
};

// 3D spherical grid, production: the reference-order FP64 crossings with FP32 accumulators
struct Sphere3DFast : Sphere3DExact
{
    using Acc = float;
};

// 3D cylindrical grid, production: the reference-order FP64 crossings with FP32 accumulators
struct Cylinder3DFast : Cylinder3DExact
{
    using Acc = float;
};

}  // namespace skg
