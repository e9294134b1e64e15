// gvx_splat.cu -- point -> brick-atlas splats.
//
// Modes
//   TRILINEAR, CUBIC (no reference counterpart): one warp per unit, a z-slab of an
//     active PADDED brick or the whole brick, PULLS the points of the brick's 27-neighbourhood
//     (points are grouped by brick by the topology sort), keeps those whose
//     footprint reaches its slab, and adds them into a shared-memory copy of
//     the slab in their global sorted order, one point at a time across the
//     warp's lanes.  Every voxel is therefore the same sum, added in the same
//     order, in the brick that owns it and in the bricks that hold it as an
//     apron voxel: the splat writes interior and apron together, the apron
//     bit-identical to the neighbours' interior (UpdateApron's copy
//     semantics), with no atomics, deterministically, and one bulk (TMA) store
//     per channel and slab.
//   REF_SCATTER: ScatterDensity semantics (gvdb_volume_gvdb.cpp:5624-5660,
//     cuda_gvdb_particles.cuh:516-573): (1 - d^2/r^2)^3 at the point's voxel
//     and its 6 face neighbours, inside the point's own padded brick, summed
//     by reductions in L2 (bricks of few points) or in shared memory instead of the reference's racy surface
//     read-modify-write.
//
// Sample convention of all modes: voxel v of the index space is sampled at the
// integer coordinate v (as gvdbGatherDensity, cuda_gvdb_particles.cuh:705).
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <map>
#include <atomic>
#include <mutex>
#include <thread>
#include <string>
#include <vector>

#include "gvx_grid.cuh"
#include "gvx_ptx.cuh"

namespace {
constexpr int kSplatThreads = 256;
constexpr int kTriWarps = 4;                // warps (brick slabs) per block of k_splat_tri
// resident blocks per SM its registers are budgeted for: 24 clouds' splat 2.63 ms at 8 (64 registers, 200
// bytes of spill), 2.37 at 7, 1.97 at 6, 2.12 at 5
constexpr int kTriMinBlocks = 6;
constexpr size_t kSlabTileMax = 48 * 1024;  // shared tile bytes of one warp at most
constexpr int kBatchMaxGrids = 256;         // grids of one batched launch
constexpr float kInvPi = 0.318309886183790671538f;
constexpr uint32_t kFull = 0xFFFFFFFFu;
}  // namespace

// the cell order of the dense leaves (k_cell_sort), for positions read again under the same grouping; leaf_dense
// null: there is none
struct CellOrder {
    const uint32_t* skeys;  // leaf key << 3 | octant
    uint32_t invalid_key;
    LeafLookup L;
    const GvxNode* nodes0;
    const int2* leaf_range;
    const int* cell_tab;
    int* leaf_dense;
};

// sorted point attributes: (x, y, z, weight) and (vx, vy, vz, radius); with
// per-point radii also the largest radius (float bits, NaN counted as huge).  A leaf with a point that is not
// in the cell it was sorted into (its position was written in place since) loses its dense number: k_tri_dense
// takes a point to be in its cell
__global__ void k_permute(const uint32_t* __restrict__ svals, uint32_t n, const char* pos, int poff, int pstride,
                          const char* vel, int voff, int vstride, const float* __restrict__ weight,
                          const float* __restrict__ radius, float tx, float ty, float tz, float4* spos,
                          float4* svel, unsigned int* rmax, CellOrder co)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (radius && rmax) {
        float r = i < n ? radius[svals[i]] : 0.0f;
        r = r != r ? 3.0e38f : fmaxf(r, 0.0f);
        const unsigned int m = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(r));
        if ((threadIdx.x & 31) == 0 && m && m > *(volatile unsigned int*)rmax) atomicMax(rmax, m);
    }
    if (i >= n) return;
    const uint32_t j = svals[i];
    const float* p = (const float*)(pos + (size_t)j * pstride + poff);
    const float w[3] = {p[0] + tx, p[1] + ty, p[2] + tz};
    spos[i] = make_float4(w[0], w[1], w[2], weight ? weight[j] : 1.0f);
    if (svel) {
        float4 v = make_float4(0.f, 0.f, 0.f, radius ? radius[j] : 0.f);
        if (vel) {
            const float* q = (const float*)(vel + (size_t)j * vstride + voff);
            v.x = q[0];
            v.y = q[1];
            v.z = q[2];
        }
        svel[i] = v;
    }
    if (!co.leaf_dense) return;
    const uint32_t key = co.skeys[i] >> 3;
    if (key >= co.invalid_key) return;
    int c[3];
    ks_unpack(co.L.ks, key, 0, c);
    const int leaf = ll_find(co.L, c[0], c[1], c[2]);
    const int dense = leaf >= 0 ? co.leaf_dense[leaf] : 0;
    if (!dense) return;
    bool in;
    const int cell = brick8_cell(w, *(const int4*)(co.nodes0 + leaf), in);
    const int* ct = co.cell_tab + (size_t)(dense - 1) * 512 + cell;
    const int end = cell == 511 ? co.leaf_range[leaf].y : ct[1];
    if (!in || (int)i < ct[0] || (int)i >= end) co.leaf_dense[leaf] = 0;
}

struct SplatArgs {
    int brick, P, apron;
    uint32_t nslots;
    const int* slot_leaf;
    const int* leaf_slot;
    const GvxNode* nodes0;
    const int* nbr;
    const int2* leaf_range;
    const int* leaf_oct;  // 8 per leaf: first sorted index of each octant of its points
    const float4* spos;
    const float4* svel;  // nullptr when no velocity and no per-point radius
    bool per_point_radius;
    float radius;
    float* den;          // channel data (slot-major, P^3 per slot) or nullptr
    float4* vel;         // or nullptr
    int slabs, slab_layers;  // z-slabs per brick, layers per slab
    // push (apron 1, not accumulating): a tile covers the interior rows and layers only (x with
    // its apron), and the slab's boundary rows go to the neighbours' y/z aprons; else the whole
    // padded brick.  tile_rows: rows of a tile layer (the brick, or the padded brick)
    bool push;
    const uint32_t* push_tab;  // one unit a brick: the boundary voxels' places (push_table), or null
    int push_count;
    int tile_rows;
    int lb;              // log2(brick)
    int reach;           // voxels a point's footprint reaches beyond its own voxel (neighbour pruning)
    const unsigned int* rmax;  // per-point radii: float bits of the largest (bounds `reach` on the device)
    float max_radius;    // per-point radii above this reach past the 26 neighbours
    bool accum;
    bool light;          // few points a unit (see kAheadUnits)
    float boundval;
    uint32_t* err;
    uint32_t* next;  // work-unit counter of the single-grid launch
    // an accumulating single-grid splat may visit only the slots whose bricks some point can
    // reach (unit_slots[0 .. *unit_count), in no particular order); null: every slot
    const uint32_t* unit_slots;
    const uint32_t* unit_count;
    // k_splat_tri, bricks of 8: per leaf 0 or 1 + its number among the dense leaves, whose points are in
    // cell order, and per dense leaf the first sorted index of each of its 512 cells; null: no such order
    const int* leaf_dense;
    const int* cell_tab;
    uint32_t* dense_units;  // units listed for k_tri_dense, and the list (grid, slot, z0, layers); null: none are
    uint4* dense_list;
};

// Shared-memory tile of one padded brick.  Density only: float per voxel.
// Velocity (with or without density): float4 per voxel (vx, vy, vz, density),
// so a contribution is one 16-byte shared read-modify-write.
template <bool HAS_DEN, bool HAS_VEL>
struct Tile {
    static constexpr bool VEC = HAS_VEL;
    static __host__ __device__ size_t bytes(int P3) { return (size_t)P3 * (VEC ? 16 : 4); }
    // The velocity sums are explicit fused multiply-adds: left to the compiler,
    // `o.x += wgt * ux` may be fused in one kernel (or one unrolled copy) and not
    // in another, and every brick must add a voxel's terms with the same rounding.
    __device__ static void add(unsigned char* t, int i, float wgt, float ux, float uy, float uz)
    {
        if (VEC) {
            float4* v = (float4*)t;
            float4 o = v[i];
            o.x = __fmaf_rn(wgt, ux, o.x);
            o.y = __fmaf_rn(wgt, uy, o.y);
            o.z = __fmaf_rn(wgt, uz, o.z);
            if (HAS_DEN) o.w = __fadd_rn(o.w, wgt);
            v[i] = o;
        } else {
            ((float*)t)[i] = __fadd_rn(((float*)t)[i], wgt);
        }
    }
    // density alone: norm * shape joins the sum in one rounding
    __device__ static void add_product(unsigned char* t, int i, float norm, float shape)
    {
        ((float*)t)[i] = __fmaf_rn(norm, shape, ((float*)t)[i]);
    }
    __device__ static void set(unsigned char* t, int i, float val)
    {
        if (VEC)
            ((float4*)t)[i] = make_float4(val, val, val, val);
        else
            ((float*)t)[i] = val;
    }
};

// one voxel out: the tile's (density in .w with velocity), or the boundary value
template <bool HAS_DEN, bool HAS_VEL>
__device__ __forceinline__ void put_voxel(const SplatArgs& a, const unsigned char* tile, int ti, size_t gi)
{
    if (HAS_VEL) {
        const float4 o = ((const float4*)tile)[ti];
        if (HAS_DEN) {
            a.den[gi] = o.w;
            a.vel[gi] = make_float4(o.x, o.y, o.z, 0.0f);
        } else {
            a.vel[gi] = o;
        }
    } else {
        a.den[gi] = ((const float*)tile)[ti];
    }
}
template <bool HAS_DEN, bool HAS_VEL>
__device__ __forceinline__ void put_bound(const SplatArgs& a, size_t gi)
{
    const float v = a.boundval;
    if (HAS_DEN) a.den[gi] = v;
    if (HAS_VEL) a.vel[gi] = make_float4(v, v, v, HAS_DEN ? 0.0f : v);
}

// The slab of a push tile to HBM (apron 1).  The tile holds the brick's interior rows and
// layers of the slab, x with its apron (computed from the points, exact copies of the
// x-neighbours' interiors by the canonical sums).  Every voxel of the padded atlas has one
// writer, the brick whose interior holds it:
//  - the tile's rows go to the brick's own slot;
//  - its boundary rows go to the y/z aprons of the neighbours B + (0, dy, dz) that exist,
//    whole rows, x aprons included (the receiver's apron row in direction -(dy, dz) holds,
//    x apart, this brick's voxels, and at its two ends the voxels of B -/+ x, which this
//    brick's x apron holds);
//  - where that neighbour B + (0, dy, dz) is missing, the end voxels of its would-be row go
//    from the bricks B + (-1|+1, dy, dz) that exist, one voxel a row (this brick's first or
//    last interior column), to B + (+1|-1, ...)'s row ends: with receiver offset (dx, dy, dz),
//    dx != 0, this brick sends when B + (dx, 0, 0) is missing;
//  - the brick's own y/z apron rows facing a missing B + (0, dy, dz) take the boundary value
//    (their end voxels too where B + (-1|+1, dy, dz) is missing as well).
// Rows of a receiver direction: dy = -1: the first interior row (to the receiver's last padded
// row), +1: the last (to its row 0), 0: every row; likewise in z, where only the slab holding
// the first (last) interior layer sends.  nbs: lane r < 27 holds the slot of neighbour r,
// r = (dx+1)*9 + (dy+1)*3 + (dz+1).
template <bool HAS_DEN, bool HAS_VEL>
__device__ __forceinline__ void push_out(const SplatArgs& a, const unsigned char* tile, uint32_t s, int z0, int nl,
                                         int nbs, int lane)
{
    const int P = a.P, P3 = P * P * P, b = a.brick, lb = a.lb, TY = b;
    // a brick with all the neighbours that its rows may go to, one unit: the boundary voxels' places come
    // from a table, 32 a step (the general code below: 1,490 instructions a brick)
    if (a.push_tab && (__ballot_sync(kFull, nbs >= 0) & 0x0043FE10u) == 0x0043FE10u) {
        float4* const tv = (float4*)tile;
        const size_t own = (size_t)s * P3;
        const int lay = TY * P;
        for (int z = 0; z < nl; z++) {
            const size_t at = own + (uint32_t)((z0 + z) * P * P + P);
            for (int e = lane; e < lay; e += 32) {
                const float4 o = tv[z * lay + e];
                a.den[at + e] = o.w;
                a.vel[at + e] = make_float4(o.x, o.y, o.z, 0.0f);
            }
        }
        for (int e = lane; e < a.push_count; e += 32) {  // (a multiple of 32, the last entries repeated)
            const uint32_t c = a.push_tab[e];
            const int r = __shfl_sync(kFull, nbs, (int)(c >> 24));
            const float4 o = tv[c & 0xFFFu];
            const size_t at = (size_t)r * P3 + ((c >> 12) & 0xFFFu);
            a.den[at] = o.w;
            a.vel[at] = make_float4(o.x, o.y, o.z, 0.0f);
        }
        return;
    }
    const uint32_t mP = 0xFFFFFFFFu / (uint32_t)P + 1u;  // e / P == umulhi(e, mP) for e < 2^16
    // the brick's own rows: a tile layer is contiguous in the slot from padded (y 1, z)
    const size_t own = (size_t)s * P3;
    const int lay = TY * P, nvox = nl * lay;
    const uint32_t mL = 0xFFFFFFFFu / (uint32_t)lay + 1u;
    for (int e = lane; e < nvox; e += 32) {
        const int lz = (int)__umulhi((uint32_t)e, mL);
        put_voxel<HAS_DEN, HAS_VEL>(a, tile, e, own + (uint32_t)((z0 + lz) * P * P + P + (e - lz * lay)));
    }
    const bool xm = __shfl_sync(kFull, nbs, 4) >= 0, xp = __shfl_sync(kFull, nbs, 22) >= 0;  // B -/+ x
#pragma unroll 1
    for (int q = 0; q < 9; q++) {
        const int dy = q / 3 - 1, dz = q % 3 - 1;
        if (dy == 0 && dz == 0) continue;
        // the sending rows (ly in [ly0, ly0 + nry), lz in [lz0, lz0 + nrz)) of direction (., dy, dz)
        int ly0 = 0, nry = TY, lz0 = 0, nrz = nl;
        if (dy != 0) {
            ly0 = dy < 0 ? 0 : TY - 1;
            nry = 1;
        }
        if (dz != 0) {
            lz0 = dz < 0 ? 1 - z0 : P - 2 - z0;  // the first (last) interior layer
            if (lz0 < 0 || lz0 >= nl) continue;
            nrz = 1;
        }
        const int nrows = nry * nrz;
        const int d0 = 9 + (dy + 1) * 3 + (dz + 1);  // (0, dy, dz); (-1|+1, dy, dz) at d0 -/+ 9
        const int r0 = __shfl_sync(kFull, nbs, d0);
        const int rm = __shfl_sync(kFull, nbs, d0 - 9), rp = __shfl_sync(kFull, nbs, d0 + 9);
        // row r of the direction: tile row, and its padded (y, z) in a receiver (-1 -> P-1, +1 -> 0)
        auto row = [&](int r, int& ti, int& yr, int& zr) {
            const int ly = ly0 + (nry == 1 ? 0 : (r & (TY - 1))), lz = lz0 + (nry == 1 ? r : (r >> lb));
            ti = (lz * TY + ly) * P;
            yr = dy < 0 ? P - 1 : (dy > 0 ? 0 : ly + 1);
            zr = dz < 0 ? P - 1 : (dz > 0 ? 0 : z0 + lz);
        };
        if (r0 >= 0) {  // whole rows to B + (0, dy, dz)
            const size_t rb = (size_t)r0 * P3;
            for (int e = lane; e < nrows * P; e += 32) {
                const int r = (int)__umulhi((uint32_t)e, mP), x = e - r * P;
                int ti, yr, zr;
                row(r, ti, yr, zr);
                put_voxel<HAS_DEN, HAS_VEL>(a, tile, ti + x, rb + (uint32_t)((zr * P + yr) * P + x));
            }
        } else if (!a.accum) {  // the brick's own apron rows facing the missing B + (0, dy, dz)
            // (their end voxels too where B -/+ x + (0, dy, dz) is missing as well)
            const bool lo = rm < 0, hi = rp < 0;
            for (int e = lane; e < nrows * P; e += 32) {
                const int r = (int)__umulhi((uint32_t)e, mP), x = e - r * P;
                if ((x == 0 && !lo) || (x == P - 1 && !hi)) continue;
                int ti, yr, zr;
                row(r, ti, yr, zr);
                const int yB = dy == 0 ? yr : P - 1 - yr, zB = dz == 0 ? zr : P - 1 - zr;  // the own side
                put_bound<HAS_DEN, HAS_VEL>(a, own + (uint32_t)((zB * P + yB) * P + x));
            }
        }
        // one voxel a row to B -/+ x + (0, dy, dz), whose row source B -/+ x is missing
        if (!xm && rm >= 0) {
            const size_t rb = (size_t)rm * P3;
            for (int r = lane; r < nrows; r += 32) {
                int ti, yr, zr;
                row(r, ti, yr, zr);
                put_voxel<HAS_DEN, HAS_VEL>(a, tile, ti + 1, rb + (uint32_t)((zr * P + yr) * P + P - 1));
            }
        }
        if (!xp && rp >= 0) {
            const size_t rb = (size_t)rp * P3;
            for (int r = lane; r < nrows; r += 32) {
                int ti, yr, zr;
                row(r, ti, yr, zr);
                put_voxel<HAS_DEN, HAS_VEL>(a, tile, ti + P - 2, rb + (uint32_t)((zr * P + yr) * P));
            }
        }
    }
}

// the apron regions `reset` (bit (dx+1)*9 + (dy+1)*3 + (dz+1)) of a slab's tile to the boundary value
template <bool HAS_DEN, bool HAS_VEL>
__device__ __forceinline__ void reset_regions(const SplatArgs& a, unsigned char* tile, uint32_t reset, int z0, int nl,
                                              int TY, int yoff, int lane)
{
    const int P = a.P;
#pragma unroll 1
    for (int k = 0; k < 27; k++) {
        if (!((reset >> k) & 1u)) continue;
        const int dx = k / 9 - 1, dy = (k / 3) % 3 - 1, dz = k % 3 - 1;
        const int xb = dx < 0 ? 0 : (dx > 0 ? P - 1 : 1), yb = dy < 0 ? 0 : (dy > 0 ? P - 1 : 1);
        const int bx = dx == 0 ? a.lb : 0, by = dy == 0 ? a.lb : 0;  // log2 of the region's x, y extents
        const int zlo = max(dz < 0 ? 0 : (dz > 0 ? P - 1 : 1), z0);
        const int zhi = min(dz < 0 ? 0 : (dz > 0 ? P - 1 : P - 2), z0 + nl - 1);
        const int cnt = zhi >= zlo ? (zhi - zlo + 1) << (bx + by) : 0;
        for (int c = lane; c < cnt; c += 32) {
            const int x = xb + (c & ((1 << bx) - 1)), y = yb + ((c >> bx) & ((1 << by) - 1));
            const int z = zlo + (c >> (bx + by));
            Tile<HAS_DEN, HAS_VEL>::set(tile, ((z - z0) * TY + (y - yoff)) * P + x, a.boundval);
        }
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------
// Work units: one warp per (brick, z-slab).  The layers of a brick's tile (the padded brick, or its
// interior for push tiles) are split into slabs of a.slab_layers layers, each with its own shared tile,
// so a warp's tile is a fraction of the brick and more warps stay resident.  Every slab sees the same
// candidate points in the same order, so a voxel's sum does not depend on the split.

// the unit's brick and slab, and what the lane needs of them
struct SplatUnit {
    uint32_t s;      // atlas slot
    int z0, nl;      // padded layers of the unit
    int leaf;
    int nl27;        // the lane's neighbour (leaf index, -1: none): lane r is neighbour (r/9, r/3%3, r%3) - 1
    int4 org;        // the node's first 16 bytes: (lev.., x, y, z)
    int start, end;  // the lane's candidates in the sorted points
};

// halves of a neighbour at offset d (bricks) whose points reach voxels [v0, v1] of the brick along an
// axis: points of floor coordinate f touch [f - below, f + above]
__device__ __forceinline__ bool unit_halves(int d, int b, int v0, int v1, int below, int above, int& lo, int& hi)
{
    const int hb = b >> 1, c = d * b;
    const bool n0 = c - below <= v1 && c + hb - 1 + above >= v0, n1 = c + hb - below <= v1 && c + b - 1 + above >= v0;
    lo = n0 ? 0 : 1;
    hi = n1 ? 1 : 0;
    return n0 || n1;
}

__device__ __forceinline__ void unit_slot(const SplatArgs& a, uint32_t u, bool push, SplatUnit& t)
{
    const uint32_t S = (uint32_t)a.slabs;
    const uint32_t ui = S == 1u ? u : u / S;
    const int y0 = push ? a.apron : 0;
    t.s = a.unit_slots ? a.unit_slots[ui] : ui;
    t.z0 = y0 + (int)(u - ui * S) * a.slab_layers;
    t.nl = min(a.slab_layers, a.P - y0 - t.z0);
    t.leaf = a.slot_leaf[t.s];
}
__device__ __forceinline__ void unit_neighbour(const SplatArgs& a, SplatUnit& t, int nbi)
{
    t.nl27 = nbi >= 0 ? a.nbr[(size_t)t.leaf * 27 + nbi] : -1;
    t.org = *(const int4*)(a.nodes0 + t.leaf);
}
// one range of candidates per neighbour: from its first octant that can reach the tile to its last one
// (a superset of the octants that can: two loads, and no list of runs; the footprint test drops the rest)
__device__ __forceinline__ void unit_octants(const SplatArgs& a, SplatUnit& t, int o0, int o1)
{
    const int* oc = a.leaf_oct + (size_t)t.nl27 * 8;
    t.start = oc[o0];
    t.end = o1 == 7 ? a.leaf_range[t.nl27].y : oc[o1 + 1];
}

// Units are claimed two at a time where there are many for every warp: the counter is one address, which
// takes an atomic every two nanoseconds (trilinear splat of 24 clouds, 2.07M bricks: 3.24 ms one at a
// time, 2.37 two, 2.44 four, 2.53 eight).  Where units are fewer, their costs differ by more than the
// claims cost: one at a time.
constexpr uint32_t kClaim = 2, kClaimUnits = 16;

// A warp that looks ahead (below) holds up to four units, taken while others have none: with few units a warp,
// and dense ones among them, the last ones wait in the queue of a warp that is busy while the chip runs empty.
// So the splats of the cells' kernel look ahead where there are kAheadUnits a warp, or kAheadLight of units that
// hold few points (SplatArgs::light), whose lookups would not be hidden otherwise.  Cubic splats of R 3.5, us
// looking ahead / not / as it was with one unit held: 100k points in 4k bricks of 8^3 534 / 330 / 418, in 9k
// bricks 338 / 286 / 324, in 2.7k of 16^3 326 / 210 / 283; density and velocity of R 2, 20k points in 17k
// bricks, 11 units a warp, 78 / 92 / 87, of R 3.5, 300k points in 3.4k bricks of 16^3, 11 a warp, 1714 / 1505 /
// 1601.  2M points of R 3 in 85k bricks, 24 a warp, 3283 / 3170 us; 24 clouds of 100k, 32 a warp, 4127 / 3486; a
// million points of radii 1-3, 80 a warp, the same.
constexpr uint32_t kAheadUnits = 64, kAheadLight = 4, kLightPoints = 1;

// Blocks an SM of a launch with fewer than kFewUnits units a warp, where registers would hold more: other
// streams' launches find room beside them.  (Frames of 300k points in 16^3 bricks, five units a warp, three in
// flight: 584 us with the SMs full, 519 with four blocks; one at a time 686 and 796, where looking ahead took 542
// and 940.  100k points in 8k bricks of 8^3, seven units a warp: 82 us and 99.)
constexpr int kFewBlocks = 4;
constexpr uint32_t kFewUnits = 6;

// Units [0, total) of all grids from the counter `next`: of(u, local) -> the number of u's grid and its
// unit there, args(k) -> that grid's arguments, range(a, t): the lane's candidates, run(a, t, k, mid): the
// unit, which calls mid() once.  Looking ahead there are three steps at a time: while unit t is summed, the
// neighbours (asked for as it starts) and then the candidate ranges of t1 arrive, and the brick of t2.
// Not looking ahead, a unit is taken when the last one is done.  AHEAD: which of the two, or, where the host does
// not know the units, as `ahead` says.
enum { kAheadNever, kAheadAlways, kAheadAsked };
template <int AHEAD, class Of, class Args, class Range, class Run>
__device__ __forceinline__ void unit_loop(uint32_t total, uint32_t* next, bool push, bool ahead, int lane, Of of,
                                          Args args, Range range, Run run)
{
    if (AHEAD != kAheadAsked) ahead = AHEAD == kAheadAlways;
    const int nbi = lane < 27 ? (lane % 3) * 9 + (lane / 3 % 3) * 3 + lane / 9 : -1;
    const uint32_t claim = total >= kClaimUnits * gridDim.x * (blockDim.x >> 5) ? kClaim : 1u;
    uint32_t cur = 0u, lim = 0u, pre = ahead && lane == 0 ? atomicAdd(next, claim) : 0u, lu;
    auto take = [&]() {  // the next unit's number (total and above: none)
        if (cur == lim) {
            if (!ahead && lane == 0) pre = atomicAdd(next, claim);
            cur = __shfl_sync(kFull, pre, 0);
            lim = cur + claim;
            if (ahead && lane == 0 && cur < total) pre = atomicAdd(next, claim);
        }
        return cur++;
    };
    uint32_t u = take();
    if (u >= total) return;
    SplatUnit t, t1;
    uint32_t k = of(u, lu), k1;
    unit_slot(args(k), lu, push, t);
    bool more = false;
    if (ahead) {
        u = take();
        more = u < total;
    }
    k1 = k;
    t1 = t;
    if (more) {
        k1 = of(u, lu);
        unit_slot(args(k1), lu, push, t1);
    }
    unit_neighbour(args(k), t, nbi);
    range(args(k), t);
    for (;;) {
        SplatUnit t2 = t1;
        uint32_t k2 = k1;
        bool more2 = false;
        if (more) {
            unit_neighbour(args(k1), t1, nbi);
            u = take();
            more2 = u < total;
            if (more2) {
                k2 = of(u, lu);
                unit_slot(args(k2), lu, push, t2);
            }
        }
        run(args(k), t, k, [&]() {
            if (more) range(args(k1), t1);
        });
        if (!ahead) {
            u = take();
            more = u < total;
            if (more) {
                k1 = of(u, lu);
                unit_slot(args(k1), lu, push, t1);
                unit_neighbour(args(k1), t1, nbi);
                range(args(k1), t1);
            }
        }
        if (!more) break;
        k = k1;
        t = t1;
        k1 = k2;
        t1 = t2;
        more = more2;
    }
}

// the lanes' ranges in a row: a lane's first candidate number `off`, the candidates' count; the ranges
// with points leave in rs, in order, their first sorted index less their first candidate number
__device__ __forceinline__ int unit_candidates(const SplatUnit& t, int lane, int& off)
{
    const int len = t.end - t.start;
    off = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, off, o);
        if (lane >= o) off += v;
    }
    const int total = __shfl_sync(kFull, off, 31);
    off -= len;
    return total;
}
__device__ __forceinline__ void unit_ranges(const SplatUnit& t, int lane, int off, int* rs)
{
    const uint32_t some = __ballot_sync(kFull, t.end > t.start);
    if (t.end > t.start) rs[__popc(some & ((1u << lane) - 1u))] = t.start - off;
}
// sorted index of candidate base + lane: its range is the number of ranges with points that start at or
// before it, less one.  base is below the candidates' count: the first range with points then starts at or
// before every candidate asked for (without candidates there is none, and rs is not to be read)
__device__ __forceinline__ int unit_candidate(const SplatUnit& t, int lane, int off, int base, const int* rs)
{
    const bool some = t.end > t.start;
    const uint32_t starts = __reduce_or_sync(kFull, some && off >= base && off < base + 32 ? 1u << (off - base) : 0u);
    const int before = __popc(__ballot_sync(kFull, some && off < base));
    return rs[before - 1 + __popc(starts & (kFull >> (31 - lane)))] + base + lane;
}

// the regions of the padded brick that voxels [xl, xh] x [yl, yh] x [zl, zh] (padded) reach, bit
// (dx+1)*9 + (dy+1)*3 + (dz+1): per axis 1 = below the interior, 2 = inside, 4 = above it; the product
// of the three spread sets has one bit per region reached (no carries)
__device__ __forceinline__ uint32_t box_regions(int xl, int xh, int yl, int yh, int zl, int zh, int P, int ap)
{
    const int hi = P - 1 - ap;
    const uint32_t tx = (uint32_t)(xl < ap) | (uint32_t)(xl <= hi && xh >= ap) << 1 | (uint32_t)(xh > hi) << 2;
    const uint32_t ty = (uint32_t)(yl < ap) | (uint32_t)(yl <= hi && yh >= ap) << 1 | (uint32_t)(yh > hi) << 2;
    const uint32_t tz = (uint32_t)(zl < ap) | (uint32_t)(zl <= hi && zh >= ap) << 1 | (uint32_t)(zh > hi) << 2;
    return ((tx & 1u) | (tx & 2u) << 8 | (tx & 4u) << 16) * ((ty & 1u) | (ty & 2u) << 2 | (ty & 4u) << 4) * tz;
}

// ---------------------------------------------------------------------------
// CUBIC splats, and TRILINEAR ones with velocity: the hits of a unit -- the candidates whose footprint
// box meets the tile -- are gathered, in the points' order, in shared memory, and their footprints' rows
// are dealt to the lanes.
//
// What bounds it: instruction issue (1M points of the 4M SPH frame's density: 65% of the issue slots,
// 6,400 warp instructions a brick, 25.7 lanes active; by ablations of the kernel before, of its 7,900,
// 3,000 were the voxels' weights and their first turn at the tile, 1,490 the pushes, 1,090 candidates and
// zeroing, 760 the lookups of a cell's point, 670 the further turns of lanes that share a row).  So:
//  - candidates come as one range per neighbour and are located without a search (unit_candidate);
//  - hits are stored where the dealing reads them, instead of being passed from lane to lane into a batch
//    and again to the lanes that deal them;
//  - deal_cells is in the code once: a second copy for the last hits cost more in instruction fetches
//    (1.3 of 8 stalled cycles) than the loop around it;
//  - a push tile's boundary voxels find their places in a table (push_table).
// 4M points 2.53 -> 2.19 ms, 778k 461 -> 405 us, a million points of radii 1-3 without velocity 1.35 ->
// 0.86 ms (with whole bricks a unit).  Tried and dropped: lanes that own rows of the tile and take their
// hits from a mask per row (3.41 ms: half the lanes idle), cells queued row by row so that lanes rarely
// share one (3.95 ms: the queue costs more than the turns it saves), predicated stores instead of
// branches in a turn (2.64 against 2.53).
constexpr int kCellWarps = 4;

// hits gathered before they are dealt: 24 with density and velocity, so that five blocks of four 10 KB
// tiles and their hits fit an SM (a 8^3 brick's interior, x with its apron)
template <bool HAS_DEN, bool HAS_VEL, int MODE, bool PPR>
struct Hits {
    static constexpr int most = HAS_DEN && HAS_VEL ? 24 : 32;
    // beside (x, y, z, weight): with velocity (vx, vy, vz, R), else with per-point radii (1/h, norm, low
    // part of R^2, R)
    static constexpr bool Q = HAS_VEL || PPR;
    static __host__ __device__ size_t bytes() { return most * sizeof(float4) * (Q ? 2 : 1); }
};

// M4 cubic spline (Monaghan & Lattanzio 1985), 3D normalisation 1/(pi h^3), support R = 2h
struct CubicRadius {
    float R, h, inv_h, norm, r2l, r2h;
    __device__ explicit CubicRadius(float R_) : R(R_), h(0.5f * R_), inv_h(1.0f / h)
    {
        norm = kInvPi * inv_h * inv_h * inv_h;
        r2h = __fmul_rn(R, R);
        r2l = fmaf(R, R, -r2h);
    }
    __device__ CubicRadius(float R_, float inv_h_, float norm_, float r2l_)
        : R(R_), h(0.5f * R_), inv_h(inv_h_), norm(norm_), r2l(r2l_)
    {
        r2h = __fmul_rn(R, R);
    }
};

// approximate reciprocal square root and quotient without the scaling of denormal arguments (none here:
// the callers' arguments are at least 1e-36, or their result is not used)
__device__ __forceinline__ float rsqrt_fast(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float div_fast(float x, float y)
{
    float q;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(q) : "f"(x), "f"(y));
    return q;
}

// The footprint cells of the hits 0 .. nb-1 (sp, sq: in shared memory, in sorted order), dealt to the
// lanes 32 at a time.  Lanes whose cells share a row apply their updates one
// after another in lane order, which is the points' sorted order (the cells of
// one point lie in distinct rows or distinct chunks of a row); rows apart apply
// together.  So every voxel sums its contributions in the same order in every
// brick that holds it.
//
// SMALL footprints (trilinear, and cubic of a uniform radius <= 2) span at most
// 4 voxels on every axis: a cell is one row of the box, and of a cubic box
// only the rows that can reach the sphere are dealt.  Their decode is a table
// of 5 bits per layer k of the box, at bit 5k: the first row (2 bits, counted
// from yl) and the number of rows (3 bits).  Other footprints deal every row
// of the box in chunks of up to 4 voxels, decoded by division with multipliers
// m = ceil(2^32 / n) (umulhi(c, m) == c / n for every c < 2^32 / n; 0 stands
// for n = 1).
template <bool HAS_DEN, bool HAS_VEL, int MODE, bool PPR, bool SMALL>
__device__ __forceinline__ void deal_cells(unsigned char* tile, const float4* sp, const float4* sq, const int nb,
                                           const int P, const int TY, const int yoff, const int nl, const int Ox,
                                           const int Oy, const int Zlo, const CubicRadius& uni, const int lane)
{
    using T = Tile<HAS_DEN, HAS_VEL>;
    constexpr bool CUBIC = MODE == GVX_SPLAT_CUBIC;
    // the lane's hit: its box in the tile (8 bits a bound), its cells; aux1, aux2: SMALL the row table,
    // else the multipliers of the chunk and row counts
    uint32_t box0 = 0u, box1 = 0u, aux1 = 0u, aux2 = 0u;
    int ncell = 0;
    if (lane < nb) {
        const float4 p = sp[lane];
        int xl, xh, yl, yh, zl, zh;
        if (!CUBIC) {
            xl = (int)floorf(p.x) - Ox, yl = (int)floorf(p.y) - Oy, zl = (int)floorf(p.z) - Zlo;
            xh = xl + 1, yh = yl + 1, zh = zl + 1;
        } else {
            const float R = PPR ? sq[lane].w : uni.R;
            xl = (int)floorf(p.x - R) + 1 - Ox, xh = (int)ceilf(p.x + R) - 1 - Ox;
            yl = (int)floorf(p.y - R) + 1 - Oy, yh = (int)ceilf(p.y + R) - 1 - Oy;
            zl = (int)floorf(p.z - R) + 1 - Zlo, zh = (int)ceilf(p.z + R) - 1 - Zlo;
        }
        xl = max(xl, 0), xh = min(xh, P - 1);
        yl = max(yl, yoff), yh = min(yh, yoff + TY - 1);
        zl = max(zl, 0), zh = min(zh, nl - 1);
        const int ny = yh - yl + 1;
        if (SMALL) {
            // A row whose float dy, dz give dy^2 + dz^2 < R^2 (1 + 1e-6) in float holds every row
            // with R^2 - dy^2 - dz^2 > 0 exactly (the rows the weights below can reach), with a
            // margin of several roundings; the rows of one layer that pass form one run.
            const float lim = uni.r2h * 1.000001f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (zl + k > zh) break;
                int first = 0, n = ny;
                if (CUBIC) {
                    const float dz = (float)(zl + k + Zlo) - p.z;
                    const float dz2 = dz * dz;
                    first = -1;
                    n = 0;
#pragma unroll
                    for (int yy = 0; yy < 4; yy++) {
                        if (yl + yy > yh) break;
                        const float dy = (float)(yl + yy + Oy) - p.y;
                        if (dy * dy + dz2 < lim) {
                            if (first < 0) first = yy;
                            n++;
                        }
                    }
                    first = max(first, 0);
                }
                aux1 |= (uint32_t)(first | (n << 2)) << (5 * k);
                ncell += n;
            }
            // a point whose box reaches the slab but whose sphere does not keeps one (empty) row,
            // so that every point of the batch owns a cell
            if (ncell == 0) {
                aux1 = 1u << 2;
                ncell = 1;
            }
            box0 = (uint32_t)xl | (uint32_t)xh << 8 | (uint32_t)yl << 16 | (uint32_t)zl << 24;
        } else {
            const uint32_t nch = (uint32_t)(xh - xl + 4) >> 2;
            aux1 = nch > 1u ? 0xFFFFFFFFu / nch + 1u : 0u;
            aux2 = ny > 1 ? 0xFFFFFFFFu / (uint32_t)ny + 1u : 0u;
            ncell = (int)nch * ny * (zh - zl + 1);
            box0 = (uint32_t)xl | (uint32_t)xh << 8 | (uint32_t)yl << 16 | (uint32_t)yh << 24;
            box1 = (uint32_t)zl;
        }
    }
    // inclusive scan of the cell counts over the lanes
    int cend = ncell;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, cend, o);
        if (lane >= o) cend += t;
    }
    const int ctot = __shfl_sync(kFull, cend, 31);
    const int cstart = cend - ncell;
    for (int g0 = 0; g0 < ctot; g0 += 32) {
        const int g = g0 + lane;
        const bool act = g < ctot;
        // the hit dealing this cell: each hit has a cell at least, so it is the number of hits that
        // start at or before g, less one
        const bool own = ncell > 0;
        const uint32_t starts =
            __reduce_or_sync(kFull, own && cstart >= g0 && cstart < g0 + 32 ? 1u << (cstart - g0) : 0u);
        const int before = __popc(__ballot_sync(kFull, own && cstart < g0));
        const int j = before - 1 + __popc(starts & (kFull >> (31 - lane)));
        const float4 p = sp[j];
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (HAS_VEL || PPR) q = sq[j];
        const uint32_t b0 = __shfl_sync(kFull, box0, j);
        const uint32_t a1 = __shfl_sync(kFull, aux1, j);
        const int cell = g - __shfl_sync(kFull, cstart, j);
        const int xl = (int)(b0 & 255u), xh = (int)((b0 >> 8) & 255u), yl = (int)((b0 >> 16) & 255u);
        int lx, ly, lz;
        if (SMALL) {
            const int s1 = (int)((a1 >> 2) & 7u), s2 = s1 + (int)((a1 >> 7) & 7u), s3 = s2 + (int)((a1 >> 12) & 7u);
            const int k = (cell >= s1) + (cell >= s2) + (cell >= s3);
            const int pre = k == 0 ? 0 : (k == 1 ? s1 : (k == 2 ? s2 : s3));
            lx = xl;
            ly = yl + (int)((a1 >> (5 * k)) & 3u) + (cell - pre);
            lz = (int)(b0 >> 24) + k;
        } else {
            const uint32_t b1 = __shfl_sync(kFull, box1, j), m2 = __shfl_sync(kFull, aux2, j);
            const int nch = (xh - xl + 4) >> 2, ny = (int)(b0 >> 24) - yl + 1;
            const int r = a1 ? (int)__umulhi((uint32_t)cell, a1) : cell;  // cell / nch
            const int zz = m2 ? (int)__umulhi((uint32_t)r, m2) : r;       // r / ny
            lx = xl + 4 * (cell - r * nch);
            ly = yl + (r - zz * ny);
            lz = (int)b1 + zz;
        }
        // the lane's voxels lx .. min(lx + 3, xh) of row (ly, lz): values, and a bit per voxel touched
        float w[4] = {0.f, 0.f, 0.f, 0.f}, norm = 0.f;
        uint32_t vm = 0u;
        const int t0 = (lz * TY + (ly - yoff)) * P + lx;  // (the tile's rows start at padded y = yoff)
        if (act) {
            if (!CUBIC) {
                const float fx0 = floorf(p.x), fy0 = floorf(p.y), fz0 = floorf(p.z);
                const float fx = p.x - fx0, fy = p.y - fy0, fz = p.z - fz0;
                const float wyz = __fmul_rn((float)(ly + Oy) == fy0 ? 1.f - fy : fy,
                                            (float)(lz + Zlo) == fz0 ? 1.f - fz : fz);
                const float wxa = (float)(lx + Ox) == fx0 ? 1.f - fx : fx;
                w[0] = __fmul_rn(__fmul_rn(p.w, wxa), wyz);
                vm = 1u;
                if (lx + 1 <= xh) {
                    w[1] = __fmul_rn(__fmul_rn(p.w, fx), wyz);  // lx + 1 is floor(px) + 1 here
                    vm |= 2u;
                }
            } else {
                // Along the row R^2 - d^2 is formed from an error-free
                // c = R^2 - dy^2 - dz^2 (two-product, two-sum) so that the outer branch
                // 0.25 (2-q)^3 = 0.25 ((R^2-d^2) / (h (R+d)))^3 keeps FP32 relative
                // accuracy up to the edge of the support.
                const CubicRadius c = !PPR ? uni : HAS_VEL ? CubicRadius(q.w) : CubicRadius(q.w, q.x, q.y, q.z);
                norm = c.norm * p.w;
                const float dy = (float)(ly + Oy) - p.y, dz = (float)(lz + Zlo) - p.z;
                // (each step rounded on its own: a fused one would not have the error it is assumed to have)
                const float qy = __fmul_rn(dy, dy), ey = fmaf(dy, dy, -qy);
                const float qz = __fmul_rn(dz, dz), ez = fmaf(dz, dz, -qz);
                const float syz = __fadd_rn(qy, qz);
                float bv = __fsub_rn(syz, qy);
                const float e1 = __fadd_rn(__fsub_rn(qy, __fsub_rn(syz, bv)), __fsub_rn(qz, bv));
                const float c1 = __fsub_rn(c.r2h, syz);
                bv = __fsub_rn(c1, c.r2h);
                const float e2 = __fadd_rn(__fsub_rn(c.r2h, __fsub_rn(c1, bv)), __fsub_rn(-syz, bv));
                const float cl = e2 + c.r2l - ((ey + ez) + e1);
                if (c1 + cl > 0.0f) {
                    // the four voxels without branches (a slot outside the row or the support
                    // is computed and masked), so that their independent chains interleave
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float dx = (float)(lx + k + Ox) - p.x;
                        const float t = fmaf(-dx, dx, c1) + cl;  // R^2 - d^2
                        const float d2 = fmaf(dx, dx, syz);
                        const float d = d2 > 1.0e-36f ? d2 * rsqrt_fast(d2) : 0.0f;
                        const float qq = d * c.inv_h;
                        const float wi = fmaf(qq * qq, fmaf(0.75f, qq, -1.5f), 1.0f);  // q < 1
                        const float uu = div_fast(t, c.h * (c.R + d));                 // 2 - q
                        const float shape = qq < 1.0f ? wi : 0.25f * uu * uu * uu;
                        const bool ok = lx + k <= xh && t > 0.0f;
                        w[k] = HAS_VEL ? __fmul_rn(norm, shape) : shape;
                        vm |= ok ? 1u << k : 0u;
                    }
                }
            }
        }
        // lanes sharing a row apply in lane order (the cells of one point lie in distinct rows
        // or distinct chunks of a row); rows apart apply together
        const int key = act ? (lz * P + ly) : -1 - lane;
        const uint32_t grp = __match_any_sync(kFull, key);
        const int rank = __popc(grp & ((1u << lane) - 1u));
        const int nph = (int)__reduce_max_sync(kFull, (uint32_t)rank) + 1;
        for (int ph = 0; ph < nph; ph++) {
            if (rank == ph && vm) {
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if ((vm >> k) & 1u) {
                        if (CUBIC && !HAS_VEL)
                            T::add_product(tile, t0 + k, norm, w[k]);
                        else
                            T::add(tile, t0 + k, w[k], q.x, q.y, q.z);
                    }
            }
            __syncwarp();
        }
    }
}

// shared memory of one warp: the tile, the hits
template <bool HAS_DEN, bool HAS_VEL>
__host__ __device__ inline size_t cell_tile_bytes(int layers, int rows, int P)
{
    return (Tile<HAS_DEN, HAS_VEL>::bytes(layers * rows * P) + 15) & ~(size_t)15;
}
template <bool HAS_DEN, bool HAS_VEL, int MODE, bool PPR>
__host__ __device__ inline size_t cell_warp_bytes(int layers, int rows, int P)
{
    return cell_tile_bytes<HAS_DEN, HAS_VEL>(layers, rows, P) + Hits<HAS_DEN, HAS_VEL, MODE, PPR>::bytes();
}

template <bool HAS_DEN, bool HAS_VEL, int MODE, bool PPR, bool SMALL, class Mid>
__device__ __forceinline__ void cell_unit(const SplatArgs& a, const SplatUnit& t, unsigned char* mem, uint64_t* bar,
                                         int* rs, uint32_t& phase, const int lane, Mid mid)
{
    using T = Tile<HAS_DEN, HAS_VEL>;
    constexpr bool CUBIC = MODE == GVX_SPLAT_CUBIC;
    // single-channel tiles go to HBM in one bulk (TMA) copy; the combined
    // density+velocity tile is split into the two channels by vector stores
    constexpr bool BULK = !(HAS_DEN && HAS_VEL);
    constexpr bool PUSHABLE = HAS_DEN && HAS_VEL;  // the host sets push for these kernels only
    const bool push = PUSHABLE && a.push;
    const CubicRadius uni(CUBIC && !PPR ? a.radius : 2.0f);
    const int P = a.P, P2 = P * P, ap = a.apron;
    const int TY = push ? a.tile_rows : P, yoff = push ? ap : 0;
    const int z0 = t.z0, nl = t.nl, nvox = nl * TY * P;
    const size_t gofs = (size_t)t.s * (P2 * P) + (size_t)z0 * P2;  // slab start in the channel (no push)
    const int Ox = t.org.y - ap, Oy = t.org.z - ap, Zlo = t.org.w - ap + z0;
    unsigned char* tile = mem;
    using H = Hits<HAS_DEN, HAS_VEL, MODE, PPR>;
    float4* sp = (float4*)(mem + cell_tile_bytes<HAS_DEN, HAS_VEL>(a.slab_layers, TY, P));
    float4* sq = sp + H::most;
    const uint32_t lt = (1u << lane) - 1u;

    int off;
    const int total = unit_candidates(t, lane, off);
    // an accumulating splat leaves a slab that no point reaches as it is: no load, no store
    if (a.accum && total == 0) {
        mid();
        return;
    }
    unit_ranges(t, lane, off, rs);
    const uint32_t nbmask = __ballot_sync(kFull, t.nl27 >= 0);  // bit r: neighbour r is active

    // ---- tile: previous values (accumulate) or zeros, once the bulk store of the warp's last
    // slab has read it (the wait is deferred to here: that read overlaps the ranges above)
    if (BULK) {
        if (lane == 0) bulk_wait_read_all();
    }
    __syncwarp();
    if (a.accum) {
        if (BULK) {
            if (lane == 0) {
                const uint32_t nb = (uint32_t)T::bytes(nvox);
                mbar_expect_tx(bar, nb);
                if (HAS_DEN) bulk_g2s(tile, a.den + gofs, nb, bar);
                else bulk_g2s(tile, a.vel + gofs, nb, bar);
            }
            if (!mbar_wait_bounded(bar, phase)) atomicOr(a.err, GVX_DERR_TIMEOUT);
            phase ^= 1u;
        } else {
            float4* tv = (float4*)tile;
            for (int i = lane; i < nvox; i += 32) {
                const float4 v = a.vel[gofs + i];
                tv[i] = make_float4(v.x, v.y, v.z, a.den[gofs + i]);
            }
        }
    } else {
        // zeros in 16-byte stores (a slab holds a multiple of 4 voxels: P is even)
        const int n16 = (int)(T::bytes(nvox) / 16);
        for (int i = lane; i < n16; i += 32) ((float4*)tile)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncwarp();
    mid();

    // ---- candidates, 32 at a time, in sorted order: those whose footprint box meets the tile join the
    // hits; hits that the next round's would overflow, and the last ones, are added to the tile
    int nb = 0;  // hits gathered (warp-uniform)
    uint32_t touched = 0u;
    for (int base = 0;; base += 32) {
        const bool done = base >= total;  // one more pass deals the last hits
        const int idx = done ? 0 : unit_candidate(t, lane, off, base, rs);
        bool hit = false;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
        if (base + lane < total) {
            p = a.spos[idx];
            if (HAS_VEL || PPR) q = a.svel[idx];
            int xl, xh, yl, yh, zl, zh;
            if (!CUBIC) {
                xl = (int)floorf(p.x) - Ox, yl = (int)floorf(p.y) - Oy, zl = (int)floorf(p.z) - Zlo;
                xh = xl + 1, yh = yl + 1, zh = zl + 1;
            } else {
                // voxels strictly inside (p - R, p + R) on every axis
                const float R = PPR ? q.w : uni.R;
                if (PPR && R > a.max_radius) atomicOr(a.err, GVX_DERR_RADIUS);
                xl = (int)floorf(p.x - R) + 1 - Ox, xh = (int)ceilf(p.x + R) - 1 - Ox;
                yl = (int)floorf(p.y - R) + 1 - Oy, yh = (int)ceilf(p.y + R) - 1 - Oy;
                zl = (int)floorf(p.z - R) + 1 - Zlo, zh = (int)ceilf(p.z + R) - 1 - Zlo;
                if (PPR && !HAS_VEL) {
                    const CubicRadius c(R);
                    q = make_float4(c.inv_h, c.norm, c.r2l, R);
                }
            }
            xl = max(xl, 0), xh = min(xh, P - 1);
            yl = max(yl, yoff), yh = min(yh, yoff + TY - 1);
            zl = max(zl, 0), zh = min(zh, nl - 1);
            hit = xl <= xh && yl <= yh && zl <= zh;
            if (hit && nbmask != 0x7FFFFFFu && ap) touched |= box_regions(xl, xh, yl, yh, z0 + zl, z0 + zh, P, ap);
        }
        // the hits that there is room for; when there is no more, all gathered are dealt first
        uint32_t hm = __ballot_sync(kFull, hit);
        do {
            const int at = nb + __popc(hm & lt);
            if (hit && at < H::most) {
                sp[at] = p;
                if (HAS_VEL || PPR) sq[at] = q;
                hit = false;
            }
            nb = min(nb + __popc(hm), H::most);
            hm = __ballot_sync(kFull, hit);
            if (hm || (done && nb > 0)) {
                __syncwarp();
                deal_cells<HAS_DEN, HAS_VEL, MODE, PPR, SMALL>(tile, sp, sq, nb, P, TY, yoff, nl, Ox, Oy, Zlo, uni, lane);
                nb = 0;
            }
        } while (hm);
        if (done) break;
    }

    // ---- apron voxels with no neighbouring brick take the boundary value (0): the apron region facing
    // each missing neighbour (apron 1), clipped to the slab.  The tile was zeroed, so with the boundary
    // value 0 only the regions that some hit reached are reset.
    uint32_t reset = ~nbmask & 0x7FFFFFFu & ~(1u << 13);
    if (a.boundval == 0.0f && reset) reset &= __reduce_or_sync(kFull, touched);
    if (push) reset &= (1u << 4) | (1u << 22);  // the tile's only apron voxels: the two x faces
    if (ap && reset && !a.accum) reset_regions<HAS_DEN, HAS_VEL>(a, tile, reset, z0, nl, TY, yoff, lane);

    // ---- out to HBM
    if (push) {
        const int nbs = t.nl27 >= 0 ? a.leaf_slot[t.nl27] : -1;
        if (PUSHABLE) push_out<HAS_DEN, HAS_VEL>(a, tile, t.s, z0, nl, nbs, lane);
        __syncwarp();
    } else if (BULK) {
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
            if (HAS_DEN) bulk_s2g(a.den + gofs, tile, (uint32_t)T::bytes(nvox));
            else bulk_s2g(a.vel + gofs, tile, (uint32_t)T::bytes(nvox));
            bulk_commit();  // (its read of the tile is waited for before the tile's next write)
        }
    } else {
        const float4* tv = (const float4*)tile;
        float* dg = a.den + gofs;
        float4* vg = a.vel + gofs;
        for (int i = lane; i < nvox; i += 32) {
            const float4 o = tv[i];
            dg[i] = o.w;
            vg[i] = make_float4(o.x, o.y, o.z, 0.0f);
        }
        __syncwarp();
    }
}

template <int AHEAD, bool HAS_DEN, bool HAS_VEL, int MODE, bool PPR, bool SMALL, class Of, class Args>
__device__ __forceinline__ void cell_loop(const SplatArgs& a0, uint32_t total, uint32_t* next, unsigned char* smem, Of of,
                                         Args args)
{
    constexpr bool CUBIC = MODE == GVX_SPLAT_CUBIC;
    __shared__ __align__(8) uint64_t s_bar[kCellWarps];
    // (a range a neighbour, no word more: with 32, five blocks of a batch's push tiles missed an SM by 128 bytes;
    // 24 clouds of 100k points, density and velocity, R 3: 3.77 ms with four blocks, 3.34 with five)
    __shared__ int s_rs[kCellWarps][28];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool push = HAS_DEN && HAS_VEL && a0.push;
    unsigned char* mem = smem + (size_t)wid * cell_warp_bytes<HAS_DEN, HAS_VEL, MODE, PPR>(a0.slab_layers, a0.tile_rows, a0.P);
    if (lane == 0) {
        mbar_init(&s_bar[wid], 1);
        mbar_fence_init();
    }
    __syncwarp();
    uint32_t phase = 0;
    const int dx = lane / 9 - 1, dy = lane / 3 % 3 - 1, dz = lane % 3 - 1;
    const bool ahead = total >= (a0.light ? kAheadLight : kAheadUnits) * gridDim.x * kCellWarps;
    unit_loop<AHEAD>(
        total, next, push, ahead, lane, of, args,
        [&](const SplatArgs& a, SplatUnit& t) {
            // the neighbour's octants whose points, whose footprints reach `reach` voxels from their own,
            // can touch the tile; with per-point radii the reach is that of the largest radius (ceil R
            // voxels, at most brick - 1)
            t.start = t.end = 0;
            if (t.nl27 < 0) return;
            const int reach = PPR && a.rmax ? min(a.reach, (int)ceilf(__uint_as_float(*a.rmax))) : a.reach;
            const int below = CUBIC ? reach : 0, b = a.brick, ap = a.apron, y0 = push ? 0 : -ap, y1 = push ? b - 1 : b - 1 + ap;
            int lx, hx, ly, hy, lz, hz;
            const bool nx = unit_halves(dx, b, -ap, b - 1 + ap, below, reach, lx, hx);
            const bool ny = unit_halves(dy, b, y0, y1, below, reach, ly, hy);
            const bool nz = unit_halves(dz, b, t.z0 - ap, t.z0 - ap + t.nl - 1, below, reach, lz, hz);
            if (nx && ny && nz) unit_octants(a, t, 4 * lx + 2 * ly + lz, 4 * hx + 2 * hy + hz);
        },
        [&](const SplatArgs& a, const SplatUnit& t, uint32_t, auto mid) {
            cell_unit<HAS_DEN, HAS_VEL, MODE, PPR, SMALL>(a, t, mem, &s_bar[wid], s_rs[wid], phase, lane, mid);
        });
    if (!(HAS_DEN && HAS_VEL) && lane == 0) bulk_wait_all();
}

// resident blocks per SM that the registers are budgeted for: 5 with density and velocity, whose tiles
// leave room for no more (778k points: frames of 865 us, 892 at 6); 6 else (frames of 300k points in 16^3
// bricks, three in flight: 684 us at 5, 572 at 6, 588 at 7; one at a time 912 / 1042 / 1135)
template <bool HAS_DEN, bool HAS_VEL>
constexpr int cell_min_blocks()
{
    return HAS_DEN && HAS_VEL ? 5 : 6;
}

template <bool HAS_DEN, bool HAS_VEL, int MODE, bool PPR, bool SMALL>
__global__ void __launch_bounds__(kCellWarps * 32, cell_min_blocks<HAS_DEN, HAS_VEL>()) k_splat_cells(SplatArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t units = (a.unit_count ? min(*a.unit_count, a.nslots) : a.nslots) * (uint32_t)a.slabs;
    cell_loop<kAheadAsked, HAS_DEN, HAS_VEL, MODE, PPR, SMALL>(
        a, units, a.next, smem,
        [&](uint32_t u, uint32_t& lu) {
            lu = u;
            return 0u;
        },
        [&](uint32_t) -> const SplatArgs& { return a; });
}

// The same work over many grids in one persistent launch: the units of grid
// k are [ustart[k], ustart[k+1]) of one global range, taken by the warps from
// the counter ustart[ngrids + 1] (zeroed before every launch); every grid has
// the same brick and tile shape (slab_layers, P).  AHEAD: the host knows the units, or the last frame's; with both
// ways compiled in one kernel its registers spill (24 clouds, 400k bricks, density 1.02 -> 1.12 ms).
template <int AHEAD, bool HAS_DEN, bool HAS_VEL, int MODE, bool PPR, bool SMALL>
__global__ void __launch_bounds__(kCellWarps * 32, cell_min_blocks<HAS_DEN, HAS_VEL>())
    k_splat_cells_batch(const SplatArgs* __restrict__ args, uint32_t* __restrict__ ustart, int ngrids)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint32_t s_us[kBatchMaxGrids + 1];
    for (int i = threadIdx.x; i <= ngrids; i += blockDim.x) s_us[i] = ustart[i];
    __syncthreads();
    uint32_t k = 0u;  // the last unit's grid: a warp's units come in rising order, so its search starts there
    cell_loop<AHEAD, HAS_DEN, HAS_VEL, MODE, PPR, SMALL>(
        args[0], s_us[ngrids], ustart + ngrids + 1, smem,
        [&](uint32_t u, uint32_t& lu) {
            while (s_us[k + 1] <= u) k++;
            lu = u - s_us[k];
            return k;
        },
        [&](uint32_t g) -> const SplatArgs& { return args[g]; });
}

// ---------------------------------------------------------------------------
// TRILINEAR density alone: the splat of sparse clouds (batches of point clouds, depth frames, small
// live clouds), 1-10 points a brick, where a brick's fixed work is most of it.
//
// What bounds it: the chain of a brick's lookups and candidates (about half of the issue slots are empty, with
// 17 to 23 of 24 warps resident), ahead of the HBM writes of the bricks; the general slab kernel was bound by
// issue (2 x 1,080 warp instructions on a brick of two points, 75% of the slots).  So, unlike the cells' kernel:
//  - a lane's candidates are ONE range per neighbour, from its first needed octant to its last one
//    (a superset of the needed octants, two loads instead of nine and no list of runs; the footprint
//    test drops the others), found from a candidate's number with one warp-wide OR of the ranges'
//    starts and a popcount, without a search;
//  - the hits of a round of candidates go to shared memory in order, and four of them are added at a
//    time, eight lanes (the corners of the footprint) each; lanes that meet on a voxel add one after
//    another in the points' order.  Every voxel's sum is that of the slab kernel, term by term;
//  - one unit is the whole padded brick where that leaves enough units for the chip (default_layers);
//  - the next unit's brick is known, and its neighbour list, ranges and origin are asked for, while
//    the current one is summed.
// 24 batched clouds, 5M points, 2.07M bricks: 7.10 -> 2.37 ms (8.3 GB written: 3.5 TB/s), 100k points
// in 36k bricks 92 -> 43 us, a fusion frame's splat 108 -> 84 us.
struct TriLane {
    int lox, hix, loy, hiy;  // first and last half of the lane's neighbour that can reach the tile, along x and y
    bool need;               // some half can, along both
};

// A unit with more than kDenseCandidates candidates in dense leaves (the core of a dense cloud:
// thousands of points a brick) is summed voxel by voxel, a lane each, from the cells around the voxel:
// the points of dense leaves are in cell order (k_cell_sort), so the terms of a voxel are eight runs of
// points, without a test of the others.  Terms are added in the sorted order of the points, as
// everywhere: leaf by leaf in key order, octant by octant, cell by cell; the two cells along an axis lie
// in different leaves, octants or cells of an octant, and an axis counts for the order the more the
// higher that level is.  The points of a leaf that is not dense are in index order inside an octant:
// its octants are scanned.
// Each voxel's lookups are a chain of loads: a brick of 3,000 points takes one warp half a millisecond,
// and every one below the bound loses against the pulled sum (fusion frames of 100-190 points a leaf:
// 84 us with the bound at 1500, 153 at 768 in whole bricks).  So the unit is put on a list, and
// k_tri_dense spreads its voxels over the chip (24 clouds of up to 10,600 points a leaf: the pulled
// sums of the densest brick alone take 3 of 6.8 ms; listed 4.07 + 0.24, before the claims of two).
constexpr int kDenseCandidates = 1500;
constexpr uint32_t kDenseCap = 65536;  // listed units at most; more are summed where they were met

// a point's weight at a voxel: every product rounded on its own, so that a voxel's sum has the same bits
// whichever way it is formed (left to the compiler, one copy of the code may fuse what another does not)
__device__ __forceinline__ float tri_weight(float w, float wx, float wy, float wz)
{
    return __fmul_rn(__fmul_rn(w, wx), __fmul_rn(wy, wz));
}

// the sums of voxels e0 + lane of the unit
__device__ __forceinline__ void tri_dense(const SplatArgs& a, const SplatUnit& t, int e0, int lane)
{
    const int P = a.P, P2 = P * P, ap = a.apron;
    const int nvox = t.nl * P2;
    float* out = a.den + (size_t)t.s * (P2 * P) + (size_t)t.z0 * P2;
    {
        const int e = e0 + lane;
        const bool live = e < nvox;
        const int lz = (live ? e : 0) / P2, r = (live ? e : 0) - lz * P2, ly = r / P, lx = r - ly * P;
        const int v[3] = {lx - ap, ly - ap, lz + t.z0 - ap};  // in the brick's voxels, -ap .. 7 + ap
        // an apron voxel of a missing neighbour takes the boundary value
        const int home = __shfl_sync(kFull, t.nl27, ((v[0] >> 3) + 1) * 9 + ((v[1] >> 3) + 1) * 3 + (v[2] >> 3) + 1);
        const bool bound = home < 0 && !a.accum;
        float sum = live && a.accum ? out[e] : 0.0f;
        // the axes in the order their two cells count: different leaves, then octants, then cells
        int lev[3], ax[3] = {0, 1, 2};
#pragma unroll
        for (int k = 0; k < 3; k++) lev[k] = (v[k] & 7) == 0 ? 2 : (v[k] & 7) == 4 ? 1 : 0;
        if (lev[1] > lev[0]) {
            ax[0] = 1;
            ax[1] = 0;
        }
        {
            const int la = max(lev[0], lev[1]), lb = min(lev[0], lev[1]);
            if (lev[2] > la) {
                ax[2] = ax[1];
                ax[1] = ax[0];
                ax[0] = 2;
            } else if (lev[2] > lb) {
                ax[2] = ax[1];
                ax[1] = 2;
            }
        }
        const float wv[3] = {(float)(t.org.y + v[0]), (float)(t.org.z + v[1]), (float)(t.org.w + v[2])};
#pragma unroll 1
        for (int c = 0; c < 8; c++) {
            int f[3], near[3];  // the cell along each axis; near: it is the voxel's own (else the one before)
#pragma unroll
            for (int k = 0; k < 3; k++) {
                near[k] = ax[0] == k ? (c >> 2) & 1 : ax[1] == k ? (c >> 1) & 1 : c & 1;
                f[k] = v[k] - 1 + near[k];
            }
            const int leaf = __shfl_sync(kFull, t.nl27, min(max(((f[0] >> 3) + 1) * 9 + ((f[1] >> 3) + 1) * 3 + (f[2] >> 3) + 1, 0), 31));
            if (!live || bound || leaf < 0 || f[0] < -8 || f[1] < -8 || f[2] < -8) continue;
            const int oct = ((f[0] >> 2) & 1) * 4 + ((f[1] >> 2) & 1) * 2 + ((f[2] >> 2) & 1);
            const int dense = a.leaf_dense[leaf];
            if (dense) {
                const int cell = oct * 64 + (f[0] & 3) * 16 + (f[1] & 3) * 4 + (f[2] & 3);
                const int* ct = a.cell_tab + (size_t)(dense - 1) * 512 + cell;
                const int i0 = ct[0], i1 = cell == 511 ? a.leaf_range[leaf].y : ct[1];
                for (int i = i0; i < i1; i += 4) {
                    float4 p[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) p[q] = a.spos[min(i + q, i1 - 1)];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float fx = p[q].x - (wv[0] - (float)(1 - near[0])), fy = p[q].y - (wv[1] - (float)(1 - near[1])),
                                    fz = p[q].z - (wv[2] - (float)(1 - near[2]));
                        const float w = tri_weight(p[q].w, near[0] ? 1.f - fx : fx, near[1] ? 1.f - fy : fy,
                                                   near[2] ? 1.f - fz : fz);
                        if (i + q < i1) sum = __fadd_rn(sum, w);
                    }
                }
            } else {
                // once per octant: where the axes whose two cells share it take the first
                if ((lev[0] == 0 && near[0]) || (lev[1] == 0 && near[1]) || (lev[2] == 0 && near[2])) continue;
                const int* oc = a.leaf_oct + (size_t)leaf * 8 + oct;
                const int i0 = oc[0], i1 = oct == 7 ? a.leaf_range[leaf].y : oc[1];
                for (int i = i0; i < i1; i += 4) {
                    float4 p[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) p[q] = a.spos[min(i + q, i1 - 1)];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float gx = floorf(p[q].x), gy = floorf(p[q].y), gz = floorf(p[q].z);
                        const float dx = wv[0] - gx, dy = wv[1] - gy, dz = wv[2] - gz;  // 0 or 1 where it reaches
                        const float fx = p[q].x - gx, fy = p[q].y - gy, fz = p[q].z - gz;
                        const float w = tri_weight(p[q].w, dx == 0.f ? 1.f - fx : fx, dy == 0.f ? 1.f - fy : fy,
                                                   dz == 0.f ? 1.f - fz : fz);
                        const bool in = (dx == 0.f || dx == 1.f) && (dy == 0.f || dy == 1.f) && (dz == 0.f || dz == 1.f);
                        if (i + q < i1 && in) sum = __fadd_rn(sum, w);
                    }
                }
            }
        }
        if (live) out[e] = bound ? a.boundval : sum;
    }
}

struct TriShared {
    int rs[kTriWarps][32];      // per range with points: its first sorted index, less its first candidate number
    float4 hit[kTriWarps][32];  // the hits of a round of candidates, in order
    uint64_t bar[kTriWarps];
};

// the sums of one unit into `tile` and out to HBM; mid(): called once, before the candidates
template <class Mid>
__device__ __forceinline__ void tri_unit(const SplatArgs& a, const SplatUnit& t, float* tile, TriShared& sh, int wid,
                                         int lane, uint32_t& phase, uint32_t grid, Mid mid)
{
    const int P = a.P, P2 = P * P, ap = a.apron;
    const int Ox = t.org.y - ap, Oy = t.org.z - ap, Zlo = t.org.w - ap + t.z0;
    const int nvox = t.nl * P2;
    const size_t gofs = (size_t)t.s * (P2 * P) + (size_t)t.z0 * P2;
    const uint32_t lt = (1u << lane) - 1u;
    int off;
    const int total = unit_candidates(t, lane, off);
    if (a.accum && total == 0) {  // no point reaches the slab: left as it is
        mid();
        return;
    }
    if (a.cell_tab && total > kDenseCandidates) {
        const bool dn = t.end > t.start && a.leaf_dense[t.nl27] != 0;
        if (__reduce_add_sync(kFull, dn ? t.end - t.start : 0) > kDenseCandidates) {
            mid();
            uint32_t at = kDenseCap;
            if (a.dense_units && lane == 0) at = atomicAdd(a.dense_units, 1u);
            at = __shfl_sync(kFull, at, 0);
            if (at < kDenseCap) {
                if (lane == 0) a.dense_list[at] = make_uint4(grid, t.s, (uint32_t)t.z0, (uint32_t)t.nl);
            } else {
                for (int e0 = 0; e0 < nvox; e0 += 32) tri_dense(a, t, e0, lane);
            }
            return;
        }
    }
    // (active neighbours: those in the lookup the table was made from, which are those with a slot)
    const uint32_t nbmask = __ballot_sync(kFull, t.nl27 >= 0);
    unit_ranges(t, lane, off, sh.rs[wid]);

    // ---- the tile, once the last unit's bulk store has read it
    if (lane == 0) bulk_wait_read_all();
    __syncwarp();
    if (a.accum) {
        if (lane == 0) {
            mbar_expect_tx(&sh.bar[wid], (uint32_t)nvox * 4u);
            bulk_g2s(tile, a.den + gofs, (uint32_t)nvox * 4u, &sh.bar[wid]);
        }
    } else {
        for (int i = lane; i < nvox / 4; i += 32) ((float4*)tile)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    bool loaded = !a.accum;
    mid();

    uint32_t touched = 0u;
    const int cx = lane & 1, cy = (lane >> 1) & 1, cz = (lane >> 2) & 1, hq = lane >> 3;
    for (int base = 0; base < total; base += 32) {
        const int idx = unit_candidate(t, lane, off, base, sh.rs[wid]);
        bool hit = false;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        if (base + lane < total) {
            p = a.spos[idx];
            const int x = (int)floorf(p.x) - Ox, y = (int)floorf(p.y) - Oy, z = (int)floorf(p.z) - Zlo;
            // the footprint is x, x + 1 and so on
            hit = (unsigned)(x + 1) <= (unsigned)P && (unsigned)(y + 1) <= (unsigned)P &&
                  (unsigned)(z + 1) <= (unsigned)t.nl;
            if (hit && nbmask != 0x7FFFFFFu && ap)
                touched |= box_regions(x, x + 1, y, y + 1, t.z0 + z, t.z0 + z + 1, P, ap);
        }
        const uint32_t hm = __ballot_sync(kFull, hit);
        if (hm == 0u) continue;
        if (hit) sh.hit[wid][__popc(hm & lt)] = p;
        if (!loaded) {
            if (!mbar_wait_bounded(&sh.bar[wid], phase)) atomicOr(a.err, GVX_DERR_TIMEOUT);
            phase ^= 1u;
            loaded = true;
        }
        __syncwarp();
        const int nh = __popc(hm);
        for (int h0 = 0; h0 < nh; h0 += 4) {
            const bool act = h0 + hq < nh;
            const float4 q = sh.hit[wid][act ? h0 + hq : 0];
            const float fx0 = floorf(q.x), fy0 = floorf(q.y), fz0 = floorf(q.z);
            const int x = (int)fx0 - Ox + cx, y = (int)fy0 - Oy + cy, z = (int)fz0 - Zlo + cz;
            const bool in = act && (unsigned)x < (unsigned)P && (unsigned)y < (unsigned)P && (unsigned)z < (unsigned)t.nl;
            const float fx = q.x - fx0, fy = q.y - fy0, fz = q.z - fz0;
            const float w = tri_weight(q.w, cx ? fx : 1.f - fx, cy ? fy : 1.f - fy, cz ? fz : 1.f - fz);
            const int i = (z * P + y) * P + x;
            // how many of the three earlier hits reach this voxel: its offset from their first cell is
            // 0 or 1 along every axis.  (Bytes x, y, z, all at least 1 here, compared at once; match_any
            // and a warp maximum held the unit they share 64% busy.)
            const uint32_t vb = (uint32_t)(x + 1) | (uint32_t)(y + 1) << 8 | (uint32_t)(z + 1) << 16;
            const uint32_t base = vb - (uint32_t)(cx | cy << 8 | cz << 16);
            int rank = 0;
#pragma unroll
            for (int o = 8; o <= 24; o += 8) {
                const uint32_t other = __shfl_up_sync(kFull, act ? base : 0u, o);
                rank += lane >= o && (((vb | 0x808080u) - other) & 0xFEFEFEu) == 0x808080u;
            }
            // (an inactive hit comes after the active ones: its base is never an earlier one)
            if (in && rank == 0) tile[i] = __fadd_rn(tile[i], w);
            __syncwarp();
            for (int ph = 1; __any_sync(kFull, in && rank >= ph); ph++) {
                if (in && rank == ph) tile[i] = __fadd_rn(tile[i], w);
                __syncwarp();
            }
        }
    }
    if (!loaded) {  // (candidates, but no hit: the slab as it was)
        if (!mbar_wait_bounded(&sh.bar[wid], phase)) atomicOr(a.err, GVX_DERR_TIMEOUT);
        phase ^= 1u;
        return;
    }
    __syncwarp();

    // ---- apron voxels with no neighbouring brick take the boundary value: regions that hits reached
    uint32_t reset = ~nbmask & 0x7FFFFFFu & ~(1u << 13);
    if (a.boundval == 0.0f && reset) reset &= __reduce_or_sync(kFull, touched);
    if (ap && reset && !a.accum) reset_regions<true, false>(a, (unsigned char*)tile, reset, t.z0, t.nl, P, 0, lane);

    // ---- out to HBM (the bulk store's read of the tile is waited for before the tile's next write)
    fence_async_smem();
    __syncwarp();
    if (lane == 0) {
        bulk_s2g(a.den + gofs, tile, (uint32_t)nvox * 4u);
        bulk_commit();
    }
}

template <class Of, class Args>
__device__ __forceinline__ void tri_loop(const SplatArgs& a0, uint32_t total, uint32_t* next, unsigned char* smem, Of of,
                                         Args args)
{
    __shared__ __align__(16) TriShared sh;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* tile = (float*)smem + (size_t)wid * (a0.slab_layers * a0.P * a0.P);
    if (lane == 0) {
        mbar_init(&sh.bar[wid], 1);
        mbar_fence_init();
    }
    __syncwarp();
    uint32_t phase = 0;
    TriLane L;
    const int dz = lane % 3 - 1;
    const bool nx = unit_halves(lane / 9 - 1, a0.brick, -a0.apron, a0.P - 1 - a0.apron, 0, 1, L.lox, L.hix);
    const bool ny = unit_halves(lane / 3 % 3 - 1, a0.brick, -a0.apron, a0.P - 1 - a0.apron, 0, 1, L.loy, L.hiy);
    L.need = nx && ny;
    unit_loop<kAheadAlways>(
        total, next, false, true, lane, of, args,
        [&](const SplatArgs& a, SplatUnit& t) {
            int lz, hz;
            t.start = t.end = 0;
            if (t.nl27 >= 0 && L.need && unit_halves(dz, a.brick, t.z0 - a.apron, t.z0 - a.apron + t.nl - 1, 0, 1, lz, hz))
                unit_octants(a, t, 4 * L.lox + 2 * L.loy + lz, 4 * L.hix + 2 * L.hiy + hz);
        },
        [&](const SplatArgs& a, const SplatUnit& t, uint32_t k, auto mid) {
            tri_unit(a, t, tile, sh, wid, lane, phase, k, mid);
        });
    if (lane == 0) bulk_wait_all();
}

__global__ void __launch_bounds__(kTriWarps * 32, kTriMinBlocks) k_splat_tri(SplatArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t units = (a.unit_count ? min(*a.unit_count, a.nslots) : a.nslots) * (uint32_t)a.slabs;
    tri_loop(
        a, units, a.next, smem,
        [&](uint32_t u, uint32_t& lu) {
            lu = u;
            return 0u;
        },
        [&](uint32_t) -> const SplatArgs& { return a; });
}

// the same over many grids: ustart as in k_splat_cells_batch, the counters after it
__global__ void __launch_bounds__(kTriWarps * 32, kTriMinBlocks)
    k_splat_tri_batch(const SplatArgs* __restrict__ args, uint32_t* __restrict__ ustart, int ngrids)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint32_t s_us[kBatchMaxGrids + 1];
    for (int i = threadIdx.x; i <= ngrids; i += blockDim.x) s_us[i] = ustart[i];
    __syncthreads();
    uint32_t k = 0u;  // the last unit's grid: a warp's units come in rising order, so its search starts there
    tri_loop(
        args[0], s_us[ngrids], ustart + ngrids + 1, smem,
        [&](uint32_t u, uint32_t& lu) {
            while (s_us[k + 1] <= u) k++;
            lu = u - s_us[k];
            return k;
        },
        [&](uint32_t g) -> const SplatArgs& { return args[g]; });
}

// the listed units of k_splat_tri (args: one grid's) or k_splat_tri_batch, 32 voxels a warp
__global__ void __launch_bounds__(kTriWarps * 32, 8)
    k_tri_dense(const SplatArgs* __restrict__ args, SplatArgs one, const uint32_t* __restrict__ units,
                const uint4* __restrict__ list, int chunks)
{
    const int lane = threadIdx.x & 31;
    const uint32_t total = min(*units, kDenseCap) * (uint32_t)chunks, nw = gridDim.x * kTriWarps;
    const int dx = lane / 9 - 1, dy = (lane / 3) % 3 - 1, dz = lane % 3 - 1;
    const int nbi = lane < 27 ? (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1) : -1;
    for (uint32_t u = blockIdx.x * kTriWarps + (threadIdx.x >> 5); u < total; u += nw) {
        const uint4 e = list[u / (uint32_t)chunks];
        const SplatArgs& a = args ? args[e.x] : one;
        SplatUnit t;
        t.s = e.y;
        t.z0 = (int)e.z;
        t.nl = (int)e.w;
        t.leaf = a.slot_leaf[t.s];
        unit_neighbour(a, t, nbi);
        const int e0 = (int)(u % (uint32_t)chunks) * 32;
        if (e0 < t.nl * a.P * a.P) tri_dense(a, t, e0, lane);
    }
}

// ScatterDensity, race-free: own points only, into the own padded tile.  With
// point colours (PT.cuh:555-571, 610-642) each point also colours the interior
// voxel it lies in: clr_mode 1 (avgColor) = integer mean of the voxel's
// points' r, g, b with alpha 255, into channel 1; clr_mode 2 = the colour of
// the voxel's highest-index point (the reference's writers race), channel 3.
// Both are counted with shared-memory integer atomics: deterministic.
struct ScatterArgs {
    int brick, P, apron;
    uint32_t nslots;
    const int* slot_leaf;
    const GvxNode* nodes0;
    const int2* leaf_range;
    const float4* spos;
    float radius;
    int expand;
    float* den;
    uint32_t* err;
    int block_points;         // bricks of at least so many points are k_scatter_ref's
    int clr_mode;             // 0 none, 1 average, 2 one point's colour
    const uint32_t* perm;     // sorted position -> point index
    const char* clr;
    int clr_off, clr_stride;
    uint32_t* clr_out;        // 4-byte channel, brick-major padded
};

// The same for bricks up to 8, a warp each.  The block per brick below stages the whole brick for its
// points, 17 in the sample's frame, and waits for every step in turn.  Here the points add their seven
// values to the channel by reductions in L2, which nothing waits for, and a warp's colour table is cleared
// by the lanes that read it, so that its cost follows the points too.
// A million points in 57k bricks, averaged colours: 278 us by blocks, 87 here.
constexpr int kScatterWarps = 4;
// bricks of so many points are k_scatter_ref's: a million points in 1728 bricks (580 each) 31 us there and
// 52 here, in 57k bricks (17 each) 278 there and 87 here
constexpr int kScatterBlock = 256;
__global__ void __launch_bounds__(kScatterWarps * 32) k_scatter_points(ScatterArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int P = a.P, P3 = P * P * P, b = a.brick, ap = a.apron, b3 = b * b * b;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // average: count, r, g, b per interior voxel, 0 between bricks; one point: 1 + its index, 0 between bricks
    uint32_t* tclr = (uint32_t*)smem + (size_t)wid * (a.clr_mode == 1 ? 4 * b3 : b3);
    if (a.clr_mode)
        for (int i = lane; i < (a.clr_mode == 1 ? 4 * b3 : b3); i += 32) tclr[i] = 0u;
    __syncwarp();
    const float r2 = a.radius * a.radius;
    const int cnt = a.expand ? 7 : 1;
    const uint32_t nw = gridDim.x * kScatterWarps;
    for (uint32_t s = blockIdx.x * kScatterWarps + wid; s < a.nslots; s += nw) {
        const int leaf = a.slot_leaf[s];
        const int2 rg = a.leaf_range[leaf];
        if (rg.y <= rg.x || rg.y - rg.x >= a.block_points) continue;  // no point: the brick is left as it is
        const int4 org = *(const int4*)(a.nodes0 + leaf);
        const float vx = (float)org.y, vy = (float)org.z, vz = (float)org.w;
        float* den = a.den + (size_t)s * P3;
        for (int e0 = rg.x; e0 < rg.y; e0 += 32) {
            const int e = e0 + lane;
            if (e >= rg.y) continue;
            const float4 w = a.spos[e];
            const float px = w.x - vx, py = w.y - vy, pz = w.z - vz;
            const float pix = (float)(int)px, piy = (float)(int)py, piz = (float)(int)pz;
            if (pix < 0 || piy < 0 || piz < 0 || pix >= b || piy >= b || piz >= b) continue;
            if (a.clr_mode) {
                const int v = ((int)piz * b + (int)piy) * b + (int)pix;
                const uint32_t pt = a.perm[e];
                if (a.clr_mode == 1) {
                    const uint32_t c = *(const uint32_t*)(a.clr + (size_t)pt * (size_t)a.clr_stride + a.clr_off);
                    atomicAdd(&tclr[v], 1u);
                    atomicAdd(&tclr[b3 + v], c & 255u);
                    atomicAdd(&tclr[2 * b3 + v], (c >> 8) & 255u);
                    atomicAdd(&tclr[3 * b3 + v], (c >> 16) & 255u);
                } else {
                    atomicMax(&tclr[v], pt + 1u);  // the highest point index
                }
            }
            for (int k = 0; k < cnt; k++) {
                const int ox = (k == 1) ? -1 : (k == 2) ? 1 : 0;
                const int oy = (k == 3) ? -1 : (k == 4) ? 1 : 0;
                const int oz = (k == 5) ? -1 : (k == 6) ? 1 : 0;
                const float bx = pix + ox - px, by = piy + oy - py, bz = piz + oz - pz;
                const float c = (bx * bx + by * by + bz * bz) / r2;
                const float v = 1.0f + c * (-3.0f + c * (3.0f - c));
                const int lx = (int)pix + ox + ap, ly = (int)piy + oy + ap, lz = (int)piz + oz + ap;
                if (lx < 0 || ly < 0 || lz < 0 || lx >= P || ly >= P || lz >= P) continue;
                atomicAdd(&den[(lz * P + ly) * P + lx], v);
            }
        }
        if (!a.clr_mode) continue;
        __syncwarp();
        // each coloured voxel by the one lane that takes its count (its point): the others find 0
        uint32_t* out = a.clr_out + (size_t)s * P3;
        for (int e0 = rg.x; e0 < rg.y; e0 += 32) {
            const int e = e0 + lane;
            if (e < rg.y) {
                const float4 w = a.spos[e];
                const int x = (int)(w.x - vx), y = (int)(w.y - vy), z = (int)(w.z - vz);
                if (x >= 0 && y >= 0 && z >= 0 && x < b && y < b && z < b) {
                    const int v = (z * b + y) * b + x, o = ((z + ap) * P + (y + ap)) * P + (x + ap);
                    const uint32_t n = atomicExch(&tclr[v], 0u);
                    if (n != 0u && a.clr_mode == 1) {
                        out[o] = (tclr[b3 + v] / n & 255u) | ((tclr[2 * b3 + v] / n & 255u) << 8) |
                                 ((tclr[3 * b3 + v] / n & 255u) << 16) | (255u << 24);
                        tclr[b3 + v] = tclr[2 * b3 + v] = tclr[3 * b3 + v] = 0u;
                    } else if (n != 0u) {
                        out[o] = *(const uint32_t*)(a.clr + (size_t)(n - 1u) * (size_t)a.clr_stride + a.clr_off);
                    }
                }
            }
            __syncwarp();
        }
    }
}

// A brick a block, staged in shared memory.  RUNS: for bricks of many points, whose neighbours in the order share
// voxels: a thread sums a run of points (see below), in 60 registers; without, in 40, two blocks more an SM (300k
// points in 2.2k bricks 15 us with runs, 12 without; 27 bricks of thousands, in cell order, 207 us with, 1590
// without).
template <bool RUNS>
__global__ void __launch_bounds__(kSplatThreads) k_scatter_ref(ScatterArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    float* tden = (float*)smem;
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ uint32_t s_list[kSplatThreads];
    __shared__ int s_n;
    const int P = a.P, P3 = P * P * P, b = a.brick, ap = a.apron, tid = threadIdx.x, b3 = b * b * b;
    const uint32_t bytes = (uint32_t)P3 * 4u;
    // colour tables after the tile: average = count, r, g, b per interior voxel; one point = its index
    uint32_t* tclr = (uint32_t*)(smem + (((size_t)P3 * 4 + 15) & ~(size_t)15));
    if (tid == 0) {
        mbar_init(&s_bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    uint32_t phase = 0;
    const float r2 = a.radius * a.radius;
    // the block's slots, a thread each: those with points enough are listed (with block_points 1 the blocks are few
    // turns long, and take their slots as they come)
    const bool direct = a.block_points <= 1;
    for (uint64_t r = blockIdx.x; r < a.nslots; r += (direct ? 1u : (uint64_t)kSplatThreads) * gridDim.x) {
        int listed = 1;
        if (!direct) {
            if (tid == 0) s_n = 0;
            __syncthreads();
            const uint64_t mine = r + (uint64_t)tid * gridDim.x;
            if (mine < a.nslots) {
                const int2 q = a.leaf_range[a.slot_leaf[mine]];
                if (q.y - q.x >= a.block_points) s_list[atomicAdd(&s_n, 1)] = (uint32_t)mine;
            }
            __syncthreads();
            listed = s_n;
        }
        for (int l = 0; l < listed; l++) {
            const uint32_t s = direct ? (uint32_t)r : s_list[l];
            const int leaf = a.slot_leaf[s];
            const GvxNode& nd = a.nodes0[leaf];
            const int2 rg = a.leaf_range[leaf];
            if (rg.y <= rg.x) break;  // no point: the brick is left as it is
            if (tid == 0) {
                mbar_expect_tx(&s_bar, bytes);
                bulk_g2s(tden, a.den + (size_t)s * P3, bytes, &s_bar);
            }
            if (a.clr_mode) {
                const int words = a.clr_mode == 1 ? 4 * b3 : b3;
                const uint32_t init = a.clr_mode == 1 ? 0u : 0xFFFFFFFFu;
                for (int i = tid; i < words; i += kSplatThreads) tclr[i] = init;
            }
            if (!mbar_wait_bounded(&s_bar, phase)) atomicOr(a.err, GVX_DERR_TIMEOUT);
            phase ^= 1u;
            if (a.clr_mode) __syncthreads();
            const float vx = (float)nd.pos[0], vy = (float)nd.pos[1], vz = (float)nd.pos[2];
            const int cnt = a.expand ? 7 : 1;
            // a run of points a thread (lanes side by side in a dense brick's order would add to one word): those
            // of one voxel, neighbours in that order, are summed in registers and added to the tile once with RUNS
            const int chunk = (rg.y - rg.x + kSplatThreads - 1) / kSplatThreads;
            const int e1 = min(rg.x + (tid + 1) * chunk, rg.y);
            float sum[7];
            uint32_t cn = 0u, cr = 0u, cg = 0u, cb = 0u;
            int cur = -1, qx = 0, qy = 0, qz = 0;
            auto flush = [&]() {
                if (cur < 0) return;
                if (a.clr_mode == 1) {
                    atomicAdd(&tclr[cur], cn);
                    atomicAdd(&tclr[b3 + cur], cr);
                    atomicAdd(&tclr[2 * b3 + cur], cg);
                    atomicAdd(&tclr[3 * b3 + cur], cb);
                } else if (a.clr_mode == 2) {
                    atomicMax((int*)&tclr[cur], (int)cn);  // the highest point index; -1 = none
                }
#pragma unroll
                for (int k = 0; k < 7; k++) {
                    if (k >= cnt) break;
                    const int lx = qx + ap + (k == 1 ? -1 : k == 2 ? 1 : 0), ly = qy + ap + (k == 3 ? -1 : k == 4 ? 1 : 0),
                              lz = qz + ap + (k == 5 ? -1 : k == 6 ? 1 : 0);
                    if (lx < 0 || ly < 0 || lz < 0 || lx >= P || ly >= P || lz >= P) continue;
                    atomicAdd(&tden[(lz * P + ly) * P + lx], sum[k]);
                }
            };
            for (int e = rg.x + tid * chunk; e < e1; e++) {
                const float4 w = a.spos[e];
                const float px = w.x - vx, py = w.y - vy, pz = w.z - vz;
                const float pix = (float)(int)px, piy = (float)(int)py, piz = (float)(int)pz;
                if (pix < 0 || piy < 0 || piz < 0 || pix >= b || piy >= b || piz >= b) continue;
                const int v = ((int)piz * b + (int)piy) * b + (int)pix;
                if (!RUNS) {
                    if (a.clr_mode) {
                        const uint32_t pt = a.perm[e];
                        if (a.clr_mode == 1) {
                            const uint32_t c = *(const uint32_t*)(a.clr + (size_t)pt * (size_t)a.clr_stride + a.clr_off);
                            atomicAdd(&tclr[v], 1u);
                            atomicAdd(&tclr[b3 + v], c & 255u);
                            atomicAdd(&tclr[2 * b3 + v], (c >> 8) & 255u);
                            atomicAdd(&tclr[3 * b3 + v], (c >> 16) & 255u);
                        } else {
                            atomicMax((int*)&tclr[v], (int)pt);
                        }
                    }
                    for (int k = 0; k < cnt; k++) {
                        const int ox = (k == 1) ? -1 : (k == 2) ? 1 : 0;
                        const int oy = (k == 3) ? -1 : (k == 4) ? 1 : 0;
                        const int oz = (k == 5) ? -1 : (k == 6) ? 1 : 0;
                        const float bx = pix + ox - px, by = piy + oy - py, bz = piz + oz - pz;
                        const float c = (bx * bx + by * by + bz * bz) / r2;
                        const int lx = (int)pix + ox + ap, ly = (int)piy + oy + ap, lz = (int)piz + oz + ap;
                        if (lx < 0 || ly < 0 || lz < 0 || lx >= P || ly >= P || lz >= P) continue;
                        atomicAdd(&tden[(lz * P + ly) * P + lx], 1.0f + c * (-3.0f + c * (3.0f - c)));
                    }
                    continue;
                }
                if (v != cur) {
                    flush();
                    cur = v, qx = (int)pix, qy = (int)piy, qz = (int)piz;
                    cn = cr = cg = cb = 0u;
#pragma unroll
                    for (int k = 0; k < 7; k++) sum[k] = 0.f;
                }
                if (a.clr_mode) {
                    const uint32_t pt = a.perm[e];
                    if (a.clr_mode == 1) {
                        const uint32_t c = *(const uint32_t*)(a.clr + (size_t)pt * (size_t)a.clr_stride + a.clr_off);
                        cn++;
                        cr += c & 255u;
                        cg += (c >> 8) & 255u;
                        cb += (c >> 16) & 255u;
                    } else {
                        cn = max(cn, pt);
                    }
                }
#pragma unroll
                for (int k = 0; k < 7; k++) {
                    if (k >= cnt) break;
                    const int ox = (k == 1) ? -1 : (k == 2) ? 1 : 0;
                    const int oy = (k == 3) ? -1 : (k == 4) ? 1 : 0;
                    const int oz = (k == 5) ? -1 : (k == 6) ? 1 : 0;
                    const float bx = pix + ox - px, by = piy + oy - py, bz = piz + oz - pz;
                    const float c = (bx * bx + by * by + bz * bz) / r2;
                    sum[k] += 1.0f + c * (-3.0f + c * (3.0f - c));
                }
            }
            if (RUNS) flush();
            fence_async_smem();
            __syncthreads();
            if (tid == 0) {
                bulk_s2g(a.den + (size_t)s * P3, tden, bytes);
                bulk_commit();
            }
            if (a.clr_mode) {
                uint32_t* out = a.clr_out + (size_t)s * P3;
                for (int v = tid; v < b3; v += kSplatThreads) {
                    const int o = (((v / (b * b)) + ap) * P + ((v / b) % b + ap)) * P + (v % b + ap);
                    if (a.clr_mode == 1) {
                        const uint32_t n = tclr[v];
                        if (n == 0u) continue;
                        out[o] = (tclr[b3 + v] / n & 255u) | ((tclr[2 * b3 + v] / n & 255u) << 8) |
                                 ((tclr[3 * b3 + v] / n & 255u) << 16) | (255u << 24);
                    } else {
                        const int pt = (int)tclr[v];
                        if (pt < 0) continue;
                        out[o] = *(const uint32_t*)(a.clr + (size_t)pt * (size_t)a.clr_stride + a.clr_off);
                    }
                }
            }
            if (tid == 0) bulk_wait_read_all();
            __syncthreads();
        }
        if (!direct) __syncthreads();  // (the list is read before its count is cleared)
    }
    if (tid == 0) bulk_wait_all();
}

// ---------------------------------------------------------------------------

static inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// InsertPoints (VG.cpp:5219-5267): group the points by brick (topology sort,
// reused when the points and translation are those of the rebuild) and write
// the sorted float4 attribute arrays the splat kernels stream through
gvx_status gvx_prepare_points(gvx_grid* g, int n, const float trans[3], bool need_svel)
{
    const float t[3] = {trans ? trans[0] : 0.f, trans ? trans[1] : 0.f, trans ? trans[2] : 0.f};
    gvx_status rc = gvx_wait_attributes(g);
    if (rc) return rc;
    rc = gvx_topo_group_points(g, n, t);
    if (rc) return rc;
    const bool want_svel = need_svel || g->pts.vel || g->pts.radius;
    const uint32_t m = g->n_sorted;
    auto attr_buffers = [&](unsigned int** rmax) -> gvx_status {
        GVX_CK(gvx_ensure(g->spos, (size_t)std::max<uint32_t>(m, 1u) * sizeof(float4)));
        if (want_svel) GVX_CK(gvx_ensure(g->svel, (size_t)std::max<uint32_t>(m, 1u) * sizeof(float4)));
        *rmax = nullptr;
        if (g->pts.radius && want_svel) {
            GVX_CK(gvx_ensure(g->d_rmax, sizeof(unsigned int)));
            GVX_CK(cudaMemsetAsync(g->d_rmax.p, 0, sizeof(unsigned int), g->stream));
            *rmax = g->d_rmax.as<unsigned int>();
        }
        return GVX_OK;
    };
    auto mark_permuted = [&]() {
        g->perm_valid = true;
        g->perm_has_svel = want_svel;
        g->perm_vel = g->pts.vel;
        g->perm_w = g->pts.weight;
        g->perm_r = g->pts.radius;
    };
    if (!g->oct_valid) {
        // a new grouping: the octant pass (the sorted attributes; the octant order itself where the
        // sort keys could not carry it)
        unsigned int* rmax = nullptr;
        rc = attr_buffers(&rmax);
        if (rc) return rc;
        GvxSortedAttr A;
        A.vel = g->pts.vel;
        A.vel_off = g->pts.vel_off;
        A.vel_stride = g->pts.vel_stride;
        A.weight = g->pts.weight;
        A.radius = g->pts.radius;
        A.spos = g->spos.as<float4>();
        A.svel = want_svel ? g->svel.as<float4>() : nullptr;
        A.rmax = rmax;
        rc = gvx_topo_octants(g, &A);
        if (rc) return rc;
        mark_permuted();
        return GVX_OK;
    }
    if (g->perm_valid && (g->perm_has_svel || !need_svel) && g->perm_vel == g->pts.vel &&
        g->perm_w == g->pts.weight && g->perm_r == g->pts.radius)
        return GVX_OK;
    // the same grouping with other attributes: the permute alone
    unsigned int* rmax = nullptr;
    rc = attr_buffers(&rmax);
    if (rc) return rc;
    if (m) {
        CellOrder co;
        memset(&co, 0, sizeof(co));
        if (g->leaf_dense && g->dense_leaves != 0) {
            co.skeys = g->keys[g->sorted_buf].as<uint32_t>();
            co.invalid_key = 1u << g->lookup.ks.total_bits;
            co.L = g->lookup;
            co.nodes0 = g->nodes[0].as<GvxNode>();
            co.leaf_range = g->leaf_range.as<int2>();
            co.cell_tab = g->cell_tab.as<int>();
            co.leaf_dense = g->leaf_dense;
        }
        k_permute<<<blocks_for(m, 256), 256, 0, g->stream>>>(
            g->vals[g->sorted_buf].as<uint32_t>(), m, g->pts.pos, g->pts.pos_off, g->pts.pos_stride, g->pts.vel,
            g->pts.vel_off, g->pts.vel_stride, g->pts.weight, g->pts.radius, t[0], t[1], t[2], g->spos.as<float4>(),
            want_svel ? g->svel.as<float4>() : nullptr, rmax, co);
        g->launches++;
    }
    GVX_CK(cudaGetLastError());
    mark_permuted();
    return GVX_OK;
}

static gvx_status check_splat_state(gvx_grid* g, const char* what)
{
    if (g->root_level < 0 || !g->lookup_valid) {
        gvx_set_error("%s: no topology", what);
        return GVX_ERR_STATE;
    }
    if (!g->atlas_valid) {
        gvx_set_error("%s: UpdateAtlas was not called after the topology changed", what);
        return GVX_ERR_STATE;
    }
    return GVX_OK;
}

static int sm_count(int device)
{
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
    return v > 0 ? v : 152;
}

// kernel variant: channel set x mode x per-point radius
struct SplatKind {
    bool has_d, has_v, ppr;
    int mode;
    bool small;  // footprint within 4 voxels a side: trilinear, or cubic of a uniform radius <= 2
    bool operator==(const SplatKind& o) const
    {
        return has_d == o.has_d && has_v == o.has_v && ppr == o.ppr && mode == o.mode && small == o.small;
    }
};

// the splats of k_splat_tri
static bool tri_kind(const SplatKind& k) { return k.mode == GVX_SPLAT_TRILINEAR && k.has_d && !k.has_v; }

// the kernel of a kind (single grid, batch, batch of few units), its warps a block and its shared memory a warp
struct SplatKernel {
    void *one, *batch, *batch_few;
    int warps;
    size_t (*warp_bytes)(int layers, int rows, int P);
};
static size_t tri_warp_bytes(int layers, int rows, int P) { return (size_t)layers * rows * P * sizeof(float); }

template <bool D, bool V, int MODE, bool PPR, bool SMALL>
static SplatKernel cell_kernel()
{
    return SplatKernel{(void*)k_splat_cells<D, V, MODE, PPR, SMALL>,
                       (void*)k_splat_cells_batch<kAheadAlways, D, V, MODE, PPR, SMALL>,
                       (void*)k_splat_cells_batch<kAheadNever, D, V, MODE, PPR, SMALL>, kCellWarps, cell_warp_bytes<D, V, MODE, PPR>};
}
template <bool D, bool V>
static SplatKernel pick_kernel(const SplatKind& k)
{
    if (k.mode == GVX_SPLAT_TRILINEAR) {
        if constexpr (D && !V)
            return SplatKernel{(void*)k_splat_tri, (void*)k_splat_tri_batch, (void*)k_splat_tri_batch, kTriWarps,
                               tri_warp_bytes};
        else
            return cell_kernel<D, V, GVX_SPLAT_TRILINEAR, false, true>();
    }
    if (k.ppr) return cell_kernel<D, V, GVX_SPLAT_CUBIC, true, false>();
    return k.small ? cell_kernel<D, V, GVX_SPLAT_CUBIC, false, true>() : cell_kernel<D, V, GVX_SPLAT_CUBIC, false, false>();
}

// whether a launch of `warps` warps over so many units has few of them
static bool few_units(uint64_t units, uint64_t warps, bool light)
{
    return units < (light ? kAheadLight : kAheadUnits) * warps;
}

static SplatKernel splat_kernel(const SplatKind& k)
{
    return k.has_d ? (k.has_v ? pick_kernel<true, true>(k) : pick_kernel<true, false>(k)) : pick_kernel<false, true>(k);
}

// Tile geometry of a grid's splat: a push tile (apron 1, not accumulating) covers the interior
// rows and layers of the padded brick, else the whole padded brick; `span` layers to cover,
// `rows` rows a layer
struct SlabShape {
    bool push;
    int span, rows;
};
static SlabShape slab_shape(const gvx_grid* g, int accum, bool dense, bool den_vel)
{
    const bool push = g->apron == 1 && !accum && dense && den_vel;
    return SlabShape{push, push ? g->brick : g->P, push ? g->brick : g->P};
}

// Points per active brick from which the push tile is used (and only by the splat of density
// with velocity, the only kernels compiled with it: the others keep their registers): its
// scattered apron stores cost a slab several hundred more instructions, which the
// interior-only dealing repays on dense clouds (4M SPH frame, 14 a brick: 3.04 -> 2.95 ms)
// and not on sparse ones (the batched clouds, 4.6 a brick: 15.3 -> 18.8 ms with it)
constexpr uint64_t kPushPointsPerBrick = 8;
static bool dense_cloud(uint64_t points, uint64_t bricks)
{
    return bricks > 0 && points >= kPushPointsPerBrick * bricks;
}

// the largest slab (in layers) whose tile fits the per-warp budget, at most `want`
static int clamp_layers(const SlabShape& sh, int P, size_t eb, int want)
{
    const int fit = (int)(kSlabTileMax / ((size_t)sh.rows * P * eb));
    return std::min(std::min(want, sh.span), fit);
}

// The slab height a splat takes by itself: a push tile the brick's whole interior (one unit a brick: the
// candidate ranges and the z pushes once), others the whole padded brick where its tile is small, else
// half of it -- and lower slabs where that leaves fewer than kUnitsWanted units, down to five layers, and, but for
// the trilinear density splat, whose units are light, to two (push tiles too) where it leaves fewer than
// kUnitsLeast: dealing a brick's candidates again for every slab costs less than warps without work.  Measured
// (bricks, density alone unless said): trilinear 36k of 8^3 whole 43 us, halves 65; 2.07M 2.4 / 3.3 ms;
// 720 of them 14 us whole, 10.1 halves, 10.9 of four layers, 11.3 of two; cubic of per-point radii 1-3,
// 238k: 0.86 ms whole, 1.13 halves, 1.67 of three layers; cubic of 8k points around one brick, 47 in all: R 2
// 1.89 ms halves, 1.64 of three layers, 1.25 of two, R 6.5 22.6 / 14.5 / 9.5, with velocity 2.57 ms whole
// interiors, 1.25 of two layers; 100k points in 729: R 3.5 0.86 ms halves, 0.48 of two layers, in 3.4k: R 2 101 us
// halves, 109 of three layers.
constexpr uint64_t kUnitsWanted = 152 * 24 * 3, kUnitsLeast = 152 * 24;
constexpr size_t kWholeTile = 6 * 1024;
static int default_layers(const SlabShape& sh, int P, size_t eb, uint64_t bricks, bool tri)
{
    int l = sh.push || (size_t)sh.span * sh.rows * P * eb <= kWholeTile ? sh.span : (sh.span + 1) / 2;
    for (;;) {
        const uint64_t units = bricks * (uint64_t)((sh.span + l - 1) / l);
        const bool few = units < kUnitsWanted && !sh.push && l > 5, very_few = units < kUnitsLeast && !tri && l > 2;
        if (!few && !very_few) return l;
        l = (l + 1) / 2;
    }
}

// validation of one grid's splat and its kernel kind (bricks: how many the launch covers); *layers in:
// the wanted slab height (<= 0: the default), out: clamped to the tile budget
static gvx_status splat_check(gvx_grid* g, int mode, float radius, int chan_d, int chan_v, int accum,
                              bool dense, uint64_t bricks, int* layers, SplatKind* kind)
{
    if (mode != GVX_SPLAT_TRILINEAR && mode != GVX_SPLAT_CUBIC) {
        gvx_set_error("Splat: unknown mode %d", mode);
        return GVX_ERR_INVALID_ARG;
    }
    const bool has_d = chan_d >= 0, has_v = chan_v >= 0;
    if (!has_d && !has_v) {
        gvx_set_error("Splat: no output channel");
        return GVX_ERR_INVALID_ARG;
    }
    if (has_d && (chan_d >= GVX_MAXCH || !g->ch[chan_d].used || g->ch[chan_d].type != GVX_T_FLOAT)) {
        gvx_set_error("Splat: density channel %d must be a T_FLOAT channel", chan_d);
        return GVX_ERR_INVALID_ARG;
    }
    if (has_v && (chan_v >= GVX_MAXCH || !g->ch[chan_v].used || g->ch[chan_v].elem_bytes != 16)) {
        gvx_set_error("Splat: velocity channel %d must be a T_FLOAT3/T_FLOAT4 channel", chan_v);
        return GVX_ERR_INVALID_ARG;
    }
    const bool ppr = mode == GVX_SPLAT_CUBIC && g->pts.radius != nullptr;
    if (mode == GVX_SPLAT_CUBIC && !ppr && !(radius > 0.f)) {
        gvx_set_error("Splat: cubic splat needs a radius > 0");
        return GVX_ERR_INVALID_ARG;
    }
    if (mode == GVX_SPLAT_CUBIC && !ppr && radius > (float)(g->brick - 1)) {
        gvx_set_error("Splat: radius %g reaches beyond the 26 neighbouring bricks", radius);
        return GVX_ERR_UNSUPPORTED;
    }
    if (g->brick < 2) {
        gvx_set_error("Splat: bricks of 1 voxel are not supported (tiles are moved in 16-byte units)");
        return GVX_ERR_UNSUPPORTED;
    }
    const int P = g->P;
    const SlabShape sh = slab_shape(g, accum, dense, has_d && has_v);
    const size_t eb = has_v ? 16 : 4;
    const bool tri = mode == GVX_SPLAT_TRILINEAR && has_d && !has_v;
    *layers = clamp_layers(sh, P, eb, *layers > 0 ? *layers : default_layers(sh, P, eb, bricks, tri));
    if (*layers < 1) {
        gvx_set_error("Splat: a %d^2 layer of the padded brick exceeds the shared tile budget", P);
        return GVX_ERR_UNSUPPORTED;
    }
    kind->has_d = has_d;
    kind->has_v = has_v;
    kind->ppr = ppr;
    kind->mode = mode;
    kind->small = mode == GVX_SPLAT_TRILINEAR || (!ppr && radius <= 2.0f);
    return GVX_OK;
}

// the kernel arguments of one grid's splat over its current grouping and atlas
static void splat_fill(gvx_grid* g, const SplatKind& k, float radius, int chan_d, int chan_v, int accum, bool dense,
                       int layers, SplatArgs* out)
{
    const bool need_svel = k.has_v || k.ppr;
    const int P = g->P;
    SplatArgs& a = *out;
    memset(&a, 0, sizeof(a));
    a.brick = g->brick;
    a.P = P;
    a.apron = g->apron;
    a.nslots = (uint32_t)g->atlas_used;
    a.slot_leaf = g->slot_leaf.as<int>();
    a.leaf_slot = g->leaf_slot.as<int>();
    a.nodes0 = g->nodes[0].as<GvxNode>();
    a.nbr = g->nbr.as<int>();
    a.leaf_range = g->leaf_range.as<int2>();
    a.leaf_oct = g->leaf_oct.as<int>();
    a.leaf_dense = g->leaf_dense;
    a.cell_tab = g->leaf_dense ? g->cell_tab.as<int>() : nullptr;
    a.spos = g->spos.as<float4>();
    a.svel = need_svel ? g->svel.as<float4>() : nullptr;
    a.per_point_radius = k.ppr;
    a.radius = radius;
    a.den = k.has_d ? g->ch[chan_d].data.as<float>() : nullptr;
    a.vel = k.has_v ? g->ch[chan_v].data.as<float4>() : nullptr;
    const SlabShape sh = slab_shape(g, accum, dense, k.has_d && k.has_v);
    a.push = sh.push;
    if (sh.push && layers == sh.span && g->push_tab_P == P) {
        a.push_tab = g->push_tab.as<uint32_t>();
        a.push_count = g->push_count;
    }
    a.tile_rows = sh.rows;
    a.slab_layers = layers;
    a.slabs = (sh.span + layers - 1) / layers;
    a.lb = 0;
    while ((1 << a.lb) < g->brick) a.lb++;
    a.max_radius = (float)(g->brick - 1);
    a.reach = k.mode == GVX_SPLAT_TRILINEAR ? 1 : (k.ppr ? g->brick - 1 : (int)ceilf(radius));
    a.rmax = k.ppr && g->n_sorted ? g->d_rmax.as<unsigned int>() : nullptr;
    a.accum = accum != 0;
    a.boundval = 0.0f;
    a.err = g->d_err.as<uint32_t>();
}

// The table of push_out for push tiles of one unit a brick: per boundary voxel and neighbour (0, dy, dz)
// that takes it, its place in the tile, its place in the neighbour's padded brick << 12, the lane that
// holds the neighbour's slot << 24; filled up to a multiple of 32 with the last entry.
static gvx_status push_table(gvx_grid* g)
{
    const int P = g->P, b = g->brick;
    if (g->push_tab_P == P) return GVX_OK;
    std::vector<uint32_t> t;
    for (int dz = -1; dz <= 1; dz++)
        for (int dy = -1; dy <= 1; dy++) {
            if (dy == 0 && dz == 0) continue;
            for (int lz = 0; lz < b; lz++)
                for (int ly = 0; ly < b; ly++) {
                    if ((dy < 0 && ly != 0) || (dy > 0 && ly != b - 1) || (dz < 0 && lz != 0) || (dz > 0 && lz != b - 1))
                        continue;
                    const int yr = dy < 0 ? P - 1 : dy > 0 ? 0 : ly + 1, zr = dz < 0 ? P - 1 : dz > 0 ? 0 : lz + 1;
                    for (int x = 0; x < P; x++)
                        t.push_back((uint32_t)((lz * b + ly) * P + x) | (uint32_t)((zr * P + yr) * P + x) << 12 |
                                    (uint32_t)(9 + (dy + 1) * 3 + (dz + 1)) << 24);
                }
        }
    while (t.size() % 32) t.push_back(t.back());
    GVX_CK(gvx_ensure(g->push_tab, t.size() * sizeof(uint32_t)));
    GVX_CK(cudaMemcpyAsync(g->push_tab.p, t.data(), t.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, g->stream));
    GVX_CK(cudaStreamSynchronize(g->stream));
    g->push_tab_P = P;
    g->push_count = (int)t.size();
    return GVX_OK;
}

// (an accumulating splat's units are the bricks that points reach, which the host does not know)
static bool light_units(uint64_t points, uint64_t units, int accum) { return !accum && points < kLightPoints * units; }

// validation, InsertPoints grouping and the kernel arguments of one grid's splat;
// layers <= 0 picks the default slab height (see splat_check); dense < 0: the tile shape from the
// grid's own points per brick, else as given (a batch decides for all its grids)
static gvx_status splat_prepare(gvx_grid* g, int mode, int n, float radius, const float trans[3], int chan_d,
                                int chan_v, int accum, int layers, int dense, uint64_t bricks, SplatArgs* out,
                                SplatKind* kind)
{
    gvx_status rc = check_splat_state(g, "Splat");
    if (rc) return rc;
    const bool dn = dense < 0 ? dense_cloud((uint64_t)n, (uint64_t)g->atlas_used) : dense != 0;
    rc = splat_check(g, mode, radius, chan_d, chan_v, accum, dn, bricks ? bricks : (uint64_t)g->atlas_used, &layers, kind);
    if (rc) return rc;
    rc = gvx_prepare_points(g, n, trans, kind->has_v || kind->ppr);
    if (rc) return rc;
    // (a tile of the whole interior has at most 4096 places: bricks up to 8)
    if (slab_shape(g, accum, dn, kind->has_d && kind->has_v).push && g->brick <= 8) GVX_CK_STATUS(push_table(g));
    splat_fill(g, *kind, radius, chan_d, chan_v, accum, dn, layers, out);
    out->light = light_units((uint64_t)n, (uint64_t)out->nslots * out->slabs, accum);
    return GVX_OK;
}

// one tile shape for the grids of a batch: from their points and bricks together
static bool batch_dense(const gvx_batch* b);

// apron state after the splat: exact copies with boundary value 0, unless an
// accumulating splat started from an apron that was not a valid copy
static void splat_finish(gvx_grid* g, int chan_d, int chan_v, int accum)
{
    for (int c : {chan_d, chan_v}) {
        if (c < 0) continue;
        GvxChannel& ch = g->ch[c];
        if (!accum) {
            ch.apron_valid = true;  // every apron voxel is the neighbour's sum, or 0 where no brick is
            ch.apron_partial_from = -1;
        } else if (ch.apron_bv != 0.0f) {
            apron_invalidate(ch);
        }
        // accumulating onto copies (all of them, or all but those near new bricks) adds the same
        // sums to both sides of every copy: the state is kept
        ch.apron_bv = 0.0f;
    }
}

static size_t splat_smem(const SplatArgs& a, const SplatKernel& k)
{
    return k.warp_bytes(a.slab_layers, a.tile_rows, a.P) * (size_t)k.warps;
}

// The slots whose brick has points of the current grouping in itself or one of its 26 neighbours:
// the only bricks an accumulating splat changes (the others it leaves as they are, loading and
// storing nothing).  Lane r < 27 of a warp tests neighbour r of eight slots at a time (each is a chain of
// three loads); a block takes its room in the list with one atomic, since those, one after the other on
// one address, were what bounded a warp per slot: 129k slots 20 us, 3.8 here.  Each unit writes its own
// brick only, so the order of the list does not matter.
constexpr int kTouchedWarps = 8, kTouchedPer = 8;
__global__ void __launch_bounds__(kTouchedWarps * 32)
    k_touched_slots(const int* __restrict__ slot_leaf, uint32_t nslots, const int* __restrict__ nbr,
                    const int2* __restrict__ leaf_range, uint32_t* __restrict__ out, uint32_t* __restrict__ count)
{
    __shared__ uint32_t s_bits[kTouchedWarps], s_base[kTouchedWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t s0 = (blockIdx.x * kTouchedWarps + wid) * kTouchedPer;
    int nl[kTouchedPer];
#pragma unroll
    for (int k = 0; k < kTouchedPer; k++) {
        const int leaf = s0 + k < nslots ? slot_leaf[s0 + k] : -1;
        nl[k] = lane < 27 && leaf >= 0 ? nbr[(size_t)leaf * 27 + lane] : -1;
    }
    uint32_t bits = 0u;
#pragma unroll
    for (int k = 0; k < kTouchedPer; k++) {
        bool has = false;
        if (nl[k] >= 0) {
            const int2 r = leaf_range[nl[k]];
            has = r.y > r.x;
        }
        if (__any_sync(0xFFFFFFFFu, has)) bits |= 1u << k;
    }
    if (lane == 0) s_bits[wid] = bits;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t n = 0u;
        for (int w = 0; w < kTouchedWarps; w++) {
            s_base[w] = n;
            n += __popc(s_bits[w]);
        }
        const uint32_t base = n ? atomicAdd(count, n) : 0u;
        for (int w = 0; w < kTouchedWarps; w++) s_base[w] += base;
    }
    __syncthreads();
    if (lane < kTouchedPer && ((bits >> lane) & 1u)) out[s_base[wid] + __popc(bits & ((1u << lane) - 1u))] = s0 + lane;
}

gvx_status gvx_splat_run(gvx_grid* g, int mode, int n, float radius, const float trans[3], int chan_d, int chan_v,
                         int accum)
{
    SplatArgs a;
    SplatKind kind;
    gvx_status rc = splat_prepare(g, mode, n, radius, trans, chan_d, chan_v, accum, 0, -1, 0, &a, &kind);
    if (rc) return rc;
    if (a.nslots) {
        const SplatKernel kern = splat_kernel(kind);
        const size_t smem = splat_smem(a, kern);
        GVX_CK_STATUS(gvx_allow_smem(kern.one, smem));
        int per_sm = 0;
        GVX_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern.one, kern.warps * 32, smem));
        const uint64_t units = (uint64_t)a.nslots * a.slabs;
        const uint64_t ctas_needed = (units + kern.warps - 1) / kern.warps;
        const uint64_t sms = (uint64_t)sm_count(g->device);
        if (!tri_kind(kind) && !accum && units < kFewUnits * sms * kFewBlocks * kern.warps)
            per_sm = std::min(per_sm, kFewBlocks);
        const uint32_t grid = (uint32_t)std::min<uint64_t>(ctas_needed, sms * std::max(per_sm, 1));
        GVX_CK(gvx_ensure(g->d_next, 3 * sizeof(uint32_t)));  // units taken, slots touched, units listed
        GVX_CK(cudaMemsetAsync(g->d_next.p, 0, 3 * sizeof(uint32_t), g->stream));
        a.next = g->d_next.as<uint32_t>();
        // (fewer points make no dense unit, and without dense leaves, where a build has counted them, there is
        // none: the launch that sums the listed ones takes 2 us, a warp that sums a unit of 1,500 points where it
        // met it 140, of 30,000 4 ms)
        const bool list_dense = tri_kind(kind) && a.cell_tab && n > kDenseCandidates && g->dense_leaves != 0;
        if (list_dense) {
            GVX_CK(gvx_ensure(g->dense_units, kDenseCap * sizeof(uint4)));
            a.dense_units = g->d_next.as<uint32_t>() + 2;
            a.dense_list = g->dense_units.as<uint4>();
        }
        if (accum) {
            // only the bricks that this grouping's points can reach (accumulating frames of a growing
            // scene touch a small part of it: the fusion frames, about a tenth of 129k bricks)
            GVX_CK(gvx_ensure(g->touched, (size_t)a.nslots * sizeof(uint32_t)));
            a.unit_count = g->d_next.as<uint32_t>() + 1;
            a.unit_slots = g->touched.as<uint32_t>();
            k_touched_slots<<<blocks_for(a.nslots, kTouchedWarps * kTouchedPer), kTouchedWarps * 32, 0, g->stream>>>(
                a.slot_leaf, a.nslots, a.nbr, a.leaf_range, g->touched.as<uint32_t>(), g->d_next.as<uint32_t>() + 1);
            g->launches++;
        }
        void* args[] = {&a};
        GVX_CK(cudaLaunchKernel(kern.one, dim3(grid), dim3(kern.warps * 32), args, smem, g->stream));
        g->launches++;
        if (list_dense) {
            k_tri_dense<<<sm_count(g->device) * 8, kTriWarps * 32, 0, g->stream>>>(
                nullptr, a, a.dense_units, a.dense_list, (a.slab_layers * a.P * a.P + 31) / 32);
            g->launches++;
            GVX_CK(cudaGetLastError());
        }
    }
    splat_finish(g, chan_d, chan_v, accum);
    return GVX_OK;
}

// ---------------------------------------------------------------------------
// Batched multi-grid splat: the splats of many grids (same brick shape and
// channel kinds) in ONE persistent launch, optionally captured in a CUDA graph
// and replayed while the grids' buffers stay where they are, with an
// autotuner over the slab height and the CTAs per SM (cached per GPU).

struct BatchTuning {
    int layers = 0, blocks_per_sm = 0;
    float ms = 0.f;
};

static std::mutex g_tune_mu;
static std::map<std::string, BatchTuning> g_tune_cache;

struct gvx_batch {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    std::vector<gvx_grid*> grids;
    DevBuf d_args, d_ustart;
    std::vector<SplatArgs> cap_args;   // arguments of the captured graph
    std::vector<uint32_t> cap_ustart;
    SplatKind cap_kind{};
    int cap_blocks = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int64_t exec_launches = 0;  // of one replay
    cudaEvent_t ev = nullptr;
    BatchTuning tuning;
    int64_t launches = 0;
    // gvx_batch_frame: the grids' planned builds and the splat, captured in one graph
    DevBuf f_args, f_ustart, f_cnt, f_caps;
    DevBuf dense_units;  // the units k_splat_tri_batch lists for k_tri_dense
    cudaEvent_t f_fork = nullptr;
    std::vector<cudaEvent_t> f_join;     // one per grid
    cudaGraph_t f_graph = nullptr;
    cudaGraphExec_t f_exec = nullptr;
    std::vector<uint64_t> f_key, f_failed_key;
    bool f_warm = false;                 // a planned frame ran without a graph since the plans were made
    float f_topo_radius = -1.f;          // the radius the plans were made for
    int64_t f_launches = 0;              // batch-stream launches of one replay
    std::vector<int64_t> f_grid_launches;
    int f_path = 0, f_void = 0;          // how the last frame ran, its grids built again without a plan
};

static uint64_t batch_points(const gvx_batch* b)
{
    uint64_t pts = 0;
    for (const gvx_grid* g : b->grids) pts += (uint64_t)(g->group_valid ? g->group_n : g->pts.n);
    return pts;
}

static uint64_t batch_bricks(const gvx_batch* b)
{
    uint64_t bricks = 0;
    for (const gvx_grid* g : b->grids) bricks += (uint64_t)g->atlas_used;
    return bricks;
}

static bool batch_dense(const gvx_batch* b) { return dense_cloud(batch_points(b), batch_bricks(b)); }

static void frame_drop_graph(gvx_batch* b)
{
    if (b->f_exec) cudaGraphExecDestroy(b->f_exec);
    if (b->f_graph) cudaGraphDestroy(b->f_graph);
    b->f_exec = nullptr;
    b->f_graph = nullptr;
    b->f_key.clear();
}

static void batch_drop_graph(gvx_batch* b)
{
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    b->cap_args.clear();
}

static std::string tune_key(int device, const SplatArgs& a, const SplatKind& k)
{
    cudaDeviceProp prop;
    memset(&prop, 0, sizeof(prop));
    cudaGetDeviceProperties(&prop, device);
    char buf[512];
    snprintf(buf, sizeof(buf), "%s|%d|P%d|p%d|m%d|d%d|v%d|r%d|s%d", prop.name, device, a.P, (int)a.push, k.mode,
             (int)k.has_d, (int)k.has_v, (int)k.ppr, (int)k.small);
    return buf;
}

// the listed units of a trilinear density batch (their count at `units`)
static gvx_status batch_dense_units(gvx_batch* b, const SplatKind& k, const SplatArgs& a0, const SplatArgs* dargs,
                                    const uint32_t* units)
{
    if (!tri_kind(k)) return GVX_OK;
    SplatArgs none;
    memset(&none, 0, sizeof(none));
    k_tri_dense<<<sm_count(b->device) * 8, kTriWarps * 32, 0, b->stream>>>(
        dargs, none, units, b->dense_units.as<uint4>(), (a0.slab_layers * a0.P * a0.P + 31) / 32);
    b->launches++;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

// where a batch's dense units are listed: the counter after the unit counter of `ustart`
static void batch_set_dense(gvx_batch* b, SplatArgs& a, DevBuf& ustart, size_t ngrids)
{
    a.dense_units = ustart.as<uint32_t>() + ngrids + 2;
    a.dense_list = b->dense_units.as<uint4>();
}

// the kernel of a batch's launch over `units` (a frame's: those of the last one)
static void* batch_kernel(const SplatKernel& kern, const SplatArgs& a0, uint64_t units, int blocks)
{
    return few_units(units, (uint64_t)blocks * kern.warps, a0.light) ? kern.batch_few : kern.batch;
}

// one launch of the batch kernel over args/ustart already on the device
static gvx_status batch_launch(gvx_batch* b, const SplatKind& k, const SplatArgs& a0, int ngrids, int blocks,
                               uint64_t units)
{
    const SplatKernel kern = splat_kernel(k);
    const size_t smem = splat_smem(a0, kern);
    const SplatArgs* dargs = b->d_args.as<SplatArgs>();
    uint32_t* dus = b->d_ustart.as<uint32_t>();
    GVX_CK(cudaMemsetAsync(dus + ngrids + 1, 0, 2 * sizeof(uint32_t), b->stream));  // units taken, units listed
    void* args[] = {(void*)&dargs, (void*)&dus, (void*)&ngrids};
    GVX_CK(cudaLaunchKernel(batch_kernel(kern, a0, units, blocks), dim3(blocks), dim3(kern.warps * 32), args, smem,
                            b->stream));
    b->launches++;
    return batch_dense_units(b, k, a0, dargs, dus + ngrids + 2);
}

// argument table of every grid for a slab height, and the unit ranges
static gvx_status batch_tables(gvx_batch* b, int mode, float radius, int chan_d, int chan_v, int accum, int layers,
                               std::vector<SplatArgs>& args, std::vector<uint32_t>& ustart, SplatKind& kind)
{
    args.resize(b->grids.size());
    ustart.assign(b->grids.size() + 1, 0u);
    GVX_CK(gvx_ensure(b->d_ustart, (ustart.size() + 2) * sizeof(uint32_t)));  // + units taken, units listed
    uint64_t tot = 0;
    const int dense = batch_dense(b) ? 1 : 0;
    const uint64_t bricks = std::max<uint64_t>(batch_bricks(b), 1);
    for (size_t i = 0; i < b->grids.size(); i++) {
        gvx_grid* g = b->grids[i];
        const int n = g->group_valid ? g->group_n : g->pts.n;
        const float* t = g->group_valid ? g->group_trans : nullptr;
        SplatKind k;
        gvx_status rc = splat_prepare(g, mode, n, radius, t, chan_d, chan_v, accum, layers, dense, bricks, &args[i], &k);
        if (rc) return rc;
        if (i == 0) {
            kind = k;
        } else if (!(k == kind) || args[i].P != args[0].P || args[i].slab_layers != args[0].slab_layers ||
                   args[i].push != args[0].push) {
            gvx_set_error("BatchSplat: grid %zu differs from grid 0 in brick shape, channels or radius kind", i);
            return GVX_ERR_INVALID_ARG;
        }
        if (tri_kind(kind)) {
            GVX_CK(gvx_ensure(b->dense_units, kDenseCap * sizeof(uint4)));
            batch_set_dense(b, args[i], b->d_ustart, b->grids.size());
        }
        ustart[i] = (uint32_t)tot;
        tot += (uint64_t)args[i].nslots * args[i].slabs;
        if (tot >= (1ull << 31)) {
            gvx_set_error("BatchSplat: more than 2^31 work units");
            return GVX_ERR_CAPACITY;
        }
    }
    ustart[b->grids.size()] = (uint32_t)tot;
    for (SplatArgs& a : args) a.light = light_units(batch_points(b), tot, accum);
    return GVX_OK;
}

static gvx_status batch_upload(gvx_batch* b, const std::vector<SplatArgs>& args, const std::vector<uint32_t>& ustart)
{
    GVX_CK(gvx_ensure(b->d_args, args.size() * sizeof(SplatArgs)));
    GVX_CK(cudaMemcpyAsync(b->d_args.p, args.data(), args.size() * sizeof(SplatArgs), cudaMemcpyHostToDevice,
                           b->stream));
    GVX_CK(cudaMemcpyAsync(b->d_ustart.p, ustart.data(), ustart.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                           b->stream));
    return GVX_OK;
}

static gvx_status batch_max_blocks(gvx_batch* b, const SplatKind& k, const SplatArgs& a0, int* per_sm)
{
    const SplatKernel kern = splat_kernel(k);
    const size_t smem = splat_smem(a0, kern);
    GVX_CK_STATUS(gvx_allow_smem(kern.batch, smem));
    GVX_CK_STATUS(gvx_allow_smem(kern.batch_few, smem));
    GVX_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern.batch, kern.warps * 32, smem));
    *per_sm = std::max(*per_sm, 1);
    return GVX_OK;
}

// tries the candidate (slab height, CTAs per SM) pairs on the live batch and
// keeps the fastest; each candidate: one warm-up, then the mean of two timed runs
static gvx_status batch_tune(gvx_batch* b, int mode, float radius, int chan_d, int chan_v, BatchTuning* best)
{
    // (the tuning splat does not accumulate)
    const int span = slab_shape(b->grids[0], 0, batch_dense(b), chan_d >= 0 && chan_v >= 0).span;
    const int cand_layers[3] = {(span + 1) / 2, span, (span + 2) / 3};
    cudaEvent_t e0, e1;
    GVX_CK(cudaEventCreate(&e0));
    GVX_CK(cudaEventCreate(&e1));
    best->ms = 1e30f;
    gvx_status rc = GVX_OK;
    for (int li = 0; li < 3 && rc == GVX_OK; li++) {
        std::vector<SplatArgs> args;
        std::vector<uint32_t> us;
        SplatKind k;
        rc = batch_tables(b, mode, radius, chan_d, chan_v, 0, cand_layers[li], args, us, k);
        if (rc) break;
        if (li > 0 && args[0].slab_layers == best->layers) continue;  // clamped to a height already tried
        rc = batch_upload(b, args, us);
        if (rc) break;
        int per_sm = 1;
        rc = batch_max_blocks(b, k, args[0], &per_sm);
        if (rc) break;
        const int sms = sm_count(b->device);
        for (int bp : {per_sm, std::max(1, (per_sm + 1) / 2)}) {
            const int blocks = sms * bp;
            float ms = 0.f;
            for (int it = 0; it < 3 && rc == GVX_OK; it++) {
                if (it == 1) cudaEventRecord(e0, b->stream);
                rc = batch_launch(b, k, args[0], (int)args.size(), blocks, us.back());
            }
            if (rc) break;
            cudaEventRecord(e1, b->stream);
            if (cudaEventSynchronize(e1) != cudaSuccess) {
                rc = gvx_cuda_fail(cudaGetLastError(), "autotune");
                break;
            }
            cudaEventElapsedTime(&ms, e0, e1);
            ms *= 0.5f;
            if (ms < best->ms) {
                best->ms = ms;
                best->layers = args[0].slab_layers;
                best->blocks_per_sm = bp;
            }
            if (bp == 1) break;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
}

// ---------------------------------------------------------------------------
// A whole frame of a batch (gvx_batch_frame): every grid's full RebuildTopology,
// UpdateAtlas and InsertPoints, then the batched splat.  Once every grid has a
// plan (gvx_topo_plan_make, from a staged full build), the builds are planned --
// no host wait, no allocation -- and, with GVX_BATCH_GRAPH, the grids' builds
// (forked onto their own streams) and the splat are captured in one CUDA graph,
// replayed every frame while no buffer has moved.  The splat's unit ranges come
// from the builds' slot counts on the device (k_batch_ustart).

// unit ranges of a batch whose slot counts are in device memory: ustart[k] = slabs * the sum
// of the slot counts of grids < k (each clamped to its capacity); the counters of units
// taken and units listed, ustart[ngrids + 1] and [ngrids + 2], zeroed
__global__ void k_batch_ustart(const uint32_t* const* __restrict__ counts, const uint32_t* __restrict__ caps,
                               int ngrids, int slabs, uint32_t* __restrict__ ustart)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    uint32_t t = 0;
    for (int k = 0; k < ngrids; k++) {
        ustart[k] = t;
        t += min(*counts[k], caps[k]) * (uint32_t)slabs;
    }
    ustart[ngrids] = t;
    ustart[ngrids + 1] = ustart[ngrids + 2] = 0u;
}

// the sorted attributes InsertPoints writes, then the planned build (whose octant pass writes them)
static gvx_status frame_build(gvx_grid* g, bool want_svel)
{
    const size_t m = (size_t)std::max(g->pts.n, 1);
    GVX_CK(gvx_ensure(g->spos, m * sizeof(float4)));
    if (want_svel) GVX_CK(gvx_ensure(g->svel, m * sizeof(float4)));
    unsigned int* rmax = nullptr;
    if (g->pts.radius && want_svel) {
        GVX_CK(gvx_ensure(g->d_rmax, sizeof(unsigned int)));
        GVX_CK(cudaMemsetAsync(g->d_rmax.p, 0, sizeof(unsigned int), g->stream));
        rmax = g->d_rmax.as<unsigned int>();
    }
    GvxSortedAttr A;
    A.vel = g->pts.vel;
    A.vel_off = g->pts.vel_off;
    A.vel_stride = g->pts.vel_stride;
    A.weight = g->pts.weight;
    A.radius = g->pts.radius;
    A.spos = g->spos.as<float4>();
    A.svel = want_svel ? g->svel.as<float4>() : nullptr;
    A.rmax = rmax;
    return gvx_topo_plan_enqueue(g, &A, true);
}

// every grid's planned build on its own stream, forked from and joined back into the batch
// stream (a grid whose build fails is joined all the same, so that a capture stays whole)
static gvx_status frame_builds(gvx_batch* b, const std::vector<char>& want_svel)
{
    gvx_status first = GVX_OK;
    GVX_CK(cudaEventRecord(b->f_fork, b->stream));
    for (size_t i = 0; i < b->grids.size(); i++) {
        gvx_grid* g = b->grids[i];
        const bool own = g->stream != b->stream;
        if (own) GVX_CK(cudaStreamWaitEvent(g->stream, b->f_fork, 0));
        gvx_status rc = frame_build(g, want_svel[i] != 0);
        if (rc != GVX_OK && first == GVX_OK) {
            const std::string m = gvx_last_error();
            gvx_set_error("BatchFrame: grid %zu: %s", i, m.c_str());
            first = rc;
        }
        if (own) {
            GVX_CK(cudaEventRecord(b->f_join[i], g->stream));
            GVX_CK(cudaStreamWaitEvent(b->stream, b->f_join[i], 0));
        }
    }
    return first;
}

// the splat arguments and the slot-count table of every grid to the device (before a capture,
// or after the builds of a frame without a graph)
static gvx_status frame_upload(gvx_batch* b, const SplatKind& kind, float radius, int chan_d, int chan_v,
                               int layers)
{
    const size_t ng = b->grids.size();
    std::vector<SplatArgs> args(ng);
    std::vector<const uint32_t*> cnt(ng);
    std::vector<uint32_t> caps(ng);
    for (size_t i = 0; i < ng; i++) {
        splat_fill(b->grids[i], kind, radius, chan_d, chan_v, 0, batch_dense(b), layers, &args[i]);
        // (the tables of the build the splat follows, not those of the grid's present grouping)
        args[i].leaf_dense = gvx_topo_plan_dense(b->grids[i]);
        args[i].cell_tab = args[i].leaf_dense ? b->grids[i]->cell_tab.as<int>() : nullptr;
        // (the bricks of the last frame)
        args[i].light = light_units(batch_points(b), batch_bricks(b) * (uint64_t)args[i].slabs, 0);
        if (tri_kind(kind)) batch_set_dense(b, args[i], b->f_ustart, ng);
        cnt[i] = gvx_topo_plan_slots(b->grids[i], &caps[i]);
    }
    GVX_CK(cudaMemcpyAsync(b->f_args.p, args.data(), ng * sizeof(SplatArgs), cudaMemcpyHostToDevice, b->stream));
    GVX_CK(cudaMemcpyAsync(b->f_cnt.p, cnt.data(), ng * sizeof(void*), cudaMemcpyHostToDevice, b->stream));
    GVX_CK(cudaMemcpyAsync(b->f_caps.p, caps.data(), ng * sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream));
    return GVX_OK;
}

// the unit ranges from the slot counts, then the batched splat
static gvx_status frame_splat(gvx_batch* b, const SplatKind& kind, const SplatArgs& a0, int blocks)
{
    const int ng = (int)b->grids.size();
    k_batch_ustart<<<1, 32, 0, b->stream>>>(b->f_cnt.as<const uint32_t*>(), b->f_caps.as<uint32_t>(), ng, a0.slabs,
                                            b->f_ustart.as<uint32_t>());
    const SplatKernel kern = splat_kernel(kind);
    const size_t smem = splat_smem(a0, kern);  // (the shared-memory limit set by batch_max_blocks)
    const SplatArgs* dargs = b->f_args.as<SplatArgs>();
    uint32_t* dus = b->f_ustart.as<uint32_t>();
    int n = ng;
    void* kargs[] = {(void*)&dargs, (void*)&dus, (void*)&n};
    GVX_CK(cudaLaunchKernel(batch_kernel(kern, a0, batch_bricks(b) * (uint64_t)a0.slabs, blocks), dim3(blocks),
                            dim3(kern.warps * 32), kargs, smem, b->stream));
    b->launches += 2;
    GVX_CK_STATUS(batch_dense_units(b, kind, a0, dargs, dus + ng + 2));
    // every grid's device error word (topology and splat) into its plan's record
    for (gvx_grid* g : b->grids) GVX_CK_STATUS(gvx_topo_plan_record_error(g, b->stream));
    return GVX_OK;
}

// what a captured frame depends on: buffer addresses (the allocation epoch), the plans, the
// points and attributes bound, the streams and the splat's parameters
static std::vector<uint64_t> frame_key(gvx_batch* b, float topo_radius, int mode, float radius, int chan_d,
                                       int chan_v, int layers, int blocks)
{
    auto fb = [](float f) {
        uint32_t u;
        memcpy(&u, &f, 4);
        return (uint64_t)u;
    };
    std::vector<uint64_t> k = {gvx_alloc_epoch(), fb(topo_radius), (uint64_t)mode, fb(radius), (uint64_t)chan_d,
                               (uint64_t)chan_v, (uint64_t)layers, (uint64_t)blocks, (uint64_t)(uintptr_t)b->stream,
                               (uint64_t)batch_dense(b)};
    for (gvx_grid* g : b->grids) {
        const GvxPoints& p = g->pts;
        for (uint64_t v : {gvx_topo_plan_id(g), (uint64_t)(uintptr_t)g->stream, (uint64_t)(uintptr_t)p.pos,
                           (uint64_t)p.pos_off, (uint64_t)p.pos_stride, (uint64_t)p.n, (uint64_t)(uintptr_t)p.vel,
                           (uint64_t)p.vel_off, (uint64_t)p.vel_stride, (uint64_t)(uintptr_t)p.weight,
                           (uint64_t)(uintptr_t)p.radius})
            k.push_back(v);
    }
    return k;
}

// the planned builds and the splat captured in b->f_exec (nothing allocated meanwhile)
static gvx_status frame_capture(gvx_batch* b, const std::vector<char>& want_svel, const SplatKind& kind,
                                const SplatArgs& a0, int blocks)
{
    const size_t ng = b->grids.size();
    std::vector<int64_t> l0(ng);
    for (size_t i = 0; i < ng; i++) l0[i] = b->grids[i]->launches;
    const int64_t b0 = b->launches;
    gvx_status rc;
    cudaGraph_t graph = nullptr;
    cudaError_t e;
    {
        GvxNoAllocScope no_alloc;
        GVX_CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
        rc = frame_builds(b, want_svel);
        if (rc == GVX_OK) rc = frame_splat(b, kind, a0, blocks);
        e = cudaStreamEndCapture(b->stream, &graph);
    }
    (void)cudaGetLastError();
    b->f_grid_launches.assign(ng, 0);
    for (size_t i = 0; i < ng; i++) {
        b->f_grid_launches[i] = b->grids[i]->launches - l0[i];
        b->grids[i]->launches = l0[i];  // counted when the graph runs
    }
    b->f_launches = b->launches - b0;
    b->launches = b0;
    if (rc != GVX_OK || e != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        return rc != GVX_OK ? rc : gvx_cuda_fail(e, "BatchFrame capture");
    }
    e = cudaGraphInstantiate(&b->f_exec, graph, 0);
    if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        b->f_exec = nullptr;
        return gvx_cuda_fail(e, "BatchFrame graph instantiation");
    }
    b->f_graph = graph;
    return GVX_OK;
}

// a frame without plans: the staged batch topology and the batched splat, then every grid's
// plan from its build
static gvx_status frame_unplanned(gvx_batch* b, float topo_radius, int mode, float radius, int chan_d, int chan_v,
                                  int flags)
{
    frame_drop_graph(b);
    b->f_warm = false;
    b->f_topo_radius = -1.f;
    b->f_path = 0;
    gvx_status rc = gvx_batch_topology(b, topo_radius, GVX_TOPO_FULL, 0);
    if (rc) return rc;
    rc = gvx_batch_splat(b, mode, radius, chan_d, chan_v, 0, flags & GVX_BATCH_TUNE);
    if (rc) return rc;
    GVX_CK(cudaStreamSynchronize(b->stream));
    bool all = true;
    for (gvx_grid* g : b->grids) all = gvx_topo_plan_make(g) == GVX_OK && all;
    if (all) b->f_topo_radius = topo_radius;
    return GVX_OK;
}

// one grid of a planned frame whose plan did not hold: built and splatted again without one,
// and planned anew
static gvx_status frame_rebuild(gvx_grid* g, float topo_radius, int mode, float radius, int chan_d, int chan_v)
{
    gvx_status rc = gvx_topo_stage1(g, g->pts.n, topo_radius, GVX_TOPO_FULL, 1);
    if (rc == GVX_OK) rc = gvx_topo_stage2(g);
    if (rc == GVX_OK) rc = gvx_topo_stage3(g);
    if (rc == GVX_OK) rc = gvx_topo_update_atlas(g);
    if (rc == GVX_OK) rc = gvx_splat_run(g, mode, g->pts.n, radius, nullptr, chan_d, chan_v, 0);
    if (rc == GVX_OK) GVX_CK(cudaStreamSynchronize(g->stream));
    if (rc == GVX_OK) (void)gvx_topo_plan_make(g);  // (without a plan the next frame runs unplanned)
    return rc;
}

extern "C" {

gvx_status gvx_batch_create(int device, gvx_batch** out)
{
    if (!out) {
        gvx_set_error("gvx_batch_create: null output");
        return GVX_ERR_INVALID_ARG;
    }
    *out = nullptr;
    GVX_CK(cudaSetDevice(device));
    gvx_batch* b = new gvx_batch();
    b->device = device;
    cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        if (b->stream) cudaStreamDestroy(b->stream);
        delete b;
        return gvx_cuda_fail(e, "gvx_batch_create");
    }
    b->own_stream = true;
    *out = b;
    return GVX_OK;
}

gvx_status gvx_batch_destroy(gvx_batch* b)
{
    if (!b) return GVX_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    batch_drop_graph(b);
    frame_drop_graph(b);
    gvx_free(b->d_args);
    gvx_free(b->d_ustart);
    gvx_free(b->dense_units);
    for (DevBuf* d : {&b->f_args, &b->f_ustart, &b->f_cnt, &b->f_caps}) gvx_free(*d);
    if (b->f_fork) cudaEventDestroy(b->f_fork);
    for (cudaEvent_t e : b->f_join) cudaEventDestroy(e);
    if (b->ev) cudaEventDestroy(b->ev);
    if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return GVX_OK;
}

gvx_status gvx_batch_set_stream(gvx_batch* b, void* stream)
{
    if (!b) {
        gvx_set_error("null batch handle");
        return GVX_ERR_INVALID_ARG;
    }
    GVX_CK(cudaSetDevice(b->device));
    GVX_CK(cudaStreamSynchronize(b->stream));
    if (b->own_stream) cudaStreamDestroy(b->stream);
    b->stream = (cudaStream_t)stream;
    b->own_stream = false;
    batch_drop_graph(b);
    frame_drop_graph(b);
    return GVX_OK;
}

gvx_status gvx_batch_set_grids(gvx_batch* b, gvx_grid* const* grids, int count)
{
    if (!b || (count > 0 && !grids) || count < 0 || count > kBatchMaxGrids) {
        gvx_set_error("BatchSetGrids: need 0..%d grids", kBatchMaxGrids);
        return GVX_ERR_INVALID_ARG;
    }
    for (int i = 0; i < count; i++) {
        if (!grids[i] || grids[i]->device != b->device) {
            gvx_set_error("BatchSetGrids: grid %d is null or on another device", i);
            return GVX_ERR_INVALID_ARG;
        }
    }
    b->grids.assign(grids, grids + count);
    batch_drop_graph(b);
    frame_drop_graph(b);
    b->f_warm = false;
    b->f_topo_radius = -1.f;
    return GVX_OK;
}

// Topology of every grid from a pool of host threads: each grid is driven by one
// thread at a time (a grid handle is not shared between threads), and builds of
// grids on different streams overlap on the GPU.  A build is mostly small kernels
// and two host readbacks, so one thread alone leaves the GPU idle most of the time.
gvx_status gvx_batch_topology(gvx_batch* b, float radius, int mode, int threads)
{
    if (!b) {
        gvx_set_error("null batch handle");
        return GVX_ERR_INVALID_ARG;
    }
    if (mode < GVX_TOPO_AUTO || mode > GVX_TOPO_ACCUMULATE) {
        gvx_set_error("BatchTopology: mode %d", mode);
        return GVX_ERR_INVALID_ARG;
    }
    const size_t n = b->grids.size();
    if (n == 0) return GVX_OK;
    if (threads <= 0) {
        // staged, from this thread: every grid's GetBoundingBox, then (one wait per grid, by
        // then mostly passed) every grid's build up to its node counts, then every grid's
        // pools, UpdateAtlas and InsertPoints; the grids' streams overlap on the GPU
        GVX_CK(cudaSetDevice(b->device));
        const char* what[3] = {"GetBoundingBox", "RebuildTopology", "pools/UpdateAtlas/InsertPoints"};
        for (int stage = 0; stage < 3; stage++) {
            for (size_t i = 0; i < n; i++) {
                gvx_grid* g = b->grids[i];
                gvx_status r = GVX_OK;
                if (stage == 0) {
                    r = gvx_wait_positions(g);
                    if (r == GVX_OK) r = gvx_topo_stage1(g, g->pts.n, radius, mode, 1);
                } else if (stage == 1) {
                    r = gvx_topo_stage2(g);
                } else {
                    r = gvx_topo_stage3(g);
                    if (r == GVX_OK) r = gvx_wait_attributes(g);
                    if (r == GVX_OK) r = gvx_topo_update_atlas(g);
                    if (r == GVX_OK) r = gvx_prepare_points(g, g->pts.n, nullptr, false);
                }
                if (r != GVX_OK) {
                    const std::string m = gvx_last_error();
                    gvx_set_error("BatchTopology: grid %zu (%s): %s", i, what[stage], m.c_str());
                    return r;
                }
            }
        }
        return GVX_OK;
    }
    const size_t nt = std::min<size_t>(n, (size_t)threads);
    std::atomic<size_t> next{0};
    std::vector<gvx_status> st(n, GVX_OK);
    std::vector<std::string> msg(n);
    const int device = b->device;
    auto work = [&]() {
        if (cudaSetDevice(device) != cudaSuccess) return;
        for (;;) {
            const size_t i = next.fetch_add(1);
            if (i >= n) break;
            gvx_grid* g = b->grids[i];
            gvx_status r = gvx_rebuild_topology(g, g->pts.n, radius, nullptr, mode, 1);
            if (r == GVX_OK) r = gvx_update_atlas(g);
            if (r == GVX_OK) r = gvx_insert_points(g, g->pts.n, nullptr, nullptr);
            st[i] = r;
            if (r != GVX_OK) msg[i] = gvx_last_error();
        }
    };
    std::vector<std::thread> pool;
    for (size_t t = 1; t < nt; t++) pool.emplace_back(work);
    work();
    for (std::thread& t : pool) t.join();
    for (size_t i = 0; i < n; i++)
        if (st[i] != GVX_OK) {
            gvx_set_error("BatchTopology: grid %zu: %s", i, msg[i].c_str());
            return st[i];
        }
    return GVX_OK;
}

gvx_status gvx_batch_splat(gvx_batch* b, int mode, float radius, int chan_density, int chan_vel, int accum, int flags)
{
    if (!b) {
        gvx_set_error("null batch handle");
        return GVX_ERR_INVALID_ARG;
    }
    GVX_CK(cudaSetDevice(b->device));
    if (b->grids.empty()) return GVX_OK;
    // the grids' own streams first (their InsertPoints work), then the batch
    for (gvx_grid* g : b->grids) {
        if (g->stream == b->stream) continue;
        GVX_CK(cudaEventRecord(b->ev, g->stream));
        GVX_CK(cudaStreamWaitEvent(b->stream, b->ev, 0));
    }
    int layers = 0, bps = 0;
    std::vector<SplatArgs> args;
    std::vector<uint32_t> us;
    SplatKind kind;
    gvx_status rc = batch_tables(b, mode, radius, chan_density, chan_vel, accum, 0, args, us, kind);
    if (rc) return rc;
    const std::string key = tune_key(b->device, args[0], kind);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end()) b->tuning = it->second;
    }
    if ((flags & GVX_BATCH_TUNE) && !accum && b->tuning.layers == 0) {
        // the grids' streams must not run during the timing
        for (gvx_grid* g : b->grids) GVX_CK(cudaStreamSynchronize(g->stream));
        batch_drop_graph(b);
        rc = batch_tune(b, mode, radius, chan_density, chan_vel, &b->tuning);
        if (rc) return rc;
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune_cache[key] = b->tuning;
    }
    layers = b->tuning.layers;
    bps = b->tuning.blocks_per_sm;
    if (layers > 0 && layers != args[0].slab_layers) {
        rc = batch_tables(b, mode, radius, chan_density, chan_vel, accum, layers, args, us, kind);
        if (rc) return rc;
    }
    int per_sm = 1;
    rc = batch_max_blocks(b, kind, args[0], &per_sm);
    if (rc) return rc;
    if (bps <= 0 || bps > per_sm) bps = per_sm;
    const uint64_t warps = (uint64_t)splat_kernel(kind).warps;
    const uint64_t ctas_needed = ((uint64_t)us.back() + warps - 1) / warps;
    const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(ctas_needed, (uint64_t)sm_count(b->device) * bps));
    const bool same = b->exec && b->cap_args.size() == args.size() && b->cap_kind == kind &&
                      b->cap_blocks == blocks &&
                      memcmp(b->cap_args.data(), args.data(), args.size() * sizeof(SplatArgs)) == 0 &&
                      b->cap_ustart == us;
    if (us.back() > 0) {
        if (flags & GVX_BATCH_GRAPH) {
            if (!same) {
                batch_drop_graph(b);
                rc = batch_upload(b, args, us);
                if (rc) return rc;
                const int64_t b0 = b->launches;
                GVX_CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
                rc = batch_launch(b, kind, args[0], (int)args.size(), blocks, us.back());
                b->exec_launches = b->launches - b0;
                b->launches = b0;  // counted when the graph runs
                cudaGraph_t graph = nullptr;
                cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
                if (rc) {
                    if (graph) cudaGraphDestroy(graph);
                    return rc;
                }
                if (e != cudaSuccess) return gvx_cuda_fail(e, "cudaStreamEndCapture");
                b->graph = graph;
                e = cudaGraphInstantiate(&b->exec, b->graph, 0);
                if (e != cudaSuccess) {
                    batch_drop_graph(b);
                    return gvx_cuda_fail(e, "cudaGraphInstantiate");
                }
                b->cap_args = args;
                b->cap_ustart = us;
                b->cap_kind = kind;
                b->cap_blocks = blocks;
            }
            GVX_CK(cudaGraphLaunch(b->exec, b->stream));
            b->launches += b->exec_launches;
        } else {
            rc = batch_upload(b, args, us);
            if (rc) return rc;
            rc = batch_launch(b, kind, args[0], (int)args.size(), blocks, us.back());
            if (rc) return rc;
        }
    }
    // the grids' streams see the splat before their next work
    GVX_CK(cudaEventRecord(b->ev, b->stream));
    for (gvx_grid* g : b->grids) {
        if (g->stream != b->stream) GVX_CK(cudaStreamWaitEvent(g->stream, b->ev, 0));
        g->launches++;
        splat_finish(g, chan_density, chan_vel, accum);
    }
    return GVX_OK;
}

gvx_status gvx_batch_get_tuning(gvx_batch* b, int* slab_layers, int* blocks_per_sm, float* ms)
{
    if (!b) {
        gvx_set_error("null batch handle");
        return GVX_ERR_INVALID_ARG;
    }
    if (slab_layers) *slab_layers = b->tuning.layers;
    if (blocks_per_sm) *blocks_per_sm = b->tuning.blocks_per_sm;
    if (ms) *ms = b->tuning.ms;
    return GVX_OK;
}

gvx_status gvx_batch_kernel_launches(gvx_batch* b, int64_t* out)
{
    if (!b || !out) {
        gvx_set_error("null batch handle");
        return GVX_ERR_INVALID_ARG;
    }
    *out = b->launches;
    return GVX_OK;
}


gvx_status gvx_batch_frame(gvx_batch* b, float topo_radius, int mode, float radius, int chan_density, int chan_vel,
                           int flags)
{
    if (!b) {
        gvx_set_error("null batch handle");
        return GVX_ERR_INVALID_ARG;
    }
    if (!(topo_radius >= 0.f)) {
        gvx_set_error("BatchFrame: topology radius must be >= 0");
        return GVX_ERR_INVALID_ARG;
    }
    GVX_CK(cudaSetDevice(b->device));
    const size_t ng = b->grids.size();
    b->f_void = 0;
    if (ng == 0) return GVX_OK;
    bool planned = b->f_topo_radius == topo_radius;
    for (gvx_grid* g : b->grids) planned = planned && gvx_topo_plan_ready(g);
    if (!planned) return frame_unplanned(b, topo_radius, mode, radius, chan_density, chan_vel, flags);

    // the splat's kind and slab height, the same for every grid
    SplatKind kind{};
    int layers = 0;
    std::vector<char> want_svel(ng);
    for (size_t i = 0; i < ng; i++) {
        gvx_grid* g = b->grids[i];
        int l = b->tuning.layers;
        SplatKind k;
        gvx_status rc = splat_check(g, mode, radius, chan_density, chan_vel, 0, batch_dense(b), batch_bricks(b), &l, &k);
        if (rc) return rc;
        if (i == 0) {
            kind = k;
            layers = l;
        } else if (!(k == kind) || g->P != b->grids[0]->P || l != layers) {
            gvx_set_error("BatchFrame: grid %zu differs from grid 0 in brick shape, channels or radius kind", i);
            return GVX_ERR_INVALID_ARG;
        }
        want_svel[i] = k.has_v || k.ppr || g->pts.vel || g->pts.radius;
    }
    SplatArgs a0;
    memset(&a0, 0, sizeof(a0));
    const SlabShape sh0 = slab_shape(b->grids[0], 0, batch_dense(b), kind.has_d && kind.has_v);
    a0.P = b->grids[0]->P;
    a0.push = sh0.push;
    a0.tile_rows = sh0.rows;
    a0.slab_layers = layers;
    a0.slabs = (sh0.span + layers - 1) / layers;
    a0.light = light_units(batch_points(b), batch_bricks(b) * (uint64_t)a0.slabs, 0);
    uint64_t units = 0;
    for (gvx_grid* g : b->grids) {
        uint32_t cap = 0;
        (void)gvx_topo_plan_slots(g, &cap);
        units += (uint64_t)cap * a0.slabs;
    }
    if (units >= (1ull << 31)) {
        gvx_set_error("BatchFrame: more than 2^31 work units");
        return GVX_ERR_CAPACITY;
    }
    int per_sm = 1;
    gvx_status rc = batch_max_blocks(b, kind, a0, &per_sm);
    if (rc) return rc;
    int bps = b->tuning.blocks_per_sm;
    if (bps <= 0 || bps > per_sm) bps = per_sm;
    const int blocks = sm_count(b->device) * bps;

    // the grids' queued work (point uploads included) before the frame
    if (!b->f_fork) GVX_CK(cudaEventCreateWithFlags(&b->f_fork, cudaEventDisableTiming));
    while (b->f_join.size() < ng) {
        cudaEvent_t e;
        GVX_CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        b->f_join.push_back(e);
    }
    for (size_t i = 0; i < ng; i++) {
        gvx_grid* g = b->grids[i];
        rc = gvx_wait_positions(g);
        if (rc == GVX_OK) rc = gvx_wait_attributes(g);
        if (rc) return rc;
        if (g->stream != b->stream) {
            GVX_CK(cudaEventRecord(b->f_join[i], g->stream));
            GVX_CK(cudaStreamWaitEvent(b->stream, b->f_join[i], 0));
        }
    }
    GVX_CK(gvx_ensure(b->f_args, ng * sizeof(SplatArgs)));
    GVX_CK(gvx_ensure(b->f_ustart, (ng + 3) * sizeof(uint32_t)));
    if (tri_kind(kind)) GVX_CK(gvx_ensure(b->dense_units, kDenseCap * sizeof(uint4)));
    GVX_CK(gvx_ensure(b->f_cnt, ng * sizeof(void*)));
    GVX_CK(gvx_ensure(b->f_caps, ng * sizeof(uint32_t)));

    bool use_graph = (flags & GVX_BATCH_GRAPH) && b->f_warm;
    if (use_graph) {
        const std::vector<uint64_t> key = frame_key(b, topo_radius, mode, radius, chan_density, chan_vel, layers, blocks);
        if (!(b->f_exec && key == b->f_key)) {
            frame_drop_graph(b);
            use_graph = key != b->f_failed_key;
            if (use_graph) {
                rc = frame_upload(b, kind, radius, chan_density, chan_vel, layers);
                if (rc) return rc;
                if (frame_capture(b, want_svel, kind, a0, blocks) == GVX_OK) {
                    b->f_key = key;
                } else {
                    b->f_failed_key = key;  // the frame runs without a graph; no new attempt with this key
                    use_graph = false;
                }
            }
        }
    }
    if (use_graph) {
        GVX_CK(cudaGraphLaunch(b->f_exec, b->stream));
        b->launches += b->f_launches;
        for (size_t i = 0; i < ng; i++) {
            b->grids[i]->launches += b->f_grid_launches[i];
            gvx_topo_plan_replayed(b->grids[i]);
        }
        b->f_path = 2;
    } else {
        rc = frame_builds(b, want_svel);
        if (rc == GVX_OK) rc = frame_upload(b, kind, radius, chan_density, chan_vel, layers);
        if (rc == GVX_OK) rc = frame_splat(b, kind, a0, blocks);
        if (rc) {
            cudaStreamSynchronize(b->stream);
            return rc;
        }
        b->f_path = 1;
    }
    GVX_CK(cudaStreamSynchronize(b->stream));

    // which plans held: the grids whose did not are built again without one
    gvx_status first = GVX_OK;
    std::vector<size_t> redo;
    for (size_t i = 0; i < ng; i++) {
        gvx_grid* g = b->grids[i];
        bool held = false;
        rc = gvx_topo_plan_finish(g, &held, true);
        if (rc != GVX_OK) {
            if (first == GVX_OK) {
                const std::string m = gvx_last_error();
                gvx_set_error("BatchFrame: grid %zu: %s", i, m.c_str());
                first = rc;
            }
            continue;
        }
        if (!held) {
            redo.push_back(i);
            continue;
        }
        g->perm_valid = true;  // as gvx_prepare_points leaves it
        g->perm_has_svel = want_svel[i] != 0;
        g->perm_vel = g->pts.vel;
        g->perm_w = g->pts.weight;
        g->perm_r = g->pts.radius;
        splat_finish(g, chan_density, chan_vel, 0);
    }
    if (first != GVX_OK) {
        frame_drop_graph(b);
        b->f_warm = false;
        b->f_topo_radius = -1.f;
        return first;
    }
    if (b->f_path == 1) b->f_warm = true;
    if (!redo.empty()) {
        frame_drop_graph(b);
        b->f_warm = false;
        b->f_void = (int)redo.size();
        for (size_t i : redo) {
            rc = frame_rebuild(b->grids[i], topo_radius, mode, radius, chan_density, chan_vel);
            if (rc) {
                const std::string m = gvx_last_error();
                gvx_set_error("BatchFrame: grid %zu: %s", i, m.c_str());
                b->f_topo_radius = -1.f;
                return rc;
            }
        }
    }
    return GVX_OK;
}

gvx_status gvx_batch_frame_path(gvx_batch* b, int* path, int* rebuilt)
{
    if (!b) {
        gvx_set_error("null batch handle");
        return GVX_ERR_INVALID_ARG;
    }
    if (path) *path = b->f_path;
    if (rebuilt) *rebuilt = b->f_void;
    return GVX_OK;
}

}  // extern "C"

gvx_status gvx_scatter_ref(gvx_grid* g, int n, float radius, const float trans[3], int expand, int avg_color)
{
    gvx_status rc = check_splat_state(g, "ScatterDensity");
    if (rc) return rc;
    if (!g->ch[0].used || g->ch[0].type != GVX_T_FLOAT) {
        gvx_set_error("ScatterDensity: channel 0 must be a T_FLOAT channel");
        return GVX_ERR_INVALID_ARG;
    }
    if (!(radius != 0.f)) {
        gvx_set_error("ScatterDensity: radius must be nonzero");
        return GVX_ERR_INVALID_ARG;
    }
    // the colour half (VG.cpp:5638-5655): with point colours, avgColor averages into channel 1; without,
    // each voxel takes a point's colour in channel 3, unless an avgColor call ever ran on this grid
    // (the reference's colour buffer then exists and silently takes the sums)
    int clr_mode = 0;
    if (g->pts.clr) {
        if (avg_color) clr_mode = 1;
        else if (!g->colavg_seen) clr_mode = 2;
    }
    const int clr_chan = clr_mode == 1 ? 1 : 3;
    if (clr_mode && (!g->ch[clr_chan].used || g->ch[clr_chan].elem_bytes != 4)) {
        gvx_set_error("ScatterDensity: point colours go to channel %d, which must be a 4-byte channel", clr_chan);
        return GVX_ERR_INVALID_ARG;
    }
    rc = gvx_prepare_points(g, n, trans, false);
    if (rc) return rc;
    if (clr_mode == 1) g->colavg_seen = true;
    const int P = g->P, P3 = P * P * P, b3 = g->brick * g->brick * g->brick;
    const size_t smem = (((size_t)P3 * 4 + 15) & ~(size_t)15) + (clr_mode == 1 ? 16 : clr_mode == 2 ? 4 : 0) * (size_t)b3;
    ScatterArgs a;
    a.brick = g->brick;
    a.P = P;
    a.apron = g->apron;
    a.nslots = (uint32_t)g->atlas_used;
    a.slot_leaf = g->slot_leaf.as<int>();
    a.nodes0 = g->nodes[0].as<GvxNode>();
    a.leaf_range = g->leaf_range.as<int2>();
    a.spos = g->spos.as<float4>();
    a.radius = radius;
    a.expand = expand;
    a.den = g->ch[0].data.as<float>();
    a.err = g->d_err.as<uint32_t>();
    a.clr_mode = clr_mode;
    a.perm = g->vals[g->sorted_buf].as<uint32_t>();
    a.clr = g->pts.clr;
    a.clr_off = g->pts.clr_off;
    a.clr_stride = g->pts.clr_stride;
    a.clr_out = clr_mode ? g->ch[clr_chan].data.as<uint32_t>() : nullptr;
    apron_invalidate(g->ch[0]);
    if (clr_mode) apron_invalidate(g->ch[clr_chan]);
    if (a.nslots == 0) return GVX_OK;
    // (cells are in order in leaves of 128 points and more of bricks of 8)
    const bool few = g->n_sorted < 192ull * a.nslots;
    const void* single = few ? (const void*)k_scatter_ref<false> : (const void*)k_scatter_ref<true>;
    int per_sm = 0;
    GVX_CK_STATUS(gvx_allow_smem(single, smem));
    GVX_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, single, kSplatThreads, smem));
    const uint32_t wave = (uint32_t)(sm_count(g->device) * std::max(per_sm, 1));
    // The blocks' kernel alone where there is a block for every brick (8k points in 330 bricks 7 us, by the two 15),
    // or six turns of the blocks do bricks of 16 points (300k points in 2.2k bricks 12 us, by the two 19; of 4.5,
    // 10k points, 10 and 8), or all are its own on average.  The warps' kernel alone for so few points that a warp
    // has them all in a few turns: nothing is gained by the other's launch (2 us).
    const uint64_t each = a.nslots <= 6u * wave ? 16 : kScatterBlock;
    const bool warps = g->brick <= 8 && a.nslots > wave && g->n_sorted < each * a.nslots;
    a.block_points = !warps ? 1 : g->n_sorted < 1024u ? 1024 : kScatterBlock;
    if (warps) {
        const size_t tab = (size_t)kScatterWarps * (clr_mode == 1 ? 16 : clr_mode == 2 ? 4 : 0) * b3;
        GVX_CK_STATUS(gvx_allow_smem((const void*)k_scatter_points, tab));
        int blocks = 0;
        GVX_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_scatter_points, kScatterWarps * 32, tab));
        const uint32_t all = (a.nslots + kScatterWarps - 1) / kScatterWarps;
        k_scatter_points<<<std::min<uint32_t>(all, (uint32_t)(sm_count(g->device) * std::max(blocks, 1))),
                           kScatterWarps * 32, tab, g->stream>>>(a);
        g->launches++;
        if (a.block_points > (int64_t)g->n_sorted) {  // (no brick can hold so many)
            GVX_CK(cudaGetLastError());
            return GVX_OK;
        }
    }
    const void* kern = warps ? (const void*)k_scatter_ref<true> : single;
    GVX_CK_STATUS(gvx_allow_smem(kern, smem));
    GVX_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSplatThreads, smem));
    const uint32_t grid = std::min<uint32_t>(a.nslots, (uint32_t)(sm_count(g->device) * std::max(per_sm, 1)));
    void* args[] = {&a};
    GVX_CK(cudaLaunchKernel(kern, dim3(grid), dim3(kSplatThreads), args, smem, g->stream));
    g->launches++;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}
