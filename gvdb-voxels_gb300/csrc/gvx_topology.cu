// gvx_topology.cu -- dynamic brick topology from points, on the device.
//
// Reference path (paths relative to the reference project):
//   VolumeGVDB::RebuildTopology          gvdb_volume_gvdb.cpp:1181-1218
//   GetBoundingBox / DetermineDepth      gvdb_volume_gvdb.cpp:5404-5467, 821-837
//   ActivateBricksGPU                    gvdb_volume_gvdb.cpp:1229-1413
//   ActivateExtraBricksGPU               gvdb_volume_gvdb.cpp:931-1016
//   gvdbCalcBrickId / CalcExtraBrickId   cuda_gvdb_particles.cuh:352-382, 467-512
//   gvdbLinkBricks                       cuda_gvdb_nodes.cuh:470-505
//   UpdateAtlas                          gvdb_volume_gvdb.cpp:2630-2704
//
// The reference computes one 64-bit key per point per level, sorts all of
// them, copies the unique keys to the host, allocates nodes in a host loop,
// links them with a root descent per node and repeats the cycle for the
// dilated ("extra") bricks.  Here the node set of every level is derived on the
// device from ONE sort of 32-bit compact level-0 keys:
//   D0 = leaves holding points, X0 = leaves of the dilation boxes not in D0,
//   level l nodes = parents of (D0 u X0), split the same way,
// each set held as a bitmap with per-word prefix popcounts, so pool order
// (sorted direct nodes, then sorted extra nodes: the order of the reference's
// two passes), parent indices and child-list slots are all O(1) rank lookups.
// The host reads back the bounding box and the per-level counts, each with the
// error word, in one copy of 384 bytes (a planned build: once, at its end).
#include <limits.h>
#include <math.h>
#include <string.h>

#include <atomic>

#include "gvx_grid.cuh"

namespace {

__device__ __forceinline__ uint32_t f2ord(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
inline float ord2f(uint32_t u)
{
    const uint32_t b = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
    float f;
    memcpy(&f, &b, 4);
    return f;
}

__device__ __forceinline__ void load_pos(const char* base, int off, int stride, uint32_t i, float* w)
{
    const float* p = (const float*)(base + (size_t)i * (size_t)stride + off);
    w[0] = p[0];
    w[1] = p[1];
    w[2] = p[2];
}

inline int ceil_log2(int64_t v)
{
    int b = 0;
    while ((int64_t(1) << b) < v) b++;
    return b;
}

}  // namespace

// the threads' bounds (order-preserving bits) into out: warp, then block, then one atomic per block and bound
// (6 addresses take every atomic)
__device__ __forceinline__ void bbox_reduce(uint32_t mn[3], uint32_t mx[3], bool nan, uint32_t* out, uint32_t* err)
{
#pragma unroll
    for (int a = 0; a < 3; a++) {
        for (int s = 16; s > 0; s >>= 1) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xFFFFFFFFu, mn[a], s));
            mx[a] = max(mx[a], __shfl_xor_sync(0xFFFFFFFFu, mx[a], s));
        }
    }
    __shared__ uint32_t s_b[32][6];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0)
        for (int a = 0; a < 3; a++) {
            s_b[wid][a] = mn[a];
            s_b[wid][3 + a] = mx[a];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t v = s_b[0][threadIdx.x];
        for (int w = 1; w < nw; w++) v = threadIdx.x < 3 ? min(v, s_b[w][threadIdx.x]) : max(v, s_b[w][threadIdx.x]);
        if (threadIdx.x < 3)
            atomicMin(&out[threadIdx.x], v);
        else
            atomicMax(&out[threadIdx.x], v);
    }
    if (nan) atomicOr(err, GVX_DERR_BADPOINT);
}

// ---------------------------------------------------------------------------
// bounding box of pos + orig over ALL points (GetBoundingBox includes points
// that the key kernel later drops)
__global__ void k_bbox(const char* pos, int off, int stride, uint32_t n, float ox, float oy, float oz,
                       uint32_t* out, uint32_t* err)
{
    uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
    bool nan = false;
    const uint32_t nt = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
    const char* base = pos + off;
    if (stride == 12 && ((uintptr_t)base & 15u) == 0 && nt % 3u == 0) {
        // packed float3, 16-byte aligned: four points in three float4 loads.  Float4 j holds
        // floats 4j .. 4j+3, whose axes are (j + k) mod 3; the thread count is a multiple of 3,
        // so j mod 3 = t mod 3 on every iteration and component k keeps one axis throughout.
        const float4* v = (const float4*)base;
        const uint64_t nflt = 3ull * n, nv = nflt / 4;
        const uint32_t ph = t % 3u;
        const float oc[3] = {ph == 0 ? ox : (ph == 1 ? oy : oz), ph == 0 ? oy : (ph == 1 ? oz : ox),
                             ph == 0 ? oz : (ph == 1 ? ox : oy)};
        uint32_t cmn[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, cmx[4] = {0u, 0u, 0u, 0u};
        for (uint64_t j = t; j < nv; j += nt) {
            const float4 q = v[j];
            const float w[4] = {q.x + oc[0], q.y + oc[1], q.z + oc[2], q.w + oc[0]};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (w[k] != w[k]) nan = true;
                const uint32_t o = f2ord(w[k]);
                cmn[k] = min(cmn[k], o);
                cmx[k] = max(cmx[k], o);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t a = (ph + (uint32_t)k) % 3u;
            mn[a] = min(mn[a], cmn[k]);
            mx[a] = max(mx[a], cmx[k]);
        }
        if (t == 0) {  // the floats after the last whole float4
            const float o3[3] = {ox, oy, oz};
            for (uint64_t f = nv * 4; f < nflt; f++) {
                const uint32_t a = (uint32_t)(f % 3u);
                const float w = ((const float*)base)[f] + o3[a];
                if (w != w) nan = true;
                mn[a] = min(mn[a], f2ord(w));
                mx[a] = max(mx[a], f2ord(w));
            }
        }
    } else {
        for (uint32_t i = t; i < n; i += nt) {
            float w[3];
            load_pos(pos, off, stride, i, w);
            w[0] += ox;
            w[1] += oy;
            w[2] += oz;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                if (w[a] != w[a]) nan = true;
                const uint32_t o = f2ord(w[a]);
                mn[a] = min(mn[a], o);
                mx[a] = max(mx[a], o);
            }
        }
    }
    bbox_reduce(mn, mx, nan, out, err);
}

// compact level-0 key of every point (invalid points -> invalid_key, sorted
// last), identity values, and the digit histograms of the sort.  kshift 3: the
// key is (leaf key << 3) | octant, octant = 4 hx + 2 hy + hz the half of the
// brick (2^lb voxels) that the point's voxel lies in on every axis, so the
// stable sort leaves every leaf's points in (octant, index) order; invalid_key
// is the shifted one then.  BBOX: the bounding box too, as k_bbox (a planned build does not wait for it: one
// launch and one pass over the positions less)
template <bool BBOX>
__global__ void k_keys(const char* pos, int off, int stride, uint32_t n, float ox, float oy, float oz,
                       KeySpace ks, float inv_b, int kshift, int lb, int passes, uint32_t invalid_key,
                       uint32_t* keys, uint32_t* vals, uint32_t* hist, uint32_t* bbox, uint32_t* err)
{
    uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
    bool nan = false;
    __shared__ uint32_t sh[4 * 256];
    for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) sh[i] = 0u;
    __syncthreads();
    bool degen = false;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float w[3];
        load_pos(pos, off, stride, i, w);
        w[0] += ox;
        w[1] += oy;
        w[2] += oz;
        if (BBOX) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                if (w[a] != w[a]) nan = true;
                mn[a] = min(mn[a], f2ord(w[a]));
                mx[a] = max(mx[a], f2ord(w[a]));
            }
        }
        uint32_t key = invalid_key;
        if (w[0] >= 0.f && w[1] >= 0.f && w[2] >= 0.f) {
            int c[3];
            bool in = true;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                c[a] = (int)(w[a] * inv_b) - ks.lo[a];  // floor(w / b), exact for a power-of-two b
                if (c[a] < 0 || c[a] >= (1 << ks.bits[a])) in = false;
            }
            if (in) {
                key = ks_pack(ks, c[0], c[1], c[2], 0) << kshift;
                if (kshift) {
                    // voxel x >= the brick's corner + half  <=>  bit lb-1 of x (x >= 0, bricks aligned)
                    int oct = 7;
                    if (lb > 0)
                        oct = ((((int)w[0]) >> (lb - 1)) & 1) << 2 | ((((int)w[1]) >> (lb - 1)) & 1) << 1 |
                              ((((int)w[2]) >> (lb - 1)) & 1);
                    key |= (uint32_t)oct;
                }
            } else {
                degen = true;
            }
        }
        keys[i] = key;
        vals[i] = i;
        gvx_sort_count_key(sh, key, passes);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += blockDim.x)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
    if (degen) atomicOr(err, GVX_DERR_DEGENERATE);
    if (BBOX) bbox_reduce(mn, mx, nan, bbox, err);
}

// The cells of a build, from the sorted keys (>> kshift: leaf keys): the first point of every run of equal
// valid ones sets its bit in d0bits.  BOX: also the leaves touched by the points' boxes
// [int(p)-r, int(p)+2r] (cuda_gvdb_particles.cuh:481-482; hi_mul = 2 for the full rebuild's box, 1 for the
// incremental box [int(p)-r, int(p)+r], PT.cuh:433-434) in x0bits, the points' own leaves among them (the
// ranks leave those out).  A point's leaves are 27 bits (dz+1)*9 + (dy+1)*3 + (dx+1); a warp's points of one
// leaf join theirs, and nine lanes a leaf set them, a lane the three along z, which are neighbours in a word;
// leaves of one word, side by side in the sorted order, are joined first where a warp has two of them and more
// a word: a word's nine rows cost 110 instructions, a leaf's a third of 40 and nine atomics of L2 (4M points
// in 777k leaves: 130 us leaf by leaf, 100 so; 300k points of a depth frame 7.4 and 8.5, always by words 13).
// lim: per axis, the first key-space coordinate past the root (a key space rounded up to powers of two may
// reach past it).
// The marks used to wait for the ranks of d0bits, which numbered a mask per leaf: three launches more, and
// two passes over the ranks (6k points a frame 96 us, 81 so; 6M points: 111 us of kernels, 90 so, although
// whole frames of them in flight went from 1.65 to 1.71 ms: the next build overlaps the last gather less).
template <bool BOX>
__global__ void __launch_bounds__(256)
    k_mark_cells(const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ svals, uint32_t n, int kshift,
                 uint32_t invalid_key, const char* pos, int off, int stride, float ox, float oy, float oz,
                 float radius, float hi_mul, int lb, KeySpace ks, int3 lim, uint32_t* d0bits, uint32_t* x0bits,
                 uint32_t* err)
{
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const uint32_t key = i < n ? skeys[i] >> kshift : invalid_key;
    const bool valid = key < invalid_key;
    uint32_t prev = __shfl_up_sync(kFull, key, 1);
    if (lane == 0) prev = valid && i > 0 ? skeys[i - 1] >> kshift : invalid_key;
    if (valid && prev != key) atomicOr(&d0bits[key >> 5], 1u << (key & 31));
    if (!BOX) return;
    uint32_t m = 0u;
    if (valid) {
        float w[3];
        load_pos(pos, off, stride, svals[i], w);
        w[0] += ox;
        w[1] += oy;
        w[2] += oz;
        uint32_t ax[3];  // per axis, bits 0 to 2: the leaf below, the own one, the one above
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int ip = (int)w[a];
            const int bmin = (int)((float)ip - radius);
            const int bmax = (int)((float)ip + hi_mul * radius);
            // C truncation of x / brick, as bmin/rres*rres
            auto cell = [&](int x) { return (x + ((x >> 31) & ((1 << lb) - 1))) >> lb; };
            const int cl = cell(ip);
            const int lo = max(cell(bmin) - cl, -1), hi = min(cell(bmax) - cl, 1);
            ax[a] = lo > hi ? 0u : (7u << (lo + 1)) & (7u >> (1 - hi));
        }
        const uint32_t y = (ax[1] & 1u) | (ax[1] & 2u) << 2 | (ax[1] & 4u) << 4;
        const uint32_t zz = (ax[2] & 1u) | (ax[2] & 2u) << 8 | (ax[2] & 4u) << 16;
        m = ax[0] * y * zz;  // (copies side by side: no carries)
    }
    const bool first = valid && (lane == 0 || prev != key);
    uint32_t runs = __ballot_sync(kFull, first);
    // equal keys are side by side: a run's first lane gets the masks of the lanes after it
    const uint32_t after = runs & ~((2u << lane) - 1u);
    const int end = after ? __ffs(after) - 1 : 32;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t m2 = __shfl_down_sync(kFull, m, o);
        if (lane + o < end) m |= m2;
    }
    bool degen = false;  // a leaf outside the root: the reference descends there
    m &= ~(1u << 13);    // (the point's own leaf)
    int c[3];
    ks_unpack(ks, key, 0, c);
    const uint32_t layers = (c[2] > 0 && c[2] - 1 < lim.z ? 0x1FFu : 0u) | (c[2] < lim.z ? 0x1FFu << 9 : 0u) |
                            (c[2] + 1 < lim.z ? 0x1FFu << 18 : 0u);
    if (m & ~layers) degen = true;
    m &= layers;
    uint32_t words = __ballot_sync(kFull, first && (lane == 0 || (prev ^ key) >> 5));
    if (ks.bits[2] >= 5 && 2 * __popc(words) < __popc(runs)) {
        // several leaves of one word (of one x and y): their nine rows, joined over the warp
        const int b = (int)(key & 31u);
        uint32_t rows = __reduce_or_sync(kFull, first ? m : 0u);
        rows |= rows >> 9 | rows >> 18;
        while (words) {
            const int src = __ffs(words) - 1;
            words &= words - 1u;
            const uint32_t W = __shfl_sync(kFull, key, src) >> 5;
            const bool mine = first && key >> 5 == W;
            int wc[3];
            ks_unpack(ks, W << 5, 0, wc);
            uint32_t row = 0u;  // lane r < 9: the bits of row r
#pragma unroll
            for (int r = 0; r < 9; r++) {
                if (!((rows >> r) & 1u)) continue;
                uint32_t z = mine ? m >> r : 0u;
                z = (z & 1u) | (z >> 8 & 2u) | (z >> 16 & 4u);
                const uint32_t bits = b == 0 ? z >> 1 : (b == 31 ? (z & 3u) << 30 : z << (b - 1));
                const uint32_t all = __reduce_or_sync(kFull, bits);
                if (lane == r) row = all;
                // past the word's ends
                if (z && (b == 0 || b == 31)) {
                    const int nx = wc[0] + r % 3 - 1, ny = wc[1] + r / 3 - 1;
                    if (nx < 0 || ny < 0 || nx >= lim.x || ny >= lim.y) {
                        degen = true;
                    } else {
                        const uint32_t k = ks_pack(ks, nx, ny, c[2], 0);
                        if (b == 0 && (z & 1u)) atomicOr(&x0bits[(k >> 5) - 1u], 0x80000000u);
                        if (b == 31 && (z & 4u)) atomicOr(&x0bits[(k >> 5) + 1u], 1u);
                    }
                }
            }
            if (row) {
                const int nx = wc[0] + lane % 3 - 1, ny = wc[1] + lane / 3 - 1;
                if (nx < 0 || ny < 0 || nx >= lim.x || ny >= lim.y)
                    degen = true;
                else
                    atomicOr(&x0bits[ks_pack(ks, nx, ny, wc[2], 0) >> 5], row);
            }
        }
        runs = 0u;
    }
    const int dx = lane % 3 - 1, dy = lane / 3 % 3 - 1;
    while (runs) {
        // three runs a turn, nine lanes each
        const int l0 = __ffs(runs) - 1;
        runs &= runs - 1u;
        const int l1 = __ffs(runs) - 1;
        runs &= runs - 1u;  // (0 stays 0)
        const int l2 = __ffs(runs) - 1;
        runs &= runs - 1u;
        const int src = lane < 9 ? l0 : lane < 18 ? l1 : lane < 27 ? l2 : -1;
        const uint32_t gm = __shfl_sync(kFull, m, max(src, 0)), gk = __shfl_sync(kFull, key, max(src, 0));
        // bits 0, 1, 2: the leaves below, beside and above
        uint32_t z = gm >> ((dy + 1) * 3 + dx + 1);
        z = (z & 1u) | (z >> 8 & 2u) | (z >> 16 & 4u);
        if (src < 0 || z == 0u) continue;
        int gc[3];
        ks_unpack(ks, gk, 0, gc);
        const int nx = gc[0] + dx, ny = gc[1] + dy;
        if (nx < 0 || ny < 0 || nx >= lim.x || ny >= lim.y) {
            degen = true;
            continue;
        }
        const uint32_t k = ks_pack(ks, nx, ny, gc[2], 0);
        const int b = (int)(k & 31u);
        const uint32_t here = b == 0 ? z >> 1 : (b == 31 ? (z & 3u) << 30 : z << (b - 1));
        if (here) atomicOr(&x0bits[k >> 5], here);
        if (b == 0 && (z & 1u)) atomicOr(&x0bits[(k >> 5) - 1u], 0x80000000u);
        if (b == 31 && (z & 4u)) atomicOr(&x0bits[(k >> 5) + 1u], 1u);
    }
    if (degen) atomicOr(err, GVX_DERR_DEGENERATE);
}

struct UpperDesc {
    int nlev;                  // levels 1..nlev are described (nlev = depth-1)
    uint32_t words[GVX_MAXLEV];
    uint32_t off[GVX_MAXLEV];  // per level: D bits, X bits, D prefix, X prefix (words each)
    int tshift[GVX_MAXLEV];
};

// parents of the cells of a word of a level-0 bitmap -> a bitmap per upper level.  Neighbouring cells share
// their parents: a parent met again ends the walk up, and above level 1 one whose bit is set is not set again
// (atomics on the few words of the top levels, one after the other, took most of 13 us in a frame of a fused
// scene; at level 1, where there are many words, waiting for the look would cost more than it saves).
__device__ __forceinline__ void upper_word(uint32_t bits, uint32_t w, const KeySpace& ks, const UpperDesc& ud,
                                           uint32_t* upper, int which)
{
    uint32_t last[GVX_MAXLEV];
#pragma unroll
    for (int l = 0; l < GVX_MAXLEV; l++) last[l] = 0xFFFFFFFFu;
    // runs of cells along z that share their level-1 parent: one of each is taken
    const int lz = min(min(ud.tshift[1], ks.bits[2]), 5);
    const uint32_t run = 0xFFFFFFFFu >> (32 - (1 << lz));
    while (bits) {
        const int b = (__ffs(bits) - 1) >> lz << lz;
        bits &= ~(run << b);
        int c[3];
        ks_unpack(ks, w * 32u + (uint32_t)b, 0, c);
#pragma unroll
        for (int l = 1; l < GVX_MAXLEV; l++) {
            if (l > ud.nlev) break;
            const int t = ud.tshift[l];
            const uint32_t k = ks_pack(ks, c[0] >> t, c[1] >> t, c[2] >> t, t);
            if (k == last[l]) break;  // (and its parents)
            last[l] = k;
            uint32_t* p = &upper[ud.off[l] + (which ? ud.words[l] : 0u) + (k >> 5)];
            if (l == 1 || !((*(volatile uint32_t*)p >> (k & 31)) & 1u)) atomicOr(p, 1u << (k & 31));
        }
    }
}

// D_l: parents of the leaves with points; A_l: of the box leaves (x0bits: blockIdx.y 1, where there are any)
__global__ void k_upper_bits(const uint32_t* __restrict__ d0bits, const uint32_t* __restrict__ x0bits, uint32_t words,
                             KeySpace ks, UpperDesc ud, uint32_t* upper)
{
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= words) return;
    uint32_t bits = d0bits[w];
    if (blockIdx.y) bits = x0bits[w] & ~bits;
    upper_word(bits, w, ks, ud, upper, (int)blockIdx.y);
}

// ---------------------------------------------------------------------------
// slots of d_counts: a planned UpdateAtlas's slot count, the dense leaves of the grouping
enum { kCntSlots = 56, kCntDense = 57 };

// The ranges of a ClearList: a block sets 4096 words of one of them, by 16 bytes where the range is aligned
struct ClearArgs {
    ClearList c;
    uint32_t chunk[ClearList::kMax];  // the first chunk of each range
};
constexpr uint32_t kClearChunk = 4096;
__global__ void __launch_bounds__(256) k_clear(ClearArgs a)
{
    int r = 0;
    while (r + 1 < a.c.n && a.chunk[r + 1] <= blockIdx.x) r++;
    const uint64_t w0 = (uint64_t)(blockIdx.x - a.chunk[r]) * kClearChunk;
    const uint64_t left = a.c.words[r] - w0;
    const uint32_t m = left < kClearChunk ? (uint32_t)left : kClearChunk;
    uint32_t* p = a.c.p[r] + w0;
    const uint32_t v = a.c.value[r];
    const uint32_t m4 = ((uintptr_t)p & 15u) ? 0u : m / 4u;
    const uint4 q = make_uint4(v, v, v, v);
    for (uint32_t i = threadIdx.x; i < m4; i += 256u) ((uint4*)p)[i] = q;
    for (uint32_t i = m4 * 4u + threadIdx.x; i < m; i += 256u) p[i] = v;
}

gvx_status gvx_clear(const ClearList& c, cudaStream_t st, int64_t* launches)
{
    if (c.full) {
        gvx_set_error("clear: more than %d ranges", ClearList::kMax);
        return c.full;
    }
    if (c.n == 0) return GVX_OK;
    ClearArgs a;
    a.c = c;
    uint64_t chunks = 0;
    for (int r = 0; r < c.n; r++) {
        a.chunk[r] = (uint32_t)chunks;
        chunks += (c.words[r] + kClearChunk - 1) / kClearChunk;
    }
    if (chunks > 0x7FFFFFFFull) {
        gvx_set_error("clear: %llu chunks", (unsigned long long)chunks);
        return GVX_ERR_CAPACITY;
    }
    k_clear<<<(unsigned)chunks, 256, 0, st>>>(a);
    (*launches)++;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

// the accumulators of GetBoundingBox and of the active leaves' box (k_bbox, k_leaf_bounds) before them
static void clear_bboxes(gvx_grid* g, ClearList& c)
{
    uint32_t* b = g->d_bbox.as<uint32_t>();
    c.add(b, 3, 0xFFFFFFFFu);  // min = all ones, max = 0 (order-preserving bits)
    c.add(b + 3, 3, 0u);
    c.add(b + 8, 3, 0x7FFFFFFFu);
    c.add(b + 11, 3, 0x80000000u);
}

// ---------------------------------------------------------------------------
// Exclusive prefix sums of several arrays in one go (of the popcounts of bitmap words, or of the words): a
// job each.  A job's word may be put together from bitmaps, (src | plus) & ~minus, and is stored then (store
// may be src: the value is the same again).  With `list` the set bits' keys, in order, go there (cap at
// most).
//
// Up to 32 blocks of 1024 words a job (a key space of 2^20 leaves), one launch does it: a block sums the
// words before its own by itself, 31 loads a thread at most, which takes less than the launch that would
// have summed them (4 us of the stream's time; with the list's, a third launch: 12 us -> 4 for 2^16 leaves).
// Above, a launch sums the blocks first: those sums would be read 32 times and more.
namespace {
struct PfxJob {
    const uint32_t *src, *plus, *minus;
    uint32_t* store;
    uint32_t* prefix;
    uint32_t words;
    uint32_t* total;
    uint32_t* list;
    uint32_t cap;
    uint32_t sums;  // where its block sums start (two launches)
};
struct PfxJobs {
    static constexpr int kMax = 2 * GVX_MAXLEV + 1;
    int n = 0;
    PfxJob j[kMax];
    PfxJob& add(const uint32_t* src, uint32_t* prefix, uint32_t words, uint32_t* total)
    {
        PfxJob& q = j[n++];
        q = PfxJob{src, nullptr, nullptr, nullptr, prefix, words, total, nullptr, 0xFFFFFFFFu, 0u};
        return q;
    }
};
constexpr uint32_t kPfxSelf = 32;
constexpr int kPfxThreads = 256, kPfxSelfThreads = 1024;
}  // namespace

// words base + k STEP, k < N, of a job, 0 from `end` on: all loads of an array before the next one's (a
// choice between arrays at each word would make every load wait for the last)
template <int N>
__device__ __forceinline__ void pfx_words(const PfxJob& q, uint32_t base, uint32_t step, uint32_t end, uint32_t (&v)[N])
{
#pragma unroll
    for (int k = 0; k < N; k++) {
        const uint32_t w = base + (uint32_t)k * step;
        v[k] = w < end ? q.src[w] : 0u;
    }
    if (q.plus) {
#pragma unroll
        for (int k = 0; k < N; k++) {
            const uint32_t w = base + (uint32_t)k * step;
            v[k] |= w < end ? q.plus[w] : 0u;
        }
    }
    if (q.minus) {
#pragma unroll
        for (int k = 0; k < N; k++) {
            const uint32_t w = base + (uint32_t)k * step;
            v[k] &= w < end ? ~q.minus[w] : 0u;
        }
    }
}

// POPC: the scanned values are the popcounts of bitmap words, else the words themselves
template <bool POPC>
__device__ __forceinline__ uint32_t pfx_value(uint32_t v)
{
    return POPC ? (uint32_t)__popc(v) : v;
}

// the sum of v over the block, in every thread
template <int THREADS>
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* s_w)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0u;
    for (int i = 0; i < THREADS / 32; i++) t += s_w[i];
    return t;
}

// per block of PER words a thread: the sum
template <bool POPC, int PER>
__global__ void __launch_bounds__(kPfxThreads) k_pfx_reduce(PfxJobs jobs, uint32_t* sums)
{
    const PfxJob& q = jobs.j[blockIdx.y];
    const uint32_t cbase = blockIdx.x * (kPfxThreads * PER);
    if (cbase >= q.words) return;
    uint32_t v[PER];
    pfx_words<PER>(q, cbase + threadIdx.x, kPfxThreads, q.words, v);
    uint32_t s = 0u;
#pragma unroll
    for (int k = 0; k < PER; k++) s += pfx_value<POPC>(v[k]);
    __shared__ uint32_t s_w[kPfxThreads / 32];
    s = block_sum<kPfxThreads>(s, s_w);
    if (threadIdx.x == 0) sums[q.sums + blockIdx.x] = s;
}

// the block's chunk in and out through shared memory (coalesced global loads and stores; index i
// of the chunk at i + i/32, so that a thread's PER consecutive values and the warps'
// strided rows are both free of bank conflicts), each thread scanning PER consecutive
// values after what comes before the block: SELF sums the words, else the earlier blocks' sums are added up
template <bool POPC, int THREADS, int PER, bool SELF>
__global__ void __launch_bounds__(THREADS) k_pfx_apply(PfxJobs jobs, const uint32_t* __restrict__ sums)
{
    constexpr uint32_t CHUNK = THREADS * PER;
    __shared__ uint32_t s_v[CHUNK + CHUNK / 32];
    __shared__ uint32_t s_w[THREADS / 32];
    const PfxJob& q = jobs.j[blockIdx.y];
    const uint32_t cbase = blockIdx.x * CHUNK;
    if (cbase >= q.words) return;
    uint32_t v[PER];
    pfx_words<PER>(q, cbase + threadIdx.x, THREADS, q.words, v);
    uint32_t before = 0u;
    if (SELF) {
        for (uint32_t w = threadIdx.x; w < cbase; w += 8u * THREADS) {
            uint32_t u[8];
            pfx_words<8>(q, w, THREADS, cbase, u);
#pragma unroll
            for (int k = 0; k < 8; k++) before += pfx_value<POPC>(u[k]);
        }
    } else {
        for (uint32_t i = threadIdx.x; i < blockIdx.x; i += THREADS) before += sums[q.sums + i];
    }
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const uint32_t i = (uint32_t)k * THREADS + threadIdx.x;
        s_v[i + (i >> 5)] = pfx_value<POPC>(v[k]);
    }
    before = block_sum<THREADS>(before, s_w);
    uint32_t cnt[PER];
    uint32_t s = 0u;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const uint32_t i = threadIdx.x * PER + k;
        cnt[k] = s_v[i + (i >> 5)];
        s += cnt[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = s;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();  // s_w is reused
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    uint32_t run = before + x - s;
    for (int k = 0; k < warp; k++) run += s_w[k];
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const uint32_t i = threadIdx.x * PER + k;
        s_v[i + (i >> 5)] = run;
        run += cnt[k];
    }
    // (the last thread of the last block: the words past the end count nothing)
    if (q.total && threadIdx.x == THREADS - 1 && q.words - cbase <= CHUNK) *q.total = run;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const uint32_t i = (uint32_t)k * THREADS + threadIdx.x, w = cbase + i;
        if (w >= q.words) break;
        uint32_t o = s_v[i + (i >> 5)];
        q.prefix[w] = o;
        if (q.store) q.store[w] = v[k];
        if (q.list) {
            uint32_t b = v[k];
            while (b && o < q.cap) {  // cap: the list's capacity
                const int bit = __ffs(b) - 1;
                b &= b - 1u;
                q.list[o++] = w * 32u + (uint32_t)bit;
            }
        }
    }
}

template <bool POPC, int PER>
static gvx_status pfx_two(PfxJobs& jobs, uint32_t most, DevBuf& tmp, cudaStream_t st, int64_t* launches)
{
    constexpr uint32_t chunk = kPfxThreads * PER;
    uint32_t sums = 0u;
    for (int i = 0; i < jobs.n; i++) {
        jobs.j[i].sums = sums;
        sums += (jobs.j[i].words + chunk - 1) / chunk;
    }
    GVX_CK(gvx_ensure(tmp, (size_t)(sums + 1) * sizeof(uint32_t)));
    const dim3 grid((most + chunk - 1) / chunk, (unsigned)jobs.n);
    k_pfx_reduce<POPC, PER><<<grid, kPfxThreads, 0, st>>>(jobs, tmp.as<uint32_t>());
    k_pfx_apply<POPC, kPfxThreads, PER, false><<<grid, kPfxThreads, 0, st>>>(jobs, tmp.as<uint32_t>());
    *launches += 2;
    return GVX_OK;
}

// (two launches: blocks of 1024 words, so that the key lists have the threads, until there are 1024 sums to
// add up in a block; then of 4096.  2^16 words with their list: 17 us by 4096, 6 by 1024)
template <bool POPC>
static gvx_status pfx_run(PfxJobs& jobs, DevBuf& tmp, cudaStream_t st, int64_t* launches)
{
    if (jobs.n == 0) return GVX_OK;
    uint32_t most = 1u;
    for (int i = 0; i < jobs.n; i++) most = std::max(most, jobs.j[i].words);
    if (most <= kPfxSelf * kPfxSelfThreads) {
        const dim3 grid((most + kPfxSelfThreads - 1) / kPfxSelfThreads, (unsigned)jobs.n);
        k_pfx_apply<POPC, kPfxSelfThreads, 1, true><<<grid, kPfxSelfThreads, 0, st>>>(jobs, nullptr);
        (*launches)++;
    } else if (most <= (1u << 20)) {
        GVX_CK_STATUS((pfx_two<POPC, 4>(jobs, most, tmp, st, launches)));
    } else {
        GVX_CK_STATUS((pfx_two<POPC, 16>(jobs, most, tmp, st, launches)));
    }
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

gvx_status gvx_bitmap_prefix(const uint32_t* bits, uint32_t* prefix, uint32_t words, uint32_t* total, DevBuf& tmp,
                             cudaStream_t st, int64_t* launches)
{
    PfxJobs jobs;
    jobs.add(bits, prefix, words, total);
    return pfx_run<true>(jobs, tmp, st, launches);
}

gvx_status gvx_scan_u32(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* total, DevBuf& tmp, cudaStream_t st,
                        int64_t* launches)
{
    PfxJobs jobs;
    jobs.add(in, out, n, total);
    return pfx_run<false>(jobs, tmp, st, launches);
}

// set bits -> sorted key lists, where the lists are sized after the prefixes (a thread a word)
__global__ void k_select(PfxJobs jobs)
{
    const PfxJob& q = jobs.j[blockIdx.y];
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= q.words) return;
    uint32_t b = q.src[w];
    uint32_t o = q.prefix[w];
    while (b && o < q.cap) {
        const int k = __ffs(b) - 1;
        b &= b - 1u;
        q.list[o++] = w * 32u + (uint32_t)k;
    }
}

static gvx_status select_run(const PfxJobs& jobs, cudaStream_t st, int64_t* launches)
{
    if (jobs.n == 0) return GVX_OK;
    uint32_t most = 1u;
    for (int i = 0; i < jobs.n; i++) most = std::max(most, jobs.j[i].words);
    k_select<<<dim3((most + 255u) / 256u, (unsigned)jobs.n), 256, 0, st>>>(jobs);
    (*launches)++;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

struct NodeLevelArgs {
    int lev, depth;
    uint32_t ucount, xcount;
    const uint32_t* dlist;
    const uint32_t* xlist;
    KeySpace ks;
    int tshift, tshift_parent, logdim_parent, res_parent;
    int lo[3];         // absolute level-l node coordinates of compact (0,0,0)
    int root_rel[3];   // root position in level-l node units (when the parent is the root)
    int range;
    BitRank pd, px;    // parent level bitmaps (unused when the parent is the root)
    uint32_t pucount;
    GvxNode* nodes;
    uint64_t* pclist;
    uint32_t* leaf_key;  // level 0 only
    // planned builds: the counts from device memory (dc[ci_u], dc[ci_x], dc[ci_pu]; ci_pu < 0: none),
    // this level's node capacity and the parent level's (0: no parent check)
    const uint32_t* dc;
    int ci_u, ci_x, ci_pu;
    uint32_t cap, pcap;
};

// the levels of a tree below its root, and the root
struct TreeArgs {
    int depth;
    int rootpos[3];
    GvxNode* root;
    NodeLevelArgs a[GVX_MAXLEV];
};

__device__ void write_root(const TreeArgs& t)
{
    GvxNode nd;
    nd.lev = (uint8_t)t.depth;
    nd.flags = 1;
    nd.prio = 0;
    nd.pad = 0;
    for (int k = 0; k < 3; k++) {
        nd.pos[k] = t.rootpos[k];
        nd.value[k] = -1;
        nd.vrange[k] = 0.f;
    }
    nd.parent = ID_UNDEFL_U64;
    nd.childlist = 1ull | ((uint64_t)t.depth << 8);
    nd.mask = 0ull;
    *t.root = nd;
}

// one node per thread, a level per blockIdx.y: Node record, parent reference, and the parent's child-list
// slot (SetupNode VG.cpp:2512-2524, gvdbLinkBricks cuda_gvdb_nodes.cuh:470-505).  A node's parent is found
// by rank, so no level waits for another.
__global__ void k_write_nodes(TreeArgs t)
{
    const NodeLevelArgs& a = t.a[blockIdx.y];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) write_root(t);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t ucount = a.ucount, xcount = a.xcount, pucount = a.pucount;
    if (a.dc) {
        ucount = min(a.dc[a.ci_u], a.cap);
        xcount = min(a.dc[a.ci_x], a.cap - ucount);
        pucount = a.ci_pu >= 0 ? a.dc[a.ci_pu] : 0u;
    }
    if (i >= ucount + xcount) return;
    const uint32_t key = i < ucount ? a.dlist[i] : a.xlist[i - ucount];
    int c[3];
    ks_unpack(a.ks, key, a.tshift, c);
    GvxNode nd;
    nd.lev = (uint8_t)a.lev;
    nd.flags = 1;
    nd.prio = 0;
    nd.pad = 0;
    for (int k = 0; k < 3; k++) {
        nd.pos[k] = (a.lo[k] + c[k]) * a.range;
        nd.value[k] = -1;
        nd.vrange[k] = 0.f;
    }
    nd.mask = 0ull;
    nd.childlist = a.lev > 0 ? (1ull | ((uint64_t)a.lev << 8) | ((uint64_t)i << 16)) : ID_UNDEFL_U64;
    uint32_t pidx;
    int rel[3];
    const int res = a.res_parent;
    bool linked = true;
    if (a.lev + 1 == a.depth) {
        pidx = 0u;
        for (int k = 0; k < 3; k++) {
            rel[k] = a.lo[k] + c[k] - a.root_rel[k];
            // (a key space rounded up to powers of two may reach past the root: a planned build's
            // points there make it void -- the frame's root differs -- and are not linked)
            linked = linked && rel[k] >= 0 && rel[k] < res;
        }
    } else {
        const int sh = a.logdim_parent;
        const uint32_t pk = ks_pack(a.ks, c[0] >> sh, c[1] >> sh, c[2] >> sh, a.tshift_parent);
        pidx = br_test(a.pd, pk) ? br_rank(a.pd, pk) : pucount + br_rank(a.px, pk);
        for (int k = 0; k < 3; k++) rel[k] = c[k] & (res - 1);
    }
    nd.parent = ((uint64_t)pidx << 16) | ((uint64_t)(a.lev + 1) << 8);
    const int bit = (rel[2] * res + rel[1]) * res + rel[0];
    // (a parent beyond its pool's capacity: no link -- the planned build is void)
    if (linked && (!a.pcap || pidx < a.pcap))
        a.pclist[(size_t)pidx * res * res * res + bit] = ((uint64_t)i << 16) | ((uint64_t)a.lev << 8);
    a.nodes[i] = nd;
    if (a.leaf_key) a.leaf_key[i] = key;
}

// run of equal leaf keys in sorted order -> [start, end) of its leaf.  With octants in the keys
// (kshift 3) also the first sorted index of every octant of the leaf's points (leaf_oct[8 l + o] =
// start + the points of octants < o), written at the starts of the octant runs and at the leaf's end
// dense_list (optional): the leaves of kDenseLeaf points and more, in no order -- the keys are sorted, so
// such a run reaches kDenseLeaf - 1 entries back from its last one
constexpr int kDenseLeaf = 128;
__device__ __forceinline__ void group_run(uint32_t i, const uint32_t* __restrict__ skeys, uint32_t n, int kshift,
                                          uint32_t invalid_key, const LeafLookup& L, int2* leaf_range, int* leaf_oct,
                                          uint32_t* dense_list, uint32_t* dense_count)
{
    const uint32_t sk = skeys[i], k = sk >> kshift;
    if (k >= invalid_key) return;
    const uint32_t prev = i == 0 ? 0xFFFFFFFFu : skeys[i - 1];
    const bool first = i == 0 || (prev >> kshift) != k;
    const bool last = i + 1 == n || (skeys[i + 1] >> kshift) != k;
    const bool ostart = kshift && (first || prev != sk);
    if (!first && !last && !ostart) return;
    int c[3];
    ks_unpack(L.ks, k, 0, c);
    const int leaf = ll_find(L, c[0], c[1], c[2]);
    if (leaf < 0) return;
    if (first) leaf_range[leaf].x = (int)i;
    if (last) {
        leaf_range[leaf].y = (int)(i + 1);
        if (dense_list && i + 1 >= (uint32_t)kDenseLeaf && (skeys[i + 1 - kDenseLeaf] >> kshift) == k)
            dense_list[atomicAdd(dense_count, 1u)] = (uint32_t)leaf;
    }
    if (kshift) {
        int* lo = leaf_oct + (size_t)leaf * 8;
        const int o = (int)(sk & 7u);
        if (ostart)
            for (int q = first ? 0 : (int)(prev & 7u) + 1; q <= o; q++) lo[q] = (int)i;
        if (last)
            for (int q = o + 1; q < 8; q++) lo[q] = (int)(i + 1);
    }
}

// Points of the dense leaves (bricks of 8, octants in the sort keys) in cell order: a stable counting
// sort of each leaf's range of sorted point indices by the cell of the point's voxel, octant first (the
// order the keys already give), then (x, y, z) inside the octant; cell_tab gets the first sorted index
// of every cell.  One block a leaf, every warp a contiguous part of its points, so that equal cells keep
// their order; the leaves differ in size by factors of a hundred, the blocks take them in turn.  A leaf
// with a point that is no longer where its key was made (written in place since) keeps its order and gets
// no dense number.
constexpr int kCellThreads = 512, kCellWarps = kCellThreads / 32;
__global__ void __launch_bounds__(kCellThreads)
    k_cell_sort(const uint32_t* __restrict__ dense_list, const uint32_t* __restrict__ dense_count,
                const int2* __restrict__ leaf_range, const GvxNode* __restrict__ nodes0,
                const uint32_t* __restrict__ skeys, const char* pos, int off, int stride, float ox, float oy, float oz,
                uint32_t* vals, uint32_t* vtmp, int* __restrict__ cell_tab, int* __restrict__ leaf_dense)
{
    __shared__ int s_cnt[kCellWarps][512];
    __shared__ int s_sum[kCellWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto cell_of = [&](uint32_t v, const int4& org, bool& in) {
        float w[3];
        load_pos(pos, off, stride, v, w);
        w[0] += ox;
        w[1] += oy;
        w[2] += oz;
        return brick8_cell(w, org, in);
    };
    const uint32_t count = *dense_count;
    for (uint32_t d = blockIdx.x; d < count; d += gridDim.x) {
        const uint32_t leaf = dense_list[d];
        const int2 r = leaf_range[leaf];
        const int4 org = *(const int4*)(nodes0 + leaf);  // (lev.., x, y, z)
        const int per = (r.y - r.x + kCellThreads - 1) / kCellThreads * 32;  // points a warp
        const int b0 = min(r.x + warp * per, r.y), b1 = min(b0 + per, r.y);
#pragma unroll
        for (int w = 0; w < kCellWarps; w++) s_cnt[w][tid] = 0;
        __syncthreads();
        bool moved = false;
        for (int i0 = b0 + lane; i0 < b1; i0 += 128) {
            int c[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                c[q] = -1;
                if (i0 + 32 * q < b1) {
                    bool in;
                    c[q] = cell_of(vals[i0 + 32 * q], org, in);
                    moved = moved || !in || (uint32_t)(c[q] >> 6) != (skeys[i0 + 32 * q] & 7u);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (c[q] >= 0) atomicAdd(&s_cnt[warp][c[q]], 1);
        }
        if (__syncthreads_or(moved)) continue;
        int run = 0;  // thread c: the places of cell c's points, warp after warp
#pragma unroll
        for (int w = 0; w < kCellWarps; w++) {
            const int n = s_cnt[w][tid];
            s_cnt[w][tid] = run;
            run += n;
        }
        int x = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_sum[warp] = x;
        __syncthreads();
        int start = r.x + x - run;
        for (int w = 0; w < warp; w++) start += s_sum[w];
#pragma unroll
        for (int w = 0; w < kCellWarps; w++) s_cnt[w][tid] += start;
        cell_tab[(size_t)d * 512 + tid] = start;
        if (tid == 0) leaf_dense[leaf] = (int)d + 1;
        __syncthreads();
        for (int i0 = b0; i0 < b1; i0 += 128) {
            uint32_t v[4];
            int c[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int i = i0 + 32 * q + lane;
                bool in;
                v[q] = i < b1 ? vals[i] : 0u;
                c[q] = i < b1 ? cell_of(v[q], org, in) : -1 - lane;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t same = __match_any_sync(0xFFFFFFFFu, c[q]);
                int at = 0;
                if (c[q] >= 0) {
                    at = s_cnt[warp][c[q]];
                    vtmp[at + __popc(same & ((1u << lane) - 1u))] = v[q];
                }
                __syncwarp();
                if (c[q] >= 0 && lane == __ffs(same) - 1) s_cnt[warp][c[q]] = at + __popc(same);
                __syncwarp();
            }
        }
        __syncthreads();
        for (int i = r.x + tid; i < r.y; i += kCellThreads) vals[i] = vtmp[i];
        __syncthreads();
    }
}

// Points of every leaf in octant order: a stable partition of the leaf's range
// of sorted point indices by the half of the brick that each point's voxel
// (floor of the translated position, as the keys take it) lies in on every
// axis, octant = 4 hx + 2 hy + hz, and the first index of every octant.  The
// sorted order becomes (leaf key, octant, point index); the splat reads only
// the octants of a neighbouring brick whose points can reach its slab.  For
// key spaces too wide for the octant in the sort key (more than 2^28 leaf
// cells; otherwise the sort itself orders the octants).  A segment of G lanes
// per leaf, launched with G = 32 (segments of 8 lanes were slower on leaves
// of very different sizes: the longest leaf of a warp sets its trip count);
// the segment's lanes 0-7 keep the octants' counters.  With A.spos the sorted
// point attributes of the leaves' points are written in the same pass (as
// k_permute writes them); entries outside the leaf ranges are not, and no
// reader takes them (a point is splatted only when its own leaf exists).
template <int G>
__global__ void k_octant_partition(const int2* __restrict__ leaf_range, DevCount nlc,
                                   const GvxNode* __restrict__ nodes0, const char* pos, int off, int stride, float ox,
                                   float oy, float oz, int half, const uint32_t* __restrict__ vin,
                                   uint32_t* __restrict__ vout, int* __restrict__ leaf_oct, GvxSortedAttr A)
{
    static_assert(G == 8 || G == 16 || G == 32, "segments of 8, 16 or 32 lanes");
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int sl = lane & (G - 1), sb = lane - sl;  // lane in the segment, the segment's first lane
    const uint32_t smask = G == 32 ? 0xFFFFFFFFu : (((1u << G) - 1u) << sb);
    const uint32_t nl = nlc.get();
    if ((gt & ~31u) / G >= nl) return;  // whole warps: the warp's first leaf is past the last
    const uint32_t leaf = gt / G;
    const bool live = leaf < nl;
    int2 r = make_int2(0, 0);
    int bx = 0, by = 0, bz = 0;
    if (live) {
        r = leaf_range[leaf];
        bx = nodes0[leaf].pos[0] + half;
        by = nodes0[leaf].pos[1] + half;
        bz = nodes0[leaf].pos[2] + half;
    }
    // translated position and octant of sorted entry i (octant -1 past the leaf's range)
    auto fetch = [&](int i, uint32_t& v, float* w) {
        if (i >= r.y) return -1;
        v = vin[i];
        load_pos(pos, off, stride, v, w);
        w[0] += ox;
        w[1] += oy;
        w[2] += oz;
        const int x = (int)floorf(w[0]), y = (int)floorf(w[1]), z = (int)floorf(w[2]);
        return (x >= bx ? 4 : 0) | (y >= by ? 2 : 0) | (z >= bz ? 1 : 0);
    };
    const int nch = __reduce_max_sync(0xFFFFFFFFu, (r.y - r.x + G - 1) / G);  // chunks of the warp's longest leaf
    int cnt = 0;  // segment lane o < 8: points of octant o
    uint32_t v0 = 0u;  // the segment's first G points, kept for the placement pass
    float w0[3] = {0.f, 0.f, 0.f};
    int o0 = -1;
    for (int c = 0; c < nch; c++) {
        uint32_t v = 0u;
        float w[3];
        const int o = fetch(r.x + c * G + sl, v, w);
        if (c == 0) {
            v0 = v;
            o0 = o;
            w0[0] = w[0];
            w0[1] = w[1];
            w0[2] = w[2];
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, o == k) & smask;
            if (sl == k) cnt += __popc(m);
        }
    }
    int incl = cnt;
#pragma unroll
    for (int s = 1; s < 8; s <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, incl, s, G);
        if (sl >= s) incl += t;
    }
    int run = r.x + incl - cnt;  // segment lane o < 8: next index of octant o
    if (live && sl < 8) leaf_oct[(size_t)leaf * 8 + sl] = run;
    for (int c = 0; c < nch; c++) {
        uint32_t v = v0;
        float w[3] = {w0[0], w0[1], w0[2]};
        int o = o0;
        if (c > 0) o = fetch(r.x + c * G + sl, v, w);
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, o < 0 ? 0xFFFFFFFFu : (uint32_t)(o | (sb << 3)));
        const int dst = __shfl_sync(0xFFFFFFFFu, run, sb + (o < 0 ? 0 : o)) + __popc(same & ((1u << lane) - 1u));
        if (o >= 0) vout[dst] = v;
        if (A.spos) {
            float rr = 0.0f;
            if (o >= 0) {
                A.spos[dst] = make_float4(w[0], w[1], w[2], A.weight ? A.weight[v] : 1.0f);
                if (A.radius) rr = A.radius[v];
                if (A.svel) {
                    float4 q = make_float4(0.f, 0.f, 0.f, rr);
                    if (A.vel) {
                        const float* u = (const float*)(A.vel + (size_t)v * A.vel_stride + A.vel_off);
                        q.x = u[0];
                        q.y = u[1];
                        q.z = u[2];
                    }
                    A.svel[dst] = q;
                }
                rr = rr != rr ? 3.0e38f : fmaxf(rr, 0.0f);
            }
            if (A.rmax) {
                const unsigned int mm = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(rr));
                // most warps find the maximum already there: read before the atomic
                if (lane == 0 && mm && mm > *(volatile unsigned int*)A.rmax) atomicMax(A.rmax, mm);
            }
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, o == k) & smask;
            if (sl == k) run += __popc(m);
        }
    }
}

// 27-neighbourhood of every leaf (leaf pool indices, -1 where no leaf; all -1
// for an inactive leaf, whose key is kNoKey)
constexpr uint32_t kNoKey = 0xFFFFFFFFu;
__device__ __forceinline__ void leaf_neighbour(uint32_t t, const uint32_t* __restrict__ leaf_key, const DevCount& nl,
                                               const LeafLookup& L, int* nbr)
{
    const uint32_t nleaves = nl.get();
    if (t >= nleaves * 27u) return;
    const uint32_t leaf = t / 27u, d = t % 27u;
    const uint32_t key = leaf_key[leaf];
    if (key == kNoKey) {
        nbr[t] = -1;
        return;
    }
    int c[3];
    ks_unpack(L.ks, key, 0, c);
    nbr[t] = ll_find(L, c[0] + (int)(d % 3u) - 1, c[1] + (int)((d / 3u) % 3u) - 1, c[2] + (int)(d / 9u) - 1);
}

// the neighbours of the leaves (the first nb blocks) and the runs of their points, which need no more of each
// other than the lookup: one launch
__global__ void k_leaf_tables(uint32_t nb, const uint32_t* __restrict__ leaf_key, DevCount nl, int* nbr,
                              const uint32_t* __restrict__ skeys, uint32_t n, int kshift, uint32_t invalid_key,
                              LeafLookup L, int2* leaf_range, int* leaf_oct, uint32_t* dense_list,
                              uint32_t* dense_count)
{
    if (blockIdx.x < nb) {
        leaf_neighbour(blockIdx.x * blockDim.x + threadIdx.x, leaf_key, nl, L, nbr);
        return;
    }
    const uint32_t i = (blockIdx.x - nb) * blockDim.x + threadIdx.x;
    if (i < n) group_run(i, skeys, n, kshift, invalid_key, L, leaf_range, leaf_oct, dense_list, dense_count);
}

// active leaves (mFlags) -> bitmap over pool indices
__global__ void k_flag_bits(const GvxNode* __restrict__ nodes, DevCount nc, uint32_t* bits)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n = nc.get();
    const bool f = i < n && nodes[i].flags;
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, f);
    if ((threadIdx.x & 31) == 0 && i < ((n + 31u) & ~31u)) bits[i >> 5] = b;
}

// UpdateAtlas: active leaf k (pool order) -> atlas slot k, mValue, atlas map
// (VG.cpp:2650-2690, AL.cpp:692-715)
// the atlas position of slot s, and its leaf i there
__device__ __forceinline__ void atlas_place(GvxNode* nodes, uint32_t i, uint32_t s, int sx, int sy, int P, int apron,
                                            int* leaf_slot, int* slot_leaf, int4* amap)
{
    const int a2 = sx * sy;
    const int z = (int)s / a2, rem = (int)s - z * a2;
    const int y = rem / sx, x = rem - y * sx;
    GvxNode* nd = nodes + i;
    nd->value[0] = x * P + apron;
    nd->value[1] = y * P + apron;
    nd->value[2] = z * P + apron;
    leaf_slot[i] = (int)s;
    slot_leaf[s] = (int)i;
    amap[s] = make_int4(nd->pos[0], nd->pos[1], nd->pos[2], (int)i);
}

// a thread per slot; the flags, their prefix and two clears of the general case below took five launches
// more, 4 us each
__global__ void k_atlas_all(GvxNode* nodes, DevCount nc, uint32_t slots, int sx, int sy, int P, int apron,
                            int* leaf_slot, int* slot_leaf, int4* amap, uint32_t* nslots)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n = nc.get();
    if (i == 0 && nslots) *nslots = n;
    if (i < n)
        atlas_place(nodes, i, i, sx, sy, P, apron, leaf_slot, slot_leaf, amap);
    else if (i < slots)
        amap[i] = make_int4(-1, -1, -1, -1);
}

__global__ void k_atlas_assign(GvxNode* nodes, DevCount nc, const uint32_t* __restrict__ fbits,
                               const uint32_t* __restrict__ fprefix, int sx, int sy, int P, int apron,
                               int* leaf_slot, int* slot_leaf, int4* amap)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc.get()) return;
    if (!((fbits[i >> 5] >> (i & 31)) & 1u)) {
        leaf_slot[i] = -1;
        return;
    }
    const uint32_t s = fprefix[i >> 5] + __popc(fbits[i >> 5] & ((1u << (i & 31)) - 1u));
    atlas_place(nodes, i, s, sx, sy, P, apron, leaf_slot, slot_leaf, amap);
}

// ComputeBounds (VG.cpp:1792-1816): bbox of active leaves (threads 0-5 of a block hold its atomics)
__device__ __forceinline__ void leaf_bounds(const GvxNode* __restrict__ nodes, uint32_t n, int range, int* out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // whole warps: the grid is a multiple of 32
    int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
    if (i < n && nodes[i].flags) {
        for (int a = 0; a < 3; a++) {
            mn[a] = nodes[i].pos[a];
            mx[a] = nodes[i].pos[a] + range;
        }
    }
    // warp, then block, then one atomic per block and bound
#pragma unroll
    for (int a = 0; a < 3; a++) {
        for (int s = 16; s > 0; s >>= 1) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xFFFFFFFFu, mn[a], s));
            mx[a] = max(mx[a], __shfl_xor_sync(0xFFFFFFFFu, mx[a], s));
        }
    }
    __shared__ int s_b[32][6];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0)
        for (int a = 0; a < 3; a++) {
            s_b[wid][a] = mn[a];
            s_b[wid][3 + a] = mx[a];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        int v = s_b[0][threadIdx.x];
        for (int w = 1; w < nw; w++) v = threadIdx.x < 3 ? min(v, s_b[w][threadIdx.x]) : max(v, s_b[w][threadIdx.x]);
        if (threadIdx.x < 3) {
            if (v != INT_MAX) atomicMin(&out[threadIdx.x], v);
        } else if (v != INT_MIN) {
            atomicMax(&out[threadIdx.x], v);
        }
    }
}

__global__ void k_leaf_bounds(const GvxNode* __restrict__ nodes, uint32_t n, int range, int* out)
{
    leaf_bounds(nodes, n, range, out);
}

// ---------------------------------------------------------------------------
// incremental rebuild: ActivateIncreBricksGPU (VG.cpp:1020-1156),
// gvdbCalcIncreBrickId / gvdbCalcIncreExtraBrickId (PT.cuh:384-465),
// gvdbLinkBricks (ND.cuh:470-505), gvdbDelinkLeafBricks / gvdbDelinkBricks
// (ND.cuh:401-467).
//
// In the reference a node is reachable by a root descent exactly when its
// parent reference is set: delinking clears the slot in the parent's child
// list and writes ID_UNDEF64 into the node, and only reachable nodes gain
// children.  The descents therefore become bitmap tests over one compact key
// space: L_l = linked level-l nodes, T_l = nodes the points' boxes touch,
// N_l = T_l & ~L_l = the nodes the reference allocates, in key order.

enum { kSetLinked = 0, kSetActive = 1 };

__device__ __forceinline__ bool node_key(const GvxNode& nd, const KeySpace& ks, int t, int range, uint32_t* key)
{
    int c[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        c[a] = nd.pos[a] / range - (ks.lo[a] >> t);
        if (c[a] < 0 || c[a] >= ks_extent(ks, a, t)) return false;
    }
    *key = ks_pack(ks, c[0], c[1], c[2], t);
    return true;
}

__device__ __forceinline__ bool in_node_set(const GvxNode& nd, int set)
{
    return set == kSetActive ? nd.flags != 0 : nd.parent != ID_UNDEF64_U64;
}

// the nodes of a level, their set's bitmap and the table k_node_remap fills; a level per blockIdx.y
struct NodeSet {
    const GvxNode* nodes;
    uint32_t n;
    int t, range;
    BitRank br;
    int* remap;
    uint32_t* leaf_key;
};
struct NodeSets {
    int n = 0;
    uint32_t most = 0u;
    NodeSet s[GVX_MAXLEV];
    void add(const GvxNode* nodes, uint32_t cnt, int t, int range, const BitRank& br, int* remap, uint32_t* leaf_key)
    {
        if (cnt == 0) return;
        s[n++] = NodeSet{nodes, cnt, t, range, br, remap, leaf_key};
        most = most < cnt ? cnt : most;
    }
    dim3 grid() const { return dim3((most + 255u) / 256u, (unsigned)n); }
};

// bitmap of a level's linked (or active) nodes; linked nodes outside the key
// space cannot be touched and are left out, an active leaf outside it is an error
__global__ void k_node_bits(NodeSets a, KeySpace ks, int set, uint32_t* err)
{
    const NodeSet& q = a.s[blockIdx.y];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.n) return;
    const GvxNode nd = q.nodes[i];
    if (!in_node_set(nd, set)) return;
    uint32_t key;
    if (node_key(nd, ks, q.t, q.range, &key))
        atomicOr(&q.br.bits[key >> 5], 1u << (key & 31));
    else if (set == kSetActive)
        atomicOr(err, GVX_DERR_DEGENERATE);
}

// rank in the set's bitmap -> pool index; with `leaf_key`, also the compact key
// of every leaf (kNoKey where the leaf is not in the set)
__global__ void k_node_remap(NodeSets a, KeySpace ks, int set)
{
    const NodeSet& q = a.s[blockIdx.y];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.n) return;
    const GvxNode nd = q.nodes[i];
    uint32_t key = kNoKey;
    if (in_node_set(nd, set) && node_key(nd, ks, q.t, q.range, &key))
        q.remap[br_rank(q.br, key)] = (int)i;
    else
        key = kNoKey;
    if (q.leaf_key) q.leaf_key[i] = key;
}

// markers of the existing leaves (VG.cpp:1028-1043, 1078-1085): a linked leaf
// inside some point's box gets 1, every other leaf keeps its flag
// (AccumulateTopology) or gets 0
__global__ void k_apply_markers(GvxNode* nodes, uint32_t n, KeySpace ks, int range, const uint32_t* __restrict__ d0,
                                const uint32_t* __restrict__ x0, int accum)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GvxNode nd = nodes[i];
    uint8_t m = accum ? nd.flags : 0;
    uint32_t key;
    if (nd.parent != ID_UNDEF64_U64 && node_key(nd, ks, 0, range, &key) &&
        (((d0[key >> 5] | x0[key >> 5]) >> (key & 31)) & 1u))
        m = 1;
    nodes[i].flags = m;
}

struct IncNodeArgs {
    int lev;
    uint32_t count;        // new nodes of this level
    uint32_t base;         // pool index of the first one (the old pool size)
    const uint32_t* keys;  // their compact keys, sorted
    KeySpace ks;
    int tshift, range;
    int lo[3];             // absolute level-l coordinates of compact (0,0,0)
    GvxNode* nodes;
    int parent_root;       // the parent level is the root's
    int root_rel[3];       // root position in level-l node units
    BitRank pl;            // linked parents, with their pool indices in premap
    const int* premap;
    BitRank pn;            // new parents (bits null when the parent level gets none)
    uint32_t pbase;        // pool index of the first new parent
    int logdim_parent, res_parent, tshift_parent;
    uint64_t* pclist;
    uint32_t* err;
};

struct IncTreeArgs {
    IncNodeArgs a[GVX_MAXLEV];
};

// one new node per thread, a level per blockIdx.y: SetupNode (VG.cpp:2512-2524) and its link
// (gvdbLinkBricks); the parent is a linked node or a new one of this build, found by rank
__global__ void k_inc_write_nodes(IncTreeArgs t)
{
    const IncNodeArgs& a = t.a[blockIdx.y];
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= a.count) return;
    const uint32_t i = a.base + j;
    int c[3];
    ks_unpack(a.ks, a.keys[j], a.tshift, c);
    GvxNode nd;
    nd.lev = (uint8_t)a.lev;
    nd.flags = 1;
    nd.prio = 0;
    nd.pad = 0;
    for (int k = 0; k < 3; k++) {
        nd.pos[k] = (a.lo[k] + c[k]) * a.range;
        nd.value[k] = -1;
        nd.vrange[k] = 0.f;
    }
    nd.mask = 0ull;
    nd.childlist = a.lev > 0 ? (1ull | ((uint64_t)a.lev << 8) | ((uint64_t)i << 16)) : ID_UNDEFL_U64;
    const int res = a.res_parent;
    uint32_t pidx = 0u;
    int rel[3];
    bool ok = true;
    if (a.parent_root) {
        for (int k = 0; k < 3; k++) {
            rel[k] = a.lo[k] + c[k] - a.root_rel[k];
            if (rel[k] < 0 || rel[k] >= res) ok = false;
        }
    } else {
        const int sh = a.logdim_parent;
        const uint32_t pk = ks_pack(a.ks, c[0] >> sh, c[1] >> sh, c[2] >> sh, a.tshift_parent);
        if (br_test(a.pl, pk))
            pidx = (uint32_t)a.premap[br_rank(a.pl, pk)];
        else if (a.pn.bits && br_test(a.pn, pk))
            pidx = a.pbase + br_rank(a.pn, pk);
        else
            ok = false;
        for (int k = 0; k < 3; k++) rel[k] = c[k] & (res - 1);
    }
    if (ok) {
        nd.parent = ((uint64_t)pidx << 16) | ((uint64_t)(a.lev + 1) << 8);
        const int bit = (rel[2] * res + rel[1]) * res + rel[0];
        a.pclist[(size_t)pidx * res * res * res + bit] = ((uint64_t)i << 16) | ((uint64_t)a.lev << 8);
    } else {
        nd.parent = ID_UNDEFL_U64;  // no parent to link to: the reference's descent fails here
        atomicOr(a.err, GVX_DERR_DEGENERATE);
    }
    a.nodes[i] = nd;
}

// clear node i's slot in its parent's child list and its parent reference
__device__ void unlink_node(GvxNode* nodes, uint32_t i, const GvxNode& nd, const GvxNode* __restrict__ pnodes,
                            uint32_t pcount, uint64_t* pclist, int res_p, int range, uint32_t* err)
{
    const uint64_t pid = nd.parent >> 16;
    if (pid >= pcount) {
        atomicOr(err, GVX_DERR_DEGENERATE);
        return;
    }
    const GvxNode& pn = pnodes[pid];
    int b[3];
    for (int a = 0; a < 3; a++) {
        const int d = nd.pos[a] - pn.pos[a];
        b[a] = d / range;
        if (d < 0 || b[a] >= res_p) {
            atomicOr(err, GVX_DERR_DEGENERATE);
            return;
        }
    }
    const uint64_t cl = pn.childlist >> 16;  // == pid: lists are allocated in lockstep with the nodes
    if (cl >= pcount) {
        atomicOr(err, GVX_DERR_DEGENERATE);
        return;
    }
    const size_t vc = (size_t)res_p * res_p * res_p;
    pclist[(size_t)cl * vc + (b[2] * res_p + b[1]) * res_p + b[0]] = ID_UNDEF64_U64;
    nodes[i].parent = ID_UNDEF64_U64;
}

// gvdbDelinkLeafBricks (ND.cuh:401-428): unmarked leaves leave the tree
__global__ void k_delink_leaves(GvxNode* nodes, uint32_t n, const GvxNode* __restrict__ pnodes, uint32_t pcount,
                                uint64_t* pclist, int res_p, int range, uint32_t* err)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GvxNode nd = nodes[i];
    if (nd.flags || nd.parent == ID_UNDEF64_U64) return;
    unlink_node(nodes, i, nd, pnodes, pcount, pclist, res_p, range, err);
}

// gvdbDelinkBricks (ND.cuh:430-467) for one level, one warp per node: a linked
// node with any child stays active, a childless one leaves the tree
__global__ void k_delink_upper(GvxNode* nodes, uint32_t n, const uint64_t* __restrict__ clist, uint32_t vc,
                               const GvxNode* __restrict__ pnodes, uint32_t pcount, uint64_t* pclist, int res_p,
                               int range, uint32_t* err)
{
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= n) return;  // warp-uniform
    const GvxNode nd = nodes[i];
    if (nd.parent == ID_UNDEF64_U64) {
        if (lane == 0) nodes[i].flags = 0;
        return;
    }
    const uint64_t* cl = clist + (size_t)i * vc;
    bool any = false;
    // eight loads a turn: one at a time, 600 ns each, a node whose children come late took 8 us
    for (uint32_t s0 = (uint32_t)lane; s0 - (uint32_t)lane < vc; s0 += 256u) {
        uint64_t c[8];
#pragma unroll
        for (int k = 0; k < 8; k++) c[k] = s0 + 32u * k < vc ? cl[s0 + 32u * k] : ID_UNDEF64_U64;
        bool here = false;
#pragma unroll
        for (int k = 0; k < 8; k++) here = here || c[k] != ID_UNDEF64_U64;
        if (__any_sync(0xFFFFFFFFu, here)) {
            any = true;
            break;
        }
    }
    if (lane != 0) return;
    if (any) {
        nodes[i].flags = 1;
        return;
    }
    nodes[i].flags = 0;
    unlink_node(nodes, i, nd, pnodes, pcount, pclist, res_p, range, err);
}

// ---------------------------------------------------------------------------
// host orchestration

static inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// decodes a device error word that was read back (and clears it on the device:
// each error is reported once)
static gvx_status report_device_error(gvx_grid* g, uint32_t e, const char* stage)
{
    if (e) GVX_CK(cudaMemsetAsync(g->d_err.p, 0, sizeof(uint32_t), g->stream));
    if (e & GVX_DERR_TIMEOUT) {
        gvx_set_error("%s: a device spin-wait timed out", stage);
        return GVX_ERR_TIMEOUT;
    }
    if (e & GVX_DERR_CAPACITY) {
        gvx_set_error("%s: device buffer capacity exceeded", stage);
        return GVX_ERR_CAPACITY;
    }
    if (e & GVX_DERR_BADPOINT) {
        gvx_set_error("%s: NaN point position", stage);
        return GVX_ERR_INVALID_ARG;
    }
    if (e & GVX_DERR_RADIUS) {
        gvx_set_error("%s: a per-point radius exceeds brick-1 (footprint beyond the 26 neighbouring bricks)", stage);
        return GVX_ERR_UNSUPPORTED;
    }
    return GVX_OK;
}

gvx_status gvx_check_device_error(gvx_grid* g, const char* stage)
{
    uint32_t e = 0;
    GVX_CK(cudaMemcpyAsync(&e, g->d_err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, g->stream));
    GVX_CK(cudaStreamSynchronize(g->stream));
    return report_device_error(g, e, stage);
}

__global__ void k_begin_errors(uint32_t* err, uint32_t* counter)
{
    *err &= GVX_DERR_TIMEOUT;
    if (counter) *counter = 0u;
}

gvx_status gvx_begin_errors(gvx_grid* g, uint32_t* counter)
{
    k_begin_errors<<<1, 1, 0, g->stream>>>(g->d_err.as<uint32_t>(), counter);
    g->launches++;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

// The counts, the bounding boxes and the device error word in one copy through pinned staging
// (queued: the copy; then, once the stream has passed it, readback_finish takes
// `bytes` from word `first` of d_counts and reports the error word as above)
static gvx_status readback_start(gvx_grid* g)
{
    if (!g->h_pin) GVX_CK(cudaMallocHost(&g->h_pin, 512));
    GVX_CK(cudaMemcpyAsync(g->h_pin, g->d_counts.p, kReadWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, g->stream));
    return GVX_OK;
}

static gvx_status readback_finish(gvx_grid* g, void* dst, int first, size_t bytes, const char* stage)
{
    GVX_CK(cudaStreamSynchronize(g->stream));
    const uint32_t* h = (const uint32_t*)g->h_pin;
    memcpy(dst, h + first, bytes);
    return report_device_error(g, h[kReadErr], stage);
}

static gvx_status readback_checked(gvx_grid* g, void* dst, int first, size_t bytes, const char* stage)
{
    gvx_status rc = readback_start(g);
    return rc ? rc : readback_finish(g, dst, first, bytes, stage);
}

static gvx_status ensure_grid_scratch(gvx_grid* g)
{
    if (g->d_err.p) return GVX_OK;  // (made with the grid)
    gvx_set_error("grid without its readback buffer");
    return GVX_ERR_STATE;
}

// sort the points by compact key in key space `ks` (positions + t), fill
// leaf_range for the leaves of `L` (whose key space must be ks)
// (octants below the leaf key when the key space leaves room for it: 28 bits of leaves)
static int sort_shift(const KeySpace& ks) { return ks.total_bits <= 28 ? 3 : 0; }

// the scratch of sort_points, its ranges to be zeroed before it
static gvx_status sort_points_scratch(gvx_grid* g, int n, const KeySpace& ks, ClearList& clear)
{
    return gvx_sort_prepare(g->sort, (uint32_t)n, ks.total_bits + sort_shift(ks) + 1, clear);
}

static gvx_status sort_points(gvx_grid* g, int n, const float t[3], const KeySpace& ks, bool bbox = false)
{
    GVX_CK(gvx_ensure(g->keys[0], (size_t)n * 4));
    GVX_CK(gvx_ensure(g->keys[1], (size_t)n * 4));
    GVX_CK(gvx_ensure(g->vals[0], (size_t)n * 4));
    GVX_CK(gvx_ensure(g->vals[1], (size_t)n * 4));
    const int kshift = sort_shift(ks);
    int lb = 0;
    while ((1 << lb) < g->brick) lb++;
    const uint32_t invalid_key = 1u << (ks.total_bits + kshift);
    const int bits = ks.total_bits + kshift + 1;
    const int passes = gvx_sort_passes(bits);
    // a block adds its digit counts up in L2: with a point or two a thread that cost as much as the keys
    // (400k points of a surface in 1216 blocks 13.6 us, in 390 6; 777k 12.8, in 759 8; 4M in 1216 23, in 304 33)
    const unsigned kb =
        std::min(blocks_for(n, 256), std::max(152u * 2u, std::min(blocks_for(n, 1024), 152u * 8u)));
    (bbox ? k_keys<true> : k_keys<false>)<<<kb, 256, 0, g->stream>>>(
        g->pts.pos, g->pts.pos_off, g->pts.pos_stride, (uint32_t)n, t[0], t[1], t[2], ks, 1.0f / (float)g->brick,
        kshift, lb, passes, invalid_key, g->keys[0].as<uint32_t>(), g->vals[0].as<uint32_t>(),
        gvx_sort_hist_ptr(g->sort), g->d_bbox.as<uint32_t>(), g->d_err.as<uint32_t>());
    g->launches++;
    uint32_t* kk[2] = {g->keys[0].as<uint32_t>(), g->keys[1].as<uint32_t>()};
    uint32_t* vv[2] = {g->vals[0].as<uint32_t>(), g->vals[1].as<uint32_t>()};
    int res = 0;
    gvx_status rc = gvx_sort_pairs(kk, vv, (uint32_t)n, bits, g->sort, true, g->stream, g->d_err.as<uint32_t>(), &res,
                                   &g->launches);
    if (rc) return rc;
    g->sorted_buf = res;
    g->full_group_gen = ~0ull;
    g->key_shift = kshift;
    g->n_sorted = (uint32_t)n;
    for (int a = 0; a < 3; a++) g->sort_trans[a] = t[a];
    g->perm_valid = false;
    g->oct_valid = false;
    return GVX_OK;
}

// the tables fill_leaf_ranges writes, their ranges to be zeroed before it
static gvx_status leaf_range_scratch(gvx_grid* g, uint32_t nleaves, ClearList& clear)
{
    GVX_CK(gvx_ensure(g->leaf_range, (size_t)(nleaves + 1) * sizeof(int2)));
    // (after the octants, and cleared with them: the dense numbers of the leaves)
    const size_t oct_words = (size_t)(nleaves + 1) * 9;
    GVX_CK(gvx_ensure(g->leaf_oct, oct_words * sizeof(int)));
    clear.add(g->leaf_range.p, (uint64_t)(nleaves + 1) * 2, 0u);
    clear.add(g->leaf_oct.p, oct_words, 0u);
    clear.add(g->d_counts.as<uint32_t>() + kCntDense, 1, 0u);
    return GVX_OK;
}

// the dense numbers of the leaves: in leaf_oct's buffer, after the octants of the nleaves its build made room
// for (null: that build orders no cells)
static int* dense_table(const gvx_grid* g, int kshift, uint32_t nleaves)
{
    return kshift && g->brick == 8 ? g->leaf_oct.as<int>() + (size_t)(nleaves + 1) * 8 : nullptr;
}

static void set_dense_table(gvx_grid* g, int* table)
{
    g->leaf_dense = table;
    g->dense_count = table ? g->d_counts.as<uint32_t>() + kCntDense : nullptr;
}

// (nl: the leaves' neighbours too, of that many)
static gvx_status fill_leaf_ranges(gvx_grid* g, uint32_t nleaves, const DevCount* nl = nullptr)
{
    uint32_t* dense_list = nullptr;
    set_dense_table(g, dense_table(g, g->key_shift, nleaves));
    g->dense_leaves = -1;
    if (g->leaf_dense) {
        const size_t most = g->n_sorted / kDenseLeaf + 1;
        GVX_CK(gvx_ensure(g->cell_tab, most * 513 * sizeof(int)));  // 512 cells a leaf, then the list of the leaves
        dense_list = g->cell_tab.as<uint32_t>() + most * 512;
    }
    const unsigned nb = nl ? blocks_for((uint64_t)nleaves * 27, 256) : 0u;
    if (g->n_sorted || nb) {
        k_leaf_tables<<<nb + blocks_for(g->n_sorted, 256), 256, 0, g->stream>>>(
            nb, g->leaf_key.as<uint32_t>(), nl ? *nl : dc_host(0), g->nbr.as<int>(),
            g->keys[g->sorted_buf].as<uint32_t>(), g->n_sorted, g->key_shift, 1u << g->lookup.ks.total_bits,
            g->lookup, g->leaf_range.as<int2>(), g->leaf_oct.as<int>(),
            dense_list, g->dense_count);
        g->launches++;
    }
    g->oct_leaves = nleaves;
    g->oct_valid = false;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

// the sorted point attributes (as k_permute writes them), one thread per sorted entry
__global__ void k_attr_permute(const uint32_t* __restrict__ svals, uint32_t n, const char* pos, int off, int stride,
                               float ox, float oy, float oz, GvxSortedAttr A)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < n;
    const uint32_t v = live ? svals[i] : 0u;
    float rr = 0.0f;
    if (live) {
        float w[3];
        load_pos(pos, off, stride, v, w);
        A.spos[i] = make_float4(w[0] + ox, w[1] + oy, w[2] + oz, A.weight ? A.weight[v] : 1.0f);
        if (A.radius) rr = A.radius[v];
        if (A.svel) {
            float4 q = make_float4(0.f, 0.f, 0.f, rr);
            if (A.vel) {
                const float* u = (const float*)(A.vel + (size_t)v * A.vel_stride + A.vel_off);
                q.x = u[0];
                q.y = u[1];
                q.z = u[2];
            }
            A.svel[i] = q;
        }
        rr = rr != rr ? 3.0e38f : fmaxf(rr, 0.0f);
    }
    if (A.rmax) {
        const unsigned int mm = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(rr));
        if ((threadIdx.x & 31) == 0 && mm && mm > *(volatile unsigned int*)A.rmax) atomicMax(A.rmax, mm);
    }
}

// Octant order inside every leaf, once per grouping, for the splats.  With the
// octants in the sort keys the sorted order is already (leaf key, octant,
// index) and fill_leaf_ranges has the octant starts: only the sorted attributes
// are written, one thread per entry.  Otherwise k_octant_partition partitions
// into the other value buffer (a copy of the sorted values, so entries outside
// the leaf ranges keep theirs), then copies back.
gvx_status gvx_topo_octants(gvx_grid* g, const GvxSortedAttr* attr)
{
    if (g->oct_valid) return GVX_OK;
    GvxSortedAttr none;
    memset(&none, 0, sizeof(none));
    const uint32_t nleaves = g->oct_leaves;
    if (g->key_shift) {
        if (g->leaf_dense && g->n_sorted >= (uint32_t)kDenseLeaf && g->dense_leaves != 0) {
            k_cell_sort<<<std::min(g->n_sorted / kDenseLeaf, 152u * 4u), kCellThreads, 0, g->stream>>>(
                g->cell_tab.as<uint32_t>() + ((size_t)g->n_sorted / kDenseLeaf + 1) * 512, g->dense_count, g->leaf_range.as<int2>(),
                g->nodes[0].as<GvxNode>(), g->keys[g->sorted_buf].as<uint32_t>(), g->pts.pos, g->pts.pos_off,
                g->pts.pos_stride, g->sort_trans[0], g->sort_trans[1], g->sort_trans[2],
                g->vals[g->sorted_buf].as<uint32_t>(), g->vals[1 - g->sorted_buf].as<uint32_t>(),
                g->cell_tab.as<int>(), g->leaf_dense);
            g->launches++;
            GVX_CK(cudaGetLastError());
        }
        if (g->n_sorted && attr && attr->spos) {
            k_attr_permute<<<blocks_for(g->n_sorted, 256), 256, 0, g->stream>>>(
                g->vals[g->sorted_buf].as<uint32_t>(), g->n_sorted, g->pts.pos, g->pts.pos_off, g->pts.pos_stride,
                g->sort_trans[0], g->sort_trans[1], g->sort_trans[2], *attr);
            g->launches++;
            GVX_CK(cudaGetLastError());
        }
    } else if (g->n_sorted && nleaves) {
        uint32_t* vin = g->vals[g->sorted_buf].as<uint32_t>();
        uint32_t* vtmp = g->vals[1 - g->sorted_buf].as<uint32_t>();
        const size_t vb = (size_t)g->n_sorted * sizeof(uint32_t);
        GVX_CK(cudaMemcpyAsync(vtmp, vin, vb, cudaMemcpyDeviceToDevice, g->stream));
        const DevCount nlc = g->oct_count.p ? g->oct_count : dc_host(nleaves);
        k_octant_partition<32><<<blocks_for((uint64_t)nleaves * 32u, 256), 256, 0, g->stream>>>(
            g->leaf_range.as<int2>(), nlc, g->nodes[0].as<GvxNode>(), g->pts.pos, g->pts.pos_off, g->pts.pos_stride,
            g->sort_trans[0], g->sort_trans[1], g->sort_trans[2], g->brick / 2, vin, vtmp, g->leaf_oct.as<int>(),
            attr ? *attr : none);
        g->launches++;
        GVX_CK(cudaMemcpyAsync(vin, vtmp, vb, cudaMemcpyDeviceToDevice, g->stream));
        GVX_CK(cudaGetLastError());
    }
    g->oct_valid = true;
    g->perm_valid = false;  // the sorted attributes follow the new order (the caller sets it when attr wrote them)
    return GVX_OK;
}

// k_mark_cells' per-axis limit: the key space's end or the root's (rootpos in voxels, the root's
// side in leaves), whichever comes first
static int3 dilate_limit(const KeySpace& ks, const int rootpos[3], int brick, int root_leaves)
{
    int l[3];
    for (int a = 0; a < 3; a++)
        l[a] = (int)std::min<int64_t>(int64_t(1) << ks.bits[a], (int64_t)rootpos[a] / brick + root_leaves - ks.lo[a]);
    return make_int3(l[0], l[1], l[2]);
}

// k_mark_cells over the sorted points (hi_mul 0: no boxes)
static void mark_cells(gvx_grid* g, int n, const float o[3], const KeySpace& ks, float radius, float hi_mul, int3 lim)
{
    (hi_mul > 0.f ? k_mark_cells<true> : k_mark_cells<false>)<<<blocks_for(n, 256), 256, 0, g->stream>>>(
        g->keys[g->sorted_buf].as<uint32_t>(), g->vals[g->sorted_buf].as<uint32_t>(), (uint32_t)n, g->key_shift,
        1u << ks.total_bits, g->pts.pos, g->pts.pos_off, g->pts.pos_stride, o[0], o[1], o[2], radius, hi_mul,
        g->logdim[0], ks, lim, g->d0_bits.as<uint32_t>(), g->x0_bits.as<uint32_t>(), g->d_err.as<uint32_t>());
    g->launches++;
}

static gvx_status grow_nodes(gvx_grid* g, int lev, int64_t cnt)
{
    GVX_CK(gvx_ensure(g->nodes[lev], (size_t)std::max<int64_t>(cnt, 1) * sizeof(GvxNode)));
    if (lev > 0) {
        const size_t vc = (size_t)g->res[lev] * g->res[lev] * g->res[lev];
        GVX_CK(gvx_ensure(g->clist[lev], (size_t)std::max<int64_t>(cnt, 1) * vc * sizeof(uint64_t)));
    }
    return GVX_OK;
}

// the child lists of levels 1..depth, cnt[l] nodes each, start empty
static void clear_clists(gvx_grid* g, int depth, const int64_t* cnt, ClearList& clear)
{
    for (int l = 1; l <= depth; l++)
        clear.add(g->clist[l].p, (uint64_t)cnt[l] * g->res[l] * g->res[l] * g->res[l] * 2u, 0xFFFFFFFFu);
}

// FULL rebuild: ActivateBricksGPU + ActivateExtraBricksGPU semantics
// A full build between its counts readback being queued and being read: what
// topo_full_complete needs of topo_full_launch.
struct FullBuild {
    int n;
    float radius;
    float o[3];
    int depth;
    int rootpos[3];
    KeySpace ks;
    uint32_t words0;
    UpperDesc ud;
    float mn[3], mx[3];  // the points' bounding box (GetBoundingBox before its margins)
};

// A staged RebuildTopology between its stages (gvx_topo_stage1..3), and the last full build of the
// grid (staged or not: what a plan is made from)
struct gvx_topo_staged {
    int n;
    float radius;
    int mode, min_depth;
    bool pending;
    FullBuild fb;
    bool last_full;     // the last full build (fb) finished, and the tree is still that one
    uint64_t last_gen;  // topo_gen after it
};

static gvx_status topo_full_scratch(gvx_grid* g, int n, int depth, const KeySpace& ks, FullBuild& fb, ClearList& clear);
static gvx_status topo_full_launch_ks(gvx_grid* g, int n, float radius, const float o[3], int depth,
                                      const int rootpos[3], const KeySpace& ks, FullBuild& fb, bool queue_readback,
                                      uint32_t* lists = nullptr, const uint32_t* list_cap = nullptr);

// the compact level-0 key space of a full build over the points' bounding box
// (+ dilation margin), inside the root
// (widen > 0: every axis's range grows by 1/widen of its length + 1 leaf on each side, inside
// the root -- the key space of a plan; hi_out: the last leaf coordinate of the range per axis)
static gvx_status full_key_space(gvx_grid* g, float radius, int depth, const int rootpos[3], const float mn[3],
                                 const float mx[3], KeySpace& ks, int widen = 0, int* hi_out = nullptr)
{
    const int b = g->brick;
    const int root_span = g->range[depth] / b;  // leaves per root side
    const int align = 1 << g->tshift[depth - 1];
    int64_t total_bits = 0;
    for (int a = 0; a < 3; a++) {
        const int rl = rootpos[a] / b;
        const float lo_v = mn[a] > 0.f ? mn[a] : 0.f;
        int lo = (int)floorf((lo_v - radius - 2.0f) / (float)b);
        int hi = mx[a] < 0.f ? rl : (int)floorf((mx[a] + 2.0f * radius + 2.0f) / (float)b);
        if (widen > 0 && hi >= lo) {
            const int m = (hi - lo + 1) / widen + 1;
            lo -= m;
            hi += m;
        }
        lo = std::max(lo, rl);
        hi = std::min(hi, rl + root_span - 1);
        if (hi < lo) hi = lo;
        lo = rl + ((lo - rl) / align) * align;
        ks.lo[a] = lo;
        ks.bits[a] = ceil_log2((int64_t)hi - lo + 1);
        if (hi_out) hi_out[a] = hi;
        total_bits += ks.bits[a];
    }
    if (total_bits > 30) {
        gvx_set_error("RebuildTopology: point extents span 2^%lld leaf cells; the compact key space holds 2^30",
                      (long long)total_bits);
        return GVX_ERR_UNSUPPORTED;
    }
    ks.total_bits = (int)total_bits;
    return GVX_OK;
}

// Everything of a full build (VG.cpp:1229-1413) up to the node counts, which are
// queued for the host; topo_full_complete reads them and writes the pools.
static gvx_status topo_full_launch(gvx_grid* g, int n, float radius, const float o[3], int depth,
                                   const int rootpos[3], const float mn[3], const float mx[3], FullBuild& fb)
{
    const int b = g->brick;
    if (radius >= 1.0f && radius > 0.5f * (float)(b - 1)) {
        gvx_set_error("RebuildTopology: radius %g exceeds (brick-1)/2 = %g (dilation beyond the 26 neighbours)",
                      radius, 0.5 * (b - 1));
        return GVX_ERR_UNSUPPORTED;
    }
    KeySpace ks;
    gvx_status rc = full_key_space(g, radius, depth, rootpos, mn, mx, ks);
    if (rc) return rc;
    for (int a = 0; a < 3; a++) {
        fb.mn[a] = mn[a];
        fb.mx[a] = mx[a];
    }
    ClearList clear;
    GVX_CK_STATUS(topo_full_scratch(g, n, depth, ks, fb, clear));
    GVX_CK_STATUS(gvx_clear(clear, g->stream, &g->launches));
    return topo_full_launch_ks(g, n, radius, o, depth, rootpos, ks, fb, true);
}

// the scratch of a full build in key space `ks` (fb.words0, fb.ud: its sizes), its ranges to be cleared
static gvx_status topo_full_scratch(gvx_grid* g, int n, int depth, const KeySpace& ks, FullBuild& fb, ClearList& clear)
{
    const uint32_t words0 = std::max<uint32_t>(1u, (uint32_t)((1ull << ks.total_bits) / 32ull));
    GVX_CK(gvx_ensure(g->d0_bits, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->d0_prefix, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->x0_bits, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->x0_prefix, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->leaf_key, (size_t)std::max(n, 1) * 4));
    UpperDesc ud;
    memset(&ud, 0, sizeof(ud));
    ud.nlev = depth - 1;
    uint32_t upper_words = 0;
    for (int l = 1; l <= ud.nlev; l++) {
        ud.tshift[l] = g->tshift[l];
        const int bl = ks_bits_at(ks, g->tshift[l]);
        ud.words[l] = std::max<uint32_t>(1u, (uint32_t)((1ull << bl) / 32ull));
        ud.off[l] = upper_words;
        upper_words += 4u * ud.words[l];
    }
    GVX_CK(gvx_ensure(g->upper, (size_t)std::max<uint32_t>(upper_words, 1u) * 4));
    clear.add(g->d0_bits.p, words0, 0u);
    clear.add(g->x0_bits.p, words0, 0u);
    clear.add(g->d_counts.p, 64, 0u);
    clear.add(g->upper.p, upper_words, 0u);
    fb.words0 = words0;
    fb.ud = ud;
    return sort_points_scratch(g, n, ks, clear);
}

// a full build in key space `ks` up to its node counts (d_counts), which are queued for the
// host when queue_readback (otherwise the bounding box is made too); its scratch (topo_full_scratch) is cleared.  lists (optional): room for the keys of
// X0 (list_cap[0]), then of D_l and X_l (list_cap[l] each) per upper level
static gvx_status topo_full_launch_ks(gvx_grid* g, int n, float radius, const float o[3], int depth,
                                      const int rootpos[3], const KeySpace& ks, FullBuild& fb, bool queue_readback,
                                      uint32_t* lists, const uint32_t* list_cap)
{
    cudaStream_t st = g->stream;
    const int b = g->brick;
    const bool extra = radius >= 1.0f;
    const uint32_t words0 = fb.words0;
    const UpperDesc& ud = fb.ud;

    // ---- one sort of the compact level-0 keys
    gvx_status rc = sort_points(g, n, o, ks, !queue_readback);
    if (rc) return rc;
    uint32_t* counts = g->d_counts.as<uint32_t>();

    // ---- D0: leaves holding points; A0: the dilation leaves with them (radius >= 1, VG.cpp:1207-1208)
    BitRank d0{g->d0_bits.as<uint32_t>(), g->d0_prefix.as<uint32_t>(), words0};
    BitRank x0{g->x0_bits.as<uint32_t>(), g->x0_prefix.as<uint32_t>(), words0};
    mark_cells(g, n, o, ks, radius, extra ? 2.0f : 0.0f, dilate_limit(ks, rootpos, b, g->range[depth] / b));

    // ---- upper levels: parents of D0 (direct) and of X0 (extra)
    if (ud.nlev > 0) {
        k_upper_bits<<<dim3(blocks_for(words0, 256), extra ? 2 : 1), 256, 0, st>>>(d0.bits, x0.bits, words0, ks, ud,
                                                                                   g->upper.as<uint32_t>());
        g->launches++;
    }
    // ---- ranks of D_l and X_l = A_l & ~D_l, and their counts; the keys too where the lists have their room
    PfxJobs ranks;
    ranks.add(d0.bits, d0.prefix, words0, counts + 0).list = g->leaf_key.as<uint32_t>();
    uint32_t* lp = lists;
    auto listed = [&](PfxJob& q, uint32_t cap) {
        if (!lists) return;
        q.list = lp;
        q.cap = cap;
        lp += cap;
    };
    PfxJob& xj = ranks.add(x0.bits, x0.prefix, words0, counts + 1);
    xj.minus = d0.bits;
    xj.store = x0.bits;
    listed(xj, list_cap ? list_cap[0] : 0u);
    for (int l = 1; l <= ud.nlev; l++) {
        uint32_t* base = g->upper.as<uint32_t>() + ud.off[l];
        const uint32_t w = ud.words[l];
        listed(ranks.add(base, base + 2u * w, w, counts + 2 + 2 * (l - 1)), list_cap ? list_cap[l] : 0u);
        PfxJob& x = ranks.add(base + w, base + 3u * w, w, counts + 3 + 2 * (l - 1));
        x.minus = base;
        x.store = base + w;
        listed(x, list_cap ? list_cap[l] : 0u);
    }
    rc = pfx_run<true>(ranks, g->tmp_scan, st, &g->launches);
    if (rc) return rc;
    GVX_CK(cudaGetLastError());

    // ---- counts to the host (the one mid-build synchronisation)
    fb.n = n;
    fb.radius = radius;
    fb.depth = depth;
    for (int a = 0; a < 3; a++) {
        fb.o[a] = o[a];
        fb.rootpos[a] = rootpos[a];
    }
    fb.ks = ks;
    return queue_readback ? readback_start(g) : GVX_OK;
}

// what a full build's level has from its key space
static void level_args(const gvx_grid* g, const FullBuild& fb, int l, NodeLevelArgs& a)
{
    memset(&a, 0, sizeof(a));
    a.lev = l;
    a.depth = fb.depth;
    a.ks = fb.ks;
    a.tshift = g->tshift[l];
    a.tshift_parent = g->tshift[l + 1];
    a.logdim_parent = g->logdim[l + 1];
    a.res_parent = g->res[l + 1];
    for (int k = 0; k < 3; k++) {
        a.lo[k] = fb.ks.lo[k] >> g->tshift[l];
        a.root_rel[k] = fb.rootpos[k] / g->range[l];
    }
    a.range = g->range[l];
    if (l + 1 < fb.depth) {
        uint32_t* base = g->upper.as<uint32_t>() + fb.ud.off[l + 1];
        const uint32_t w = fb.ud.words[l + 1];
        a.pd = BitRank{base, base + 2 * w, w};
        a.px = BitRank{base + w, base + 3 * w, w};
    }
    a.nodes = g->nodes[l].as<GvxNode>();
    a.pclist = g->clist[l + 1].as<uint64_t>();
    a.leaf_key = l == 0 ? g->leaf_key.as<uint32_t>() : nullptr;
}

// the nodes of all levels (most nodes a level) and the root
static void write_tree(gvx_grid* g, const FullBuild& fb, TreeArgs& t, uint32_t most)
{
    t.depth = fb.depth;
    for (int a = 0; a < 3; a++) t.rootpos[a] = fb.rootpos[a];
    t.root = g->nodes[fb.depth].as<GvxNode>();
    k_write_nodes<<<dim3(blocks_for(most, 256), (unsigned)fb.depth), 256, 0, g->stream>>>(t);
    g->launches++;
}

static gvx_status topo_full_complete(gvx_grid* g, const FullBuild& fb)
{
    cudaStream_t st = g->stream;
    const int n = fb.n, depth = fb.depth;
    const float* o = fb.o;
    const int* rootpos = fb.rootpos;
    const KeySpace ks = fb.ks;
    const uint32_t words0 = fb.words0;
    const UpperDesc& ud = fb.ud;
    const BitRank d0{g->d0_bits.as<uint32_t>(), g->d0_prefix.as<uint32_t>(), words0};
    const BitRank x0{g->x0_bits.as<uint32_t>(), g->x0_prefix.as<uint32_t>(), words0};
    uint32_t hc[64];
    gvx_status rc = readback_finish(g, hc, 0, sizeof(hc), "RebuildTopology");
    if (rc) return rc;
    const uint32_t U0 = hc[0], X0 = hc[1];
    uint32_t Ul[GVX_MAXLEV] = {}, Xl[GVX_MAXLEV] = {};
    Ul[0] = U0;
    Xl[0] = X0;
    for (int l = 1; l < depth; l++) {
        Ul[l] = hc[2 + 2 * (l - 1)];
        Xl[l] = hc[3 + 2 * (l - 1)];
    }

    // ---- pools and lists
    for (int l = 0; l < GVX_MAXLEV; l++) g->count[l] = 0;
    for (int l = 0; l < depth; l++) {
        rc = grow_nodes(g, l, (int64_t)Ul[l] + Xl[l]);
        if (rc) return rc;
        g->count[l] = (int64_t)Ul[l] + Xl[l];
    }
    rc = grow_nodes(g, depth, 1);
    if (rc) return rc;
    g->count[depth] = 1;
    const uint32_t L0 = U0 + X0;
    ClearList clear;
    clear_clists(g, depth, g->count, clear);
    GVX_CK_STATUS(leaf_range_scratch(g, L0, clear));
    GVX_CK_STATUS(gvx_clear(clear, st, &g->launches));
    size_t list_words = (size_t)X0 + 1;
    for (int l = 1; l < depth; l++) list_words += (size_t)Ul[l] + Xl[l];
    GVX_CK(gvx_ensure(g->lists, list_words * 4));
    uint32_t* x0list = g->lists.as<uint32_t>();
    PfxJobs sel;
    sel.add(x0.bits, x0.prefix, words0, nullptr).list = x0list;
    uint32_t* lp = x0list + X0 + 1;
    const uint32_t* dl[GVX_MAXLEV] = {};
    const uint32_t* xl[GVX_MAXLEV] = {};
    xl[0] = x0list;
    for (int l = 1; l < depth; l++) {
        uint32_t* base = g->upper.as<uint32_t>() + ud.off[l];
        const uint32_t w = ud.words[l];
        sel.add(base, base + 2 * w, w, nullptr).list = lp;
        dl[l] = lp;
        lp += Ul[l];
        sel.add(base + w, base + 3 * w, w, nullptr).list = lp;
        xl[l] = lp;
        lp += Xl[l];
    }
    // leaf keys in pool order: the D0 list of the first half, again (the buffer may have been replaced),
    // and X0's, which level 0's nodes append
    GVX_CK(gvx_ensure(g->leaf_key, (size_t)std::max<uint64_t>((uint64_t)U0 + X0, (uint64_t)n) * 4 + 4));
    sel.add(d0.bits, d0.prefix, words0, nullptr).list = g->leaf_key.as<uint32_t>();
    dl[0] = g->leaf_key.as<uint32_t>();
    GVX_CK_STATUS(select_run(sel, st, &g->launches));

    // ---- nodes, parents and child lists
    TreeArgs t;
    uint32_t most = 1u;
    for (int l = depth - 1; l >= 0; l--) {
        NodeLevelArgs& a = t.a[l];
        level_args(g, fb, l, a);
        a.ucount = Ul[l];
        a.xcount = Xl[l];
        a.dlist = dl[l];
        a.xlist = xl[l];
        a.pucount = l + 1 < depth ? Ul[l + 1] : 0u;
        most = std::max(most, Ul[l] + Xl[l]);
    }
    write_tree(g, fb, t, most);

    // ---- leaf lookup, neighbours, point ranges
    g->lookup.ks = ks;
    g->lookup.a = d0;
    g->lookup.b = x0;
    g->lookup.b_offset = U0;
    g->lookup.remap = nullptr;
    g->lookup.b_offset_p = nullptr;
    g->lookup.cap = 0;
    g->lookup_valid = true;
    GVX_CK(gvx_ensure(g->nbr, (size_t)std::max<uint32_t>(L0, 1u) * 27 * sizeof(int)));
    g->nbr_valid = true;
    const DevCount nl = dc_host(L0);
    rc = fill_leaf_ranges(g, L0, &nl);
    if (rc) return rc;
    g->group_valid = true;
    g->full_group_gen = g->topo_gen;
    g->group_pos = g->pts.pos;
    g->group_n = n;
    for (int a = 0; a < 3; a++) g->group_trans[a] = o[a];

    g->root_level = depth;
    for (int a = 0; a < 3; a++) g->root_pos[a] = rootpos[a];
    g->used_leaves = L0;
    g->atlas_valid = false;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

static gvx_status topo_full(gvx_grid* g, int n, float radius, const float o[3], int depth, const int rootpos[3],
                            const float mn[3], const float mx[3])
{
    FullBuild fb{};
    gvx_status rc = topo_full_launch(g, n, radius, o, depth, rootpos, mn, mx, fb);
    if (rc == GVX_OK) rc = topo_full_complete(g, fb);
    // recorded for a plan (gvx_topo_plan_make)
    if (!g->staged) g->staged = new gvx_topo_staged();
    g->staged->fb = fb;
    g->staged->last_full = rc == GVX_OK;
    g->staged->last_gen = g->topo_gen;
    return rc;
}

// slots of d_counts read back by the incremental build
enum { kCntNew = 0, kCntActive = 48 };

// grows a pool buffer keeping its first `keep` bytes (PoolAlloc "preserve
// existing on expand", VG.cpp:1096)
static gvx_status grow_keep(gvx_grid* g, DevBuf& b, size_t bytes, size_t keep)
{
    if (b.p && bytes <= b.cap) return GVX_OK;
    DevBuf nb;
    GVX_CK(gvx_ensure(nb, bytes));
    cudaError_t e = cudaSuccess;
    if (b.p && keep) e = cudaMemcpyAsync(nb.p, b.p, keep, cudaMemcpyDeviceToDevice, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    if (e != cudaSuccess) {
        gvx_free(nb);
        return gvx_cuda_fail(e, "pool growth");
    }
    gvx_free(b);
    b = nb;
    return GVX_OK;
}

// leaf lookup over the ACTIVE leaves in key space `ks` (bitmap + rank -> pool
// index), the per-leaf keys, the neighbour table and the point ranges of the
// grouping made in `ks`.  readback: kReadUsed = the active count becomes
// used_leaves (one synchronisation, with the device error word); kReadError =
// the device error word only; kReadNone = no synchronisation (the caller knows
// the active count; a device error stays in the word for the next readback)
enum { kReadNone = 0, kReadError = 1, kReadUsed = 2 };
static gvx_status build_active_lookup(gvx_grid* g, const KeySpace& ks, uint32_t words0, int readback)
{
    cudaStream_t st = g->stream;
    const uint32_t L0 = (uint32_t)g->count[0];
    GVX_CK(gvx_ensure(g->lk_bits, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->lk_prefix, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->remap, (size_t)L0 * 4 + 4));
    GVX_CK(gvx_ensure(g->leaf_key, (size_t)L0 * 4 + 4));
    ClearList clear;
    clear.add(g->lk_bits.p, words0, 0u);
    GVX_CK_STATUS(leaf_range_scratch(g, L0, clear));
    GVX_CK_STATUS(gvx_clear(clear, st, &g->launches));
    uint32_t* counts = g->d_counts.as<uint32_t>();
    const BitRank lk{g->lk_bits.as<uint32_t>(), g->lk_prefix.as<uint32_t>(), words0};
    NodeSets act;
    act.add(g->nodes[0].as<GvxNode>(), L0, 0, g->range[0], lk, g->remap.as<int>(), g->leaf_key.as<uint32_t>());
    if (L0) {
        k_node_bits<<<act.grid(), 256, 0, st>>>(act, ks, kSetActive, g->d_err.as<uint32_t>());
        g->launches++;
    }
    gvx_status rc = gvx_bitmap_prefix(g->lk_bits.as<uint32_t>(), g->lk_prefix.as<uint32_t>(), words0,
                                      counts + kCntActive, g->tmp_scan, st, &g->launches);
    if (rc) return rc;
    if (L0) {
        k_node_remap<<<act.grid(), 256, 0, st>>>(act, ks, kSetActive);
        g->launches++;
    }
    g->lookup.ks = ks;
    g->lookup.a = lk;
    g->lookup.b = BitRank{nullptr, nullptr, 0u};
    g->lookup.b_offset = 0u;
    g->lookup.remap = g->remap.as<int>();
    g->lookup.b_offset_p = nullptr;
    g->lookup.cap = 0;
    g->lookup_valid = true;
    GVX_CK(gvx_ensure(g->nbr, (size_t)std::max<uint32_t>(L0, 1u) * 27 * sizeof(int)));
    g->nbr_valid = true;
    const DevCount nl = dc_host(L0);
    rc = fill_leaf_ranges(g, L0, &nl);
    if (rc) return rc;
    if (readback == kReadUsed) {
        uint32_t used = 0;
        gvx_status rc = readback_checked(g, &used, kCntActive, 4, "RebuildTopology");
        if (rc) return rc;
        g->used_leaves = used;
        return GVX_OK;
    }
    if (readback == kReadNone) {
        GVX_CK(cudaGetLastError());
        return GVX_OK;
    }
    return gvx_check_device_error(g, "RebuildTopology");
}

// Incremental rebuild (ActivateIncreBricksGPU, VG.cpp:1020-1156) of the tree
// rooted at g->root_level over levels 0..depth-1; AccumulateTopology
// (VG.cpp:1158-1178) may pass a depth below the root's level.  act[6] is the
// box of the active leaves (voxels, max exclusive; empty when min > max).
static gvx_status topo_incremental(gvx_grid* g, int n, float radius, const float o[3], int depth, bool accum,
                                   const float mn[3], const float mx[3], const int act[6])
{
    cudaStream_t st = g->stream;
    const int b = g->brick, R = g->root_level;
    if (g->count[0] == 0) return GVX_OK;  // no leaf: the reference returns at once (VG.cpp:1022)
    if (radius > (float)(b - 1)) {
        gvx_set_error("RebuildTopology: incremental radius %g exceeds brick-1 = %d (box beyond the 26 neighbours)",
                      radius, b - 1);
        return GVX_ERR_UNSUPPORTED;
    }
    if (depth > R) {
        gvx_set_error("AccumulateTopology: points need %d levels, the tree's root is at level %d", depth + 1, R);
        return GVX_ERR_DEPTH;
    }
    const int top = depth < R ? depth : depth - 1;  // highest level whose linked set is needed
    uint32_t old[GVX_MAXLEV] = {};
    for (int l = 0; l <= R; l++) old[l] = (uint32_t)g->count[l];

    // ---- key space: the points' boxes and the active leaves, inside the root
    KeySpace ks;
    const int root_span = g->range[R] / b;
    const int align = 1 << g->tshift[top];
    int64_t total_bits = 0;
    for (int a = 0; a < 3; a++) {
        const int rl = g->root_pos[a] / b;
        const float lo_v = mn[a] > 0.f ? mn[a] : 0.f;
        int lo = (int)floorf((lo_v - radius - 2.0f) / (float)b);
        int hi = mx[a] < 0.f ? rl : (int)floorf((mx[a] + radius + 2.0f) / (float)b);
        if (act[a] < act[3 + a]) {
            lo = std::min(lo, act[a] / b);
            hi = std::max(hi, act[3 + a] / b - 1);
        }
        lo = std::max(lo, rl);
        hi = std::min(hi, rl + root_span - 1);
        if (hi < lo) hi = lo;
        lo = rl + ((lo - rl) / align) * align;
        ks.lo[a] = lo;
        ks.bits[a] = ceil_log2((int64_t)hi - lo + 1);
        total_bits += ks.bits[a];
    }
    if (total_bits > 30) {
        gvx_set_error("RebuildTopology: points and active bricks span 2^%lld leaf cells; the key space holds 2^30",
                      (long long)total_bits);
        return GVX_ERR_UNSUPPORTED;
    }
    ks.total_bits = (int)total_bits;
    const uint32_t words0 = std::max<uint32_t>(1u, (uint32_t)((1ull << total_bits) / 32ull));

    // ---- scratch: D0 / X0 (touched level-0 cells), L0 / N0 (linked / new), upper levels
    GVX_CK(gvx_ensure(g->d0_bits, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->d0_prefix, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->x0_bits, (size_t)words0 * 4));
    GVX_CK(gvx_ensure(g->inc0, (size_t)words0 * 16));
    ClearList clear;
    clear.add(g->d0_bits.p, words0, 0u);
    clear.add(g->x0_bits.p, words0, 0u);
    clear.add(g->inc0.p, (uint64_t)words0 * 4u, 0u);
    clear.add(g->d_counts.p, 64, 0u);
    // per upper level: D (touched via direct leaves), A (via box leaves), L bits, L prefix, N bits, N prefix
    UpperDesc ud;
    memset(&ud, 0, sizeof(ud));
    ud.nlev = depth - 1;
    uint32_t upper_words = 0;
    for (int l = 1; l <= top; l++) {
        ud.tshift[l] = g->tshift[l];
        ud.words[l] = std::max<uint32_t>(1u, (uint32_t)((1ull << ks_bits_at(ks, g->tshift[l])) / 32ull));
        ud.off[l] = upper_words;
        upper_words += 6u * ud.words[l];
    }
    GVX_CK(gvx_ensure(g->upper, (size_t)std::max<uint32_t>(upper_words, 1u) * 4));
    clear.add(g->upper.p, upper_words, 0u);
    GVX_CK_STATUS(sort_points_scratch(g, n, ks, clear));
    GVX_CK_STATUS(gvx_clear(clear, st, &g->launches));
    uint32_t* upper = g->upper.as<uint32_t>();
    uint32_t* counts = g->d_counts.as<uint32_t>();
    uint32_t* err = g->d_err.as<uint32_t>();

    // ---- touched cells: the points' leaves (D0) and their boxes [int(p)-r, int(p)+r] (X0), PT.cuh:420-465
    gvx_status rc = sort_points(g, n, o, ks);
    if (rc) return rc;
    const BitRank d0{g->d0_bits.as<uint32_t>(), nullptr, words0};
    mark_cells(g, n, o, ks, radius, radius > 0.f ? 1.0f : 0.0f, dilate_limit(ks, g->root_pos, b, g->range[R] / b));
    if (ud.nlev > 0) {
        k_upper_bits<<<dim3(blocks_for(words0, 256), radius > 0.f ? 2 : 1), 256, 0, st>>>(
            d0.bits, g->x0_bits.as<uint32_t>(), words0, ks, ud, upper);
        g->launches++;
    }

    // ---- linked sets L_l with rank -> pool index, levels 0..top
    size_t roff[GVX_MAXLEV] = {}, rtotal = 0;
    for (int l = 0; l <= top; l++) {
        roff[l] = rtotal;
        rtotal += old[l];
    }
    GVX_CK(gvx_ensure(g->inc_remap, rtotal * 4 + 4));
    BitRank Lb[GVX_MAXLEV] = {}, Nb[GVX_MAXLEV] = {};
    NodeSets linked;
    PfxJobs lranks;
    for (int l = 0; l <= top; l++) {
        uint32_t* base = l == 0 ? g->inc0.as<uint32_t>() : upper + ud.off[l] + 2u * ud.words[l];
        const uint32_t w = l == 0 ? words0 : ud.words[l];
        Lb[l] = BitRank{base, base + w, w};
        Nb[l] = BitRank{base + 2u * w, base + 3u * w, w};
        linked.add(g->nodes[l].as<GvxNode>(), old[l], g->tshift[l], g->range[l], Lb[l],
                   g->inc_remap.as<int>() + roff[l], nullptr);
        lranks.add(Lb[l].bits, Lb[l].prefix, w, nullptr);
    }
    if (linked.n) {
        k_node_bits<<<linked.grid(), 256, 0, st>>>(linked, ks, kSetLinked, err);
        g->launches++;
    }
    rc = pfx_run<true>(lranks, g->tmp_scan, st, &g->launches);
    if (rc) return rc;
    if (linked.n) {
        k_node_remap<<<linked.grid(), 256, 0, st>>>(linked, ks, kSetLinked);
        g->launches++;
    }
    // ---- new nodes N_l = T_l & ~L_l = (D_l | A_l) & ~L_l (touched by a point or by a point's box, and not
    // linked), levels 0..depth-1
    PfxJobs nranks;
    for (int l = 0; l < depth; l++) {
        PfxJob& q = nranks.add(l == 0 ? d0.bits : upper + ud.off[l], Nb[l].prefix, Nb[l].words, counts + kCntNew + l);
        q.plus = l == 0 ? g->x0_bits.as<uint32_t>() : upper + ud.off[l] + ud.words[l];
        q.minus = Lb[l].bits;
        q.store = Nb[l].bits;
    }
    rc = pfx_run<true>(nranks, g->tmp_scan, st, &g->launches);
    if (rc) return rc;
    GVX_CK(cudaGetLastError());

    // ---- new-node counts to the host
    uint32_t hc[64];
    rc = readback_checked(g, hc, 0, sizeof(hc), "RebuildTopology");
    if (rc) return rc;
    uint32_t nnew[GVX_MAXLEV] = {};
    uint64_t total_new = 0;
    for (int l = 0; l < depth; l++) {
        nnew[l] = hc[kCntNew + l];
        total_new += nnew[l];
    }
    g->group_valid = false;  // the grouping now follows `ks`
    if (total_new == 0) {
        // no new node: the reference returns before it applies the markers (VG.cpp:1066)
        rc = build_active_lookup(g, ks, words0, accum ? kReadNone : kReadError);
        if (rc) return rc;
        g->last_rebuild = 0;
    } else {
        k_apply_markers<<<blocks_for(old[0], 256), 256, 0, st>>>(g->nodes[0].as<GvxNode>(), old[0], ks, g->range[0],
                                                                 d0.bits, g->x0_bits.as<uint32_t>(), accum ? 1 : 0);
        g->launches++;
        // ---- pools grow, keeping their nodes and child lists; new lists start empty
        ClearList grown;
        for (int l = 0; l < depth; l++) {
            if (!nnew[l]) continue;
            const size_t cnt = (size_t)old[l] + nnew[l];
            rc = grow_keep(g, g->nodes[l], cnt * sizeof(GvxNode), (size_t)old[l] * sizeof(GvxNode));
            if (rc) return rc;
            if (l > 0) {
                const size_t vb = (size_t)g->res[l] * g->res[l] * g->res[l] * sizeof(uint64_t);
                rc = grow_keep(g, g->clist[l], cnt * vb, (size_t)old[l] * vb);
                if (rc) return rc;
                grown.add((char*)g->clist[l].p + (size_t)old[l] * vb, (uint64_t)nnew[l] * (vb / 4), 0xFFFFFFFFu);
            }
        }
        GVX_CK_STATUS(gvx_clear(grown, st, &g->launches));
        // ---- sorted keys of the new nodes
        GVX_CK(gvx_ensure(g->lists, (size_t)(total_new + 1) * 4));
        const uint32_t* nl[GVX_MAXLEV] = {};
        uint32_t* lp = g->lists.as<uint32_t>();
        PfxJobs sel;
        for (int l = 0; l < depth; l++) {
            if (!nnew[l]) continue;
            sel.add(Nb[l].bits, Nb[l].prefix, Nb[l].words, nullptr).list = lp;
            nl[l] = lp;
            lp += nnew[l];
        }
        GVX_CK_STATUS(select_run(sel, st, &g->launches));
        // ---- new nodes and their links (gvdbLinkBricks, VG.cpp:1121-1129)
        IncTreeArgs tree;
        unsigned nlev = 0;
        uint32_t most = 0u;
        for (int l = depth - 1; l >= 0; l--) {
            if (!nnew[l]) continue;
            IncNodeArgs& a = tree.a[nlev++];
            memset(&a, 0, sizeof(a));
            most = std::max(most, nnew[l]);
            a.lev = l;
            a.count = nnew[l];
            a.base = old[l];
            a.keys = nl[l];
            a.ks = ks;
            a.tshift = g->tshift[l];
            a.range = g->range[l];
            for (int k = 0; k < 3; k++) {
                a.lo[k] = ks.lo[k] >> g->tshift[l];
                a.root_rel[k] = g->root_pos[k] / g->range[l];
            }
            a.nodes = g->nodes[l].as<GvxNode>();
            a.parent_root = l + 1 == R;
            if (!a.parent_root) {
                a.pl = Lb[l + 1];
                a.premap = g->inc_remap.as<int>() + roff[l + 1];
                if (l + 1 < depth && nnew[l + 1]) a.pn = Nb[l + 1];
                a.pbase = old[l + 1];
            }
            a.logdim_parent = g->logdim[l + 1];
            a.res_parent = g->res[l + 1];
            a.tshift_parent = g->tshift[l + 1];
            a.pclist = g->clist[l + 1].as<uint64_t>();
            a.err = err;
        }
        k_inc_write_nodes<<<dim3(blocks_for(most, 256), nlev), 256, 0, st>>>(tree);
        g->launches++;
        for (int l = 0; l < depth; l++) g->count[l] = (int64_t)old[l] + nnew[l];
        // ---- delink, bottom-up (VG.cpp:1131-1140)
        const uint32_t L0 = (uint32_t)g->count[0];
        k_delink_leaves<<<blocks_for(L0, 256), 256, 0, st>>>(g->nodes[0].as<GvxNode>(), L0,
                                                             g->nodes[1].as<GvxNode>(), (uint32_t)g->count[1],
                                                             g->clist[1].as<uint64_t>(), g->res[1], g->range[0], err);
        g->launches++;
        for (int l = 1; l < depth; l++) {
            const uint32_t cnt = (uint32_t)g->count[l];
            const uint32_t vc = (uint32_t)(g->res[l] * g->res[l] * g->res[l]);
            k_delink_upper<<<blocks_for((uint64_t)cnt * 32u, 256), 256, 0, st>>>(
                g->nodes[l].as<GvxNode>(), cnt, g->clist[l].as<uint64_t>(), vc, g->nodes[l + 1].as<GvxNode>(),
                (uint32_t)g->count[l + 1], g->clist[l + 1].as<uint64_t>(), g->res[l + 1], g->range[l], err);
            g->launches++;
        }
        GVX_CK(cudaGetLastError());
        // accumulating, no leaf is delinked and a dead one stays dead (its parent reference is
        // gone, k_apply_markers): the active count grows by the new leaves, known on the host
        rc = build_active_lookup(g, ks, words0, accum ? kReadNone : kReadUsed);
        if (rc) return rc;
        if (accum) g->used_leaves += nnew[0];
        g->atlas_valid = false;
        g->last_rebuild = 2;
    }
    g->group_valid = true;
    g->group_pos = g->pts.pos;
    g->group_n = n;
    for (int a = 0; a < 3; a++) g->group_trans[a] = o[a];
    return GVX_OK;
}

// the incremental build checks its limits (UNSUPPORTED, DEPTH) before it
// touches anything; any later failure leaves no usable tree
static gvx_status incremental_status(gvx_grid* g, gvx_status rc)
{
    if (rc == GVX_OK) g->pools_appended = true;  // the pools kept their nodes, new ones appended
    if (rc == GVX_OK || rc == GVX_ERR_UNSUPPORTED || rc == GVX_ERR_DEPTH) return rc;
    g->rebuild_topo = true;
    g->root_level = -1;
    g->lookup_valid = false;
    g->group_valid = false;
    return rc;
}

// the grid's state after a full build: a failed one leaves no usable tree
static gvx_status full_status(gvx_grid* g, gvx_status rc)
{
    if (rc) {
        g->root_level = -1;
        g->lookup_valid = false;
        g->group_valid = false;
        return rc;
    }
    g->rebuild_topo = false;
    g->last_rebuild = 1;
    return GVX_OK;
}

// GetBoundingBox's box read back (hb[0..5], order-preserving float bits) -> the points' box
// (mn, mx), bbox_min/max with the reference's margins (VG.cpp:5452-5460), and DetermineDepth:
// the lowest level whose node covers posMin and posMax, and that node's position (depth -1: none)
static void bbox_depth(gvx_grid* g, const uint32_t* hb, float mn[3], float mx[3], int* depth, int rootpos[3])
{
    int pmin[3], pmax[3];
    for (int a = 0; a < 3; a++) {
        mn[a] = ord2f(hb[a]);
        mx[a] = ord2f(hb[3 + a]);
        float lo = mn[a] - 1.0f, hi = mx[a] + 2.0f;
        lo = 0 > lo ? 0 : lo;
        hi = 0 > hi ? 0 : hi;
        g->bbox_min[a] = lo;
        g->bbox_max[a] = hi;
        pmin[a] = (int)lo;
        pmax[a] = (int)hi;
    }
    *depth = -1;
    for (int l = 0; l < g->levels; l++) {
        const int r = g->range[l];
        if (pmin[0] / r == pmax[0] / r && pmin[1] / r == pmax[1] / r && pmin[2] / r == pmax[2] / r) {
            *depth = l;
            for (int a = 0; a < 3; a++) rootpos[a] = pmin[a] / r * r;
            break;
        }
    }
}

// the blocks of k_bbox (256 threads): a multiple of 3, since the packed path needs the thread count divisible
// by 3; four an SM, as their atomics on six words come one after the other (400k points: eight an SM 7.9 us,
// four 5.8; 4M: 20 and 19, two 28)
static unsigned bbox_blocks(int n) { return (std::min(blocks_for(n, 256), 152u * 4u) + 2u) / 3u * 3u; }

// RebuildTopology up to GetBoundingBox's readback, which is queued
static gvx_status rebuild_begin(gvx_grid* g, int n, float radius, const float orig[3], int mode)
{
    if (!g->configured) {
        gvx_set_error("RebuildTopology: Configure was not called");
        return GVX_ERR_NOT_CONFIGURED;
    }
    if (n <= 0 || n > g->pts.n || !g->pts.pos) {
        gvx_set_error("RebuildTopology: %d points requested, %d bound by SetPoints", n, g->pts.n);
        return GVX_ERR_INVALID_ARG;
    }
    if (!(radius >= 0.f)) {
        gvx_set_error("RebuildTopology: radius must be >= 0");
        return GVX_ERR_INVALID_ARG;
    }
    gvx_status rc = ensure_grid_scratch(g);
    if (rc) return rc;
    g->sc_valid = false;
    g->pools_appended = false;
    const float o[3] = {orig ? orig[0] : 0.f, orig ? orig[1] : 0.f, orig ? orig[2] : 0.f};
    cudaStream_t st = g->stream;
    // (the device error word is not cleared here: an error left by the unchecked tail of an
    // accumulating build is reported by this build's first readback)

    // ---- GetBoundingBox: one reduction
    ClearList clear;
    clear_bboxes(g, clear);
    GVX_CK_STATUS(gvx_clear(clear, st, &g->launches));
    const unsigned bb = bbox_blocks(n);
    k_bbox<<<bb, 256, 0, st>>>(g->pts.pos, g->pts.pos_off, g->pts.pos_stride, (uint32_t)n, o[0], o[1], o[2],
                               g->d_bbox.as<uint32_t>(), g->d_err.as<uint32_t>());
    g->launches++;
    // an incremental build also needs the box of the active leaves: same readback
    const bool maybe_incremental = g->root_level >= 0 && !g->rebuild_topo && mode != GVX_TOPO_FULL;
    int* act_dev = g->d_bbox.as<int>() + 8;
    if (maybe_incremental && g->count[0] > 0) {
        k_leaf_bounds<<<blocks_for(g->count[0], 256), 256, 0, st>>>(g->nodes[0].as<GvxNode>(),
                                                                     (uint32_t)g->count[0], g->range[0], act_dev);
        g->launches++;
    }
    return readback_start(g);
}

// the rest of RebuildTopology, from the bounding box (and active-leaf box) read
// back; a full build with `fb` stops after queueing its counts readback (*pending),
// for topo_full_complete
static gvx_status rebuild_after_bbox(gvx_grid* g, int n, float radius, const float orig[3], int mode, int min_depth,
                                     const uint32_t hb[14], FullBuild* fb, bool* pending)
{
    gvx_status rc = GVX_OK;
    const float o[3] = {orig ? orig[0] : 0.f, orig ? orig[1] : 0.f, orig ? orig[2] : 0.f};
    if (pending) *pending = false;
    float mn[3], mx[3];
    int depth = -1, rootpos[3] = {0, 0, 0};
    bbox_depth(g, hb, mn, mx, &depth, rootpos);
    int act[6];
    memcpy(act, hb + 8, sizeof(act));
    if (mode == GVX_TOPO_ACCUMULATE && !g->rebuild_topo) {
        // AccumulateTopology (VG.cpp:1158-1178): depth raised to min_depth, no depth-change check
        int d = depth;
        if (d >= 0 && d < min_depth) d = min_depth;
        if (d <= 0 || d >= g->levels) {
            gvx_set_error("AccumulateTopology: depth %d outside 1..%d", d, g->levels - 1);
            return GVX_ERR_DEPTH;
        }
        g->topo_gen++;
        return incremental_status(g, topo_incremental(g, n, radius, o, d, true, mn, mx, act));
    }
    if (depth <= 0) {
        gvx_set_error(depth == 0 ? "RebuildTopology: point extents smaller than 1 brick"
                                 : "RebuildTopology: point extents exceed the configured levels");
        return GVX_ERR_DEPTH;
    }
    if (depth >= g->levels) {
        gvx_set_error("RebuildTopology: point extents need %d levels, %d configured", depth + 1, g->levels);
        return GVX_ERR_DEPTH;
    }
    // ---- state machine of RebuildTopology (VG.cpp:1195-1217)
    if (mode == GVX_TOPO_FULL) g->rebuild_topo = true;
    if (!g->rebuild_topo && depth != g->curr_depth) {
        g->rebuild_topo = true;  // "Depth change in rebuild": Clear + full rebuild
        g->curr_depth = depth;
    }
    g->topo_gen++;  // the device tree changes (or is rebuilt) from here on
    if (!g->rebuild_topo) return incremental_status(g, topo_incremental(g, n, radius, o, depth, false, mn, mx, act));
    g->atlas_prefix = -1;  // the pools are rebuilt from scratch
    if (fb) {
        rc = topo_full_launch(g, n, radius, o, depth, rootpos, mn, mx, *fb);
        if (rc == GVX_OK) {
            *pending = true;
            return GVX_OK;
        }
    } else {
        rc = topo_full(g, n, radius, o, depth, rootpos, mn, mx);
    }
    return full_status(g, rc);
}


// Staged RebuildTopology for batches of grids (gvx_batch_topology): stage 1
// queues GetBoundingBox and its readback; stage 2, once the grid's stream has
// passed it, reads the box and queues a full build up to its node counts (any
// other kind of build runs to its end here); stage 3 reads the counts and
// finishes the full build.  The host waits on a grid only where its stream
// has had the time of the other grids' stages to get there.

gvx_status gvx_topo_stage1(gvx_grid* g, int n, float radius, int mode, int min_depth)
{
    if (!g->staged) g->staged = new gvx_topo_staged();
    gvx_topo_staged& S = *g->staged;
    S.n = n;
    S.radius = radius;
    S.mode = mode;
    S.min_depth = min_depth;
    S.pending = false;
    S.last_full = false;
    return rebuild_begin(g, n, radius, nullptr, mode);
}

gvx_status gvx_topo_stage2(gvx_grid* g)
{
    gvx_topo_staged& S = *g->staged;
    uint32_t hb[14];
    gvx_status rc = readback_finish(g, hb, kReadBbox, sizeof(hb), "GetBoundingBox");
    if (rc) return rc;
    return rebuild_after_bbox(g, S.n, S.radius, nullptr, S.mode, S.min_depth, hb, &S.fb, &S.pending);
}

gvx_status gvx_topo_stage3(gvx_grid* g)
{
    gvx_topo_staged& S = *g->staged;
    if (!S.pending) return GVX_OK;
    S.pending = false;
    gvx_status rc = full_status(g, topo_full_complete(g, S.fb));
    S.last_full = rc == GVX_OK;
    S.last_gen = g->topo_gen;
    return rc;
}

void gvx_topo_staged_free(gvx_grid* g)
{
    delete g->staged;
    g->staged = nullptr;
}

// ---------------------------------------------------------------------------
// Planned full builds, for batches of grids rebuilt every frame (gvx_batch_frame).
// A full build waits on the host twice: for the bounding box, from which the
// host takes the depth, the root and the compact key space, and for the node
// counts, which size the pools.  A plan fixes both from the grid's last full
// build: the key space (that build's, widened on every side by an eighth of its
// extent and a leaf), the depth and root, and every pool's capacity (its count + 25% + 64).
// A planned build then queues GetBoundingBox, the full RebuildTopology, UpdateAtlas
// and the octant/attribute pass of InsertPoints with no host wait and no
// allocation, so that a batch of them can be captured in one CUDA graph: its
// kernels take the counts from device memory (DevCount) and clamp every write to
// the capacities.  The counts, the bounding box and the device error word go to
// pinned memory at the end.  Once the stream has passed them, gvx_topo_plan_finish
// checks that the plan held: the frame's own DetermineDepth gives the plan's root,
// the frame's own key space lies inside the plan's, and every count fits its
// capacity.  Then the pools, lists and atlas are those of an unplanned build --
// the pool order is the order of the leaf coordinates (x, y, z lexicographic),
// the same in every key space that holds them -- and the host state is set as an
// unplanned build sets it.  Otherwise the planned build is void and the caller
// builds the grid again without a plan.

enum { kRecCounts = 0, kRecBbox = kReadBbox, kRecErr = kReadErr, kRecWords = kReadWords };

struct gvx_topo_plan {
    FullBuild fb;                      // key space, depth, root, points, radius (words0, ud after enqueue)
    uint32_t cap[GVX_MAXLEV] = {};     // node capacity of levels 0 .. depth-1
    uint32_t* rec = nullptr;           // pinned: counts, bounding box, error word of the last build
    int sorted_buf = 0;                // where the planned sort leaves the keys
    uint64_t id = 0;
    bool enqueued = false;
};

static std::atomic<uint64_t> g_plan_ids{0};

void gvx_topo_plan_free(gvx_grid* g)
{
    if (!g->plan) return;
    if (g->plan->rec) cudaFreeHost(g->plan->rec);
    delete g->plan;
    g->plan = nullptr;
}

// (a plan fixes sizes, not addresses: any points of the same count may be built under it)
bool gvx_topo_plan_ready(const gvx_grid* g)
{
    return g->plan && g->plan->id && g->pts.pos && g->pts.n == g->plan->fb.n;
}

uint64_t gvx_topo_plan_id(const gvx_grid* g) { return g->plan ? g->plan->id : 0; }

int* gvx_topo_plan_dense(const gvx_grid* g)
{
    return g->plan ? dense_table(g, sort_shift(g->plan->fb.ks), g->plan->cap[0]) : nullptr;
}

const uint32_t* gvx_topo_plan_slots(const gvx_grid* g, uint32_t* cap)
{
    *cap = g->plan ? g->plan->cap[0] : 0u;
    return g->d_counts.as<uint32_t>() + kCntSlots;
}

gvx_status gvx_topo_plan_make(gvx_grid* g)
{
    const gvx_topo_staged* S = g->staged;
    if (!S || !S->last_full || S->last_gen != g->topo_gen || g->root_level < 0 || !g->lookup_valid) {
        gvx_set_error("plan: the grid's tree is not the result of a staged full build");
        return GVX_ERR_STATE;
    }
    if (!g->plan) g->plan = new gvx_topo_plan();
    gvx_topo_plan& P = *g->plan;
    P.id = 0;
    P.enqueued = false;
    if (!P.rec) GVX_CK(cudaMallocHost(&P.rec, kRecWords * sizeof(uint32_t)));
    const FullBuild& last = S->fb;
    KeySpace ks;
    // the widened key space, unless it would hold more than 8x the build's cells
    if (full_key_space(g, last.radius, last.depth, last.rootpos, last.mn, last.mx, ks, 8) != GVX_OK ||
        ks.total_bits > last.ks.total_bits + 3)
        ks = last.ks;
    P.fb = last;
    P.fb.ks = ks;
    for (int l = 0; l < GVX_MAXLEV; l++) P.cap[l] = 0;
    for (int l = 0; l < last.depth; l++) {
        const uint64_t c = (uint64_t)g->count[l];
        const uint64_t cap = c + c / 4 + 64;
        if (cap >= (1ull << 31)) {
            gvx_set_error("plan: level %d holds %llu nodes", l, (unsigned long long)c);
            return GVX_ERR_CAPACITY;
        }
        P.cap[l] = (uint32_t)cap;
    }
    P.id = ++g_plan_ids;
    return GVX_OK;
}

// pools, child lists, leaf keys, lookup, neighbours and point ranges of a planned build (the
// part of topo_full_complete after the counts), every launch over the capacities
static gvx_status plan_pools(gvx_grid* g, const gvx_topo_plan& P, const FullBuild& fb)
{
    const int depth = fb.depth;
    const KeySpace ks = fb.ks;
    const uint32_t words0 = fb.words0;
    const uint32_t* dcnt = g->d_counts.as<uint32_t>();
    const uint32_t cap0 = P.cap[0];
    const BitRank d0{g->d0_bits.as<uint32_t>(), g->d0_prefix.as<uint32_t>(), words0};
    const BitRank x0{g->x0_bits.as<uint32_t>(), g->x0_prefix.as<uint32_t>(), words0};

    // ---- nodes, parents and child lists, counts from d_counts; the lists as topo_full_launch_ks wrote them
    TreeArgs t;
    uint32_t most = 1u;
    const uint32_t* lp = g->lists.as<uint32_t>();
    for (int l = 0; l < depth; l++) {
        NodeLevelArgs& a = t.a[l];
        level_args(g, fb, l, a);
        if (l > 0) {
            a.dlist = lp;
            lp += P.cap[l];
        } else {
            a.dlist = g->leaf_key.as<uint32_t>();  // the D0 list; level 0's nodes append X0 to it
        }
        a.xlist = lp;
        lp += P.cap[l];
        a.ci_pu = l + 1 < depth ? 2 + 2 * l : -1;
        a.pcap = l + 1 < depth ? P.cap[l + 1] : 0u;
        a.dc = dcnt;
        a.ci_u = l == 0 ? 0 : 2 + 2 * (l - 1);
        a.ci_x = a.ci_u + 1;
        a.cap = P.cap[l];
        most = std::max(most, P.cap[l]);
    }
    write_tree(g, fb, t, most);

    // ---- leaf lookup (X0 offset U0 from d_counts), neighbours, point ranges
    g->lookup.ks = ks;
    g->lookup.a = d0;
    g->lookup.b = x0;
    g->lookup.b_offset = 0u;
    g->lookup.remap = nullptr;
    g->lookup.b_offset_p = dcnt;
    g->lookup.cap = cap0;
    GVX_CK(gvx_ensure(g->nbr, (size_t)cap0 * 27 * sizeof(int)));
    const DevCount nl = dc_dev(dcnt, 0, 1, cap0);
    return fill_leaf_ranges(g, cap0, &nl);
}

// UpdateAtlas where every leaf of the pool is active: leaf i in slot i, the other slots free (atlas map -1)
static gvx_status atlas_all(gvx_grid* g, DevCount nl, int64_t slots, uint32_t* nslots)
{
    k_atlas_all<<<blocks_for((uint64_t)std::max<int64_t>(slots, 1), 256), 256, 0, g->stream>>>(
        g->nodes[0].as<GvxNode>(), nl, (uint32_t)slots, g->sub[0], g->sub[1], g->P, g->apron, g->leaf_slot.as<int>(),
        g->slot_leaf.as<int>(), g->amap.as<int4>(), nslots);
    g->launches++;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

// UpdateAtlas of a planned build: slots in pool order over the leaf capacity, the slot count
// to d_counts[kCntSlots]
static gvx_status plan_atlas(gvx_grid* g, const gvx_topo_plan& P)
{
    const uint32_t cap0 = P.cap[0];
    const DevCount nl = dc_dev(g->d_counts.as<uint32_t>(), 0, 1, cap0);
    GVX_CK_STATUS(gvx_grow_atlas(g, cap0));
    const int64_t slots = (int64_t)g->sub[0] * g->sub[1] * g->sub[2];
    GVX_CK(gvx_ensure(g->amap, (size_t)slots * sizeof(int4)));
    GVX_CK(gvx_ensure(g->leaf_slot, (size_t)cap0 * 4));
    GVX_CK(gvx_ensure(g->slot_leaf, (size_t)std::max<int64_t>(slots, 1) * 4));
    return atlas_all(g, nl, slots, g->d_counts.as<uint32_t>() + kCntSlots);  // a full build: every leaf is active
}

gvx_status gvx_topo_plan_enqueue(gvx_grid* g, const GvxSortedAttr* attr, bool frame)
{
    if (!gvx_topo_plan_ready(g)) {
        gvx_set_error("planned build: no plan for the grid's points");
        return GVX_ERR_STATE;
    }
    gvx_topo_plan& P = *g->plan;
    cudaStream_t st = g->stream;
    const int n = P.fb.n, depth = P.fb.depth;
    const uint32_t cap0 = P.cap[0];
    const float o[3] = {0.f, 0.f, 0.f};
    GVX_CK_STATUS(ensure_grid_scratch(g));
    P.enqueued = false;

    // ---- everything the build clears, sized by the capacities
    GVX_CK(gvx_ensure(g->leaf_key, ((size_t)std::max<uint32_t>(cap0, (uint32_t)n) + 1) * 4));
    FullBuild fb{};
    ClearList clear;
    clear_bboxes(g, clear);
    GVX_CK_STATUS(topo_full_scratch(g, n, depth, P.fb.ks, fb, clear));
    int64_t cap[GVX_MAXLEV] = {};
    for (int l = 0; l <= depth; l++) {
        cap[l] = l < depth ? P.cap[l] : 1;
        GVX_CK_STATUS(grow_nodes(g, l, cap[l]));
    }
    clear_clists(g, depth, cap, clear);
    GVX_CK_STATUS(leaf_range_scratch(g, cap0, clear));
    GVX_CK_STATUS(gvx_clear(clear, st, &g->launches));

    // ---- GetBoundingBox (read by gvx_topo_plan_finish) and the full build in the plan's key space, sized by
    // the capacities
    size_t list_words = cap0;  // X0's keys, then those of D_l and X_l per upper level
    for (int l = 1; l < depth; l++) list_words += 2 * (size_t)P.cap[l];
    GVX_CK(gvx_ensure(g->lists, list_words * 4 + 4));
    GVX_CK_STATUS(topo_full_launch_ks(g, n, P.fb.radius, o, depth, P.fb.rootpos, P.fb.ks, fb, false,
                                      g->lists.as<uint32_t>(), P.cap));
    P.fb.words0 = fb.words0;
    P.fb.ud = fb.ud;
    gvx_status rc = plan_pools(g, P, fb);
    if (rc == GVX_OK && frame) rc = plan_atlas(g, P);
    // ---- InsertPoints: octant order and the sorted attributes over the leaf capacity
    if (rc == GVX_OK && frame) {
        g->oct_count = dc_dev(g->d_counts.as<uint32_t>(), 0, 1, cap0);
        g->oct_valid = false;
        rc = gvx_topo_octants(g, attr);
    }
    // the kernels took the device counts by value: the host state goes back to host counts
    g->oct_count = DevCount{};
    g->lookup.b_offset_p = nullptr;
    g->lookup.cap = 0;
    g->lookup_valid = false;
    if (rc) return rc;
    // (with the error word; a frame records that again after its splat)
    GVX_CK(cudaMemcpyAsync(P.rec, g->d_counts.p, kReadWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    GVX_CK(cudaGetLastError());
    P.sorted_buf = g->sorted_buf;
    P.enqueued = true;
    return GVX_OK;
}

// a captured planned build queued again (its graph launched)
void gvx_topo_plan_replayed(gvx_grid* g)
{
    if (g->plan) g->plan->enqueued = true;
}

// the device error word into the plan's record, on `st` after the work that may set it (the
// caller's: after the splat of the frame)
gvx_status gvx_topo_plan_record_error(gvx_grid* g, cudaStream_t st)
{
    GVX_CK(cudaMemcpyAsync(g->plan->rec + kRecErr, g->d_err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    return GVX_OK;
}

// a void planned build: nothing of the grid's tree, atlas or grouping is usable
static void plan_void(gvx_grid* g)
{
    g->root_level = -1;
    g->rebuild_topo = true;
    g->lookup_valid = false;
    g->group_valid = false;
    g->nbr_valid = false;
    g->atlas_valid = false;
    g->atlas_prefix = -1;
    g->oct_valid = false;
    g->perm_valid = false;
    g->used_leaves = 0;
    for (int c = 0; c < GVX_MAXCH; c++) apron_invalidate(g->ch[c]);
}

gvx_status gvx_topo_plan_finish(gvx_grid* g, bool* held, bool frame)
{
    *held = false;
    if (!g->plan || !g->plan->enqueued) {
        gvx_set_error("planned build: nothing queued");
        return GVX_ERR_STATE;
    }
    gvx_topo_plan& P = *g->plan;
    P.enqueued = false;
    const uint32_t* rec = P.rec;
    const int depth = P.fb.depth;
    // as rebuild_begin / rebuild_after_bbox
    g->sc_valid = false;
    g->pools_appended = false;
    g->topo_gen++;
    g->atlas_gen++;
    gvx_status rc = report_device_error(g, rec[kRecErr], frame ? "BatchFrame" : "RebuildTopology");  // (clears it)
    if (rc) {
        plan_void(g);
        return rc;
    }
    // did the plan hold?
    float mn[3], mx[3];
    int fdepth = -1, rootpos[3] = {0, 0, 0};
    bbox_depth(g, rec + kRecBbox, mn, mx, &fdepth, rootpos);
    bool ok = fdepth == depth;
    for (int a = 0; a < 3; a++) ok = ok && rootpos[a] == P.fb.rootpos[a];
    if (ok) {
        KeySpace ks;
        int hi[3];
        if (full_key_space(g, P.fb.radius, depth, rootpos, mn, mx, ks, 0, hi) != GVX_OK) {
            ok = false;
        } else {
            for (int a = 0; a < 3; a++)
                ok = ok && ks.lo[a] >= P.fb.ks.lo[a] && (int64_t)hi[a] < (int64_t)P.fb.ks.lo[a] + (1ll << P.fb.ks.bits[a]);
        }
    }
    uint64_t cnt[GVX_MAXLEV] = {};
    for (int l = 0; l < depth && ok; l++) {
        const int ci = l == 0 ? 0 : 2 + 2 * (l - 1);
        cnt[l] = (uint64_t)rec[kRecCounts + ci] + rec[kRecCounts + ci + 1];
        ok = cnt[l] <= P.cap[l];
    }
    ok = ok && (!frame || rec[kRecCounts + kCntSlots] == cnt[0]);  // every leaf of a full build is active
    if (!ok) {
        plan_void(g);
        return GVX_OK;
    }
    // ---- the host state of a full build (topo_full_complete, full_status) ...
    const uint32_t U0 = rec[kRecCounts + 0];
    for (int l = 0; l < GVX_MAXLEV; l++) g->count[l] = 0;
    for (int l = 0; l < depth; l++) g->count[l] = (int64_t)cnt[l];
    g->count[depth] = 1;
    g->lookup.ks = P.fb.ks;
    g->lookup.a = BitRank{g->d0_bits.as<uint32_t>(), g->d0_prefix.as<uint32_t>(), P.fb.words0};
    g->lookup.b = BitRank{g->x0_bits.as<uint32_t>(), g->x0_prefix.as<uint32_t>(), P.fb.words0};
    g->lookup.b_offset = U0;
    g->lookup.remap = nullptr;
    g->lookup.b_offset_p = nullptr;
    g->lookup.cap = 0;
    g->lookup_valid = true;
    g->nbr_valid = true;
    g->sorted_buf = P.sorted_buf;
    g->n_sorted = (uint32_t)P.fb.n;
    // (a replayed graph ran none of the host code that sets these, and another grouping may have set them since)
    g->key_shift = sort_shift(P.fb.ks);
    set_dense_table(g, gvx_topo_plan_dense(g));
    for (int a = 0; a < 3; a++) {
        g->sort_trans[a] = 0.f;
        g->group_trans[a] = 0.f;
        g->root_pos[a] = P.fb.rootpos[a];
    }
    g->group_valid = true;
    g->full_group_gen = g->topo_gen;
    g->group_pos = g->pts.pos;
    g->group_n = P.fb.n;
    g->root_level = depth;
    g->used_leaves = (int64_t)cnt[0];
    g->rebuild_topo = false;
    g->last_rebuild = 1;
    g->oct_leaves = (uint32_t)cnt[0];
    g->perm_valid = false;
    g->dense_leaves = (int64_t)rec[kRecCounts + kCntDense];
    if (!frame) {  // the topology alone: UpdateAtlas and the octant pass are the caller's next calls
        g->atlas_valid = false;
        g->atlas_prefix = -1;
        g->oct_valid = false;
        *held = true;
        return GVX_OK;
    }
    // ... of UpdateAtlas (gvx_topo_update_atlas: every brick in a new slot) ...
    g->atlas_used = (int64_t)cnt[0];
    g->atlas_valid = true;
    for (int c = 0; c < GVX_MAXCH; c++) apron_invalidate(g->ch[c]);
    g->atlas_prefix = g->atlas_used;
    // ... and of the octant pass of InsertPoints (the attributes: the caller)
    g->oct_valid = true;
    *held = true;
    return GVX_OK;
}

// A full RebuildTopology under the plan of the grid's last full build (same point count and
// radius, no origin): the whole build queued at once and one host wait at its end, for the
// counts, the bounding box and the error word, instead of a wait for the bounding box and
// another for the counts.  *done false: the plan did not hold (or there is none), nothing of
// the grid's tree is left, and the caller builds without it.
static gvx_status rebuild_planned(gvx_grid* g, int n, float radius, const float orig[3], int mode, bool* done)
{
    *done = false;
    const bool no_orig = !orig || (orig[0] == 0.f && orig[1] == 0.f && orig[2] == 0.f);
    if (mode != GVX_TOPO_FULL || !no_orig || !g->configured || !gvx_topo_plan_ready(g) || n != g->plan->fb.n ||
        radius != g->plan->fb.radius)
        return GVX_OK;
    gvx_status rc = gvx_topo_plan_enqueue(g, nullptr, false);
    if (rc == GVX_OK) GVX_CK(cudaStreamSynchronize(g->stream));
    bool held = false;
    if (rc == GVX_OK) rc = gvx_topo_plan_finish(g, &held, false);
    if (rc) {
        plan_void(g);
        return rc;
    }
    *done = held;
    if (held) {
        g->staged->last_full = false;  // (the plan stays: it is not remade from its own builds)
        g->planned_builds++;
    }
    return GVX_OK;
}

gvx_status gvx_topo_rebuild(gvx_grid* g, int n, float radius, const float orig[3], int mode, int min_depth)
{
    bool done = false;
    gvx_status rc = rebuild_planned(g, n, radius, orig, mode, &done);
    if (rc || done) return rc;
    rc = rebuild_begin(g, n, radius, orig, mode);
    if (rc) return rc;
    uint32_t hb[14];
    rc = readback_finish(g, hb, kReadBbox, sizeof(hb), "GetBoundingBox");
    if (rc) return rc;
    rc = rebuild_after_bbox(g, n, radius, orig, mode, min_depth, hb, nullptr, nullptr);
    // a full build plans the next ones (any points of the same count and radius)
    if (rc == GVX_OK && mode == GVX_TOPO_FULL) (void)gvx_topo_plan_make(g);
    return rc;
}



// A tree given as node pools and child lists (LoadVBX, VG.cpp:507-686: Configure, PoolRead per level,
// FinishTopology).  The pools are taken as they are; the leaf lookup, leaf keys and neighbour table
// are derived from the level-0 pool as after a build, over a compact key space spanning the leaves;
// the next RebuildTopology is a full one (Clear, VG.cpp:2487-2503, sets mRebuildTopo).
gvx_status gvx_topo_import(gvx_grid* g, int root_level, const int64_t* counts, const GvxNode* const* nodes,
                           const uint64_t* const* clists)
{
    if (!g->configured) {
        gvx_set_error("topology import: Configure was not called");
        return GVX_ERR_NOT_CONFIGURED;
    }
    if (root_level < 1 || root_level >= g->levels || counts[root_level] < 1) {
        gvx_set_error("topology import: root level %d of a %d-level tree", root_level, g->levels);
        return GVX_ERR_INVALID_ARG;
    }
    gvx_status rc = ensure_grid_scratch(g);
    if (rc) return rc;
    cudaStream_t st = g->stream;
    const int b = g->brick, R = root_level;
    // ---- compact key space over the leaves, aligned as a build aligns it inside the root
    const GvxNode& root = nodes[R][0];
    KeySpace ks;
    const int root_span = g->range[R] / b;
    const int align = 1 << g->tshift[R - 1];
    int64_t total_bits = 0;
    for (int a = 0; a < 3; a++) {
        const int rl = root.pos[a] / b;
        int lo = rl + root_span - 1, hi = rl;
        for (int64_t i = 0; i < counts[0]; i++) {
            const int c = nodes[0][i].pos[a] / b;
            lo = std::min(lo, c);
            hi = std::max(hi, c);
        }
        lo = std::max(lo, rl);
        hi = std::min(hi, rl + root_span - 1);
        if (hi < lo) hi = lo;
        lo = rl + ((lo - rl) / align) * align;
        ks.lo[a] = lo;
        ks.bits[a] = ceil_log2((int64_t)hi - lo + 1);
        total_bits += ks.bits[a];
    }
    if (total_bits > 30) {
        gvx_set_error("topology import: the leaves span 2^%lld leaf cells; the compact key space holds 2^30",
                      (long long)total_bits);
        return GVX_ERR_UNSUPPORTED;
    }
    ks.total_bits = (int)total_bits;
    // ---- pools
    for (int l = 0; l < g->levels; l++) {
        const int64_t c = l <= R ? counts[l] : 0;
        g->count[l] = c;
        if (c == 0) continue;
        rc = grow_nodes(g, l, c);
        if (rc) return rc;
        GVX_CK(cudaMemcpyAsync(g->nodes[l].p, nodes[l], (size_t)c * sizeof(GvxNode), cudaMemcpyHostToDevice, st));
        if (l > 0) {
            const size_t vc = (size_t)g->res[l] * g->res[l] * g->res[l];
            GVX_CK(cudaMemcpyAsync(g->clist[l].p, clists[l], (size_t)c * vc * sizeof(uint64_t),
                                   cudaMemcpyHostToDevice, st));
        }
    }
    g->root_level = R;
    g->topo_gen++;
    g->pools_appended = false;
    g->atlas_prefix = -1;
    for (int a = 0; a < 3; a++) g->root_pos[a] = root.pos[a];
    g->rebuild_topo = true;
    g->last_rebuild = 1;
    g->n_sorted = 0;
    g->group_valid = false;
    g->perm_valid = false;
    g->sc_valid = false;
    g->atlas_valid = false;
    GVX_CK_STATUS(gvx_begin_errors(g));
    const uint32_t words0 = std::max<uint32_t>(1u, (uint32_t)((1ull << total_bits) / 32ull));
    return build_active_lookup(g, ks, words0, kReadUsed);
}

gvx_status gvx_topo_update_atlas(gvx_grid* g)
{
    if (g->root_level < 0) {
        gvx_set_error("UpdateAtlas: no topology");
        return GVX_ERR_STATE;
    }
    if (!g->have_atlas) {
        gvx_set_error("UpdateAtlas: no channel added");
        return GVX_ERR_STATE;
    }
    cudaStream_t st = g->stream;
    const int64_t used = g->used_leaves;
    // Slots go to the active leaves in pool order.  When the last UpdateAtlas gave every leaf
    // below atlas_prefix its own index as slot and the build since only appended leaves, all of
    // them active (AccumulateTopology), those leaves keep their slots and values: the aprons stay
    // copies except in the new bricks and around them.
    const int64_t from = g->pools_appended && g->atlas_prefix >= 0 && g->atlas_prefix <= used &&
                                 used == g->count[0]
                             ? g->atlas_prefix
                             : -1;
    gvx_status rc = gvx_grow_atlas(g, used);
    if (rc) return rc;
    const int64_t slots = (int64_t)g->sub[0] * g->sub[1] * g->sub[2];
    const uint32_t L0 = (uint32_t)g->count[0];
    const uint32_t fw = std::max<uint32_t>(1u, (L0 + 31u) / 32u);
    GVX_CK(gvx_ensure(g->amap, (size_t)slots * sizeof(int4)));
    GVX_CK(gvx_ensure(g->leaf_slot, (size_t)std::max<uint32_t>(L0, 1u) * 4));
    GVX_CK(gvx_ensure(g->slot_leaf, (size_t)std::max<int64_t>(slots, 1) * 4));
    if (used == g->count[0]) {
        GVX_CK_STATUS(atlas_all(g, dc_host(L0), slots, nullptr));
    } else {
        GVX_CK(gvx_ensure(g->bm_a, (size_t)fw * 4));
        GVX_CK(gvx_ensure(g->bm_a_prefix, (size_t)fw * 4));
        ClearList clear;
        clear.add(g->amap.p, (uint64_t)slots * 4u, 0xFFFFFFFFu);
        clear.add(g->bm_a.p, fw, 0u);
        GVX_CK_STATUS(gvx_clear(clear, st, &g->launches));
    }
    if (L0 && used != g->count[0]) {
        k_flag_bits<<<blocks_for(L0, 256), 256, 0, st>>>(g->nodes[0].as<GvxNode>(), dc_host(L0), g->bm_a.as<uint32_t>());
        g->launches++;
        rc = gvx_bitmap_prefix(g->bm_a.as<uint32_t>(), g->bm_a_prefix.as<uint32_t>(), fw, nullptr, g->tmp_scan, st,
                               &g->launches);
        if (rc) return rc;
        k_atlas_assign<<<blocks_for(L0, 256), 256, 0, st>>>(
            g->nodes[0].as<GvxNode>(), dc_host(L0), g->bm_a.as<uint32_t>(), g->bm_a_prefix.as<uint32_t>(), g->sub[0],
            g->sub[1], g->P, g->apron, g->leaf_slot.as<int>(), g->slot_leaf.as<int>(), g->amap.as<int4>());
        g->launches++;
    }
    GVX_CK(cudaGetLastError());
    g->atlas_used = used;
    g->atlas_valid = true;
    g->sc_valid = false;  // subcell indices follow the atlas slots
    for (int c = 0; c < GVX_MAXCH; c++) {
        GvxChannel& ch = g->ch[c];
        if (from < 0 || !(ch.apron_valid || ch.apron_partial_from >= 0)) {
            apron_invalidate(ch);  // bricks moved to new slots
        } else if (from < used) {
            ch.apron_partial_from = ch.apron_valid ? from : std::min(ch.apron_partial_from, from);
            ch.apron_valid = false;
        }
    }
    g->atlas_prefix = used == g->count[0] ? used : -1;
    g->atlas_gen++;
    return GVX_OK;
}

// ComputeBounds (VG.cpp:1792-1816) runs on the device: min and max both start
// at level-0 pool node 0's position whatever its flags (a delinked node 0
// still seeds them), then the active leaves lower the minimum to their
// positions and raise the maximum to position + range.  mVoxResMax (the
// largest max - min per axis since Configure) is kept on the device beside
// them.  The result is read when the host asks for it (gvx_get_info), so
// FinishTopology adds no synchronisation.  host_stage: ints [0..2] min,
// [3..5] max, [6..8] res max.
// One launch: the blocks lower and raise the accumulators (ints [10..15]), and the last of them to get there
// (counter [9]) writes the result and leaves accumulators and counter as it found them.
__global__ void k_compute_bounds(const GvxNode* __restrict__ nodes, uint32_t n, int range, int* out, int reset_res_max)
{
    leaf_bounds(nodes, n, range, out + 10);
    __shared__ bool s_last;
    if (threadIdx.x < 6) __threadfence();  // (the threads that hold the block's atomics)
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd((unsigned int*)out + 9, 1u) + 1u == gridDim.x;
    __syncthreads();
    if (!s_last || threadIdx.x >= 3) return;
    __threadfence();
    const int a = threadIdx.x;
    volatile int* acc = out + 10;
    int mn = n ? nodes[0].pos[a] : 0x7FFFFFFF, mx = n ? nodes[0].pos[a] : (int)0x80000000;
    mn = min(mn, acc[a]);
    mx = max(mx, acc[3 + a]);
    out[a] = mn;
    out[3 + a] = mx;
    const int rm = reset_res_max ? 0 : out[6 + a];
    out[6 + a] = n ? max(rm, mx - mn) : rm;
    acc[a] = 0x7FFFFFFF;
    acc[3 + a] = (int)0x80000000;
    if (a == 0) out[9] = 0;
}

gvx_status gvx_topo_compute_bounds(gvx_grid* g)
{
    if (g->root_level < 0) return GVX_OK;
    gvx_status rc = ensure_grid_scratch(g);
    if (rc) return rc;
    const uint32_t L0 = (uint32_t)g->count[0];
    if (!g->host_stage.p) {
        GVX_CK(gvx_ensure(g->host_stage, 64));
        ClearList clear;
        clear.add(g->host_stage.p, 10, 0u);
        clear.add(g->host_stage.as<int>() + 10, 3, 0x7FFFFFFFu);
        clear.add(g->host_stage.as<int>() + 13, 3, 0x80000000u);
        GVX_CK_STATUS(gvx_clear(clear, g->stream, &g->launches));
    }
    k_compute_bounds<<<blocks_for(std::max(L0, 1u), 256), 256, 0, g->stream>>>(
        g->nodes[0].as<GvxNode>(), L0, g->range[0], g->host_stage.as<int>(), g->vox_res_max_reset ? 1 : 0);
    g->launches++;
    g->vox_res_max_reset = false;
    GVX_CK(cudaGetLastError());
    g->bounds_pending = true;
    return GVX_OK;
}

gvx_status gvx_topo_read_bounds(gvx_grid* g)
{
    if (!g->bounds_pending) return GVX_OK;
    int hb[9];
    GVX_CK(cudaMemcpyAsync(hb, g->host_stage.p, sizeof(hb), cudaMemcpyDeviceToHost, g->stream));
    GVX_CK(cudaStreamSynchronize(g->stream));
    const bool any = g->count[0] > 0;
    for (int a = 0; a < 3; a++) {
        g->obj_min[a] = any ? (float)hb[a] : 0.f;
        g->obj_max[a] = any ? (float)hb[3 + a] : 0.f;
        g->vox_res_max[a] = (float)hb[6 + a];
    }
    g->bounds_pending = false;
    return GVX_OK;
}

// InsertPoints: group the points by leaf for positions + trans, reusing the
// grouping of the topology build when it was made from the same points
gvx_status gvx_topo_group_points(gvx_grid* g, int n, const float trans[3])
{
    if (!g->lookup_valid) {
        gvx_set_error("InsertPoints: no topology");
        return GVX_ERR_STATE;
    }
    if (n <= 0 || n > g->pts.n || !g->pts.pos) {
        gvx_set_error("InsertPoints: %d points requested, %d bound", n, g->pts.n);
        return GVX_ERR_INVALID_ARG;
    }
    const float t[3] = {trans ? trans[0] : 0.f, trans ? trans[1] : 0.f, trans ? trans[2] : 0.f};
    if (g->group_valid && g->group_pos == g->pts.pos && g->group_n == n && t[0] == g->group_trans[0] &&
        t[1] == g->group_trans[1] && t[2] == g->group_trans[2])
        return GVX_OK;
    gvx_status rc = ensure_grid_scratch(g);
    if (rc) return rc;
    ClearList clear;
    GVX_CK_STATUS(sort_points_scratch(g, n, g->lookup.ks, clear));
    GVX_CK_STATUS(leaf_range_scratch(g, (uint32_t)g->count[0], clear));
    GVX_CK_STATUS(gvx_clear(clear, g->stream, &g->launches));
    rc = sort_points(g, n, t, g->lookup.ks);
    if (rc) return rc;
    rc = fill_leaf_ranges(g, (uint32_t)g->count[0]);
    if (rc) return rc;
    g->group_valid = true;
    g->group_pos = g->pts.pos;
    g->group_n = n;
    for (int a = 0; a < 3; a++) g->group_trans[a] = t[a];
    return GVX_OK;
}
