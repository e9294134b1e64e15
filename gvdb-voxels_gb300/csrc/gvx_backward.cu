// gvx_backward.cu -- adjoint of the TRILINEAR / CUBIC density splat (no
// reference counterpart).
//
// Forward (gvx_splat.cu): rho_v = sum_i w_i W(v - p_i; R_i) over the interior
// voxels v of the active bricks, W the CIC weight or the M4 cubic spline
// norm(h) M4(|v - p| / h), norm = 1 / (pi h^3), h = R / 2, support R.
// Backward: with G_v = dL/drho_v,
//   dL/dw_i = sum_v G_v W
//   dL/dp_i = sum_v G_v w_i dW/dp
//   dL/dR_i = sum_v G_v w_i dW/dR,   dW/dR = -(3 M4 + q M4') / (2 pi h^4)
// gathered per point, one warp per point over its support, in the sorted
// order of the forward's grouping (re-keyed and re-sorted when the points
// changed), reduced by a fixed butterfly: deterministic, no atomics.  Only
// interior voxels are read: an apron voxel is a copy of its owner's interior.
#include <math.h>

#include "gvx_grid.cuh"

namespace {

constexpr float kInvPi = 0.318309886183790671538f;
constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kBackThreads = 256;

inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

struct BackArgs {
    int brick, lb, P, apron;  // lb = log2(brick)
    bool ppr;
    float radius;
    uint32_t n;               // sorted points
    const uint32_t* skeys;    // compact level-0 keys, sorted
    const uint32_t* svals;    // sorted -> original point index
    int kshift;               // the sort keys are leaf key << kshift | octant
    uint32_t invalid_key;
    const float4* spos;       // (x, y, z, w), sorted
    const float4* svel;       // (., ., ., R), sorted (per-point radius) or null
    LeafLookup L;
    const int* nbr;           // 27 neighbours of every leaf
    const int* leaf_slot;
    const float* G;           // dL/drho, density channel layout
    float* gpos;              // 3 per original point
    float* gw;
    float* gr;                // or null
    uint32_t* err;
    uint32_t* next;           // point counter (zeroed before the launch)
};

}  // namespace

// sums of four values over the warp: lane 0 gets a, lane 8 b, lane 16 c, lane 24 d -- halves of the
// warp exchange what the other half sums, so that ten shuffles do what four butterflies take twenty for
__device__ __forceinline__ float sum4(float a, float b, float c, float d, int lane)
{
    const bool hi = lane & 16, hi8 = lane & 8;
    float x = (hi ? c : a) + __shfl_xor_sync(kFull, hi ? a : c, 16);
    const float y = (hi ? d : b) + __shfl_xor_sync(kFull, hi ? b : d, 16);
    x = (hi8 ? y : x) + __shfl_xor_sync(kFull, hi8 ? x : y, 8);
    for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    return x;
}

// One warp per point.  What bounds it: instruction issue (650 warp instructions a point of radius 1-3,
// 77% of the issue slots), and, one point a claim, the counter, whose one address takes an atomic every
// one to two nanoseconds.  So points are claimed kBackClaim at a time; they are neighbours in the sorted
// order, and most lie in the brick of the last one, whose 27 neighbours' slots the lanes keep; a cell's
// place in the support needs no division; dL/drho is asked for before the distances are formed.
// A million points of radii 1-3: 1.07 -> 0.68 ms.
// Of few points a warp takes fewer at a time, and none ahead of the one it works on, so that all warps have some
// (2000 points of R 6.5: claims of eight 213 us, one by one 40).
constexpr uint32_t kBackClaim = 8;
template <int MODE>
__global__ void __launch_bounds__(kBackThreads) k_splat_backward(BackArgs a)
{
    const int lane = threadIdx.x & 31;
    const int P = a.P, P3 = P * P * P, ap = a.apron, b = a.brick, lb = a.lb;
    // ceil(2^32 / n): c / n == umulhi(c, s_recip[n]) for n > 1, c < 2^32 / n (supports of up to 126
    // voxels a side: R < brick <= 64)
    __shared__ uint32_t s_recip[129];
    for (uint32_t n = threadIdx.x + 1; n <= 128u; n += blockDim.x) s_recip[n] = 0xFFFFFFFFu / n + 1u;
    __syncthreads();
    const uint32_t warps = gridDim.x * (kBackThreads / 32);
    const uint32_t claim = min(max(a.n / (3u * warps), 1u), kBackClaim);
    const bool ahead = a.n >= 4u * warps;
    uint32_t cur = 0u, lim = 0u, pre = ahead && lane == 0 ? atomicAdd(a.next, claim) : 0u;
    uint32_t brick_key = 0xFFFFFFFFu;  // the leaf that own, myslot and bx, by, bz are of
    int own = -1, myslot = -1, bx = 0, by = 0, bz = 0;
    for (;;) {
        if (cur == lim) {
            if (!ahead && lane == 0) pre = atomicAdd(a.next, claim);
            cur = __shfl_sync(0xFFFFFFFFu, pre, 0);
            lim = min(cur + claim, a.n);
            if (cur >= a.n) break;
            if (ahead && lane == 0) pre = atomicAdd(a.next, claim);
        }
        const uint32_t i = cur++;
        const uint32_t key = a.skeys[i] >> a.kshift;
        const uint32_t orig = a.svals[i];
        if (key != brick_key) {
            // the point takes part iff its own brick is in the lookup (as in the forward); lane k < 27 keeps
            // the atlas slot of neighbour k (-1 if none)
            brick_key = key;
            own = myslot = -1;
            if (key < a.invalid_key) {
                int c[3];
                ks_unpack(a.L.ks, key, 0, c);
                own = ll_find(a.L, c[0], c[1], c[2]);
                bx = c[0] + a.L.ks.lo[0];
                by = c[1] + a.L.ks.lo[1];
                bz = c[2] + a.L.ks.lo[2];
                if (own >= 0 && lane < 27) {
                    const int leaf = a.nbr[(size_t)own * 27 + lane];
                    myslot = leaf >= 0 ? a.leaf_slot[leaf] : -1;
                }
            }
        }
        float gx = 0.f, gy = 0.f, gz = 0.f, gwv = 0.f, grv = 0.f;
        if (own >= 0) {
            const float4 p = a.spos[i];
            const float R = a.ppr ? a.svel[i].w : a.radius;
            if (MODE == GVX_SPLAT_CUBIC && R > (float)(b - 1)) {
                if (lane == 0) atomicOr(a.err, GVX_DERR_RADIUS);
            }
            // a point that has left the brick of its key (written in place since the grouping): the bricks
            // around where it is, found one by one, for this point alone
            const int qx = (int)floorf(p.x) >> lb, qy = (int)floorf(p.y) >> lb, qz = (int)floorf(p.z) >> lb;
            if (((qx ^ bx) | (qy ^ by) | (qz ^ bz)) != 0) {
                bx = qx;
                by = qy;
                bz = qz;
                const int leaf = lane < 27 ? ll_find(a.L, bx + lane % 3 - 1 - a.L.ks.lo[0],
                                                     by + lane / 3 % 3 - 1 - a.L.ks.lo[1], bz + lane / 9 - 1 - a.L.ks.lo[2])
                                           : -1;
                myslot = leaf >= 0 ? a.leaf_slot[leaf] : -1;
                brick_key = 0xFFFFFFFFu;
            }
            // support box (world voxels), in the point's brick and its neighbours
            int lo[3], hi[3];
            const float pc[3] = {p.x, p.y, p.z};
            const int corner[3] = {bx, by, bz};
            for (int k = 0; k < 3; k++) {
                if (MODE == GVX_SPLAT_CUBIC) {
                    lo[k] = (int)floorf(pc[k] - R) + 1;
                    hi[k] = (int)ceilf(pc[k] + R) - 1;
                } else {
                    lo[k] = (int)floorf(pc[k]);
                    hi[k] = lo[k] + 1;
                }
                lo[k] = max(lo[k], max(0, (corner[k] - 1) << lb));
                hi[k] = min(hi[k], ((corner[k] + 2) << lb) - 1);
            }
            const int nx = hi[0] - lo[0] + 1, ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1;
            const int ncell = (nx > 0 && ny > 0 && nz > 0) ? nx * ny * nz : 0;
            const uint32_t mx = s_recip[min(max(nx, 1), 128)], my = s_recip[min(max(ny, 1), 128)];
            float h = 0.f, inv_h = 0.f, norm = 0.f, r2h = 0.f, r2l = 0.f;
            if (MODE == GVX_SPLAT_CUBIC) {
                h = 0.5f * R;
                inv_h = 1.0f / h;
                norm = kInvPi * inv_h * inv_h * inv_h;
                r2h = R * R;
                r2l = fmaf(R, R, -r2h);
            }
            const float fx0 = floorf(p.x), fy0 = floorf(p.y), fz0 = floorf(p.z);
            for (int c0 = 0; c0 < ncell; c0 += 32) {
                const int c = c0 + lane;
                const uint32_t cc = c < ncell ? (uint32_t)c : 0u;
                const uint32_t r = nx > 1 ? __umulhi(cc, mx) : cc, z = ny > 1 ? __umulhi(r, my) : r;
                const int vx = lo[0] + (int)(cc - r * nx), vy = lo[1] + (int)(r - z * ny), vz = lo[2] + (int)z;
                const int kb = ((vz >> lb) - bz + 1) * 9 + ((vy >> lb) - by + 1) * 3 + (vx >> lb) - bx + 1;
                const int slot = __shfl_sync(kFull, myslot, kb & 31);
                // (G arrives while the distances are formed)
                const int lx = vx & (b - 1), ly = vy & (b - 1), lz = vz & (b - 1);
                const bool there = c < ncell && slot >= 0;
                const float Gv = there ? a.G[(size_t)slot * P3 + (uint32_t)(((lz + ap) * P + (ly + ap)) * P + (lx + ap))] : 0.0f;
                const float dx = (float)vx - p.x, dy = (float)vy - p.y, dz = (float)vz - p.z;
                if (MODE == GVX_SPLAT_TRILINEAR) {
                    if (Gv == 0.0f) continue;
                    const float fx = p.x - fx0, fy = p.y - fy0, fz = p.z - fz0;
                    const bool ux = (float)vx == fx0, uy = (float)vy == fy0, uz = (float)vz == fz0;
                    const float wx = ux ? 1.f - fx : fx, wy = uy ? 1.f - fy : fy, wz = uz ? 1.f - fz : fz;
                    const float gwx = Gv * p.w;
                    gwv += Gv * wx * wy * wz;
                    gx += gwx * (ux ? -1.f : 1.f) * wy * wz;
                    gy += gwx * wx * (uy ? -1.f : 1.f) * wz;
                    gz += gwx * wx * wy * (uz ? -1.f : 1.f);
                } else {
                    // R^2 - d^2 error-free, as in the forward
                    const float qy = dy * dy, ey = fmaf(dy, dy, -qy);
                    const float qz = dz * dz, ez = fmaf(dz, dz, -qz);
                    const float syz = qy + qz;
                    float bv = syz - qy;
                    const float e1 = (qy - (syz - bv)) + (qz - bv);
                    const float c1 = r2h - syz;
                    bv = c1 - r2h;
                    const float e2 = (r2h - (c1 - bv)) + (-syz - bv);
                    const float cl = e2 + r2l - ((ey + ez) + e1);
                    const float t = fmaf(-dx, dx, c1) + cl;  // R^2 - d^2
                    if (!there || t <= 0.0f) continue;
                    const float d = sqrtf(fmaf(dx, dx, syz));
                    const float q = d * inv_h;
                    float m4, dm_over_hd, qdm;  // M4(q), M4'(q) / (h d), q M4'(q)
                    if (q < 1.0f) {
                        m4 = fmaf(q * q, fmaf(0.75f, q, -1.5f), 1.0f);
                        const float dm_over_q = fmaf(2.25f, q, -3.0f);  // M4'(q) / q
                        dm_over_hd = dm_over_q * inv_h * inv_h;
                        qdm = dm_over_q * q * q;
                    } else {
                        const float uu = t / (h * (R + d));  // 2 - q
                        m4 = 0.25f * uu * uu * uu;
                        const float dm = -0.75f * uu * uu;
                        dm_over_hd = dm / (h * d);
                        qdm = q * dm;
                    }
                    if (Gv == 0.0f) continue;
                    const float gnw = Gv * norm;
                    gwv += gnw * m4;
                    // dW/dp = norm M4'(q) / (h d) (p - v)
                    const float s = gnw * p.w * dm_over_hd;
                    gx -= s * dx;
                    gy -= s * dy;
                    gz -= s * dz;
                    // dW/dR = -(3 M4 + q M4') / (2 pi h^4) = -norm (3 M4 + q M4') / (2 h)
                    grv -= gnw * p.w * (3.0f * m4 + qdm) * (0.5f * inv_h);
                }
            }
        }
        // a fixed tree: the same sum order on every run
        const float g4 = sum4(gx, gy, gz, gwv, lane);
        if (a.gr) {
            for (int o = 16; o > 0; o >>= 1) grv += __shfl_xor_sync(kFull, grv, o);
            if (lane == 1) a.gr[orig] = grv;
        }
        if ((lane & 7) == 0) {
            if (lane == 24)
                a.gw[orig] = g4;
            else  // lanes 0, 8, 16
                a.gpos[(size_t)orig * 3 + (lane >> 3)] = g4;
        }
    }
}

extern "C" gvx_status gvx_splat_backward_ex(gvx_grid* g, int mode, int n, float radius, const float trans[3],
                                            const float* dL_drho, float* grad_pos, float* grad_w, float* grad_r,
                                            int flags)
{
    if (!g) {
        gvx_set_error("null grid handle");
        return GVX_ERR_INVALID_ARG;
    }
    GVX_CK(cudaSetDevice(g->device));
    if (g->root_level < 0 || !g->lookup_valid || !g->atlas_valid || !g->nbr_valid) {
        gvx_set_error("SplatBackward: no topology / atlas");
        return GVX_ERR_STATE;
    }
    if (mode != GVX_SPLAT_TRILINEAR && mode != GVX_SPLAT_CUBIC) {
        gvx_set_error("SplatBackward: mode %d has no adjoint", mode);
        return GVX_ERR_INVALID_ARG;
    }
    if (!dL_drho || !grad_pos || !grad_w) {
        gvx_set_error("SplatBackward: dL_drho, grad_pos and grad_w are required");
        return GVX_ERR_INVALID_ARG;
    }
    const bool ppr = mode == GVX_SPLAT_CUBIC && g->pts.radius != nullptr;
    if (mode == GVX_SPLAT_CUBIC && !ppr && !(radius > 0.f && radius <= (float)(g->brick - 1))) {
        gvx_set_error("SplatBackward: cubic radius %g outside (0, brick-1]", radius);
        return GVX_ERR_INVALID_ARG;
    }
    GVX_CK(gvx_ensure(g->d_next, sizeof(uint32_t)));
    GVX_CK_STATUS(gvx_begin_errors(g, g->d_next.as<uint32_t>()));
    // the grouping of the forward: reused when valid, else re-keyed and re-sorted.
    // GVX_BWD_RECOMPUTE drops it first, so the permutation is recomputed from the
    // positions (keys with their octants, radix sort, the sorted attributes)
    // rather than taken from the forward; the sort is deterministic, so the new
    // grouping equals the forward's and the gradients are the same bit for bit.
    if (flags & GVX_BWD_RECOMPUTE) {
        g->group_valid = false;
        g->oct_valid = false;
        g->perm_valid = false;
    }
    gvx_status rc = gvx_prepare_points(g, n, trans, ppr);
    if (rc) return rc;
    BackArgs a;
    a.brick = g->brick;
    a.lb = 0;
    while ((1 << a.lb) < g->brick) a.lb++;
    a.P = g->P;
    a.apron = g->apron;
    a.ppr = ppr;
    a.radius = radius;
    a.n = g->n_sorted;
    a.skeys = g->keys[g->sorted_buf].as<uint32_t>();
    a.svals = g->vals[g->sorted_buf].as<uint32_t>();
    a.kshift = g->key_shift;
    a.invalid_key = 1u << g->lookup.ks.total_bits;
    a.spos = g->spos.as<float4>();
    a.svel = ppr ? g->svel.as<float4>() : nullptr;
    a.L = g->lookup;
    a.nbr = g->nbr.as<int>();
    a.leaf_slot = g->leaf_slot.as<int>();
    a.G = dL_drho;
    a.gpos = grad_pos;
    a.gw = grad_w;
    a.gr = grad_r;
    a.err = g->d_err.as<uint32_t>();
    if (a.n) {
        a.next = g->d_next.as<uint32_t>();
        const unsigned blocks = std::min<unsigned>(blocks_for((uint64_t)a.n * 32u, kBackThreads), 152u * 8u);
        if (mode == GVX_SPLAT_CUBIC)
            k_splat_backward<GVX_SPLAT_CUBIC><<<blocks, kBackThreads, 0, g->stream>>>(a);
        else
            k_splat_backward<GVX_SPLAT_TRILINEAR><<<blocks, kBackThreads, 0, g->stream>>>(a);
        g->launches++;
    }
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

extern "C" gvx_status gvx_splat_backward(gvx_grid* g, int mode, int n, float radius, const float trans[3],
                                         const float* dL_drho, float* grad_pos, float* grad_w, float* grad_r)
{
    return gvx_splat_backward_ex(g, mode, n, radius, trans, dL_drho, grad_pos, grad_w, grad_r, 0);
}
