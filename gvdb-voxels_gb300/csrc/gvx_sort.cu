// gvx_sort.cu -- hand-written onesweep LSD radix sort of 32-bit brick keys.
//
// Replaces the reference's thrust::sort of 64-bit keys (gvdb_cutils.cu:11-16,
// called from VolumeGVDB::RadixSortByByte, gvdb_volume_gvdb.cpp:904-928).
// Only the significant bits of the compact brick key are sorted (8 bits per
// pass), the digit histograms of all passes come from one upfront count (fused
// into the key producer when it can), and every pass is a single kernel: tile
// ranking by warp ballots, decoupled look-back across tiles for the digit
// offsets, then a scatter staged through shared memory so that global writes
// of one digit bucket are contiguous.  Stable: equal keys keep input order.
//
// Every look-back wait is bounded: after ~2 s of polling the kernel records
// GVX_DERR_TIMEOUT in the device error word and carries on, so a lost
// predecessor can never hang the GPU.
#include <algorithm>

#include "gvx_internal.cuh"

namespace {
constexpr int kWindow = 8;  // predecessors a look-back round loads at once
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kFlagMask = 3u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1u;
constexpr long long kSpinCycles = 4000000000LL;
}  // namespace

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v)
{
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// the digit of a pair; the pairs past the end of the input (not live) have digit 255
__device__ __forceinline__ uint32_t i_digit(uint32_t key, int shift, bool live)
{
    return live ? (key >> shift) & 255u : 255u;
}

__global__ void k_sort_hist(const uint32_t* __restrict__ keys, uint32_t n, int passes, uint32_t* hist)
{
    __shared__ uint32_t sh[4 * 256];
    for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        gvx_sort_count_key(sh, keys[i], passes);
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += blockDim.x)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// One pass over a tile of THREADS * ITEMS pairs per block.
//
// What bounds it: the chain of tiles and instruction issue (half of the slots), not HBM (16 bytes a pair and pass).
// Every tile needs the digit counts of all tiles before it; the resident tiles start together, so
// the look-back of a late tile walks over many predecessors before it meets a finished prefix.
//  - A thread (one digit) loads kWindow predecessors at a time, independent loads in flight, and
//    polls a single word while its next predecessor has published nothing.
//  - The walk starts only after the tile has been put in digit order in shared memory, which needs
//    the tile's own counts alone: the predecessors publish theirs meanwhile.
//  - Tiles of 8192 pairs (512 threads, half of which look back) keep fewer tiles in flight than
//    tiles of 4096 would: less walking per pair.
//  - Equal digits of a warp are found by eight ballots (match_any waits longer for its result than
//    the eight votes take to issue).
//  - The pairs past the end of the last tile rank as digit 255, after every pair of the input, and
//    are taken out of the tile's count of that digit.
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
    k_onesweep(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
               uint32_t* __restrict__ vout, uint32_t n, int shift, const uint32_t* __restrict__ hist,
               uint32_t* lookback, uint32_t* counter, uint32_t* err)
{
    constexpr uint32_t TILE = (uint32_t)THREADS * ITEMS;
    constexpr int WARPS = THREADS / 32;
    extern __shared__ __align__(16) uint32_t s_dyn[];  // (s_whist is cleared 16 bytes at a time)
    uint32_t* s_keys = s_dyn;                     // TILE
    uint32_t* s_vals = s_dyn + TILE;              // TILE
    uint32_t(*s_whist)[256] = (uint32_t(*)[256])(s_dyn + 2 * TILE);  // per warp: digit counts, then offsets
    __shared__ uint32_t s_gofs[256];              // where the digit's pairs go, less their place in the tile
    __shared__ uint32_t s_wsum[8], s_hsum[8];
    __shared__ uint32_t s_tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(counter, 1u);
    for (int i = tid; i < WARPS * 64; i += THREADS) ((uint4*)&s_whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t tbase = tile * TILE;
    const uint32_t cnt_tile = min(TILE, n - tbase);
    const uint32_t w0 = (uint32_t)warp * 32u * ITEMS + lane;  // the thread's first pair in the tile

    uint32_t k[ITEMS], r[ITEMS / 2];  // r: places among the equal digits, 16 bits each
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        const uint32_t i = w0 + (uint32_t)j * 32u;
        k[j] = i < cnt_tile ? kin[tbase + i] : 0xFFFFFFFFu;
    }
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        const uint32_t d = i_digit(k[j], shift, w0 + (uint32_t)j * 32u < cnt_tile);
        uint32_t peers = 0xFFFFFFFFu;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, (d >> q) & 1u);
            peers &= ~(m ^ (0u - ((d >> q) & 1u)));
        }
        const int leader = __ffs(peers) - 1;
        uint32_t prev = 0u;
        if (lane == leader) {
            prev = s_whist[warp][d];
            s_whist[warp][d] = prev + __popc(peers);
        }
        prev = __shfl_sync(0xFFFFFFFFu, prev, leader);
        prev += __popc(peers & lt);
        r[j / 2] = (j & 1) ? r[j / 2] | prev << 16 : prev;
        __syncwarp();
    }
    // (the values are asked for here, past the ranking that needs the registers; they arrive while
    // the counts are scanned)
    uint32_t v[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        const uint32_t i = w0 + (uint32_t)j * 32u;
        v[j] = i < cnt_tile ? vin[tbase + i] : 0u;
    }
    __syncthreads();

    // thread tid < 256 owns digit tid: the tile's count, published for the later tiles, and the
    // places of the warps' pairs of that digit in the tile
    uint32_t cnt = 0u, tstart = 0u, gbase = 0u;
    uint32_t* my = lookback + (size_t)tile * 256u + tid;
    if (tid < 256) {
#pragma unroll
        for (int w = 0; w < WARPS; w++) cnt += s_whist[w][tid];
        if (tid == 255) cnt -= TILE - cnt_tile;
        st_relaxed(my, (tile == 0 ? kFlagPrefix : kFlagAgg) | cnt);
        // exclusive scans over the digits: of the tile's counts, and of the whole input's
        const uint32_t all = hist[tid];
        uint32_t x = cnt, h = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o), z = __shfl_up_sync(0xFFFFFFFFu, h, o);
            if (lane >= o) {
                x += y;
                h += z;
            }
        }
        if (lane == 31) {
            s_wsum[warp] = x;
            s_hsum[warp] = h;
        }
        tstart = x - cnt;
        gbase = h - all;
    }
    __syncthreads();
    if (tid < 256) {
        for (int w = 0; w < warp; w++) {
            tstart += s_wsum[w];
            gbase += s_hsum[w];
        }
        uint32_t at = tstart;
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
            const uint32_t c = s_whist[w][tid];
            s_whist[w][tid] = at;
            at += c;
        }
    }
    __syncthreads();

    // the tile in digit order
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        if (w0 + (uint32_t)j * 32u < cnt_tile) {
            const uint32_t pos = s_whist[warp][(k[j] >> shift) & 255u] + (r[j / 2] >> (16 * (j & 1)) & 0xFFFFu);
            s_keys[pos] = k[j];
            s_vals[pos] = v[j];
        }
    }

    // look-back: the digit's count in all earlier tiles, kWindow tiles a round
    if (tid < 256) {
        uint32_t excl = 0u;
        if (tile > 0) {
            const uint32_t* lb = lookback + (size_t)(tile - 1) * 256u + tid;  // the next predecessor's word
            int left = (int)tile;                                              // predecessors not yet counted
            const long long t0 = clock64();
            bool done = false;
            while (!done) {
                uint32_t w[kWindow];
                w[0] = ld_relaxed(lb);
                while ((w[0] & kFlagMask) == 0u) {  // nothing published yet
                    if (clock64() - t0 > kSpinCycles) {
                        atomicOr(err, GVX_DERR_TIMEOUT);
                        done = true;
                        break;
                    }
                    w[0] = ld_relaxed(lb);
                }
                if (done) break;
#pragma unroll
                for (int i = 1; i < kWindow; i++) w[i] = i < left ? ld_relaxed(lb - i * 256) : 0u;
                int used = 0;
                bool run = true;  // up to the first prefix, or the first word without a flag
#pragma unroll
                for (int i = 0; i < kWindow; i++) {
                    run = run && (w[i] & kFlagMask) != 0u;
                    if (run) {
                        excl += w[i] & kCountMask;
                        used = i + 1;
                        done = (w[i] & kFlagPrefix) != 0u;
                        run = !done;
                    }
                }
                lb -= used * 256;
                left -= used;
            }
            st_relaxed(my, kFlagPrefix | ((excl + cnt) & kCountMask));
        }
        s_gofs[tid] = gbase + excl - tstart;
    }
    __syncthreads();

#pragma unroll 4
    for (uint32_t i = tid; i < cnt_tile; i += THREADS) {
        const uint32_t key = s_keys[i];
        const uint32_t g = s_gofs[(key >> shift) & 255u] + i;
        kout[g] = key;
        vout[g] = s_vals[i];
    }
}

template <int THREADS, int ITEMS>
static gvx_status onesweep_launch(uint32_t tiles, const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                                  uint32_t* vout, uint32_t n, int shift, const uint32_t* hist, uint32_t* lookback,
                                  uint32_t* counter, uint32_t* err, cudaStream_t st)
{
    const size_t smem = ((size_t)THREADS * ITEMS * 2 + (size_t)THREADS / 32 * 256) * sizeof(uint32_t);
    if (smem > 46 * 1024)  // (with the static arrays, past the 48 KB a kernel has without asking)
        GVX_CK(cudaFuncSetAttribute(k_onesweep<THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem));
    k_onesweep<THREADS, ITEMS><<<tiles, THREADS, smem, st>>>(kin, vin, kout, vout, n, shift, hist, lookback, counter,
                                                             err);
    return GVX_OK;
}

gvx_status gvx_onesweep_pass(uint32_t tile, uint32_t tiles, const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                             uint32_t* vout, uint32_t n, int shift, const uint32_t* hist, uint32_t* lookback,
                             uint32_t* counter, uint32_t* err, cudaStream_t st)
{
    if (tile == 1024)
        return onesweep_launch<256, 4>(tiles, kin, vin, kout, vout, n, shift, hist, lookback, counter, err, st);
    if (tile == 4096)
        return onesweep_launch<256, 16>(tiles, kin, vin, kout, vout, n, shift, hist, lookback, counter, err, st);
    return onesweep_launch<512, 16>(tiles, kin, vin, kout, vout, n, shift, hist, lookback, counter, err, st);
}

// Pairs per tile: small inputs are spread over more SMs (100k pairs, 24 bits, three passes and the
// copies around them: 61 us with tiles of 1024, 69 with 4096, 81 with 8192), large ones keep fewer
// tiles in flight (400k: 86 / 86 / 97 us; 1.5M: 128 / 104 / 113; 3M: 190 / 159 / 149; 32M: 1424 /
// 805 / 802, where one predecessor per look-back step and match_any took 1071)
static uint32_t sort_tile(uint32_t n)
{
    return n <= 300000u ? 1024u : n <= 2000000u ? 4096u : 8192u;
}

int gvx_sort_passes(int bits) { return bits <= 0 ? 0 : (bits + 7) / 8; }

// scratch of one sort, zeroed together: the digit histograms of four passes, their tile counters
// (64 words), the look-back words of every pass
constexpr size_t kHistWords = 4 * 256, kCounterWords = 64;

uint32_t* gvx_sort_hist_ptr(SortScratch& s) { return s.buf.as<uint32_t>(); }

gvx_status gvx_sort_prepare(SortScratch& s, uint32_t n, int bits, ClearList& clear)
{
    const uint32_t tile = sort_tile(n), tiles = (n + tile - 1) / tile;
    const size_t words = kHistWords + kCounterWords + (size_t)gvx_sort_passes(bits) * tiles * 256;
    GVX_CK(gvx_ensure(s.buf, words * sizeof(uint32_t)));
    clear.add(s.buf.p, words, 0u);
    return GVX_OK;
}

static gvx_status sort_limits(uint32_t n, int bits)
{
    if (bits > 32) {
        gvx_set_error("sort: %d key bits exceed 32", bits);
        return GVX_ERR_INVALID_ARG;
    }
    if (n > kCountMask) {
        gvx_set_error("sort: %u keys exceed the 2^30 limit", n);
        return GVX_ERR_CAPACITY;
    }
    return GVX_OK;
}

// the passes of a prepared sort whose histograms are in: pass p reads what pass p - 1 wrote (the
// first one kin, vin) and writes k[to], v[to] with to = `first` on even p, the other one on odd p
static gvx_status sort_run(const uint32_t* kin, const uint32_t* vin, uint32_t* const k[2], uint32_t* const v[2],
                           int first, uint32_t n, int bits, SortScratch& s, cudaStream_t st, uint32_t* d_err,
                           int64_t* launches)
{
    const int passes = gvx_sort_passes(bits);
    const uint32_t tile = sort_tile(n), tiles = (n + tile - 1) / tile;
    uint32_t* hist = s.buf.as<uint32_t>();
    uint32_t* counter = hist + kHistWords;
    uint32_t* lookback = counter + kCounterWords;
    int to = first;
    for (int p = 0; p < passes; p++, to ^= 1) {
        GVX_CK_STATUS(gvx_onesweep_pass(tile, tiles, kin, vin, k[to], v[to], n, 8 * p, hist + p * 256,
                                        lookback + (size_t)p * tiles * 256, counter + p, d_err, st));
        (*launches)++;
        kin = k[to];
        vin = v[to];
    }
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}

static gvx_status sort_histograms(const uint32_t* keys, uint32_t n, int bits, SortScratch& s, cudaStream_t st,
                                  int64_t* launches)
{
    ClearList clear;
    GVX_CK_STATUS(gvx_sort_prepare(s, n, bits, clear));
    GVX_CK(cudaMemsetAsync(clear.p[0], 0, clear.words[0] * sizeof(uint32_t), st));
    const uint32_t blocks = std::min<uint32_t>((n + 4095u) / 4096u, 1024u);
    k_sort_hist<<<blocks, 256, 0, st>>>(keys, n, gvx_sort_passes(bits), gvx_sort_hist_ptr(s));
    (*launches)++;
    return GVX_OK;
}

gvx_status gvx_sort_pairs(uint32_t* keys[2], uint32_t* vals[2], uint32_t n, int bits, SortScratch& s,
                          bool prepared, cudaStream_t st, uint32_t* d_err, int* result, int64_t* launches)
{
    *result = 0;
    const int passes = gvx_sort_passes(bits);
    if (n <= 1 || passes == 0) return GVX_OK;
    GVX_CK_STATUS(sort_limits(n, bits));
    if (!prepared) GVX_CK_STATUS(sort_histograms(keys[0], n, bits, s, st, launches));
    GVX_CK_STATUS(sort_run(keys[0], vals[0], keys, vals, 1, n, bits, s, st, d_err, launches));
    *result = passes & 1;
    return GVX_OK;
}

gvx_status gvx_sort_pairs_to(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout,
                             uint32_t* ktmp, uint32_t* vtmp, uint32_t n, int bits, SortScratch& s, cudaStream_t st,
                             uint32_t* d_err, int64_t* launches)
{
    GVX_CK_STATUS(sort_limits(n, bits));
    GVX_CK_STATUS(sort_histograms(kin, n, bits, s, st, launches));
    uint32_t* const k[2] = {kout, ktmp};
    uint32_t* const v[2] = {vout, vtmp};
    return sort_run(kin, vin, k, v, (gvx_sort_passes(bits) & 1) ^ 1, n, bits, s, st, d_err, launches);
}

// One pass of the sort with its first tile withheld (a test of the bounded
// look-back): the tile counter starts at 1 and tiles - 1 blocks run, so every
// block takes a tile in range, and the tile after the withheld one waits for a
// flag that nothing sets.  Its wait gives up after kSpinCycles and records
// GVX_DERR_TIMEOUT; it then publishes the prefix it has (a lower bound of the
// true one, so every scatter index stays below n) and the later tiles finish.
gvx_status gvx_sort_pass_withheld_tile(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout,
                                       uint32_t n, SortScratch& s, cudaStream_t st, uint32_t* d_err,
                                       int64_t* launches)
{
    constexpr uint32_t kTile = 4096;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    if (tiles < 2) {
        gvx_set_error("sort test: %u keys make one tile; at least two are needed", n);
        return GVX_ERR_INVALID_ARG;
    }
    const size_t words = kHistWords + kCounterWords + (size_t)tiles * 256;
    GVX_CK(gvx_ensure(s.buf, words * sizeof(uint32_t)));
    GVX_CK(cudaMemsetAsync(s.buf.p, 0, words * sizeof(uint32_t), st));
    uint32_t* hist = s.buf.as<uint32_t>();
    uint32_t* counter = hist + kHistWords;
    k_sort_hist<<<tiles < 1024 ? tiles : 1024, 256, 0, st>>>(kin, n, 1, hist);
    static const uint32_t one = 1u;
    GVX_CK(cudaMemcpyAsync(counter, &one, sizeof(one), cudaMemcpyHostToDevice, st));
    GVX_CK_STATUS(gvx_onesweep_pass(kTile, tiles - 1, kin, vin, kout, vout, n, 0, hist, counter + kCounterWords,
                                    counter, d_err, st));
    *launches += 2;
    GVX_CK(cudaGetLastError());
    return GVX_OK;
}
