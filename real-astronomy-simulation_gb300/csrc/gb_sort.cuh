// Stable LSD radix sort of (key, 32-bit value) pairs, 8-bit digits, shared by
// the tree build (Morton keys) and the neighbour grid (cell keys).
//
// The kernel that makes the keys counts the digits of every pass as it writes
// them (RsCount).  Each pass is then one kernel: a CTA takes the next tile of 2048
// keys from a counter, ranks them stably in index order (digit ballots within
// a warp, warp offsets within the tile), stages the tile in shared memory in
// digit order (so that global writes run in contiguous digit runs),
// publishes the tile's per-digit counts and finds the counts of all earlier
// tiles by decoupled look-back
// (Merrill and Garland, "Single-pass Parallel Prefix Scan with Decoupled
// Look-back", 2016) on two levels: a CTA adds the counts of the earlier tiles of
// its group of 16, then the groups' sums, back to a group whose inclusive prefix
// is published.  Tiles are handed out
// in counter order, so every tile a CTA waits for belongs to a CTA that is
// already running and publishes its count without waiting itself.  Each wait
// is bounded: after RS_SPIN_LIMIT polls the CTA counts DIAG_WAIT_TIMEOUT and
// goes on with the prefix it has (its scatter still stays inside [0, n)).
//
// Smaller sorts (radix_small) take up to three kernels instead: blocks of 1,024
// keys are made and sorted in shared memory, then every key finds its place
// among a group of blocks, and among the groups, by binary search.
#pragma once

#include <algorithm>

#include "gb_common.cuh"

namespace gb {

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;  // 2048 keys per CTA
constexpr int RS_BINS = 256;
constexpr int RS_MAX_PASSES = 8;                // 64-bit keys
constexpr int RS_COUNTERS = 32;                 // tile counters, one per pass
constexpr uint32_t RS_AGG = 1u << 30;           // status: a tile's own count
constexpr uint32_t RS_PRE = 2u << 30;           // status: a group's inclusive prefix
constexpr uint32_t RS_VAL = RS_AGG - 1u;        // count bits (n < 2^30)
constexpr int RS_SPIN_LIMIT = 1 << 20;          // polls of one status word before a wait gives up
constexpr int RS_LOOKBACK = 8;                  // tile words a look-back step reads at once
constexpr int RS_GROUP = 16;                    // tiles per group
constexpr int RS_GROUPS = 4;                    // groups a look-back step reads at once
constexpr uint32_t RS_GROUP_ONE = 1u << 24;     // group sums: one more tile added
static_assert(RS_GROUP * RS_TILE < RS_GROUP_ONE, "a group's counts stay below the number of tiles");

inline int64_t radix_tiles(int64_t n) { return (n + RS_TILE - 1) / RS_TILE; }

// Status words of a pass (RsStatus).
inline int64_t radix_status_words(int64_t n) {
    const int64_t nb = std::max<int64_t>(radix_tiles(n), 1);
    return (nb + 2 * ((nb + RS_GROUP - 1) / RS_GROUP)) * RS_BINS;
}

// 32-bit scratch words a sort of up to n keys needs: digit counts of every
// pass, the per-pass tile counters and two arrays of status words, used by
// alternate passes.
inline int64_t radix_scratch_size(int64_t n) {
    return (int64_t)RS_MAX_PASSES * RS_BINS + RS_COUNTERS + 2 * radix_status_words(n);
}

// Keys a sort accepts (status words hold counts below 2^30).
constexpr int64_t RS_MAX_N = (int64_t)RS_VAL;

__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_gpu(uint32_t *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void red_relaxed_gpu(uint32_t *p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The status words of a pass, zero when it starts: a word per tile and digit
// (RS_AGG and the tile's count), then per group of RS_GROUP tiles the sum of
// their counts, with the number of tiles that added theirs in the bits from
// RS_GROUP_ONE up, then per group its inclusive prefix (RS_PRE).
struct RsStatus {
    uint32_t *tile, *gsum, *gpre;
    __device__ __forceinline__ RsStatus(uint32_t *s, int nb)
        : tile(s), gsum(s + (int64_t)nb * RS_BINS),
          gpre(gsum + (int64_t)((nb + RS_GROUP - 1) / RS_GROUP) * RS_BINS) {}
};

// Publishes count c of digit d of tile t.
__device__ __forceinline__ void rs_publish(const RsStatus &st, int t, int d, uint32_t c) {
    st_relaxed_gpu(st.tile + (int64_t)t * RS_BINS + d, RS_AGG | c);
    red_relaxed_gpu(st.gsum + (int64_t)(t / RS_GROUP) * RS_BINS + d, RS_GROUP_ONE + c);
}

// Decoupled look-back for digit d of tile t, which has published count c: sums
// the counts of the group's earlier tiles and then
// the sums of earlier groups down to one whose last tile has published its
// prefix; a group's last tile publishes the group's.  Words are read
// RS_LOOKBACK at once and added as far as they are published.  What is not
// published yet is polled at most spin_limit times; then the wait counts
// DIAG_WAIT_TIMEOUT and ends with the sum it has.
//
// The words a pass reads and the round trips it waits for are what a pass of
// many tiles spends its time on.  Walking tile by tile down to a published
// prefix the tiles of a pass, which all start together, read up to 90 words a
// digit in 11 trips at 1,000,000 keys (489 tiles); with groups up to 45, in 2 to
// 4.  A pass of 1,000,000 32-bit keys: 16.9 to 13.3 us, and 12.3 with the staging
// between the publication and the look-back; 300,000: 10.1 to 8.7; 2,000,000:
// 25.6 to 21.0 (8 or 32 tiles a group, 2 or 8 groups a step: 13.3 to 13.8).
__device__ __forceinline__ uint32_t rs_lookback(const RsStatus &st, int t, int d, uint32_t c, int spin_limit,
                                                unsigned long long *diag) {
    const int g = t / RS_GROUP, r = t - g * RS_GROUP;
    uint32_t excl = 0;
    int spins = 0;
    // The group's tiles r-1, r-2, ..., 0.
    for (int j = r - 1; j >= 0;) {
        const uint32_t *p = st.tile + ((int64_t)g * RS_GROUP + j) * RS_BINS + d;
        uint32_t w[RS_LOOKBACK];
#pragma unroll
        for (int q = 0; q < RS_LOOKBACK; ++q) w[q] = j - q >= 0 ? ld_relaxed_gpu(p - q * RS_BINS) : 0u;
        int used = 0;
#pragma unroll
        for (int q = 0; q < RS_LOOKBACK; ++q)
            if (used == q && w[q] != 0u) {
                excl += w[q] & RS_VAL;
                used = q + 1;
            }
        j -= used;
        if (j >= 0 && used < RS_LOOKBACK && ++spins > spin_limit) {  // a tile has not published yet
            atomicAdd(diag + DIAG_WAIT_TIMEOUT, 1ull);
            return excl;
        }
    }
    // Groups g-1, g-2, ...
    for (int j = g - 1; j >= 0;) {
        const int64_t at = (int64_t)j * RS_BINS + d;
        uint32_t s[RS_GROUPS], p[RS_GROUPS];
#pragma unroll
        for (int q = 0; q < RS_GROUPS; ++q) {
            s[q] = j - q >= 0 ? ld_relaxed_gpu(st.gsum + at - q * RS_BINS) : 0u;
            p[q] = j - q >= 0 ? ld_relaxed_gpu(st.gpre + at - q * RS_BINS) : RS_PRE;
        }
        int used = 0;
        bool done = false;
#pragma unroll
        for (int q = 0; q < RS_GROUPS; ++q) {
            if (done || used < q) continue;
            done = (p[q] & RS_PRE) != 0u;
            if (!done && s[q] / RS_GROUP_ONE < RS_GROUP) continue;  // not complete
            excl += done ? p[q] & RS_VAL : s[q] % RS_GROUP_ONE;
            used = q + 1;
        }
        if (done) break;
        j -= used;
        if (j >= 0 && used < RS_GROUPS && ++spins > spin_limit) {
            atomicAdd(diag + DIAG_WAIT_TIMEOUT, 1ull);
            return excl;
        }
    }
    if (r == RS_GROUP - 1) st_relaxed_gpu(st.gpre + (int64_t)g * RS_BINS + d, RS_PRE | ((excl + c) & RS_VAL));
    return excl;
}

// Lanes of the warp holding the same 8-bit digit as this lane (among the
// lanes with ok set; a lane without ok matches only itself): eight ballots,
// one per digit bit.
__device__ __forceinline__ uint32_t warp_digit_peers(uint32_t dig, bool ok, int lane) {
    uint32_t m = __ballot_sync(0xffffffffu, ok);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (dig >> b) & 1u;
        const uint32_t bal = __ballot_sync(0xffffffffu, bit);
        m &= bit ? bal : ~bal;
    }
    return ok ? m : (1u << lane);
}

// Digit counts of all passes, taken by the kernel that makes the keys (it
// starts with all scratch words of radix_zero_words zero): counts[p * 256 +
// digit] += keys with that digit p (bits 8p .. 8p + 7).  Counted in shared
// memory, in COPIES copies by lane (equal digits of a warp's keys meet fewer
// conflicts), then one global add per non-zero bin and CTA.  A separate kernel
// that read the keys again took 16.4 us at n = 1,000,000 (8 ballots per digit).
template <int PASSES>
struct RsCount {
    static constexpr int COPIES = PASSES <= 4 ? 4 : 2;
    uint32_t h[COPIES][PASSES * RS_BINS];

    __device__ __forceinline__ void clear() {
        for (int i = threadIdx.x; i < COPIES * PASSES * RS_BINS; i += blockDim.x) (&h[0][0])[i] = 0u;
        __syncthreads();
    }
    template <typename KeyT>
    __device__ __forceinline__ void add(KeyT k, int passes) {
        uint32_t *c = h[threadIdx.x & (COPIES - 1)];
#pragma unroll
        for (int p = 0; p < PASSES; ++p)
            if (p < passes) atomicAdd(c + p * RS_BINS + ((uint32_t)(k >> (8 * p)) & 0xFFu), 1u);
    }
    __device__ __forceinline__ void flush(uint32_t *counts, int passes) {
        __syncthreads();
        for (int i = threadIdx.x; i < passes * RS_BINS; i += blockDim.x) {
            uint32_t n = 0;
#pragma unroll
            for (int q = 0; q < COPIES; ++q) n += h[q][i];
            if (n) atomicAdd(counts + i, n);
        }
    }
};

// Words that a kernel running before the keys' zeroes for the kernels behind
// it (a memset node each would cost a launch).
struct ZeroWords {
    uint32_t *p[3];
    int64_t n[3];
};

__device__ __forceinline__ void zero_words(const ZeroWords &z) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < z.n[k];
             i += (int64_t)gridDim.x * blockDim.x)
            z.p[k][i] = 0u;
}

// Exclusive scan of 256 values held one per thread of a 256-thread CTA.
__device__ __forceinline__ uint32_t cta256_exclusive_scan(uint32_t v, uint32_t *wsum) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const uint32_t w = lane < RS_WARPS ? wsum[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < RS_WARPS) wsum[lane] = wi - w;
    }
    __syncthreads();
    return wsum[wid] + inc - v;
}

// One pass: stable scatter of the tile the CTA takes from *counter.  Keys
// of a tile are ranked in index order (warp, round, lane) among equal
// digits; the destination is the digit's global start (scan of this pass's
// counts) + the digit's count in earlier tiles (look-back) + the rank within
// the tile.  status holds this pass's words (RsStatus, zeroed); status_next, when
// given, is zeroed here for the next pass.  IOTA (the first pass): the values
// are the keys' indices and are not read.
template <typename KeyT, bool IOTA>
__global__ void __launch_bounds__(RS_THREADS, 4)
rs_onesweep_kernel(const KeyT *__restrict__ kin, const uint32_t *__restrict__ vin, KeyT *__restrict__ kout,
                   uint32_t *__restrict__ vout, int64_t n, int shift, const uint32_t *__restrict__ counts,
                   uint32_t *counter, uint32_t *status, uint32_t *status_next, int nb,
                   int64_t status_words, unsigned long long *diag) {
    static_assert(RS_THREADS == RS_BINS, "one thread per digit");
    __shared__ uint32_t whist[RS_WARPS][RS_BINS];
    __shared__ uint32_t boff[RS_BINS];
    __shared__ uint32_t wsum[RS_WARPS];
    __shared__ int tile_s;
    __shared__ uint32_t wsum2[RS_WARPS];
    __shared__ uint32_t tst[RS_BINS];
    __shared__ KeyT skey[RS_TILE];  // the tile in digit order
    __shared__ uint32_t sval[RS_TILE];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, d = threadIdx.x;
    if (status_next) {
        for (int64_t i = (int64_t)blockIdx.x * RS_THREADS + threadIdx.x; i < status_words;
             i += (int64_t)gridDim.x * RS_THREADS)
            status_next[i] = 0u;
    }
    if (threadIdx.x == 0) tile_s = (int)atomicAdd(counter, 1u);
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) whist[w][d] = 0;
    __syncthreads();
    const int t = tile_s;
    const int64_t wbase = (int64_t)t * RS_TILE + (int64_t)wid * (RS_ITEMS * 32);
    const uint32_t lt_mask = (1u << lane) - 1u;
    KeyT key[RS_ITEMS];
    uint32_t val[RS_ITEMS];
    uint32_t rank[RS_ITEMS];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int64_t i = wbase + r * 32 + lane;
        const bool ok = i < n;
        key[r] = ok ? kin[i] : (KeyT)0;
        val[r] = IOTA ? (uint32_t)i : (ok ? vin[i] : 0u);
        const uint32_t dig = (uint32_t)(key[r] >> shift) & 0xFFu;
        const uint32_t peers = warp_digit_peers(dig, ok, lane);
        const uint32_t before = ok ? whist[wid][dig] : 0u;
        rank[r] = before + __popc(peers & lt_mask);
        __syncwarp();
        if (ok && (peers & lt_mask) == 0) whist[wid][dig] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Thread d: warp offsets of digit d within the tile, and its tile count.
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
        const uint32_t x = whist[w][d];
        whist[w][d] = c;
        c += x;
    }
    const RsStatus st(status, nb);
    rs_publish(st, t, d, c);
    // Digit d's first position in the tile; the tile's keys are staged in
    // shared memory in digit order, and position p of the staged tile goes
    // to boff[digit] + p (mod 2^32), so consecutive threads write
    // consecutive addresses within each digit's run.  The look-back comes
    // after the staging: by then most earlier tiles have published.
    const uint32_t start = counts[d];
    const uint32_t tstart = cta256_exclusive_scan(c, wsum2);
    tst[d] = tstart;
    const uint32_t gstart = cta256_exclusive_scan(start, wsum);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int64_t i = wbase + r * 32 + lane;
        if (i < n) {
            const uint32_t dig = (uint32_t)(key[r] >> shift) & 0xFFu;
            const uint32_t q = tst[dig] + whist[wid][dig] + rank[r];  // < RS_TILE for a consistent count
            if (q < (uint32_t)RS_TILE) {
                skey[q] = key[r];
                sval[q] = val[r];
            }
        }
    }
    boff[d] = gstart + rs_lookback(st, t, d, c, RS_SPIN_LIMIT, diag) - tstart;
    __syncthreads();
    const int64_t left = n - (int64_t)t * RS_TILE;
    const int cnt = left < (int64_t)RS_TILE ? (int)left : RS_TILE;
    for (int q = threadIdx.x; q < cnt; q += RS_THREADS) {
        const KeyT k = skey[q];
        const uint32_t dst = boff[(uint32_t)(k >> shift) & 0xFFu] + (uint32_t)q;
        if (dst < n) {
            kout[dst] = k;
            vout[dst] = sval[q];
        } else {
            atomicAdd(diag + DIAG_BAD_TREE, 1ull);
        }
    }
}

// ------------------------------------------------------------ small sorts
// First kernel: a CTA makes 1,024 keys (src(i): the key of index i) and sorts
// them with their indices: 32 at a time by a bitonic network in each warp,
// then five rounds that merge neighbouring runs, a key's place in its pair of
// runs being its place in its own plus the keys before it in the other
// (binary search; equal keys of the earlier run come first, so the sort is
// stable).
constexpr int SS_BLOCK = 1024;

template <typename KeyT>
__device__ __forceinline__ int ss_count(const KeyT *run, int len, KeyT key, bool equal_too) {
    int at = 0;  // len is a power of two; at < len before the last comparison
    for (int step = len >> 1; step > 0; step >>= 1) {
        const KeyT x = run[at + step - 1];
        if (x < key || (equal_too && x == key)) at += step;
    }
    const KeyT x = run[at];
    return at + (x < key || (equal_too && x == key));
}

template <typename KeyT, typename Source>
__global__ void __launch_bounds__(SS_BLOCK)
ss_block_kernel(Source src, int n, KeyT *__restrict__ kout, uint32_t *__restrict__ vout) {
    __shared__ KeyT sk[2][SS_BLOCK];
    __shared__ uint32_t sv[2][SS_BLOCK];
    const int tid = threadIdx.x, lane = tid & 31, g = blockIdx.x * SS_BLOCK + tid;
    KeyT key = g < n ? src(g) : ~(KeyT)0;  // above every key: the last ones
    uint32_t val = (uint32_t)g;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const KeyT ok = __shfl_xor_sync(0xffffffffu, key, j);
            const uint32_t ov = __shfl_xor_sync(0xffffffffu, val, j);
            const bool less = ok < key || (ok == key && ov < val);        // the other one comes first
            const bool want_first = ((lane & k) == 0) == ((lane & j) == 0);  // k = 32: ascending
            if (less == want_first) {
                key = ok;
                val = ov;
            }
        }
    int buf = 0;
    sk[0][tid] = key;
    sv[0][tid] = val;
    __syncthreads();
#pragma unroll
    for (int len = 32; len < SS_BLOCK; len <<= 1) {
        const int other = (tid & ~(len - 1)) ^ len;
        const int to = (tid & ~(2 * len - 1)) + (tid & (len - 1)) + ss_count(sk[buf] + other, len, key, other < tid);
        sk[buf ^ 1][to] = key;
        sv[buf ^ 1][to] = val;
        buf ^= 1;
        __syncthreads();
        key = sk[buf][tid];
        val = sv[buf][tid];
    }
    if (g < n) {
        kout[g] = key;
        vout[g] = val;
    }
}

// First index in [0, n) with key >= c (above: > c), found by a warp: 32 probes
// per step.
template <typename KeyT, typename IndexT>
__device__ __forceinline__ IndexT warp_bound(const KeyT *__restrict__ keys, IndexT n, KeyT c, bool above = false) {
    const int lane = threadIdx.x & 31;
    IndexT lo = 0, hi = n;
    while (lo < hi) {
        const IndexT step = (hi - lo + 32) / 33, at = lo + (lane + 1) * step - 1;
        const KeyT x = at < hi ? __ldg(keys + at) : (KeyT)0;
        const int below = __popc(__ballot_sync(0xffffffffu, at < hi && (x < c || (above && x == c))));
        hi = below < 32 ? min(hi, lo + (below + 1) * step - 1) : hi;
        lo += below * step;
    }
    return lo;
}

// Second kernel: a group of neighbouring sorted blocks becomes one.  The place
// of a key is its place in its block plus the keys before it in every other
// block of the group (those of earlier blocks where equal).  A CTA takes
// SS_KEYS consecutive keys of a block and passes over the group's blocks,
// SS_SIDE of them at a time in shared memory, whose searches run side by side;
// a warp's keys are neighbours, so they read the same or neighbouring words.
constexpr int SS_KEYS = 256;
constexpr int SS_SIDE = 4;

template <typename KeyT>
__global__ void __launch_bounds__(SS_KEYS)
ss_group_kernel(const KeyT *__restrict__ kin, const uint32_t *__restrict__ vin, int n, int group,
                KeyT *__restrict__ kout, uint32_t *__restrict__ vout) {
    __shared__ KeyT blk[SS_SIDE][SS_BLOCK];
    const int tid = threadIdx.x, g = blockIdx.x * SS_KEYS + tid, mine = blockIdx.x / (SS_BLOCK / SS_KEYS);
    const int first = mine / group * group, end = min(first + group, (n + SS_BLOCK - 1) / SS_BLOCK);
    const KeyT key = g < n ? __ldg(kin + g) : ~(KeyT)0;
    int place = first * SS_BLOCK + (g - mine * SS_BLOCK);
    for (int b0 = first; b0 < end; b0 += SS_SIDE) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < SS_SIDE * SS_BLOCK / SS_KEYS; ++q) {
            const int i = q * SS_KEYS + tid, x = b0 * SS_BLOCK + i;
            (&blk[0][0])[i] = x < min(n, end * SS_BLOCK) ? __ldg(kin + x) : ~(KeyT)0;
        }
        __syncthreads();
        int at[SS_SIDE];
#pragma unroll
        for (int q = 0; q < SS_SIDE; ++q) at[q] = 0;
#pragma unroll
        for (int step = SS_BLOCK >> 1; step > 0; step >>= 1)
#pragma unroll
            for (int q = 0; q < SS_SIDE; ++q) {
                const KeyT x = blk[q][at[q] + step - 1];
                if (x < key || (b0 + q < mine && x == key)) at[q] += step;
            }
#pragma unroll
        for (int q = 0; q < SS_SIDE; ++q) {
            const KeyT x = blk[q][at[q]];
            if (x < key || (b0 + q < mine && x == key)) ++at[q];
            if (b0 + q != mine) place += at[q];  // past the group's end no key is below ~0
        }
    }
    if (g < n && place < n) {
        kout[place] = key;
        vout[place] = __ldg(vin + g);
    }
}

// Third kernel: all groups, sorted blocks of len keys, become one.  The places
// of a CTA's first and last key bound its searches in another block (a 32-way
// search by a warp each), which are short and read neighbouring words of L1.
constexpr int SS_MAX_GROUPS = 16;

template <typename KeyT>
__global__ void __launch_bounds__(SS_KEYS)
ss_merge_kernel(const KeyT *__restrict__ kin, const uint32_t *__restrict__ vin, int n, int len,
                KeyT *__restrict__ kout, uint32_t *__restrict__ vout) {
    __shared__ int from[SS_MAX_GROUPS], size[SS_MAX_GROUPS];  // the window in each block
    const int tid = threadIdx.x, wid = tid >> 5, g0 = blockIdx.x * SS_KEYS, g = g0 + tid;
    const int mine = g0 / len, blocks = (n + len - 1) / len;
    const KeyT key = g < n ? __ldg(kin + g) : ~(KeyT)0;
    const KeyT kmin = __ldg(kin + g0), kmax = __ldg(kin + min(g0 + SS_KEYS, n) - 1);
    for (int t = wid; t < blocks; t += SS_KEYS / 32) {
        const int start = t * len, cnt = min(len, n - start);
        int lo = 0, m = 0;
        if (t != mine) {
            lo = warp_bound(kin + start, cnt, kmin);
            m = warp_bound(kin + start + lo, cnt - lo, kmax, true);
        }
        if ((tid & 31) == 0) {
            from[t] = start + lo;
            size[t] = m;
        }
    }
    __syncthreads();
    int place = g - mine * len;
    for (int t0 = 0; t0 < blocks; t0 += SS_SIDE) {
        int at[SS_SIDE], m[SS_SIDE], most = 0;
        const KeyT *win[SS_SIDE];
#pragma unroll
        for (int q = 0; q < SS_SIDE; ++q) {
            const bool in = t0 + q < blocks;
            const int f = in ? from[t0 + q] : 0;
            win[q] = kin + f;
            m[q] = in ? size[t0 + q] : 0;
            most = max(most, m[q]);
            at[q] = 0;
            if (in && t0 + q != mine) place += f - (t0 + q) * len;
        }
        for (int step = most > 0 ? 1 << (31 - __clz(most)) : 0; step > 0; step >>= 1)
#pragma unroll
            for (int q = 0; q < SS_SIDE; ++q)
                if (at[q] + step <= m[q]) {
                    const KeyT x = __ldg(win[q] + at[q] + step - 1);
                    if (x < key || (t0 + q < mine && x == key)) at[q] += step;
                }
#pragma unroll
        for (int q = 0; q < SS_SIDE; ++q) place += at[q];
    }
    if (g < n && place < n) {
        kout[place] = key;
        vout[place] = __ldg(vin + g);
    }
}

// Whether a sort of n keys in `passes` digits takes these kernels.  Bounding
// box, keys and sort on the disk (us, with a kernel per digit in brackets),
// 63-bit keys (8 digits): 1,000: 19 (72); 10,000: 28 (94); 33,000: 40 (96);
// 100,000: 54 (104); 131,072: 58 (114); 200,000: 93 (121); 262,144: 108 (123).
// 30-bit keys (4): 10,000: 24 (52); 33,000: 36 (56); 100,000: 49 (62); 131,072:
// 51 (64); 200,000: 79 (72).  A kernel per digit costs 7 to 9 us whatever its
// size, mostly launch, look-back and ranking latency; these grow with the
// number of blocks each key is compared with.  Groups of 32: 63 at 100,000;
// blocks' windows instead of whole blocks in the second kernel too: 36 at
// 10,000, 65 at 100,000; one stage over all blocks: 98 at 100,000.
constexpr int64_t SS_ONE_N = 32 * SS_BLOCK;  // one group
constexpr int64_t SS_GROUP = 16;             // blocks per group above
constexpr int64_t SS_MAX_N8 = 262144, SS_MAX_N4 = 131072, SS_MAX_N3 = 65536;
static_assert(SS_MAX_N8 <= SS_MAX_GROUPS * SS_GROUP * SS_BLOCK, "a window per group");
inline bool radix_small(int64_t n, int passes) {
    return n <= (passes > 4 ? SS_MAX_N8 : passes == 4 ? SS_MAX_N4 : SS_MAX_N3);
}

// Kernels of such a sort.
inline int radix_small_launches(int64_t n) { return n <= SS_BLOCK ? 1 : n <= SS_ONE_N ? 2 : 3; }

// Sorts the keys src(0 .. n - 1) with their indices.  The result is in k[0] and
// v[0] whatever n is, like that of an even number of digits: two kernels start
// in the other pair.
template <typename KeyT, typename Source>
static void radix_sort_small(const Source &src, KeyT *k[2], uint32_t *v[2], int64_t n, cudaStream_t s) {
    const int launches = radix_small_launches(n), a = launches == 2 ? 1 : 0, b = a ^ 1;
    const unsigned gr = (unsigned)((n + SS_KEYS - 1) / SS_KEYS);
    ss_block_kernel<KeyT, Source><<<(unsigned)((n + SS_BLOCK - 1) / SS_BLOCK), SS_BLOCK, 0, s>>>(src, (int)n, k[a],
                                                                                               v[a]);
    if (launches > 1)
        ss_group_kernel<KeyT><<<gr, SS_KEYS, 0, s>>>(k[a], v[a], (int)n, launches == 2 ? 32 : (int)SS_GROUP, k[b],
                                                     v[b]);
    if (launches > 2)
        ss_merge_kernel<KeyT><<<gr, SS_KEYS, 0, s>>>(k[1], v[1], (int)n, (int)(SS_GROUP * SS_BLOCK), k[0], v[0]);
}

// Scratch words that are zero when the kernel that makes the keys starts:
// the digit counts, the tile counters and the first pass's status array.
inline int64_t radix_zero_words(int64_t n) {
    return (int64_t)RS_MAX_PASSES * RS_BINS + RS_COUNTERS + radix_status_words(n);
}

// Sorts k[0], with the indices 0 .. n - 1 as values, by the low 8 * passes
// bits of the keys (n < 2^30, 1 <= passes <= 8), ping-ponging with k[1] and
// v; returns the index of the pair holding the result.  scratch holds
// radix_scratch_size(n) words, zeroed (radix_zero_words) and with the digit
// counts added (RsCount).  Launches: one kernel per pass.
template <typename KeyT>
static int radix_sort_counted(KeyT *k[2], uint32_t *v[2], int64_t n, int passes, uint32_t *scratch,
                              unsigned long long *diag, cudaStream_t s) {
    const int nb = (int)radix_tiles(n);
    const int64_t words = radix_status_words(n);
    uint32_t *counts = scratch;
    uint32_t *counters = counts + RS_MAX_PASSES * RS_BINS;
    uint32_t *status[2] = {counters + RS_COUNTERS, counters + RS_COUNTERS + words};
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        uint32_t *next = p + 1 < passes ? status[(p + 1) & 1] : nullptr;
        if (p == 0)
            rs_onesweep_kernel<KeyT, true><<<nb, RS_THREADS, 0, s>>>(k[0], v[0], k[1], v[1], n, 0, counts, counters,
                                                                     status[0], next, nb, words, diag);
        else
            rs_onesweep_kernel<KeyT, false><<<nb, RS_THREADS, 0, s>>>(k[cur], v[cur], k[cur ^ 1], v[cur ^ 1], n, 8 * p,
                                                                      counts + p * RS_BINS, counters + p, status[p & 1],
                                                                      next, nb, words, diag);
        cur ^= 1;
    }
    return cur;
}

}  // namespace gb
