// LBVH Barnes-Hut on the GB300 (sm_103a): every stage on the device.
//
// Replaces BarnesHut.compute (core/solvers/barnes_hut.py:242-259), which runs
// Morton keys and the stable sort on the host in numpy and the tree kernels
// in Taichi.  Stages (one CUDA graph per step when driven by gb_bh_kdk):
//   0 bbox      per-axis min/max (optionally after the fused kick+drift),
//               last-CTA-done combine -> FP64 quantisation parameters
//   1 morton    keys bit-identical to morton_codes (:27-46): FP64
//               (x - lo) * scale with separate roundings, clip, truncate,
//               interleave x,y,z into bits 3b, 3b+1, 3b+2
//   2 sort      stable LSD radix sort (8-bit digits) of (key, index): the
//               permutation of np.argsort(kind="stable") (:247)
//   3 tree      particles into key order (leaf records), the binary radix
//               tree, identical to _build_radix (:84-121), and node mass,
//               first moment and AABB (FP32) in one pass upwards, in shared
//               memory within chunks of leaves; no floating-point atomics,
//               and the result is independent of scheduling (:124-177 use
//               FP64 atomics on every ancestor instead)
//   4 traverse  per-particle walk: 4 to 32 key-consecutive targets share a
//               warp and its list of opened nodes (for large theta one node
//               at a time); every target applies the reference's own acceptance
//               test size^2 < theta^2 (r^2 + eps^2) (:204-210), so each
//               particle accepts exactly the node set of _traverse
//               (:180-217); the max_stack rule (:212) is kept and the skipped
//               pushes are counted instead of being lost silently.  Closing
//               kick fused in the epilogue for KDK steps.
#include <algorithm>
#include <cstdio>

#include "gb_common.cuh"
#include "gb_sort.cuh"

namespace gb {

struct BHParams {
    double lo[3];
    double scale;
    float lof[3], sh, sl;  // the same for cell_fp32
};



constexpr int BBOX_THREADS = 256;
constexpr int KEY_THREADS = 256;

// ------------------------------------------------------------------ bbox
template <bool KDK>
__global__ void __launch_bounds__(BBOX_THREADS)
bh_bbox_kernel(float4 *xm, float4 *vel, const float4 *acc, int64_t n, float h, float dt, float4 *part,
               unsigned *ticket, BHParams *prm, int bits, ZeroWords zero, unsigned long long *diag) {
    zero_words(zero);
    float mn0 = INFINITY, mn1 = INFINITY, mn2 = INFINITY;
    float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY;
    unsigned long long bad = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float4 x = xm[i];
        if (KDK) {
            const float4 v = vel[i], a = acc[i];
            const float vx = kick(v.x, a.x, h), vy = kick(v.y, a.y, h), vz = kick(v.z, a.z, h);
            x = make_float4(drift(x.x, vx, dt), drift(x.y, vy, dt), drift(x.z, vz, dt), x.w);
            xm[i] = x;
            vel[i] = make_float4(vx, vy, vz, v.w);
        }
        if (isfinite(x.x) && isfinite(x.y) && isfinite(x.z)) {
            mn0 = fminf(mn0, x.x); mn1 = fminf(mn1, x.y); mn2 = fminf(mn2, x.z);
            mx0 = fmaxf(mx0, x.x); mx1 = fmaxf(mx1, x.y); mx2 = fmaxf(mx2, x.z);
        } else {
            ++bad;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn0 = fminf(mn0, __shfl_xor_sync(0xffffffffu, mn0, o));
        mn1 = fminf(mn1, __shfl_xor_sync(0xffffffffu, mn1, o));
        mn2 = fminf(mn2, __shfl_xor_sync(0xffffffffu, mn2, o));
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        mx2 = fmaxf(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
        bad += __shfl_xor_sync(0xffffffffu, bad, o);
    }
    __shared__ float4 smn[BBOX_THREADS / 32], smx[BBOX_THREADS / 32];
    __shared__ bool is_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        smn[wid] = make_float4(mn0, mn1, mn2, 0.f);
        smx[wid] = make_float4(mx0, mx1, mx2, 0.f);
        if (bad) atomicAdd(diag + DIAG_NONFINITE, bad);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float4 a = smn[0], b = smx[0];
        for (int w = 1; w < BBOX_THREADS / 32; ++w) {
            a.x = fminf(a.x, smn[w].x); a.y = fminf(a.y, smn[w].y); a.z = fminf(a.z, smn[w].z);
            b.x = fmaxf(b.x, smx[w].x); b.y = fmaxf(b.y, smx[w].y); b.z = fmaxf(b.z, smx[w].z);
        }
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = b;
        __threadfence();
        is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    // Last CTA: merge every CTA's partial with all its threads (strided L2
    // reads, then the same warp/CTA reduction).
    __threadfence();
    float4 a = make_float4(INFINITY, INFINITY, INFINITY, 0.f), b = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
    for (unsigned k = threadIdx.x; k < gridDim.x; k += BBOX_THREADS) {
        const float4 c = __ldcg(part + 2 * k), d = __ldcg(part + 2 * k + 1);
        a.x = fminf(a.x, c.x); a.y = fminf(a.y, c.y); a.z = fminf(a.z, c.z);
        b.x = fmaxf(b.x, d.x); b.y = fmaxf(b.y, d.y); b.z = fmaxf(b.z, d.z);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a.x = fminf(a.x, __shfl_xor_sync(0xffffffffu, a.x, o));
        a.y = fminf(a.y, __shfl_xor_sync(0xffffffffu, a.y, o));
        a.z = fminf(a.z, __shfl_xor_sync(0xffffffffu, a.z, o));
        b.x = fmaxf(b.x, __shfl_xor_sync(0xffffffffu, b.x, o));
        b.y = fmaxf(b.y, __shfl_xor_sync(0xffffffffu, b.y, o));
        b.z = fmaxf(b.z, __shfl_xor_sync(0xffffffffu, b.z, o));
    }
    __syncthreads();  // smn/smx reused
    if (lane == 0) {
        smn[wid] = a;
        smx[wid] = b;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    a = smn[0];
    b = smx[0];
    for (int w = 1; w < BBOX_THREADS / 32; ++w) {
        a.x = fminf(a.x, smn[w].x); a.y = fminf(a.y, smn[w].y); a.z = fminf(a.z, smn[w].z);
        b.x = fmaxf(b.x, smx[w].x); b.y = fmaxf(b.y, smx[w].y); b.z = fmaxf(b.z, smx[w].z);
    }
    // span = largest per-axis extent (:41); 1.0 when not > 0 (:42).
    const double lo0 = a.x, lo1 = a.y, lo2 = a.z;
    double span = __dsub_rn((double)b.x, lo0);
    span = fmax(span, __dsub_rn((double)b.y, lo1));
    span = fmax(span, __dsub_rn((double)b.z, lo2));
    if (!(span > 0.0)) span = 1.0;
    const double qmax = (double)((1ull << bits) - 1ull);
    prm->lo[0] = lo0;
    prm->lo[1] = lo1;
    prm->lo[2] = lo2;
    const double scale = __ddiv_rn(qmax, __dmul_rn(span, 1.0000001));
    prm->scale = scale;
    prm->lof[0] = a.x;
    prm->lof[1] = a.y;
    prm->lof[2] = a.z;
    split_fp32(scale, prm->sh, prm->sl);
    *ticket = 0u;
}

// ---------------------------------------------------------------- morton
template <int BITS>
__device__ __forceinline__ uint64_t interleave3(uint32_t x, uint32_t y, uint32_t z) {
    uint64_t r = 0;
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
        const uint64_t t = ((x >> b) & 1u) | (((y >> b) & 1u) << 1) | (((z >> b) & 1u) << 2);
        r |= t << (3 * b);
    }
    return r;
}

// The FP64 quantisation, where FP32 cannot decide.
__device__ __noinline__ uint32_t quantise_fp64(float x, double lo, double scale, double qmax) {
    double t = __dmul_rn(__dsub_rn((double)x, lo), scale);
    t = t > qmax ? qmax : t;
    t = t >= 0.0 ? t : 0.0;  // also maps NaN to 0 (counted in the bbox pass)
    return __double2uint_rz(t);
}

// The Morton key of particle i.
template <typename KeyT, int BITS>
struct MortonKey {
    const float4 *__restrict__ xm;
    const BHParams *__restrict__ prm;

    __device__ __forceinline__ KeyT operator()(int64_t i) const {
        constexpr uint32_t QMAX = (1u << BITS) - 1u;
        const float4 x = xm[i];
        const float sh = prm->sh, sl = prm->sl;
        uint32_t qx, qy, qz;
        if (!cell_fp32(x.x, prm->lof[0], sh, sl, qx)) qx = quantise_fp64(x.x, prm->lo[0], prm->scale, (double)QMAX);
        if (!cell_fp32(x.y, prm->lof[1], sh, sl, qy)) qy = quantise_fp64(x.y, prm->lo[1], prm->scale, (double)QMAX);
        if (!cell_fp32(x.z, prm->lof[2], sh, sl, qz)) qz = quantise_fp64(x.z, prm->lo[2], prm->scale, (double)QMAX);
        return (KeyT)interleave3<BITS>(min(qx, QMAX), min(qy, QMAX), min(qz, QMAX));
    }
};

// Keys and, beside them, the digit counts of the sort (4 CTAs per SM share the
// particles, so that a CTA counts many keys before it adds them up).  1M
// particles, 30-bit keys: 11.2 us, against 35.1 us for FP64 keys alone and
// 16.4 us for a kernel that counted their digits.
template <typename KeyT, int BITS>
__global__ void __launch_bounds__(KEY_THREADS)
bh_morton_kernel(const float4 *__restrict__ xm, int64_t n, const BHParams *__restrict__ prm,
                 KeyT *__restrict__ keys, uint32_t *__restrict__ counts) {
    constexpr int PASSES = (3 * BITS + 7) / 8;
    __shared__ RsCount<PASSES> cnt;
    cnt.clear();
    const MortonKey<KeyT, BITS> key{xm, prm};
    for (int64_t i = (int64_t)blockIdx.x * KEY_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * KEY_THREADS) {
        const KeyT k = key(i);
        keys[i] = k;
        cnt.add(k, PASSES);
    }
    cnt.flush(counts, PASSES);
}

// ------------------------------------------------------------------ tree
// Common-prefix length of keys i and j over bits 62..0; equal keys continue
// with the index bits 30..0 (63 + prefix); -1 outside [0, n) (:71-81).
__device__ __forceinline__ int clz63(uint64_t x) { return __clzll(x) - 1; }
__device__ __forceinline__ int clz63(uint32_t x) { return __clz(x) + 31; }

template <typename KeyT>
__device__ __forceinline__ int kdelta(const KeyT *__restrict__ k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const KeyT x = __ldg(k + i) ^ __ldg(k + j);
    if (x == 0) return 63 + (__clz(i ^ j) - 1);
    return clz63(x);
}

// Node summary in FP32: mass, first moment about the node's AABB minimum
// corner, and the AABB.  Moments about the corner keep the centre of mass
// accurate to rounding of the node size (a cluster of coincident particles
// gets its exact position); the reference keeps FP64 moments about the
// origin (core/solvers/barnes_hut.py:143-177).
struct NodeSum {
    float m, sx, sy, sz;    // mass, moment about (lx, ly, lz)
    float lx, ly, lz, hx, hy, hz;
};

__device__ __forceinline__ NodeSum leaf_sum(float4 p) {
    NodeSum s;
    s.m = p.w;
    s.sx = s.sy = s.sz = 0.f;
    s.lx = s.hx = p.x;
    s.ly = s.hy = p.y;
    s.lz = s.hz = p.z;
    return s;
}

__device__ __forceinline__ NodeSum merge_sums(const NodeSum &a, const NodeSum &b) {
    NodeSum s;
    s.lx = fminf(a.lx, b.lx); s.ly = fminf(a.ly, b.ly); s.lz = fminf(a.lz, b.lz);
    s.hx = fmaxf(a.hx, b.hx); s.hy = fmaxf(a.hy, b.hy); s.hz = fmaxf(a.hz, b.hz);
    s.m = a.m + b.m;
    s.sx = __fmaf_rn(b.m, b.lx - s.lx, __fmaf_rn(a.m, a.lx - s.lx, a.sx + b.sx));
    s.sy = __fmaf_rn(b.m, b.ly - s.ly, __fmaf_rn(a.m, a.ly - s.ly, a.sy + b.sy));
    s.sz = __fmaf_rn(b.m, b.lz - s.lz, __fmaf_rn(a.m, a.lz - s.lz, a.sz + b.sz));
    return s;
}

// Centre of mass and mass; a node without mass keeps a zero centre, like the
// freshly allocated com field of the reference.
__device__ __forceinline__ float4 trav_com(const NodeSum &s) {
    if (!(s.m > 0.f)) return make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(s.lx + __fdiv_rn(s.sx, s.m), s.ly + __fdiv_rn(s.sy, s.m), s.lz + __fdiv_rn(s.sz, s.m), s.m);
}

// Squared largest AABB extent (:207).
__device__ __forceinline__ float size2_of(const NodeSum &s) {
    const float e = fmaxf(fmaxf(s.hx - s.lx, s.hy - s.ly), s.hz - s.lz);
    return e * e;
}

// The binary radix tree and its summaries in one kernel (the reference's
// _build_radix and summary passes, core/solvers/barnes_hut.py:84-177).
//
// The internal node that splits its leaves between g and g + 1 joins the two
// subtrees that end at g and start at g + 1, and a subtree over leaves [l, r]
// is a left child, split at r, when its keys share more with leaf r + 1 than
// with leaf l - 1, else a right child, split at l - 1 (Apetrei, "Fast and
// Simple Agglomerative LBVH Construction", 2014).  In the numbering of the
// reference (Karras) a left child has index r, a right child index l and the
// root 0.  So a node's place, parent and children follow from its leaf range
// alone, and its summary from its children's: leaves, topology and summaries
// need one pass upwards and no searches.
//
// A CTA joins its TREE_CHUNK consecutive leaves in shared memory: a subtree
// that comes to the split of its parent first stays there, and the second
// makes the parent.  While there are many parents to make they are queued and
// spread over the CTA, round by round; the last 32 each take a lane of one
// warp and go upwards on their own.  What is left are the maximal subtrees inside the chunk, at most one per tree
// level and side (a dozen or two in practice).  The last CTA of TREE_GROUP
// chunks to finish takes the subtrees of all of them as the leaves of the
// same procedure, and so on up to the root.  No floating-point atomics, and
// no CTA waits for another; the result does not depend on scheduling (the
// reference uses FP64 atomics on every ancestor).  The merge keeps its
// operands' order, so results are those of a node-by-node pass, bit for bit.
//
// Bound by latency: that of the levels in shared memory and of the hand-over
// between CTAs.  Disk, 63-bit keys to 100,000, 30-bit above (us): 10,000: 20;
// 100,000: 34; 300,000: 44; 1M: 102, against 57, 72, 98 and 211 for a gather,
// a search-based topology pass and a pass with one global arrival ticket per
// node.  Measured at 10,000 / 1M (us): tickets at every node, topology from
// ranges: 59 / 155; nodes of a chunk in queued rounds, records inside: 47 /
// 168; records apart: 27 / 129; one thread per leaf upwards instead of
// rounds: 24 / 122; rounds down to 32 nodes: 20 / 105; 4 CTAs per SM (64
// registers): 20 / 102.  128 threads: 27 / 110; 512, one CTA per SM: 18 / 152.
// So 512 threads while every unit has an SM of its own (77,824 leaves on 152
// SMs; tree stage, 256 / 512: 500: 15.0 / 12.6; 10,000: 24.6 / 22.7; 20,000:
// 35.4 / 30.9; 60,000: 35.8 / 31.6; 80,000: 37.9 / 39.3; 300,000: 47.8 / 58.8).
constexpr int TREE_THREADS = 256, TREE_WIDE = 512;  // per CTA; TREE_WIDE while every unit has an SM of its own
constexpr int TREE_CHUNK = 512;   // leaves or subtrees joined at a time
constexpr int TREE_GROUP = 32;    // units of a level that the next one joins (one per lane)
// Subtrees left of a unit: in sorted keys the common prefix grows from one to
// the next up to the longest and falls again, so 63 key bits + 31 index bits on
// each side.  Keys out of order, which an expired wait of the sort can leave,
// may keep any number apart (alternating ones all 512): those past the bound are
// dropped and counted as bad_tree.
constexpr int TREE_PEND = 192;
// Leaves per group of the group walk (traversal shape 3).
constexpr int GW_GROUP = 32;

// A finished subtree over leaves [l, r] and the common prefixes beyond its ends.
struct alignas(16) TreeItem {
    NodeSum s;
    int l, r, dl, dr;
};

struct TreeArgs {
    const float4 *xm;
    const uint32_t *order;
    int n;
    float4 *leaf;
    int2 *child;
    int *parent;
    // Subtrees left of every unit (level after level, TREE_PEND each), their
    // number, and the finished units of every group (zero at launch).
    TreeItem *items;
    int *count;
    unsigned *done;
    float4 *sums, *bmin, *bmax, *inode, *root;
    // The group walk's groups, when it is asked for (NULL or zero at launch):
    // the maximal subtrees with at most GW_GROUP leaves; gsize[first leaf] =
    // its leaf count.  They partition the leaves into key-order ranges, each
    // inside one node's box (32 key-consecutive leaves can straddle a jump of
    // the Morton curve and span most of the system).
    int *gsize;
    unsigned long long *diag;
};

// Writes the node of leaves [l, r] split at p, with index k; s: its summary, a
// and b: its children's.  The traversal record of k holds its two children as
// (left, right) pairs:
//   inode[3k] = {x_L, x_R, y_L, y_R}, inode[3k+1] = {z_L, z_R, m_L, m_R},
//   inode[3k+2] = {size2_L, size2_R, id_L, id_R} (ids as bits; size2 = -1
//   marks a leaf child), pre-packed for .f32x2 arithmetic.
__device__ __forceinline__ void tree_record(const TreeArgs &t, const NodeSum &s, const NodeSum &a, const NodeSum &b,
                                            int l, int r, int p, int k) {
    const int n = t.n;
    const int lc = l == p ? p : p + n, rc = r == p + 1 ? r : p + 1 + n;
    t.child[k] = make_int2(lc, rc);
    t.parent[lc] = k + n;
    t.parent[rc] = k + n;
    t.sums[k] = make_float4(s.m, s.sx, s.sy, s.sz);
    t.bmin[k] = make_float4(s.lx, s.ly, s.lz, 0.f);
    t.bmax[k] = make_float4(s.hx, s.hy, s.hz, 0.f);
    const float4 ca = trav_com(a), cb = trav_com(b);
    t.inode[3 * (int64_t)k] = make_float4(ca.x, cb.x, ca.y, cb.y);
    t.inode[3 * (int64_t)k + 1] = make_float4(ca.z, cb.z, ca.w, cb.w);
    t.inode[3 * (int64_t)k + 2] = make_float4(l == p ? -1.f : size2_of(a), r == p + 1 ? -1.f : size2_of(b),
                                              __int_as_float(lc), __int_as_float(rc));
    const bool is_root = l == 0 && r == n - 1;
    if (is_root) {
        t.root[0] = trav_com(s);
        t.root[1] = make_float4(size2_of(s), 0.f, 0.f, 0.f);
        t.parent[n] = -1;
    }
    if (t.gsize) {
        const int cnt = r - l + 1, cl = p - l + 1, cr = r - p;
        if (cnt > GW_GROUP) {
            if (cl <= GW_GROUP) t.gsize[l] = cl;
            if (cr <= GW_GROUP) t.gsize[p + 1] = cr;
        } else if (is_root) {
            t.gsize[0] = cnt;  // the whole system is one group
        }
    }
}

struct TreeShared {
    // Summaries: of the leaves or subtrees to join (the items), then of the
    // nodes above them, each at the place of its first or last item (as the
    // node is a right or a left child), whose own summary is then in use no
    // more except in the records.
    float sum[10][TREE_CHUNK];
    float4 leaf[TREE_CHUNK];                  // the items, while they are leaves
    int first[TREE_CHUNK], last[TREE_CHUNK];  // their leaf ranges
    // Per split (j lies before item j; 0 and m are the outer ones): 1 + the
    // first item of the left child that came, and 1 + the last item of the
    // right one in the upper half.
    unsigned came[TREE_CHUNK + 1];
    signed char delta[TREE_CHUNK + 1];        // per split: common prefix of the leaves beside it
    unsigned queue[2][TREE_CHUNK / 2];        // nodes to make: first item | last item << 10 | split << 20
    int queued[3];
    short end[TREE_CHUNK];
    int scan[TREE_CHUNK / 32];
    int before[TREE_GROUP + 1];               // subtrees of the units before each one of a group
    bool last_unit;

    __device__ __forceinline__ NodeSum get(int i) const {
        NodeSum s;
        s.m = sum[0][i]; s.sx = sum[1][i]; s.sy = sum[2][i]; s.sz = sum[3][i];
        s.lx = sum[4][i]; s.ly = sum[5][i]; s.lz = sum[6][i];
        s.hx = sum[7][i]; s.hy = sum[8][i]; s.hz = sum[9][i];
        return s;
    }
    __device__ __forceinline__ void put(int i, const NodeSum &s) {
        sum[0][i] = s.m; sum[1][i] = s.sx; sum[2][i] = s.sy; sum[3][i] = s.sz;
        sum[4][i] = s.lx; sum[5][i] = s.ly; sum[6][i] = s.lz;
        sum[7][i] = s.hx; sum[8][i] = s.hy; sum[9][i] = s.hz;
    }
};

// The subtree over the items [a, b] comes to the split of its parent (not the
// root).  Returns whether it is the second there: then [a, b] is the parent's
// range and j its split.
__device__ __forceinline__ bool tree_come(TreeShared &w, bool left, int &a, int &b, int &j) {
    j = left ? b + 1 : a;
    __threadfence_block();  // its summary first
    const unsigned old = atomicOr(&w.came[j], left ? (unsigned)(a + 1) : (unsigned)(b + 1) << 16);
    const int sib = (int)(left ? old >> 16 : old & 0xFFFFu) - 1;
    if (sib < 0) return false;  // the sibling is not there yet, or lies outside
    __threadfence_block();
    if (left) b = sib;
    else a = sib;
    return true;
}

// Makes the node over the items [a, b], split at j; false for the root.
__device__ __forceinline__ bool tree_make(TreeShared &w, int a, int b, int j, bool &left) {
    const int da = w.delta[a], db = w.delta[b + 1];
    left = db > da;
    w.put(left ? b : a, merge_sums(w.get(j - 1), w.get(j)));
    return da >= 0 || db >= 0;
}

// Joins the m items in w (summaries, leaf ranges, deltas; m >= 1) as far as
// they reach.  Complete after the barrier at its end.
template <int THREADS>
__device__ __forceinline__ void tree_join(TreeShared &w, int m) {
    const int tid = threadIdx.x;
    for (int i = tid; i <= m; i += THREADS) w.came[i] = 0u;
    if (tid < 3) w.queued[tid] = 0;
    __syncthreads();
    auto push = [&](int a, int b, int j, int q, int c) {
        w.queue[q][atomicAdd(&w.queued[c], 1)] = (unsigned)a | (unsigned)b << 10 | (unsigned)j << 20;
    };
    for (int i = tid; i < m; i += THREADS) {
        int a = i, b = i, j;
        const int da = w.delta[i], db = w.delta[i + 1];
        if ((da >= 0 || db >= 0) && tree_come(w, db > da, a, b, j)) push(a, b, j, 0, 0);
    }
    __syncthreads();
    int q = 0, c = 0;
    for (;;) {
        const int ready = w.queued[c], c1 = c == 2 ? 0 : c + 1;
        if (ready <= 32) break;
        if (tid == 0) w.queued[c1 == 2 ? 0 : c1 + 1] = 0;  // read one round ago, used by the next one
        for (int i = tid; i < ready; i += THREADS) {
            const unsigned e = w.queue[q][i];
            int a = (int)(e & 1023u), b = (int)(e >> 10 & 1023u), j = (int)(e >> 20);
            bool left;
            if (tree_make(w, a, b, j, left) && tree_come(w, left, a, b, j)) push(a, b, j, q ^ 1, c1);
        }
        __syncthreads();
        q ^= 1;
        c = c1;
    }
    if (tid < w.queued[c]) {  // 32 at most: a lane each
        const unsigned e = w.queue[q][tid];
        int a = (int)(e & 1023u), b = (int)(e >> 10 & 1023u), j = (int)(e >> 20);
        bool left;
        while (tree_make(w, a, b, j, left) && tree_come(w, left, a, b, j)) {
        }
    }
    __syncthreads();
}

// The records of the nodes that tree_join made; base(i): the summary of item
// i.  Apart from the joining, because the divisions of the centres and the 13
// stores of a node would lengthen every level.
template <int THREADS, typename F>
__device__ __forceinline__ void tree_records(const TreeShared &w, const TreeArgs &t, int m, F base) {
    for (int j = threadIdx.x + 1; j < m; j += THREADS) {
        const int a = (int)(w.came[j] & 0xFFFFu) - 1, b = (int)(w.came[j] >> 16) - 1;
        if (a < 0 || b < 0) continue;
        const int da = w.delta[a], db = w.delta[b + 1], l = w.first[a], r = w.last[b];
        const bool left = db > da;
        const NodeSum x = a == j - 1 ? base(a) : w.get(j - 1), y = b == j ? base(b) : w.get(j);
        tree_record(t, w.get(left ? b : a), x, y, l, r, w.last[j - 1], da < 0 && db < 0 ? 0 : left ? r : l);
    }
}

// Writes the subtrees that are left, in leaf order, to dst; returns how many,
// TREE_PEND at most.
template <int THREADS>
__device__ __forceinline__ int tree_left(TreeShared &w, TreeItem *dst, int m, unsigned long long *diag) {
    constexpr int PER = TREE_CHUNK / THREADS;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < TREE_CHUNK; i += THREADS) w.end[i] = 0;  // 1 + the last item of the subtree from here
    __syncthreads();
    for (int j = tid; j <= m; j += THREADS) {
        const int a = (int)(w.came[j] & 0xFFFFu) - 1, b = (int)(w.came[j] >> 16) - 1;
        if (a >= 0 && b < 0) w.end[a] = (short)j;
        else if (b >= 0 && a < 0) w.end[j] = (short)(b + 1);
    }
    __syncthreads();
    int own = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) own += w.end[tid * PER + q] != 0;
    int inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) w.scan[wid] = inc;
    __syncthreads();
    int at = inc - own, total = 0;
#pragma unroll
    for (int k = 0; k < THREADS / 32; ++k) {
        if (k < wid) at += w.scan[k];
        total += w.scan[k];
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int a = tid * PER + q, b = w.end[a] - 1;
        if (b < 0) continue;
        TreeItem x;
        x.dl = w.delta[a];
        x.dr = w.delta[b + 1];
        x.s = w.get(x.dr > x.dl ? b : a);
        x.l = w.first[a];
        x.r = w.last[b];
        if (at < TREE_PEND) dst[at] = x;
        ++at;
    }
    if (total <= TREE_PEND) return total;
    if (tid == 0) atomicAdd(diag + DIAG_BAD_TREE, (unsigned long long)(total - TREE_PEND));
    return TREE_PEND;
}

__device__ __forceinline__ void tree_take(TreeShared &w, const TreeItem &x, int i, bool last) {
    w.put(i, x.s);
    w.first[i] = x.l;
    w.last[i] = x.r;
    w.delta[i] = (signed char)x.dl;
    if (last) w.delta[i + 1] = (signed char)x.dr;
}

__device__ __forceinline__ TreeItem load_item(const TreeItem *p) {  // written by other CTAs: read past L1
    static_assert(sizeof(TreeItem) == 64, "four 16-byte loads");
    union {
        float4 v[4];
        TreeItem x;
    } u;
#pragma unroll
    for (int k = 0; k < 4; ++k) u.v[k] = __ldcg(reinterpret_cast<const float4 *>(p) + k);
    return u.x;
}

template <typename KeyT, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == TREE_WIDE ? 1 : 4)
bh_tree_kernel(const KeyT *__restrict__ keys, TreeArgs t) {
    __shared__ TreeShared w;
    const int tid = threadIdx.x, n = t.n;
    int unit = blockIdx.x, units = gridDim.x, base = 0, groups = 0;  // units and groups of the levels below
    int m = min(TREE_CHUNK, n - unit * TREE_CHUNK);
    for (int i = tid; i <= m; i += THREADS) {
        const int g = unit * TREE_CHUNK + i;
        w.delta[i] = g >= 1 ? (signed char)kdelta(keys, n, g - 1, g) : (signed char)-1;
        if (i == m) continue;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t.order) {
            const uint32_t o = t.order[g];
            if (o < (uint32_t)n) x = __ldg(t.xm + o);
            else atomicAdd(t.diag + DIAG_BAD_TREE, 1ull);
            t.leaf[g] = x;
        } else {
            x = t.leaf[g];
        }
        w.leaf[i] = x;
        w.put(i, leaf_sum(x));
        w.first[i] = w.last[i] = g;
    }
    if (n == 1) {  // the root is the leaf
        if (tid == 0) t.parent[0] = t.parent[1] = -1;
        return;
    }
    __syncthreads();
    tree_join<THREADS>(w, m);
    if (units == 1) {
        tree_records<THREADS>(w, t, m, [&](int i) { return leaf_sum(w.leaf[i]); });
        return;
    }
    TreeItem *items = nullptr;  // the items of levels above the leaves
    bool apart = true;          // unit u's at items[u * TREE_PEND ..], not back to back
    auto item = [&](int i) {
        if (!apart) return items + i;
        int u = 0;
#pragma unroll
        for (int o = TREE_GROUP / 2; o > 0; o >>= 1)
            if (i >= w.before[u + o]) u += o;
        return items + u * TREE_PEND + (i - w.before[u]);
    };
    auto above = [&](int i) { return load_item(item(i)).s; };
    for (int level = 0; units > 1; ++level) {
        const int left = tree_left<THREADS>(w, t.items + (int64_t)(base + unit) * TREE_PEND, m, t.diag);
        // The last unit of the group to finish goes on with all of its
        // subtrees; the records are written while that is being found out.
        static_assert(TREE_GROUP == 32, "one unit of a group per lane");
        const int group = unit / TREE_GROUP, gn = min(TREE_GROUP, units - group * TREE_GROUP);
        __syncthreads();
        if (tid == 0) {
            t.count[base + unit] = left;
            __threadfence();
            w.last_unit = atomicAdd(t.done + groups + group, 1u) == (unsigned)(gn - 1);
        }
        if (level == 0) tree_records<THREADS>(w, t, m, [&](int i) { return leaf_sum(w.leaf[i]); });
        else tree_records<THREADS>(w, t, m, above);
        __syncthreads();
        if (!w.last_unit) return;
        __threadfence();
        if (tid < 32) {
            int c = tid < gn ? __ldcg(t.count + base + group * TREE_GROUP + tid) : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, c, o);
                if (tid >= o) c += v;
            }
            w.before[tid + 1] = c;
            if (tid == 0) w.before[0] = 0;
        }
        __syncthreads();
        items = t.items + (int64_t)(base + group * TREE_GROUP) * TREE_PEND;
        apart = true;
        int total = w.before[TREE_GROUP];
        // More than fit (trees far deeper than log2 n): join them piece by
        // piece; what a piece leaves goes back to the front of the same
        // storage.  A full piece leaves at most TREE_PEND of TREE_CHUNK items,
        // so every sweep leaves fewer than it took, whatever the keys.
        static_assert(TREE_PEND < TREE_CHUNK, "a sweep ends with fewer items");
        while (total > TREE_CHUNK) {
            int out = 0;
            for (int i0 = 0; i0 < total; i0 += TREE_CHUNK) {
                m = min(TREE_CHUNK, total - i0);
                __syncthreads();
                for (int i = tid; i < m; i += THREADS) tree_take(w, load_item(item(i0 + i)), i, i == m - 1);
                __syncthreads();
                tree_join<THREADS>(w, m);
                tree_records<THREADS>(w, t, m, [&](int i) { return load_item(item(i0 + i)).s; });
                __syncthreads();  // the items are read
                out += tree_left<THREADS>(w, items + out, m, t.diag);
            }
            __syncthreads();
            __threadfence();
            apart = false;
            total = out;
        }
        __syncthreads();
        m = total;
        for (int i = tid; i < m; i += THREADS) tree_take(w, load_item(item(i)), i, i == m - 1);
        __syncthreads();
        tree_join<THREADS>(w, m);
        base += units;
        groups += (units + TREE_GROUP - 1) / TREE_GROUP;
        unit = group;
        units = (units + TREE_GROUP - 1) / TREE_GROUP;
    }
    tree_records<THREADS>(w, t, m, above);
}

// Units and groups of all levels for n leaves.
static void tree_units(int64_t n, int64_t *units, int64_t *groups) {
    *units = *groups = 0;
    for (int64_t u = (n + TREE_CHUNK - 1) / TREE_CHUNK; u > 1; u = (u + TREE_GROUP - 1) / TREE_GROUP) {
        *units += u;
        *groups += (u + TREE_GROUP - 1) / TREE_GROUP;
    }
}

}  // namespace gb

#include "gb_bh_traverse.cuh"

namespace gb {

// ----------------------------------------------------------------- export
// Tree arrays in the reference's layout for parity checks.
enum ExportWhat {
    EXP_CODES = 0,   // uint64[n]  keys in sorted order
    EXP_ORDER = 1,   // int32[n]
    EXP_LEFT = 2,    // int32[n-1]
    EXP_RIGHT = 3,   // int32[n-1]
    EXP_PARENT = 4,  // int32[2n-1]
    EXP_MASS = 5,    // double[2n-1]
    EXP_COM = 6,     // double[2n-1][3]
    EXP_MIN = 7,     // double[2n-1][3]
    EXP_MAX = 8      // double[2n-1][3]
};

template <typename KeyT>
__global__ void bh_export_kernel(int what, int n, const KeyT *keys, const uint32_t *order, const int2 *child,
                                 const int *parent, const float4 *leaf, const float4 *sums, const float4 *bmin,
                                 const float4 *bmax, void *dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nodes = 2 * (int64_t)n - 1;
    switch (what) {
        case EXP_CODES:
            if (i < n) ((uint64_t *)dst)[i] = (uint64_t)keys[i];
            break;
        case EXP_ORDER:
            if (i < n) ((int *)dst)[i] = (int)order[i];
            break;
        case EXP_LEFT:
            if (i < n - 1) ((int *)dst)[i] = child[i].x;
            break;
        case EXP_RIGHT:
            if (i < n - 1) ((int *)dst)[i] = child[i].y;
            break;
        case EXP_PARENT:
            if (i < nodes) ((int *)dst)[i] = i < n ? parent[i] : parent[i];
            break;
        default: {
            if (i >= nodes) break;
            double m, c[3], lo[3], hi[3];
            if (i < n) {
                const float4 p = leaf[i];
                m = p.w;
                c[0] = lo[0] = hi[0] = p.x;
                c[1] = lo[1] = hi[1] = p.y;
                c[2] = lo[2] = hi[2] = p.z;
            } else {
                const int k = (int)(i - n);
                const float4 q = sums[k];
                m = q.x;
                lo[0] = bmin[k].x; lo[1] = bmin[k].y; lo[2] = bmin[k].z;
                c[0] = m > 0.0 ? lo[0] + q.y / m : 0.0;
                c[1] = m > 0.0 ? lo[1] + q.z / m : 0.0;
                c[2] = m > 0.0 ? lo[2] + q.w / m : 0.0;
                hi[0] = bmax[k].x; hi[1] = bmax[k].y; hi[2] = bmax[k].z;
            }
            double *o = (double *)dst;
            if (what == EXP_MASS) o[i] = m;
            else {
                const double *src = what == EXP_COM ? c : (what == EXP_MIN ? lo : hi);
                o[3 * i] = src[0];
                o[3 * i + 1] = src[1];
                o[3 * i + 2] = src[2];
            }
        }
    }
}

}  // namespace gb

// ================================================================ C ABI
using namespace gb;

struct gb_bh {
    int device, sms;
    int64_t n_max;
    int key_bits;
    int64_t n;  // n of the last build (-1: none)
    // Radix ping-pong.  Every sort ends in pair 0, whatever n is: a replayed
    // graph sorts again without passing through the host code.
    void *keys[2];
    uint32_t *vals[2];
    uint32_t *sort_scratch;  // radix_scratch_size(n_max) words
    float4 *bbox_part;
    int bbox_blocks;
    unsigned *ticket;
    BHParams *prm;
    float4 *leaf;
    int2 *child;
    int *parent;
    TreeItem *tree_items;  // scratch of the build between chunks
    int *tree_count;
    unsigned *tree_done;
    float4 *sums;
    float4 *bmin, *bmax;
    float4 *inode;
    float4 *root;
    unsigned long long *diag;
    // Stage timing (gb_bh_timing): events recorded on the launch stream at
    // stage boundaries, GB_BH_STAGES + 1 per step, reused cyclically.
    int timing;
    int ev_used;
    cudaEvent_t ev[GB_BH_TIMING_STEPS * (GB_BH_STAGES + 1)];
    uint64_t launches;  // kernels launched by this handle (host count)
    int pending_slot;   // timing slot of the last gb_bh_build
    int tpl;            // traversal shape: -1 .. 2 the particle walk, 3 the group walk
    // One KDK step captured as a CUDA graph (gb_bh_kdk), replayed per step
    // on the handle's own stream and joined to the caller's by events.
    // gexec[0]: a plain step; gexec[1]: a step that also writes the tree
    // potential (gb_bh_kdk_phi); each captured again when its key changes.
    int use_graph;
    cudaStream_t gstream;
    cudaEvent_t gev_in, gev_out;
    cudaGraphExec_t gexec[2];
    struct Key {
        const void *xm, *vel, *acc, *phi;
        int64_t n;
        float theta, eps2, G, dt;
        int max_stack, tpl;
        bool operator==(const Key &o) const {
            return xm == o.xm && vel == o.vel && acc == o.acc && phi == o.phi && n == o.n && theta == o.theta &&
                   eps2 == o.eps2 && G == o.G && dt == o.dt && max_stack == o.max_stack && tpl == o.tpl;
        }
    } gkey[2];
    uint64_t graph_launches[2];  // kernels in each captured step
    int64_t graph_groups[2];     // groups_n after each captured step
    double2 *epart;              // energy block partials (gb_bh_energy)
    int epart_cap;
    int *gsize;                  // group-walk groups of the last build (mode 3)
    int64_t groups_n;            // n of the build that marked them (-1: none)
    // Failure checks (GB_CHECK, gb_bh_set_check): the failure counters as
    // read by the last checked call (or zero after a diag reset).
    int check;
    unsigned long long seen[DIAG_COUNT];  // failure counters at the last checked call
};

static void mark(gb_bh_t *h, int step_slot, int stage, cudaStream_t s) {
    if (!h->timing) return;
    cudaEventRecord(h->ev[step_slot * (GB_BH_STAGES + 1) + stage], s);
}

static size_t key_size(int bits) { return bits <= 10 ? sizeof(uint32_t) : sizeof(uint64_t); }

extern "C" int gb_bh_destroy(gb_bh_t *h) {
    if (!h) return GB_OK;
    void *ptrs[] = {h->keys[0], h->keys[1], h->vals[0], h->vals[1], h->sort_scratch, h->bbox_part, h->ticket,
                    h->prm, h->leaf, h->child, h->parent, h->tree_items, h->tree_count, h->tree_done, h->sums, h->bmin, h->bmax,
                    h->inode, h->root, h->diag, h->epart, h->gsize};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    for (auto &g : h->gexec)
        if (g) cudaGraphExecDestroy(g);
    if (h->gev_in) cudaEventDestroy(h->gev_in);
    if (h->gev_out) cudaEventDestroy(h->gev_out);
    if (h->gstream) cudaStreamDestroy(h->gstream);
    for (auto &e : h->ev)
        if (e) cudaEventDestroy(e);
    delete h;
    return GB_OK;
}

extern "C" int gb_bh_create(gb_bh_t **out, int64_t n_max, int key_bits) {
    if (!out) return fail(GB_EINVAL, "out is NULL");
    *out = nullptr;
    if (n_max < 1 || n_max > RS_MAX_N) return fail(GB_EINVAL, "n_max=%lld out of range", (long long)n_max);
    if (key_bits != 10 && key_bits != 21) return fail(GB_EINVAL, "key_bits must be 10 or 21 (got %d)", key_bits);
    gb_bh_t *h = new gb_bh();
    GB_CUDA_TRY(cudaGetDevice(&h->device));
    h->sms = num_sms();
    h->n_max = n_max;
    h->key_bits = key_bits;
    h->tpl = -1;
    h->use_graph = 1;
    h->n = -1;
    const int64_t nn = n_max, ni = std::max<int64_t>(n_max - 1, 1), nodes = 2 * n_max;
    h->bbox_blocks = std::max(1, std::min(h->sms * 4, (int)((n_max + BBOX_THREADS - 1) / BBOX_THREADS)));
    bool ok = true;
    auto A = [&](void **p, size_t bytes) {
        if (ok && cudaMalloc(p, bytes) != cudaSuccess) ok = false;
    };
    A(&h->keys[0], key_size(key_bits) * nn);
    A(&h->keys[1], key_size(key_bits) * nn);
    A((void **)&h->vals[0], sizeof(uint32_t) * nn);
    A((void **)&h->vals[1], sizeof(uint32_t) * nn);
    A((void **)&h->sort_scratch, sizeof(uint32_t) * radix_scratch_size(n_max));
    A((void **)&h->bbox_part, sizeof(float4) * 2 * h->bbox_blocks);
    A((void **)&h->ticket, sizeof(unsigned));
    A((void **)&h->prm, sizeof(BHParams));
    A((void **)&h->leaf, sizeof(float4) * nn);
    A((void **)&h->child, sizeof(int2) * ni);
    A((void **)&h->parent, sizeof(int) * nodes);
    int64_t units, groups;
    tree_units(n_max, &units, &groups);
    A((void **)&h->tree_items, sizeof(TreeItem) * TREE_PEND * std::max<int64_t>(units, 1));
    A((void **)&h->tree_count, sizeof(int) * std::max<int64_t>(units, 1));
    A((void **)&h->tree_done, sizeof(unsigned) * std::max<int64_t>(groups, 1));
    A((void **)&h->sums, sizeof(float4) * ni);
    A((void **)&h->bmin, sizeof(float4) * ni);
    A((void **)&h->bmax, sizeof(float4) * ni);
    A((void **)&h->inode, sizeof(float4) * 3 * ni);
    A((void **)&h->root, sizeof(float4) * 2);
    A((void **)&h->diag, sizeof(unsigned long long) * DIAG_COUNT);
    h->epart_cap = 4 * h->sms;
    A((void **)&h->epart, sizeof(double2) * (h->epart_cap + ENERGY_EXTRA));
    A((void **)&h->gsize, sizeof(int) * nn);
    h->groups_n = -1;
    if (!ok) {
        gb_bh_destroy(h);
        return fail(GB_ENOMEM, "gb_bh_create: device allocation failed for n_max=%lld", (long long)n_max);
    }
    if (cudaMemset(h->ticket, 0, sizeof(unsigned)) != cudaSuccess ||
        cudaMemset(h->diag, 0, sizeof(unsigned long long) * DIAG_COUNT) != cudaSuccess ||
        cudaMemset(h->epart, 0, sizeof(double2) * (h->epart_cap + ENERGY_EXTRA)) != cudaSuccess) {
        gb_bh_destroy(h);
        return fail(GB_ECUDA, "gb_bh_create: memset failed");
    }
    *out = h;
    return GB_OK;
}

// The tree over the handle's sorted keys; groups: also marks the group walk's
// groups.  order: the particles of xm in key order; NULL: the leaves are there
// already.  h->tree_done (and h->gsize) are zero.
template <typename KeyT>
static int build_tree(gb_bh_t *h, const float4 *xm, const uint32_t *order, int64_t n, bool groups, cudaStream_t s) {
    TreeArgs t;
    t.xm = xm;
    t.order = order;
    t.n = (int)n;
    t.leaf = h->leaf;
    t.child = h->child;
    t.parent = h->parent;
    t.items = h->tree_items;
    t.count = h->tree_count;
    t.done = h->tree_done;
    t.sums = h->sums;
    t.bmin = h->bmin;
    t.bmax = h->bmax;
    t.inode = h->inode;
    t.root = h->root;
    t.gsize = groups ? h->gsize : nullptr;
    t.diag = h->diag;
    const unsigned grid = (unsigned)((n + TREE_CHUNK - 1) / TREE_CHUNK);
    const KeyT *keys = (const KeyT *)h->keys[0];
    if (grid <= (unsigned)h->sms) bh_tree_kernel<KeyT, TREE_WIDE><<<grid, TREE_WIDE, 0, s>>>(keys, t);
    else bh_tree_kernel<KeyT, TREE_THREADS><<<grid, TREE_THREADS, 0, s>>>(keys, t);
    GB_CUDA_TRY(cudaGetLastError());
    h->groups_n = groups ? n : -1;
    h->launches += 1;
    return GB_OK;
}

template <typename KeyT, int BITS>
static int build_impl(gb_bh_t *h, float4 *xm, float4 *vel, const float4 *acc, int64_t n, float dt, bool kdk,
                      cudaStream_t s, int slot) {
    mark(h, slot, 0, s);
    const int nblk = std::max(1, std::min(h->bbox_blocks, (int)((n + BBOX_THREADS - 1) / BBOX_THREADS)));
    // The sort's scratch, the tree's finished units and the group walk's marks.
    constexpr int passes = (3 * BITS + 7) / 8;
    static_assert(passes % 2 == 0, "the sorted keys are in pair 0");
    const bool groups = h->tpl == 3, small = radix_small(n, passes);
    int64_t units, ngroups;
    tree_units(n, &units, &ngroups);
    const ZeroWords zero = {{h->sort_scratch, h->tree_done, (uint32_t *)h->gsize},
                            {small ? 0 : radix_zero_words(n), ngroups, groups ? n : 0}};
    if (kdk)
        bh_bbox_kernel<true><<<nblk, BBOX_THREADS, 0, s>>>(xm, vel, acc, n, 0.5f * dt, dt, h->bbox_part, h->ticket,
                                                           h->prm, BITS, zero, h->diag);
    else
        bh_bbox_kernel<false><<<nblk, BBOX_THREADS, 0, s>>>(xm, nullptr, nullptr, n, 0.f, 0.f, h->bbox_part,
                                                            h->ticket, h->prm, BITS, zero, h->diag);
    KeyT *kk[2] = {(KeyT *)h->keys[0], (KeyT *)h->keys[1]};
    if (small) {
        mark(h, slot, 1, s);
        radix_sort_small<KeyT>(MortonKey<KeyT, BITS>{xm, h->prm}, kk, h->vals, n, s);
    } else {
        const unsigned gk = std::min((unsigned)(h->sms * 4), (unsigned)((n + KEY_THREADS - 1) / KEY_THREADS));
        bh_morton_kernel<KeyT, BITS><<<gk, KEY_THREADS, 0, s>>>(xm, n, h->prm, kk[0], h->sort_scratch);
        mark(h, slot, 1, s);
        radix_sort_counted<KeyT>(kk, h->vals, n, passes, h->sort_scratch, h->diag, s);
    }
    mark(h, slot, 2, s);
    // The group walk's groups are marked when the handle walks groups.
    GB_TRY(build_tree<KeyT>(h, xm, h->vals[0], n, groups, s));
    mark(h, slot, 3, s);
    GB_CUDA_TRY(cudaGetLastError());
    mark(h, slot, 4, s);
    h->launches += small ? 1 + radix_small_launches(n) : 2 + passes;
    h->n = n;
    return GB_OK;
}

static int next_slot(gb_bh_t *h) {
    if (!h->timing) return 0;
    const int slot = h->ev_used % GB_BH_TIMING_STEPS;
    ++h->ev_used;
    return slot;
}

static int build_any(gb_bh_t *h, float4 *xm, float4 *vel, const float4 *acc, int64_t n, float dt, bool kdk,
                     cudaStream_t s, int slot) {
    if (h->key_bits == 10) return build_impl<uint32_t, 10>(h, xm, vel, acc, n, dt, kdk, s, slot);
    return build_impl<uint64_t, 21>(h, xm, vel, acc, n, dt, kdk, s, slot);
}

static int check_bh(gb_bh_t *h, int64_t n) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (n < 0 || n > h->n_max) return fail(GB_EINVAL, "n=%lld outside [0, n_max=%lld]", (long long)n, (long long)h->n_max);
    return GB_OK;
}

static int check_ptr(const void *p, const char *name) {
    if (!p) return fail(GB_EINVAL, "%s is NULL", name);
    if (!aligned16(p)) return fail(GB_EINVAL, "%s is not 16-byte aligned", name);
    return GB_OK;
}

// Dispatches L<KDK, COUNT, PHI>::go(args...) on run-time flags.
template <template <bool, bool, bool> class L, typename... Args>
static void dispatch3(bool kdk, bool count, bool phi, Args... args) {
    const int sel = (kdk ? 4 : 0) + (count ? 2 : 0) + (phi ? 1 : 0);
    switch (sel) {
        case 0: L<false, false, false>::go(args...); break;
        case 1: L<false, false, true>::go(args...); break;
        case 2: L<false, true, false>::go(args...); break;
        case 3: L<false, true, true>::go(args...); break;
        case 4: L<true, false, false>::go(args...); break;
        case 5: L<true, false, true>::go(args...); break;
        case 6: L<true, true, false>::go(args...); break;
        default: L<true, true, true>::go(args...); break;
    }
}
template <bool KDK, bool COUNT, bool PHI>
struct GroupLaunch {
    static void go(unsigned grid, const TravArgs *a, const int *gsize, float *phi, int2 r, cudaStream_t s) {
        bh_group_kernel<KDK, COUNT, PHI><<<grid, GW_WARPS * 32, 0, s>>>(*a, gsize, phi, r.x, r.y);
    }
};
template <bool KDK, bool COUNT, bool PHI>
struct ShortWalkLaunch {
    static void go(WalkForm form, int2 r, const TravArgs *a, float *phi, cudaStream_t s) {
        const int64_t nt = (int64_t)r.y - r.x;
        if (form == WALK_WARP) {
            constexpr int T = WARP_WALK_WARPS * 32;
            bh_warp_walk_kernel<KDK, COUNT, PHI><<<(unsigned)((nt + T - 1) / T), T, 0, s>>>(*a, phi, r.x, r.y);
        } else {
            constexpr int T = LANE_WALK_THREADS;
            const int room = std::min(a->max_stack, LANE_WALK_STACK);
            bh_lane_walk_kernel<KDK, COUNT, PHI>
                <<<(unsigned)((nt + T - 1) / T), T, sizeof(unsigned) * room * T, s>>>(*a, phi, r.x, r.y, room);
        }
    }
};
template <bool KDK, bool COUNT, bool PHI>
struct WalkLaunch {
    template <int T>
    static void run(int2 r, const TravArgs *a, float *phi, cudaStream_t s) {
        const int64_t groups = ((int64_t)r.y - r.x + T - 1) / T;
        bh_walk_kernel<KDK, COUNT, PHI, T><<<(unsigned)((groups + WALK_WARPS - 1) / WALK_WARPS), WALK_WARPS * 32,
                                             WALK_WARPS * sizeof(WalkWarp<T>), s>>>(*a, phi, r.x, r.y);
    }
    static void go(int group, int2 r, const TravArgs *a, float *phi, cudaStream_t s) {
        if (group == 4) run<4>(r, a, phi, s);
        else if (group == 8) run<8>(r, a, phi, s);
        else if (group == 16) run<16>(r, a, phi, s);
        else run<32>(r, a, phi, s);
    }
};

// The traversal of the last build: accelerations into acc (KDK: the
// closing kick into vel too) and, when phi is not NULL, the tree potential
// sums into phi.
// Targets: key-order indices [s0, s1) (s1 < 0: all n).
static int traverse(gb_bh_t *h, float4 *acc, float4 *vel, float *phi, float theta, float eps2, float G, float dt,
                    int max_stack, int flags, bool kdk, cudaStream_t s, int slot, const ExtPot &pot = ExtPot{},
                    int64_t s0 = 0, int64_t s1 = -1) {
    const int64_t n = h->n;
    if (n <= 0) return GB_OK;
    if (s1 < 0) s1 = n;
    if (s1 <= s0) return GB_OK;
    const int64_t nt = s1 - s0;
    const int2 range = make_int2((int)s0, (int)s1);  // key-order targets [s0, s1)
    TravArgs a;
    a.leaf = h->leaf;
    a.inode = h->inode;
    a.root = h->root;
    a.order = h->vals[0];
    a.acc = acc;
    a.vel = vel;
    a.n = (int)n;
    a.theta2 = theta * theta;
    a.eps2 = eps2;
    a.G = G;
    a.h = 0.5f * dt;
    a.max_stack = max_stack;
    a.accumulate = (flags & GB_ACCUMULATE) ? 1 : 0;
    a.diag = h->diag;
    a.pot = pot;
    const bool count = (flags & GB_COUNT_WORK) != 0;
    if (h->tpl == 3) {
        const int64_t warps = (nt + 31) / 32;
        const unsigned grid = (unsigned)((warps + GW_WARPS - 1) / GW_WARPS);
        if (h->groups_n != n) {
            // Built in another traversal mode: mark the groups by a second
            // pass over the same build (identical values).
            GB_CUDA_TRY(cudaMemsetAsync(h->gsize, 0, sizeof(int) * n, s));
            int64_t units, groups;
            tree_units(n, &units, &groups);
            GB_CUDA_TRY(cudaMemsetAsync(h->tree_done, 0, sizeof(unsigned) * groups, s));
            if (h->key_bits == 10) GB_TRY(build_tree<uint32_t>(h, nullptr, nullptr, n, true, s));
            else GB_TRY(build_tree<uint64_t>(h, nullptr, nullptr, n, true, s));
        }
        dispatch3<GroupLaunch>(kdk, count, phi != nullptr, grid, &a, (const int *)h->gsize, phi, range, s);
    } else if (const WalkForm form = walk_form(n, theta); form != WALK_ROUNDS) {
        dispatch3<ShortWalkLaunch>(kdk, count, phi != nullptr, form, range, &a, phi, s);
    } else {
        const int group = n < WALK_4_N ? 4 : n < WALK_8_N ? 8 : n < WALK_16_N ? 16 : 32;
        dispatch3<WalkLaunch>(kdk, count, phi != nullptr, group, range, &a, phi, s);
    }
    GB_CUDA_TRY(cudaGetLastError());
    mark(h, slot, 5, s);
    h->launches += 1;
    return GB_OK;
}

// Synchronises `s` and compares the failure counters (stack drops, stack
// overflow, non-finite positions, bad tree, expired waits) with the values
// the last check saw: anything counted since then fails the call.
// Non-finite positions and index guards give GB_EINVAL, an expired wait
// GB_ETIMEOUT, dropped or overflowed pushes GB_ESTACK.
static int check_failures(gb_bh_t *h, cudaStream_t s, const char *call) {
    unsigned long long d[DIAG_COUNT];
    GB_CUDA_TRY(cudaMemcpyAsync(d, h->diag, sizeof(d), cudaMemcpyDeviceToHost, s));
    GB_CUDA_TRY(cudaStreamSynchronize(s));
    unsigned long long inc[DIAG_COUNT];
    for (int k = 0; k < DIAG_COUNT; ++k) {
        inc[k] = d[k] - h->seen[k];
        h->seen[k] = d[k];
    }
    if (inc[DIAG_NONFINITE])
        return fail(GB_EINVAL, "%s: %llu non-finite particle positions", call, inc[DIAG_NONFINITE]);
    if (inc[DIAG_BAD_TREE])
        return fail(GB_EINVAL, "%s: inconsistent tree (%llu index guards taken)", call, inc[DIAG_BAD_TREE]);
    if (inc[DIAG_WAIT_TIMEOUT])
        return fail(GB_ETIMEOUT, "%s: %llu bounded device waits expired (radix sort look-back)", call,
                    inc[DIAG_WAIT_TIMEOUT]);
    if (inc[DIAG_STACK_DROPS] || inc[DIAG_STACK_OVERFLOW])
        return fail(GB_ESTACK, "%s: the max_stack rule dropped %llu pushes; %llu overflowed the traversal stack",
                    call, inc[DIAG_STACK_DROPS], inc[DIAG_STACK_OVERFLOW]);
    return GB_OK;
}

static int check_params(float theta, float eps2, int max_stack) {
    if (!(theta >= 0.f)) return fail(GB_EINVAL, "theta must be >= 0");
    if (!(eps2 > 0.f)) return fail(GB_EINVAL, "eps2 must be > 0");
    if (max_stack < 1) return fail(GB_EINVAL, "max_stack must be >= 1");
    return GB_OK;
}

extern "C" int gb_bh_build(gb_bh_t *h, const float *xm, int64_t n, void *stream) {
    GB_TRY(check_bh(h, n));
    if (n == 0) {
        h->n = 0;
        return GB_OK;
    }
    GB_TRY(check_ptr(xm, "xm"));
    h->pending_slot = next_slot(h);
    return build_any(h, (float4 *)xm, nullptr, nullptr, n, 0.f, false, (cudaStream_t)stream, h->pending_slot);
}

extern "C" int gb_bh_accel(gb_bh_t *h, float *acc, float theta, float eps2, float G, int max_stack, int flags,
                           void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (h->n < 0) return fail(GB_ENOTREADY, "gb_bh_accel before gb_bh_build");
    if (h->n == 0) return GB_OK;
    GB_TRY(check_ptr(acc, "acc"));
    GB_TRY(check_params(theta, eps2, max_stack));
    GB_TRY(traverse(h, (float4 *)acc, nullptr, nullptr, theta, eps2, G, 0.f, max_stack, flags, false,
                    (cudaStream_t)stream, h->pending_slot));
    if ((flags & GB_CHECK) || h->check) return check_failures(h, (cudaStream_t)stream, "gb_bh_accel");
    return GB_OK;
}

extern "C" int gb_bh_accel_range(gb_bh_t *h, float *acc, float *phi, int64_t s0, int64_t ns, float theta,
                                 float eps2, float G, int max_stack, int flags, void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (h->n < 0) return fail(GB_ENOTREADY, "gb_bh_accel_range before gb_bh_build");
    if (s0 < 0 || ns < 0 || s0 > h->n || ns > h->n - s0)
        return fail(GB_EINVAL, "target range [%lld, %lld) outside the %lld particles of the last build",
                    (long long)s0, (long long)(s0 + ns), (long long)h->n);
    if (flags & ~(GB_ACCUMULATE | GB_CHECK))
        return fail(GB_EINVAL, "gb_bh_accel_range: flags 0x%x: only GB_ACCUMULATE and GB_CHECK apply", flags);
    if (ns == 0) return GB_OK;
    GB_TRY(check_ptr(acc, "acc"));
    GB_TRY(check_params(theta, eps2, max_stack));
    GB_TRY(traverse(h, (float4 *)acc, nullptr, phi, theta, eps2, G, 0.f, max_stack, flags, false,
                    (cudaStream_t)stream, h->pending_slot, ExtPot{}, s0, s0 + ns));
    if ((flags & GB_CHECK) || h->check) return check_failures(h, (cudaStream_t)stream, "gb_bh_accel_range");
    return GB_OK;
}

extern "C" int gb_bh_accel_phi(gb_bh_t *h, float *acc, float *phi, float theta, float eps2, float G, int max_stack,
                               int flags, void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (h->n < 0) return fail(GB_ENOTREADY, "gb_bh_accel_phi before gb_bh_build");
    if (h->n == 0) return GB_OK;
    GB_TRY(check_ptr(acc, "acc"));
    if (!phi) return fail(GB_EINVAL, "phi is NULL");
    GB_TRY(check_params(theta, eps2, max_stack));
    GB_TRY(traverse(h, (float4 *)acc, nullptr, phi, theta, eps2, G, 0.f, max_stack, flags, false,
                    (cudaStream_t)stream, h->pending_slot));
    if ((flags & GB_CHECK) || h->check) return check_failures(h, (cudaStream_t)stream, "gb_bh_accel_phi");
    return GB_OK;
}

extern "C" int gb_bh_accel_ext(gb_bh_t *h, float *acc, float theta, float eps2, float G, int max_stack,
                               const gb_potential_t *pot, int flags, void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    ExtPot ep;
    GB_TRY(make_extpot(pot, G, &ep));
    if (h->n < 0) return fail(GB_ENOTREADY, "gb_bh_accel_ext before gb_bh_build");
    if (h->n == 0) return GB_OK;
    GB_TRY(check_ptr(acc, "acc"));
    GB_TRY(check_params(theta, eps2, max_stack));
    GB_TRY(traverse(h, (float4 *)acc, nullptr, nullptr, theta, eps2, G, 0.f, max_stack, flags, false,
                    (cudaStream_t)stream, h->pending_slot, ep));
    if ((flags & GB_CHECK) || h->check) return check_failures(h, (cudaStream_t)stream, "gb_bh_accel_ext");
    return GB_OK;
}

extern "C" int gb_bh_compute(gb_bh_t *h, const float *xm, float *acc, int64_t n, float theta, float eps2, float G,
                             int max_stack, int flags, void *stream) {
    GB_TRY(check_bh(h, n));
    if (n > 0) {
        GB_TRY(check_ptr(acc, "acc"));
        GB_TRY(check_params(theta, eps2, max_stack));
    }
    GB_TRY(gb_bh_build(h, xm, n, stream));
    return gb_bh_accel(h, acc, theta, eps2, G, max_stack, flags, stream);
}

// One KDK step: tree build with the fused kick and drift, then the traversal
// with the closing kick (and the tree potential of the new positions when
// phi is not NULL).
static int kdk_step(gb_bh_t *h, float4 *xm, float4 *vel, float4 *acc, float *phi, int64_t n, float theta,
                    float eps2, float G, float dt, int max_stack, cudaStream_t s) {
    const int slot = next_slot(h);
    GB_TRY(build_any(h, xm, vel, acc, n, dt, true, s, slot));
    return traverse(h, acc, vel, phi, theta, eps2, G, dt, max_stack, 0, true, s, slot);
}

// Graph slot g (0 plain, 1 with the potential) holds one captured step with
// this key, captured again when the key changed.
static int ensure_graph(gb_bh_t *h, int g, const gb_bh::Key &key, float4 *x, float4 *v, float4 *a, float *phi,
                        int64_t n, float theta, float eps2, float G, float dt, int max_stack) {
    if (h->gexec[g] && h->gkey[g] == key) return GB_OK;
    if (h->gexec[g]) cudaGraphExecDestroy(h->gexec[g]);
    h->gexec[g] = nullptr;
    GB_CUDA_TRY(cudaStreamBeginCapture(h->gstream, cudaStreamCaptureModeThreadLocal));
    // What a step leaves on the handle is true once it has run: it is noted
    // here and set after the replay.
    const uint64_t l0 = h->launches;
    const int64_t n0 = h->n, groups0 = h->groups_n;
    const int st = kdk_step(h, x, v, a, phi, n, theta, eps2, G, dt, max_stack, h->gstream);
    h->graph_launches[g] = h->launches - l0;
    h->graph_groups[g] = h->groups_n;
    h->launches = l0;
    h->n = n0;
    h->groups_n = groups0;
    cudaGraph_t graph = nullptr;
    const cudaError_t e = cudaStreamEndCapture(h->gstream, &graph);
    if (st != GB_OK) {
        if (graph) cudaGraphDestroy(graph);
        return st;
    }
    if (e != cudaSuccess) return fail(GB_ECUDA, "graph capture: %s", cudaGetErrorString(e));
    const cudaError_t ei = cudaGraphInstantiate(&h->gexec[g], graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) {
        h->gexec[g] = nullptr;
        return fail(GB_ECUDA, "graph instantiate: %s", cudaGetErrorString(ei));
    }
    h->gkey[g] = key;
    return GB_OK;
}

// nsteps KDK steps; with phi, the last step also writes the tree potential.
static int bh_kdk_impl(gb_bh_t *h, float *xm, float *vel, float *acc, float *phi, int64_t n, float theta, float eps2,
                       float G, float dt, int64_t nsteps, int max_stack, void *stream, const char *call) {
    GB_TRY(check_bh(h, n));
    if (nsteps < 0) return fail(GB_EINVAL, "nsteps < 0");
    if (n == 0 || nsteps == 0) return GB_OK;
    GB_TRY(check_ptr(xm, "xm"));
    GB_TRY(check_ptr(vel, "vel"));
    GB_TRY(check_ptr(acc, "acc"));
    GB_TRY(check_params(theta, eps2, max_stack));
    cudaStream_t s = (cudaStream_t)stream;
    float4 *x = (float4 *)xm, *v = (float4 *)vel, *a = (float4 *)acc;
    if (!h->use_graph || h->timing) {
        for (int64_t k = 0; k < nsteps; ++k)
            GB_TRY(kdk_step(h, x, v, a, k == nsteps - 1 ? phi : nullptr, n, theta, eps2, G, dt, max_stack, s));
        return h->check ? check_failures(h, s, call) : GB_OK;
    }
    if (!h->gstream) {
        GB_CUDA_TRY(cudaStreamCreateWithFlags(&h->gstream, cudaStreamNonBlocking));
        GB_CUDA_TRY(cudaEventCreateWithFlags(&h->gev_in, cudaEventDisableTiming));
        GB_CUDA_TRY(cudaEventCreateWithFlags(&h->gev_out, cudaEventDisableTiming));
    }
    const int64_t plain_steps = phi ? nsteps - 1 : nsteps;
    gb_bh::Key key{xm, vel, acc, nullptr, n, theta, eps2, G, dt, max_stack, h->tpl};
    if (plain_steps) GB_TRY(ensure_graph(h, 0, key, x, v, a, nullptr, n, theta, eps2, G, dt, max_stack));
    if (phi) {
        key.phi = phi;
        GB_TRY(ensure_graph(h, 1, key, x, v, a, phi, n, theta, eps2, G, dt, max_stack));
    }
    GB_CUDA_TRY(cudaEventRecord(h->gev_in, s));
    GB_CUDA_TRY(cudaStreamWaitEvent(h->gstream, h->gev_in, 0));
    for (int64_t k = 0; k < plain_steps; ++k) GB_CUDA_TRY(cudaGraphLaunch(h->gexec[0], h->gstream));
    if (phi) GB_CUDA_TRY(cudaGraphLaunch(h->gexec[1], h->gstream));
    GB_CUDA_TRY(cudaEventRecord(h->gev_out, h->gstream));
    GB_CUDA_TRY(cudaStreamWaitEvent(s, h->gev_out, 0));
    h->launches += h->graph_launches[0] * (uint64_t)plain_steps + (phi ? h->graph_launches[1] : 0);
    h->n = n;
    h->groups_n = h->graph_groups[phi ? 1 : 0];  // of the step replayed last
    return h->check ? check_failures(h, s, call) : GB_OK;
}

extern "C" int gb_bh_kdk(gb_bh_t *h, float *xm, float *vel, float *acc, int64_t n, float theta, float eps2, float G,
                         float dt, int64_t nsteps, int max_stack, void *stream) {
    return bh_kdk_impl(h, xm, vel, acc, nullptr, n, theta, eps2, G, dt, nsteps, max_stack, stream, "gb_bh_kdk");
}

extern "C" int gb_bh_kdk_phi(gb_bh_t *h, float *xm, float *vel, float *acc, float *phi, int64_t n, float theta,
                             float eps2, float G, float dt, int64_t nsteps, int max_stack, void *stream) {
    if (!phi && n > 0 && nsteps > 0) return fail(GB_EINVAL, "phi is NULL");
    return bh_kdk_impl(h, xm, vel, acc, phi, n, theta, eps2, G, dt, nsteps, max_stack, stream, "gb_bh_kdk_phi");
}

extern "C" int gb_bh_energy(gb_bh_t *h, const float *xm, const float *vel, const float *phi, int64_t n, float G,
                            double *out3, void *stream) {
    GB_TRY(check_bh(h, n));
    if (n > 0) {
        GB_TRY(check_ptr(xm, "xm"));
        GB_TRY(check_ptr(vel, "vel"));
        if (!phi) return fail(GB_EINVAL, "phi is NULL");
    }
    if (!out3) return fail(GB_EINVAL, "out3 is NULL");
    GB_TRY(launch_energy((const float4 *)xm, (const float4 *)vel, phi, n, G, h->epart, h->epart_cap, out3,
                         (cudaStream_t)stream));
    h->launches += 1;
    return GB_OK;
}

// One CTA runs the radix sort's look-back for tile t (1: the first of its
// group's earlier tiles is tile 0; RS_GROUP: the first tile behind a whole
// group) of a status array of t + 1 tiles, digit d in thread d; every earlier
// tile counts d.  publish = 0: one earlier tile has not published, so every
// wait runs out after spin_limit polls; 1: all have; 2 (t = RS_GROUP): the
// group's inclusive prefix is there and its sum is not.
__global__ void sort_wait_probe_kernel(uint32_t *status, int t, int spin_limit, int publish, uint32_t *excl,
                                       unsigned long long *diag) {
    const int d = threadIdx.x;
    const RsStatus st(status, t + 1);
    for (int k = 0; k < (publish ? t : t - 1); ++k) rs_publish(st, k, d, (uint32_t)d);
    if (publish == 2) {
        rs_lookback(st, t - 1, d, (uint32_t)d, spin_limit, diag);  // publishes the group's prefix
        st_relaxed_gpu(st.gsum + d, 0u);
    }
    rs_publish(st, t, d, 1u);
    excl[d] = rs_lookback(st, t, d, 1u, spin_limit, diag);
}

static int sort_wait_probe(const char *call, int t, int spin_limit, int publish, uint32_t *excl_out,
                           uint64_t *timeouts_out) {
    if (spin_limit < 1 || spin_limit > RS_SPIN_LIMIT)
        return fail(GB_EINVAL, "spin_limit must be in [1, %d] (got %d)", RS_SPIN_LIMIT, spin_limit);
    if (!excl_out || !timeouts_out) return fail(GB_EINVAL, "NULL argument");
    uint32_t *status = nullptr, *excl = nullptr;
    unsigned long long *diag = nullptr;
    const size_t bytes = sizeof(uint32_t) * radix_status_words((int64_t)(t + 1) * RS_TILE);
    int rc = GB_OK;
    if (cudaMalloc(&status, bytes) != cudaSuccess || cudaMalloc(&excl, sizeof(uint32_t) * RS_BINS) != cudaSuccess ||
        cudaMalloc(&diag, sizeof(unsigned long long) * DIAG_COUNT) != cudaSuccess) {
        rc = fail(GB_ENOMEM, "%s: device allocation failed", call);
    }
    if (rc == GB_OK && (cudaMemset(status, 0, bytes) != cudaSuccess ||
                        cudaMemset(diag, 0, sizeof(unsigned long long) * DIAG_COUNT) != cudaSuccess))
        rc = fail(GB_ECUDA, "%s: memset failed", call);
    if (rc == GB_OK) {
        sort_wait_probe_kernel<<<1, RS_BINS>>>(status, t, spin_limit, publish, excl, diag);
        unsigned long long d[DIAG_COUNT];
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
            cudaMemcpy(excl_out, excl, sizeof(uint32_t) * RS_BINS, cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(d, diag, sizeof(d), cudaMemcpyDeviceToHost) != cudaSuccess) {
            rc = fail(GB_ECUDA, "%s: %s", call, cudaGetErrorString(cudaGetLastError()));
        } else {
            *timeouts_out = (uint64_t)d[DIAG_WAIT_TIMEOUT];
            if (d[DIAG_WAIT_TIMEOUT]) rc = fail(GB_ETIMEOUT, "%s: %llu waits expired", call, d[DIAG_WAIT_TIMEOUT]);
        }
    }
    if (status) cudaFree(status);
    if (excl) cudaFree(excl);
    if (diag) cudaFree(diag);
    return rc;
}

extern "C" int gb_sort_wait_probe(int spin_limit, int publish_first, uint32_t *excl_out, uint64_t *timeouts_out) {
    return sort_wait_probe("gb_sort_wait_probe", 1, spin_limit, publish_first ? 1 : 0, excl_out, timeouts_out);
}

extern "C" int gb_sort_group_wait_probe(int spin_limit, int publish, uint32_t *excl_out, uint64_t *timeouts_out) {
    if (publish < 0 || publish > 2) return fail(GB_EINVAL, "publish must be 0, 1 or 2 (got %d)", publish);
    return sort_wait_probe("gb_sort_group_wait_probe", RS_GROUP, spin_limit, publish, excl_out, timeouts_out);
}

extern "C" int gb_bh_tree_probe(gb_bh_t *h, const float *xm, const void *keys, const uint32_t *order, int64_t n,
                                void *stream) {
    GB_TRY(check_bh(h, n));
    if (n < 1) return fail(GB_EINVAL, "n must be >= 1");
    GB_TRY(check_ptr(xm, "xm"));
    if (!keys || !order) return fail(GB_EINVAL, "NULL argument");
    cudaStream_t s = (cudaStream_t)stream;
    const bool groups = h->tpl == 3;
    int64_t units, ngroups;
    tree_units(n, &units, &ngroups);
    GB_CUDA_TRY(cudaMemcpyAsync(h->keys[0], keys, key_size(h->key_bits) * n, cudaMemcpyDeviceToDevice, s));
    GB_CUDA_TRY(cudaMemcpyAsync(h->vals[0], order, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s));
    GB_CUDA_TRY(cudaMemsetAsync(h->tree_done, 0, sizeof(unsigned) * ngroups, s));
    if (groups) GB_CUDA_TRY(cudaMemsetAsync(h->gsize, 0, sizeof(int) * n, s));
    if (h->key_bits == 10) GB_TRY(build_tree<uint32_t>(h, (const float4 *)xm, h->vals[0], n, groups, s));
    else GB_TRY(build_tree<uint64_t>(h, (const float4 *)xm, h->vals[0], n, groups, s));
    h->n = n;
    return GB_OK;
}

extern "C" int gb_bh_set_check(gb_bh_t *h, int on) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    h->check = on ? 1 : 0;
    return GB_OK;
}

extern "C" int gb_bh_set_graph(gb_bh_t *h, int on) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    h->use_graph = on ? 1 : 0;
    return GB_OK;
}

extern "C" int gb_bh_export(gb_bh_t *h, int what, void *dst, void *stream) {
    if (!h || !dst) return fail(GB_EINVAL, "NULL argument");
    if (h->n < 1) return fail(GB_ENOTREADY, "no tree built");
    if (what < EXP_CODES || what > EXP_MAX) return fail(GB_EINVAL, "unknown export %d", what);
    const int n = (int)h->n;
    const int64_t count = 2 * (int64_t)n;
    const unsigned grid = (unsigned)((count + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    if (h->key_bits == 10)
        bh_export_kernel<uint32_t><<<grid, 256, 0, s>>>(what, n, (const uint32_t *)h->keys[0], h->vals[0],
                                                        h->child, h->parent, h->leaf, h->sums, h->bmin, h->bmax, dst);
    else
        bh_export_kernel<uint64_t><<<grid, 256, 0, s>>>(what, n, (const uint64_t *)h->keys[0], h->vals[0],
                                                        h->child, h->parent, h->leaf, h->sums, h->bmin, h->bmax, dst);
    GB_CUDA_TRY(cudaGetLastError());
    return GB_OK;
}

extern "C" int gb_bh_diag(gb_bh_t *h, gb_diag_t *out, int reset) {
    if (!h || !out) return fail(GB_EINVAL, "NULL argument");
    GB_TRY(read_diag(h->diag, out, reset));
    if (reset)
        for (auto &v : h->seen) v = 0;
    return GB_OK;
}

extern "C" int gb_bh_timing(gb_bh_t *h, int enable) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (enable && !h->ev[0]) {
        for (auto &e : h->ev) GB_CUDA_TRY(cudaEventCreate(&e));
    }
    h->timing = enable ? 1 : 0;
    h->ev_used = 0;
    return GB_OK;
}

extern "C" int gb_bh_stage_times(gb_bh_t *h, float *ms, int *steps) {
    if (!h || !ms || !steps) return fail(GB_EINVAL, "NULL argument");
    for (int k = 0; k < GB_BH_STAGES; ++k) ms[k] = 0.f;
    const int used = std::min(h->ev_used, GB_BH_TIMING_STEPS);
    GB_CUDA_TRY(cudaDeviceSynchronize());
    for (int st = 0; st < used; ++st)
        for (int k = 0; k < GB_BH_STAGES; ++k) {
            float t = 0.f;
            GB_CUDA_TRY(cudaEventElapsedTime(&t, h->ev[st * (GB_BH_STAGES + 1) + k],
                                             h->ev[st * (GB_BH_STAGES + 1) + k + 1]));
            ms[k] += t;
        }
    *steps = used;
    h->ev_used = 0;
    return GB_OK;
}

extern "C" uint64_t gb_bh_launch_count(gb_bh_t *h) { return h ? h->launches : 0; }

extern "C" int gb_bh_set_traversal(gb_bh_t *h, int targets_per_lane) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (targets_per_lane < -1 || targets_per_lane > 3)
        return fail(GB_EINVAL, "traversal mode must be -1, 0, 1, 2 or 3 (got %d)", targets_per_lane);
    h->tpl = targets_per_lane;
    return GB_OK;
}
