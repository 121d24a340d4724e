// Tree traversal kernels of the LBVH Barnes-Hut path (included by gb_bh.cu,
// which builds the tree they walk):
//   bh_walk_kernel   the per-particle walk (traversal shapes -1, 0, 1, 2):
//                    each particle accepts exactly the node set of the
//                    reference's _traverse (core/solvers/barnes_hut.py:
//                    180-217)
//   bh_lane_walk_kernel, bh_warp_walk_kernel
//                    the same walk, one node at a time, for large opening
//                    angles, with the same results
//   bh_group_kernel  the opt-in group walk (a refinement of each target's
//                    node set, one walk per leaf group)
// Node records: inode[3k .. 3k+2] = the two children of internal node k as
// (left, right) pairs {x, y, z, m, size^2, id}; root[0..1] = the root's.
#pragma once

#include "gb_common.cuh"

namespace gb {

// --------------------------------------------------------------- traverse
struct TravArgs {
    const float4 *__restrict__ leaf;
    const float4 *__restrict__ inode;
    const float4 *__restrict__ root;
    const uint32_t *__restrict__ order;
    float4 *acc;
    float4 *vel;
    int n;
    float theta2, eps2, G, h;
    int max_stack;
    int accumulate;
    unsigned long long *diag;
    ExtPot pot;  // analytic potential added in the epilogue (pot.on)
};

// The acceleration G s of particle p, the analytic potential's added (and the
// closing kick), written at its own index: the traversals' epilogue.
template <bool KDK>
__device__ __forceinline__ void trav_write(const TravArgs &a, uint32_t p, float px, float py, float pz, float sx,
                                           float sy, float sz) {
    float gx = a.G * sx, gy = a.G * sy, gz = a.G * sz;
    if (a.pot.on) ext_acc_add(a.pot, px, py, pz, gx, gy, gz);
    if (KDK) {
        const float4 vh = a.vel[p];
        a.vel[p] = make_float4(kick(vh.x, gx, a.h), kick(vh.y, gy, a.h), kick(vh.z, gz, a.h), vh.w);
        a.acc[p] = make_float4(gx, gy, gz, 0.f);
    } else if (a.accumulate) {
        float4 o = a.acc[p];
        o.x += gx; o.y += gy; o.z += gz;
        a.acc[p] = o;
    } else {
        a.acc[p] = make_float4(gx, gy, gz, 0.f);
    }
}

// ----------------------------------------------------------- particle walk
// Per-particle walk: T key-consecutive targets share a warp.  The nodes that
// some target opened form a list in the order of the reference's walk (a
// node, then its right subtree, then its left one); a round
//   expands  up to 32 unexpanded nodes of the list, the first ones, one per
//            lane: loads their two-children records and applies the
//            reference's own test size^2 < theta^2 (|d|^2 + eps^2)
//            (core/solvers/barnes_hut.py:204-210) of both children to all T
//            targets, two targets per .f32x2 instruction, broadcast from
//            shared memory.  An expanded node keeps the masks of the targets
//            that accepted its children; an opened child enters the list
//            behind it;
//   emits    the expanded nodes at the list's head, up to the first
//            unexpanded one, into a buffer of records;
//   sums     a full buffer: every lane adds the records, in order, to its
//            target; children outside the target's mask add zero.
// So every target sums exactly the node set of the reference's _traverse
// (:180-217), its accepted left children and its accepted right children
// each in the order of the reference's walk, whatever its group: results
// depend neither on T, nor on the range of targets, nor on scheduling.
//
// Leaves carry size^2 = -1 in the record, so the one comparison accepts every
// leaf.  A target's own leaf (:198) sits at distance 0 and adds a zero force.
// depth is the depth of the reference's per-particle stack when the node is
// popped; it depends only on the node's path (a right child is popped at
// depth + 1, a left child at depth), so the max_stack rule (:212) holds per
// node, and the skipped pushes of all its targets are counted.
//
// The list cannot overflow: a round expands no more nodes than half the free
// elements above WALK_RESERVE (an expanded node stays until it is emitted and
// adds at most two), and at least one, the first, which the next round emits;
// single expansions are a depth-first walk, which needs at most one more
// element per tree level (63 key bits + 31 index bits) and two in all.
//
// Bound by issue: 67% of the slots at n = 400,000, the FMA pipe at 55%, the
// shared-memory pipe at 69%.  1M disk, theta 0.5: 2.35 ms, against 3.40 ms for
// a walk that expanded one node per warp step (74 instructions for 32
// targets' tests and terms of a record, 61% of the lanes in use for the
// tests and 31% for the terms); 100,000: 218 against 442 us; 10,000, theta
// 0.6: 48 against 129 us for one walk per lane.  A round's test costs 344
// instructions for 32 records, a summed record 23.  Measured on the disk:
//   - T by n (us, theta 0.5): 4,000: 41.1 (T = 4), 44.3 (8); 8,000: 52.0,
//     54.0; 12,000: 60.8 (8), 69.6 (16); 25,000: 87.6, 87.2; 50,000: 123
//     (16), 157 (32); 70,000: 172, 172; 150,000: 346, 330; 1M: 2.69 ms, 2.35.
//     Small groups give a small system more warps and shorter rounds, large
//     ones share records and rounds among more targets.
//   - CAP 512 with 10 CTAs per SM: 2.53 ms at 1M before the last two items,
//     608 with 8: 2.64, 448 with 11: 2.61 (a short list expands fewer nodes
//     per round, 24 of 32 lanes at 512).
//   - a node that no target accepted a child of leaves the list: 2.82 to
//     2.64 ms with the sums below it.
//   - the buffer's sums and the list's chase between the record loads and the
//     tests, emitted records stored a round later: 2.51 and 2.38 ms; eight
//     records unrolled in the sums: 2.35.
//   - asynchronous copies of the emitted records: 2.34 ms, but 6% slower below
//     100,000; not kept.
//   - sums in round order instead of the reference's: 1.71 ms, but the last
//     bits then depend on the group, and over several steps a changed last
//     bit flips acceptance tests; not kept.
// Targets per group by n: 4, 8, 16 below these, then 32.
constexpr int64_t WALK_4_N = 8192, WALK_8_N = 20480, WALK_16_N = 65536;
constexpr int WALK_WARPS = 2;
constexpr int WALK_RESERVE = 100;
constexpr int WALK_LIST = 32;  // buffered records per warp
// Greatest depth of an element, the 7 bits below the expanded flag.  A consistent
// tree has 63 key bits + 31 index bits; in any other the depth stays there and
// the bound on the rounds ends the walk.  (A branch for each of these two guards
// took 1.3% of the walk at 1M, a minimum each takes nothing.)
constexpr int WALK_DEPTH = 0x7F;
template <int T>
struct WalkShape {
    static constexpr int CAP = 512;  // list elements; the last one ends the list
    static constexpr int CTAS = T == 32 ? 10 : 11;   // resident CTAs per SM
};

template <int T>
struct WalkWarp {
    static constexpr int CAP = WalkShape<T>::CAP;
    float4 tx[T / 4], ty[T / 4], tz[T / 4];  // the targets
    // Buffered records: T = 32 the record's own {x_L, x_R, y_L, y_R} and
    // {z_L, z_R, m_L, m_R}, else the left and the right child {x, y, z, m}.
    float4 ra[WALK_LIST], rb[WALK_LIST];
    uint2 rm[T == 32 ? WALK_LIST : 1];          // masks (left, right)
    unsigned rmask[T == 32 ? 1 : WALK_LIST];    // left | right << T
    // The list: node, masks (unexpanded: targets that opened it; expanded:
    // that accepted the left and right child), next element, and flags
    // (unexpanded: depth; expanded: 0x80).
    int ek[CAP];
    unsigned ea[CAP];
    unsigned eb[T == 32 ? CAP : 1];
    unsigned short nx[CAP];
    // Free elements from the front; unexpanded ones, in list order, at the back.
    unsigned short sf[CAP];
    unsigned char fl[CAP];
};

// Two targets against one node: shifts the outcomes (1: accepted) of the
// second and the first into the mask.  size^2 < t is the sign of size^2 - t,
// which rounding keeps (a NaN's is positive: not accepted).  The difference
// is an FMA by -1 (NEG, not known to the compiler), because the compiler
// contracts a packed product and difference into one rounding.
__device__ __forceinline__ unsigned walk_test(unsigned mask, f2 x, f2 y, f2 z, f2 TX, f2 TY, f2 TZ, f2 S2, f2 E2,
                                              f2 TH2, f2 NEG) {
    const f2 dx = sub2(x, TX), dy = sub2(y, TY), dz = sub2(z, TZ);
    f2 r2 = fma2(dx, dx, E2);
    r2 = fma2(dy, dy, r2);
    r2 = fma2(dz, dz, r2);
    float d0, d1;
    unpack2(fma2(mul2(TH2, r2), NEG, S2), d0, d1);
    mask = __funnelshift_l(__float_as_uint(d1), mask, 1);
    return __funnelshift_l(__float_as_uint(d0), mask, 1);
}

// A lane's sums.  T = 32: packed over the (left, right) children; else the
// lane's own side in the low half.
struct WalkSum {
    f2 X, Y, Z, W;
};

// Adds the buffered records [0, cnt) to the lane's target at (px, py, pz).
template <bool PHI, int T>
__device__ __forceinline__ void walk_eval(const WalkWarp<T> &w, int cnt, int lane, float px, float py, float pz,
                                          float eps2, WalkSum &s) {
    if constexpr (T == 32) {
        const f2 PX = pack2(px, px), PY = pack2(py, py), PZ = pack2(pz, pz), E2 = pack2(eps2, eps2);
        const unsigned bit = 1u << lane;
        const ulonglong2 *RA = reinterpret_cast<const ulonglong2 *>(w.ra),
                         *RB = reinterpret_cast<const ulonglong2 *>(w.rb);
#pragma unroll 8
        for (int i = 0; i < cnt; ++i) {
            const ulonglong2 A = RA[i], B = RB[i];
            const uint2 k = w.rm[i];
            const f2 dx = sub2(A.x, PX), dy = sub2(A.y, PY), dz = sub2(B.x, PZ);
            f2 r2 = fma2(dx, dx, E2);
            r2 = fma2(dy, dy, r2);
            r2 = fma2(dz, dz, r2);
            const f2 inv = rsqrt2(r2);
            float c0, c1;
            unpack2(mul2(mul2(B.y, inv), mul2(inv, inv)), c0, c1);
            const f2 sc = pack2((k.x & bit) ? c0 : 0.f, (k.y & bit) ? c1 : 0.f);
            s.X = fma2(sc, dx, s.X);
            s.Y = fma2(sc, dy, s.Y);
            s.Z = fma2(sc, dz, s.Z);
            if (PHI) s.W = fma2(sc, r2, s.W);
        }
    } else {
        const unsigned bit = 1u << (lane & (2 * T - 1));
        const float4 *R = (lane & T) ? w.rb : w.ra;
        float sx, sy, sz, sw, none;
        unpack2(s.X, sx, none);
        unpack2(s.Y, sy, none);
        unpack2(s.Z, sz, none);
        unpack2(s.W, sw, none);
#pragma unroll 8
        for (int i = 0; i < cnt; ++i) {
            const float4 q = R[i];
            const unsigned k = w.rmask[i];
            const float dx = __fsub_rn(q.x, px), dy = __fsub_rn(q.y, py), dz = __fsub_rn(q.z, pz);
            const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, eps2)));
            const float inv = rsqrt_approx(r2);
            const float c = __fmul_rn(__fmul_rn(q.w, inv), __fmul_rn(inv, inv));
            const float sc = (k & bit) ? c : 0.f;
            sx = __fmaf_rn(sc, dx, sx);
            sy = __fmaf_rn(sc, dy, sy);
            sz = __fmaf_rn(sc, dz, sz);
            if (PHI) sw = __fmaf_rn(sc, r2, sw);
        }
        s.X = pack2(sx, 0.f);
        s.Y = pack2(sy, 0.f);
        s.Z = pack2(sz, 0.f);
        s.W = pack2(sw, 0.f);
    }
}

// left + right sum of a lane's target.
template <int T>
__device__ __forceinline__ float walk_total(f2 v) {
    float lo, hi;
    unpack2(v, lo, hi);
    if (T < 32) hi = __shfl_xor_sync(0xffffffffu, lo, T);
    return lo + hi;
}

template <bool KDK, bool COUNT, bool PHI, int T>
__global__ void __launch_bounds__(WALK_WARPS * 32, WalkShape<T>::CTAS)
bh_walk_kernel(TravArgs a, float *__restrict__ phi, int s0, int s1) {
    constexpr int CAP = WalkShape<T>::CAP, END = CAP - 1;
    extern __shared__ __align__(16) unsigned char walk_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    WalkWarp<T> &w = reinterpret_cast<WalkWarp<T> *>(walk_smem)[wid];
    const int n = a.n;
    const int g0 = s0 + (blockIdx.x * WALK_WARPS + wid) * T;  // the group's first target
    if (g0 >= s1) return;  // whole warp out of range
    const int gn = min(T, s1 - g0);
    // The lane's target: g0 + t (T < 32: its left side in lanes t, its right
    // side in lanes t + T).
    const int t = lane & (T - 1);
    float px = 0.f, py = 0.f, pz = 0.f, pm = 0.f;
    if (t < gn) {
        const float4 p = __ldg(a.leaf + g0 + t);
        px = p.x; py = p.y; pz = p.z; pm = p.w;
    }
    if (lane < T) {
        reinterpret_cast<float *>(w.tx)[lane] = px;
        reinterpret_cast<float *>(w.ty)[lane] = py;
        reinterpret_cast<float *>(w.tz)[lane] = pz;
    }
    const f2 E2 = pack2(a.eps2, a.eps2), TH2 = pack2(a.theta2, a.theta2);
    const float neg = __int_as_float((int)0xBF800000 | (n >> 30));  // -1 (n < 2^30)
    const f2 NEG = pack2(neg, neg);
    const unsigned lt = (1u << lane) - 1u;
    WalkSum sum;
    sum.X = sum.Y = sum.Z = sum.W = 0ull;
    unsigned drops = 0, bad = 0, reads = 0, n_int = 0, n_test = 0, self = 0;
    float ax = 0.f, ay = 0.f, az = 0.f, aw = 0.f;  // the root's term
    int ns = 0;     // unexpanded elements, the first at sf[CAP - ns]
    int nfree = 0;  // free elements in sf[0 .. nfree)
    int fresh = 0;  // elements never used: fresh .. END - 1
    int head = END, live = 0, cnt = 0;
    if (n >= 2) {
        // The root is popped first, with an empty stack (depth 0).
        const float4 R0 = __ldg(a.root), R1 = __ldg(a.root + 1);
        const float dx = R0.x - px, dy = R0.y - py, dz = R0.z - pz;
        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, a.eps2)));
        const bool acc = R1.x < a.theta2 * r2;
        if (acc) {
            const float inv = rsqrt_approx(r2);
            const float sc = R0.w * inv * inv * inv;
            ax = __fmul_rn(sc, dx);
            ay = __fmul_rn(sc, dy);
            az = __fmul_rn(sc, dz);
            aw = R0.w * inv;
        }
        const bool mine = lane < gn;
        unsigned om = __ballot_sync(0xffffffffu, mine && !acc);
        if (COUNT && lane == 0) {
            n_int += gn - __popc(om);
            n_test += gn;
        }
        if (a.max_stack < 2) {
            drops += lane == 0 ? __popc(om) : 0;
            om = 0;
        }
        if (lane == 0) {
            w.nx[END] = END;
            w.fl[END] = 0;
            w.ek[0] = 0;
            w.ea[0] = om;
            w.fl[0] = 0;
            w.nx[0] = END;
            w.sf[END] = 0;
        }
        if (om) {
            ns = live = fresh = 1;
            head = 0;
        }
    }
    __syncwarp();
    // Emits the expanded elements among the first 32 of the list, of which lane
    // i holds the i-th (h: the one after them), and frees their elements; lane
    // i < cnt then has the i-th one's record in U, V and masks in uL, uR.
    float4 U = make_float4(0.f, 0.f, 0.f, 0.f), V = U;
    unsigned uL = 0, uR = 0;
    auto emit = [&](int mine, int h, int got) {
        const unsigned stop = __ballot_sync(0xffffffffu, !(w.fl[mine] & 0x80));
        cnt = stop ? __ffs(stop) - 1 : 32;
        head = cnt < got ? __shfl_sync(0xffffffffu, mine, cnt) : h;
        if (lane < cnt) {
            // An index that the round found out of range is still in the list, with empty masks.
            const float4 *rc = a.inode + 3 * (int64_t)min((unsigned)w.ek[mine], (unsigned)(n - 2));
            U = __ldg(rc);
            V = __ldg(rc + 1);
            uL = w.ea[mine];
            if constexpr (T == 32) uR = w.eb[mine];
            w.sf[nfree + lane] = (unsigned short)mine;
        }
        nfree += cnt;
        live -= cnt;
    };
    auto buffer = [&]() {
        if (lane < cnt) {
            if constexpr (T == 32) {
                w.ra[lane] = U;
                w.rb[lane] = V;
                w.rm[lane] = make_uint2(uL, uR);
            } else {
                w.ra[lane] = make_float4(U.x, U.z, V.x, V.z);
                w.rb[lane] = make_float4(U.y, U.w, V.y, V.w);
                w.rmask[lane] = uL;
            }
        }
        __syncwarp();
    };
    // The list's first elements, the i-th in lane i's `mine`, as far as the
    // expanded ones reach (in eights); h: the one after them.
    auto chase = [&](int &mine, int &h) {
        mine = END;
        h = head;
        int got = 0;
        do {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (lane == got + i) mine = h;
                h = w.nx[h];
            }
            got += 8;
        } while (got < 32 && (w.fl[h] & 0x80));
        return got;
    };
    // A consistent tree expands each internal node at most once per group,
    // so more than n - 1 rounds mean a corrupted tree: stop.
    for (int round = 0; ns > 0; ++round) {
        const int take = min(ns, max(1, min(32, (CAP - WALK_RESERVE - live) >> 1)));
        const bool act = lane < take;
        const int e = act ? w.sf[CAP - ns + lane] : END;
        int k = 0, depth = 0;
        unsigned m = 0;
        if (act) {
            k = w.ek[e];
            m = w.ea[e];
            depth = w.fl[e];
        }
        ns -= take;
        if (round >= n || (unsigned)k >= (unsigned)(n - 1)) {  // never for a consistent tree
            bad += __popc(m);
            k = 0;
            m = 0;
        }
        // Idle lanes read record 0 with an empty mask.
        const float4 *rec = a.inode + 3 * (int64_t)k;
        const float4 A = __ldg(rec), B = __ldg(rec + 1), C = __ldg(rec + 2);
        if (COUNT) reads += __popc(__ballot_sync(0xffffffffu, m != 0));
        // While the records arrive: the list's head as the last round left it
        // (a chain of shared-memory loads), and the buffer's sums.
        int mine, h;
        const int got = chase(mine, h);
        buffer();
        walk_eval<PHI>(w, cnt, lane, px, py, pz, a.eps2, sum);
        unsigned aL = 0, aR = 0;
        {
            const f2 XL = pack2(A.x, A.x), YL = pack2(A.z, A.z), ZL = pack2(B.x, B.x), SL = pack2(C.x, C.x);
            const f2 XR = pack2(A.y, A.y), YR = pack2(A.w, A.w), ZR = pack2(B.y, B.y), SR = pack2(C.y, C.y);
            const ulonglong2 *TX = reinterpret_cast<const ulonglong2 *>(w.tx),
                             *TY = reinterpret_cast<const ulonglong2 *>(w.ty),
                             *TZ = reinterpret_cast<const ulonglong2 *>(w.tz);
#pragma unroll
            for (int j = T / 4 - 1; j >= 0; --j) {  // target 4 j + 3 first: its bit is shifted furthest
                const ulonglong2 X = TX[j], Y = TY[j], Z = TZ[j];
                aL = walk_test(aL, XL, YL, ZL, X.y, Y.y, Z.y, SL, E2, TH2, NEG);
                aR = walk_test(aR, XR, YR, ZR, X.y, Y.y, Z.y, SR, E2, TH2, NEG);
                aL = walk_test(aL, XL, YL, ZL, X.x, Y.x, Z.x, SL, E2, TH2, NEG);
                aR = walk_test(aR, XR, YR, ZR, X.x, Y.x, Z.x, SR, E2, TH2, NEG);
            }
        }
        emit(mine, h, got);
        __syncwarp();
        const int idL = __float_as_int(C.z), idR = __float_as_int(C.w);
        unsigned oL = m & ~aL, oR = m & ~aR;
        aL &= m;
        aR &= m;
        if (COUNT) {
            n_int += __popc(aL) + __popc(aR);
            n_test += (C.x >= 0.f ? __popc(m) : 0) + (C.y >= 0.f ? __popc(m) : 0);
        }
        if (idL < n) {
            if (PHI || COUNT) {  // a target's own leaf
                const unsigned o = (unsigned)(idL - g0) < (unsigned)T ? aL & (1u << (idL - g0)) : 0u;
                self |= o;
                if (COUNT && o) n_int -= 1u;
            }
            bad += __popc(oL);  // a leaf that fails the test has a non-finite distance
            oL = 0;
        }
        if (idR < n) {
            if (PHI || COUNT) {
                const unsigned o = (unsigned)(idR - g0) < (unsigned)T ? aR & (1u << (idR - g0)) : 0u;
                self |= o;
                if (COUNT && o) n_int -= 1u;
            }
            bad += __popc(oR);
            oR = 0;
        }
        if (depth + 3 > a.max_stack) {  // the rule only bites near max_stack
            drops += __popc(oR);
            oR = 0;
            if (depth + 2 > a.max_stack) {
                drops += __popc(oL);
                oL = 0;
            }
        }
        // The opened children in list order: right, left of lane 0, then of
        // lane 1, ...  A node that no target accepted a child of leaves the
        // list: its first opened child takes its element.  The others' are
        // freed ones first, then fresh ones.
        const unsigned cL = __ballot_sync(0xffffffffu, oL != 0), cR = __ballot_sync(0xffffffffu, oR != 0);
        const bool swap = (aL | aR) == 0 && (oL | oR) != 0;
        const unsigned cS = __ballot_sync(0xffffffffu, swap);
        const int np = __popc(cL) + __popc(cR), na = np - __popc(cS);
        if (fresh + max(0, na - nfree) > END) {  // never for a consistent tree
            bad += lane == 0 ? 1u : 0u;
            break;
        }
        const int rank = __popc(cL & lt) + __popc(cR & lt);
        const int q = rank - __popc(cS & lt);  // the lane's first new element
        const int n0 = q < nfree ? w.sf[nfree - 1 - q] : fresh + q - nfree;
        const int n1 = q + 1 < nfree ? w.sf[nfree - 2 - q] : fresh + q + 1 - nfree;
        __syncwarp();  // the popped and the free elements are read
        ns += np;
        live += na;
        fresh += max(0, na - nfree);
        nfree = max(0, nfree - na);
        if (act) {
            const int c1 = swap ? e : n0, c2 = swap ? n0 : n1;  // the first and the second opened child
            int link = w.nx[e];
            if (oL) {
                const int el = oR ? c2 : c1;
                w.ek[el] = idL - n;
                w.ea[el] = oL;
                w.fl[el] = (unsigned char)depth;
                w.nx[el] = (unsigned short)link;
                w.sf[CAP - ns + rank + (oR ? 1 : 0)] = (unsigned short)el;
                link = el;
            }
            if (oR) {
                w.ek[c1] = idR - n;
                w.ea[c1] = oR;
                w.fl[c1] = (unsigned char)min(depth + 1, WALK_DEPTH);
                w.nx[c1] = (unsigned short)link;
                w.sf[CAP - ns + rank] = (unsigned short)c1;
                link = c1;
            }
            if (!swap) {
                w.nx[e] = (unsigned short)link;
                w.fl[e] = 0x80;
                if constexpr (T == 32) {
                    w.ea[e] = aL;
                    w.eb[e] = aR;
                } else {
                    w.ea[e] = aL | aR << T;
                }
            }
        }
        __syncwarp();
    }
    if (n >= 2) {  // the elements left are all expanded
        do {
            int mine, h;
            const int got = chase(mine, h);
            buffer();
            walk_eval<PHI>(w, cnt, lane, px, py, pz, a.eps2, sum);
            emit(mine, h, got);
            __syncwarp();
        } while (cnt > 0);
    }
    // Counters: one atomic per warp and counter.
    const unsigned dsum = __reduce_add_sync(0xffffffffu, drops), bsum = __reduce_add_sync(0xffffffffu, bad);
    if (lane == 0) {
        if (dsum) atomicAdd(a.diag + DIAG_STACK_DROPS, (unsigned long long)dsum);
        if (bsum) atomicAdd(a.diag + DIAG_BAD_TREE, (unsigned long long)bsum);
    }
    if (COUNT) {
        const unsigned isum = __reduce_add_sync(0xffffffffu, n_int), tsum = __reduce_add_sync(0xffffffffu, n_test);
        if (lane == 0) {
            atomicAdd(a.diag + DIAG_NODE_READS, (unsigned long long)reads);
            atomicAdd(a.diag + DIAG_ROOT_READS, 1ull);
            atomicAdd(a.diag + DIAG_INTERACTIONS, (unsigned long long)isum);
            atomicAdd(a.diag + DIAG_TESTS, (unsigned long long)tsum);
        }
    }
    const float tx = walk_total<T>(sum.X), ty = walk_total<T>(sum.Y), tz = walk_total<T>(sum.Z);
    float pw = 0.f;
    if (PHI) {
        // The records' terms include the target's own leaf: remove it.
        pw = aw + walk_total<T>(sum.W);
        if ((__reduce_or_sync(0xffffffffu, self) >> t) & 1u) {
            const float inv = rsqrt_approx(a.eps2);
            pw = __fmaf_rn(-((pm * inv) * (inv * inv)), a.eps2, pw);
        }
    }
    if (lane >= gn) return;
    const int s = g0 + lane;
    const uint32_t p = __ldg(a.order + s);
    if (p >= (uint32_t)n) return;
    if (PHI) phi[p] = pw;
    trav_write<KDK>(a, p, px, py, pz, ax + tx, ay + ty, az + tz);
}

// ------------------------------------------------------------- short walks
// Large opening angles make short walks: most of the rounds of bh_walk_kernel go
// down the tree towards the targets with few nodes each, at the price of 32.
// These two kernels expand one node at a time, per warp or per lane, and add
// every accepted child where they meet it.  Right subtrees come first, so each
// target sums the same nodes in the same order as in bh_walk_kernel, bit for bit.
//
// Walk time over that of bh_walk_kernel (disk, Plummer sphere, uniform cube; eps
// 0.05; 63-bit keys), per lane at theta 1.0 / 1.1 / 1.2 / 1.3 (15,000 and 22,000,
// theta 1.4: 0.94 1.20 0.79, 0.89 1.12 0.77):
//   25,000: 1.43 1.90 1.35 / 1.20 1.59 1.03 / 1.05 1.36 0.91 / 0.90 1.17 0.82
//   40,000: 1.26 1.69 1.17 / 1.11 1.41 0.84 / 1.03 1.19 0.79 / 0.87 1.08 0.68
//   50,000: 1.23 1.42 1.00 / 1.06 1.18 0.78 / 0.93 0.95 0.69 / 0.79 0.85 0.58
//   85,000: 0.94 1.20 0.88 / 0.83 0.97 0.65 / 0.71 0.81 0.60 / 0.63 0.71 0.53
//  100,000: 0.92 1.10 0.75 / 0.77 0.94 0.53 / 0.64 0.79 0.50 / 0.57 0.68 0.44
// and per warp at theta 0.8 / 0.9 / 1.0 / 1.2:
//  131,072: 1.35 1.15 1.17 / 1.23 1.08 0.97 / 1.10 0.96 0.80 / 0.81 0.74 0.59
//  250,000: 1.22 1.23 1.08 / 1.11 1.12 0.88 / 1.00 0.97 0.70 / 0.74 0.72 0.49
//  500,000: 1.10 1.07 0.94 / 0.98 0.97 0.74 / 0.85 0.84 0.57 / 0.64 0.61 0.38
//  1.5M:    1.01 1.04 0.79 / 0.90 0.92 0.60 / 0.77 0.79 0.46 / 0.57 0.59 0.31
//  4M:      1.01 1.02 0.72 / 0.89 0.91 0.54 / 0.76 0.77 0.41 / 0.54 0.58 0.29
// (100,000, theta 1.2: 96 us in rounds, 62 per lane, 82 per warp on the disk; 1M:
// 813 in rounds, 473 per warp.)  Per lane is the faster of the two up to about
// 120,000 (100,000: see above; 131,072, theta 1.2: 0.71 0.96 0.63).  The lines of
// walk_form lie where the geometric mean of the three crosses 1.
enum WalkForm { WALK_ROUNDS, WALK_LANE, WALK_WARP };
static inline WalkForm walk_form(int64_t n, float theta) {
    if (n < 12000) return WALK_ROUNDS;
    if (n < 131072) {
        const float line = n < 25000 ? 1.4f : n < 40000 ? 1.3f : n < 50000 ? 1.2f : n < 85000 ? 1.1f : 1.0f;
        return theta >= line ? WALK_LANE : WALK_ROUNDS;
    }
    const float line = n < 150000 ? 1.0f : n < 300000 ? 0.95f : n < 500000 ? 0.9f : n < 1200000 ? 0.85f : 0.8f;
    return theta >= line ? WALK_WARP : WALK_ROUNDS;
}

// One lane's target s and its sums.
struct OneWalk {
    float px, py, pz, pm;
    f2 PX, PY, PZ;
    float ax, ay, az, aw;  // the root's term
    WalkSum sum;           // over the (left, right) children
    unsigned n_int, n_test, drops;
    bool self;             // met the target's own leaf
};

__device__ __forceinline__ OneWalk one_target(const TravArgs &a, int s, bool valid) {
    OneWalk w;
    const float4 p = valid ? __ldg(a.leaf + s) : make_float4(0.f, 0.f, 0.f, 0.f);
    w.px = p.x; w.py = p.y; w.pz = p.z; w.pm = p.w;
    w.PX = pack2(p.x, p.x);
    w.PY = pack2(p.y, p.y);
    w.PZ = pack2(p.z, p.z);
    w.ax = w.ay = w.az = w.aw = 0.f;
    w.sum.X = w.sum.Y = w.sum.Z = w.sum.W = 0ull;
    w.n_int = w.n_test = w.drops = 0;
    w.self = false;
    return w;
}

// Whether a target that opens a node popped at `depth` may push its children (:212).
__device__ __forceinline__ bool one_room(OneWalk &w, bool open, int depth, int max_stack) {
    if (depth + 2 <= max_stack) return open;
    w.drops += open ? 1u : 0u;
    return false;
}

// The root, popped first with an empty stack; returns whether it is opened.
__device__ __forceinline__ bool one_root(OneWalk &w, const TravArgs &a, bool valid) {
    const float4 R0 = __ldg(a.root), R1 = __ldg(a.root + 1);
    const float dx = R0.x - w.px, dy = R0.y - w.py, dz = R0.z - w.pz;
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, a.eps2)));
    const bool acc = valid && R1.x < a.theta2 * r2;
    if (acc) {
        const float inv = rsqrt_approx(r2);
        const float sc = R0.w * inv * inv * inv;
        w.ax = __fmul_rn(sc, dx);
        w.ay = __fmul_rn(sc, dy);
        w.az = __fmul_rn(sc, dz);
        w.aw = R0.w * inv;
        w.n_int = 1;
    }
    w.n_test = valid ? 1 : 0;
    return one_room(w, valid && !acc, 0, a.max_stack);
}

// Both children of record {A, B, C} for the lane's target, when `in`: accepted
// ones are added, and the ones to open returned.
template <bool COUNT, bool PHI>
__device__ __forceinline__ void one_pair(OneWalk &w, const TravArgs &a, ulonglong2 A, ulonglong2 B, float4 C, int s,
                                         bool in, f2 E2, f2 TH2, bool &openL, bool &openR) {
    const f2 dx = sub2(A.x, w.PX), dy = sub2(A.y, w.PY), dz = sub2(B.x, w.PZ);
    f2 r2 = fma2(dx, dx, E2);
    r2 = fma2(dy, dy, r2);
    r2 = fma2(dz, dz, r2);
    float tL, tR, cL, cR;
    unpack2(mul2(TH2, r2), tL, tR);
    const bool accL = in && C.x < tL, accR = in && C.y < tR;
    const f2 inv = rsqrt2(r2);
    unpack2(mul2(mul2(B.y, inv), mul2(inv, inv)), cL, cR);
    const f2 sc = pack2(accL ? cL : 0.f, accR ? cR : 0.f);
    w.sum.X = fma2(sc, dx, w.sum.X);
    w.sum.Y = fma2(sc, dy, w.sum.Y);
    w.sum.Z = fma2(sc, dz, w.sum.Z);
    if (PHI) w.sum.W = fma2(sc, r2, w.sum.W);
    if (PHI || COUNT) {
        const bool ownL = __float_as_int(C.z) == s, ownR = __float_as_int(C.w) == s;
        if (PHI) w.self |= (accL && ownL) || (accR && ownR);
        if (COUNT) {
            w.n_int += (accL && !ownL ? 1u : 0u) + (accR && !ownR ? 1u : 0u);
            w.n_test += (in && C.x >= 0.f ? 1u : 0u) + (in && C.y >= 0.f ? 1u : 0u);
        }
    }
    openL = in && !accL;
    openR = in && !accR;
}

// The warp's counters, and the lane's target written.  reads, roots: records
// read by the lane or its warp.
template <bool KDK, bool COUNT, bool PHI>
__device__ __forceinline__ void one_write(OneWalk &w, const TravArgs &a, float *__restrict__ phi, int s, bool valid,
                                          unsigned bad, unsigned reads, unsigned roots) {
    const int lane = threadIdx.x & 31;
    const unsigned dsum = __reduce_add_sync(0xffffffffu, w.drops), bsum = __reduce_add_sync(0xffffffffu, bad);
    if (lane == 0) {
        if (dsum) atomicAdd(a.diag + DIAG_STACK_DROPS, (unsigned long long)dsum);
        if (bsum) atomicAdd(a.diag + DIAG_BAD_TREE, (unsigned long long)bsum);
    }
    if (COUNT) {
        const unsigned isum = __reduce_add_sync(0xffffffffu, w.n_int), tsum = __reduce_add_sync(0xffffffffu, w.n_test);
        const unsigned rsum = __reduce_add_sync(0xffffffffu, reads), osum = __reduce_add_sync(0xffffffffu, roots);
        if (lane == 0) {
            atomicAdd(a.diag + DIAG_NODE_READS, (unsigned long long)rsum);
            atomicAdd(a.diag + DIAG_ROOT_READS, (unsigned long long)osum);
            atomicAdd(a.diag + DIAG_INTERACTIONS, (unsigned long long)isum);
            atomicAdd(a.diag + DIAG_TESTS, (unsigned long long)tsum);
        }
    }
    if (!valid) return;
    const uint32_t p = __ldg(a.order + s);
    if (p >= (uint32_t)a.n) return;
    float xl, xr, yl, yr, zl, zr;
    unpack2(w.sum.X, xl, xr);
    unpack2(w.sum.Y, yl, yr);
    unpack2(w.sum.Z, zl, zr);
    if (PHI) {  // the children's terms include the target's own leaf: remove it
        float wl, wr;
        unpack2(w.sum.W, wl, wr);
        float pw = w.aw + (wl + wr);
        if (w.self) {
            const float inv = rsqrt_approx(a.eps2);
            pw = __fmaf_rn(-((w.pm * inv) * (inv * inv)), a.eps2, pw);
        }
        phi[p] = pw;
    }
    trav_write<KDK>(a, p, w.px, w.py, w.pz, w.ax + (xl + xr), w.ay + (yl + yr), w.az + (zl + zr));
}

// Per warp: 32 key-consecutive targets share a stack of {node, mask of the
// targets that opened it, depth}.
constexpr int WARP_WALK_WARPS = 4;
constexpr int WARP_WALK_STACK = 128;  // one pending left child per level of right turns: 94 in a consistent tree

template <bool KDK, bool COUNT, bool PHI>
__global__ void __launch_bounds__(WARP_WALK_WARPS * 32)
bh_warp_walk_kernel(TravArgs a, float *__restrict__ phi, int s0, int s1) {
    __shared__ int4 stk[WARP_WALK_WARPS][WARP_WALK_STACK];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, n = a.n;
    const int g0 = s0 + (blockIdx.x * WARP_WALK_WARPS + wid) * 32, s = g0 + lane;
    if (g0 >= s1) return;  // whole warp out of range
    const bool valid = s < s1;
    OneWalk w = one_target(a, s, valid);
    const f2 E2 = pack2(a.eps2, a.eps2), TH2 = pack2(a.theta2, a.theta2);
    unsigned bad = 0, reads = 0, m = 0;
    int top = 0, k = 0, depth = 0;
    if (n >= 2) m = __ballot_sync(0xffffffffu, one_root(w, a, valid));
    // A consistent tree expands each internal node at most once per warp, so
    // more than n - 1 nodes mean a corrupted tree.
    for (int left = n; m;) {
        unsigned mL = 0, mR = 0;
        int idL = 0, idR = 0;
        if (--left < 0 || (unsigned)k >= (unsigned)(n - 1)) {  // never for a consistent tree
            bad += (m >> lane) & 1u;
        } else {
            const float4 *rec = a.inode + 3 * (int64_t)k;
            const ulonglong2 A = __ldg(reinterpret_cast<const ulonglong2 *>(rec));
            const ulonglong2 B = __ldg(reinterpret_cast<const ulonglong2 *>(rec + 1));
            const float4 C = __ldg(rec + 2);
            idL = __float_as_int(C.z);
            idR = __float_as_int(C.w);
            reads += lane == 0 ? 1u : 0u;
            bool openL, openR;
            one_pair<COUNT, PHI>(w, a, A, B, C, s, (m >> lane) & 1u, E2, TH2, openL, openR);
            if (depth + 3 > a.max_stack) {  // the rule only bites near max_stack
                openR = one_room(w, openR, depth + 1, a.max_stack);
                openL = one_room(w, openL, depth, a.max_stack);
            }
            mL = __ballot_sync(0xffffffffu, openL);
            mR = __ballot_sync(0xffffffffu, openR);
        }
        if (mR) {  // the right child next; a left child waits on the stack
            if (mL) {
                if (top < WARP_WALK_STACK) stk[wid][top++] = make_int4(idL - n, (int)mL, depth, 0);
            }
            k = idR - n;
            m = mR;
            ++depth;
        } else if (mL) {
            k = idL - n;
            m = mL;
        } else if (top > 0) {
            __syncwarp();
            const int4 e = stk[wid][--top];
            __syncwarp();
            k = e.x;
            m = (unsigned)e.y;
            depth = e.z;
        } else {
            m = 0;
        }
    }
    one_write<KDK, COUNT, PHI>(w, a, phi, s, valid, bad, reads, lane == 0 ? 1u : 0u);
}

// Per lane: every lane walks for its own target, its pending left children as
// {node, 25 bits; depth, 7 bits} on a stack of its own, laid out so that lanes
// meet no bank conflicts whatever their depth.
constexpr int LANE_WALK_THREADS = 128;
constexpr int LANE_WALK_BITS = 25;
constexpr int LANE_WALK_STACK = 96;  // one pending left child per level of right turns (94)

template <bool KDK, bool COUNT, bool PHI>
__global__ void __launch_bounds__(LANE_WALK_THREADS)
bh_lane_walk_kernel(TravArgs a, float *__restrict__ phi, int s0, int s1, int room) {
    extern __shared__ unsigned lane_stk[];  // [room][LANE_WALK_THREADS]
    const int tid = threadIdx.x, n = a.n, s = s0 + blockIdx.x * LANE_WALK_THREADS + tid;
    const bool valid = s < s1;
    OneWalk w = one_target(a, s, valid);
    const f2 E2 = pack2(a.eps2, a.eps2), TH2 = pack2(a.theta2, a.theta2);
    unsigned bad = 0, reads = 0;
    int k = 0, depth = 0, top = 0;
    bool active = n >= 2 && one_root(w, a, valid);
    for (int left = n;;) {
        if (!active) {
            if (top == 0) break;
            const unsigned e = lane_stk[--top * LANE_WALK_THREADS + tid];
            k = (int)(e & ((1u << LANE_WALK_BITS) - 1u));
            depth = (int)(e >> LANE_WALK_BITS);
            active = true;
        }
        if (--left < 0 || (unsigned)k >= (unsigned)(n - 1)) {  // never for a consistent tree
            ++bad;
            break;
        }
        const float4 *rec = a.inode + 3 * (int64_t)k;
        const ulonglong2 A = __ldg(reinterpret_cast<const ulonglong2 *>(rec));
        const ulonglong2 B = __ldg(reinterpret_cast<const ulonglong2 *>(rec + 1));
        const float4 C = __ldg(rec + 2);
        const int idL = __float_as_int(C.z), idR = __float_as_int(C.w);
        if (COUNT) ++reads;
        bool openL, openR;
        one_pair<COUNT, PHI>(w, a, A, B, C, s, true, E2, TH2, openL, openR);
        if (depth + 3 > a.max_stack) {
            openR = one_room(w, openR, depth + 1, a.max_stack);
            openL = one_room(w, openL, depth, a.max_stack);
        }
        if (openR) {
            if (openL) {
                if (top < room) lane_stk[top++ * LANE_WALK_THREADS + tid] =
                    (unsigned)(idL - n) | (unsigned)depth << LANE_WALK_BITS;
                else ++bad;  // never for a consistent tree
            }
            k = idR - n;
            ++depth;
        } else if (openL) {
            k = idL - n;
        } else {
            active = false;
        }
    }
    __syncwarp();
    one_write<KDK, COUNT, PHI>(w, a, phi, s, valid, bad, reads, n >= 2 && valid ? 1u : 0u);
}

// ------------------------------------------------------------- group walk
// Group walk (gb_bh_set_traversal 3): the warp's 32 key-consecutive targets
// share one walk and one interaction list.  A node is accepted for the whole
// group when size^2 < theta^2 (dmin^2 + eps^2), dmin the distance from its
// centre of mass to the group's bounding box; since every target is at
// least dmin away, each target then also passes the reference's own test
// (core/solvers/barnes_hut.py:204-210), so the group accepts a refinement of
// every target's node set: more, smaller nodes, never a coarser one.  Leaves
// are always accepted.  The walk keeps a stack of internal nodes in shared
// memory; each iteration pops up to 32 of them, one per lane, loads their
// two-children records and tests both children: accepted children go to the
// interaction list (compacted by ballots), opened ones are pushed.  The list
// is evaluated by every lane for its own target, two entries per packed
// .f32x2 instruction, whenever it fills and at the end.  Deterministic (no
// atomics); not the reference's per-particle node set, so its results are
// not bit-identical to the other shapes; the max_stack rule does not apply.
// A push that would overflow the warp's stack takes the child as a monopole
// instead and counts it in stack_overflow.
constexpr int GW_WARPS = 2;
constexpr int GW_STACK = 640;            // internal nodes per warp (the 1M disk peaks near 310)
constexpr int GW_LIST = 256;             // list entries per warp
constexpr int GW_FLUSH = GW_LIST - 64;   // an iteration appends at most 64

// The list holds entry pairs as {x0, x1, y0, y1} in la and {z0, z1, m0, m1}
// in lb (two arrays: the scalar stores of 32 consecutive entries meet 2-way
// bank conflicts, against 4-way with the two halves interleaved).
struct GwWarp {
    int stk[GW_STACK];
    float4 la[GW_LIST / 2];
    float4 lb[GW_LIST / 2];
};

__device__ __forceinline__ void gw_put(GwWarp &w, int j, float x, float y, float z, float m) {
    float *a = reinterpret_cast<float *>(&w.la[j >> 1]);
    float *b = reinterpret_cast<float *>(&w.lb[j >> 1]);
    const int h = j & 1;
    a[h] = x;
    a[2 + h] = y;
    b[h] = z;
    b[2 + h] = m;
}

// Squared distance from (x, y, z) to the box [lo, hi].
__device__ __forceinline__ float box_dist2(float x, float y, float z, float lx, float ly, float lz, float hx, float hy,
                                           float hz) {
    const float dx = fmaxf(fmaxf(lx - x, x - hx), 0.f);
    const float dy = fmaxf(fmaxf(ly - y, y - hy), 0.f);
    const float dz = fmaxf(fmaxf(lz - z, z - hz), 0.f);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
}

// Adds entries [0, cnt) of the list (cnt even) to the lane's target.
template <bool PHI>
__device__ __forceinline__ void gw_eval(const GwWarp &w, int cnt, f2 PX, f2 PY, f2 PZ, f2 E2, f2 &AX, f2 &AY,
                                        f2 &AZ, f2 &PW) {
    const ulonglong2 *LA = reinterpret_cast<const ulonglong2 *>(w.la);
    const ulonglong2 *LB = reinterpret_cast<const ulonglong2 *>(w.lb);
#pragma unroll 4
    for (int q = 0; q < (cnt >> 1); ++q) {
        const ulonglong2 A = LA[q], B = LB[q];
        const f2 dx = sub2(A.x, PX), dy = sub2(A.y, PY), dz = sub2(B.x, PZ);
        f2 r2 = fma2(dx, dx, E2);
        r2 = fma2(dy, dy, r2);
        r2 = fma2(dz, dz, r2);
        const f2 inv = rsqrt2(r2);
        const f2 mi = mul2(B.y, inv);
        const f2 sc = mul2(mi, mul2(inv, inv));
        AX = fma2(sc, dx, AX);
        AY = fma2(sc, dy, AY);
        AZ = fma2(sc, dz, AZ);
        if (PHI) PW = add2(PW, mi);
    }
}

// One group: leaves [g0, g0 + size) (size <= 32), lane l walks with target
// g0 + l.
template <bool KDK, bool COUNT, bool PHI>
__device__ __forceinline__ void gw_group(GwWarp &w, const TravArgs &a, float *__restrict__ phi, int g0, int size,
                                         int lane, unsigned &reads, unsigned &evals, unsigned &overflow,
                                         unsigned &bad) {
    const int n = a.n;
    const int s = g0 + lane;
    const bool valid = lane < size;
    float px = 0.f, py = 0.f, pz = 0.f, pm = 0.f;
    if (valid) {
        const float4 p = __ldg(a.leaf + s);
        px = p.x; py = p.y; pz = p.z; pm = p.w;
    }
    // The group's bounding box.
    float lx = valid ? px : INFINITY, ly = valid ? py : INFINITY, lz = valid ? pz : INFINITY;
    float hx = valid ? px : -INFINITY, hy = valid ? py : -INFINITY, hz = valid ? pz : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o));
        ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o));
        lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o));
        hx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, o));
        hy = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, o));
        hz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, o));
    }
    const f2 PX = pack2(px, px), PY = pack2(py, py), PZ = pack2(pz, pz), E2 = pack2(a.eps2, a.eps2);
    f2 AX = 0ull, AY = 0ull, AZ = 0ull, PW = 0ull;
    const unsigned lt = (1u << lane) - 1u;
    unsigned selfbits = 0;
    int cnt = 0, top = 0;
    if (n >= 2) {
        // The root, tested for the whole group: a monopole, or its children.
        const float4 R0 = __ldg(a.root), R1 = __ldg(a.root + 1);
        const float d2 = box_dist2(R0.x, R0.y, R0.z, lx, ly, lz, hx, hy, hz);
        if (R1.x < a.theta2 * (d2 + a.eps2)) {
            if (lane == 0) gw_put(w, 0, R0.x, R0.y, R0.z, R0.w);
            cnt = 1;
        } else {
            if (lane == 0) w.stk[0] = 0;
            top = 1;
        }
        __syncwarp();
    }
    // A consistent tree expands each internal node at most once per group,
    // so more than n - 1 iterations means a corrupted tree: stop.
    for (int iter = 0; top > 0; ++iter) {
        if (iter >= n) {
            bad += lane == 0 ? 1u : 0u;
            break;
        }
        const int take = min(top, 32);
        top -= take;
        bool act = lane < take;
        const int k = act ? w.stk[top + lane] : 0;
        __syncwarp();  // the popped entries are read before pushes reuse them
        if (act && (unsigned)k >= (unsigned)(n - 1)) {  // never for a consistent tree
            ++bad;
            act = false;
        }
        float4 A = make_float4(0.f, 0.f, 0.f, 0.f), B = A, C = A;
        if (act) {
            const float4 *rec = a.inode + 3 * (int64_t)k;
            A = __ldg(rec);      // {x_L, x_R, y_L, y_R}
            B = __ldg(rec + 1);  // {z_L, z_R, m_L, m_R}
            C = __ldg(rec + 2);  // {size2_L, size2_R, id_L, id_R}
        }
        if (COUNT) reads += __popc(__ballot_sync(0xffffffffu, act));
        // A leaf child carries size2 = -1 and is always accepted.
        const bool accL = act && C.x < a.theta2 * (box_dist2(A.x, A.z, B.x, lx, ly, lz, hx, hy, hz) + a.eps2);
        const bool accR = act && C.y < a.theta2 * (box_dist2(A.y, A.w, B.y, lx, ly, lz, hx, hy, hz) + a.eps2);
        const bool openL = act && !accL, openR = act && !accR;
        const int idL = __float_as_int(C.z), idR = __float_as_int(C.w);
        const unsigned bL = __ballot_sync(0xffffffffu, accL), bR = __ballot_sync(0xffffffffu, accR);
        if (accL) gw_put(w, cnt + __popc(bL & lt), A.x, A.z, B.x, B.z);
        if (accR) gw_put(w, cnt + __popc(bL) + __popc(bR & lt), A.y, A.w, B.y, B.w);
        cnt += __popc(bL) + __popc(bR);
        if (PHI) {
            // Own leaves of the group's targets in the list: their terms are
            // removed from the potential at the end.
            unsigned bit = 0;
            if (accL && (unsigned)(idL - g0) < (unsigned)size) bit |= 1u << (idL - g0);
            if (accR && (unsigned)(idR - g0) < (unsigned)size) bit |= 1u << (idR - g0);
            selfbits |= __reduce_or_sync(0xffffffffu, bit);
        }
        const unsigned cL = __ballot_sync(0xffffffffu, openL), cR = __ballot_sync(0xffffffffu, openR);
        const int np = __popc(cL) + __popc(cR);
        if (top + np <= GW_STACK) {
            if (openL) w.stk[top + __popc(cL & lt)] = idL - n;
            if (openR) w.stk[top + __popc(cL) + __popc(cR & lt)] = idR - n;
            top += np;
        } else {  // no room: the opened children enter the list as monopoles
            if (openL) gw_put(w, cnt + __popc(cL & lt), A.x, A.z, B.x, B.z);
            if (openR) gw_put(w, cnt + __popc(cL) + __popc(cR & lt), A.y, A.w, B.y, B.w);
            cnt += np;
            overflow += np;
        }
        __syncwarp();
        if (cnt > GW_FLUSH) {
            if ((cnt & 1) && lane == 0) gw_put(w, cnt, 0.f, 0.f, 0.f, 0.f);
            __syncwarp();
            gw_eval<PHI>(w, cnt + (cnt & 1), PX, PY, PZ, E2, AX, AY, AZ, PW);
            if (COUNT) evals += cnt * size;
            cnt = 0;
            __syncwarp();  // the list is read before the next appends
        }
    }
    if (cnt > 0) {
        if ((cnt & 1) && lane == 0) gw_put(w, cnt, 0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        gw_eval<PHI>(w, cnt + (cnt & 1), PX, PY, PZ, E2, AX, AY, AZ, PW);
        if (COUNT) evals += cnt * size;
    }
    __syncwarp();  // the next group reuses the stack and the list
    if (!valid) return;
    const uint32_t p = __ldg(a.order + s);
    if (p >= (uint32_t)n) {
        ++bad;
        return;
    }
    float xl, xr, yl, yr, zl, zr;
    unpack2(AX, xl, xr);
    unpack2(AY, yl, yr);
    unpack2(AZ, zl, zr);
    if (PHI) {
        float wl, wr;
        unpack2(PW, wl, wr);
        float pw = wl + wr;
        if ((selfbits >> lane) & 1u) pw -= pm * rsqrt_approx(a.eps2);  // the term the list added
        phi[p] = pw;
    }
    trav_write<KDK>(a, p, px, py, pz, xl + xr, yl + yr, zl + zr);
}

// Warp w walks the groups whose first leaf lies in [32 w, 32 w + 32) (gsize
// from bh_tree_kernel), one after the other.
// 32 resident warps per SM (64 registers, 13 KB of shared memory per CTA of
// 2 warps): 7.8% less time than 24 warps on the 1M disk; CTAs of 2 warps
// against 4: 1.3% less (a CTA retires when its slowest warp is done).
template <bool KDK, bool COUNT, bool PHI>
__global__ void __launch_bounds__(GW_WARPS * 32, 16)
bh_group_kernel(TravArgs a, const int *__restrict__ gsize, float *__restrict__ phi, int s0, int s1) {
    __shared__ GwWarp sw[GW_WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    GwWarp &w = sw[wid];
    // Groups whose first leaf lies in [s0, s1) (a group may end past s1).
    const int c0 = s0 + (blockIdx.x * GW_WARPS + wid) * 32;
    if (c0 >= s1) return;  // whole warp out of range
    const int n = a.n;
    int gs = (c0 + lane < s1) ? __ldg(gsize + c0 + lane) : 0;
    if (n == 1 && lane == 0) gs = 1;  // a single particle: no internal node, one group
    unsigned starts = __ballot_sync(0xffffffffu, gs > 0 && gs <= GW_GROUP);
    unsigned reads = 0, evals = 0, overflow = 0, bad = 0, ngroups = 0;
    while (starts) {
        const int j = __ffs(starts) - 1;
        starts &= starts - 1u;
        const int size = min(__shfl_sync(0xffffffffu, gs, j), n - (c0 + j));
        gw_group<KDK, COUNT, PHI>(w, a, phi, c0 + j, size, lane, reads, evals, overflow, bad);
        ++ngroups;
    }
    const unsigned bsum = __reduce_add_sync(0xffffffffu, bad);
    if (lane == 0) {
        if (overflow) atomicAdd(a.diag + DIAG_STACK_OVERFLOW, (unsigned long long)overflow);
        if (bsum) atomicAdd(a.diag + DIAG_BAD_TREE, (unsigned long long)bsum);
        if (COUNT) {
            atomicAdd(a.diag + DIAG_NODE_READS, (unsigned long long)reads);
            atomicAdd(a.diag + DIAG_ROOT_READS, (unsigned long long)ngroups);
            atomicAdd(a.diag + DIAG_INTERACTIONS, (unsigned long long)evals);
            atomicAdd(a.diag + DIAG_TESTS, 2ull * reads + ngroups);
        }
    }
}

}  // namespace gb
