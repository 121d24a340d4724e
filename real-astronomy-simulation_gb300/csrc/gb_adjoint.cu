// Hand-written adjoint (reverse mode) of the direct-sum KDK leapfrog.
//
// Forward step (core/engine.py:108-116, core/integrators/leapfrog.py:11-22):
//   vh = v + h a,  x' = x + dt vh,  a' = F(x'),  v' = vh + h a'   (h = dt/2)
// with F_j = G sum_i m_i (x_i - x_j) (|x_i - x_j|^2 + eps2)^{-3/2}
// (core/solvers/gravity.py:13-26).  Given the adjoints (lx', lv', la') of
// x', v', a', one backward step returns those of x, v, a and accumulates the
// mass gradient:
//   w   = la' + h lv'                       (adjoint of a')
//   gx  = J_x^T w,  gm = J_m^T w             (VJP of F at x')
//   lxt = lx' + gx
//   lvh = lv' + dt lxt
//   lx = lxt,  lv = lvh,  la = h lvh,  lm += gm
// and the priming evaluation a0 = F(x0) adds J^T la to (lx, lm) at the end.
//
// VJP of the pairwise force, for target j and source i, d = x_j - x_i,
// r2 = |d|^2 + eps2, s = r2^{-3/2}, t = r2^{-5/2}:
//   gx_j = G sum_i (s I - 3 t d d^T)(m_j w_i - m_i w_j)
//   gm_j = G sum_i s d.w_i
// With u = m_j w_i - m_i w_j the self pair contributes exactly zero.  The
// kernel uses the stream-K layout of the force kernel (equal unit runs per
// CTA, partials merged in CTA order by the fix-up, which also applies the
// elementwise part of the backward step).
#include <algorithm>

#include "gb_direct_core.cuh"

namespace gb {

struct VjpArgs {
    const float4 *__restrict__ xm;  // positions and masses at which F was evaluated
    const float4 *__restrict__ lv;  // adjoint of v' (ignored when prime)
    const float4 *__restrict__ la;  // adjoint of a'
    float4 *__restrict__ part;
    int64_t n, num_ju, U, P;
    int smax;
    float eps2, h;
    int prime;
};

__device__ __forceinline__ float4 load_w(const VjpArgs &a, int64_t i) {
    if (i >= a.n) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 la = __ldg(a.la + i);
    if (a.prime) return la;
    const float4 lv = __ldg(a.lv + i);
    return make_float4(__fmaf_rn(a.h, lv.x, la.x), __fmaf_rn(a.h, lv.y, la.y), __fmaf_rn(a.h, lv.z, la.z), 0.f);
}

__device__ __forceinline__ float4 load_x(const VjpArgs &a, int64_t i) {
    return i < a.n ? __ldg(a.xm + i) : make_float4(0.f, 0.f, 0.f, 0.f);
}

template <int K, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, K == 2 ? 1024 / (WARPS * 32) : 1)
adjoint_vjp_kernel(VjpArgs a) {
    constexpr int TILE = 32 * K;
    constexpr int ST = WARPS * TILE;
    constexpr int JU = WARPS * 32;
    __shared__ float4 sx[JU], sw[JU];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t c = blockIdx.x;
    const int64_t u_begin = unit_begin(a.U, a.P, c), u_end = unit_begin(a.U, a.P, c + 1);
    if (u_begin >= u_end) return;
    const int64_t st0 = u_begin / a.num_ju;
    int64_t u = u_begin;
    while (u < u_end) {
        const int64_t st = u / a.num_ju;
        const int64_t run_end = min(u_end, (st + 1) * a.num_ju);
        const int64_t tbase = st * ST + wib * TILE + lane;
        float X[K], Y[K], Z[K], M[K], WX[K], WY[K], WZ[K];
        float SX[K], SY[K], SZ[K], SG[K];
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const float4 x = load_x(a, tbase + q * 32), w = load_w(a, tbase + q * 32);
            X[q] = x.x; Y[q] = x.y; Z[q] = x.z; M[q] = x.w;
            WX[q] = w.x; WY[q] = w.y; WZ[q] = w.z;
            SX[q] = SY[q] = SZ[q] = SG[q] = 0.f;
        }
        for (; u < run_end; ++u) {
            const int64_t j = (u - st * a.num_ju) * JU + threadIdx.x;
            const float4 xj = load_x(a, j), wj = load_w(a, j);
            __syncthreads();
            sx[threadIdx.x] = xj;
            sw[threadIdx.x] = wj;
            __syncthreads();
            float PX[K], PY[K], PZ[K], PG[K];
#pragma unroll
            for (int q = 0; q < K; ++q) PX[q] = PY[q] = PZ[q] = PG[q] = 0.f;
#pragma unroll 2
            for (int jj = 0; jj < JU; ++jj) {
                const float4 xs = sx[jj], ws = sw[jj];
#pragma unroll
                for (int q = 0; q < K; ++q) {
                    const float dx = X[q] - xs.x, dy = Y[q] - xs.y, dz = Z[q] - xs.z;
                    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, a.eps2)));
                    const float inv = rsqrt_approx(r2);
                    const float inv2 = inv * inv;
                    const float s = inv * inv2;
                    const float t3 = s * (3.f * inv2);
                    const float ux = __fmaf_rn(-xs.w, WX[q], M[q] * ws.x);
                    const float uy = __fmaf_rn(-xs.w, WY[q], M[q] * ws.y);
                    const float uz = __fmaf_rn(-xs.w, WZ[q], M[q] * ws.z);
                    const float du = __fmaf_rn(dz, uz, __fmaf_rn(dy, uy, dx * ux));
                    const float cf = t3 * du;
                    PX[q] = __fmaf_rn(-cf, dx, __fmaf_rn(s, ux, PX[q]));
                    PY[q] = __fmaf_rn(-cf, dy, __fmaf_rn(s, uy, PY[q]));
                    PZ[q] = __fmaf_rn(-cf, dz, __fmaf_rn(s, uz, PZ[q]));
                    const float dw = __fmaf_rn(dz, ws.z, __fmaf_rn(dy, ws.y, dx * ws.x));
                    PG[q] = __fmaf_rn(s, dw, PG[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < K; ++q) {
                SX[q] += PX[q]; SY[q] += PY[q]; SZ[q] += PZ[q]; SG[q] += PG[q];
            }
        }
        const int64_t slot = (c * a.smax + (st - st0)) * ST + wib * TILE + lane;
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int64_t sq = slot + q * 32;
            a.part[2 * sq] = make_float4(SX[q], SY[q], SZ[q], SG[q]);  // (the lo half is unused)
        }
    }
}

struct VjpFix {
    const float4 *__restrict__ part;
    float4 *lx, *lv, *la;
    float *lm;
    int64_t n, num_ju, U, P, st_size;
    int smax;
    float G, h, dt;
    int prime;
};

__global__ void adjoint_fixup_kernel(VjpFix f) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= f.n) return;
    const int64_t st = i / f.st_size, off = i - st * f.st_size;
    const int64_t c_lo = unit_owner(f.U, f.P, st * f.num_ju);
    const int64_t c_hi = unit_owner(f.U, f.P, (st + 1) * f.num_ju - 1);
    float gx = 0.f, gy = 0.f, gz = 0.f, gm = 0.f;
    for (int64_t c = c_lo; c <= c_hi; ++c) {
        const int64_t st0c = unit_begin(f.U, f.P, c) / f.num_ju;
        const float4 p = f.part[2 * ((c * f.smax + (st - st0c)) * f.st_size + off)];
        gx += p.x; gy += p.y; gz += p.z; gm += p.w;
    }
    gx *= f.G; gy *= f.G; gz *= f.G; gm *= f.G;
    f.lm[i] += gm;
    const float4 lx = f.lx[i];
    const float tx = lx.x + gx, ty = lx.y + gy, tz = lx.z + gz;
    if (f.prime) {
        f.lx[i] = make_float4(tx, ty, tz, 0.f);
        return;
    }
    const float4 lv = f.lv[i];
    const float hx = __fmaf_rn(f.dt, tx, lv.x), hy = __fmaf_rn(f.dt, ty, lv.y), hz = __fmaf_rn(f.dt, tz, lv.z);
    f.lx[i] = make_float4(tx, ty, tz, 0.f);
    f.lv[i] = make_float4(hx, hy, hz, 0.f);
    f.la[i] = make_float4(f.h * hx, f.h * hy, f.h * hz, 0.f);
}

constexpr int VJP_K = 2;
constexpr int VJP_WARPS = 8;

// --------------------------------------------------- symmetric evaluation
// Every unordered pair {i, j} once (Newton's third law).  With d = x_j - x_i
// and P = K(d) (m_j w_i - m_i w_j) (K = s I - 3 t d d^T, symmetric in i, j):
//   gx_j += P,  gx_i -= P,  gm_j += s d.w_i,  gm_i -= s d.w_j.
// Tiles of ST_T = 256 particles; unordered tile pairs (I <= J) are numbered
// row-major and split into equal runs over a persistent grid.  A CTA (4 warps,
// 2 targets per lane) keeps tile I's sums in registers along its row; tile J
// sits in shared memory with per-source accumulators.  In round r warp w
// works on source group g = (2w + r) mod 8 and at step k lane l on source
// 32g + (l + k) mod 32: no two lanes touch one accumulator at once, so there
// are no atomics.  Row sums go to slot (I + CTA) and each tile pair's source
// sums to slot (pair); the fix-up merges them in a fixed order.
constexpr int SYM_T = 256;
constexpr int SYM_WARPS = 4;


struct SymArgs {
    const float4 *__restrict__ xm;
    const float4 *__restrict__ lv;
    const float4 *__restrict__ la;
    float4 *__restrict__ rowpart;  // (nt + P) x SYM_T
    float4 *__restrict__ colpart;  // NP x SYM_T
    int64_t n, nt, NP, P;
    float eps2, h;
    int prime;
};

__device__ __forceinline__ float4 sym_w(const SymArgs &a, int64_t i) {
    if (i >= a.n) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 la = __ldg(a.la + i);
    if (a.prime) return la;
    const float4 lv = __ldg(a.lv + i);
    return make_float4(__fmaf_rn(a.h, lv.x, la.x), __fmaf_rn(a.h, lv.y, la.y), __fmaf_rn(a.h, lv.z, la.z), 0.f);
}

__global__ void __launch_bounds__(SYM_WARPS * 32) adjoint_vjp_sym_kernel(SymArgs a) {
    __shared__ float4 sxm[SYM_T], sw[SYM_T], sacc[SYM_T];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, tid = threadIdx.x;
    const int64_t c = blockIdx.x;
    const int64_t p0 = a.NP * c / a.P, p1 = a.NP * (c + 1) / a.P;
    if (p0 >= p1) return;
    int64_t p = p0;
    int64_t I = sym_row(p, a.nt);
    int64_t rbase = sym_base(I, a.nt);
    float X[2], Y[2], Z[2], M[2], WX[2], WY[2], WZ[2], AX[2], AY[2], AZ[2], AG[2];
    auto load_row = [&]() {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int64_t i = I * SYM_T + 64 * wib + 32 * q + lane;
            const float4 x = i < a.n ? __ldg(a.xm + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 w = sym_w(a, i);
            X[q] = x.x; Y[q] = x.y; Z[q] = x.z; M[q] = x.w;
            WX[q] = w.x; WY[q] = w.y; WZ[q] = w.z;
            AX[q] = AY[q] = AZ[q] = AG[q] = 0.f;
        }
    };
    load_row();
    while (p < p1) {
        const int64_t J = I + (p - rbase);
        const bool diag = J == I;
        // Stage tile J.
        __syncthreads();
        for (int t = tid; t < SYM_T; t += SYM_WARPS * 32) {
            const int64_t j = J * SYM_T + t;
            sxm[t] = j < a.n ? __ldg(a.xm + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            sw[t] = sym_w(a, j);
            sacc[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        if (!diag) {
            // Off-diagonal tile pair: every (target, source) pair, no masks.
            for (int r = 0; r < 8; ++r) {
                const int g = (2 * wib + r) & 7;
                const float4 *bx = sxm + g * 32, *bw = sw + g * 32;
                float4 *bacc = sacc + g * 32;
#pragma unroll 4
                for (int k = 0; k < 32; ++k) {
                    const int jj = (lane + k) & 31;
                    const float4 xs = bx[jj], ws = bw[jj];
                    float px = 0.f, py = 0.f, pz = 0.f, pg = 0.f;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float dx = xs.x - X[q], dy = xs.y - Y[q], dz = xs.z - Z[q];
                        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, a.eps2)));
                        const float inv = rsqrt_approx(r2);
                        const float inv2 = inv * inv;
                        const float sv = inv * inv2;
                        // P = sv (u - 3 inv2 (d.u) d), applied with opposite
                        // signs to both sides without forming P.
                        const float ux = __fmaf_rn(-M[q], ws.x, xs.w * WX[q]);
                        const float uy = __fmaf_rn(-M[q], ws.y, xs.w * WY[q]);
                        const float uz = __fmaf_rn(-M[q], ws.z, xs.w * WZ[q]);
                        const float du = __fmaf_rn(dz, uz, __fmaf_rn(dy, uy, dx * ux));
                        const float e = (3.f * inv2) * du;
                        const float vx = __fmaf_rn(-e, dx, ux), vy = __fmaf_rn(-e, dy, uy), vz = __fmaf_rn(-e, dz, uz);
                        const float dwi = __fmaf_rn(dz, WZ[q], __fmaf_rn(dy, WY[q], dx * WX[q]));
                        const float dwj = __fmaf_rn(dz, ws.z, __fmaf_rn(dy, ws.y, dx * ws.x));
                        AX[q] = __fmaf_rn(-sv, vx, AX[q]);
                        AY[q] = __fmaf_rn(-sv, vy, AY[q]);
                        AZ[q] = __fmaf_rn(-sv, vz, AZ[q]);
                        AG[q] = __fmaf_rn(-sv, dwj, AG[q]);
                        px = __fmaf_rn(sv, vx, px);
                        py = __fmaf_rn(sv, vy, py);
                        pz = __fmaf_rn(sv, vz, pz);
                        pg = __fmaf_rn(sv, dwi, pg);
                    }
                    float4 acc = bacc[jj];
                    acc.x += px; acc.y += py; acc.z += pz; acc.w += pg;
                    bacc[jj] = acc;
                    __syncwarp();
                }
                __syncthreads();
            }
        } else {
            for (int r = 0; r < 8; ++r) {
                const int g = (2 * wib + r) & 7;
                // Diagonal tile: slot group ga meets group g fully if ga < g, half
                // the in-group pairs if ga == g, and not at all if ga > g.
                int act[2];
    #pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int ga = 2 * wib + q;
                    act[q] = !diag ? 2 : (ga < g ? 2 : (ga == g ? 1 : 0));
                }
                // Warp-uniform skip; every warp still reaches the barrier below.
                const int nsteps = (act[0] == 0 && act[1] == 0) ? 0 : 32;
    #pragma unroll 2
                for (int k = 0; k < nsteps; ++k) {
                    const int jj = g * 32 + ((lane + k) & 31);
                    const float4 xs = sxm[jj], ws = sw[jj];
                    const bool half_on = (k >= 1 && k < 16) || (k == 16 && lane < 16);
                    float px = 0.f, py = 0.f, pz = 0.f, pg = 0.f;
    #pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const bool on = act[q] == 2 || (act[q] == 1 && half_on);
                        const float dx = xs.x - X[q], dy = xs.y - Y[q], dz = xs.z - Z[q];
                        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, a.eps2)));
                        const float inv = rsqrt_approx(r2);
                        const float inv2 = inv * inv;
                        const float sv = on ? inv * inv2 : 0.f;
                        const float ux = __fmaf_rn(-M[q], ws.x, xs.w * WX[q]);
                        const float uy = __fmaf_rn(-M[q], ws.y, xs.w * WY[q]);
                        const float uz = __fmaf_rn(-M[q], ws.z, xs.w * WZ[q]);
                        const float du = __fmaf_rn(dz, uz, __fmaf_rn(dy, uy, dx * ux));
                        const float e = (3.f * inv2) * du;
                        const float vx = __fmaf_rn(-e, dx, ux), vy = __fmaf_rn(-e, dy, uy), vz = __fmaf_rn(-e, dz, uz);
                        const float dwi = __fmaf_rn(dz, WZ[q], __fmaf_rn(dy, WY[q], dx * WX[q]));
                        const float dwj = __fmaf_rn(dz, ws.z, __fmaf_rn(dy, ws.y, dx * ws.x));
                        AX[q] = __fmaf_rn(-sv, vx, AX[q]);
                        AY[q] = __fmaf_rn(-sv, vy, AY[q]);
                        AZ[q] = __fmaf_rn(-sv, vz, AZ[q]);
                        AG[q] = __fmaf_rn(-sv, dwj, AG[q]);
                        px = __fmaf_rn(sv, vx, px);
                        py = __fmaf_rn(sv, vy, py);
                        pz = __fmaf_rn(sv, vz, pz);
                        pg = __fmaf_rn(sv, dwi, pg);
                    }
                    float4 acc = sacc[jj];
                    acc.x += px; acc.y += py; acc.z += pz; acc.w += pg;
                    sacc[jj] = acc;
                    __syncwarp();
                }
                __syncthreads();
            }
        }
        // Source-side sums of this tile pair.
        for (int t = tid; t < SYM_T; t += SYM_WARPS * 32) a.colpart[p * SYM_T + t] = sacc[t];
        ++p;
        if (p == p1 || p == rbase + (a.nt - I)) {  // row (or run) ends: flush tile I's sums
#pragma unroll
            for (int q = 0; q < 2; ++q)
                a.rowpart[(I + c) * SYM_T + 64 * wib + 32 * q + lane] = make_float4(AX[q], AY[q], AZ[q], AG[q]);
            if (p < p1) {
                ++I;
                rbase = sym_base(I, a.nt);
                load_row();
            }
        }
    }
}

// ------------------------------------- symmetric evaluation, packed pairs
// The pair algebra of adjoint_vjp_sym_kernel in .f32x2 arithmetic, where one
// instruction serves two (target, source) pairs.  Tiles of SYM2_T = 512
// particles; 4 warps, 4 targets per lane held as two packed pairs (targets
// q = 0, 1 and q = 2, 3; lane l of warp w owns targets 128 w + 32 q + l).
// A unit is one unordered tile pair (I <= J) and one of Q source slices of
// tile J (512 / Q sources, G = 16 / Q groups of 32).  CTAs take units from
// an atomic counter, so CTAs that the schedulers favour take more units and
// all of them stay resident until the work runs out; each unit writes its
// own row slot (tile I's sums over the slice) and its slice of the pair's
// column slot, and the fix-up adds the slots in a fixed order, so results
// do not depend on which CTA did which unit.  In round r warp w takes group
// g = (G/4 w + r) mod G of the slice (distinct across the warps of a round)
// and at step k lane l source 32 g + (l + k) mod 32, so no two lanes update
// one source accumulator at once.  Target sums N = sum sv v (and sum sv
// d.w_source) stay in registers and are written negated.  On the diagonal
// tile a pair (t, s) counts when t < s; the self pair is exactly zero.
constexpr int SYM2_T = 512;
template <int TILE>
constexpr int SYM2_WARPS = TILE / 128;
// Small systems (at most SYM2_SMALL_N particles): tiles of 256, two warps, four
// source slices per tile pair.  As in the force pass the time is one unit's
// length while the units fit one wave, and half of it here.  Microseconds per
// VJP with its fix-up, tiles of 512 / 256: 1,000: 21.4 / 13.2; 4,096: 22.3 / 20.5;
// 6,144: 48.7 / 34.7; 8,000: 63.0 / 60.6 (10,000: 94.3 / 88.2, so the line could
// lie a little higher).
constexpr int SYM2_SMALL_T = 256, SYM2_SMALL_Q = 4;
constexpr int64_t SYM2_SMALL_N = 8192;

struct Sym2Args {
    const float4 *__restrict__ xm;
    const float4 *__restrict__ lv;
    const float4 *__restrict__ la;
    float4 *__restrict__ rowpart;  // NU x SYM2_T (one row slot per unit)
    float4 *__restrict__ colpart;  // band pairs x SYM2_T
    unsigned long long *counter;   // zero at launch; NULL: one unit per CTA
    int64_t n, nt, NU, p0;         // units of the band, its first tile pair
    float eps2, h;
    int prime;
};

__device__ __forceinline__ float4 sym2_w(const Sym2Args &a, int64_t i) {
    if (i >= a.n) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 la = __ldg(a.la + i);
    if (a.prime) return la;
    const float4 lv = __ldg(a.lv + i);
    return make_float4(__fmaf_rn(a.h, lv.x, la.x), __fmaf_rn(a.h, lv.y, la.y), __fmaf_rn(a.h, lv.z, la.z), 0.f);
}

// A lane's four targets, two by two, with their sums.
struct Sym2Half {
    f2 TX, TY, TZ, TNM, TWX, TWY, TWZ, NX, NY, NZ, NG;
};

// One source against two of the lane's targets, HH the first (0) or the second
// half; the source's sums in PX .. PG.  -3 d.u, with u = m_s w_t - m_t w_s, comes
// from the two dot products: (-3 m_s) d.w_t + (3 m_t) d.w_s.  DIAG masks the
// pairs with target index >= source index (diagonal tile).
template <bool DIAG, int HH>
__device__ __forceinline__ void sym2_half(Sym2Half &t, float4 xs, float4 ws, int jj, int lane, int wib, float eps2,
                                          f2 &PX, f2 &PY, f2 &PZ, f2 &PG) {
    const f2 sx = pack2(xs.x, xs.x), sy = pack2(xs.y, xs.y), sz = pack2(xs.z, xs.z), sm = pack2(xs.w, xs.w);
    const f2 swx = pack2(ws.x, ws.x), swy = pack2(ws.y, ws.y), swz = pack2(ws.z, ws.z);
    const f2 E = pack2(eps2, eps2), NEG3 = pack2(-3.f, -3.f);
    const f2 sm3 = mul2(sm, NEG3), TM3 = mul2(t.TNM, NEG3);
    const f2 dx = sub2(sx, t.TX), dy = sub2(sy, t.TY), dz = sub2(sz, t.TZ);
    const f2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, E)));
    const f2 inv = rsqrt2(r2);
    const f2 inv2 = mul2(inv, inv);
    f2 sv = mul2(inv, inv2);
    if (DIAG) {
        float q0, q1;
        unpack2(sv, q0, q1);
        const int t0 = 128 * wib + 64 * HH + lane;
        q0 = t0 < jj ? q0 : 0.f;
        q1 = t0 + 32 < jj ? q1 : 0.f;
        sv = pack2(q0, q1);
    }
    const f2 ux = fma2(t.TNM, swx, mul2(sm, t.TWX));
    const f2 uy = fma2(t.TNM, swy, mul2(sm, t.TWY));
    const f2 uz = fma2(t.TNM, swz, mul2(sm, t.TWZ));
    const f2 dwt = fma2(dz, t.TWZ, fma2(dy, t.TWY, mul2(dx, t.TWX)));
    const f2 dws = fma2(dz, swz, fma2(dy, swy, mul2(dx, swx)));
    const f2 ne = mul2(inv2, fma2(sm3, dwt, mul2(TM3, dws)));
    const f2 vx = fma2(ne, dx, ux), vy = fma2(ne, dy, uy), vz = fma2(ne, dz, uz);
    t.NX = fma2(sv, vx, t.NX);
    t.NY = fma2(sv, vy, t.NY);
    t.NZ = fma2(sv, vz, t.NZ);
    t.NG = fma2(sv, dws, t.NG);
    PX = fma2(sv, vx, PX);
    PY = fma2(sv, vy, PY);
    PZ = fma2(sv, vz, PZ);
    PG = fma2(sv, dwt, PG);
}

// One round of sym2 pair steps: lane l at step k takes source jj =
// 32 g + (l + k) mod 32 of the staged tile against its 4 targets.  Bound by the
// FMA pipe (math-pipe throttle at 65% of it, issue 63%): one half in scalar
// arithmetic, twice as many targets a lane, sources staged twice against
// register moves and fewer barriers measured the same or slower (n = 65,536:
// 2.95, 3.00, 3.18 and 3.06 ms, this 2.94).
template <bool DIAG, int UNROLL>
__device__ __forceinline__ void sym2_round(const float4 *__restrict__ sxm, const float4 *__restrict__ sw,
                                           float4 *sacc, int g, int lane, int wib, float eps2, Sym2Half &A,
                                           Sym2Half &B) {
    // The next step's source is read one step ahead: where a block is alone on
    // its SM the read's latency was not covered (VJP and fix-up of 1,000
    // particles: 18.7 to 16.7 us; of 4,096 and more: the same).
    float4 xn = sxm[g * 32 + lane], wn = sw[g * 32 + lane];
#pragma unroll UNROLL
    for (int k = 0; k < 32; ++k) {
        const int jj = g * 32 + ((lane + k) & 31), jn = g * 32 + ((lane + k + 1) & 31);
        const float4 xs = xn, ws = wn;
        xn = sxm[jn];
        wn = sw[jn];
        f2 PX = 0ull, PY = 0ull, PZ = 0ull, PG = 0ull;
        sym2_half<DIAG, 0>(A, xs, ws, jj, lane, wib, eps2, PX, PY, PZ, PG);
        sym2_half<DIAG, 1>(B, xs, ws, jj, lane, wib, eps2, PX, PY, PZ, PG);
        float4 acc = sacc[jj];
        float lo, hi;
        unpack2(PX, lo, hi);
        acc.x += lo + hi;
        unpack2(PY, lo, hi);
        acc.y += lo + hi;
        unpack2(PZ, lo, hi);
        acc.z += lo + hi;
        unpack2(PG, lo, hi);
        acc.w += lo + hi;
        sacc[jj] = acc;
        __syncwarp();
    }
}

template <int Q, int TILE>
__global__ void __launch_bounds__(SYM2_WARPS<TILE> * 32, 16 / SYM2_WARPS<TILE>) adjoint_vjp_sym2_kernel(Sym2Args a) {
    constexpr int WARPS = SYM2_WARPS<TILE>, G = TILE / 32 / Q, SPAN = G * 32;
    // Steps unrolled, 2 / 3: 4,096 particles 26.7 / 25.4 us; 65,536 (two slices): 2.94
    // / 3.01 ms; in one slice 72,000: 3.65 / 3.56 ms, 80,000: 4.51 / 4.43, 130,000:
    // 11.60 / 11.48.
    constexpr int UNROLL = TILE == SYM2_SMALL_T || Q == 1 ? 3 : 2;
    static_assert(G >= WARPS, "each warp of a round takes its own source group");
    __shared__ float4 sxm[TILE], sw[TILE], sacc[TILE];
    __shared__ long long s_unit;
    __shared__ int s_gend, s_ntgt;  // source groups and targets of the unit that hold particles
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, tid = threadIdx.x;
    const int64_t NU = a.NU;
    if (tid == 0) s_unit = -1;
    for (;;) {
        __syncthreads();  // the previous unit is done with s_unit and shared memory
        if (tid == 0)
            s_unit = a.counter ? (long long)atomicAdd(a.counter, 1ull) : s_unit < 0 ? (long long)blockIdx.x : (long long)NU;
        __syncthreads();
        Sym2Half half[2];
        bool diag;
        int gbase;
        {
        // Unit bookkeeping is re-read from shared memory after the pair
        // loop, so none of it stays in registers across the loop.
        const int64_t u = s_unit;
        if (u >= NU) break;
        const int64_t p = u / Q;
        const int sl = (int)(u - p * Q);
        const int64_t pg = a.p0 + p;  // pair index in the triangle
        const int64_t I = sym_row(pg, a.nt);
        const int64_t J = I + (pg - sym_base(I, a.nt));
        diag = J == I;
        gbase = sl * G;
        // Padding of the last tile (zero mass and zero w) adds exact zeros:
        // its source groups and all-padding target warps are skipped.
        if (tid == 0) {
            s_gend = (int)((min(a.n - J * TILE, (int64_t)TILE) + 31) / 32);
            s_ntgt = (int)min(a.n - I * TILE, (int64_t)TILE);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float4 x[2], w[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int64_t i = I * TILE + 128 * wib + 32 * (2 * h + e) + lane;
                x[e] = i < a.n ? __ldg(a.xm + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                w[e] = sym2_w(a, i);
            }
            Sym2Half &q = half[h];
            q.TX = pack2(x[0].x, x[1].x);
            q.TY = pack2(x[0].y, x[1].y);
            q.TZ = pack2(x[0].z, x[1].z);
            q.TNM = pack2(-x[0].w, -x[1].w);
            q.TWX = pack2(w[0].x, w[1].x);
            q.TWY = pack2(w[0].y, w[1].y);
            q.TWZ = pack2(w[0].z, w[1].z);
            q.NX = q.NY = q.NZ = q.NG = 0ull;
        }
        // Stage the slice's sources (tile-local indices sl*SPAN .. +SPAN-1).
        for (int t = tid; t < SPAN; t += WARPS * 32) {
            const int tt = sl * SPAN + t;
            const int64_t j = J * TILE + tt;
            sxm[tt] = j < a.n ? __ldg(a.xm + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            sw[tt] = sym2_w(a, j);
            sacc[tt] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        }
        __syncthreads();
        for (int r = 0; r < G; ++r) {
            const int g = gbase + (((G / WARPS) * wib + r) & (G - 1));
            // Diagonal tile: targets 128 w .. 128 w + 127 against sources
            // 32 g .. 32 g + 31; no pair has t < s when 4 w > g.
            // Warp-uniform branches; every warp still reaches the barrier.
            if (128 * wib < s_ntgt && g < s_gend) {
                if (!diag)
                    sym2_round<false, UNROLL>(sxm, sw, sacc, g, lane, wib, a.eps2, half[0], half[1]);
                else if (4 * wib <= g)
                    sym2_round<true, UNROLL>(sxm, sw, sacc, g, lane, wib, a.eps2, half[0], half[1]);
            }
            __syncthreads();
        }
        const int64_t u = s_unit;
        const int64_t p = u / Q;
        const int sl = (int)(u - p * Q);
        for (int t = tid; t < SPAN; t += WARPS * 32) {
            const int tt = sl * SPAN + t;
            a.colpart[p * TILE + tt] = sacc[tt];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float x0, x1, y0, y1, z0, z1, g0, g1;
            unpack2(half[h].NX, x0, x1);
            unpack2(half[h].NY, y0, y1);
            unpack2(half[h].NZ, z0, z1);
            unpack2(half[h].NG, g0, g1);
            float4 *row = a.rowpart + u * TILE + 128 * wib + 64 * h + lane;
            row[0] = make_float4(-x0, -y0, -z0, -g0);
            row[32] = make_float4(-x1, -y1, -z1, -g1);
        }
    }
}

struct Sym2Fix {
    const float4 *__restrict__ rowpart;
    const float4 *__restrict__ colpart;
    float4 *lx, *lv, *la;
    float *lm;
    float4 *aux;  // running sums of particles past the band (one float4 each)
    int64_t n, nt, Ib, Ie, p0;
    int Q;
    float G, h, dt;
    int prime;
};

// Particle i (in tile T, at or after the band's first row Ib) adds, in a
// fixed order: the running sum left by earlier bands, its row units
// (T, J, slice) for J = T .. nt-1 when T is in the band, then its column
// slots (I', T) for the band's rows I' <= T.  A particle of the band is
// complete and gets the elementwise part of the backward step; one past the
// band keeps its running sum in aux.  Later bands never read a finished
// tile, so its adjoint state may change.  One band (Ib = 0, Ie = nt) is the
// whole pass.  A CTA takes 32 particles: warp w adds slots w, w + 8, ...
// (512-byte rows), and warp 0 adds the warps' sums in order.  n = 65,536:
// 38 us against 55 us with one thread for all slots of a particle, 4,096: 3.5
// us against 4.8.
constexpr int SYM2_FIX_WARPS = 8;

template <int TILE>
__global__ void __launch_bounds__(SYM2_FIX_WARPS * 32) adjoint_sym2_fixup_kernel(Sym2Fix f) {
    __shared__ float4 part[SYM2_FIX_WARPS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i0 = f.Ib * TILE + (int64_t)blockIdx.x * 32, i = i0 + lane;
    const int64_t T = i0 / TILE, r = i - T * TILE;
    const bool in_band = T < f.Ie;
    const int64_t R = in_band ? (f.nt - T) * f.Q : 0;          // row slots
    const int64_t C = (in_band ? T : f.Ie - 1) - f.Ib + 1;     // column slots
    const int64_t rbase = (sym_base(T, f.nt) - f.p0) * f.Q;
    float gx = 0.f, gy = 0.f, gz = 0.f, gm = 0.f;
    auto add = [&](float4 v) {
        gx += v.x; gy += v.y; gz += v.z; gm += v.w;
    };
    // Slots of padded particles (i >= n) lie inside the scratch; their sums are dropped below.
    const float4 *row = f.rowpart + rbase * TILE + r;
    const int nr = (int)R, nc = (int)C;
#pragma unroll 4
    for (int k = w; k < nr; k += SYM2_FIX_WARPS) add(row[(int64_t)k * TILE]);
    const float4 *col = f.colpart + (T - f.p0) * TILE + r;
#pragma unroll 4
    for (int k = (nr + SYM2_FIX_WARPS - 1 - w) / SYM2_FIX_WARPS * SYM2_FIX_WARPS + w - nr; k < nc; k += SYM2_FIX_WARPS) {
        const int64_t I2 = f.Ib + k;
        add(col[(sym_base(I2, f.nt) - I2) * TILE]);
    }
    part[w][lane] = make_float4(gx, gy, gz, gm);
    __syncthreads();
    if (w != 0 || i >= f.n) return;
    gx = gy = gz = gm = 0.f;
    if (f.Ib > 0) add(f.aux[i]);
#pragma unroll
    for (int q = 0; q < SYM2_FIX_WARPS; ++q) add(part[q][lane]);
    if (!in_band) {
        f.aux[i] = make_float4(gx, gy, gz, gm);
        return;
    }
    gx *= f.G; gy *= f.G; gz *= f.G; gm *= f.G;
    f.lm[i] += gm;
    const float4 lx = f.lx[i];
    const float tx = lx.x + gx, ty = lx.y + gy, tz = lx.z + gz;
    if (f.prime) {
        f.lx[i] = make_float4(tx, ty, tz, 0.f);
        return;
    }
    const float4 lv = f.lv[i];
    const float hx = __fmaf_rn(f.dt, tx, lv.x), hy = __fmaf_rn(f.dt, ty, lv.y), hz = __fmaf_rn(f.dt, tz, lv.z);
    f.lx[i] = make_float4(tx, ty, tz, 0.f);
    f.lv[i] = make_float4(hx, hy, hz, 0.f);
    f.la[i] = make_float4(f.h * hx, f.h * hy, f.h * hz, 0.f);
}

struct SymFix {
    const float4 *__restrict__ rowpart;
    const float4 *__restrict__ colpart;
    float4 *lx, *lv, *la;
    float *lm;
    int64_t n, nt, NP, P;
    float G, h, dt;
    int prime;
};

__global__ void adjoint_sym_fixup_kernel(SymFix f) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= f.n) return;
    const int64_t I = i / SYM_T, r = i - I * SYM_T;
    const int64_t b0 = sym_base(I, f.nt), b1 = b0 + (f.nt - I) - 1;
    const int64_t c_lo = ((b0 + 1) * f.P - 1) / f.NP, c_hi = ((b1 + 1) * f.P - 1) / f.NP;
    float gx = 0.f, gy = 0.f, gz = 0.f, gm = 0.f;
    for (int64_t c = c_lo; c <= c_hi; ++c) {
        const float4 v = f.rowpart[(I + c) * SYM_T + r];
        gx += v.x; gy += v.y; gz += v.z; gm += v.w;
    }
    for (int64_t I2 = 0; I2 <= I; ++I2) {
        const float4 v = f.colpart[(sym_base(I2, f.nt) + (I - I2)) * SYM_T + r];
        gx += v.x; gy += v.y; gz += v.z; gm += v.w;
    }
    gx *= f.G; gy *= f.G; gz *= f.G; gm *= f.G;
    f.lm[i] += gm;
    const float4 lx = f.lx[i];
    const float tx = lx.x + gx, ty = lx.y + gy, tz = lx.z + gz;
    if (f.prime) {
        f.lx[i] = make_float4(tx, ty, tz, 0.f);
        return;
    }
    const float4 lv = f.lv[i];
    const float hx = __fmaf_rn(f.dt, tx, lv.x), hy = __fmaf_rn(f.dt, ty, lv.y), hz = __fmaf_rn(f.dt, tz, lv.z);
    f.lx[i] = make_float4(tx, ty, tz, 0.f);
    f.lv[i] = make_float4(hx, hy, hz, 0.f);
    f.la[i] = make_float4(f.h * hx, f.h * hy, f.h * hz, 0.f);
}


// Grows the handle's symmetric scratch to at least need float4 elements.

}  // namespace gb

using namespace gb;

extern "C" int gb_adjoint_step(gb_direct_t *h, const float *xm, float *lx, float *lv, float *la, float *lm,
                               int64_t n, float G, float eps2, float dt, int prime, void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (n < 0 || n > h->n_max) return fail(GB_EINVAL, "n=%lld outside [0, n_max=%lld]", (long long)n,
                                           (long long)h->n_max);
    if (n == 0) return GB_OK;
    const void *ptrs[] = {xm, lx, lv, la};
    const char *names[] = {"xm", "lx", "lv", "la"};
    for (int k = 0; k < 4; ++k) {
        if (!ptrs[k]) return fail(GB_EINVAL, "%s is NULL", names[k]);
        if (!aligned16(ptrs[k])) return fail(GB_EINVAL, "%s is not 16-byte aligned", names[k]);
    }
    if (!lm) return fail(GB_EINVAL, "lm is NULL");
    if (!(eps2 > 0.f)) return fail(GB_EINVAL, "eps2 must be > 0");
    cudaStream_t s = (cudaStream_t)stream;
    if (h->adj_variant == 2) {
        // Small tiles where one band holds their slots.
        const bool small = n <= SYM2_SMALL_N && sym_one_band(n, SYM2_SMALL_T, SYM2_SMALL_Q, h->sym_band);
        const int tile = small ? SYM2_SMALL_T : SYM2_T;
        const int64_t nt = (n + tile - 1) / tile, NP = nt * (nt + 1) / 2;
        int occs = 0;
        if (small)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occs, adjoint_vjp_sym2_kernel<SYM2_SMALL_Q, SYM2_SMALL_T>,
                                                          SYM2_WARPS<SYM2_SMALL_T> * 32, 0);
        else
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occs, adjoint_vjp_sym2_kernel<1, SYM2_T>,
                                                          SYM2_WARPS<SYM2_T> * 32, 0);
        const int64_t slots = (int64_t)h->sms * std::max(occs, 1);
        const int Q = small ? SYM2_SMALL_Q : direct_sym_slices(NP, slots, 16 / SYM2_WARPS<SYM2_T>);
        // Bands of tile rows within the handle's slot budget, as for the
        // symmetric force pass.
        std::vector<int64_t> rows;
        const int64_t max_pairs =
            sym_bands(nt, h->sym_band / ((int64_t)sizeof(float4) * tile * (Q + 1)), rows);
        const int64_t aux = rows.size() > 2 ? n : 0;
        const int64_t need = max_pairs * Q * tile + max_pairs * tile + aux + 1;  // + the unit counter
        const bool counted = max_pairs * Q > slots;
        if (need * (int64_t)sizeof(float4) <= SYM_MAX_BYTES) {
            GB_TRY(ensure_sym(h, need, [&] {
                int occ1 = 0;
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ1, adjoint_vjp_sym2_kernel<1, SYM2_T>,
                                                              SYM2_WARPS<SYM2_T> * 32, 0);
                return sym_most(n, h->sym_band, SYM2_T, (int64_t)h->sms * std::max(occ1, 1), 16 / SYM2_WARPS<SYM2_T>,
                                SYM2_SMALL_T, SYM2_SMALL_Q, SYM2_SMALL_N, 1);
            }));
            Sym2Args a;
            a.xm = (const float4 *)xm;
            a.lv = (const float4 *)lv;
            a.la = (const float4 *)la;
            a.rowpart = h->sym;
            a.colpart = h->sym + max_pairs * Q * tile;
            a.counter = counted ? (unsigned long long *)(h->sym + need - 1) : nullptr;
            a.n = n;
            a.nt = nt;
            a.eps2 = eps2;
            a.h = 0.5f * dt;
            a.prime = prime ? 1 : 0;
            Sym2Fix f;
            f.rowpart = a.rowpart;
            f.colpart = a.colpart;
            f.aux = a.colpart + max_pairs * tile;
            f.lx = (float4 *)lx;
            f.lv = (float4 *)lv;
            f.la = (float4 *)la;
            f.lm = lm;
            f.n = n;
            f.nt = nt;
            f.Q = Q;
            f.G = G;
            f.h = 0.5f * dt;
            f.dt = dt;
            f.prime = a.prime;
            for (size_t b = 0; b + 1 < rows.size(); ++b) {
                a.p0 = host_sym_base(rows[b], nt);
                a.NU = (host_sym_base(rows[b + 1], nt) - a.p0) * Q;
                f.Ib = rows[b];
                f.Ie = rows[b + 1];
                f.p0 = a.p0;
                const unsigned P = (unsigned)std::min(slots, a.NU);
                if (counted) GB_CUDA_TRY(cudaMemsetAsync(a.counter, 0, sizeof(unsigned long long), s));
                const unsigned b1 = SYM2_WARPS<SYM2_T> * 32;
                if (small)
                    adjoint_vjp_sym2_kernel<SYM2_SMALL_Q, SYM2_SMALL_T><<<P, SYM2_WARPS<SYM2_SMALL_T> * 32, 0, s>>>(a);
                else if (Q == 1) adjoint_vjp_sym2_kernel<1, SYM2_T><<<P, b1, 0, s>>>(a);
                else if (Q == 2) adjoint_vjp_sym2_kernel<2, SYM2_T><<<P, b1, 0, s>>>(a);
                else adjoint_vjp_sym2_kernel<4, SYM2_T><<<P, b1, 0, s>>>(a);
                GB_CUDA_TRY(cudaGetLastError());
                const unsigned fgrid = (unsigned)((n - f.Ib * tile + 31) / 32);
                if (small) adjoint_sym2_fixup_kernel<SYM2_SMALL_T><<<fgrid, SYM2_FIX_WARPS * 32, 0, s>>>(f);
                else adjoint_sym2_fixup_kernel<SYM2_T><<<fgrid, SYM2_FIX_WARPS * 32, 0, s>>>(f);
                GB_CUDA_TRY(cudaGetLastError());
                h->launches += 2;
            }
            return GB_OK;
        }
    }
    if (h->adj_variant == 1) {
        const int64_t nt = (n + SYM_T - 1) / SYM_T, NP = nt * (nt + 1) / 2;
        int occs = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occs, adjoint_vjp_sym_kernel, SYM_WARPS * 32, 0);
        const int64_t P = std::max<int64_t>(1, std::min<int64_t>((int64_t)h->sms * std::max(occs, 1), NP));
        const int64_t need = (nt + P) * SYM_T + NP * SYM_T;
        if (need * (int64_t)sizeof(float4) <= SYM_MAX_BYTES) {
            GB_TRY(ensure_sym(h, need, [&] { return need; }));
            SymArgs a;
            a.xm = (const float4 *)xm;
            a.lv = (const float4 *)lv;
            a.la = (const float4 *)la;
            a.rowpart = h->sym;
            a.colpart = h->sym + (nt + P) * SYM_T;
            a.n = n;
            a.nt = nt;
            a.NP = NP;
            a.P = P;
            a.eps2 = eps2;
            a.h = 0.5f * dt;
            a.prime = prime ? 1 : 0;
            adjoint_vjp_sym_kernel<<<(unsigned)P, SYM_WARPS * 32, 0, s>>>(a);
            GB_CUDA_TRY(cudaGetLastError());
            SymFix f;
            f.rowpart = a.rowpart;
            f.colpart = a.colpart;
            f.lx = (float4 *)lx;
            f.lv = (float4 *)lv;
            f.la = (float4 *)la;
            f.lm = lm;
            f.n = n;
            f.nt = nt;
            f.NP = NP;
            f.P = P;
            f.G = G;
            f.h = 0.5f * dt;
            f.dt = dt;
            f.prime = a.prime;
            adjoint_sym_fixup_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(f);
            GB_CUDA_TRY(cudaGetLastError());
            h->launches += 2;
            return GB_OK;
        }
    }
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, adjoint_vjp_kernel<VJP_K, VJP_WARPS>, VJP_WARPS * 32, 0);
    int64_t P = (int64_t)h->sms * std::max(occ, 1);
    DirectPlan pl;
    make_plan(n, VJP_K / 2, VJP_WARPS, P, &pl);
    while (plan_partials(pl) > h->part_cap && P > 1) {  // stay inside the handle's scratch
        P = P / 2;
        make_plan(n, VJP_K / 2, VJP_WARPS, P, &pl);
    }
    if (plan_partials(pl) > h->part_cap) return fail(GB_EINVAL, "adjoint scratch too small for n=%lld", (long long)n);
    VjpArgs a;
    a.xm = (const float4 *)xm;
    a.lv = (const float4 *)lv;
    a.la = (const float4 *)la;
    a.part = h->part;
    a.n = n;
    a.num_ju = pl.num_ju;
    a.U = pl.U;
    a.P = pl.P;
    a.smax = pl.smax;
    a.eps2 = eps2;
    a.h = 0.5f * dt;
    a.prime = prime ? 1 : 0;
    adjoint_vjp_kernel<VJP_K, VJP_WARPS><<<(unsigned)pl.P, VJP_WARPS * 32, 0, s>>>(a);
    GB_CUDA_TRY(cudaGetLastError());
    VjpFix f;
    f.part = h->part;
    f.lx = (float4 *)lx;
    f.lv = (float4 *)lv;
    f.la = (float4 *)la;
    f.lm = lm;
    f.n = n;
    f.num_ju = pl.num_ju;
    f.U = pl.U;
    f.P = pl.P;
    f.st_size = pl.st_size;
    f.smax = pl.smax;
    f.G = G;
    f.h = 0.5f * dt;
    f.dt = dt;
    f.prime = a.prime;
    adjoint_fixup_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(f);
    GB_CUDA_TRY(cudaGetLastError());
    h->launches += 2;
    return GB_OK;
}

extern "C" int gb_adjoint_trajectory(gb_direct_t *h, float *xm, float *vel, float *acc, float *traj, int64_t n, float G,
                                     float eps2, float dt, int64_t nsteps, int flags, void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (n < 0 || n > h->n_max) return fail(GB_EINVAL, "n=%lld outside [0, n_max=%lld]", (long long)n,
                                           (long long)h->n_max);
    if (nsteps < 0) return fail(GB_EINVAL, "nsteps < 0");
    if (flags & ~GB_PLAIN_FP32) return fail(GB_EINVAL, "flags 0x%x: only GB_PLAIN_FP32 applies", flags);
    if (n > 0 && nsteps > 0) {
        if (!traj) return fail(GB_EINVAL, "traj is NULL");
        if (!aligned16(traj)) return fail(GB_EINVAL, "traj is not 16-byte aligned");
    }
    for (int64_t k = 0; k < nsteps; ++k) {
        GB_TRY(gb_direct_kdk(h, xm, vel, acc, n, G, eps2, dt, 1, flags, stream));
        if (n > 0)
            GB_CUDA_TRY(cudaMemcpyAsync(traj + 4 * k * n, xm, (size_t)n * 4 * sizeof(float), cudaMemcpyDeviceToDevice,
                                        (cudaStream_t)stream));
    }
    return GB_OK;
}

extern "C" int gb_adjoint_segment(gb_direct_t *h, const float *traj, const float *x_end, float *lx, float *lv,
                                  float *la, float *lm, int64_t n, float G, float eps2, float dt, int64_t nsteps,
                                  void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (nsteps < 0) return fail(GB_EINVAL, "nsteps < 0");
    if (n > 0 && nsteps > 1 && !traj) return fail(GB_EINVAL, "traj is NULL");
    for (int64_t k = nsteps - 1; k >= 0; --k)
        GB_TRY(gb_adjoint_step(h, k == nsteps - 1 ? x_end : traj + 4 * k * n, lx, lv, la, lm, n, G, eps2, dt, 0,
                               stream));
    return GB_OK;
}

extern "C" int gb_adjoint_set_variant(gb_direct_t *h, int variant) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    if (variant < 0 || variant > 2) return fail(GB_EINVAL, "variant must be 0, 1 or 2 (got %d)", variant);
    h->adj_variant = variant;
    return GB_OK;
}
