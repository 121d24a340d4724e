// Uniform neighbour grid over the gas particles, rebuilt on the device:
// NeighborGrid.rebuild / rebuild_all (core/solvers/neighbor_grid.py:49-136),
// which the reference runs in host numpy before uploading gsort and
// cell_start.  Same outputs, bit for bit:
//   cell   = max(2 h_max, min_radius) (1 if not > 1e-9), grown by 1.3 while
//            the grid has more than max_cells = max(64, 4n) cells;
//   dims   = max(floor((max - min) / cell) + 1, 1) per axis;
//   ijk    = clip(trunc((x - min) / cell), 0, dims - 1), all in FP64;
//   flat   = (i dims_y + j) dims_z + k;
//   gsort  = gas indices in stable order of flat, zero-padded to n;
//   cell_start[c] = number of gas particles with flat < c for c <= n_cells,
//            zero above.
// Stages (one stream, no host round trip):
//   1 grid_reduce_kernel  gas count, bounding box and h_max (block partials,
//                         merged by the last CTA, which also derives the
//                         geometry in FP64);
//   2 grid_key_kernel     cell key per particle; stars (and every particle
//                         when there is no gas) get a key that sorts last;
//   3 radix sort          stable, 8-bit digits, enough passes for max_cells;
//   4 grid_gsort_kernel / grid_start_kernel: outputs (skipped when there is
//                         no gas, which leaves them as the reference does).
#include <algorithm>
#include <climits>
#include <cmath>

#include "gb_common.cuh"
#include "gb_sort.cuh"

namespace gb {

constexpr int GRID_THREADS = 256;
constexpr int GRID_MAX_GROW = 4096;  // bound on the cell-growth loop

// Geometry of the last rebuild (device-resident; copied to gb_grid_info_t).
struct GridGeom {
    long long ngas, n_cells;
    int nx, ny, nz, status;  // status: 0 ok, 1 non-finite input, 2 growth loop did not converge
    double lo[3], cell, inv_cell;
    int active;              // this rebuild writes the outputs (ngas > 0)
    float lof[3], ih, il;    // lo and 1 / cell for cell_fp32
};

// The geometry and the sort's counters behind it in one allocation, read back
// in one copy (with a second one, of the counters: 126 us per rebuild
// of 1,000,000 particles, 116 without).
struct GridBack {
    GridGeom g;
    unsigned long long diag[DIAG_COUNT];
};
static_assert(sizeof(GridBack) == sizeof(GridGeom) + sizeof(unsigned long long) * DIAG_COUNT, "no padding");

struct GridPart {
    float mn[3], mx[3], hmax;
    unsigned long long count, nonfinite;
};

// numpy's float64 -> int64 cast on x86-64: truncation, and the "integer
// indefinite" value INT64_MIN for NaN and out-of-range inputs.
__device__ __forceinline__ long long np_trunc_i64(double t) {
    if (!(t < 9.2233720368547758e18 && t > -9.2233720368547758e18)) return (long long)(-9223372036854775807ll - 1);
    return __double2ll_rz(t);
}

__device__ __forceinline__ GridPart empty_part() {
    GridPart p;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        p.mn[a] = INFINITY;
        p.mx[a] = -INFINITY;
    }
    p.hmax = -INFINITY;
    p.count = p.nonfinite = 0;
    return p;
}

__device__ __forceinline__ GridPart merge_part(const GridPart &x, const GridPart &y) {
    GridPart p;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        p.mn[a] = fminf(x.mn[a], y.mn[a]);
        p.mx[a] = fmaxf(x.mx[a], y.mx[a]);
    }
    p.hmax = fmaxf(x.hmax, y.hmax);
    p.count = x.count + y.count;
    p.nonfinite = x.nonfinite + y.nonfinite;
    return p;
}

// Merge of a CTA's threads' partials, complete in thread 0; w: one per warp.
__device__ __forceinline__ GridPart cta_merge(GridPart p, GridPart *w) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        GridPart q;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            q.mn[a] = __shfl_xor_sync(0xffffffffu, p.mn[a], o);
            q.mx[a] = __shfl_xor_sync(0xffffffffu, p.mx[a], o);
        }
        q.hmax = __shfl_xor_sync(0xffffffffu, p.hmax, o);
        q.count = __shfl_xor_sync(0xffffffffu, p.count, o);
        q.nonfinite = __shfl_xor_sync(0xffffffffu, p.nonfinite, o);
        p = merge_part(p, q);
    }
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = p;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 1; k < GRID_THREADS / 32; ++k) p = merge_part(p, w[k]);
    return p;
}

// Bound by the latency of its tail, the merge and the FP64 divisions of the
// geometry.  The last CTA's threads share the merge of the block partials: at
// n = 1,000,000 10.8 us, against 71 us with 608 partials read one after the
// other by one thread.
__global__ void __launch_bounds__(GRID_THREADS)
grid_reduce_kernel(const float4 *__restrict__ xm, const float *__restrict__ hsml, const int *__restrict__ is_star,
                   int64_t n, double min_radius, long long max_cells, GridPart *part, unsigned *ticket,
                   GridGeom *geom, ZeroWords zero) {
    zero_words(zero);  // the sort's scratch
    float mn0 = INFINITY, mn1 = INFINITY, mn2 = INFINITY, mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY;
    float hm = -INFINITY;
    unsigned long long cnt = 0, bad = 0;
    // Four particles' loads at once: with one at a time, and its position read
    // after its star flag, the kernel took 15.5 us at n = 1,000,000, now 10.8.
    constexpr int U = 4;
    const int64_t step = (int64_t)gridDim.x * GRID_THREADS;
    for (int64_t i0 = (int64_t)blockIdx.x * GRID_THREADS + threadIdx.x; i0 < n; i0 += U * step) {
        float4 p[U];
        float hv[U];
        int star[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t i = i0 + u * step;
            star[u] = 1;
            if (i < n) {
                star[u] = is_star ? __ldg(is_star + i) : 0;
                p[u] = __ldg(xm + i);
                hv[u] = __ldg(hsml + i);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (star[u] != 0) continue;
            if (!(isfinite(p[u].x) && isfinite(p[u].y) && isfinite(p[u].z) && isfinite(hv[u]))) ++bad;
            mn0 = fminf(mn0, p[u].x); mn1 = fminf(mn1, p[u].y); mn2 = fminf(mn2, p[u].z);
            mx0 = fmaxf(mx0, p[u].x); mx1 = fmaxf(mx1, p[u].y); mx2 = fmaxf(mx2, p[u].z);
            hm = fmaxf(hm, hv[u]);
            ++cnt;
        }
    }
    __shared__ GridPart wpart[GRID_THREADS / 32];
    __shared__ bool last;
    GridPart bp;
    bp.mn[0] = mn0; bp.mn[1] = mn1; bp.mn[2] = mn2;
    bp.mx[0] = mx0; bp.mx[1] = mx1; bp.mx[2] = mx2;
    bp.hmax = hm;
    bp.count = cnt;
    bp.nonfinite = bad;
    bp = cta_merge(bp, wpart);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = bp;
        __threadfence();
        const unsigned t = atomicAdd(ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    // Last CTA: merge the block partials, one or a few per thread, and derive
    // the grid.
    __threadfence();
    bp = empty_part();
    for (unsigned b = threadIdx.x; b < gridDim.x; b += GRID_THREADS) {
        const GridPart *q = part + b;  // written by other CTAs: read past L1
        GridPart o;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            o.mn[a] = __ldcg(q->mn + a);
            o.mx[a] = __ldcg(q->mx + a);
        }
        o.hmax = __ldcg(&q->hmax);
        o.count = __ldcg(&q->count);
        o.nonfinite = __ldcg(&q->nonfinite);
        bp = merge_part(bp, o);
    }
    __syncthreads();  // wpart is read
    bp = cta_merge(bp, wpart);
    if (threadIdx.x != 0) return;
    *ticket = 0;  // ready for the next rebuild (stream-ordered)
    const float *mn = bp.mn, *mx = bp.mx, hmax = bp.hmax;
    const unsigned long long count = bp.count, nonfinite = bp.nonfinite;
    GridGeom g = *geom;  // a rebuild without gas keeps the previous geometry
    g.ngas = (long long)count;
    g.active = count > 0 ? 1 : 0;
    g.status = nonfinite ? 1 : 0;
    if (count > 0) {
        double cell = fmax(__dmul_rn(2.0, (double)hmax), min_radius);
        cell = cell > 1e-9 ? cell : 1.0;
        double lo[3], span[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = (double)mn[a];
            span[a] = __dsub_rn((double)mx[a], lo[a]);
        }
        long long dims[3];
        auto set_dims = [&]() {
            for (int a = 0; a < 3; ++a) {
                const long long f = np_trunc_i64(floor(__ddiv_rn(span[a], cell)));
                dims[a] = (f != LLONG_MIN && f + 1 > 1) ? f + 1 : 1;
            }
        };
        set_dims();
        int grow = 0;
        // Products past 2^53 are inexact in FP64 but far above max_cells.
        while ((double)dims[0] * (double)dims[1] * (double)dims[2] > (double)max_cells) {
            if (++grow > GRID_MAX_GROW) {
                g.status = 2;
                break;
            }
            cell = __dmul_rn(cell, 1.3);
            set_dims();
        }
        if (g.status == 2) {
            g.active = 0;
        } else {
            g.nx = (int)dims[0];
            g.ny = (int)dims[1];
            g.nz = (int)dims[2];
            g.n_cells = dims[0] * dims[1] * dims[2];
            for (int a = 0; a < 3; ++a) g.lo[a] = lo[a];
            g.cell = cell;
            g.inv_cell = __ddiv_rn(1.0, cell);
            for (int a = 0; a < 3; ++a) g.lof[a] = mn[a];
            split_fp32(g.inv_cell, g.ih, g.il);
        }
    }
    *geom = g;
}

// The FP64 cell index on one axis, where FP32 cannot decide.
__device__ __noinline__ uint32_t cell_fp64(float x, double lo, double cell, int dim) {
    const long long v = np_trunc_i64(__ddiv_rn(__dsub_rn((double)x, lo), cell));
    return (uint32_t)(v < 0 ? 0 : (v > dim - 1 ? dim - 1 : v));
}

// Cell key of particle i; stars and inactive rebuilds get n_cells (or 0),
// which sorts after every gas key.
struct CellKey {
    const float4 *__restrict__ xm;
    const int *__restrict__ is_star;
    const GridGeom *__restrict__ geom;

    __device__ __forceinline__ uint32_t operator()(int64_t i) const {
        const GridGeom &g = *geom;
        if (!g.active) return 0u;
        if (is_star && __ldg(is_star + i) != 0) return (uint32_t)g.n_cells;
        const float4 p = __ldg(xm + i);
        const float c[3] = {p.x, p.y, p.z}, ih = g.ih, il = g.il;
        const int dim[3] = {g.nx, g.ny, g.nz};
        uint32_t q[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (!cell_fp32(c[a], g.lof[a], ih, il, q[a])) q[a] = cell_fp64(c[a], g.lo[a], g.cell, dim[a]);
            q[a] = min(q[a], (uint32_t)(dim[a] - 1));
        }
        return (q[0] * (uint32_t)dim[1] + q[1]) * (uint32_t)dim[2] + q[2];
    }
};

// All keys, and the digit counts of the sort.  1M particles: 11.4 us, against
// 67.7 us with FP64 divisions and 13.7 us for a kernel that counted the digits.
__global__ void __launch_bounds__(GRID_THREADS)
grid_key_kernel(CellKey key, int64_t n, uint32_t *keys, uint32_t *counts, int passes) {
    __shared__ RsCount<4> cnt;
    cnt.clear();
    for (int64_t i = (int64_t)blockIdx.x * GRID_THREADS + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * GRID_THREADS) {
        const uint32_t k = key(i);
        keys[i] = k;
        cnt.add(k, passes);
    }
    cnt.flush(counts, passes);
}

__global__ void grid_gsort_kernel(const uint32_t *__restrict__ vals, int64_t n, const GridGeom *__restrict__ geom,
                                  int *gsort) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n || !geom->active) return;
    gsort[p] = p < geom->ngas ? (int)vals[p] : 0;
}

// cell_start[c] = lower bound of c in the sorted gas keys (c <= n_cells);
// 0 above n_cells, as the reference re-zeroes its field each rebuild.  A CTA
// takes START_CELLS consecutive cells: two warps search for the range of
// their keys, then every thread searches that range for its cells, all at
// once.  Most CTAs hold few keys or none, and their cells need few steps;
// the searches are chains of reads, so the chain is what counts.
// At n = 1,000,000 (4,000,000 cells): 8.3 us, against 17.7 us with one search
// over all keys (20 dependent reads) per cell, and 34.7 us with the range's
// keys counted per cell in shared memory (dense cells put most keys in a few
// CTAs).
constexpr int START_CELLS = 1024;

__global__ void __launch_bounds__(GRID_THREADS)
grid_start_kernel(const uint32_t *__restrict__ keys, const GridGeom *__restrict__ geom, long long max_cells,
                  int *__restrict__ cell_start) {
    constexpr int PER = START_CELLS / GRID_THREADS;  // cells per thread
    if (!geom->active) return;
    __shared__ int range[2];
    const int tid = threadIdx.x;
    const long long c0 = (long long)blockIdx.x * START_CELLS;
    const long long nc = geom->n_cells, ng = geom->ngas;
    int at[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) at[q] = 0;
    if (c0 <= nc) {
        if (tid < 64) {
            const int k = tid >> 5;
            const long long r = warp_bound(keys, ng, (uint32_t)(c0 + k * START_CELLS));
            if ((tid & 31) == 0) range[k] = (int)r;
        }
        __syncthreads();
        int len = range[1] - range[0];
#pragma unroll
        for (int q = 0; q < PER; ++q) at[q] = range[0];
        while (len > 0) {
            const int half = (len + 1) >> 1;
#pragma unroll
            for (int q = 0; q < PER; ++q)
                if ((long long)__ldg(keys + at[q] + half - 1) < c0 + q * GRID_THREADS + tid) at[q] += half;
            len -= half;
        }
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const long long c = c0 + q * GRID_THREADS + tid;
        if (c <= max_cells) cell_start[c] = c <= nc ? at[q] : 0;
    }
}

}  // namespace gb

using namespace gb;

struct gb_grid {
    int device;
    int64_t n;
    long long max_cells;
    double min_radius;
    int passes, red_blocks;
    uint32_t *keys[2], *vals[2], *sort_scratch;
    unsigned long long timeouts_seen;  // DIAG_WAIT_TIMEOUT at the last rebuild with info
    GridPart *part;
    unsigned *ticket;
    GridGeom *geom;            // a GridBack
    unsigned long long *diag;  // its counters
    uint64_t launches;
};

extern "C" int gb_grid_destroy(gb_grid_t *h) {
    if (!h) return GB_OK;
    void *ptrs[] = {h->keys[0], h->keys[1], h->vals[0], h->vals[1], h->sort_scratch, h->part, h->ticket,
                    h->geom};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    delete h;
    return GB_OK;
}

extern "C" int gb_grid_create(gb_grid_t **out, int64_t n, double min_radius) {
    if (!out) return fail(GB_EINVAL, "out is NULL");
    *out = nullptr;
    if (n < 0 || n > ((int64_t)1 << 29)) return fail(GB_EINVAL, "n=%lld out of range", (long long)n);
    if (!(min_radius >= 0.0) || !std::isfinite(min_radius)) return fail(GB_EINVAL, "min_radius must be finite and >= 0");
    gb_grid_t *h = new gb_grid();
    GB_CUDA_TRY(cudaGetDevice(&h->device));
    h->n = n;
    h->max_cells = std::max<long long>(64, 4 * (long long)n);
    h->min_radius = min_radius;
    int bits = 1;
    while (bits < 32 && (1ll << bits) <= h->max_cells) ++bits;  // keys <= max_cells
    h->passes = (bits + 7) / 8;
    const int64_t nn = std::max<int64_t>(n, 1);
    h->red_blocks = std::max(1, std::min(num_sms() * 4, (int)((nn + GRID_THREADS - 1) / GRID_THREADS)));
    bool ok = true;
    auto A = [&](void **p, size_t bytes) {
        if (ok && cudaMalloc(p, bytes) != cudaSuccess) ok = false;
    };
    A((void **)&h->keys[0], sizeof(uint32_t) * nn);
    A((void **)&h->keys[1], sizeof(uint32_t) * nn);
    A((void **)&h->vals[0], sizeof(uint32_t) * nn);
    A((void **)&h->vals[1], sizeof(uint32_t) * nn);
    A((void **)&h->sort_scratch, sizeof(uint32_t) * radix_scratch_size(nn));
    A((void **)&h->part, sizeof(GridPart) * h->red_blocks);
    A((void **)&h->ticket, sizeof(unsigned));
    A((void **)&h->geom, sizeof(GridBack));
    if (!ok) {
        gb_grid_destroy(h);
        return fail(GB_ENOMEM, "gb_grid_create: device allocation failed for n=%lld", (long long)n);
    }
    h->diag = (unsigned long long *)(h->geom + 1);
    GridBack g0 = {};
    g0.g.nx = g0.g.ny = g0.g.nz = 1;
    g0.g.cell = g0.g.inv_cell = 1.0;
    if (cudaMemset(h->ticket, 0, sizeof(unsigned)) != cudaSuccess ||
        cudaMemcpy(h->geom, &g0, sizeof(GridBack), cudaMemcpyHostToDevice) != cudaSuccess) {
        gb_grid_destroy(h);
        return fail(GB_ECUDA, "gb_grid_create: initialisation failed");
    }
    *out = h;
    return GB_OK;
}

extern "C" int64_t gb_grid_max_cells(gb_grid_t *h) { return h ? (int64_t)h->max_cells : -1; }

extern "C" int gb_grid_rebuild(gb_grid_t *h, const float *xm, const float *hsml, const int32_t *is_star,
                               int32_t *gsort, int32_t *cell_start, gb_grid_info_t *info, void *stream) {
    if (!h) return fail(GB_EINVAL, "handle is NULL");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t n = h->n;
    if (n > 0) {
        if (!xm || !aligned16(xm)) return fail(GB_EINVAL, "xm is NULL or not 16-byte aligned");
        if (!hsml) return fail(GB_EINVAL, "hsml is NULL");
        if (!gsort || !cell_start) return fail(GB_EINVAL, "gsort and cell_start must not be NULL");
        const int nblk = std::max(1, std::min(h->red_blocks, (int)((n + GRID_THREADS - 1) / GRID_THREADS)));
        const bool small = radix_small(n, h->passes);
        grid_reduce_kernel<<<nblk, GRID_THREADS, 0, s>>>((const float4 *)xm, hsml, is_star, n, h->min_radius,
                                                        h->max_cells, h->part, h->ticket, h->geom,
                                                        ZeroWords{{h->sort_scratch}, {small ? 0 : radix_zero_words(n)}});
        const unsigned g = (unsigned)((n + GRID_THREADS - 1) / GRID_THREADS);
        const CellKey key{(const float4 *)xm, is_star, h->geom};
        int cur = 0;
        if (small) {
            radix_sort_small<uint32_t>(key, h->keys, h->vals, n, s);
        } else {
            grid_key_kernel<<<nblk, GRID_THREADS, 0, s>>>(key, n, h->keys[0], h->sort_scratch, h->passes);
            cur = radix_sort_counted<uint32_t>(h->keys, h->vals, n, h->passes, h->sort_scratch, h->diag, s);
        }
        grid_gsort_kernel<<<g, GRID_THREADS, 0, s>>>(h->vals[cur], n, h->geom, gsort);
        const unsigned gc = (unsigned)((h->max_cells + START_CELLS) / START_CELLS);
        grid_start_kernel<<<gc, GRID_THREADS, 0, s>>>(h->keys[cur], h->geom, h->max_cells, cell_start);
        GB_CUDA_TRY(cudaGetLastError());
        h->launches += small ? 3 + radix_small_launches(n) : 4 + h->passes;
    }
    if (info) {
        GridBack back;
        GB_CUDA_TRY(cudaMemcpyAsync(&back, h->geom, sizeof(GridBack), cudaMemcpyDeviceToHost, s));
        GB_CUDA_TRY(cudaStreamSynchronize(s));
        GridGeom &g = back.g;
        if (n == 0) g.ngas = 0;
        info->ngas = g.ngas;
        info->n_cells = g.n_cells;
        info->nx = g.nx;
        info->ny = g.ny;
        info->nz = g.nz;
        info->status = g.status;
        for (int a = 0; a < 3; ++a) info->lo[a] = g.lo[a];
        info->cell = g.cell;
        info->inv_cell = g.inv_cell;
        if (g.status == 1) return fail(GB_EINVAL, "gb_grid_rebuild: non-finite gas position or smoothing length");
        if (g.status == 2) return fail(GB_EINVAL, "gb_grid_rebuild: cell growth did not converge");
        const unsigned long long to = back.diag[DIAG_WAIT_TIMEOUT];
        const unsigned long long inc = to - h->timeouts_seen;
        h->timeouts_seen = to;
        if (inc) return fail(GB_ETIMEOUT, "gb_grid_rebuild: %llu bounded device waits expired (radix sort)", inc);
    }
    return GB_OK;
}

extern "C" uint64_t gb_grid_launch_count(gb_grid_t *h) { return h ? h->launches : 0; }
