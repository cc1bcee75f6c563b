// slices.cu -- power iteration of one level on row slices.
//
// The recurrence, stopping rule and result are k_power_iter's (eigen.cu).
// The matrix is laid out once per level as units of 128-entry steps, each
// read by one warp with coalesced loads and no row search: a group of 32 rows
// is cut into 2^g units of 32 >> g rows, 2^g lanes a row, four consecutive
// entries a lane and step, the smallest g that leaves a lane at most `epl`
// entries; rows above 32 * epl entries are cut into units of that size.  Rows
// are summed by their lanes in entry order and combined by a butterfly.
//
// Four forms, chosen per level (slice_form; the direct ones take a second
// barrier where a row is far above a block's share, kLongRowGlobal):
//   direct, shared   the whole iterate in every block's shared memory
//                    (n <= kSlicePW), one grid barrier an iteration
//   panels           columns cut into panels of kSlicePW; a block loads the
//                    panels of its share of the units one after another,
//                    writes one sum per row and panel, and after a second
//                    barrier the rows add their panels
//   direct, global   iterate gathered from L2 (sparse levels wider than one
//                    panel), one grid barrier an iteration
//   direct, hub      the same in degree order, the leading kSlicePW entries (the
//                    most referenced) in shared memory (skewed levels)
// Destinations are 16 bits inside a panel, weights 8 / 16 / 32 / 64 bits, or
// none: a level whose total weight is at most 1.25 times its entries repeats
// them instead (first coarse levels of unweighted graphs: 1.09 at R-MAT 22).
//
// What bounds it: the cooperative kernel gathers the iterate through L1, about
// 1.2 gathers a clock and SM whatever the cache holds.  Shared memory serves a
// half warp's 64-bit gathers in one pass when its 16 banks differ: 6.4 passes
// a warp load with the entries in row order, 3.0 with the places chosen by
// bank (R-MAT 20's first coarse level, 30.6M entries).  An iteration of R-MAT
// 22's level 1 (117M entries) goes from 341 us to 116, of R-MAT 20's from 96
// to 37, of a weighted Chung-Lu level of 5.9M entries from 49 to 20, of a mesh
// level of 16,799 vertices from 11.1 to 5.9, of one of 190,000 from 26 to 10.5.
// What is left is the shared-memory passes (49 us of the 116) and the 2-byte
// matrix stream (47 us) overlapped with them, the rows' panel sums (15 us) and,
// below a million entries, the barrier and the trips to L2 behind it (about 4
// us an iteration).
//
// Sums are taken in an order fixed by the level and the grid (static unit
// ranges per warp), so results are reproducible run to run.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "common.cuh"
#include "internal.h"
#include "pi_common.cuh"

namespace sgpb {

constexpr uint32_t kSlicePW = 25600;        // iterate entries per panel (200 KB of shared memory)
// Shared memory serves a warp's 64-bit gathers 16 lanes at a time from 16
// banks of 8 bytes.  Entries are placed so that the lanes of a half warp read
// different banks where a row's destinations allow it (place below); the
// destination of an empty place is a zero behind the panel in that bank.
constexpr uint32_t kBanks = 16;
constexpr size_t kSliceSmem = (size_t)(kSlicePW + kBanks) * sizeof(double);
enum SliceForm { kFormShared = 0, kFormGlobal = 1, kFormPanels = 2, kFormHub = 3 };

// Threads of a block.  512 leave each 128 registers for the batches in flight:
// against 1024 threads the weighted Chung-Lu partition takes 70 instead of 78
// ms and R-MAT 16 22 instead of 25.  Panels without weights hold no weights in
// registers and gain from the warps instead (R-MAT 22's level 1 125 -> 122 us).
__host__ __device__ constexpr int slice_threads(int form, int wb) {
    return form == kFormPanels && wb == 0 ? 1024 : 512;
}
constexpr uint32_t kSliceItem = 2048;       // entries of a row that one warp lays out
constexpr uint32_t kSliceMaxPanels = 32;    // a lane holds a panel's bounds in the layout kernels
constexpr int kSumK = 3;                    // sum r, sum r^2, sum u r
constexpr uint32_t kSpinLimit = 1u << 23;   // polls of a grid barrier before giving up, about 6 s


struct SliceArgs {
    uint32_t n, n32, P;
    uint32_t nu;                  // units
    const uint4 *unit;            // x step offset, y first row, z steps | lanes log2 << 16, w slot of a chunk or ~0
    const uint32_t *cpre;         // [nu+1] prefix of the units' cost
    const uint32_t *pan_u;        // [P+1] first unit of each panel
    const void *col;              // uint16 (shared, panels) or uint32 (global)
    const void *w;
    const uint32_t *sptr;         // [n+1] chunk slots of each row
    uint32_t nslots;
    double *spart;                // sums of chunks
    uint32_t ncross;              // (direct) > 0: the chunks of a row are anywhere, its rows are added up ...
    const uint32_t *cross;        // ... behind a second barrier: the rows with chunks, ascending
    double *y;                    // [P][n32] row sums of the panels
    const double *deg;            // [n] weighted degrees
    const uint32_t *inv;          // new id -> level vertex id (null: identity)
    const double *x_in;
    const uint32_t *vcmap;
    double *va, *vb;              // n32 doubles each, zero behind n
    double *out;
    double *partials;             // [2][grid][4]
    uint32_t *bar;                // grid barrier counter and err, 0 at launch; 8-byte aligned
    uint32_t *err;                // set by a block that gave up waiting; the others leave at their next barrier
    uint32_t spin;                // polls of a grid barrier before giving up
    double tol;
    uint64_t iter_max;
    double *res;                  // [0] niter [1] dot [2] gb [3] lambda [4] capped [5] barrier gave up
                                  // [7] least distance of an iteration's change from tol, 0 if an iterate cancelled
    // continued run: iterations already done and the last dot product but one
    uint64_t iter0;
    double dot0;
};

// ------------------------------------------------------------- barrier --
// Grid barrier of a cooperative launch: arrivals are counted in one word that
// only grows, thread 0 polls it with a limit.  Returns false, and the kernel
// then returns, when the limit ran out here (err is set), or err was set before
// or while this block waited (err is the word behind the counter, one load).
struct GridBar {
    uint32_t *ctr;
    uint32_t target, limit;
    // by warp 0 alone, after a block barrier behind the other warps' stores
    __device__ __forceinline__ void arrive() {
        target += gridDim.x;
        __syncwarp();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
        }
    }
    // by every thread; target is warp 0's
    __device__ __forceinline__ bool wait(uint32_t *s_ok) {
        if (threadIdx.x == 0) {
            unsigned long long both;
            uint32_t k = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(both) : "l"(ctr) : "memory");
            } while ((int32_t)((uint32_t)both - target) < 0 && !(both >> 32) && ++k < limit);
            const bool ok = (int32_t)((uint32_t)both - target) >= 0 && !(both >> 32) && limit;
            if (!ok) atomicExch(ctr + 1, 1u);
            *s_ok = ok ? 1u : 0u;
        }
        __syncthreads();
        return *s_ok != 0;
    }
    __device__ __forceinline__ bool sync(uint32_t *s_ok) {
        __syncthreads();
        if (threadIdx.x < 32) arrive();
        return wait(s_ok);
    }
};

// The block's sums of p[3], written to dst[0..2] by warp 0 (sm: 3 x 32).
template <int WARPS>
__device__ __forceinline__ void block_sum3_to(const double (&p)[kSumK], double (*sm)[kSumK], double *dst) {
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double v = warp_sum3(p[0], p[1], p[2]);
    if (lane < kSumK) sm[wid][lane] = v;
    __syncthreads();
    if (wid == 0) {
        const bool in = lane < WARPS;
        const double t = warp_sum3(in ? sm[lane][0] : 0.0, in ? sm[lane][1] : 0.0, in ? sm[lane][2] : 0.0);
        if (lane < kSumK) dst[lane] = t;
    }
}

// The grid's sums from the blocks' partials, by one warp, left in s[0..2].
__device__ __forceinline__ void grid_sum3(const double *part, double *s) {
    const unsigned lane = threadIdx.x & 31;
    double a = 0, b = 0, c = 0;
    for (uint32_t k = lane; k < gridDim.x; k += 32) {
        const double2 ab = __ldcg(reinterpret_cast<const double2 *>(part + 4 * (size_t)k));
        a += ab.x;
        b += ab.y;
        c += __ldcg(part + 4 * (size_t)k + 2);
    }
    const double t = warp_sum3(a, b, c);
    if (lane < kSumK) s[lane] = t;
}

__device__ __forceinline__ uint32_t slice_lower_bound(const uint32_t *pre, uint32_t lo, uint32_t hi, uint64_t t) {
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if ((uint64_t)pre[mid] < t) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// ------------------------------------------------------------ row sums --
// four destinations of a lane's step (16 or 32 bits)
struct Col16 {
    uint2 v;
    __device__ __forceinline__ void load(const void *p, uint64_t i) {
        asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];"
                     : "=r"(v.x), "=r"(v.y)
                     : "l"((const uint2 *)p + i));
    }
    __device__ __forceinline__ uint32_t get(int k) const {
        const uint32_t x = k < 2 ? v.x : v.y;
        return (k & 1) ? x >> 16 : x & 0xFFFFu;
    }
};
struct Col32 {
    uint4 v;
    __device__ __forceinline__ void load(const void *p, uint64_t i) {
        asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "l"((const uint4 *)p + i));
    }
    __device__ __forceinline__ uint32_t get(int k) const { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
};
// four weights of WB bytes
template <int WB>
struct Wgt4 {
    uint32_t v[WB ? WB : 1];
    __device__ __forceinline__ void load(const void *p, uint64_t i) {
        const uint32_t *q = (const uint32_t *)p + i * (WB ? WB : 1);
        if constexpr (WB == 1) {
            asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v[0]) : "l"(q));
        } else if constexpr (WB == 2) {
            asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(q));
        } else if constexpr (WB >= 4) {
#pragma unroll
            for (int h = 0; h < WB / 4; h++)
                asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(v[4 * h]), "=r"(v[4 * h + 1]), "=r"(v[4 * h + 2]), "=r"(v[4 * h + 3])
                             : "l"(q + 4 * h));
        }
    }
    __device__ __forceinline__ double get(int k) const {
        if constexpr (WB == 0) return 1.0;
        else if constexpr (WB == 1) return (double)((v[0] >> (8 * k)) & 0xFFu);
        else if constexpr (WB == 2) return (double)((v[k >> 1] >> (16 * (k & 1))) & 0xFFFFu);
        else if constexpr (WB == 4) return (double)v[k];
        else return (double)(((unsigned long long)v[2 * k + 1] << 32) | v[2 * k]);
    }
};

// A warp's units [k0, k1) of one panel: their steps are consecutive, so the
// destinations and weights are one stream, loaded a batch of U steps ahead of
// its use across unit ends.  begin() loads the first batch (it depends on the
// layout alone, so a barrier can follow); run() consumes the stream and calls
// done(unit, next unit, whether there is one, sum) on every lane at each unit's end (the sum complete on all
// lanes of a row).
template <int FORM, int WB>
struct Stream {
    static constexpr bool GLOBAL = FORM == kFormGlobal || FORM == kFormHub, PANELS = FORM == kFormPanels;
    typedef typename std::conditional<GLOBAL, Col32, Col16>::type Col;
    static constexpr int U = (GLOBAL || WB >= 4) ? 2 : 4;
    uint32_t k, k1, pos, end;   // unit, last unit's end, stream position and end in steps
    uint4 d, dn, dm;            // records of this unit and of the next two
    Col c[U];
    Wgt4<WB> w[U];

    __device__ __forceinline__ void begin(const SliceArgs &a, uint32_t k0_, uint32_t k1_) {
        k = k0_;
        k1 = k1_;
        pos = end = 0;
        if (k >= k1) return;
        d = __ldg(a.unit + k);
        dn = __ldg(a.unit + (k + 1 < k1 ? k + 1 : k));
        dm = __ldg(a.unit + (k + 2 < k1 ? k + 2 : k));
        const uint4 dl = __ldg(a.unit + k1 - 1);
        pos = d.x;
        end = dl.x + (dl.z & 0xFFFFu);
        load(a, pos, c, w);
    }
    __device__ __forceinline__ void load(const SliceArgs &a, uint32_t p, Col (&cc)[U], Wgt4<WB> (&ww)[U]) const {
        const uint64_t i = (uint64_t)p * 32 + (threadIdx.x & 31);
#pragma unroll
        for (int q = 0; q < U; q++)
            if (p + q < end) {
                cc[q].load(a.col, i + 32 * q);
                if (WB) ww[q].load(a.w, i + 32 * q);
            }
    }
    template <typename Done>
    __device__ __forceinline__ void run(const SliceArgs &a, const double *x, const double *g, Done &&done) {
        if (k >= k1) return;
        uint32_t left = d.z & 0xFFFFu;
        double s0 = 0, s1 = 0;
        // ends the unit (and units without steps behind it)
        auto flush = [&]() {
            do {
                const uint32_t lg = d.z >> 16;
                double s = s0 + s1;
                for (uint32_t o = 1; o < (1u << lg); o <<= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
                done(d, dn, k + 1 < k1, s);
                s0 = s1 = 0;
                d = dn;
                k++;
                dn = dm;
                if (k + 2 < k1) dm = __ldg(a.unit + k + 2);
                left = d.z & 0xFFFFu;
            } while (left == 0 && k < k1);
        };
        if (left == 0) flush();
        auto gather = [&](int q, double (&v)[4]) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint32_t j = c[q].get(e);
                // x: shared memory; g: the whole iterate
                if (FORM == kFormHub) v[e] = j < kSlicePW ? x[j] : j != 0xFFFFFFFFu ? g[j] : 0.0;
                else if (GLOBAL) v[e] = j != 0xFFFFFFFFu ? g[j] : 0.0;
                else v[e] = x[j];
            }
        };
        auto add = [&](int q, const double (&v)[4]) {
            if (WB == 0) {
                s0 += v[0] + v[1];
                s1 += v[2] + v[3];
            } else {
                s0 = fma(w[q].get(0), v[0], s0);
                s1 = fma(w[q].get(1), v[1], s1);
                s0 = fma(w[q].get(2), v[2], s0);
                s1 = fma(w[q].get(3), v[3], s1);
            }
        };
        while (pos < end) {
            Col cn[U];
            Wgt4<WB> wn[U];
            load(a, pos + U, cn, wn);
            if (left > U) {
                // the batch is inside the unit: every gather in flight at once
                double v[U][4];
#pragma unroll
                for (int q = 0; q < U; q++) gather(q, v[q]);
#pragma unroll
                for (int q = 0; q < U; q++) add(q, v[q]);
                left -= U;
            } else {
#pragma unroll
                for (int q = 0; q < U; q++) {
                    if (pos + q < end) {
                        double v[4];
                        gather(q, v);
                        add(q, v);
                        if (--left == 0) flush();
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < U; q++) {
                c[q] = cn[q];
                if (WB) w[q] = wn[q];
            }
            pos += U;
        }
    }
};

// Panel copies: one bulk copy of the panel into shared memory, completion
// counted on an mbarrier.  The iterate was written by generic stores of other
// blocks before the last grid barrier, and the shared memory read by this
// block's loads before its own: both sides of the copy are fenced.
struct PanelCopy {
    uint64_t *bar;
    uint32_t phase;
    __device__ __forceinline__ void init() {
        if (threadIdx.x == 0) {
            mbar_init(bar);
            mbar_fence_init();
        }
    }
    // by warp 0, all threads past a block barrier behind the panel's last use
    __device__ __forceinline__ void issue(const double *src, uint32_t len, double *xs) {
        if (threadIdx.x >= 32) return;
        const uint32_t bytes = ((len + 1) & ~1u) * (uint32_t)sizeof(double);
        if (threadIdx.x == 0) mbar_expect_tx(bar, bytes);
        __syncwarp();
        // a slice for each of eight lanes, multiples of 16 bytes
        const uint32_t per = ((bytes / 8) + 127) & ~127u;
        const uint32_t b = threadIdx.x * per;
        if (threadIdx.x < 8 && b < bytes) {
            asm volatile("fence.proxy.async;" ::: "memory");
            bulk_load((char *)xs + b, (const char *)src + b, bytes - b < per ? bytes - b : per, bar);
        }
    }
    // by every thread; false when the wait limit ran out (the copy is waited
    // for once more, so that the block does not leave under it)
    __device__ __forceinline__ bool wait() {
        const bool ok = mbar_wait(bar, phase);
        if (!ok) mbar_wait(bar, phase);
        phase ^= 1;
        return ok;
    }
};

// the calling warp's share of the units [u, ue): equal cost
template <int kSliceWarps>
__device__ __forceinline__ void warp_units(const SliceArgs &a, uint32_t u, uint32_t ue, unsigned wid, uint32_t &k0,
                                           uint32_t &k1) {
    const uint64_t c0 = a.cpre[u], c1 = a.cpre[ue];
    k0 = wid == 0 ? u : slice_lower_bound(a.cpre, u, ue, c0 + (c1 - c0) * wid / kSliceWarps);
    k1 = wid + 1 == kSliceWarps ? ue : slice_lower_bound(a.cpre, u, ue, c0 + (c1 - c0) * (wid + 1) / kSliceWarps);
}

// FORM: the level's form; WB: bytes per weight (0: none); CROSS: a row's chunks
// are anywhere (ncross; as a branch it cost every other level 0.25 us an iteration).
template <int FORM, int WB, bool CROSS>
__global__ void __launch_bounds__(slice_threads(FORM, WB), 1) k_pi_slices(SliceArgs a) {
    constexpr int kSliceThreads = slice_threads(FORM, WB), kSliceWarps = kSliceThreads / 32;
    constexpr bool PANELS = FORM == kFormPanels, GLOBAL = FORM == kFormGlobal || FORM == kFormHub;
    constexpr bool COPY = FORM != kFormGlobal;   // the iterate or a part of it in shared memory
    extern __shared__ __align__(16) double xs[];
    __shared__ double sm[kSliceWarps][kSumK];
    __shared__ double s_sum[4];
    __shared__ double s_it[3];   // mean, 1 / norm and dot product of the last iteration
    __shared__ double s_margin;  // res[7]
    __shared__ uint32_t s_ok;
    const uint32_t n = a.n;
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t gtid = blockIdx.x * kSliceThreads + threadIdx.x, gthr = gridDim.x * kSliceThreads;
    __shared__ __align__(8) uint64_t s_mbar;
    GridBar bar{a.bar, 0, a.spin};
    PanelCopy panel{&s_mbar, 0};
    if (threadIdx.x == 0) s_margin = 1e300;
    if (COPY) panel.init();   // seen by the block behind the start vector's barriers
    double *part0 = a.partials, *part1 = a.partials + 4 * (size_t)gridDim.x;
    if (COPY && threadIdx.x < kBanks) xs[kSlicePW + threadIdx.x] = 0.0;
    // units of this block: an equal share of the cost; the direct forms keep
    // the units of a row (its chunks) in one block, unless a row is much longer
    // than a block's share (ncross)
    const uint64_t call = a.cpre[a.nu];
    auto block_unit = [&](uint32_t b) -> uint32_t {
        if (b == 0) return 0u;
        if (b >= gridDim.x) return a.nu;
        uint32_t u = slice_lower_bound(a.cpre, 0, a.nu, call * b / gridDim.x);
        if (!PANELS && !CROSS)
            while (u < a.nu && u > 0 && a.unit[u].y == a.unit[u - 1].y) u++;
        return u;
    };
    const uint32_t U0 = block_unit(blockIdx.x), U1 = block_unit(blockIdx.x + 1);
    uint32_t wu0 = 0, wu1 = 0, R0 = 0, R1 = 0;
    if (!PANELS) {
        warp_units<kSliceWarps>(a, U0, U1, wid, wu0, wu1);
        if (U0 < U1) {
            R0 = a.unit[U0].y;
            R1 = U1 < a.nu ? a.unit[U1].y : n;
        }
    }
    // ---- start vector, largest degree, mean, norm
    double mu, gb, inv_nu;
    {
        double s = 0, mx = 0;
        for (uint32_t i = gtid; i < n; i += gthr) {
            const uint32_t o = a.inv ? a.inv[i] : i;
            const double x = a.vcmap ? a.x_in[a.vcmap[o]] : a.x_in[o];
            const double d = a.deg[i];
            a.va[i] = x;
            s += x;
            mx = d > mx ? d : mx;
        }
        mx = warp_max(mx);
        if (lane == 0) sm[wid][0] = mx;
        __syncthreads();
        if (wid == 0) {
            const double t = warp_max(lane < kSliceWarps ? sm[lane][0] : 0.0);
            if (lane == 0) part0[4 * (size_t)blockIdx.x + 3] = t;
        }
        __syncthreads();
        double p[kSumK] = {s, 0, 0};
        block_sum3_to<kSliceWarps>(p, sm, part0 + 4 * (size_t)blockIdx.x);
        if (!bar.sync(&s_ok)) return;
        if (wid == 0) {
            grid_sum3(part0, s_sum);
            double t = 0;
            for (uint32_t k = lane; k < gridDim.x; k += 32) {
                const double v = __ldcg(part0 + 4 * (size_t)k + 3);
                t = v > t ? v : t;
            }
            t = warp_max(t);
            if (lane == 0) s_sum[3] = t;
        }
        __syncthreads();
        gb = 2.0 * s_sum[3];
        if (gb < 2.0) gb = 2.0;
        mu = s_sum[0] / (double)n;
        double q = 0;
        for (uint32_t i = gtid; i < n; i += gthr) {
            const double x = a.va[i] - mu;
            q += x * x;
        }
        double p2[kSumK] = {q, 0, 0};
        if (COPY) asm volatile("fence.proxy.async;" ::: "memory");
        block_sum3_to<kSliceWarps>(p2, sm, part1 + 4 * (size_t)blockIdx.x);
        if (!bar.sync(&s_ok)) return;
        if (wid == 0) grid_sum3(part1, s_sum);
        __syncthreads();
        inv_nu = 1.0 / sqrt(s_sum[0]);
        if (threadIdx.x == 0 && !(s_sum[0] > kCancel * (double)n * mu * mu)) s_margin = 0;
        __syncthreads();
    }
    // ---- iterations
    double dot = a.dot0;
    uint64_t niter = a.iter0;
    double *part = part0, *part_n = part1;   // partials of the running iteration, of the last
    double *src = a.va, *dst = a.vb;
    bool first = true;
    // this warp's first units: their stream starts before each barrier
    Stream<FORM, WB> st;
    uint32_t p0 = 0, ue0 = 0;
    if (PANELS) {
        while (U0 < U1 && a.pan_u[p0 + 1] <= U0) p0++;
        ue0 = U0 < U1 && a.pan_u[p0 + 1] < U1 ? a.pan_u[p0 + 1] : U1;
        warp_units<kSliceWarps>(a, U0, ue0, wid, wu0, wu1);
    }
    st.begin(a, wu0, wu1);
    // (direct) the first unit's row of this lane
    uint32_t ri0 = 0;
    bool row0 = false;
    double di0 = 0;
    if (!PANELS && wu0 < wu1) {
        const uint32_t lg = st.d.z >> 16;
        ri0 = st.d.y + (lane >> lg);
        row0 = st.d.w == 0xFFFFFFFFu && (lane & ((1u << lg) - 1u)) == 0 && ri0 < n;
        if (row0) di0 = a.deg[ri0];
    }
    while (true) {
        // the iterate (its first panel); beside it one warp takes the last
        // iteration's sums
        if (COPY && !PANELS) panel.issue(src, n < kSlicePW ? n : kSlicePW, xs);
        if (PANELS && U0 < U1)
            panel.issue(src + p0 * kSlicePW, n - p0 * kSlicePW < kSlicePW ? n - p0 * kSlicePW : kSlicePW, xs);
        if (!first && wid == kSliceWarps - 1) {
            grid_sum3(part_n, s_sum);
            __syncwarp();
            if (lane == 0) {
                const double m = s_sum[0] / (double)n;
                const double nsq = s_sum[1] - m * s_sum[0];
                const double inv = 1.0 / sqrt(nsq);
                s_it[0] = m;
                s_it[1] = inv;
                s_it[2] = s_sum[2] * inv;
                s_margin = nsq > kCancel * gb * gb ? fmin(s_margin, fabs(fabs(s_it[2] - dot) - a.tol)) : 0.0;
            }
        }
        if (COPY && (!PANELS || U0 < U1))
            if (!panel.wait() && lane == 0) atomicExch(a.err, 1u);
        __syncthreads();
        if (!first) {
            const double last = dot;
            dot = s_it[2];
            niter++;
            const double delta = fabs(dot - last);
            if (!(delta > a.tol && niter < a.iter_max)) {
                // the reference returns u of the last iteration, whose raw
                // values are still in the buffer the next one would overwrite
                const double s_ur = s_sum[2];
                double uu = 0;
                for (uint32_t i = gtid; i < n; i += gthr) {
                    const double u = (__ldcg(dst + i) - mu) * inv_nu;
                    a.out[a.inv ? a.inv[i] : i] = u;
                    uu += u * u;
                }
                double p[kSumK] = {uu, 0, 0};
                __syncthreads();
                block_sum3_to<kSliceWarps>(p, sm, part + 4 * (size_t)blockIdx.x);
                if (wid == 0) bar.arrive();
                if (!bar.wait(&s_ok)) return;
                if (blockIdx.x == 0 && wid == 0) {
                    grid_sum3(part, s_sum);
                    __syncwarp();
                    if (lane == 0) {
                        const double S5 = s_sum[0];
                        a.res[0] = (double)niter;
                        a.res[1] = dot;
                        a.res[2] = gb;
                        a.res[3] = (gb * S5 - s_ur) / S5;
                        a.res[4] = niter >= a.iter_max ? 1.0 : 0.0;
                        a.res[5] = 0.0;
                        a.res[7] = s_margin;
                    }
                }
                return;
            }
            mu = s_it[0];
            inv_nu = s_it[1];
        }
        first = false;
        double P[kSumK] = {0, 0, 0};
        // row i from its sum, its raw value and its degree
        auto fin = [&](uint32_t i, double acc, double xi, double d) {
            const double ui = (xi - mu) * inv_nu;
            const double r = next_value<false>(0, gb, mu, inv_nu, ui, acc, d);
            dst[i] = r;
            P[0] += r;
            P[1] += r * r;
            P[2] += ui * r;
        };
        if (PANELS) {
            uint32_t p = p0, ue = ue0;
            while (true) {
                double *y = a.y + (size_t)p * a.n32;
                st.run(a, xs, src, [&](const uint4 &d, const uint4 &, bool, double s) {
                    const uint32_t lg = d.z >> 16;
                    if (d.w != 0xFFFFFFFFu) {
                        if (lane == 0) a.spart[d.w] = s;
                    } else if ((lane & ((1u << lg) - 1u)) == 0) {
                        y[d.y + (lane >> lg)] = s;   // y has n32 entries a panel
                    }
                });
                if (ue >= U1) break;
                // the block's units of the next panel
                const uint32_t u = ue;
                while (a.pan_u[p + 1] <= u) p++;
                ue = a.pan_u[p + 1] < U1 ? a.pan_u[p + 1] : U1;
                uint32_t k0, k1;
                warp_units<kSliceWarps>(a, u, ue, wid, k0, k1);
                st.begin(a, k0, k1);
                __syncthreads();   // every warp is done with the previous panel
                panel.issue(src + p * kSlicePW, n - p * kSlicePW < kSlicePW ? n - p * kSlicePW : kSlicePW, xs);
                if (!panel.wait() && lane == 0) atomicExch(a.err, 1u);
            }
            if (!bar.sync(&s_ok)) return;
            // the rows: their panels in order, then their chunks
            for (uint32_t i = gtid; i < n; i += gthr) {
                const double xi = __ldcg(src + i), di = a.deg[i];
                const uint32_t b = a.nslots ? a.sptr[i] : 0u, e = a.nslots ? a.sptr[i + 1] : 0u;
                double acc = 0;
#pragma unroll 4
                for (uint32_t q = 0; q < a.P; q++) acc += __ldcg(a.y + (size_t)q * a.n32 + i);
#pragma unroll 4
                for (uint32_t q = b; q < e; q++) acc += __ldcg(a.spart + q);
                fin(i, acc, xi, di);
            }
        } else {
            auto own = [&](uint32_t i) -> double {
                return FORM == kFormShared || (FORM == kFormHub && i < kSlicePW) ? xs[i] : src[i];
            };
            // a row's own value and degree load one unit ahead of its sum
            uint32_t ri = 0;
            bool row = false;
            double di = 0, xi = 0;
            auto fetch = [&](const uint4 &d) {
                const uint32_t lg = d.z >> 16;
                ri = d.y + (lane >> lg);
                row = d.w == 0xFFFFFFFFu && (lane & ((1u << lg) - 1u)) == 0 && ri < n;
                if (row) {
                    di = __ldg(a.deg + ri);
                    xi = own(ri);
                }
            };
            if (wu0 < wu1) {
                ri = ri0;
                row = row0;
                di = di0;
                if (row) xi = own(ri);
            }
            st.run(a, xs, src, [&](const uint4 &d, const uint4 &dn, bool more, double s) {
                if (row) fin(ri, s, xi, di);
                else if (d.w != 0xFFFFFFFFu && lane == 0) a.spart[d.w] = s;
                if (more) fetch(dn);
            });
            if (CROSS) {
                if (!bar.sync(&s_ok)) return;
                for (uint32_t q = blockIdx.x * kSliceWarps + wid; q < a.ncross; q += gridDim.x * kSliceWarps) {
                    const uint32_t i = a.cross[q];
                    double acc = 0;
                    for (uint32_t k = a.sptr[i] + lane; k < a.sptr[i + 1]; k += 32) acc += __ldcg(a.spart + k);
                    acc = warp_sum(acc);
                    if (lane == 0) fin(i, acc, own(i), a.deg[i]);
                }
            } else if (a.nslots) {
                __syncthreads();   // the chunks of the block's rows are summed
                for (uint32_t i = R0 + threadIdx.x; i < R1; i += kSliceThreads) {
                    const uint32_t b = a.sptr[i], e = a.sptr[i + 1];
                    if (b == e) continue;
                    double acc = 0;
                    for (uint32_t q = b; q < e; q++) acc += a.spart[q];
                    fin(i, acc, own(i), a.deg[i]);
                }
            }
        }
        // the iterate's next readers copy it through the async proxy
        if (COPY) asm volatile("fence.proxy.async;" ::: "memory");
        block_sum3_to<kSliceWarps>(P, sm, part + 4 * (size_t)blockIdx.x);
        if (wid == 0) bar.arrive();
        st.begin(a, wu0, wu1);
        if (!bar.wait(&s_ok)) return;
        double *t = src; src = dst; dst = t;
        t = part; part = part_n; part_n = t;
    }
}

// --------------------------------------------------------------- layout --
// longest row and the number of kSliceItem-entry items of each row
__global__ void k_sl_rows(uint32_t n, const uint32_t *rp, uint32_t *items, uint32_t *maxlen) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t len = 0;
    if (i < n) {
        len = rp[i + 1] - rp[i];
        items[i] = len ? (len + kSliceItem - 1) / kSliceItem : 0u;
    }
    const uint32_t mx = __reduce_max_sync(0xFFFFFFFFu, len);
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(maxlen, mx);
}

__global__ void k_sl_item_rows(uint32_t n, const uint32_t *iptr, uint32_t *irow) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (uint32_t s = iptr[i]; s < iptr[i + 1]; s++) irow[s] = i;
}

// weighted degrees (one warp per item), their total and the largest weight
template <typename W>
__global__ void __launch_bounds__(256) k_sl_weights(uint32_t nitems, const uint32_t *iptr, const uint32_t *irow,
                                                   const uint32_t *rp, const W *__restrict__ w,
                                                   unsigned long long *dsum, unsigned long long *stat) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t nw = gridDim.x * blockDim.x / 32;
    unsigned long long tot = 0, mx = 0;
    for (uint32_t it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < nitems; it += nw) {
        const uint32_t i = irow[it];
        const uint32_t b = rp[i] + (it - iptr[i]) * kSliceItem;
        const uint32_t e = rp[i + 1] - b < kSliceItem ? rp[i + 1] : b + kSliceItem;
        unsigned long long s = 0;
#pragma unroll 4
        for (uint32_t j = b + lane; j < e; j += 32) {
            const unsigned long long x = (unsigned long long)__ldg(w + j);
            s += x;
            mx = x > mx ? x : mx;
        }
        s = warp_sum(s);
        if (lane == 0) {
            if (iptr[i + 1] - iptr[i] == 1) dsum[i] = s;
            else atomicAdd(dsum + i, s);
        }
        tot += s;
    }
    mx = warp_max(mx);
    if (lane == 0) {
        atomicAdd(stat, tot);
        atomicMax(stat + 1, mx);
    }
}

// entries of the leading kSlicePW rows in degree order
__global__ void k_sl_lead(const uint32_t *rp, const uint32_t *inv, unsigned long long *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long s = 0;
    if (i < kSlicePW) s = rp[inv[i] + 1] - rp[inv[i]];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, s);
}

struct SliceBuild {
    uint32_t n, n32, ng, P, epl, nitems;
    int direct, expand, l2;
    const uint32_t *rp, *col;
    const void *w;
    const uint32_t *perm, *inv;          // null: identity
    const uint32_t *iptr, *irow;         // items of each row, row of each item
    const uint32_t *mptr;                // [n+1] items before row i's of rows of several items
    uint32_t *tcol;                      // permuted destinations (panels)
    uint32_t *icnt;                      // items of rows of several: [item][P*16] base ranks
    uint32_t *mtot;                      // rows of several items, at their first item: [P*16] entries
    uint32_t *cnt;                       // [P][n32] entries (copies) of a row in a panel
    uint32_t *nun, *nst;                 // [P*ng] units and steps of a group
    const uint32_t *unb, *stb;           // their scans
    uint32_t *slotc;                     // [n] chunk slots of a row
    const uint32_t *sptr;
    uint32_t *roff;                      // [P][n32] step offset of a row's first unit
    uint32_t *rst;                       // [P][n32] steps of a row | log2 of its lanes << 24
    uint4 *unit;
    uint32_t *ucost;
    uint32_t *pan_u;
    void *ocol, *ow;
    double *deg;
    const unsigned long long *dsum;
};
constexpr int kLayWarps = 4;             // warps per block of the layout kernels
constexpr uint32_t kMaxKeys = kSliceMaxPanels * kBanks;

// items of the rows of more than one
__global__ void k_sl_multi(uint32_t n, const uint32_t *iptr, uint32_t *items) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = iptr[i + 1] - iptr[i];
    items[i] = c > 1 ? c : 0u;
}

// Entries of an item by panel and bank.  An item that is its whole row leaves
// its panel counts in cnt; an item of a longer row its (panel, bank) counts in
// icnt.  The permuted destinations are kept for the fill.  only_multi: whole
// rows are skipped (one panel: their count is the row length).
template <typename W>
__global__ void __launch_bounds__(32 * kLayWarps) k_sl_count(SliceBuild b, int only_multi) {
    __shared__ uint32_t s_hist[kLayWarps][kMaxKeys];
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t nw = gridDim.x * kLayWarps, keys = b.P * kBanks;
    const W *w = (const W *)b.w;
    uint32_t *hist = s_hist[wid];
    for (uint32_t it = blockIdx.x * kLayWarps + wid; it < b.nitems; it += nw) {
        const uint32_t i = b.irow[it];
        const bool multi = b.iptr[i + 1] - b.iptr[i] > 1;
        if (only_multi && !multi) continue;
        const uint32_t s = b.rp[i] + (it - b.iptr[i]) * kSliceItem;
        const uint32_t e = b.rp[i + 1] - s < kSliceItem ? b.rp[i + 1] : s + kSliceItem;
        for (uint32_t k = lane; k < keys; k += 32) hist[k] = 0;
        __syncwarp();
        for (uint32_t j0 = s; j0 < e; j0 += 128) {
            uint32_t c[4], m[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t j = j0 + 32 * k + lane;
                c[k] = j < e ? __ldg(b.col + j) : 0u;
                m[k] = b.expand && j < e ? (uint32_t)__ldg(w + j) : 1u;
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (b.perm && j0 + 32 * k + lane < e) c[k] = __ldg(b.perm + c[k]);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t j = j0 + 32 * k + lane;
                if (j < e) {
                    if (b.tcol) b.tcol[j] = c[k];
                    const uint32_t p = b.P > 1 ? c[k] / kSlicePW : 0u;
                    atomicAdd(&hist[p * kBanks + (c[k] & (kBanks - 1))], m[k]);   // kSlicePW is a multiple of 16
                }
            }
        }
        __syncwarp();
        if (multi) {
            uint32_t *o = b.icnt + (size_t)(b.mptr[i] + it - b.iptr[i]) * keys;
            for (uint32_t k = lane; k < keys; k += 32) o[k] = hist[k];
        } else if (lane < b.P) {
            uint32_t t = 0;
            for (uint32_t k = 0; k < kBanks; k++) t += hist[lane * kBanks + k];
            b.cnt[(size_t)lane * b.n32 + (b.perm ? b.perm[i] : i)] = t;
        }
        __syncwarp();
    }
}

// Rows of several items (a warp each, found by their first item): the base
// ranks of every item by panel and bank, the row's totals, its panel counts.
__global__ void __launch_bounds__(32 * kLayWarps) k_sl_row_counts(SliceBuild b) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t nw = gridDim.x * kLayWarps, keys = b.P * kBanks;
    for (uint32_t i = blockIdx.x * kLayWarps + (threadIdx.x >> 5); i < b.n; i += nw) {
        const uint32_t i0 = b.mptr[i], i1 = b.mptr[i + 1];
        if (i0 == i1) continue;
        for (uint32_t k0 = 0; k0 < keys; k0 += 32) {   // keys is a multiple of 16
            const uint32_t k = k0 + lane;
            uint32_t run = 0;
            if (k < keys) {
                for (uint32_t it = i0; it < i1; it++) {
                    const uint32_t c = b.icnt[(size_t)it * keys + k];
                    b.icnt[(size_t)it * keys + k] = run;
                    run += c;
                }
                b.mtot[(size_t)i0 * keys + k] = run;
            }
            uint32_t t = run;
            for (int o = 1; o < (int)kBanks; o <<= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
            if (k < keys && (lane & (kBanks - 1)) == 0)
                b.cnt[(size_t)(k / kBanks) * b.n32 + (b.perm ? b.perm[i] : i)] = t;
        }
    }
}

__global__ void k_sl_chunked(uint32_t n, const uint32_t *sptr, uint8_t *flags) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flags[i] = sptr[i + 1] > sptr[i];
}

// row lengths in the layout's numbering (one panel) and weighted degrees
__global__ void k_sl_degrees(SliceBuild b) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.n32) return;
    uint32_t len = 0;
    if (i < b.n) {
        const uint32_t o = b.inv ? b.inv[i] : i;
        len = b.rp[o + 1] - b.rp[o];
        b.deg[i] = b.w ? (len ? (double)b.dsum[o] : 0.0) : (double)len;
    }
    if (b.P == 1) b.cnt[i] = len;
}

// The units of group g in panel p for the lane's row: lanes per row (log2),
// the row's unit inside the group, that unit's steps, and for a chunked row
// its chunks.
struct GroupPlan {
    uint32_t len, lg, steps, chunks;
};
__device__ __forceinline__ GroupPlan group_plan(const SliceBuild &b, uint32_t p, uint32_t g) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t i = g * 32 + lane;
    GroupPlan r;
    r.len = b.cnt[(size_t)p * b.n32 + i];
    const uint32_t mx = __reduce_max_sync(0xFFFFFFFFu, r.len);
    r.lg = 0;
    while (r.lg < 5 && mx > (b.epl << r.lg)) r.lg++;
    uint32_t um = r.len;   // longest row of the unit: 32 >> lg lanes
    for (uint32_t o = 1; o < (32u >> r.lg); o <<= 1) {
        const uint32_t t = __shfl_xor_sync(0xFFFFFFFFu, um, o);
        um = t > um ? t : um;
    }
    r.steps = (um + (4u << r.lg) - 1) / (4u << r.lg);
    r.chunks = r.lg == 5 ? (r.len + 32 * b.epl - 1) / (32 * b.epl) : 1u;
    return r;
}

__global__ void __launch_bounds__(256) k_sl_groups(SliceBuild b) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= (uint64_t)b.P * b.ng) return;
    const uint32_t p = (uint32_t)(t / b.ng), g = (uint32_t)(t % b.ng);
    const GroupPlan r = group_plan(b, p, g);
    const bool head = (lane & ((32u >> r.lg) - 1u)) == 0;   // first row of its unit
    uint32_t nu = 0, ns = 0;
    if (head) {
        ns = r.steps;
        nu = r.chunks > 1 ? r.chunks : ((b.direct ? g * 32 + lane < b.n : r.steps > 0) ? 1u : 0u);
    }
    if (r.chunks > 1) atomicAdd(b.slotc + g * 32 + lane, r.chunks);
    nu = __reduce_add_sync(0xFFFFFFFFu, nu);
    ns = __reduce_add_sync(0xFFFFFFFFu, ns);
    if (lane == 0) {
        b.nun[t] = nu;
        b.nst[t] = ns;
    }
}

// cost of a unit in the split over blocks and warps, in half steps: its steps,
// a quarter more where every lane has a row of its own (short rows share banks
// more often: R-MAT 22's level 1 122 -> 118 us), plus the price of two steps for
// the record, the butterfly and the row's value.  Gathers from L2 (l2) cost by
// their number too, and a unit the price of four steps: rows of a few entries
// leave most places of a step empty, and 512 rows of 2,000 entries among a million
// of six had 7 blocks to themselves (79 -> 51 us; with a unit at two steps 36, but
// the weighted Chung-Lu input of 262,147 vertices 47 in place of 39.5 -> 38.4)
__global__ void __launch_bounds__(256) k_sl_units(SliceBuild b) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= (uint64_t)b.P * b.ng) return;
    const uint32_t p = (uint32_t)(t / b.ng), g = (uint32_t)(t % b.ng);
    const GroupPlan r = group_plan(b, p, g);
    const uint32_t i = g * 32 + lane;
    const bool head = (lane & ((32u >> r.lg) - 1u)) == 0;
    uint32_t nu = 0, ns = 0;
    if (head) {
        ns = r.steps;
        nu = r.chunks > 1 ? r.chunks : ((b.direct ? i < b.n : r.steps > 0) ? 1u : 0u);
    }
    uint32_t us = nu, ss = ns;   // inclusive scans over the lanes
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, us, o), y = __shfl_up_sync(0xFFFFFFFFu, ss, o);
        if ((int)lane >= o) { us += x; ss += y; }
    }
    const uint32_t u0 = b.unb[t] + us - nu;
    const uint32_t off = b.stb[t] + ss - ns;
    if (g == 0 && lane == 0) b.pan_u[p] = b.unb[t];
    if (t == (uint64_t)b.P * b.ng - 1 && lane == 31) b.pan_u[b.P] = b.unb[t] + us;
    b.roff[(size_t)p * b.n32 + i] = __shfl_sync(0xFFFFFFFFu, off, lane & ~((32u >> r.lg) - 1u));
    b.rst[(size_t)p * b.n32 + i] = r.steps | (r.lg << 24);
    uint32_t entries = r.len;   // of the unit
    for (uint32_t o = 1; o < (32u >> r.lg); o <<= 1) entries += __shfl_xor_sync(0xFFFFFFFFu, entries, o);
    if (!nu) return;
    if (r.chunks <= 1) {
        b.unit[u0] = make_uint4(off, i, r.steps | (r.lg << 16), 0xFFFFFFFFu);
        b.ucost[u0] = b.l2 ? 4 * r.steps + entries / 16 + 16 : 2 * r.steps + (r.lg == 0 ? r.steps / 2 : 0) + 4;
        return;
    }
    uint32_t slot = b.sptr[i];
    for (uint32_t q = 0; q < p; q++) {
        const uint32_t c = b.cnt[(size_t)q * b.n32 + i];
        if (c > 32 * b.epl) slot += (c + 32 * b.epl - 1) / (32 * b.epl);
    }
    const uint32_t full = b.epl / 4;   // steps of a whole chunk
    for (uint32_t k = 0; k < r.chunks; k++) {
        const uint32_t st = k + 1 < r.chunks ? full : r.steps - k * full;
        b.unit[u0 + k] = make_uint4(off + k * full, i, st | (5u << 16), slot + k);
        const uint32_t left = r.len - k * 32 * b.epl;
        b.ucost[u0 + k] = b.l2 ? 4 * st + (left < 32 * b.epl ? left : 32 * b.epl) / 16 + 16 : 2 * st + 4;
    }
}

// The places of a row's entries with bank b when the row has 2^lg lanes, is
// the sub-th row of its unit and has S slots a lane.  In every slot the half
// warp's lanes get different banks: with G <= 16 lanes a row and R = 16 / G
// rows a half warp, lane j reads bank j R + (t + sub) mod R in slot t; with 32
// lanes, lanes j and j + 16 read bank j.
struct BankPlaces {
    uint32_t cap, t0, step, lane;
    __device__ __forceinline__ BankPlaces(uint32_t bk, uint32_t lg, uint32_t sub, uint32_t S) {
        if (lg == 5) {
            cap = 2 * S;
            t0 = 0;
            step = 0;
            lane = bk;
            return;
        }
        const uint32_t lr = 4 - lg, R = 1u << lr;
        t0 = (bk - sub) & (R - 1);
        step = R;
        cap = S > t0 ? (S - t0 + R - 1) >> lr : 0u;
        lane = (sub << lg) + (bk >> lr);
    }
    // slot and lane of the bank's k-th place
    __device__ __forceinline__ uint32_t slot(uint32_t k) const { return step ? t0 + k * step : k >> 1; }
    __device__ __forceinline__ uint32_t lane_of(uint32_t k) const { return step ? lane : lane + 16 * (k & 1); }
};

// every place of every unit: the zero of its bank
__global__ void __launch_bounds__(256) k_sl_preset(SliceBuild b, uint32_t nu) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t nw = gridDim.x * blockDim.x / 32;
    for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < nu; u += nw) {
        const uint4 d = b.unit[u];
        const uint32_t lg = d.z >> 16, steps = d.z & 0xFFFFu;
        const uint32_t sub = lg == 5 ? 0u : lane >> lg, j = lg == 5 ? lane & 15u : lane & ((1u << lg) - 1u);
        const uint32_t lr = lg == 5 ? 0u : 4 - lg, R = 1u << lr;
        uint2 *o = (uint2 *)b.ocol + (size_t)d.x * 32 + lane;
        for (uint32_t s = 0; s < steps; s++, o += 32) {
            uint32_t c[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) c[k] = kSlicePW + (j << lr) + ((4 * s + k + sub) & (R - 1));
            *o = make_uint2(c[0] | (c[1] << 16), c[2] | (c[3] << 16));
        }
    }
}

// One warp per item: every entry to a place of its bank, by its rank among the
// row's entries of that panel and bank; entries beyond the bank's places take
// the places other banks leave free, in order.  WI: the level's weights, WO:
// the layout's (char: none).  CO uint32_t: the global form, places by rank
// alone.
template <typename WI, typename WO, typename CO>
__global__ void __launch_bounds__(32 * kLayWarps) k_sl_fill(SliceBuild b) {
    constexpr bool BANKED = sizeof(CO) == 2;
    __shared__ uint32_t s_cur[kLayWarps][BANKED ? kMaxKeys : 1];    // next rank of a key
    __shared__ uint32_t s_tot[kLayWarps][BANKED ? kMaxKeys : 1];    // entries of a key
    __shared__ uint32_t s_ovb[kLayWarps][BANKED ? kMaxKeys : 1];    // overflow of the panel's banks before
    __shared__ uint32_t s_hob[kLayWarps][BANKED ? kMaxKeys : 1];    // free places of the panel's banks before
    __shared__ uint32_t s_off[kLayWarps][kSliceMaxPanels], s_rst[kLayWarps][kSliceMaxPanels];
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t nw = gridDim.x * kLayWarps, keys = b.P * kBanks;
    uint32_t *cur = s_cur[wid], *tot = s_tot[wid], *ovb = s_ovb[wid], *hob = s_hob[wid];
    CO *ocol = (CO *)b.ocol;
    WO *ow = (WO *)b.ow;
    const WI *w = (const WI *)b.w;
    for (uint32_t it = blockIdx.x * kLayWarps + wid; it < b.nitems; it += nw) {
        const uint32_t o = b.irow[it];
        const uint32_t i = b.perm ? b.perm[o] : o;
        const uint32_t k0 = (it - b.iptr[o]) * kSliceItem;
        const uint32_t s = b.rp[o] + k0;
        const uint32_t e = b.rp[o + 1] - s < kSliceItem ? b.rp[o + 1] : s + kSliceItem;
        __syncwarp();
        if (lane < b.P) {
            s_off[wid][lane] = b.roff[(size_t)lane * b.n32 + i];
            s_rst[wid][lane] = b.rst[(size_t)lane * b.n32 + i];
        }
        auto dest = [&](uint32_t j) -> uint32_t {
            return b.tcol ? b.tcol[j] : (b.perm ? __ldg(b.perm + b.col[j]) : b.col[j]);
        };
        if constexpr (!BANKED) {
            __syncwarp();
            const uint32_t off = s_off[wid][0], lg = s_rst[wid][0] >> 24;
            const uint32_t sub = (i & ((32u >> lg) - 1u)) << lg;
            for (uint32_t j = s + lane; j < e; j += 32) {
                const uint32_t r = k0 + j - s;
                const uint64_t at =
                    ((uint64_t)(off + (r >> (2 + lg))) * 32 + sub + ((r >> 2) & ((1u << lg) - 1u))) * 4 + (r & 3u);
                ocol[at] = (CO)dest(j);
                if (ow) ow[at] = (WO)w[j];
            }
        } else {
            const bool multi = b.iptr[o + 1] - b.iptr[o] > 1;
            if (multi) {
                for (uint32_t k = lane; k < keys; k += 32) {
                    cur[k] = b.icnt[(size_t)(b.mptr[o] + it - b.iptr[o]) * keys + k];
                    tot[k] = b.mtot[(size_t)b.mptr[o] * keys + k];
                }
            } else {
                for (uint32_t k = lane; k < keys; k += 32) {
                    cur[k] = 0;
                    tot[k] = 0;
                }
                __syncwarp();
                for (uint32_t j = s + lane; j < e; j += 32) {
                    const uint32_t c = dest(j);
                    const uint32_t p = b.P > 1 ? c / kSlicePW : 0u;
                    atomicAdd(&tot[p * kBanks + (c & (kBanks - 1))], b.expand ? (uint32_t)w[j] : 1u);
                }
            }
            __syncwarp();
            for (uint32_t kk = 0; kk < keys; kk += 32) {   // 16 lanes a panel
                const uint32_t k = kk + lane, p = (k < keys ? k : 0u) / kBanks;
                const uint32_t st = s_rst[wid][p], lg = st >> 24;
                const uint32_t sub = lg == 5 ? 0u : i & ((32u >> lg) - 1u);
                const BankPlaces bp(k & (kBanks - 1), lg, sub, 4 * (st & 0xFFFFFFu));
                const uint32_t c = k < keys ? tot[k] : 0u;
                const uint32_t ov = c > bp.cap ? c - bp.cap : 0u, ho = c < bp.cap ? bp.cap - c : 0u;
                uint32_t x = ov, y = ho;
                for (int d = 1; d < (int)kBanks; d <<= 1) {
                    const uint32_t tx = __shfl_up_sync(0xFFFFFFFFu, x, d, kBanks);
                    const uint32_t ty = __shfl_up_sync(0xFFFFFFFFu, y, d, kBanks);
                    if ((lane & (kBanks - 1)) >= (unsigned)d) { x += tx; y += ty; }
                }
                if (k < keys) { ovb[k] = x - ov; hob[k] = y - ho; }
            }
            __syncwarp();
            for (uint32_t j0 = s; j0 < e; j0 += 32) {
                const uint32_t j = j0 + lane;
                const bool ok = j < e;
                uint32_t c = 0, m = 0;
                WI wt = 0;
                if (ok) {
                    c = dest(j);
                    if (w) wt = w[j];
                    m = b.expand ? (uint32_t)wt : 1u;
                }
                const uint32_t p = b.P > 1 ? c / kSlicePW : 0u;
                const uint32_t key = ok ? p * kBanks + (c & (kBanks - 1)) : 0xFFFFFFFFu;
                const unsigned peers = __match_any_sync(0xFFFFFFFFu, key);
                uint32_t before = __popc(peers & ((1u << lane) - 1u)), all = __popc(peers);
                if (b.expand) {   // entries of several copies
                    unsigned many = __ballot_sync(0xFFFFFFFFu, ok && m != 1u);
                    while (many) {
                        const int q = __ffs(many) - 1;
                        const uint32_t more = __shfl_sync(0xFFFFFFFFu, m, q) - 1u;
                        if (peers >> q & 1u) {
                            all += more;
                            if (q < (int)lane) before += more;
                        }
                        many &= many - 1;
                    }
                }
                uint32_t rank = 0;
                if (ok) rank = cur[key] + before;
                __syncwarp();
                if (ok && (int)lane == __ffs(peers) - 1) cur[key] = rank + all;
                __syncwarp();
                if (!ok) continue;
                const uint32_t st = s_rst[wid][p], lg = st >> 24, S = 4 * (st & 0xFFFFFFu), off = s_off[wid][p];
                const uint32_t sub = lg == 5 ? 0u : i & ((32u >> lg) - 1u);
                const BankPlaces mine(c & (kBanks - 1), lg, sub, S);
                for (uint32_t q = 0; q < m; q++) {
                    uint32_t k = rank + q, t, ln;
                    if (k < mine.cap) {
                        t = mine.slot(k);
                        ln = mine.lane_of(k);
                    } else {
                        // the free place of the overflow's number
                        const uint32_t v = ovb[key] + k - mine.cap;
                        const uint32_t *hb = hob + p * kBanks;
                        uint32_t lo = 0, hi = kBanks - 1;   // last bank with hb <= v
                        while (lo < hi) {
                            const uint32_t mid = (lo + hi + 1) >> 1;
                            if (hb[mid] <= v) lo = mid;
                            else hi = mid - 1;
                        }
                        const BankPlaces f(lo, lg, sub, S);
                        k = tot[p * kBanks + lo] + v - hb[lo];
                        t = f.slot(k);
                        ln = f.lane_of(k);
                    }
                    const uint64_t at = ((uint64_t)(off + (t >> 2)) * 32 + ln) * 4 + (t & 3u);
                    ocol[at] = (CO)(c - p * kSlicePW);
                    if (ow) ow[at] = (WO)wt;
                }
            }
        }
    }
}

// ------------------------------------------------------------------ host --
// levels of fewer mean entries per row and panel gather from L2 instead
constexpr double kSliceMinSeg = 5.0;

// largest weight that is laid out as copies of its entry (R-MAT 22's level 1
// has 160)
constexpr uint64_t kMaxCopies = 4096;

// levels whose gathers beyond the leading kSlicePW vertices in degree order
// are at most this many take the hub form: panels cost a second barrier and a
// pass over the rows' panel sums, about 5 us, a gather from L2 two clocks of an
// SM
constexpr uint64_t kHubTail = 1ull << 20;

// A row in one block takes its entries' time there: a row this much longer than
// a block's share (gathers from L2 / from shared memory) costs more than the
// second barrier, about 3 us.  A star of 100,000 vertices 39 -> 9 us an iteration
// (the main kernel 33), of 30,000 and 60,000 random pairs 18 -> 9.2 (12), 4 hubs
// among 1,000,000 vertices of six entries 142 -> 38 (105); rows of 7,500 in the
// hub form are quicker in one block (8.7 against 9.6).
constexpr uint64_t kLongRowGlobal = 4096, kLongRowShared = 16384;

// The form of a level.  skew: its longest row is at least four times the mean;
// tail: its entries beyond the leading kSlicePW vertices in degree order.
// Mesh level of 57,210 vertices, 4.1 entries per row and panel: panels 12.6 us
// an iteration, global 7.1; R-MAT 16's input level, 19 entries: 17 and 24.
static SliceForm slice_form(uint32_t n, uint64_t m, bool skew, uint64_t tail) {
    if (n <= kSlicePW) return kFormShared;
    if (skew && tail <= kHubTail) return kFormHub;
    const uint64_t P = cdiv(n, kSlicePW);
    if (P <= kSliceMaxPanels && (double)m >= kSliceMinSeg * (double)n * (double)P) return kFormPanels;
    return kFormGlobal;
}

bool power_iter_slices_ok(const Level &L, const PowerIterOpts &o) {
    if (pi_plain(o)) return false;
    if (L.n == 0 || L.m == 0 || L.n > 0x7FFFFFFFu) return false;
    return L.wbytes == 0 || L.wbytes == 4 || L.wbytes == 8;
}

template <int FORM, bool CROSS>
static const void *slice_kernel(int wb) {
    switch (wb) {
        case 0: return (const void *)k_pi_slices<FORM, 0, CROSS>;
        case 1: return (const void *)k_pi_slices<FORM, 1, CROSS>;
        case 2: return (const void *)k_pi_slices<FORM, 2, CROSS>;
        case 4: return (const void *)k_pi_slices<FORM, 4, CROSS>;
        default: return (const void *)k_pi_slices<FORM, 8, CROSS>;
    }
}

template <int FORM>
static const void *direct_kernel(int wb, bool cross) {
    return cross ? slice_kernel<FORM, true>(wb) : slice_kernel<FORM, false>(wb);
}

template <typename WI>
static int slice_fill(Context &C, const SliceBuild &b, bool wide, int wb, uint32_t grid) {
    constexpr int T = 32 * kLayWarps;
    auto go = [&](auto co) {
        using CO = decltype(co);
        if (wb == 0) k_sl_fill<WI, char, CO><<<grid, T, 0, C.stream>>>(b);
        else if (wb == 1) k_sl_fill<WI, uint8_t, CO><<<grid, T, 0, C.stream>>>(b);
        else if (wb == 2) k_sl_fill<WI, uint16_t, CO><<<grid, T, 0, C.stream>>>(b);
        else if (wb == 4) k_sl_fill<WI, uint32_t, CO><<<grid, T, 0, C.stream>>>(b);
        else k_sl_fill<WI, unsigned long long, CO><<<grid, T, 0, C.stream>>>(b);
    };
    if (wide) go((uint32_t)0);
    else go((uint16_t)0);
    C.kernel_launches++;
    SGPB_CUDA(cudaGetLastError());
    return SGP_B200_OK;
}

// Lays the level out and runs it; *tight: the layout did not fit, nothing ran.
static int slices_run(Context &C, const Level &L, const double *x_in, const uint32_t *vcmap, double *x_out,
                      const PowerIterOpts &o, uint64_t iter_max, uint64_t iter0, double dot0, PowerIterResult *res,
                      bool *tight) {
    const uint32_t n = L.n;
    SliceBuild b;
    memset(&b, 0, sizeof(b));
    SliceArgs a;
    memset(&a, 0, sizeof(a));
    b.n = n;
    b.n32 = cdiv(n, 32) * 32;
    b.ng = b.n32 / 32;
    b.rp = L.rp; b.col = L.col; b.w = L.w;
    // rows and items
    uint32_t *items, *iptr, *head;
    SGPB_TRY(dalloc_t(C, &items, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &iptr, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &head, 8));
    SGPB_TRY(dzero(C, head, 32));
    k_sl_rows<<<cdiv(n, 256), 256, 0, C.stream>>>(n, L.rp, items, head);
    C.kernel_launches++;
    SGPB_TRY(scan_u32(C, items, iptr, n, nullptr));
    // at most one item a row and one more for each kSliceItem entries
    const uint64_t max_items = (uint64_t)n + L.m / kSliceItem + 1;
    uint32_t *irow;
    SGPB_TRY(dalloc_t(C, &irow, max_items));
    k_sl_item_rows<<<cdiv(n, 256), 256, 0, C.stream>>>(n, iptr, irow);
    C.kernel_launches++;
    SGPB_CUDA(cudaMemcpyAsync(head + 1, iptr + n, 4, cudaMemcpyDeviceToDevice, C.stream));
    uint32_t h[6];
    SGPB_TRY(read_u32(C, head, h, 2));
    const uint32_t maxlen = h[0];
    b.nitems = h[1];
    b.iptr = iptr; b.irow = irow;
    const uint32_t wgrid = b.nitems / 8 + 1 < (uint32_t)C.num_sms * 16 ? b.nitems / 8 + 1 : (uint32_t)C.num_sms * 16;
    // weighted degrees, total and largest weight
    uint64_t wtot = 0, wmax = 0;
    if (L.w) {
        unsigned long long *dsum, *stat;
        SGPB_TRY(dalloc_t(C, &dsum, n));
        SGPB_TRY(dalloc_t(C, &stat, 2));
        SGPB_TRY(dzero(C, dsum, sizeof(*dsum) * (size_t)n));
        SGPB_TRY(dzero(C, stat, 16));
        if (L.wbytes == 8)
            k_sl_weights<unsigned long long><<<wgrid, 256, 0, C.stream>>>(b.nitems, iptr, irow, L.rp,
                                                                          (const unsigned long long *)L.w, dsum, stat);
        else
            k_sl_weights<uint32_t><<<wgrid, 256, 0, C.stream>>>(b.nitems, iptr, irow, L.rp, (const uint32_t *)L.w,
                                                                dsum, stat);
        C.kernel_launches++;
        uint64_t st[2];
        SGPB_TRY(read_u64(C, (const uint64_t *)stat, st, 2));
        wtot = st[0];
        wmax = st[1];
        b.dsum = dsum;
    }
    // skewed levels are laid out in degree order: rows of a group then have
    // like lengths, and the most referenced columns share the first panels
    const double avg = (double)L.m / n;
    const bool skew = maxlen >= 4.0 * avg && avg >= 4.0;
    uint64_t tail = 0;
    if (skew) {
        uint32_t *perm, *inv;
        SGPB_TRY(degree_order(C, n, L.rp, &perm, &inv));
        b.perm = perm;
        b.inv = inv;
        if (n > kSlicePW) {
            unsigned long long *lead;
            SGPB_TRY(dalloc_t(C, &lead, 1));
            SGPB_TRY(dzero(C, lead, 8));
            k_sl_lead<<<cdiv(kSlicePW, 256), 256, 0, C.stream>>>(L.rp, inv, lead);
            C.kernel_launches++;
            SGPB_TRY(read_u64(C, (const uint64_t *)lead, &tail));
            tail = L.m - tail;
        }
    }
    const SliceForm form = slice_form(n, L.m, skew, tail);
    if (form == kFormGlobal) b.perm = b.inv = nullptr;   // its gathers keep the level's locality
    const bool wide = form == kFormGlobal || form == kFormHub;   // 32-bit destinations, places by rank
    b.l2 = form == kFormGlobal;
    b.direct = form != kFormPanels;
    b.P = form == kFormPanels ? cdiv(n, kSlicePW) : 1u;
    // (one lane writes an entry's copies: at most kMaxCopies)
    b.expand = form == kFormPanels && L.w && wmax <= kMaxCopies && wtot <= 0xFFFFFFFFull &&
               (double)wtot <= 1.25 * (double)L.m;
    const int wb = !L.w || b.expand ? 0 : wmax <= 0xFF ? 1 : wmax <= 0xFFFF ? 2 : wmax <= 0xFFFFFFFFull ? 4 : 8;
    const uint64_t me = b.expand ? wtot : L.m;
    // entries per lane and unit, 8 .. 64: units of at most a warp's share (with
    // a quarter of it R-MAT 16's 6,915 vertices took 7.5 instead of 6.6 us an
    // iteration, a mesh level of 190,000 14.3 instead of 10.5)
    uint32_t epl = 8;
    while (epl < 64 && (uint64_t)epl * 2 * C.num_sms * 16 * 16 <= me) epl *= 2;
    b.epl = epl;
    const size_t pn = (size_t)b.P * b.n32, pg = (size_t)b.P * b.ng;
    double *deg;
    uint32_t *unb, *stb, *sptr;
    SGPB_TRY(dalloc_t(C, &deg, b.n32));
    SGPB_TRY(dalloc_t(C, &b.cnt, pn));
    SGPB_TRY(dalloc_t(C, &b.roff, pn));
    SGPB_TRY(dalloc_t(C, &b.nun, pg + 1));
    SGPB_TRY(dalloc_t(C, &b.nst, pg + 1));
    SGPB_TRY(dalloc_t(C, &unb, pg + 1));
    SGPB_TRY(dalloc_t(C, &stb, pg + 1));
    SGPB_TRY(dalloc_t(C, &b.slotc, (size_t)b.n32 + 1));
    SGPB_TRY(dalloc_t(C, &sptr, (size_t)b.n32 + 1));
    SGPB_TRY(dzero(C, b.slotc, sizeof(uint32_t) * b.n32));
    b.deg = deg;
    SGPB_TRY(dalloc_t(C, &b.rst, pn));
    const uint32_t lgrid = cdiv(b.nitems, kLayWarps) < (uint32_t)C.num_sms * 16 ? cdiv(b.nitems, kLayWarps)
                                                                              : (uint32_t)C.num_sms * 16;
    const bool multi = !wide && maxlen > kSliceItem;
    if (b.P > 1) {
        SGPB_TRY(dalloc_t(C, &b.tcol, L.m));
        SGPB_TRY(dzero(C, b.cnt, sizeof(uint32_t) * pn));
    }
    if (multi) {
        // (panel, bank) counts of the items of rows longer than one item
        // (such a row has at most twice its entries / kSliceItem items)
        const size_t max_multi = 2 * (size_t)(L.m / kSliceItem) + 2;
        uint32_t *mptr;
        SGPB_TRY(dalloc_t(C, &mptr, (size_t)n + 1));
        k_sl_multi<<<cdiv(n, 256), 256, 0, C.stream>>>(n, iptr, items);
        SGPB_TRY(scan_u32(C, items, mptr, n, nullptr));
        SGPB_TRY(dalloc_t(C, &b.icnt, max_multi * b.P * kBanks));
        SGPB_TRY(dalloc_t(C, &b.mtot, max_multi * b.P * kBanks));
        b.mptr = mptr;
        C.kernel_launches++;
    }
    if (b.P > 1 || multi) {
        if (L.wbytes == 8) k_sl_count<unsigned long long><<<lgrid, 32 * kLayWarps, 0, C.stream>>>(b, b.P == 1);
        else k_sl_count<uint32_t><<<lgrid, 32 * kLayWarps, 0, C.stream>>>(b, b.P == 1);
        C.kernel_launches++;
    }
    if (multi) {
        const uint32_t g = cdiv(n, kLayWarps) < (uint32_t)C.num_sms * 16 ? cdiv(n, kLayWarps) : (uint32_t)C.num_sms * 16;
        k_sl_row_counts<<<g, 32 * kLayWarps, 0, C.stream>>>(b);
        C.kernel_launches++;
    }
    k_sl_degrees<<<cdiv(b.n32, 256), 256, 0, C.stream>>>(b);
    k_sl_groups<<<cdiv(pg * 32, 256), 256, 0, C.stream>>>(b);
    C.kernel_launches += 2;
    SGPB_TRY(scan_u32(C, b.nun, unb, (uint32_t)pg, nullptr));
    SGPB_TRY(scan_u32(C, b.nst, stb, (uint32_t)pg, nullptr));
    SGPB_TRY(scan_u32(C, b.slotc, sptr, b.n32, nullptr));
    SGPB_CUDA(cudaMemcpyAsync(head + 2, unb + pg, 4, cudaMemcpyDeviceToDevice, C.stream));
    SGPB_CUDA(cudaMemcpyAsync(head + 3, stb + pg, 4, cudaMemcpyDeviceToDevice, C.stream));
    SGPB_CUDA(cudaMemcpyAsync(head + 4, sptr + b.n32, 4, cudaMemcpyDeviceToDevice, C.stream));
    SGPB_TRY(read_u32(C, head, h, 5));
    const uint32_t nu = h[2], nst = h[3], nslots = h[4];
    b.unb = unb; b.stb = stb; b.sptr = sptr;
    uint32_t *cpre;
    const size_t cb = wide ? 4 : 2;
    if (const char *e = getenv("SGPB_PI_SLICES_MB"))   // a limit on the laid-out matrix
        if (*e && (uint64_t)nst * 128 * (cb + wb) > strtoull(e, nullptr, 10) << 20) {
            *tight = true;
            return SGP_B200_ERR_DEVICE;
        }
    SGPB_TRY(dalloc_t(C, &b.unit, (size_t)nu + 1));
    SGPB_TRY(dalloc_t(C, &b.ucost, (size_t)nu + 1));
    SGPB_TRY(dalloc_t(C, &cpre, (size_t)nu + 1));
    SGPB_TRY(dalloc_t(C, &b.pan_u, (size_t)b.P + 1));
    SGPB_TRY(dalloc(C, &b.ocol, (size_t)nst * 128 * cb));
    if (wide) SGPB_CUDA(cudaMemsetAsync(b.ocol, 0xFF, (size_t)nst * 128 * cb, C.stream));
    if (wb) {
        SGPB_TRY(dalloc(C, &b.ow, (size_t)nst * 128 * wb));
        SGPB_TRY(dzero(C, b.ow, (size_t)nst * 128 * wb));
    }
    k_sl_units<<<cdiv(pg * 32, 256), 256, 0, C.stream>>>(b);
    C.kernel_launches++;
    SGPB_TRY(scan_u32(C, b.ucost, cpre, nu, nullptr));
    if (!wide) {
        const uint32_t g = cdiv(nu, 8) < (uint32_t)C.num_sms * 16 ? cdiv(nu, 8) : (uint32_t)C.num_sms * 16;
        k_sl_preset<<<g, 256, 0, C.stream>>>(b, nu);
        C.kernel_launches++;
    }
    if (L.wbytes == 8) SGPB_TRY(slice_fill<unsigned long long>(C, b, wide, wb, lgrid));
    else SGPB_TRY(slice_fill<uint32_t>(C, b, wide, wb, lgrid));
    // the run
    a.n = n; a.n32 = b.n32; a.P = b.P; a.nu = nu; a.unit = b.unit; a.cpre = cpre; a.pan_u = b.pan_u;
    a.col = b.ocol; a.w = b.ow; a.sptr = sptr; a.nslots = nslots; a.deg = deg; a.inv = b.inv;
    a.x_in = x_in; a.vcmap = vcmap; a.out = x_out;
    SGPB_TRY(dalloc_t(C, &a.spart, (size_t)nslots + 1));
    if (b.direct && nslots && maxlen > me / C.num_sms + (b.l2 ? kLongRowGlobal : kLongRowShared)) {
        uint8_t *flags;
        uint32_t *list, *cnt;
        SGPB_TRY(dalloc_t(C, &flags, n));
        SGPB_TRY(dalloc_t(C, &list, (size_t)n + 1));
        SGPB_TRY(dalloc_t(C, &cnt, 1));
        k_sl_chunked<<<cdiv(n, 256), 256, 0, C.stream>>>(n, sptr, flags);
        C.kernel_launches++;
        SGPB_TRY(compact_flags(C, flags, n, list, cnt));
        SGPB_TRY(read_u32(C, cnt, &a.ncross));
        a.cross = list;
    }
    SGPB_TRY(dalloc_t(C, &a.va, b.n32));
    SGPB_TRY(dalloc_t(C, &a.vb, b.n32));
    SGPB_CUDA(cudaMemsetAsync(a.va + (n & ~1u), 0, sizeof(double) * (b.n32 - (n & ~1u)), C.stream));
    SGPB_CUDA(cudaMemsetAsync(a.vb + (n & ~1u), 0, sizeof(double) * (b.n32 - (n & ~1u)), C.stream));
    if (b.P > 1) {
        SGPB_TRY(dalloc_t(C, &a.y, pn));
        SGPB_TRY(dzero(C, a.y, sizeof(double) * pn));
    }
    double *res_d;
    SGPB_TRY(dalloc_t(C, &res_d, 8));
    SGPB_TRY(dalloc_t(C, &a.bar, 2));
    SGPB_TRY(dzero(C, a.bar, 8));
    SGPB_TRY(dzero(C, res_d, 64));
    a.err = a.bar + 1;
    a.spin = kSpinLimit;
    if (const char *e = getenv("SGPB_PI_SPIN"))   // another limit (0: the first wait gives up)
        if (*e) a.spin = (uint32_t)strtoul(e, nullptr, 10);
    a.res = res_d;
    a.tol = o.tol;
    a.iter_max = iter_max;
    a.iter0 = iter0;
    a.dot0 = dot0;
    const int threads = slice_threads(form, wb);
    uint32_t grid = cdiv(nu, (uint32_t)threads / 32);
    if (grid > (uint32_t)C.num_sms) grid = C.num_sms;
    if (C.grid_cap && grid > C.grid_cap) grid = C.grid_cap;
    if (grid < 1) grid = 1;
    SGPB_TRY(dalloc_t(C, &a.partials, (size_t)8 * grid));
    const void *k = form == kFormShared   ? direct_kernel<kFormShared>(wb, a.ncross != 0)
                    : form == kFormGlobal ? direct_kernel<kFormGlobal>(wb, a.ncross != 0)
                    : form == kFormHub    ? direct_kernel<kFormHub>(wb, a.ncross != 0)
                                          : slice_kernel<kFormPanels, false>(wb);
    const size_t dyn = form == kFormGlobal ? 0 : kSliceSmem;
    if (dyn) SGPB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSliceSmem));
    cudaEvent_t ev[2];
    for (auto &e : ev) SGPB_CUDA(cudaEventCreate(&e));
    struct EvFree {
        cudaEvent_t *e;
        ~EvFree() { cudaEventDestroy(e[0]); cudaEventDestroy(e[1]); }
    } evfree{ev};
    SGPB_CUDA(cudaEventRecord(ev[0], C.stream));
    void *args[] = {&a};
    SGPB_CUDA(cudaLaunchCooperativeKernel(k, dim3(grid), dim3((unsigned)threads), args, dyn, C.stream));
    C.kernel_launches++;
    SGPB_CUDA(cudaEventRecord(ev[1], C.stream));
    SGPB_CUDA(cudaMemcpyAsync(C.h_pinned, res_d, 8 * sizeof(double), cudaMemcpyDeviceToHost, C.stream));
    SGPB_CUDA(cudaMemcpyAsync((double *)C.h_pinned + 8, a.err, 4, cudaMemcpyDeviceToHost, C.stream));
    SGPB_CUDA(cudaStreamSynchronize(C.stream));
    const double *r = (const double *)C.h_pinned;
    if (*(const uint32_t *)(r + 8)) {
        set_error("power iteration: a grid barrier did not complete within its wait limit");
        return SGP_B200_ERR_DEVICE;
    }
    res->niter = (uint64_t)r[0];
    res->dot = r[1];
    res->gb = r[2];
    res->lambda = r[3];
    res->capped = r[4] != 0.0;
    res->resid = 0;
    res->close = r[7] < kStopMargin;
    float t = 0;
    cudaEventElapsedTime(&t, ev[0], ev[1]);
    res->kernel_ms = t;
    return SGP_B200_OK;
}

int power_iter_slices(Context &C, const Level &L, const double *x_in, const uint32_t *vcmap, double *x_out,
                      const PowerIterOpts &o, uint64_t iter_max, uint64_t iter0, double dot0, PowerIterResult *res,
                      bool *fits) {
    const size_t mark = C.owned.size();
    bool tight = false;
    C.out_of_memory = false;
    const int rc = slices_run(C, L, x_in, vcmap, x_out, o, iter_max, iter0, dot0, res, &tight);
    // the layout is this call's alone: give it back before the next level
    for (size_t q = mark; q < C.owned.size(); q++) cudaFreeAsync(C.owned[q], C.stream);
    C.owned.resize(mark);
    *fits = rc == SGP_B200_OK || !(tight || C.out_of_memory);
    return *fits ? rc : SGP_B200_OK;
}

}  // namespace sgpb
