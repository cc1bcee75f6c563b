// fm.cu -- FM refinement of a bisection on the device.
//
// The reference's FM (cmg/eigensolve_kokkos.h:973-1240, fm_refine) is a
// host-serial pass over gain-bucket lists whose initial order comes from a
// parallel build, and its parallel variant (:695-971, fm_refine_par, disabled
// there) orders moves through atomics and picks the best prefix with a
// non-associative scan.  This pass keeps fm_refine_par's structure with
// deterministic rules (oracle/sgpar_oracle.c orc_fm_refine restates them):
//   1. gain(u) = neighbours across the cut minus those inside (the finest
//      level's edges all weigh 1);
//   2. each side's positive-gain vertices ordered by (gain clamped to
//      kFmBuckets - 1 descending, id ascending) -- a stable counting sort of
//      the id-ordered candidates;
//   3. the two lists interleaved by the serial FM's balance rule
//      (:1105-1140): side 0 while the balance (part-0 minus part-1 vertices)
//      is positive, side 1 while negative, at zero the head of larger gain
//      (side 0 on a tie), the other list once one runs out.  With unit
//      vertex weights this order has a closed form: ceil(|d| / 2) moves from
//      the heavy side, then pairs (fixed order at balance -+1, by gain at 0),
//      then the rest of the longer list;
//   4. sequential gains: the gain of the i-th move given that the first i
//      have moved; cut after k moves = cut - their sum;
//   5. k* = the k (0 included) of least cut whose |balance| is within the
//      serial FM's target max(|d| / 10, 20) (:1073-1076), the largest such k
//      on a tie (its "<="); the first k* moves are applied.
// Passes repeat until one applies nothing or leaves the cut unchanged.
#include <cooperative_groups.h>

#include <stdlib.h>

#include <type_traits>

#include "bits.cuh"
#include "common.cuh"
#include "internal.h"

namespace cg = cooperative_groups;

namespace sgpb {

constexpr int kFmBuckets = 1024;
constexpr int kFmTile = 1024;   // candidates per block in the counting sort

// Gains, candidate flags, cut and balance.  Unit edge weights (the finest
// level): a symmetric graph with fewer than 2^32 directed entries has every
// degree below 2^31, so 32-bit sums are exact.  The parts are a bitmap, in
// the block's shared memory when it fits (SHARED); rows of more than kLongRow
// entries take a block each, the others G lanes each with four entries per
// lane in flight.  R-MAT 18 (7.6M entries, hubs of 30,000): with parts
// gathered through L1 and hub rows on a warp each 177 us a pass, now 24.
struct FmGraph {
    uint32_t n;
    const uint32_t *rp, *col;
    const uint32_t *bits;     // part 1
    const uint32_t *longs;    // rows of more than kLongRow entries
    const uint32_t *nlong;
};

template <int G, bool SHARED>
__global__ void __launch_bounds__(1024) k_fm_gain(FmGraph a, long long *__restrict__ gain,
                                                  uint32_t *__restrict__ flag /* [2n]: side 0, side 1 */,
                                                  unsigned long long *__restrict__ sums /* [0] 2 cut, [1] balance,
                                                                                           [2], [3] candidates */) {
    extern __shared__ uint32_t s_bits[];
    __shared__ int s_sum;
    if (SHARED) bits_load(a.bits, bit_words(a.n), s_bits);
    const uint32_t *bits = SHARED ? (const uint32_t *)s_bits : a.bits;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    unsigned long long cut2 = 0;
    long long bal = 0;
    uint32_t c0 = 0, c1 = 0;
    auto done = [&](uint32_t u, uint32_t pu, int across, int deg) {
        const int g = 2 * across - deg;   // across minus inside
        gain[u] = g;
        flag[u] = pu == 0 && g > 0;
        flag[(size_t)a.n + u] = pu != 0 && g > 0;
        c0 += pu == 0 && g > 0;
        c1 += pu != 0 && g > 0;
        cut2 += (unsigned)across;
        bal += pu == 0 ? 1 : -1;
    };
    const uint32_t nl = *a.nlong;
    for (uint32_t r = blockIdx.x; r < nl; r += gridDim.x) {
        const uint32_t u = __ldg(a.longs + r), b = __ldg(a.rp + u), e = __ldg(a.rp + u + 1);
        const uint32_t pu = bit_of(bits, u);
        int across = 0;
#pragma unroll 4
        for (uint64_t j = (uint64_t)b + threadIdx.x; j < e; j += 1024) across += bit_of(bits, __ldg(a.col + j)) != pu;
        across = __reduce_add_sync(0xFFFFFFFFu, across);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, across);
        __syncthreads();
        if (threadIdx.x == 0) {
            done(u, pu, s_sum, (int)(e - b));
            s_sum = 0;
        }
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & (G - 1);
    const uint64_t ng = ((uint64_t)gridDim.x * blockDim.x) / G;
    for (uint64_t u = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; u < a.n; u += ng) {
        const uint32_t b = __ldg(a.rp + u), e = __ldg(a.rp + u + 1);
        if (e - b > kLongRow) continue;   // uniform in the row's group
        const uint32_t pu = bit_of(bits, (uint32_t)u);
        int across = 0;
        for (uint32_t j0 = b + lane; j0 < e; j0 += 4 * G) {
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = j0 + q * G < e ? __ldg(a.col + j0 + q * G) : (uint32_t)u;
#pragma unroll
            for (int q = 0; q < 4; q++) across += bit_of(bits, v[q]) != pu;
        }
        across = group_sum<G>(across);
        if (lane == 0) done((uint32_t)u, pu, across, (int)(e - b));
    }
    cut2 = warp_sum(cut2);
    bal = warp_sum(bal);
    c0 = __reduce_add_sync(0xFFFFFFFFu, c0);
    c1 = __reduce_add_sync(0xFFFFFFFFu, c1);
    if ((threadIdx.x & 31) == 0) {
        if (cut2) atomicAdd(sums, cut2);
        if (bal) atomicAdd(sums + 1, (unsigned long long)bal);
        if (c0) atomicAdd(sums + 2, (unsigned long long)c0);
        if (c1) atomicAdd(sums + 3, (unsigned long long)c1);
    }
}

__device__ __forceinline__ uint32_t fm_bucket(long long g) {
    return g < kFmBuckets - 1 ? (uint32_t)g : (uint32_t)(kFmBuckets - 1);
}

// flagged vertices in order (n2 = 2n flags: side 0 before side 1)
__global__ void k_fm_list(uint32_t n2, const uint32_t *__restrict__ flag, const uint32_t *__restrict__ pos, uint32_t n,
                          uint32_t *__restrict__ idx) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n2 && flag[i]) idx[pos[i]] = (uint32_t)(i < n ? i : i - n);
}

// Counting sort of both sides' candidates (the first na of the list are side
// 0's): key = side, then the descending bucket.  Above kFmJoint candidates a side
// at a time (half the keys, na = len), so that keys times tiles fit 32 bits and
// the histogram stays at 8 bytes a candidate.
constexpr int kFmKeys = 2 * kFmBuckets;
constexpr uint64_t kFmJoint = 1ull << 28;
__device__ __forceinline__ uint32_t fm_key(uint32_t i, uint32_t na, long long g) {
    return (i < na ? 0u : (uint32_t)kFmBuckets) + (uint32_t)(kFmBuckets - 1) - fm_bucket(g);
}

// counts per (key, tile): hist[key * ntiles + t]
__global__ void __launch_bounds__(kFmTile) k_fm_hist(uint32_t len, uint32_t na, const uint32_t *__restrict__ idx,
                                                     const long long *__restrict__ gain, uint32_t ntiles,
                                                     int keys, uint32_t *__restrict__ hist) {
    __shared__ uint32_t cnt[kFmKeys];
    for (int b = threadIdx.x; b < keys; b += blockDim.x) cnt[b] = 0;
    __syncthreads();
    const uint32_t i = blockIdx.x * kFmTile + threadIdx.x;
    if (i < len) atomicAdd(&cnt[fm_key(i, na, gain[idx[i]])], 1u);
    __syncthreads();
    for (int b = threadIdx.x; b < keys; b += blockDim.x) hist[(size_t)b * ntiles + blockIdx.x] = cnt[b];
}

// stable placement: within a tile the warps take turns in order, and lanes
// of one key rank by lane
__global__ void __launch_bounds__(kFmTile) k_fm_place(uint32_t len, uint32_t na, const uint32_t *__restrict__ idx,
                                                      const long long *__restrict__ gain, uint32_t ntiles,
                                                      int keys, const uint32_t *__restrict__ off,
                                                      uint32_t *__restrict__ sorted) {
    __shared__ uint32_t cnt[kFmKeys];
    for (int b = threadIdx.x; b < keys; b += blockDim.x) cnt[b] = 0;
    __syncthreads();
    const uint32_t i = blockIdx.x * kFmTile + threadIdx.x;
    const bool valid = i < len;
    const uint32_t u = valid ? idx[i] : 0u;
    const uint32_t b = valid ? fm_key(i, na, gain[u]) : 0u;
    const uint32_t base = valid ? off[(size_t)b * ntiles + blockIdx.x] : 0u;
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned act = __ballot_sync(0xFFFFFFFFu, valid);
    const unsigned peers = valid ? __match_any_sync(act, b) : 0u;
    for (unsigned turn = 0; turn < kFmTile / 32; turn++) {
        if (wid == turn && valid) {
            const uint32_t r = cnt[b] + __popc(peers & ((1u << lane) - 1u));
            sorted[base + r] = u;
            __syncwarp(peers);
            if ((int)lane == __ffs(peers) - 1) cnt[b] += __popc(peers);
        }
        __syncthreads();
    }
}

// closed-form interleave (see the header): order[pos] = vertex, rank[v] = pos
__global__ void k_fm_interleave(uint32_t na, uint32_t nb, const uint32_t *__restrict__ A,
                                const uint32_t *__restrict__ B, const long long *__restrict__ gain, long long d,
                                uint32_t *__restrict__ order, uint32_t *__restrict__ rank,
                                uint32_t *__restrict__ listed, uint8_t *__restrict__ side,
                                unsigned long long key0, unsigned long long *__restrict__ best) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *best = key0;   // k = 0
    // phase 1: ceil(|d| / 2) moves from the heavier side (as many as it has)
    const bool heavy0 = d > 0;
    const uint64_t want = d > 0 ? (uint64_t)(d + 1) / 2 : (uint64_t)(-d + 1) / 2;
    const uint32_t nh = heavy0 ? na : nb;
    const uint32_t p0 = (uint32_t)(want < nh ? want : nh);
    // balance after phase 1 when the heavy side lasted: 0 or -+1
    const long long r = heavy0 ? d - 2 * (long long)p0 : d + 2 * (long long)p0;
    const uint32_t ra = heavy0 ? na - p0 : na, rb = heavy0 ? nb : nb - p0;   // left after phase 1
    const uint32_t a0 = heavy0 ? p0 : 0, b0 = heavy0 ? 0 : p0;                // first index left
    const uint32_t m = ra < rb ? ra : rb;                                     // full pairs
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t tot = na > nb ? na : nb;
    for (uint64_t i = tid; i < tot; i += stride) {
        for (int s = 0; s < 2; s++) {
            const uint32_t len = s == 0 ? na : nb;
            if (i >= len) continue;
            const uint32_t u = s == 0 ? A[i] : B[i];
            uint64_t pos;
            const uint32_t first = s == 0 ? a0 : b0;
            if ((s == 0) == heavy0 && i < p0 && d != 0) {
                pos = i;                                      // phase 1
            } else if (i - first < m) {
                const uint32_t k = i - first;                 // pair k
                bool a_first;
                if (r > 0) a_first = true;                    // balance +1: side 0 then side 1
                else if (r < 0) a_first = false;
                else a_first = gain[A[a0 + k]] >= gain[B[b0 + k]];
                const bool me_first = (s == 0) == a_first;
                pos = (uint64_t)p0 + 2ull * k + (me_first ? 0 : 1);
            } else {
                pos = (uint64_t)p0 + 2ull * m + (i - first - m);   // tail of the longer list
            }
            order[pos] = u;
            rank[u] = (uint32_t)pos;
            atomicOr(listed + (u >> 5), 1u << (u & 31u));
            side[pos] = (uint8_t)s;
        }
    }
}

// Sequential gain of the i-th move (unit weights, 32-bit sums as above).  A
// second bitmap says which vertices are listed, so ranks are read of those
// alone.
template <int G, bool SHARED>
__global__ void __launch_bounds__(1024) k_fm_seqgain(FmGraph a, uint32_t k, const uint32_t *__restrict__ listed,
                                                     const uint32_t *__restrict__ order,
                                                     const uint32_t *__restrict__ rank, long long *__restrict__ gseq) {
    extern __shared__ uint32_t s_bits[];
    __shared__ int s_sum;
    const uint32_t words = bit_words(a.n);
    if (SHARED) {
        bits_load(a.bits, words, s_bits);
        bits_load(listed, words, s_bits + words);
    }
    const uint32_t *bits = SHARED ? (const uint32_t *)s_bits : a.bits;
    const uint32_t *lst = SHARED ? (const uint32_t *)(s_bits + words) : listed;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    // an entry counts +1: across xor moved before
    auto term = [&](uint32_t v, uint32_t pu, uint32_t i) -> int {
        const bool across = bit_of(bits, v) != pu;
        const bool moved = bit_of(lst, v) && __ldg(rank + v) < i;
        return across != moved;
    };
    const uint32_t nl = *a.nlong;
    for (uint32_t r = blockIdx.x; r < nl; r += gridDim.x) {
        const uint32_t u = __ldg(a.longs + r);
        if (!bit_of(lst, u)) continue;   // uniform in the block
        const uint32_t i = __ldg(rank + u), b = __ldg(a.rp + u), e = __ldg(a.rp + u + 1), pu = bit_of(bits, u);
        int plus = 0;
#pragma unroll 4
        for (uint64_t j = (uint64_t)b + threadIdx.x; j < e; j += 1024) plus += term(__ldg(a.col + j), pu, i);
        plus = __reduce_add_sync(0xFFFFFFFFu, plus);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, plus);
        __syncthreads();
        if (threadIdx.x == 0) {
            gseq[i] = 2 * s_sum - (int)(e - b);
            s_sum = 0;
        }
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & (G - 1);
    const uint64_t ng = ((uint64_t)gridDim.x * blockDim.x) / G;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; i < k; i += ng) {
        const uint32_t u = __ldg(order + i);
        const uint32_t b = __ldg(a.rp + u), e = __ldg(a.rp + u + 1);
        if (e - b > kLongRow) continue;   // uniform in the row's group
        const uint32_t pu = bit_of(bits, u);
        int plus = 0;
        for (uint32_t j0 = b + lane; j0 < e; j0 += 4 * G) {
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = j0 + q * G < e ? __ldg(a.col + j0 + q * G) : 0xFFFFFFFFu;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (v[q] != 0xFFFFFFFFu) plus += term(v[q], pu, (uint32_t)i);
        }
        plus = group_sum<G>(plus);
        if (lane == 0) gseq[i] = 2 * plus - (int)(e - b);
    }
}

// best prefix: one contiguous chunk per block, chunk sums, then a scan per
// chunk evaluating every k; key = cut << 32 | ~k, minimised (least cut,
// then the largest k)
struct FmBestArgs {
    uint32_t k;
    const long long *gseq;
    const uint8_t *side;
    long long cut0, bal0, target;
    long long *chunk_g, *chunk_b;   // [gridDim]
    unsigned long long *best;
};

__global__ void __launch_bounds__(256) k_fm_best(FmBestArgs a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ uint64_t sm[33];
    const uint32_t chunk = (a.k + gridDim.x - 1) / gridDim.x;
    const uint64_t c0 = (uint64_t)blockIdx.x * chunk;
    const uint64_t c1 = c0 + chunk < a.k ? c0 + chunk : a.k;
    long long sg = 0, sb = 0;
    for (uint64_t i = c0 + threadIdx.x; i < c1; i += blockDim.x) {
        sg += a.gseq[i];
        sb += a.side[i] == 0 ? -2 : 2;
    }
    uint64_t t1, t2;
    block_scan_u64((uint64_t)sg, sm, &t1);
    block_scan_u64((uint64_t)sb, sm, &t2);
    if (threadIdx.x == 0) {
        a.chunk_g[blockIdx.x] = (long long)t1;
        a.chunk_b[blockIdx.x] = (long long)t2;
    }
    grid.sync();
    long long base_g = 0, base_b = 0;
    for (uint32_t b = 0; b < blockIdx.x; b++) {
        base_g += a.chunk_g[b];
        base_b += a.chunk_b[b];
    }
    unsigned long long best = ~0ull;
    for (uint64_t s0 = c0; s0 < c1; s0 += blockDim.x) {
        const uint64_t i = s0 + threadIdx.x;
        const long long g = i < c1 ? a.gseq[i] : 0;
        const long long sbv = i < c1 ? (a.side[i] == 0 ? -2 : 2) : 0;
        uint64_t tg, tb;
        const long long ig = (long long)block_scan_u64((uint64_t)g, sm, &tg);
        const long long ib = (long long)block_scan_u64((uint64_t)sbv, sm, &tb);
        if (i < c1) {
            const long long cut = a.cut0 - (base_g + ig);
            long long bal = a.bal0 + base_b + ib;
            bal = bal < 0 ? -bal : bal;
            if (bal <= a.target) {
                const unsigned long long key = ((unsigned long long)cut << 32) | (0xFFFFFFFFu - (uint32_t)(i + 1));
                best = key < best ? key : best;
            }
        }
        base_g += (long long)tg;
        base_b += (long long)tb;
    }
    // block minimum, one atomic
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xFFFFFFFFu, best, o);
        best = x < best ? x : best;
    }
    if ((threadIdx.x & 31) == 0 && best != ~0ull) atomicMin(a.best, best);
}

__global__ void k_fm_apply(uint32_t k, const uint32_t *__restrict__ order, uint32_t *__restrict__ part,
                           uint32_t *__restrict__ bits) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += stride) {
        const uint32_t u = order[i];
        part[u] ^= 1u;
        atomicXor(bits + (u >> 5), 1u << (u & 31u));
    }
}

static uint32_t fm_grid(Context &C, uint64_t items) {
    uint64_t g = (items + 255) / 256;
    const uint64_t cap = (uint64_t)C.num_sms * 16;
    if (g > cap) g = cap;
    return g ? (uint32_t)g : 1u;
}

template <typename W>
static int fm_impl(Context &C, const Level &L, const W *w, uint32_t *part, uint32_t max_passes, uint64_t *cut_out,
                   uint32_t *passes_out, uint64_t *moves_out) {
    const uint32_t n = L.n;
    long long *gain, *gseq, *chunk_g, *chunk_b;
    uint8_t *side;
    uint32_t *flag, *pos, *idx, *sorted, *order, *rank, *hist = nullptr, *off = nullptr;
    unsigned long long *sums, *best;
    SGPB_TRY(dalloc_t(C, &gain, n));
    SGPB_TRY(dalloc_t(C, &gseq, n));
    SGPB_TRY(dalloc_t(C, &flag, 2 * (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &pos, 2 * (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &side, n));
    SGPB_TRY(dalloc_t(C, &idx, n));
    // once the candidates are listed, flags and positions have been read
    sorted = pos;
    order = flag;
    rank = flag + n;
    SGPB_TRY(dalloc_t(C, &sums, 4));
    SGPB_TRY(dalloc_t(C, &best, 1));
    size_t hist_room = 0;   // entries of hist and off
    uint64_t joint = kFmJoint;
    if (const char *e = getenv("SGPB_FM_JOINT"))   // another bound (0: always a side at a time)
        if (*e) joint = strtoull(e, nullptr, 10);
    // len candidates (the first na are side 0's) of src in order into dst
    auto sort = [&](uint32_t len, uint32_t na, const uint32_t *src, uint32_t *dst, int keys) -> int {
        if (!len) return SGP_B200_OK;
        const uint32_t nt = cdiv(len, kFmTile);
        const uint64_t cells = (uint64_t)keys * nt;
        if (cells > 0xFFFFFFFFull) {
            set_error("FM: %u candidates of one side", len);
            return SGP_B200_ERR_TOO_LARGE;
        }
        if (cells > hist_room) {
            SGPB_TRY(dalloc_t(C, &hist, cells + 1));
            SGPB_TRY(dalloc_t(C, &off, cells + 1));
            hist_room = cells;
        }
        k_fm_hist<<<nt, kFmTile, 0, C.stream>>>(len, na, src, gain, nt, keys, hist);
        SGPB_TRY(scan_u32(C, hist, off, (uint32_t)cells, nullptr));
        k_fm_place<<<nt, kFmTile, 0, C.stream>>>(len, na, src, gain, nt, keys, off, dst);
        C.kernel_launches += 2;
        return SGP_B200_OK;
    };
    int per_sm = 0;
    SGPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fm_best, 256, 0));
    if (per_sm < 1) {
        set_error("FM best-prefix kernel does not fit on an SM");
        return SGP_B200_ERR_DEVICE;
    }
    const uint32_t bgrid_max = (uint32_t)per_sm * C.num_sms;
    SGPB_TRY(dalloc_t(C, &chunk_g, bgrid_max));
    SGPB_TRY(dalloc_t(C, &chunk_b, bgrid_max));
    const double avg = n ? (double)L.m / n : 0;
    // parts and listed vertices as bitmaps, the long rows' list
    const uint32_t words = bit_words(n);
    uint32_t *bits, *listed, *longs, *nlong;
    SGPB_TRY(dalloc_t(C, &bits, words));
    SGPB_TRY(dalloc_t(C, &listed, words));
    SGPB_TRY(dalloc_t(C, &longs, n));
    SGPB_TRY(dalloc_t(C, &nlong, 1));
    SGPB_TRY(dzero(C, nlong, 4));
    SGPB_TRY(part_bits(C, n, part, bits));
    SGPB_TRY(long_rows(C, n, L.rp, longs, nlong));
    const FmGraph fg{n, L.rp, L.col, bits, longs, nlong};
    // blocks of 1024 threads: two an SM while their bitmaps fit
    auto row_grid = [&](uint64_t threads, uint32_t smem_words) -> uint32_t {
        const uint32_t cap = (uint32_t)C.num_sms * (smem_words <= kBitsMaxWords / 2 ? 2u : 1u);
        const uint64_t g = (threads + 1023) / 1024;
        return g > cap ? cap : g ? (uint32_t)g : 1u;
    };
    const bool sh1 = words <= kBitsMaxWords, sh2 = 2 * words <= kBitsMaxWords;
    auto gain_pass = [&](auto gt) -> int {
        constexpr int G = decltype(gt)::value;
        const uint32_t g = row_grid((uint64_t)n * G, sh1 ? words : 0);
        if (sh1) {
            SGPB_CUDA(cudaFuncSetAttribute(k_fm_gain<G, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(kBitsMaxWords * 4)));
            k_fm_gain<G, true><<<g, 1024, (size_t)words * 4, C.stream>>>(fg, gain, flag, sums);
        } else {
            k_fm_gain<G, false><<<g, 1024, 0, C.stream>>>(fg, gain, flag, sums);
        }
        return SGP_B200_OK;
    };
    auto seq_pass = [&](auto gt, uint32_t k) -> int {
        constexpr int G = decltype(gt)::value;
        const uint32_t g = row_grid((uint64_t)k * G, sh2 ? 2 * words : 0);
        if (sh2) {
            SGPB_CUDA(cudaFuncSetAttribute(k_fm_seqgain<G, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(kBitsMaxWords * 4)));
            k_fm_seqgain<G, true><<<g, 1024, (size_t)words * 8, C.stream>>>(fg, k, listed, order, rank, gseq);
        } else {
            k_fm_seqgain<G, false><<<g, 1024, 0, C.stream>>>(fg, k, listed, order, rank, gseq);
        }
        return SGP_B200_OK;
    };
    // lanes for about a trip of four entries each a row
    typedef std::integral_constant<int, 2> G2;
    typedef std::integral_constant<int, 8> G8;
    typedef std::integral_constant<int, 32> G32;
    uint64_t moves = 0;
    uint32_t pass = 0;
    for (; pass < max_passes; pass++) {
        SGPB_TRY(dzero(C, sums, 4 * sizeof(unsigned long long)));
        SGPB_TRY(avg <= 10 ? gain_pass(G2()) : avg <= 100 ? gain_pass(G8()) : gain_pass(G32()));
        uint64_t s[4];
        SGPB_TRY(read_u64(C, (const uint64_t *)sums, s, 4));
        const long long cut0 = (long long)(s[0] / 2), bal0 = (long long)s[1];
        if (pass == 0 && cut_out) *cut_out = (uint64_t)cut0;
        const uint32_t na = (uint32_t)s[2], nb = (uint32_t)s[3], k = na + nb;
        C.kernel_launches += 1;
        if (k == 0) break;
        // both sides' candidates in id order, sorted by descending clamped gain
        if (n < 0x80000000u) {
            SGPB_TRY(scan_u32(C, flag, pos, 2 * n, nullptr));
            k_fm_list<<<cdiv(2 * (uint64_t)n, 256), 256, 0, C.stream>>>(2 * n, flag, pos, n, idx);
        } else {   // one side at a time: 2n does not fit 32 bits
            for (int sd = 0; sd < 2; sd++) {
                SGPB_TRY(scan_u32(C, flag + (size_t)sd * n, pos, n, nullptr));
                k_fm_list<<<cdiv(n, 256), 256, 0, C.stream>>>(n, flag + (size_t)sd * n, pos, n, idx + (sd ? na : 0));
            }
        }
        C.kernel_launches += 1;
        if (k <= joint) {
            SGPB_TRY(sort(k, na, idx, sorted, kFmKeys));
        } else {
            SGPB_TRY(sort(na, na, idx, sorted, kFmBuckets));
            SGPB_TRY(sort(nb, nb, idx + na, sorted + na, kFmBuckets));
        }
        const uint32_t *sa = sorted, *sb = sorted + na;
        const unsigned long long key0 = ((unsigned long long)cut0 << 32) | 0xFFFFFFFFull;
        SGPB_TRY(dzero(C, listed, sizeof(uint32_t) * words));   // ranks are read of listed vertices alone
        k_fm_interleave<<<fm_grid(C, na > nb ? na : nb), 256, 0, C.stream>>>(na, nb, sa, sb, gain, bal0, order, rank,
                                                                             listed, side, key0, best);
        SGPB_TRY(avg <= 10 ? seq_pass(G2(), k) : avg <= 100 ? seq_pass(G8(), k) : seq_pass(G32(), k));
        FmBestArgs ba;
        ba.k = k;
        ba.gseq = gseq;
        ba.side = side;
        ba.cut0 = cut0;
        ba.bal0 = bal0;
        const long long ab = bal0 < 0 ? -bal0 : bal0;
        ba.target = ab / 10 > 20 ? ab / 10 : 20;
        ba.chunk_g = chunk_g;
        ba.chunk_b = chunk_b;
        ba.best = best;
        uint32_t bg = cdiv(k, 1024);
        if (bg > bgrid_max) bg = bgrid_max;
        if (bg < 1) bg = 1;
        void *args[] = {&ba};
        SGPB_CUDA(cudaLaunchCooperativeKernel((const void *)k_fm_best, dim3(bg), dim3(256), args, 0, C.stream));
        C.kernel_launches += 3;
        uint64_t bk = 0;
        SGPB_TRY(read_u64(C, (const uint64_t *)best, &bk));
        const uint32_t kstar = 0xFFFFFFFFu - (uint32_t)(bk & 0xFFFFFFFFu);
        const long long best_cut = (long long)(bk >> 32);
        if (kstar == 0 || best_cut == cut0) break;
        k_fm_apply<<<fm_grid(C, kstar), 256, 0, C.stream>>>(kstar, order, part, bits);
        C.kernel_launches++;
        SGPB_CUDA(cudaGetLastError());
        moves += kstar;
        if (cut_out) *cut_out = (uint64_t)best_cut;
    }
    SGPB_CUDA(cudaGetLastError());
    if (passes_out) *passes_out = pass;
    if (moves_out) *moves_out = moves;
    return SGP_B200_OK;
}

// On the finest level, whose edges all weigh 1 in the reference (its loader
// sets every value to 1), so the cut is the edge count the split reports.
int fm_refine_level(Context &C, const Level &L, uint32_t *part, uint32_t max_passes, uint64_t *cut_out,
                    uint32_t *passes_out, uint64_t *moves_out) {
    if (L.n == 0 || max_passes == 0) {
        if (passes_out) *passes_out = 0;
        if (moves_out) *moves_out = 0;
        return SGP_B200_OK;
    }
    return fm_impl<uint32_t>(C, L, nullptr, part, max_passes, cut_out, passes_out, moves_out);
}

__global__ void k_count_zero(uint32_t n, const uint32_t *__restrict__ part, uint32_t *__restrict__ out) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t z = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) z += part[i] == 0;
    z = warp_sum(z);
    if (lane == 0 && z) atomicAdd(out, z);
}

int count_part0(Context &C, const uint32_t *part, uint32_t n, uint32_t *out) {
    uint32_t *d;
    SGPB_TRY(dalloc_t(C, &d, 1));
    SGPB_TRY(dzero(C, d, 4));
    k_count_zero<<<fm_grid(C, n), 256, 0, C.stream>>>(n, part, d);
    C.kernel_launches++;
    SGPB_CUDA(cudaGetLastError());
    return read_u32(C, d, out);
}

}  // namespace sgpb
