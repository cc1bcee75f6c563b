// split.cu -- median split of the Fiedler vector and its edge cut.
//
// Reference: cmg/sgpar.h:1969-2071 (sgp_compute_partition, local search off):
// sort (ev, u) ascending, ties by u; the first n - imbr vertices form part 0,
// the rest part 1; vertices at sorted positions [imbl, imbr) move to part 0
// while that does not raise the cut; edge cut = directed cross entries / 2.
//
// The reference sorts all n pairs on the host.  Only the order statistic at
// position imbl matters for the split, so this is a radix *select* over the 64
// key bits of the order-preserving image of the double, then the 32 index
// bits, in one cooperative kernel: 11 bits a pass, each pass a histogram and a
// grid barrier, until at most kSelSmall candidates are left, which every
// block ranks for itself.  part[i] = ((key_i, i) < threshold) ? 0 : 1, also as
// a bitmap.  A pass over the CSR then counts the cut from the bitmap in
// shared memory, and the single sweep vertex of an odd n
// (perc_imbalance_allowed = 0, the value the reference's driver passes,
// sgpar.cpp:55) is decided on the device.
//
// What bounds it: the select is a chain of grid barriers (three or four where
// the 12 digit passes of 8 bits took 13), the cut the row lookups of short
// rows and the destination stream.  Erdos-Renyi, 1M vertices, 8M entries: 380
// -> 80 us.
#include <mutex>

#include <cooperative_groups.h>

#include "bits.cuh"
#include "common.cuh"
#include "internal.h"

namespace sgpb {

constexpr int kSplitThreads = 512;

constexpr int kSelBits = 11, kSelBins = 1 << kSelBits;
constexpr uint32_t kSelSmall = 1024;       // candidates ranked directly

struct SplitArgs {
    uint32_t n;
    const uint32_t *rp;
    const uint32_t *col;
    const double *evec;
    uint32_t k;            // imbl: sorted position of the threshold element
    uint32_t sweep;        // 1 when position k is also the sweep vertex (imbr - imbl == 1)
    uint32_t *hist;        // [3][kSelBins], then the candidate and the long-row counter: all zero at launch
    unsigned long long *cand;       // [2 * kSelSmall] (key, index) of the last candidates
    uint32_t *bits;        // [bit_words(n)] part 1
    uint32_t *longs;       // rows of more than kLongRow entries, in any order
    uint32_t *part;
    unsigned long long *out;        // [0] edgecut [1] part0 size [2] threshold index [3] directed cross entries
    double gap;                     // >= 0: out[4..7] too, see below
};
// The certificate of a split (gap >= 0): out[4] largest key below the
// threshold's, out[5] least key of the vertices behind the threshold, out[6]
// the threshold's key, out[7] whether a vertex on the other side of a decision
// lies within gap of the threshold.
constexpr size_t kSplitOutWords = 8;
constexpr size_t kSplitHistWords = 3 * kSelBins + 2;

__device__ __forceinline__ unsigned long long order_key(double x) {
    if (x == 0.0) x = 0.0;   // -0.0 == +0.0 in the reference's comparator
    unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ double key_value(unsigned long long k) {
    return __longlong_as_double((long long)((k >> 63) ? k & ~(1ull << 63) : ~k));
}

__global__ void __launch_bounds__(kSplitThreads) k_split(SplitArgs a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ uint32_t sh[kSelBins];
    __shared__ uint64_t sm[64];
    __shared__ unsigned long long s_key[kSelSmall];
    __shared__ uint32_t s_idx[kSelSmall];
    __shared__ uint32_t s_sel[3];
    const uint32_t n = a.n;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    uint32_t *ncand = a.hist + 3 * kSelBins, *nlong = ncand + 1;
    if (a.gap >= 0 && tid == 0) {   // next used behind a grid barrier
        a.out[4] = 0;
        a.out[5] = ~0ull;
    }
    // select: prefix over (key:64, index:32), digits MSB first: the key in five
    // of 11 bits and one of 9, the index in two of 11 and one of 10
    unsigned long long kpre = 0;   // selected key bits so far
    uint32_t ipre = 0;             // selected index bits so far
    uint32_t rank = a.k;           // rank among candidates matching the prefix
    for (int pass = 0; pass < 9; pass++) {
        uint32_t *h = a.hist + (pass % 3) * kSelBins;
        // Clear the buffer of the next pass.  It was last read after the barrier
        // of pass - 2, which every block has passed; it is next written after the
        // barrier of this pass.
        if (blockIdx.x == 0 && pass > 0)
            for (int t = threadIdx.x; t < kSelBins; t += blockDim.x) a.hist[((pass + 1) % 3) * kSelBins + t] = 0;
        for (int t = threadIdx.x; t < kSelBins; t += blockDim.x) sh[t] = 0;
        __syncthreads();
        const bool by_key = pass < 6;
        const int shift = by_key ? (pass < 5 ? 53 - 11 * pass : 0) : (pass < 8 ? 21 - 11 * (pass - 6) : 0);
        const uint32_t width = by_key ? (pass < 5 ? 11u : 9u) : (pass < 8 ? 11u : 10u), mask = (1u << width) - 1u;
        for (uint64_t i = tid; i < n; i += nth) {
            const unsigned long long key = order_key(a.evec[i]);
            uint32_t digit;
            if (by_key) {
                // candidates: key bits above the current digit equal the prefix
                if (pass && (key >> (shift + width)) != (kpre >> (shift + width))) continue;
                digit = (uint32_t)(key >> shift) & mask;
            } else {
                if (key != kpre) continue;
                if (pass > 6 && ((uint32_t)i >> (shift + width)) != (ipre >> (shift + width))) continue;
                digit = ((uint32_t)i >> shift) & mask;
            }
            atomicAdd(&sh[digit], 1u);
        }
        if (pass == 0)   // beside the first pass: the rows the cut gives to whole blocks
            for (uint64_t i = tid; i < n; i += nth)
                if (a.rp[i + 1] - a.rp[i] > kLongRow) a.longs[atomicAdd(nlong, 1u)] = (uint32_t)i;
        __syncthreads();
        for (int t = threadIdx.x; t < kSelBins; t += blockDim.x)
            if (sh[t]) atomicAdd(&h[t], sh[t]);
        grid.sync();
        // every block picks the same digit from the global histogram
        {
            constexpr int per = kSelBins / kSplitThreads;
            uint32_t c[per];
            uint64_t sum = 0, tot;
#pragma unroll
            for (int q = 0; q < per; q++) {
                c[q] = __ldcg(h + threadIdx.x * per + q);
                sum += c[q];
            }
            uint64_t acc = block_scan_u64(sum, sm, &tot) - sum;
#pragma unroll
            for (int q = 0; q < per; q++) {
                if (rank >= acc && rank < acc + c[q]) {
                    s_sel[0] = threadIdx.x * per + q;
                    s_sel[1] = rank - (uint32_t)acc;
                    s_sel[2] = c[q];
                }
                acc += c[q];
            }
        }
        __syncthreads();
        const uint32_t d = s_sel[0], left = s_sel[2];
        rank = s_sel[1];
        if (by_key) kpre |= (unsigned long long)d << shift;
        else ipre |= d << shift;
        __syncthreads();
        if (pass == 8) break;
        if (left > kSelSmall) continue;
        // few enough: list them, and every block ranks the list
        for (uint64_t i = tid; i < n; i += nth) {
            const unsigned long long key = order_key(a.evec[i]);
            const bool in = by_key ? (key >> shift) == (kpre >> shift)
                                   : key == kpre && ((uint32_t)i >> shift) == (ipre >> shift);
            if (in) {
                const uint32_t q = atomicAdd(ncand, 1u);
                a.cand[2 * q] = key;
                a.cand[2 * q + 1] = i;
            }
        }
        grid.sync();
        for (uint32_t q = threadIdx.x; q < left; q += blockDim.x) {
            s_key[q] = __ldcg(a.cand + 2 * q);
            s_idx[q] = (uint32_t)__ldcg(a.cand + 2 * q + 1);
        }
        __syncthreads();
        for (uint32_t q = threadIdx.x; q < left; q += blockDim.x) {
            const unsigned long long key = s_key[q];
            const uint32_t idx = s_idx[q];
            uint32_t before = 0;
            for (uint32_t t = 0; t < left; t++) before += s_key[t] < key || (s_key[t] == key && s_idx[t] < idx);
            if (before == rank) {   // one entry of the list: no two are equal
                sm[40] = key;
                s_sel[0] = idx;
            }
        }
        __syncthreads();
        kpre = sm[40];
        ipre = s_sel[0];
        break;
    }
    // assign parts; a.k elements precede the threshold
    unsigned long long lo = 0, hi = ~0ull;
    for (uint64_t i0 = tid & ~31ull; i0 < n; i0 += nth) {
        const uint64_t i = i0 + (threadIdx.x & 31);
        bool less = true;
        if (i < n) {
            const unsigned long long key = order_key(a.evec[i]);
            less = key < kpre || (key == kpre && (uint32_t)i < ipre);
            a.part[i] = less ? 0u : 1u;
            if (less) lo = key > lo ? key : lo;
            else if ((uint32_t)i != ipre) hi = key < hi ? key : hi;
        }
        const unsigned b = __ballot_sync(0xFFFFFFFFu, !less);
        if ((threadIdx.x & 31) == 0) a.bits[i0 >> 5] = b;
    }
    if (tid == 0) {
        a.out[1] = a.k;
        a.out[2] = ipre;
        a.out[3] = 0;
    }
    if (a.gap >= 0) {
        for (int o = 16; o; o >>= 1) {
            const unsigned long long l = __shfl_xor_sync(0xFFFFFFFFu, lo, o), h = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
            lo = l > lo ? l : lo;
            hi = h < hi ? h : hi;
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMax(a.out + 4, lo);
            atomicMin(a.out + 5, hi);
        }
        if (tid == 0) a.out[6] = kpre;
    }
}

// the bitmap of a part array
__global__ void k_part_bits(uint32_t n, const uint32_t *__restrict__ part, uint32_t *__restrict__ bits) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned b = __ballot_sync(0xFFFFFFFFu, i < n && part[i] != 0);
    if ((threadIdx.x & 31) == 0 && i < n) bits[i >> 5] = b;
}

__global__ void k_long_rows(uint32_t n, const uint32_t *__restrict__ rp, uint32_t *__restrict__ longs,
                            uint32_t *__restrict__ nlong) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && rp[i + 1] - rp[i] > kLongRow) longs[atomicAdd(nlong, 1u)] = i;
}

// Cross entries of rows of at most kLongRow entries, G lanes a row and four
// entries a lane in flight.
template <int G>
__device__ __forceinline__ uint64_t cut_rows(uint32_t n, const uint32_t *__restrict__ rp,
                                             const uint32_t *__restrict__ col, const uint32_t *bits) {
    const uint32_t lane = threadIdx.x & (G - 1);
    const uint64_t ng = ((uint64_t)gridDim.x * blockDim.x) / G;
    uint64_t cut = 0;
    for (uint64_t u = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; u < n; u += ng) {
        const uint32_t b = __ldg(rp + u), e = __ldg(rp + u + 1);
        if (e - b > kLongRow) continue;
        const uint32_t pu = bit_of(bits, (uint32_t)u);
        uint32_t c = 0;
        for (uint32_t j0 = b + lane; j0 < e; j0 += 4 * G) {
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = j0 + q * G < e ? __ldg(col + j0 + q * G) : (uint32_t)u;
#pragma unroll
            for (int q = 0; q < 4; q++) c += bit_of(bits, v[q]) != pu;
        }
        cut += c;
    }
    return cut;
}

// Directed cross entries of a bisection given as a bitmap, added to *out.
// SHARED: the bitmap in the block's shared memory.
template <bool SHARED>
__global__ void __launch_bounds__(1024) k_cut_bits(uint32_t n, const uint32_t *__restrict__ rp,
                                                   const uint32_t *__restrict__ col, const uint32_t *__restrict__ gbits,
                                                   const uint32_t *__restrict__ longs,
                                                   const uint32_t *__restrict__ nlong, unsigned long long *out) {
    extern __shared__ uint32_t s_bits[];
    __shared__ uint64_t sm[33];
    const uint32_t m = __ldg(rp + n);
    if (SHARED) {
        bits_load(gbits, bit_words(n), s_bits);
        __syncthreads();
    }
    const uint32_t *bits = SHARED ? (const uint32_t *)s_bits : gbits;
    uint64_t cut;
    // a row's latency is what short rows cost: lanes for about a trip a row
    if (m <= 10ull * n) cut = cut_rows<2>(n, rp, col, bits);
    else if (m <= 20ull * n) cut = cut_rows<4>(n, rp, col, bits);
    else if (m <= 100ull * n) cut = cut_rows<8>(n, rp, col, bits);
    else cut = cut_rows<32>(n, rp, col, bits);
    // long rows, a block each
    const uint32_t nl = *nlong;
    for (uint32_t r = blockIdx.x; r < nl; r += gridDim.x) {
        const uint32_t u = __ldg(longs + r), b = __ldg(rp + u), e = __ldg(rp + u + 1);
        const uint32_t pu = bit_of(bits, u);
#pragma unroll 4
        for (uint64_t j = (uint64_t)b + threadIdx.x; j < e; j += 1024) cut += bit_of(bits, __ldg(col + j)) != pu;
    }
    uint64_t tot;
    block_scan_u64(cut, sm, &tot);
    if (threadIdx.x == 0 && tot) atomicAdd(out, (unsigned long long)tot);
}

// sweep of the vertex at position k (sgpar.h:2046-2071) and the results
__global__ void __launch_bounds__(kSplitThreads) k_split_sweep(SplitArgs a) {
    __shared__ uint64_t sm[64];
    long long upd = 0;
    const uint32_t u = (uint32_t)a.out[2];
    if (a.sweep) {
        long long c = 0;
        for (uint32_t j = a.rp[u] + threadIdx.x; j < a.rp[u + 1]; j += blockDim.x)
            c += (a.part[a.col[j]] == 1) ? 1 : -1;
        uint64_t uc = (uint64_t)(c + (1ll << 40));   // bias to keep the scan unsigned
        uint64_t tt;
        block_scan_u64(uc, sm, &tt);
        upd = (long long)tt - (long long)blockDim.x * (1ll << 40);
    }
    if (threadIdx.x == 0) {
        long long best = (long long)a.out[3];
        if (a.sweep) {
            const long long cur = best + 2 * upd;
            if (cur <= best) {
                a.part[u] = 0;
                best = cur;
                a.out[1]++;
            }
        }
        a.out[0] = (unsigned long long)(best / 2);
        if (a.gap >= 0) {
            // below the threshold: who is in part 0; behind it, too, where the
            // threshold's vertex is the sweep's
            const double t = key_value(a.out[6]);
            a.out[7] = (a.k > 0 && t - key_value(a.out[4]) <= a.gap) ||
                       (a.sweep && a.k + 1 < a.n && key_value(a.out[5]) - t <= a.gap);
        }
    }
}

static int launch_cut_bits(cudaStream_t s, int num_sms, uint32_t n, const uint32_t *rp, const uint32_t *col,
                           const uint32_t *bits, const uint32_t *longs, const uint32_t *nlong,
                           unsigned long long *out) {
    const uint32_t words = bit_words(n);
    const size_t bytes = (size_t)words * 4;
    // two blocks an SM while two bitmaps fit, of at least 256 rows each
    uint32_t g = (uint32_t)num_sms * (words <= kBitsMaxWords / 2 || words > kBitsMaxWords ? 2u : 1u);
    if (g > cdiv(n, 256)) g = cdiv(n, 256);
    if (words <= kBitsMaxWords) {
        SGPB_CUDA(cudaFuncSetAttribute(k_cut_bits<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(kBitsMaxWords * 4)));
        k_cut_bits<true><<<g, 1024, bytes, s>>>(n, rp, col, bits, longs, nlong, out);
    } else {
        k_cut_bits<false><<<g, 1024, 0, s>>>(n, rp, col, bits, longs, nlong, out);
    }
    SGPB_CUDA(cudaGetLastError());
    return SGP_B200_OK;
}

// the kernels of a split whose SplitArgs are complete and whose histogram
// words are zero
static int launch_split(cudaStream_t s, int num_sms, uint32_t grid, SplitArgs &a) {
    void *args[] = {&a};
    SGPB_CUDA(cudaLaunchCooperativeKernel((const void *)k_split, dim3(grid), dim3(kSplitThreads), args, 0, s));
    SGPB_TRY(launch_cut_bits(s, num_sms, a.n, a.rp, a.col, a.bits, a.longs, a.hist + 3 * kSelBins + 1, a.out + 3));
    k_split_sweep<<<1, kSplitThreads, 0, s>>>(a);
    SGPB_CUDA(cudaGetLastError());
    return SGP_B200_OK;
}

int split_level(Context &C, const Level &L, const double *evec, int perc_imbalance, uint32_t *part,
                uint64_t *edgecut, uint32_t *n_part0, bool *close) {
    const uint32_t n = L.n;
    if (close) *close = false;
    if (n == 0) { *edgecut = 0; if (n_part0) *n_part0 = 0; return SGP_B200_OK; }
    if (perc_imbalance != 0) {
        set_error("perc_imbalance_allowed must be 0 (the value sgpar.cpp passes); got %d", perc_imbalance);
        return SGP_B200_ERR_INVALID;
    }
    // sgpar.h:2009-2012
    long long max_part_size = (long long)ceil(n / 2.0);
    uint32_t imbr = (uint32_t)floor(max_part_size * (1.0 + perc_imbalance / 100.0));
    uint32_t imbl = n - imbr;
    SplitArgs a;
    a.n = n; a.rp = L.rp; a.col = L.col; a.evec = evec; a.part = part;
    // With imbl == n there is no threshold element (cannot happen for p = 0).
    a.k = imbl < n ? imbl : n - 1;
    a.sweep = (imbr > imbl) ? 1u : 0u;
    SGPB_TRY(dalloc_t(C, &a.hist, kSplitHistWords));
    SGPB_TRY(dzero(C, a.hist, kSplitHistWords * sizeof(uint32_t)));
    SGPB_TRY(dalloc_t(C, &a.cand, 2 * kSelSmall));
    SGPB_TRY(dalloc_t(C, &a.bits, bit_words(n)));
    SGPB_TRY(dalloc_t(C, &a.longs, n));
    SGPB_TRY(dalloc_t(C, &a.out, kSplitOutWords));
    a.gap = close ? kTieGap / sqrt((double)n) : -1.0;
    int per_sm = 0;
    SGPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)k_split, kSplitThreads, 0));
    if (per_sm < 1) { set_error("split kernel does not fit"); return SGP_B200_ERR_DEVICE; }
    if (per_sm > 2) per_sm = 2;
    uint64_t maxg = (uint64_t)per_sm * C.num_sms;
    uint64_t want = cdiv(n, kSplitThreads * 8ull);
    uint32_t grid = (uint32_t)(want < maxg ? want : maxg);
    if (grid < 1) grid = 1;
    SGPB_TRY(launch_split(C.stream, C.num_sms, grid, a));
    C.kernel_launches += 3;
    uint64_t out[kSplitOutWords];
    SGPB_TRY(read_u64(C, (const uint64_t *)a.out, out, close ? kSplitOutWords : 3));
    if (close) *close = out[7] != 0;
    *edgecut = out[0];
    if (n_part0) *n_part0 = (uint32_t)out[1];
    return SGP_B200_OK;
}

// --------------------------------------------------- split, no allocation --
// Scratch of sgp_b200_split_noalloc: the long-row list and the bitmap of
// SGP_B200_NOALLOC_MAX_N vertices, the last candidates, the digit histograms
// and the result words.  It is a file-scope device array, so every GPU that
// loads this library holds it (about 4 MiB) until the process exits, and every
// call on a device shares it.
constexpr uint32_t kNoAllocMaxBlocks = 1024;
constexpr size_t kNoAllocBitsOff = (size_t)SGP_B200_NOALLOC_MAX_N * sizeof(uint32_t);
constexpr size_t kNoAllocCandOff = kNoAllocBitsOff + (size_t)SGP_B200_NOALLOC_MAX_N / 8;
constexpr size_t kNoAllocOutOff = kNoAllocCandOff + 2 * (size_t)kSelSmall * sizeof(unsigned long long);
constexpr size_t kNoAllocHistOff = kNoAllocOutOff + 4 * sizeof(unsigned long long);
constexpr size_t kNoAllocBytes = kNoAllocHistOff + kSplitHistWords * sizeof(uint32_t);
static __device__ __align__(256) unsigned char g_split_scratch[kNoAllocBytes];

// Per-device set-up, done by the first call on that device: the host
// address of g_split_scratch is only a stand-in, so the device address comes
// from cudaGetSymbolAddress with the device current.  The address belongs to
// the context that loaded the module: after cudaDeviceReset (or any new
// context on the device) the cached one is stale, so the set-up is keyed by
// the current context's id and redone when that id changes.
struct NoAllocDevice {
    unsigned char *scratch = nullptr;
    int num_sms = 0;
    int per_sm = 0;
    unsigned long long ctx_id = 0;
    bool ready = false;
};
static std::mutex g_noalloc_mu;
static NoAllocDevice g_noalloc_dev[64];

// Unique id of the calling thread's current context (cuCtxGetCurrent and
// cuCtxGetId through the runtime's driver entry points, so the library does
// not link the driver library itself).  Every context ever created in the
// process gets a distinct id.
typedef int (*CtxGetCurrentFn)(void **ctx);
typedef int (*CtxGetIdFn)(void *ctx, unsigned long long *id);
static int current_ctx_id(int device, unsigned long long *id) {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = (CtxGetCurrentFn)f;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (CtxGetIdFn)f;
    });
    if (!get_current || !get_id) {
        set_error("the CUDA driver does not provide cuCtxGetCurrent / cuCtxGetId");
        return SGP_B200_ERR_DEVICE;
    }
    // makes the device's primary context current if no context is yet
    SGPB_CUDA(cudaSetDevice(device));
    void *ctx = nullptr;
    if (get_current(&ctx) != 0 || !ctx || get_id(ctx, id) != 0) {
        set_error("no current CUDA context on device %d", device);
        return SGP_B200_ERR_DEVICE;
    }
    return SGP_B200_OK;
}

static int noalloc_setup(int device, NoAllocDevice **out) {
    if (device < 0 || device >= 64) {
        set_error("device %d out of range for the no-allocation entry point", device);
        return SGP_B200_ERR_INVALID;
    }
    unsigned long long id = 0;
    SGPB_TRY(current_ctx_id(device, &id));
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoAllocDevice &d = g_noalloc_dev[device];
    if (!d.ready || d.ctx_id != id) {
        d.ready = false;
        void *p = nullptr;
        SGPB_CUDA(cudaGetSymbolAddress(&p, g_split_scratch));
        SGPB_CUDA(cudaDeviceGetAttribute(&d.num_sms, cudaDevAttrMultiProcessorCount, device));
        SGPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.per_sm, (const void *)k_split, kSplitThreads, 0));
        if (d.per_sm < 1) {
            set_error("split kernel does not fit on an SM");
            return SGP_B200_ERR_DEVICE;
        }
        d.scratch = (unsigned char *)p;
        d.ctx_id = id;
        d.ready = true;
    }
    *out = &d;
    return SGP_B200_OK;
}

// ------------------------------------------------------------- edge cut --
int part_bits(Context &C, uint32_t n, const uint32_t *part, uint32_t *bits) {
    k_part_bits<<<cdiv(n, 256), 256, 0, C.stream>>>(n, part, bits);
    C.kernel_launches++;
    SGPB_CUDA(cudaGetLastError());
    return SGP_B200_OK;
}

int long_rows(Context &C, uint32_t n, const uint32_t *rp, uint32_t *longs, uint32_t *nlong) {
    k_long_rows<<<cdiv(n, 256), 256, 0, C.stream>>>(n, rp, longs, nlong);
    C.kernel_launches++;
    SGPB_CUDA(cudaGetLastError());
    return SGP_B200_OK;
}

int edge_cut_device(Context &C, const Level &L, const uint32_t *part, uint64_t *edgecut) {
    unsigned long long *o;
    SGPB_TRY(dalloc_t(C, &o, 2));
    SGPB_TRY(dzero(C, o, 16));
    if (L.n) {
        uint32_t *bits, *longs, *nlong = (uint32_t *)(o + 1);
        SGPB_TRY(dalloc_t(C, &bits, bit_words(L.n)));
        SGPB_TRY(dalloc_t(C, &longs, L.n));
        SGPB_TRY(part_bits(C, L.n, part, bits));
        SGPB_TRY(long_rows(C, L.n, L.rp, longs, nlong));
        SGPB_TRY(launch_cut_bits(C.stream, C.num_sms, L.n, L.rp, L.col, bits, longs, nlong, o));
        C.kernel_launches++;
    }
    uint64_t h;
    SGPB_TRY(read_u64(C, (const uint64_t *)o, &h));
    *edgecut = h / 2;
    return SGP_B200_OK;
}

// --------------------------------------------------------- local search --
// sgpar.h:2080-2170: after the split, alternately flip the vertex of largest
// positive gain (cross minus same-side neighbours; first id on a tie) among
// ids [mid - n/3, mid) and then among [mid, mid + n/3), mid being the part-0
// size the split left; a missing second move undoes the first and ends the
// search, as does a missing first move or n/3 completed pairs.  The
// reference recomputes every candidate's gain per move (O(n m) in all); here
// the gains are kept incrementally -- a flip negates the vertex's own gain
// and moves each neighbour's by 2 -- and each half-step is a grid-wide
// argmax plus one row update in a single cooperative launch.
//
// Ordering: a flip of part[v] is deferred to the next phase (after a grid
// barrier), so no thread reads part[v] while it is written; the argmax
// phase reads gains only.  Four argmax slots rotate; the slot two
// half-steps ahead is cleared while the current one is read.  Gains and
// parts change between barriers on other SMs, so after the first phase
// they are read with ld.global.cg (L2), never from a possibly stale L1 line.
constexpr int kLSThreads = 512;

struct LSArgs {
    uint32_t n;
    const uint32_t *rp, *col;
    uint32_t *part;
    int *gain;
    uint32_t lo, mid, hi, max_swaps;
    unsigned long long *key;   // [4], zero on entry
    uint32_t *out;             // [0] swaps
};

namespace cgls = cooperative_groups;

__global__ void __launch_bounds__(kLSThreads) k_local_search(LSArgs a) {
    cgls::grid_group grid = cgls::this_grid();
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    __shared__ unsigned long long wmax[kLSThreads / 32];
    // gains, a warp per row
    for (uint64_t u = tid >> 5; u < a.n; u += nthreads >> 5) {
        const uint32_t pu = a.part[u];
        int x = 0;
        for (uint32_t j = a.rp[u] + lane; j < a.rp[u + 1]; j += 32) x += a.part[__ldg(a.col + j)] != pu ? 1 : -1;
        x = warp_sum(x);
        if (lane == 0) a.gain[u] = x;
    }
    grid.sync();
    uint32_t pending = 0xFFFFFFFFu, first = 0xFFFFFFFFu, swaps = 0, slot = 0;
    for (int half = 0;; half ^= 1) {
        if (half == 0 && swaps >= a.max_swaps) break;
        // ---- argmax of (gain, -id) over this half's range, gains > 0 only
        if (leader && pending != 0xFFFFFFFFu) a.part[pending] = __ldcg(a.part + pending) ^ 1u;
        pending = 0xFFFFFFFFu;
        const uint32_t b = half == 0 ? a.lo : a.mid, e = half == 0 ? a.mid : a.hi;
        unsigned long long best = 0;
        for (uint64_t i = b + tid; i < e; i += nthreads) {
            const int g = __ldcg(a.gain + i);
            if (g > 0) {
                const unsigned long long k = ((unsigned long long)(uint32_t)g << 32) | (0xFFFFFFFFu - (uint32_t)i);
                best = k > best ? k : best;
            }
        }
        best = warp_max(best);
        if (lane == 0) wmax[wid] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long m = 0;
            for (int w = 0; w < kLSThreads / 32; w++) m = wmax[w] > m ? wmax[w] : m;
            if (m) atomicMax(a.key + slot, m);
        }
        grid.sync();
        // ---- apply: flip the winner (deferred) and move its neighbours' gains
        const unsigned long long k = *(volatile unsigned long long *)(a.key + slot);
        if (leader) a.key[(slot + 2) & 3] = 0;
        slot = (slot + 1) & 3;
        uint32_t v;
        if (k == 0) {
            if (half == 0) break;   // no first move: done
            v = first;              // no second move: undo the first, then done
        } else {
            v = 0xFFFFFFFFu - (uint32_t)(k & 0xFFFFFFFFu);
        }
        const uint32_t old = __ldcg(a.part + v);
        for (uint64_t j = a.rp[v] + tid; j < a.rp[v + 1]; j += nthreads) {
            const uint32_t u = __ldg(a.col + j);
            // rows hold u once: no other writer of gain[u] in this phase
            a.gain[u] = __ldcg(a.gain + u) + (__ldcg(a.part + u) != old ? -2 : 2);
        }
        if (leader) a.gain[v] = -__ldcg(a.gain + v);
        pending = v;
        grid.sync();
        if (k == 0) break;          // the undo above ends the search
        if (half == 0) first = v;
        else swaps++;
    }
    grid.sync();
    if (leader) {
        if (pending != 0xFFFFFFFFu) a.part[pending] = __ldcg(a.part + pending) ^ 1u;
        a.out[0] = swaps;
    }
    grid.sync();
    // part-0 size after the search (the moves need not balance)
    uint32_t z = 0;
    for (uint64_t i = tid; i < a.n; i += nthreads) z += __ldcg(a.part + i) == 0;
    z = warp_sum(z);
    if (lane == 0 && z) atomicAdd(a.out + 1, z);
}

int local_search_level(Context &C, const Level &L, uint32_t *part, uint32_t mid, uint32_t *swaps_out,
                       uint32_t *part0_out) {
    const uint32_t n = L.n;
    if (n < 3) {
        if (swaps_out) *swaps_out = 0;
        if (part0_out) *part0_out = mid;
        return SGP_B200_OK;
    }
    LSArgs a;
    a.n = n;
    a.rp = L.rp;
    a.col = L.col;
    a.part = part;
    a.mid = mid;
    a.lo = mid > n / 3 ? mid - n / 3 : 0;
    a.hi = (uint64_t)mid + n / 3 < n ? mid + n / 3 : n;
    a.max_swaps = n / 3;
    SGPB_TRY(dalloc_t(C, &a.gain, n));
    SGPB_TRY(dalloc_t(C, &a.key, 4));
    SGPB_TRY(dalloc_t(C, &a.out, 2));
    SGPB_TRY(dzero(C, a.out, 2 * sizeof(uint32_t)));
    SGPB_TRY(dzero(C, a.key, 4 * sizeof(unsigned long long)));
    int per_sm = 0;
    SGPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_local_search, kLSThreads, 0));
    if (per_sm < 1) {
        set_error("local-search kernel does not fit on an SM");
        return SGP_B200_ERR_DEVICE;
    }
    // one block per SM at most: the per-move barriers cost less with fewer
    // blocks, and a range of n/3 gains is a light scan
    uint32_t grid = cdiv((uint64_t)n, 4096);
    if (grid > (uint32_t)C.num_sms) grid = C.num_sms;
    if (grid < 1) grid = 1;
    void *args[] = {&a};
    SGPB_CUDA(cudaLaunchCooperativeKernel((const void *)k_local_search, dim3(grid), dim3(kLSThreads), args, 0,
                                          C.stream));
    C.kernel_launches++;
    uint32_t o[2] = {0, 0};
    SGPB_TRY(read_u32(C, a.out, o, 2));
    if (swaps_out) *swaps_out = o[0];
    if (part0_out) *part0_out = o[1];
    return SGP_B200_OK;
}

// ------------------------------------------------- induced sub-graphs --
// sgpar.h:2666-2752: vertices of each part relabelled in ascending order,
// edges inside each part kept in row order.
__global__ void k_same_part_counts(uint32_t n, const uint32_t *rp, const uint32_t *col, const uint32_t *part,
                                   uint32_t *cnt0, uint32_t *cnt1, uint32_t *is0, uint32_t *is1) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t wid = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = wid; i < n; i += nw) {
        const uint32_t pi = part[i];
        uint32_t c = 0;
        for (uint32_t j = rp[i] + lane; j < rp[i + 1]; j += 32) c += (part[col[j]] == pi);
        c = warp_sum(c);
        if (lane == 0) {
            cnt0[i] = pi == 0 ? c : 0;
            cnt1[i] = pi == 0 ? 0 : c;
            is0[i] = pi == 0;
            is1[i] = pi != 0;
        }
    }
}

__global__ void k_fill_sub(uint32_t n, const uint32_t *rp, const uint32_t *col, const uint32_t *part,
                           const uint32_t *map0, const uint32_t *map1, const uint32_t *off0, const uint32_t *off1,
                           uint32_t *rp1, uint32_t *col1, uint32_t *rp2, uint32_t *col2) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t wid = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = wid; i < n; i += nw) {
        const uint32_t pi = part[i];
        uint32_t o = pi == 0 ? off0[i] : off1[i];
        uint32_t *dst = pi == 0 ? col1 : col2;
        if (lane == 0) {
            if (pi == 0) rp1[map0[i]] = o; else rp2[map1[i]] = o;
        }
        const uint32_t b = rp[i], e = rp[i + 1];
        for (uint32_t j0 = b; j0 < e; j0 += 32) {
            uint32_t j = j0 + lane;
            bool keep = false;
            uint32_t v = 0;
            if (j < e) { v = col[j]; keep = part[v] == pi; }
            unsigned m = __ballot_sync(0xFFFFFFFFu, keep);
            if (keep) dst[o + __popc(m & ((1u << lane) - 1u))] = pi == 0 ? map0[v] : map1[v];
            o += __popc(m);
        }
    }
}

int induced_subgraphs(Context &C, const Level &L, const uint32_t *part, Level *g1, Level *g2, uint32_t **map0_out,
                      uint32_t **map1_out) {
    const uint32_t n = L.n;
    uint32_t *cnt0, *cnt1, *is0, *is1, *off0, *off1, *map0, *map1;
    SGPB_TRY(dalloc_t(C, &cnt0, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &cnt1, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &is0, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &is1, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &off0, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &off1, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &map0, (size_t)n + 1));
    SGPB_TRY(dalloc_t(C, &map1, (size_t)n + 1));
    uint32_t g = n ? cdiv(n, 8) : 1;
    if (g > (uint32_t)C.num_sms * 8) g = C.num_sms * 8;
    if (n) k_same_part_counts<<<g, 256, 0, C.stream>>>(n, L.rp, L.col, part, cnt0, cnt1, is0, is1);
    SGPB_TRY(scan_u32(C, cnt0, off0, n, nullptr));
    SGPB_TRY(scan_u32(C, cnt1, off1, n, nullptr));
    SGPB_TRY(scan_u32(C, is0, map0, n, nullptr));
    SGPB_TRY(scan_u32(C, is1, map1, n, nullptr));
    uint32_t tots[2], nn[2];
    SGPB_TRY(read_u32(C, off0 + n, &tots[0]));
    SGPB_TRY(read_u32(C, off1 + n, &tots[1]));
    SGPB_TRY(read_u32(C, map0 + n, &nn[0]));
    SGPB_TRY(read_u32(C, map1 + n, &nn[1]));
    g1->n = nn[0]; g1->m = tots[0]; g1->wbytes = 0; g1->w = nullptr;
    g2->n = nn[1]; g2->m = tots[1]; g2->wbytes = 0; g2->w = nullptr;
    SGPB_TRY(dalloc_t(C, &g1->rp, (size_t)nn[0] + 1));
    SGPB_TRY(dalloc_t(C, &g2->rp, (size_t)nn[1] + 1));
    SGPB_TRY(dalloc_t(C, &g1->col, (size_t)tots[0] + 1));
    SGPB_TRY(dalloc_t(C, &g2->col, (size_t)tots[1] + 1));
    if (n)
        k_fill_sub<<<g, 256, 0, C.stream>>>(n, L.rp, L.col, part, map0, map1, off0, off1, g1->rp, g1->col, g2->rp,
                                            g2->col);
    SGPB_CUDA(cudaMemcpyAsync(g1->rp + nn[0], off0 + n, 4, cudaMemcpyDeviceToDevice, C.stream));
    SGPB_CUDA(cudaMemcpyAsync(g2->rp + nn[1], off1 + n, 4, cudaMemcpyDeviceToDevice, C.stream));
    C.kernel_launches += 2;
    SGPB_CUDA(cudaGetLastError());
    if (map0_out) *map0_out = map0;
    if (map1_out) *map1_out = map1;
    return SGP_B200_OK;
}

}  // namespace sgpb

using namespace sgpb;

// Median split + edge cut of a device eigenvector without any allocation: the
// scratch is g_split_scratch above.  Meant for callers that cannot allocate
// device memory at that point: a host application that owns every device
// allocation through its own pool, code running inside an out-of-memory
// handler, or a plug-in whose allocation calls are forbidden by its host.
// The first call on a device (and the first after the device's context
// changed, e.g. after cudaDeviceReset) fetches the scratch address (see
// noalloc_setup); make that first call before any stream capture.  The stream
// must belong to the current device.  Calls that overlap on the GPU
// (different streams, or graphs replayed concurrently) share the scratch and
// race; serialise them.
extern "C" int sgp_b200_split_noalloc(void *stream, uint32_t n, const uint32_t *row_ptr, const uint32_t *col,
                                      const double *evec, uint32_t *part, uint64_t *result) {
    // col may be NULL for a graph without edges, as for sgp_b200_split
    if (!row_ptr || !evec || !part || !result) {
        set_error("null argument");
        return SGP_B200_ERR_INVALID;
    }
    if (n == 0 || n > SGP_B200_NOALLOC_MAX_N) {
        set_error("sgp_b200_split_noalloc handles 1 .. %u vertices (its fixed scratch size); got %u",
                  (unsigned)SGP_B200_NOALLOC_MAX_N, n);
        return SGP_B200_ERR_TOO_LARGE;
    }
    int device = 0;
    SGPB_CUDA(cudaGetDevice(&device));
    cudaStream_t s = (cudaStream_t)stream;
    if (s) {
        int sdev = -1;
        SGPB_CUDA(cudaStreamGetDevice(s, &sdev));
        if (sdev != device) {
            set_error("sgp_b200_split_noalloc: the stream belongs to device %d but device %d is current; "
                      "make the stream's device current",
                      sdev, device);
            return SGP_B200_ERR_INVALID;
        }
    }
    NoAllocDevice *d = nullptr;
    SGPB_TRY(noalloc_setup(device, &d));
    SplitArgs a;
    a.n = n;
    a.rp = row_ptr;
    a.col = col;
    a.evec = evec;
    a.part = part;
    // sgpar.h:2009-2012 with perc_imbalance_allowed = 0
    const uint32_t imbr = (uint32_t)ceil(n / 2.0);
    const uint32_t imbl = n - imbr;
    a.k = imbl < n ? imbl : n - 1;
    a.sweep = imbr > imbl ? 1u : 0u;
    a.gap = -1.0;
    a.longs = reinterpret_cast<uint32_t *>(d->scratch);
    a.bits = reinterpret_cast<uint32_t *>(d->scratch + kNoAllocBitsOff);
    a.cand = reinterpret_cast<unsigned long long *>(d->scratch + kNoAllocCandOff);
    a.hist = reinterpret_cast<uint32_t *>(d->scratch + kNoAllocHistOff);
    a.out = reinterpret_cast<unsigned long long *>(d->scratch + kNoAllocOutOff);
    // the scratch keeps the previous call's contents: the histograms and
    // counters must start at zero; the rest is written before use
    SGPB_CUDA(cudaMemsetAsync(a.hist, 0, kSplitHistWords * sizeof(uint32_t), s));
    const int per_sm = d->per_sm > 2 ? 2 : d->per_sm;
    uint64_t grid = (uint64_t)per_sm * d->num_sms;
    const uint64_t want = cdiv(n, kSplitThreads * 8ull);
    if (want < grid) grid = want;
    if (grid > kNoAllocMaxBlocks) grid = kNoAllocMaxBlocks;
    if (grid < 1) grid = 1;
    SGPB_TRY(launch_split(s, d->num_sms, (uint32_t)grid, a));
    // result[0] = edge cut, result[1] = size of part 0 (device array)
    SGPB_CUDA(cudaMemcpyAsync(result, a.out, 2 * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s));
    SGPB_CUDA(cudaGetLastError());
    return SGP_B200_OK;
}
