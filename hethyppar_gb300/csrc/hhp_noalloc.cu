// hhp_noalloc.cu -- y = alpha*A*x + beta*y on caller-owned device CSR arrays, without allocating.
//
// For callers that cannot call cudaMalloc: code that must not trigger the implicit device-wide
// synchronisation of cudaMalloc/cudaFree in the middle of its stream work, or that runs under a
// memory budget owned by someone else (a host application or framework that pre-sizes and owns
// all device memory). The caller passes every input and output; the only scratch this path
// needs -- one carry (row, partial sum) per CTA for rows split between CTAs -- lives in a
// file-scope __device__ array of kMaxCarry entries that every GPU loading the library holds
// until the process exits.
//
// Work split (merge path): the rows' end offsets and the nonzeros form one merged list of
// m + nnz items; CTA c takes items [c*D, (c+1)*D), in tiles of at most 1664 items. Per tile the
// CTA stages the row ends, the values and the gathered x of its nonzeros in shared memory
// (coalesced loads); each thread walks up to 13 items, summing in CSR order with one FMA per
// nonzero, and leaves the sums of the rows that start and end inside its walk in shared memory;
// rows that cross threads are combined in a fixed order, the finished rows are stored as
// alpha*sum + beta*y in one dense pass, and a row still open at the end of a tile carries into the
// next. The row open at the end of the CTA's range goes to the CTA's carry slot, and a second
// kernel adds the carries of each row, in CTA order, to the row's y. Rows inside one thread's
// walk are summed exactly as hhp_spmv_dev sums them; rows split between threads or CTAs differ
// from it only in rounding.
//
// Set-up: the first call on a device resolves the array's device address with
// cudaGetSymbolAddress, with that device current, and remembers it; make that first call before
// any stream capture. All calls share the one array and it keeps the last call's contents. Nothing
// in it needs to start at zero: a call writes every slot of its CTAs (an unused slot is marked
// row -1) before its second kernel reads any. Calls that overlap on the GPU (on different streams,
// or from different host threads on one device) race on the array and give wrong results.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "hhp_device.cuh"
#include "hhp_internal.h"

namespace {

constexpr int kMaxCarry = 4096;                          // CTAs of one call (= carry slots)
constexpr long long kItemsPerCtaMax = 1LL << 16;         // merge items of one CTA, at most
constexpr long long kMaxItems = kMaxCarry * kItemsPerCtaMax;  // largest m + nnz accepted (2^28)
constexpr int kThreads = 128;
constexpr int kCtasPerSm = 5;               // 95 registers a thread: at 6 the prefetched words spill and
                                              // every spill waits for its load (55 -> 80 us, 450k banded rows)
constexpr int kMaxDevices = 64;
constexpr int kIpt = 13;                  // merge items per thread per tile, at most (odd: see the walk)
constexpr int kTile = kThreads * kIpt;    // merge items per tile, at most (1664)
constexpr int kLaneSteps = 48;            // longest row x rounds of rows a lane-per-row tile may have
constexpr int kMaxTiles = static_cast<int>((kItemsPerCtaMax + kTile - 1) / kTile);

static __device__ __align__(256) double g_carry_val[kMaxCarry];
static __device__ __align__(256) int g_carry_row[kMaxCarry];

struct Scratch {
    double *val = nullptr;
    int *row = nullptr;
    int sms = 0;
};
std::mutex g_mu;
Scratch g_scratch[kMaxDevices];
bool g_ready[kMaxDevices] = {};

// Merge-path coordinate on diagonal d of (row end offsets rowptr[1..m]) x (nonzeros 0..nnz-1),
// found by one whole warp: the number of rows completed (d minus it nonzeros are consumed). Every
// round trip to memory tests 32 rows. The first tries rows at doubling distances around the row
// that equal row lengths would give, which ends the search in two rounds on regular matrices;
// what interval is left shrinks 32-fold a round (3.5M rows: 5 rounds against 22 halvings).
__device__ __forceinline__ int merge_path(const int *__restrict__ rowptr, int m, int nnz, int d, int lane) {
    int lo = max(d - nnz, 0), hi = min(d, m);
    auto done = [&](int r) { return rowptr[r + 1] <= d - r - 1; };  // row r ends before diagonal d
    if (hi - lo > 32) {
        const int guess = static_cast<int>(static_cast<long long>(d) * m / (static_cast<long long>(m) + nnz));
        // lanes 0..15: guess - 2^15 + ... - 2^0; lanes 16..31: guess + 2^0 - 1 ... (ascending rows)
        const int r = lane < 16 ? guess - (1 << (15 - lane)) : guess + (1 << (lane - 16)) - 1;
        const bool in = r >= lo && r < hi;
        // rows below the range count as done, rows above it as not
        const unsigned yes = __ballot_sync(0xffffffffu, in ? done(r) : r < lo);
        const int c = __popc(yes);  // a prefix of the lanes: the rows ascend and done() is monotone
        const int below = __shfl_sync(0xffffffffu, r, max(c - 1, 0)), above = __shfl_sync(0xffffffffu, r, min(c, 31));
        if (c > 0) lo = max(lo, min(below + 1, hi));
        if (c < 32) hi = max(lo, min(hi, above));
    }
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32;
        const int r = lo + (lane + 1) * step - 1;
        const unsigned yes = __ballot_sync(0xffffffffu, r < hi && done(r));
        const int c = __popc(yes);
        const int next = lo + c * step + step - 1;  // the first tested row that is not done (if below hi)
        lo = min(lo + c * step, hi);
        hi = min(hi, next);
    }
    return lo;
}

// Inclusive segmented scan over the block, in thread order, of (row, v) pairs whose rows do not
// decrease with the thread index: the sum of v over the run of threads up to and including this
// one that carry the same row, earlier values first. Fixed order: reproducible.
__device__ __forceinline__ double seg_scan(int row, double v, int *srow, double *sv) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int r2 = __shfl_up_sync(0xffffffffu, row, o);
        const double v2 = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o && r2 == row) v = v2 + v;
    }
    if (lane == 31) {
        srow[warp] = row;
        sv[warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // the warps' totals, in order
        for (int w = 1; w < nw; ++w)
            if (srow[w] == srow[w - 1]) sv[w] = sv[w - 1] + sv[w];
    }
    __syncthreads();
    if (warp > 0 && srow[warp - 1] == row) v = sv[warp - 1] + v;
    return v;
}

// Merge-path SpMV, thread-sequential (see the file's head). What bounds it: loads in flight and
// the FP64 pipe (~19 clocks per warp instruction and SM), so
//  * the tile boundaries are found by whole warps (merge_path), the next tile's columns and values
//    are requested before this tile's walk, and a tile costs one gather latency;
//  * a nonzero's value and x lie side by side (one 16-byte shared load), walks are an odd number of
//    items apart (no bank conflicts between the lanes of a quarter warp when rows are long);
//  * FP64 instructions are the walk's one FMA per step, the additions that join rows across
//    threads, and alpha*s + beta*y once per row with all lanes busy: the walk itself only stores
//    raw sums;
//  * rows that span at most 4 threads join by a short walk back over the threads' open sums, 1 to
//    4 additions; only a tile with a longer row pays the segmented scan (5 per warp).
// 450k rows of 17 entries (7.65M nonzeros), beta != 0: 110.6 -> 43.8 us (ncu, 2.4 TB/s
// of 12 nnz + 28 m bytes).
__global__ void __launch_bounds__(kThreads, kCtasPerSm) k_mp_spmv(int m, int nnz, const int *__restrict__ rowptr,
                                                                  const int *__restrict__ col,
                                                                  const double *__restrict__ val, double alpha,
                                                                  const double *__restrict__ x, double beta,
                                                                  double *y, int D, int tile_items, double *carry_val,
                                                                  int *carry_row) {
    // one pool: the tile's nonzeros {value, x}, then its rows' sums, then their end offsets
    __shared__ double2 s_pool[kTile + 1];
    __shared__ int s_bound[kMaxTiles + 1];  // rows completed at each tile boundary
    __shared__ int s_trow[kThreads];        // row open at the end of each thread's walk
    __shared__ double s_tail[kThreads];     // its sum so far within the walk
    __shared__ int s_srow[kThreads / 32];
    __shared__ double s_sv[kThreads / 32], s_carry;
    const int c = blockIdx.x, t = threadIdx.x, lane = t & 31;
    const int total = m + nnz;
    const int c0 = static_cast<int>(min(static_cast<long long>(c) * D, static_cast<long long>(total)));
    const int c1 = static_cast<int>(min(static_cast<long long>(c0) + D, static_cast<long long>(total)));
    const int ntiles = (c1 - c0 + tile_items - 1) / tile_items;
    for (int b = t >> 5; b <= ntiles; b += kThreads / 32) {
        const int r = merge_path(rowptr, m, nnz, min(c0 + b * tile_items, c1), lane);
        if (lane == 0) s_bound[b] = r;
    }
    __syncthreads();
    int cc[kIpt];
    double vv[kIpt];
    auto request = [&](int tile) {  // the columns and values of a tile
        const int ka = min(c0 + tile * tile_items, c1) - s_bound[tile];
        const int nk = min(c0 + (tile + 1) * tile_items, c1) - s_bound[tile + 1] - ka;
#pragma unroll
        for (int i = 0; i < kIpt; ++i) {
            const int q = t + i * kThreads;
            cc[i] = q < nk ? __ldg(col + ka + q) : 0;
            vv[i] = q < nk ? __ldg(val + ka + q) : 0.0;
        }
    };
    if (ntiles > 0) request(0);
    double tile_carry = 0.0;  // the open row's sum from earlier tiles of this CTA (row s_bound[tile])
    for (int tile = 0; tile < ntiles; ++tile) {
        const int ra = s_bound[tile], ka = c0 + tile * tile_items - ra;
        const int nr = s_bound[tile + 1] - ra, T = min(tile_items, c1 - c0 - tile * tile_items), nk = T - nr;
        double *s_sum = reinterpret_cast<double *>(s_pool + nk);
        int *s_rend = reinterpret_cast<int *>(s_sum + nr);
        // row ends from the tile's first nonzero; row nr is the one open at the tile's end
        const int rounds = nr / kThreads + 1;
        bool uneven = false;
        for (int i = t; i <= nr; i += kThreads) {
            const int b = i > 0 ? rowptr[ra + i] - ka : 0, e = i < nr ? rowptr[ra + i + 1] - ka : nk;
            s_rend[i] = e;
            uneven = uneven || (e - b) * rounds > kLaneSteps;
        }
        double yold = 0.0;
        if (beta != 0.0 && t < nr) yold = y[ra + t];
        double xv[kIpt];
#pragma unroll
        for (int i = 0; i < kIpt; ++i) xv[i] = t + i * kThreads < nk ? __ldg(x + cc[i]) : 0.0;
#pragma unroll
        for (int i = 0; i < kIpt; ++i)
            if (t + i * kThreads < nk) s_pool[t + i * kThreads] = make_double2(vv[i], xv[i]);
        uneven = __syncthreads_or(uneven);
        if (tile + 1 < ntiles) request(tile + 1);
        if (!uneven) {
            // a lane per row, the carried row continuing its sum and the open one starting its own
            for (int i = t; i <= nr; i += kThreads) {
                double acc = i == 0 ? tile_carry : 0.0;
                int k = i > 0 ? s_rend[i - 1] : 0;
                const int e = s_rend[i];
                for (; k + 4 <= e; k += 4) {
                    const double2 q0 = s_pool[k], q1 = s_pool[k + 1], q2 = s_pool[k + 2], q3 = s_pool[k + 3];
                    acc = fma(q3.x, q3.y, fma(q2.x, q2.y, fma(q1.x, q1.y, fma(q0.x, q0.y, acc))));
                }
                for (; k < e; ++k) acc = fma(s_pool[k].x, s_pool[k].y, acc);
                if (i < nr) {
                    const double s = alpha * acc;
                    y[ra + i] = beta != 0.0 ? fma(beta, i == t ? yold : y[ra + i], s) : s;
                } else {
                    s_carry = acc;
                }
            }
            __syncthreads();
            tile_carry = s_carry;
            continue;
        }
        // this thread's start on the tile's merge path (row ends and nonzeros counted from the tile's
        // first), then its items: a nonzero of row r, or the end of row r
        const int ipt = (T + kThreads - 1) / kThreads | 1;
        const int dt = min(t * ipt, T), steps = min(ipt, T - dt), last = (T - 1) / ipt;
        int lo = max(dt - nk, 0), hi = min(dt, nr);
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s_rend[mid] <= dt - mid - 1) lo = mid + 1;
            else hi = mid;
        }
        int r = lo, k = dt - lo, first_row = -1, end = r < nr ? s_rend[r] : T;
        double acc = 0.0, first_acc = 0.0;
        for (int i = 0; i < steps; ++i) {
            if (k < end) {
                const double2 e = s_pool[k];
                acc = fma(e.x, e.y, acc);
                ++k;
            } else {
                if (first_row < 0) {
                    first_row = r;
                    first_acc = acc;
                } else {
                    s_sum[r] = acc;
                }
                acc = 0.0;
                end = ++r < nr ? s_rend[r] : T;
            }
        }
        s_trow[t] = r;
        s_tail[t] = acc;
        __syncthreads();
        const bool far = t >= 4 && t <= last && s_trow[t - 4] == r;  // a row open over 5 threads
        if (!__syncthreads_or(far)) {
            // the open sums of the threads before t, back to the one that started t's first row
            if (t <= last && (first_row >= 0 || t == last)) {
                double cin = 0.0;
                int u = t - 1;
                for (; u >= 0; --u) {
                    cin = s_tail[u] + cin;
                    if (s_trow[u] != (u > 0 ? s_trow[u - 1] : 0)) break;  // u started this row
                }
                if (u < 0) cin = tile_carry + cin;
                if (first_row >= 0) s_sum[first_row] = cin + first_acc;
                if (t == last) s_carry = first_row >= 0 ? acc : cin + acc;
            }
        } else {
            // thread 0's run continues the tile's carried row; the scan joins the runs across threads
            const double own = (t == 0 && first_row < 0) ? tile_carry + acc : acc;
            const double run = seg_scan(r, own, s_srow, s_sv);
            const double prev = __shfl_up_sync(0xffffffffu, run, 1);
            const int prow = __shfl_up_sync(0xffffffffu, r, 1);
            if (first_row >= 0) {
                // the runs of the earlier threads on this row, or the tile's carry for thread 0
                double cin = t == 0 ? tile_carry : 0.0;
                if (lane != 0) {
                    if (prow == first_row) cin = prev;
                } else if (t > 0 && s_srow[(t >> 5) - 1] == first_row) {
                    cin = s_sv[(t >> 5) - 1];
                }
                s_sum[first_row] = cin + first_acc;
            }
            if (t == kThreads - 1) s_carry = run;
        }
        __syncthreads();
        tile_carry = s_carry;
        for (int i = t; i < nr; i += kThreads) {
            const double s = alpha * s_sum[i];
            y[ra + i] = beta != 0.0 ? fma(beta, i == t ? yold : y[ra + i], s) : s;
        }
        __syncthreads();
    }
    if (t == 0) {
        // the row left open at the end of the CTA's range, if this CTA consumed any of its nonzeros
        const int ro = s_bound[ntiles], ko = c1 - ro, k0 = c0 - s_bound[0];
        const bool open = ntiles > 0 && ro < m && ko > max(rowptr[ro], k0);
        carry_val[c] = open ? tile_carry : 0.0;
        carry_row[c] = open ? ro : -1;
    }
}

// Adds each row's carries to its y, once: the first CTA carrying a row stands for its run (CTAs c, c + 1, ...
// with that row, as the rows ascend). A run of up to kRun carries, as between even tiles, is its thread's: all
// requested at once, added in CTA order. A longer one is its warp's: strided over the lanes, four requests each,
// then added across them, in an order that the run's length alone decides. (A thread that walked a long run
// alone waited for each carry: one row of 777,777 entries over 760 CTAs 106.7 us a call, so 12.4. A warp for every
// carry cost rows of 17 entries 0.5 us of 45.)
constexpr int kRun = 4;
__global__ void k_mp_fixup(int n_cta, double alpha, double *y, const double *carry_val, const int *carry_row) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the first kernel's stores are complete and visible
    auto row_of = [&](int q) { return q >= 0 && q < n_cta ? carry_row[q] : -1; };
    const int row = row_of(c), before = row_of(c - 1);
    int next[kRun];
    double v[kRun];
#pragma unroll
    for (int u = 0; u < kRun; ++u) {
        next[u] = row_of(c + u + 1);
        v[u] = c + u < n_cta ? carry_val[c + u] : 0.0;
    }
    const bool first = row >= 0 && before != row, far = first && next[kRun - 1] == row;
    if (first && !far) {
        double s = v[0];
#pragma unroll
        for (int u = 1; u < kRun; ++u)
            if (next[u - 1] == row) s += v[u];
        y[row] = fma(alpha, s, y[row]);
    }
    for (unsigned left = __ballot_sync(0xffffffffu, far); left != 0; left &= left - 1) {
        const int src = __ffs(left) - 1, r = __shfl_sync(0xffffffffu, row, src);
        double s = 0.0;
        for (int q = c + src;; q += 32 * kRun) {  // this lane's: the run's first carry + lane, ...
            bool on[kRun];
#pragma unroll
            for (int u = 0; u < kRun; ++u) {
                on[u] = row_of(q + 32 * u) == r;
                v[u] = on[u] ? carry_val[q + 32 * u] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kRun; ++u)
                if (on[u]) s += v[u];
            if (!on[kRun - 1]) break;
        }
        s = hhp::warp_sum(s);
        if (lane == 0) y[r] = fma(alpha, s, y[r]);
    }
}

hhp_status scratch_for_current_device(Scratch &out) {
    int dev = 0;
    HHP_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        hhp::set_error("hhp_spmv_csr_noalloc: device %d outside the supported range 0..%d", dev, kMaxDevices - 1);
        return HHP_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_ready[dev]) {
        Scratch s;
        HHP_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&s.val), g_carry_val));
        HHP_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&s.row), g_carry_row));
        HHP_CUDA(cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev));
        g_scratch[dev] = s;
        g_ready[dev] = true;
    }
    out = g_scratch[dev];
    return HHP_OK;
}

}  // namespace

extern "C" hhp_status hhp_spmv_csr_noalloc(int m, int n, int nnz, const int *rowptr_dev, const int *col_dev,
                                           const double *val_dev, double alpha, const double *x_dev, double beta,
                                           double *y_dev, void *stream) {
    HHP_API_BEGIN
    if (m < 0 || n < 0 || nnz < 0 || !rowptr_dev || (nnz > 0 && (!col_dev || !val_dev)) || (m > 0 && !y_dev) ||
        (nnz > 0 && !x_dev)) {
        hhp::set_error("hhp_spmv_csr_noalloc: invalid sizes or null pointers");
        return HHP_ERR_ARG;
    }
    const long long total = static_cast<long long>(m) + nnz;
    if (total > kMaxItems) {
        hhp::set_error("hhp_spmv_csr_noalloc: m + nnz = %lld exceeds the maximum %lld (%d CTAs x %lld items)", total,
                       kMaxItems, kMaxCarry, kItemsPerCtaMax);
        return HHP_ERR_ARG;
    }
    if (m == 0) return HHP_OK;
    Scratch sc;
    HHP_TRY(scratch_for_current_device(sc));
    // one resident wave of CTAs that share the list evenly, but no CTA below 4 items a thread; lists
    // too long for that take the CTAs of all carry slots
    long long n_cta = std::min<long long>(static_cast<long long>(sc.sms) * kCtasPerSm, kMaxCarry);
    n_cta = std::max(1LL, std::min(n_cta, total / (4 * kThreads)));
    if ((total + n_cta - 1) / n_cta > kItemsPerCtaMax) n_cta = kMaxCarry;
    const int D = static_cast<int>((total + n_cta - 1) / n_cta), tiles = (D + kTile - 1) / kTile;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_mp_spmv<<<static_cast<int>(n_cta), kThreads, 0, st>>>(m, nnz, rowptr_dev, col_dev, val_dev, alpha, x_dev,
                                                            beta, y_dev, D, (D + tiles - 1) / tiles, sc.val, sc.row);
    // launched programmatically: it is set up while the first kernel still runs and starts when that one's
    // last block has ended, not a launch later (450k banded rows 46.8 -> 45.1 us a call, one row of 100,000 entries
    // 10.3 -> 8.3)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>((n_cta + 255) / 256));
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    HHP_CUDA(cudaLaunchKernelEx(&cfg, k_mp_fixup, static_cast<int>(n_cta), alpha, y_dev,
                                static_cast<const double *>(sc.val), static_cast<const int *>(sc.row)));
    HHP_CUDA(cudaGetLastError());
    return HHP_OK;
    HHP_API_END
}
