// hhp_small.cuh -- the BiCGStab solve of a small system as one kernel, in FP64 and in the mixed form.
//
// 5-point stencils, us an iteration against the graph loop: 32^2 7.9 / 19.4, 64^2 9.1 / 19.7, 128^2
// 11.7 / 20.1 (classic 64^2 10.1 / 25.0); 17 entries per row: 4,000 rows 14.0 / 27.5, 20,000 rows
// 17.9 / 30.0.
//
// On a system of few rows an iteration of the graph loop is 4 (classic: 5) launches of
// ~5 us each, nearly all of it launch gaps and chains of latencies: the work list, the partial
// records, operands that left the registers a kernel ago. Here the whole system lives on the SMs: a
// row per thread, its matrix entries in shared memory, its elements of x, r, r0, p, v, s and t in
// registers; what other rows need (p, and r with v, or s) goes through L2. The initial and the final
// residual are formed here too, so a solve is this one launch. An iteration has three grid-wide
// exchanges (classic: four):
//   v = A p               -> sum of r0.v                      (and every v is visible)
//   s = r - alpha v, t = A s -> sums of t.s, t.t, r0.t, s.s, r0.s
//   x, r, p               -> (every p and r is visible)
// t = A s forms s_j = r_j - alpha v_j for the entries it gathers, one more multiply-add each, which is
// cheaper than a fourth exchange up to kSmallPubS entries per row; above, s is published.
//
// Up to kSmallClusterRows rows the blocks are one thread-block cluster: an exchange is partial sums
// pushed into every block's shared memory and the hardware's cluster barrier (556 cycles at 16
// blocks). Above that the FP64 work of 16 SMs outweighs the cheaper exchange: the grid is launched
// cooperatively (all blocks resident) and an exchange is records in L2 and an arrival count that every
// block polls (1.2 us; polling all blocks' records instead took 3.3 us at 152 blocks). Every such wait
// is bounded: one that runs out sets the context's error word and the block leaves, as the others then
// do. All blocks add the same numbers in the same order, so they compute the same scalars bit for bit and
// take the same branches.
#pragma once

constexpr int kSmallThreads = 512;
constexpr int kSmallMaxK = 64;            // entries per row, at most
constexpr int kSmallPubS = 9;             // above: t = A s gathers published s (an exchange costs what
                                          // some ten FP64 instructions of every warp do)
constexpr int kSmallQ = 5;                // quantities of the widest exchange
constexpr int kSmallMaxGrid = 160;        // blocks (5 records per lane of the reading warp)
constexpr int kSmallCluster = 16;         // blocks of the one-cluster form, at most
constexpr int kSmallClusterRows = 6144;   // 5-point, 4096 rows: 9.1 against 13.9 us an iteration on the
                                          // whole grid, 8100 rows: 12.3 against 12.4; 17 entries per
                                          // row, 4000 rows: 14.0 against 19.1, 8000 rows: 19.1 against 17.8
// The count starts one below 2^32: a launch of 152 blocks passes 2^32 every 28 million exchanges, and so
// every launch does in its first.
constexpr unsigned kSmallCount0 = 0xffffffffu;
constexpr int kSmallPolls = 1 << 20;      // reads of the count before giving up (~0.5 us each); the
                                          // variable HHP_SMALL_POLLS sets another limit

struct SmallArgs {
    DevScal *sc;
    const long long *slice_ptr;
    const int *pos_row;       // the row at each position of the slices (null: the position)
    const int *pos_len;       // row lengths, or masks of diagonals (uni)
    const double *sval;
    const int *scol;
    const short *scol16;
    int uni, nd, H, K, n, rows;  // rows: of a block
    int doff[kMaxDiag];
    double *X, *P, *S;
    const double *B;
    double2 *RV;              // {r, v}
    float *P32;               // mixed form: p, {r, v}
    float2 *RV32;
    double *rec;              // 2 sets of kSmallQ * grid partial sums, used in turn
    unsigned *arrived;        // blocks that have arrived, over all exchanges, from kSmallCount0
    double *hist;
    int hist_cap, polls;
    int *dev_err;
};

struct SmallShared {
    double red[kSmallQ * kSmallThreads];
    double in[2][kSmallQ][kSmallCluster];  // cluster form: the blocks' partial sums, used in turn
    double tot[kSmallQ];
    double bc[4];
    int mode, ok;
};

// The block's sum of v[q] over its threads, in all lanes of warp q mod (number of warps). Dense tree
// (T a power of two), then a butterfly in one warp per quantity.
template <int NQ>
__device__ __forceinline__ void block_tree(SmallShared &sh, const double (&v)[NQ]) {
    const int t = threadIdx.x, T = blockDim.x;
#pragma unroll
    for (int q = 0; q < NQ; ++q) sh.red[q * T + t] = v[q];
    __syncthreads();
    for (int h = T >> 1; h >= 32; h >>= 1) {
        if (t < h) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) sh.red[q * T + t] += sh.red[q * T + t + h];
        }
        __syncthreads();
    }
}

// The first exchange writes other blocks' shared memory, which may only be done once every block of the
// cluster runs. cluster_start() says so of this block, cluster_started() waits for all; between the two a
// kernel stages its matrix, so the wait costs nothing. (Not .aligned: lanes may arrive apart.)
__device__ __forceinline__ void cluster_start() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_started() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One exchange of NQ sums (NQ = 0: a barrier), number e = 1, 2, ... of the launch; the sums in sh.tot.
// (CLUSTER: after cluster_started().) The blocks' earlier global stores are visible to every block after
// it. The buffers of e are written again at e + 2, which a block reaches only after every block has arrived at
// e + 1, that is has read e's. Returns false when the wait ran out (uniform across the block).
template <int NQ, bool CLUSTER>
__device__ __forceinline__ bool exchange(const SmallArgs &a, SmallShared &sh, const double (&v)[NQ > 0 ? NQ : 1],
                                         unsigned &e) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, T = blockDim.x, G = gridDim.x, NW = T >> 5;
    ++e;
    if constexpr (NQ > 0) block_tree<NQ>(sh, v);
    if constexpr (CLUSTER) {
        if constexpr (NQ > 0) {
            for (int q = w; q < NQ; q += NW) {
                const double mine = warp_sum(sh.red[q * T + lane]);
                if (lane < G) {
                    uint32_t to;
                    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(&sh.in[e & 1u][q][blockIdx.x]));
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(at), "r"(lane));
                    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(mine) : "memory");
                }
            }
        }
        cluster_barrier();
        if constexpr (NQ > 0) {
            for (int q = w; q < NQ; q += NW) {
                double s = lane < G ? sh.in[e & 1u][q][lane & (kSmallCluster - 1)] : 0.0;
#pragma unroll
                for (int o = kSmallCluster / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) sh.tot[q] = s;
            }
            __syncthreads();
        }
        return true;
    } else {
        double *set = a.rec + (e & 1u) * (kSmallQ * kSmallMaxGrid);
        if constexpr (NQ > 0) {
            for (int q = w; q < NQ; q += NW) {
                const double mine = warp_sum(sh.red[q * T + lane]);
                if (lane == 0) __stcg(set + q * kSmallMaxGrid + blockIdx.x, mine);
            }
        }
        __syncthreads();
        if (t == 0) {
            // the block's stores (ordered before this by the barrier) before its arrival
            asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(a.arrived) : "memory");
            const unsigned target = kSmallCount0 + e * static_cast<unsigned>(G);
            bool all = false;
            for (int i = 0; i < a.polls && !all; ++i) {
                unsigned seen;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.arrived) : "memory");
                all = count_reached(seen, target);
            }
            sh.ok = all;
        }
        __syncthreads();
        if (!sh.ok) {
            if (t == 0) atomicExch(a.dev_err, DEV_ERR_TIMEOUT);
            return false;
        }
        if constexpr (NQ > 0) {
            for (int q = w; q < NQ; q += NW) {
                double r[kSmallMaxGrid / 32], s = 0.0;
#pragma unroll
                for (int i = 0; i < kSmallMaxGrid / 32; ++i)
                    r[i] = lane + 32 * i < G ? __ldcg(set + q * kSmallMaxGrid + lane + 32 * i) : 0.0;
#pragma unroll
                for (int i = 0; i < kSmallMaxGrid / 32; ++i)
                    if (32 * i < G) s += r[i];
                s = warp_sum(s);
                if (lane == 0) sh.tot[q] = s;
            }
            __syncthreads();
        }
        return true;
    }
}

// Sum over a row's entries, in order, of val * get(col): eight gathers in flight, as many steps as the
// warp's longest row has, kmax (a multiply-add that no lane needs still takes the FP64 pipe's slot).
template <typename T, typename G>
__device__ __forceinline__ T small_row_sum(const T *sv, const int *sc, int ld, int len, int kmax, G get) {
    T acc = T(0);
    auto steps = [&](auto n, int k) {
        constexpr int N = decltype(n)::value;
        T g[N];
#pragma unroll
        for (int u = 0; u < N; ++u) g[u] = k + u < len ? get(sc[(k + u) * ld]) : T(0);
#pragma unroll
        for (int u = 0; u < N; ++u)
            if (k + u < len) acc = tfma(sv[(k + u) * ld], g[u], acc);
    };
    int k = 0;
    for (; k + 8 <= kmax; k += 8) steps(std::integral_constant<int, 8>(), k);
    switch (kmax - k) {
        case 1: steps(std::integral_constant<int, 1>(), k); break;
        case 2: steps(std::integral_constant<int, 2>(), k); break;
        case 3: steps(std::integral_constant<int, 3>(), k); break;
        case 4: steps(std::integral_constant<int, 4>(), k); break;
        case 5: steps(std::integral_constant<int, 5>(), k); break;
        case 6: steps(std::integral_constant<int, 6>(), k); break;
        case 7: steps(std::integral_constant<int, 7>(), k); break;
        default: break;
    }
    return acc;
}

template <bool MERGED, bool CLUSTER>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small(const __grid_constant__ SmallArgs a) {
    extern __shared__ double s_mat[];  // val[K][rows], then col[K][rows]
    __shared__ SmallShared sh;
    const int t = threadIdx.x, pos = blockIdx.x * a.rows + t;
    const bool own = t < a.rows && pos < a.n, lead = blockIdx.x == 0 && t == 0;
    const int row = own && a.pos_row ? a.pos_row[pos] : pos;
    if constexpr (CLUSTER) cluster_start();
    double *sv = s_mat + t;
    int *sc_ = reinterpret_cast<int *>(s_mat + a.K * a.rows) + t;
    const int ld = a.rows;
    DevScal *sc = a.sc;
    // control words, and on a restart the counts and threshold of the passes before (the lead thread
    // writes them at the end, which no block reaches before all have taken part in the first exchange)
    const int restart = sc->restart, maxit = sc->maxit, fixed = sc->fixed;
    const double rtol2 = sc->rtol2, thr2_in = sc->thr2, rr0_in = sc->rr0;
    const int it0 = restart ? sc->iter : 0;
    unsigned e = 0;
    int iter = it0, status = ST_RUNNING;
    int len = 0;
    double x = 0.0, b = 0.0, r = 0.0, p = 0.0, v = 0.0, s = 0.0, tv = 0.0;
    if (own) {
        const long long base = a.uni ? static_cast<long long>(pos / a.H) * a.nd * a.H + pos % a.H
                                     : a.slice_ptr[pos / a.H] + pos % a.H;
        const int pl = a.pos_len[pos];
        if (a.uni) {
            for (int k = 0; k < a.nd; ++k)
                if (pl >> k & 1) {
                    sv[len * ld] = a.sval[base + static_cast<long long>(k) * a.H];
                    sc_[len * ld] = row + a.doff[k];
                    ++len;
                }
        } else {
            for (int k = 0; k < pl; ++k) {
                const long long q = base + static_cast<long long>(k) * a.H;
                sv[k * ld] = a.sval[q];
                sc_[k * ld] = a.scol16 ? row + a.scol16[q] : a.scol[q];
            }
            len = pl;
        }
        x = a.X[row];
        b = a.B[row];
    }
    const int kmax = __reduce_max_sync(0xffffffffu, len);
    auto row_sum = [&](auto get) { return small_row_sum<double>(sv, sc_, ld, len, kmax, get); };
    const double none[1] = {0.0};
    // r = b - A x, p = r; ||r||^2, ||b||^2 and whether x0 has a nonzero. x0 = 0 means r = b, also where
    // A holds an infinity or a NaN (the loop finds it): formed again then.
    r = b - row_sum([&](int c) { return __ldcg(a.X + c); });
    auto publish = [&] {
        p = r;
        if (own) {
            a.P[row] = p;
            a.RV[row].x = r;
        }
    };
    publish();
    const double di[3] = {own ? r * r : 0.0, own ? b * b : 0.0, own && x != 0.0 ? 1.0 : 0.0};
    if constexpr (CLUSTER) cluster_started();
    bool good = exchange<3, CLUSTER>(a, sh, di, e);
    double rr = sh.tot[0], alpha = 1.0, omega = 1.0;
    const double bb = sh.tot[1], thr2 = restart ? thr2_in : fixed ? -1.0 : rtol2 * bb;
    if (good && !isfinite(rr) && sh.tot[2] == 0.0) {
        r = b;
        rr = bb;
        publish();
        good = exchange<0, CLUSTER>(a, sh, none, e);
    }
    const double r0 = r;
    double rho = rr;
    // stop tests on the initial residual (K_P's first run)
    if (thr2 >= 0.0 && rr <= thr2) status = ST_CONVERGED;
    else if (iter >= maxit) status = ST_MAXIT;
    else if (!finite_nonzero(rho) || !isfinite(rr)) status = ST_BREAKDOWN;
    __syncthreads();  // sh.tot has been read
    while (status == ST_RUNNING && good) {
        // v = A p, alpha
        v = row_sum([&](int c) { return __ldcg(a.P + c); });
        if (own) a.RV[row].y = v;
        const double dv[1] = {own ? v * r0 : 0.0};
        good = exchange<1, CLUSTER>(a, sh, dv, e);
        if (!good) break;
        if (t == 0) {
            const double rv = sh.tot[0], al = rho / rv;
            sh.mode = finite_nonzero(rv) && isfinite(al);
            sh.bc[0] = al;
        }
        __syncthreads();
        if (!sh.mode) {
            status = ST_BREAKDOWN;
            break;
        }
        alpha = sh.bc[0];
        ++iter;
        // s, t = A s
        s = fma(-alpha, v, r);
        if (a.K > kSmallPubS) {
            if (own) a.S[row] = s;
            good = exchange<0, CLUSTER>(a, sh, none, e);
            if (!good) break;
            tv = row_sum([&](int c) { return __ldcg(a.S + c); });
        } else {
            tv = row_sum([&](int c) {
                const double2 q = __ldcg(a.RV + c);
                return fma(-alpha, q.y, q.x);
            });
        }
        if constexpr (MERGED) {
            const double d[5] = {own ? tv * s : 0.0, own ? tv * tv : 0.0, own ? tv * r0 : 0.0, own ? s * s : 0.0,
                                 own ? s * r0 : 0.0};
            good = exchange<5, CLUSTER>(a, sh, d, e);
            if (!good) break;
            if (t == 0) {  // the step of K_XRP
                const double ts = sh.tot[0], tt = sh.tot[1], r0t = sh.tot[2], ss = sh.tot[3], r0s = sh.tot[4];
                int mode = 0, term = ST_RUNNING;
                double rn = ss, om = 0.0, beta = 0.0, rho_new = rho;
                if (thr2 >= 0.0 && ss <= thr2) {
                    mode = 2;
                    term = ST_CONVERGED_HALF;
                } else {
                    om = ts / tt;
                    if (!finite_nonzero(tt) || !isfinite(om)) {
                        term = ST_BREAKDOWN;
                    } else {
                        rn = fmax(ss - om * ts, 0.0);
                        mode = 3;
                        if (thr2 >= 0.0 && fmax(rn, kCancel * ss) <= thr2) {
                            term = ST_CONVERGED;
                        } else if (iter >= maxit) {
                            term = ST_MAXIT;
                        } else {
                            rho_new = r0s - om * r0t;
                            if (!finite_nonzero(rho_new) || !isfinite(rn)) {
                                term = ST_BREAKDOWN;
                            } else {
                                beta = (rho_new / rho) * (alpha / om);
                                mode = 1;
                            }
                        }
                    }
                }
                sh.mode = mode | term << 8;
                sh.bc[0] = om;
                sh.bc[1] = beta;
                sh.bc[2] = rn;
                sh.bc[3] = rho_new;
            }
            __syncthreads();
            const int mode = sh.mode & 255;
            status = sh.mode >> 8;
            omega = sh.bc[0];
            rho = sh.bc[3];
            if (mode != 0) {
                rr = sh.bc[2];
                if (lead && iter >= 1 && iter - 1 < a.hist_cap) a.hist[iter - 1] = rr;
                if (mode == 2) {
                    x = fma(alpha, p, x);
                    r = s;
                } else {
                    x = fma(omega, s, fma(alpha, p, x));
                    r = fma(-omega, tv, s);
                    if (mode == 1) p = fma(sh.bc[1], fma(-omega, v, p), r);
                }
            }
        } else {
            const double d[3] = {own ? tv * s : 0.0, own ? tv * tv : 0.0, own ? s * s : 0.0};
            good = exchange<3, CLUSTER>(a, sh, d, e);
            if (!good) break;
            if (t == 0) {  // the step of K_XR
                const double ss = sh.tot[2];
                int mode = thr2 >= 0.0 && ss <= thr2 ? 2 : 1;
                double om = 0.0;
                if (mode == 1) {
                    om = sh.tot[0] / sh.tot[1];
                    if (!finite_nonzero(sh.tot[1]) || !isfinite(om)) mode = 0;
                }
                sh.mode = mode;
                sh.bc[0] = om;
                sh.bc[1] = ss;
            }
            __syncthreads();
            const int mode = sh.mode;
            const double ss = sh.bc[1];
            if (mode == 0) {
                status = ST_BREAKDOWN;
                break;
            }
            if (mode == 2) {
                x = fma(alpha, p, x);
                r = s;
            } else {
                omega = sh.bc[0];
                x = fma(omega, s, fma(alpha, p, x));
                r = fma(-omega, tv, s);
            }
            const double d2[2] = {own ? r * r0 : 0.0, own ? r * r : 0.0};
            good = exchange<2, CLUSTER>(a, sh, d2, e);
            if (!good) break;
            if (t == 0) {  // the step of K_P
                double beta = 0.0;
                const double rho_new = sh.tot[0], rn = sh.tot[1];
                const int term = step_p(ST_RUNNING, iter, it0, maxit, thr2, rho_new, rn, ss, rho, alpha, omega, false, beta);
                sh.mode = term;
                sh.bc[0] = beta;
                sh.bc[1] = rn;
                sh.bc[2] = rho_new;
                if (lead && iter - 1 < a.hist_cap) a.hist[iter - 1] = rn;
            }
            __syncthreads();
            status = sh.mode;
            rr = sh.bc[1];
            if (status == ST_RUNNING) {
                rho = sh.bc[2];
                p = fma(sh.bc[0], fma(-omega, v, p), r);
            }
        }
        if (status != ST_RUNNING) break;
        if (own) {
            a.RV[row].x = r;
            a.P[row] = p;
        }
        good = exchange<0, CLUSTER>(a, sh, none, e);
    }
    if (own) a.X[row] = x;
    // the true residual of the result
    double true_rr = rr;
    if (good) good = exchange<0, CLUSTER>(a, sh, none, e);
    if (good) {
        const double res = b - row_sum([&](int c) { return __ldcg(a.X + c); });
        const double df[1] = {own ? res * res : 0.0};
        good = exchange<1, CLUSTER>(a, sh, df, e);
        true_rr = sh.tot[0];
    }
    if (lead) {
        sc->status = good ? status : ST_DEVICE_ERROR;
        sc->rr0 = restart ? rr0_in : bb;
        sc->thr2 = sc->thr2_rec = thr2;
        sc->bb = bb;
        sc->iter = iter;
        sc->iter_start = it0;
        sc->bodies = 0;
        sc->arrivals = 0;
        sc->rr_last = rr;
        sc->true_rr = true_rr;
    }
}

// Growth of the FP32 recursive ||r||^2 over the last true ||b - A x||^2 taken as divergence
// (a factor 1e5 in the norm: BiCGStab's residual peaks stay far below it when it converges).
constexpr double kDivergence2 = 1e10;
// Mixed form, stagnation: an FP64 update whose true ||b - A x||^2 is above kStall2 times the last
// one's (the norm fell by less than 10%), kStallUpdates times in a row.
constexpr double kStall2 = 0.81;
constexpr int kStallUpdates = 3;

// The mixed form of a small system (see K_MIX_INIT to K_MIX_FINAL): the FP32 recurrences as in k_small,
// the FP64 iterate and residual per row in the thread's registers. 5-point stencils, us an inner iteration
// against the graph loop: 100^2 11.9 / 22.7, 125^2 11.2 / 23.2; whole solves: 4,291 and 10,033 rows of 17
// entries 364 / 936 and 396 / 944 us, 16^3 7-point 537 / 1651 us.
// An FP64 update is two exchanges (every x visible; the sums) and a product with the FP64 values from
// L2, a few times per solve. t = A s always forms s from r and v: an FP32 multiply-add an entry costs
// next to nothing beside an exchange.
template <bool MERGED, bool CLUSTER>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small_mix(const __grid_constant__ SmallArgs a) {
    extern __shared__ double s_mat[];  // float val[K][rows], then col[K][rows]
    __shared__ SmallShared sh;
    const int t = threadIdx.x, pos = blockIdx.x * a.rows + t;
    const bool own = t < a.rows && pos < a.n, lead = blockIdx.x == 0 && t == 0;
    const int row = own && a.pos_row ? a.pos_row[pos] : pos;
    if constexpr (CLUSTER) cluster_start();
    float *sv = reinterpret_cast<float *>(s_mat) + t;
    int *sc_ = reinterpret_cast<int *>(reinterpret_cast<float *>(s_mat) + a.K * a.rows) + t;
    const int ld = a.rows;
    DevScal *sc = a.sc;
    const int restart = sc->restart, maxit = sc->maxit;
    const double rtol2 = sc->rtol2, inner2 = sc->inner_rtol2, thr2_in = sc->thr2, rr0_in = sc->rr0, bb_in = sc->bb;
    const int it0 = restart ? sc->iter : 0;
    unsigned e = 0;
    int iter = it0, updates = restart ? sc->updates : 0, stalls = 0, status = ST_RUNNING, len = 0, mask = 0;
    long long base = 0;
    double x = 0.0, b = 0.0;
    float d = 0.f, r = 0.f, p = 0.f, v = 0.f, s = 0.f, tv = 0.f;
    if (own) {
        base = a.uni ? static_cast<long long>(pos / a.H) * a.nd * a.H + pos % a.H : a.slice_ptr[pos / a.H] + pos % a.H;
        mask = a.pos_len[pos];
        if (a.uni) {
            for (int k = 0; k < a.nd; ++k)
                if (mask >> k & 1) {
                    sv[len * ld] = static_cast<float>(a.sval[base + static_cast<long long>(k) * a.H]);
                    sc_[len * ld] = row + a.doff[k];
                    ++len;
                }
        } else {
            for (int k = 0; k < mask; ++k) {
                const long long q = base + static_cast<long long>(k) * a.H;
                sv[k * ld] = static_cast<float>(a.sval[q]);
                sc_[k * ld] = a.scol16 ? row + a.scol16[q] : a.scol[q];
            }
            len = mask;
        }
        x = a.X[row];
        b = a.B[row];
    }
    const int kmax = __reduce_max_sync(0xffffffffu, len);
    auto row_sum = [&](auto get) { return small_row_sum<float>(sv, sc_, ld, len, kmax, get); };
    // b - A x of this row in FP64 (every block's x is in a.X)
    auto residual = [&] {
        double acc = 0.0;
        if (a.uni) {
            int j = 0;
            for (int k = 0; k < a.nd; ++k)
                if (mask >> k & 1)
                    acc = fma(a.sval[base + static_cast<long long>(k) * a.H], __ldcg(a.X + sc_[j++ * ld]), acc);
        } else {
#pragma unroll 4
            for (int k = 0; k < len; ++k)
                acc = fma(a.sval[base + static_cast<long long>(k) * a.H], __ldcg(a.X + sc_[k * ld]), acc);
        }
        return b - acc;
    };
    const double none[1] = {0.0};
    auto publish = [&] {  // r and p, for the other rows after the next exchange
        if (own) {
            a.RV32[row].x = r;
            a.P32[row] = p;
        }
    };
    double rd = residual();
    r = static_cast<float>(rd);
    p = r;
    publish();
    const double di[4] = {own ? rd * rd : 0.0, own ? b * b : 0.0, own && x != 0.0 ? 1.0 : 0.0,
                          static_cast<double>(r) * r};
    if constexpr (CLUSTER) cluster_started();
    bool good = exchange<4, CLUSTER>(a, sh, di, e);
    double rd2 = sh.tot[0], rho = sh.tot[3], alpha = 1.0, omega = 1.0;
    const double bb = restart ? bb_in : sh.tot[1], thr2 = restart ? thr2_in : rtol2 * bb;
    if (good && !isfinite(rd2) && sh.tot[2] == 0.0) {  // x0 = 0: r = b whatever A holds (see k_small)
        rd2 = sh.tot[1];
        r = static_cast<float>(b);
        p = r;
        publish();
        const double dr[1] = {static_cast<double>(r) * r};
        good = exchange<1, CLUSTER>(a, sh, dr, e);
        rho = sh.tot[0];
    }
    const float r0 = r;
    double true_rr = rd2, rr_max = rd2, rr_last = rd2;
    // the stop tests of K_MIX_INIT, then of K_P's first run
    if (rd2 <= rtol2 * bb) {
        status = ST_CONVERGED;
    } else if (!isfinite(rd2)) {
        status = ST_BREAKDOWN;
    } else {
        double beta;
        status = step_p(ST_RUNNING, iter, it0, maxit, -1.0, rho, rho, 0.0, 1.0, 1.0, 1.0, false, beta);
        rr_last = rho;
    }
    __syncthreads();  // sh.tot has been read
    while (status == ST_RUNNING && good) {
        // v = A p, alpha
        v = row_sum([&](int c) { return __ldcg(a.P32 + c); });
        if (own) a.RV32[row].y = v;
        const double dv[1] = {own ? static_cast<double>(v) * r0 : 0.0};
        good = exchange<1, CLUSTER>(a, sh, dv, e);
        if (!good) break;
        if (t == 0) {
            const double rv = sh.tot[0], al = rho / rv;
            sh.mode = finite_nonzero(rv) && isfinite(al);
            sh.bc[0] = al;
        }
        __syncthreads();
        if (!sh.mode) {
            status = ST_BREAKDOWN;
            break;
        }
        alpha = sh.bc[0];
        const float ta = static_cast<float>(alpha);
        ++iter;
        // s, t = A s
        s = fmaf(-ta, v, r);
        tv = row_sum([&](int c) {
            const float2 q = __ldcg(a.RV32 + c);
            return fmaf(-ta, q.y, q.x);
        });
        const double sd = s, td = tv;
        // what: 0 nothing (the pass ends), 1 d, r and p, 2 an FP64 update
        if constexpr (MERGED) {
            const double ds[5] = {own ? td * sd : 0.0, own ? td * td : 0.0, own ? td * r0 : 0.0, own ? sd * sd : 0.0,
                                  own ? sd * r0 : 0.0};
            good = exchange<5, CLUSTER>(a, sh, ds, e);
            if (!good) break;
            if (t == 0) {  // the step of K_XRP_RU
                const double ts = sh.tot[0], tt = sh.tot[1], r0t = sh.tot[2], ss = sh.tot[3], r0s = sh.tot[4];
                const double om = ts / tt, rr = fmax(ss - om * ts, 0.0);
                int what = 0;
                sh.bc[0] = om;
                sh.bc[2] = rr;
                if (finite_nonzero(tt) && isfinite(om) && isfinite(rr) && !(rr > kDivergence2 * true_rr)) {
                    if (rr <= thr2 || rr < inner2 * rr_max || iter >= maxit) {
                        what = 2;
                    } else {
                        const double rho_new = r0s - om * r0t;
                        if (finite_nonzero(rho_new)) {
                            sh.bc[1] = (rho_new / rho) * (alpha / om);
                            sh.bc[3] = rho_new;
                            what = 1;
                        }
                    }
                    if (lead && iter - 1 < a.hist_cap) a.hist[iter - 1] = rr;
                }
                sh.mode = what;
            }
            __syncthreads();
        } else {
            const double ds[2] = {own ? td * sd : 0.0, own ? td * td : 0.0};
            good = exchange<2, CLUSTER>(a, sh, ds, e);
            if (!good) break;
            if (t == 0) {  // the step of K_XR
                const double om = sh.tot[0] / sh.tot[1];
                sh.mode = finite_nonzero(sh.tot[1]) && isfinite(om);
                sh.bc[0] = om;
            }
            __syncthreads();
            if (!sh.mode) {
                status = ST_BREAKDOWN;
                break;
            }
            const double rn = fmaf(-static_cast<float>(sh.bc[0]), tv, s);
            const double d2[2] = {own ? rn * r0 : 0.0, own ? rn * rn : 0.0};
            good = exchange<2, CLUSTER>(a, sh, d2, e);
            if (!good) break;
            if (t == 0) {  // the step of K_P_RU
                const double rho_new = sh.tot[0], rr = sh.tot[1];
                int what = 0;
                sh.bc[2] = rr;
                if (isfinite(rr) && !(rr > kDivergence2 * true_rr)) {
                    if (rr <= thr2 || rr < inner2 * rr_max || iter >= maxit) {
                        what = 2;
                    } else if (finite_nonzero(rho_new)) {
                        sh.bc[1] = (rho_new / rho) * (alpha / sh.bc[0]);
                        sh.bc[3] = rho_new;
                        what = 1;
                    }
                    if (lead && iter - 1 < a.hist_cap) a.hist[iter - 1] = rr;
                }
                sh.mode = what;
            }
            __syncthreads();
        }
        const int what = sh.mode;
        if (what == 0) {  // d is dropped: x stays as of the last update
            status = ST_BREAKDOWN;
            break;
        }
        omega = sh.bc[0];
        const float tw = static_cast<float>(omega);
        d = fmaf(tw, s, fmaf(ta, p, d));
        if (what == 1) {
            const float tb = static_cast<float>(sh.bc[1]);
            rho = sh.bc[3];
            rr_last = sh.bc[2];
            rr_max = fmax(rr_max, rr_last);
            r = fmaf(-tw, tv, s);
            p = fmaf(tb, fmaf(-tw, v, p), r);
        } else {
            // x += d and the true residual; its FP32 value replaces r (K_RU_APPLY, then K_P)
            x += static_cast<double>(d);
            d = 0.f;
            if (own) a.X[row] = x;
            good = exchange<0, CLUSTER>(a, sh, none, e);
            if (!good) break;
            rd = residual();
            r = static_cast<float>(rd);
            const double du[3] = {own ? rd * rd : 0.0, own ? static_cast<double>(r) * r0 : 0.0,
                                  own ? static_cast<double>(r) * r : 0.0};
            good = exchange<3, CLUSTER>(a, sh, du, e);
            if (!good) break;
            rd2 = sh.tot[0];
            const double rho_new = sh.tot[1], rr = sh.tot[2];
            rr_max = rd2;
            ++updates;
            stalls = rd2 > kStall2 * true_rr ? stalls + 1 : 0;
            true_rr = rd2;
            if (rd2 <= thr2) status = ST_CONVERGED;
            else if (!isfinite(rd2) || stalls >= kStallUpdates) status = ST_BREAKDOWN;
            else if (iter >= maxit) status = ST_MAXIT;
            if (status != ST_RUNNING) break;
            if (lead && iter - 1 < a.hist_cap) a.hist[iter - 1] = rr;
            rr_last = rr;
            if (t == 0) {
                double beta = 0.0;
                sh.mode = step_p(ST_RUNNING, iter, it0, maxit, -1.0, rho_new, rr, 0.0, rho, alpha, omega, false, beta);
                sh.bc[1] = beta;
            }
            __syncthreads();
            status = sh.mode;
            if (status != ST_RUNNING) break;
            rho = rho_new;
            p = fmaf(static_cast<float>(sh.bc[1]), fmaf(-tw, v, p), r);
        }
        publish();
        good = exchange<0, CLUSTER>(a, sh, none, e);
    }
    // (x holds every folded increment; the one since is zero or, after a breakdown, dropped)
    if (own) a.X[row] = x;
    if (good) good = exchange<0, CLUSTER>(a, sh, none, e);
    if (good) {
        const double res = residual();
        const double df[1] = {own ? res * res : 0.0};
        good = exchange<1, CLUSTER>(a, sh, df, e);
        true_rr = sh.tot[0];
    }
    if (lead) {
        sc->status = good ? status : ST_DEVICE_ERROR;
        sc->rr0 = restart ? rr0_in : bb;
        sc->bb = bb;
        sc->thr2 = thr2;
        sc->thr2_rec = -1.0;
        sc->iter = iter;
        sc->iter_start = it0;
        sc->updates = updates;
        sc->stalls = stalls;
        sc->bodies = 0;
        sc->arrivals = 0;
        sc->ru_flag = 0;
        sc->rr_last = rr_last;
        sc->true_rr = true_rr;
    }
}
