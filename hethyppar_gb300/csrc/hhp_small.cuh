// hhp_small.cuh -- the FP64 BiCGStab loop of a small system as one cooperative kernel.
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
// block polls (1.2 us; polling all blocks' records instead took 3.3 us at 152 blocks). Every such wait is bounded: one that runs out sets the
// context's error word and the block leaves, as the others then do. All blocks add the same numbers in
// the same order, so they compute the same scalars bit for bit and take the same branches.
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
constexpr int kSmallPolls = 1 << 20;      // reads of the count before giving up (~0.5 us each)

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
    double *rec;              // 2 sets of kSmallQ * grid partial sums, used in turn
    unsigned *arrived;        // blocks that have arrived, over all exchanges (zero at the launch)
    double *hist;
    int hist_cap;
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

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One exchange of NQ sums (NQ = 0: a barrier), number e = 1, 2, ... of the launch; the sums in
// sh.tot. The blocks' earlier global stores are visible to every block after it. The buffers of e are
// written again at e + 2, which a block reaches only after every block has arrived at e + 1, that is
// has read e's. Returns false when the wait ran out (uniform across the block).
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
            const unsigned target = e * static_cast<unsigned>(G);
            unsigned seen = 0;
            for (int i = 0; i < kSmallPolls && seen < target; ++i)
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.arrived) : "memory");
            sh.ok = seen >= target;
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

template <bool MERGED, bool CLUSTER>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small(const __grid_constant__ SmallArgs a) {
    extern __shared__ double s_mat[];  // val[K][rows], then col[K][rows]
    __shared__ SmallShared sh;
    const int t = threadIdx.x, pos = blockIdx.x * a.rows + t;
    const bool own = t < a.rows && pos < a.n, lead = blockIdx.x == 0 && t == 0;
    const int row = own && a.pos_row ? a.pos_row[pos] : pos;
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
    // sum over the row's entries, in order, of val * get(col): eight gathers in flight, as many steps as
    // the warp's longest row has (a multiply-add that no lane needs still takes the FP64 pipe's slot)
    const int kmax = __reduce_max_sync(0xffffffffu, len);
    auto row_sum = [&](auto get) {
        double acc = 0.0;
        auto steps = [&](auto n, int k) {
            constexpr int N = decltype(n)::value;
            double g[N];
#pragma unroll
            for (int u = 0; u < N; ++u) g[u] = k + u < len ? get(sc_[(k + u) * ld]) : 0.0;
#pragma unroll
            for (int u = 0; u < N; ++u)
                if (k + u < len) acc = fma(sv[(k + u) * ld], g[u], acc);
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
    };
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
