// pcg_resident.cuh -- the pressure solve of scenes whose chunks fit the SMs (included by pcg.cu after
// its helpers; FP64 and MIXED with the elementwise preconditioner).
//
// k_pcg_fast keeps every scene of the launch in step: one grid barrier and one pass over all
// partial sums per iteration, and every cell's state crosses L2 in every iteration.  A scene that
// fits the SMs needs neither:
//   - a block keeps its chunks for the whole solve.  r, w, s stay in registers, p, x, u and the
//     operator data in shared memory.  Only cells with a neighbour in another block write
//     (r, w, s, pc) to L2, at their list position, for those blocks to read.  Neighbours inside
//     the block take the owner's u from shared memory, computed once per cell instead of once per
//     neighbour;
//   - a block waits only for the blocks of its own scene, on the scene's own arrival counter.
// Scenes are packed into groups of at most gridDim.x block positions; a block takes its position
// of each group in turn, so small scenes run side by side and large ones one after another, each
// out of shared memory, instead of all of them streaming through L2.
//
// ms per solve, k_pcg_fast before -> here: MIXED 32^3 0.54 -> 0.30, 64^3 1.11 -> 0.66, 128^3 (0.50 M
// FLUID cells) 3.90 -> 2.15 (10.0 -> 5.5 us per iteration), FP64 77^3 1.76 -> 1.48; eight scenes of
// 32^3-128^3, two of them of 0.9 M cells, 24.5 -> 18.4.  What an iteration of the 128^3 dam break
// spends, in SM cycles of about 10,800: 2,300 own update and halo, 2,400 the operator (shared
// memory bandwidth: 11 words per cell), 900 block sums, 2,500-3,500 arrival and wait (a release, a
// reduction and an acquire through L2), 2,200 reading 291 partials and the fp64 divisions of alpha
// and beta.  At 64^3 the last three are 5,500 of 6,500 cycles.
//
// The arithmetic, the chunk of every cell, the entries of every thread and every summation tree
// are those of k_pcg_fast, so both kernels give the same bits.
#pragma once

__device__ __forceinline__ float4 ldcg4(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ double4 ldcg4(const double4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldcg(q), b = __ldcg(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

// Waits until `want` arrivals are counted.  Bounded: gives up, with the error words set, when nothing has
// moved for `timeout_ns`, or when another block has given up.  The beat counts the exchanges of all
// scenes, since a block of the scene that is waited for may still be busy with one of an earlier group.
__device__ __forceinline__ bool wait_arrivals(const unsigned* count, unsigned want, Barrier* bar, int* dev_error,
                                              unsigned long long timeout_ns) {
    unsigned spin = 0, beat = 0;
    unsigned long long t_start = 0;
    while (!arrived(ld_acquire_cnt(count), want)) {
        if ((++spin & 255u) != 0) continue;
        if (*(volatile int*)&bar->error) return false;
        const unsigned long long now = gtimer();
        const unsigned bt = *(volatile unsigned*)&bar->beat;
        if (t_start == 0 || bt != beat) {
            t_start = now;
            beat = bt;
        } else if (now - t_start > timeout_ns) {
            atomicExch(&bar->error, 1);
            if (dev_error) atomicExch(dev_error, 1);
            return false;
        }
    }
    return true;
}

// Self test of that wait, one block: an arrival that never comes, one that comes after three times
// the limit while others move, and an error of another block, with the count wrapping around at the
// first two arrivals.  1 into *err when it did as it should.  The latter two with a limit of at most 50 ms,
// so that the test of a long one takes little longer than the limit; the last has 5 ms more than half the
// limit, since the wait looks at the error every 256 polls.
__global__ void k_wait_selftest(Barrier* bar, unsigned* count, int* err, unsigned long long timeout_ns) {
    const int tid = threadIdx.x;
    const unsigned long long limit = timeout_ns < 50000000ull ? timeout_ns : 50000000ull;
    if (tid == 0) {
        *bar = Barrier{};
        *count = 0xffffffffu;
        const bool gave_up = !wait_arrivals(count, 1u, bar, nullptr, timeout_ns) && *(volatile int*)&bar->error == 1;
        *err = gave_up;
        *bar = Barrier{};
        __threadfence();
    }
    __syncthreads();
    if (tid == 32) {
        for (int i = 0; i < 6; ++i) {
            const unsigned long long t0 = gtimer();
            while (gtimer() - t0 < limit / 2) __nanosleep(1000);
            atomicAdd(&bar->beat, 1u);
        }
        red_release_add(count, 2u);
    } else if (tid == 0) {
        const bool came = wait_arrivals(count, 1u, bar, nullptr, limit) && *(volatile int*)&bar->error == 0;
        atomicExch(&bar->error, 1);
        const unsigned long long t0 = gtimer();
        const bool left = !wait_arrivals(count, 2u, bar, nullptr, limit) && gtimer() - t0 < limit / 2 + 5000000ull;
        *err = *err && came && left;
    }
}

// One block per SM: two halves of kPcgThreads threads, each with one chunk or more.  Fewer arrivals and
// pollers make the barrier cheaper than two blocks per SM do (148 against 291 blocks: 2.2 against
// 2.9 us for an arrival, the wait and the reading of three sums per chunk).
constexpr int kResThreads = 2 * kPcgThreads;

// One block's part in one scene's solve: C chunks per half, Q rounds of one cell per thread in
// each (csize <= 256 Q).  BIG: blocks of up to four full-size chunks, whose (p, x), cell indices and
// halo cells stay in global memory, read ahead of use.  False when a wait gave up.
template <int MODE, int Q, int C, bool BIG>
__device__ __forceinline__ bool res_scene(const PcgArgs& A, int sc, int v) {
    using T = typename VT<MODE>::T;
    using T2 = typename V2<T>::type;
    using T4 = typename V4<T>::type;
    constexpr int R = Q * C, kWarps = kPcgThreads / 32;
    // halo entries of a thread loaded ahead of alpha and beta, in registers
    constexpr int kAhead = R <= 2 ? 2 : (MODE == kFp64 ? 2 : (BIG ? 4 : 5));
    const DevState& S = A.S;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int half = tid / kPcgThreads, htid = tid % kPcgThreads, hwid = htid >> 5;
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double dsum[2 * C][3][kWarps], total[3];
    __shared__ int s_nhalo;
    // the scene's solver state, kept by thread 0; the others read alpha, beta and stop
    __shared__ struct {
        double bb, rr, rho, alpha, beta, target, rr_out;
        int iters, outer, converged, stop;
    } st;
    const T* pcv = MODE == kFp64 ? (const T*)(const void*)A.pc64 : (const T*)(const void*)A.pc32;
    T4* const Av0 = (T4*)A.va0;
    T4* const Av1 = (T4*)A.va1;
    const unsigned long long tmo = A.timeout_ns;
    const SceneDev& D = S.scenes[sc];
    const int4 pl = A.res[sc];
    // this block's first chunk and its chunks (cpb for all blocks but perhaps the last); half h
    // has the chunks ch0 + h, ch0 + h + 2, ...
    const int nch = pl.z, cpb = (nch + pl.y - 1) / pl.y;
    const int ch0 = (v - pl.x) * cpb;
    const int n = D.n;
    const int nf = A.sc[sc].nf, csize = A.sc[sc].csize;
    // list positions of the block: [t0, t0 + blen)
    const long long t0 = A.fl_pref[sc] + (long long)ch0 * csize;
    const int blen = min(cpb * csize, nf - ch0 * csize);
    // round q of this thread: whether it has a cell, and its position in the block
    auto cell_of = [&](int q, int& o) -> bool {
        const int i = htid + (q % Q) * kPcgThreads;
        o = (half + 2 * (q / Q)) * csize + i;
        return i < csize && o < blen;
    };
    // Shared memory: per cell (p, x), the diagonal, pc, u and three words of neighbour positions in
    // u (x, y, z pairs of 14 bits; bit 28 of the first: some neighbour lies in another block); u
    // continues with the halo -- the neighbours in other blocks -- and a slot that stays 0 for
    // neighbours that are not FLUID; the halo's list positions, where its owners publish.  BIG: these in
    // hlist, which has six for every list position (a slot a cell was too few for a scene's last block,
    // often a short one: its neighbours are mostly not its own, and the scene was handed over).
    const int cells = cpb * csize, hcap = res_halo_slots(MODE, cells, BIG), zero = cells + hcap;
    T2* const px = BIG ? (T2*)A.vb + t0 : reinterpret_cast<T2*>(dyn);
    T* const dgs = reinterpret_cast<T*>(dyn + (BIG ? 0 : sizeof(T2) * cells));
    T* const pcs = dgs + cells;
    T* const ub = pcs + cells;
    uint32_t* const nw = reinterpret_cast<uint32_t*>(ub + zero + 1);
    uint32_t* const hpos = BIG ? A.hlist + 6 * t0 : nw + 3 * cells;
    const uint32_t* const cs = A.fl + t0;
    const unsigned arrivals = (unsigned)pl.y;
    unsigned* const count = A.res_count + 32 * (size_t)sc;
    unsigned epoch = 0;
    // The scene's partial sums, in two sets used in turn: a block can be one exchange ahead
    // of another block of its scene, never two.
    auto partial = [&](unsigned e) {
        return A.partial + (e & 1 ? 3 * (size_t)A.max_chunks : 0) + 3 * (size_t)pl.w;
    };
    // Publishes the `nsum` sums of this block's chunks and waits for the scene's other blocks
    // (nsum 0: a barrier).  False when the wait gave up.
    auto arrive_wait = [&](int nsum, double (&a)[C], double (&b)[C], double (&c)[C]) -> bool {
        ++epoch;
        if (nsum > 0) {
#pragma unroll
            for (int j = 0; j < C; ++j) {
                a[j] = warp_sum(a[j]);
                b[j] = warp_sum(b[j]);
                if (nsum > 2) c[j] = warp_sum(c[j]);
            }
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    dsum[half + 2 * j][0][hwid] = a[j];
                    dsum[half + 2 * j][1][hwid] = b[j];
                    dsum[half + 2 * j][2][hwid] = c[j];
                }
            }
        }
        __syncthreads();
        if (hwid < nsum) {
#pragma unroll
            for (int j = 0; j < C; ++j) {
                // block_sum2's second step: its tree over a warp whose lanes past the eight warp
                // sums hold zeros
                const int i = half + 2 * j;
                double x = lane < kWarps ? dsum[i][hwid][lane] : 0.0;
                static_assert(kWarps == 8, "three steps sum the warps");
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
                if (lane == 0 && i < cpb && ch0 + i < nch) partial(epoch)[hwid * nch + ch0 + i] = x;
            }
        }
        __syncthreads();
        bool ok = true;
        if (tid == 0) {
            // release: orders the block's writes (collected by the barrier above) before the
            // arrival; acquire: the others' writes before what follows the barrier below
            red_release_add(count, 1u);
            ok = wait_arrivals(count, epoch * arrivals, A.bar, S.dev_error, tmo);
            if (ch0 == 0) atomicAdd(&A.bar->beat, 1u);
        }
        return __syncthreads_and(ok) != 0;
    };
    // The scene's sums into total[], then `f` by thread 0; ends with a block barrier.  `ahead`
    // issues loads to overlap with it: after those of the partials, but before them where their
    // registers and those of the partials together would spill.
    auto sums = [&](int nsum, auto&& ahead, auto&& f) {
        constexpr int kU = ((BIG ? kResBigChunks : kResMaxChunks) + 31) / 32;
        // scene_sum3's order: partials a lane at a time, ascending
        if (R > 2) ahead();
        double x[kU];
        if (wid < nsum) {
            const double* const p0 = partial(epoch) + wid * nch;
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int c0 = u * 32 + lane;
                x[u] = c0 < nch ? __ldcg(p0 + c0) : 0.0;
            }
        }
        if (R <= 2) ahead();
        if (wid < nsum) {
            double y = 0.0;
#pragma unroll
            for (int u = 0; u < kU; ++u) y += x[u];
            y = warp_sum(y);
            if (lane == 0) total[wid] = y;
        }
        if (wid < 3) asm volatile("bar.sync 1, 96;" ::: "memory");
        if (tid == 0) f();
        __syncthreads();
    };

    // ---- the block's operator data --------------------------------------------------------
    if (tid == 0) {
        st = {};
        s_nhalo = 0;
        ub[zero] = (T)0;
    }
    __syncthreads();
    for (int q = 0; q < R; ++q) {
        int o;
        if (!cell_of(q, o)) continue;
        const uint4 rc = A.rec[t0 + o];
        const uint32_t c = rc.x, m = rc.y;
        T dg;
        dec_diag(rc, dg);
        int i, j, kk;
        cell_ijk(D, (long long)c - D.c_begin, i, j, kk);
        bool out = false;
        auto code = [&](int d, int a, int b, int e) -> uint32_t {
            if (!((m >> d) & 1u)) return (uint32_t)zero;
            const long long p = (long long)A.flscan[D.c_begin + list_order(MODE, n, a, b, e)] - t0;
            if (p >= 0 && p < blen) return (uint32_t)p;
            out = true;
            // one slot for each active lane, in lane order
            const unsigned act = __activemask();
            const int lead = __ffs(act) - 1;
            int h = 0;
            if (lane == lead) h = atomicAdd(&s_nhalo, __popc(act));
            h = __shfl_sync(act, h, lead) + __popc(act & ((1u << lane) - 1u));
            if (h < hcap) hpos[h] = (uint32_t)(p + t0);
            return (uint32_t)(cells + h);
        };
        const uint32_t x0 = code(0, i - 1, j, kk), x1 = code(1, i + 1, j, kk);
        const uint32_t y0 = code(2, i, j - 1, kk), y1 = code(3, i, j + 1, kk);
        const uint32_t z0 = code(4, i, j, kk - 1), z1 = code(5, i, j, kk + 1);
        dgs[o] = dg;
        pcs[o] = pcv[c];
        nw[o] = x0 | x1 << 14 | (out ? 1u << 28 : 0u);
        nw[cells + o] = y0 | y1 << 14;
        nw[2 * cells + o] = z0 | z1 << 14;
    }
    // (every thread reads back only its own entries of dgs, pcs, nw and px)
    __syncthreads();
    const int nhalo = s_nhalo;
    // More neighbours in other blocks than slots for them (liquid in sheets along the bricks' faces):
    // the scene is left to the streaming kernel.  Its blocks learn of it at their first exchange.
    if (tid == 0 && nhalo > hcap) atomicExch(count + 1, 1u);

    const T scale = (T)(1.0 / (double)D.ax_h);
    const int cap = A.max_iters > 0 ? A.max_iters : n * n * n;
    T r[R], w[R], sv[R];

    for (int outer = 0;; ++outer) {
        // ---- residual r = b - A x, |b|^2 ----------------------------------------------------
        double a0[C], a1[C], a2[C];
        auto clear = [&] {
#pragma unroll
            for (int j = 0; j < C; ++j) a0[j] = a1[j] = a2[j] = 0.0;
        };
        clear();
#pragma unroll
        for (int j = 0; j < C; ++j)
            for (int q = j * Q; q < (j + 1) * Q; ++q) {
                int o;
                if (!cell_of(q, o)) break;
                const long long c = cs[o];
                const double bv = (double)S.D[c];
                const double xc = __ldcg(S.P64 + c);
                const double ax = ax_diag<double>(A, D, c, xc, [&](long long p) { return __ldcg(S.P64 + p); });
                const double rv = bv - ax;
                if (MODE == kMixed)
                    A.r64[c] = rv;
                else
                    ((T*)A.r)[c] = (T)rv;
                a0[j] += rv * rv;
                a1[j] += bv * bv;
            }
        if (!arrive_wait(2, a0, a1, a2)) return false;
        if (outer == 0 && *(volatile unsigned*)(count + 1)) {
            if (ch0 == 0 && tid == 0) {
                A.res[sc].x = kNotResident;
                atomicAdd(&A.ctl->nstream, 1);
            }
            return true;
        }
        sums(2, [] {}, [&] {
            const double rr = total[0];
            if (outer == 0) st.bb = total[1];
            st.rr_out = rr;
            if (MODE == kMixed) st.outer += 1;
            const double lim2 = A.tol * A.tol * st.bb;
            const double abs_eps = (double)(1.0e-2f * (float)(n * n * n));
            bool conv = false;
            if (A.stop_rule == ARIEL_STOP_REL)
                conv = rr <= lim2;
            else if (MODE == kMixed)
                conv = outer > 0 && rr <= abs_eps;
            if (conv) {
                st.stop = 1;
                st.converged = 1;
            } else if (MODE == kMixed && (st.outer > A.max_outer || st.iters >= cap)) {
                st.stop = 1;
            }
            if (st.stop) return;
            st.rr = rr;
            if (MODE == kMixed) {
                // the correction solve stops at the final tolerance itself (its fp32
                // residual); the true residual then decides whether another sweep is needed
                const double a = A.inner_tol * A.inner_tol * rr;
                const double b = A.stop_rule == ARIEL_STOP_REL ? lim2 : 0.0;
                st.target = a > b ? a : b;
            } else {
                st.target = A.stop_rule == ARIEL_STOP_REL ? lim2 : abs_eps;
            }
        });
        if (st.stop) break;
        // ---- u = M r, w = A u, p = 0 ----------------------------------------------------
        auto r0 = [&](long long q) -> T {
            return MODE == kMixed ? (T)__ldcg(A.r64 + q) : __ldcg((const T*)A.r + q);
        };
        clear();
#pragma unroll
        for (int q = 0; q < R; ++q) {
            int o;
            if (cell_of(q, o)) {
                const long long c = cs[o];
                const uint32_t m = A.mask[c];
                const T rv = r0(c), pcc = pcs[o];
                const T uv = (rv * pcc) * pcc;
                T acc = dgs[o] * uv;
#pragma unroll
                for (int d = 0; d < 6; ++d)
                    if (m & (1u << d)) {
                        const long long qq = c + nb_off(d, n);
                        const T pq = pcv[qq];
                        acc -= (r0(qq) * pq) * pq;
                    }
                const T wv = acc * scale;
                const T xv = MODE == kMixed ? (T)0 : (T)S.P64[c];
                if (nw[o] >> 28) st4(Av0 + t0 + o, mk4<T>(rv, wv, (T)0, pcc));
                r[q] = rv;
                w[q] = wv;
                sv[q] = (T)0;
                px[o] = mk2<T>((T)0, xv);
                a0[q / Q] += (double)rv * (double)uv;
                a1[q / Q] += (double)wv * (double)uv;
            }
        }
        if (!arrive_wait(2, a0, a1, a2)) return false;
        // BIG: this thread's halo positions, and (p, x) a group of rounds ahead of use
        constexpr int kGroup = 4;
        uint32_t hreg[BIG ? kAhead : 1];
        T2 bn[BIG ? kGroup : 1];
        auto load_px = [&](int q0) {
            if constexpr (BIG) {
#pragma unroll
                for (int u = 0; u < kGroup; ++u) {
                    int o;
                    if (q0 + u < R && cell_of(q0 + u, o)) bn[u] = px[o];
                }
            }
        };
        if constexpr (BIG) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int h = tid + u * kResThreads;
                hreg[u] = h < nhalo ? hpos[h] : 0u;
            }
        }
        // ---- iterations: k_pcg_fast's update of (r, w, s, p, x, u), one exchange each ---
        // The halo comes from L2 as its owners' (r, w, s, pc) of the last iteration; the loads
        // are issued as soon as the wait ends, ahead of alpha and beta.
        for (int it = 0;; ++it) {
            const T4* const Ac = (it & 1) ? Av1 : Av0;
            T4* const mine = ((it & 1) ? Av0 : Av1) + t0;
            T4 eh[kAhead];
            auto load_halo = [&] {
#pragma unroll
                for (int u = 0; u < kAhead; ++u) {
                    const int h = tid + u * kResThreads;
                    if (h < nhalo) eh[u] = ldcg4(Ac + (BIG ? hreg[u] : hpos[h]));
                }
                if (BIG) load_px(0);
            };
            if (it == 0)
                sums(2, load_halo, [&] {
                    st.rho = total[0];
                    st.alpha = total[1] != 0.0 ? total[0] / total[1] : 0.0;
                    st.beta = 0.0;
                    st.stop = 0;
                });
            else
                sums(3, load_halo, [&] {
                    const double g = total[0], d = total[1];
                    st.iters += 1;
                    st.rr = total[2];
                    const bool conv = total[2] <= st.target;
                    if (conv || st.iters >= cap) {
                        if (MODE != kMixed) st.converged = conv;
                        st.stop = 1;
                        return;
                    }
                    const double beta = st.rho != 0.0 ? g / st.rho : 0.0;
                    const double den = d - (st.alpha != 0.0 ? beta * g / st.alpha : 0.0);
                    st.beta = beta;
                    st.alpha = den != 0.0 ? g / den : 0.0;
                    st.rho = g;
                });
            if (st.stop) break;
            const T al = (T)st.alpha, bt = (T)st.beta;
            auto u_of = [&](const T4& e) -> T {
                const T sq = e.y + bt * e.z;
                const T rq = e.x - al * sq;
                return (rq * e.w) * e.w;
            };
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int h = tid + u * kResThreads;
                if (h < nhalo) ub[cells + h] = u_of(eh[u]);
            }
            // (BIG: hpos made anew from t0, which is at hand: kept across the iterations, its registers
            // are spilled elsewhere, 160^3 6.0 -> 6.4 ms)
            long long tb = t0;
            if (BIG) asm volatile("" : "+l"(tb));
            const uint32_t* const hp = BIG ? A.hlist + 6 * tb : hpos;
            for (int h = tid + kAhead * kResThreads; h < nhalo; h += kResThreads)
                ub[cells + h] = u_of(ldcg4(Ac + hp[h]));
            T2 bc[BIG ? kGroup : 1];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if constexpr (BIG) {
                    if (q % kGroup == 0) {
#pragma unroll
                        for (int u = 0; u < kGroup; ++u) bc[u] = bn[u];
                        load_px(q + kGroup);
                    }
                }
                int o;
                if (cell_of(q, o)) {
                    const T pc = pcs[o];
                    const T2 b = BIG ? bc[BIG ? q % kGroup : 0] : px[o];
                    const T s1 = w[q] + bt * sv[q];
                    const T ui = (r[q] * pc) * pc;
                    const T pv = ui + bt * b.x;
                    const T xv = b.y + al * pv;
                    const T rn = r[q] - al * s1;
                    sv[q] = s1;
                    r[q] = rn;
                    px[o] = mk2<T>(pv, xv);
                    ub[o] = (rn * pc) * pc;
                }
            }
            __syncthreads();
            clear();
#pragma unroll
            for (int q = 0; q < R; ++q) {
                int o;
                if (cell_of(q, o)) {
                    const uint32_t nb[3] = {nw[o], nw[cells + o], nw[2 * cells + o]};
                    const T un = ub[o];
                    T a = dgs[o] * un;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        a -= ub[nb[d] & 0x3fffu];  // 0 where the neighbour is not FLUID
                        a -= ub[nb[d] >> 14 & 0x3fffu];
                    }
                    const T wn = a * scale;
                    w[q] = wn;
                    if (nb[0] >> 28) st4(mine + o, mk4<T>(r[q], wn, sv[q], pcs[o]));
                    if (MODE == kMixed) {
                        // products of two floats are exact in double, so the fused sums round as
                        // the separate ones
                        const double dr = (double)r[q], du = (double)un;
                        a0[q / Q] = __fma_rn(dr, du, a0[q / Q]);
                        a1[q / Q] = __fma_rn((double)wn, du, a1[q / Q]);
                        a2[q / Q] = __fma_rn(dr, dr, a2[q / Q]);
                    } else {
                        a0[q / Q] += (double)r[q] * (double)un;
                        a1[q / Q] += (double)wn * (double)un;
                        a2[q / Q] += (double)r[q] * (double)r[q];
                    }
                }
            }
            if (!arrive_wait(3, a0, a1, a2)) return false;
        }
        __syncthreads();
        if (tid == 0) st.stop = 0;
        // fold the solve's x back: MIXED adds the correction to x64, FP64 stores x64
        for (int q = 0; q < R; ++q) {
            int o;
            if (!cell_of(q, o)) continue;
            const uint32_t c = cs[o];
            S.P64[c] = MODE == kMixed ? S.P64[c] + (double)px[o].y : (double)px[o].y;
        }
        if (MODE != kMixed) break;
        if (!arrive_wait(0, a0, a1, a2)) return false;
    }
    if (ch0 == 0 && tid == 0) {
        PcgScene o = load_sc(A.sc + sc);
        o.bb = st.bb;
        o.rr = st.rr;
        o.rho = st.rho;
        o.alpha = st.alpha;
        o.beta = st.beta;
        o.rr_out = st.rr_out;
        o.target = st.target;
        o.iters = st.iters;
        o.outer = st.outer;
        o.done = 1;
        o.inner_done = 1;
        o.converged = st.converged;
        A.sc[sc] = o;
        PcgTotals& Tt = A.totals[sc];
        const int sweeps = MODE == kMixed ? st.outer : 1;
        Tt.solves += 1;
        Tt.iterations += st.iters;
        Tt.outer += sweeps;
        Tt.cell_iterations += (double)nf * (double)st.iters;
        Tt.cell_outer += (double)nf * (double)sweeps;
        Tt.not_converged += st.converged ? 0 : 1;
    }
    for (int q = 0; q < R; ++q) {
        int o;
        if (!cell_of(q, o)) continue;
        const uint32_t c = cs[o];
        S.P[c] = (float)S.P64[c];
    }
    return true;
}

// One kernel per class of scenes (res_class), so that none carries the code and the registers of
// rounds that its threads do not have.
template <int MODE, int CLASS>
__global__ void __launch_bounds__(kResThreads, 1) k_pcg_res(PcgArgs A) {
    if (A.ctl->any_ordered) return;  // the ordered preconditioner runs in k_pcg
    const DevState& S = A.S;
    const int tid = threadIdx.x, nvirt = A.ctl->nvirt[CLASS], k = S.k;
    __shared__ int s_scene;
    if (blockIdx.x == 0)
        for (int s = tid; s < k; s += kResThreads) {
            const int4 e = A.res[s];
            if (e.x < 0 || e.z > 0 || res_class(k, A.sc[s].csize, A.res[s].z) != CLASS) continue;
            // a scene without FLUID cells: solved as it is
            PcgScene o = load_sc(A.sc + s);
            o.outer = MODE == kMixed ? 1 : 0;
            o.done = o.inner_done = o.converged = 1;
            A.sc[s] = o;
            A.totals[s].solves += 1;
            A.totals[s].outer += 1;
        }
    for (int v = blockIdx.x; v < nvirt; v += gridDim.x) {
        __syncthreads();
        if (tid == 0) s_scene = -1;
        __syncthreads();
        for (int s = tid; s < k; s += kResThreads) {
            const int4 e = A.res[s];
            if (v >= e.x && v < e.x + e.y && res_class(k, A.sc[s].csize, A.res[s].z) == CLASS) s_scene = s;
        }
        __syncthreads();
        const int sc = s_scene;
        if (sc < 0) continue;  // no chunk for this block in this group
        if (!res_scene<MODE, res_rounds(CLASS), res_chunks(CLASS), CLASS == kResBig>(A, sc, v)) return;
    }
}
