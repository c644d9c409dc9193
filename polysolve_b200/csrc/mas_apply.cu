// MAS preconditioner apply (sm_100a): z = sum_l P_l A_l^-1 P_l^T r.
//
// The reference (MASPreconditioner.cu:1099-1164) zeroes two multi-level vectors, restricts with
// warp segmented sums plus FP64 atomics, multiplies every level's packed 96 x 96 inverse with one
// 96-thread CTA each (symv_upper_packed, :665-705), and prolongs in a third kernel. Here a PCG
// iteration's apply is two launches:
//
//  * the level-0 restriction (per-bank sums of each connected component) is fused into the kernel
//    that produces r (update_xr; k_restrict after a true-residual SpMV);
//  * k_coarse_levels: every coarse level above the first in one launch -- one CTA per third-level
//    node sums its second-level children (a warp each, lane per child) and then itself, so both
//    levels take one round; the last CTA to finish (atomic ticket) sums a fourth level;
//  * k_mas_apply: persistent warps stream every inverse -- the level-0 subdomain matrices, then
//    the active coarse matrices -- through shared memory with cp.async.bulk (two stages per warp,
//    mbarrier completion) and write z0 = A_0^-1 r and zc = A_l^-1 rc with per-CTA partial dots;
//    the last CTA (atomic ticket) sums them in a fixed order and runs the reference's per-iteration
//    scalar work and convergence test. The prolongation z = z0 + P zc is fused into the p update
//    (update_p): PCG uses z only there and in r . z = r . z0 + (P^T r) . zc.
//
// Inverses are stored tile-packed (mas_internal.h): the same N (N + 1) / 2 values as packed upper
// storage, in 32 x 32 tiles that shared memory serves without bank conflicts by rows and by columns,
// so a lane forms its whole row of the product from either side of the diagonal and no sum crosses
// lanes. Storage is FP64, FP32 or binary16 with one power-of-two scale per matrix (FP32 arithmetic
// for both reduced formats; binary16 runs on the tensor cores).

#include "mas_apply.cuh"

namespace pmas
{
    namespace
    {
        // Partial dots of the apply, per CTA: r.z0 and r.z0_old over banks with coupled rows, the
        // same over banks of isolated rows, rc.zc and rc.zc_old over the coarse matrices.
        constexpr int APPLY_PARTS = 6;

        // Whether the solve has stopped, for a whole CTA; read past L1 (see mas_apply_body) and once, not by each
        // of some 2,000 warps from the same line.
        __device__ __forceinline__ bool solve_done(const PcgState *st)
        {
            __shared__ int stop;
            if (threadIdx.x == 0)
                stop = __ldcg(&st->done);
            __syncthreads();
            return warp_uniform(stop) != 0;
        }

        // Work item m: m < banks -> level-0 matrix m (input r, output z0); otherwise coarse matrix
        // g = coarse_active[m - banks] (matrix banks + g, input rc, output zc, 32 coarse nodes
        // from g * 32). mode 0: plain apply; 1: initial PCG apply (rz0); 2: PCG iteration.
        // prefetch_first: issue the first two inverse copies before waiting for the predecessor
        // (a chained launch of one system); otherwise a finished solve returns before any copy
        // (the batched launch, where most CTAs may belong to finished systems).
        //
        // Both forms below return with part[] the thread's partial dots, or false on a solve that is
        // already done. This one: FP32 and binary16 inverses, a warp per matrix.
        template <int BD, class Store, int MODE>
        __device__ __forceinline__ bool mas_apply_warps(const MasView &mas, const double *__restrict__ r,
                                                        double *__restrict__ z0, PcgState *st, const PcgConfig &cfg,
                                                        Cta cta, bool early, double (&part)[APPLY_PARTS])
        {
            using L = ApplyLayout<BD, Store>;
            using Real = typename L::Real;
            constexpr int N = L::N, S = L::S, WARPS = L::WARPS;
            extern __shared__ __align__(128) unsigned char smem[];
            const int w = warp_index(), lane = threadIdx.x & 31;
            unsigned char *base = smem + (size_t)w * L::TEAM_BYTES;
            Store *stage0 = reinterpret_cast<Store *>(base);
            Store *stage1 = reinterpret_cast<Store *>(base + L::STAGE_BYTES);
            Real *xs = reinterpret_cast<Real *>(base + 2 * L::STAGE_BYTES);
            __half *xh = reinterpret_cast<__half *>(base + 2 * L::STAGE_BYTES);
            __half *xl = xh + N;
            float *ys = reinterpret_cast<float *>(base + 2 * L::STAGE_BYTES + 4 * N);
            uint64_t *bar = reinterpret_cast<uint64_t *>(base + 2 * L::STAGE_BYTES + L::XS_BYTES);
            const Store *__restrict__ inv = static_cast<const Store *>(mas.inv);
            const int banks = mas.banks;
            const int items = banks + mas.n_coarse_active;
            const int total_warps = cta.n * WARPS;
            const int gw = cta.x * WARPS + w;
            int *errp = st ? &st->error : nullptr;
            const bool pr = (MODE == 2) && cfg.polak_ribiere;
            // Matrix index and input vector of an item (coarse vectors: g * N).
            auto mat_of = [&](int m) { return m < banks ? m : banks + mas.coarse_active[m - banks]; };
            auto in_of = [&](int m) -> const double * {
                return m < banks ? r + (size_t)m * N : mas.rc + (size_t)(mat_of(m) - banks) * N;
            };

            const uint64_t pol = l2_evict_first_policy(); // the inverses stream, the vectors stay
            if (lane == 0)
            {
                mbar_init(&bar[0], 1);
                mbar_init(&bar[1], 1);
                fence_mbar_init();
            }
            __syncwarp();
            if (lane == 0)
            {
                if (gw < items)
                    bulk_load_stream(stage0, inv + (size_t)mat_of(gw) * S, L::STAGE_BYTES, &bar[0], pol);
                if (gw + total_warps < items)
                    bulk_load_stream(stage1, inv + (size_t)mat_of(gw + total_warps) * S, L::STAGE_BYTES, &bar[1], pol);
            }
            // Copies issued and not yet consumed, per stage (drained if a wait gives up).
            bool pending[2] = {gw < items, gw + total_warps < items};
            // The first two inverses are on their way (no kernel of a solve writes them); now wait
            // for the predecessor (launched chained in a PCG iteration), or at the first coarse matrix.
            if (!early)
                pdl_wait();
            if (MODE != 0 && solve_done(st))
            {
                if (lane == 0)
                    mbar_drain(bar, pending, {0u, 0u});
                __syncwarp();
                return false;
            }
            uint32_t phase0 = 0, phase1 = 0;
            bool ok = true;
            // Input (and binary16 scale) of the current item, prefetched one item ahead.
            double r_next[BD], scale_next = 1.0;
            if (gw < items)
            {
                if (early && gw >= banks)
                    pdl_wait();
                const double *in = in_of(gw);
#pragma unroll
                for (int t = 0; t < BD; ++t)
                    r_next[t] = __ldcg(in + t * 32 + lane);
                if (StoreTraits<Store>::SCALED)
                    scale_next = mas.inv_scale[mat_of(gw)];
            }
            int k = 0;
            for (int m = gw; m < items; m += total_warps, ++k)
            {
                const bool s1 = (k & 1) != 0;
                Store *stage = s1 ? stage1 : stage0;
                uint64_t *b = s1 ? &bar[1] : &bar[0];
                const bool coarse = m >= banks;
                const int mat = mat_of(m);
                double *out = coarse ? mas.zc + (size_t)(mat - banks) * N : z0 + (size_t)m * N;
                double r64[BD];
#pragma unroll
                for (int t = 0; t < BD; ++t)
                    r64[t] = r_next[t];
                const double mscale = scale_next;
                double xscale = 1.0; // binary16 input: x * xscale split into hi + lo
                if constexpr (L::MMA)
                {
                    xscale = half_scale<BD>(r64);
#pragma unroll
                    for (int t = 0; t < BD; ++t)
                    {
                        const float v = (float)(r64[t] * xscale);
                        const __half h = __float2half_rn(v);
                        xh[t * 32 + lane] = h;
                        xl[t * 32 + lane] = __float2half_rn(v - __half2float(h));
                    }
                }
                else
                {
#pragma unroll
                    for (int t = 0; t < BD; ++t)
                        xs[t * 32 + lane] = (Real)r64[t];
                }
                const int mnext = m + total_warps;
                if (mnext < items)
                {
                    if (early && mnext >= banks)
                        pdl_wait();
                    const double *in = in_of(mnext);
#pragma unroll
                    for (int t = 0; t < BD; ++t)
                        r_next[t] = __ldcg(in + t * 32 + lane);
                    if (StoreTraits<Store>::SCALED)
                        scale_next = mas.inv_scale[mat_of(mnext)];
                }
                double zold[BD];
                if (pr)
#pragma unroll
                    for (int t = 0; t < BD; ++t)
                        zold[t] = out[t * 32 + lane];
                __syncwarp();
                if (!mbar_wait_bounded(b, s1 ? phase1 : phase0, errp, cfg.wait_limit))
                {
                    ok = false;
                    break;
                }
                pending[s1 ? 1 : 0] = false;
                if (s1)
                    phase1 ^= 1u;
                else
                    phase0 ^= 1u;
                // Coarse matrices of isolated rows are exactly the identity: z = r, unrounded.
                const bool ident = coarse && warp_uniform(mas.identity[mat - banks]);
                Real yr[BD];
                if (!ident)
                {
                    if constexpr (L::MMA)
                        symv_mma16<BD>(stage, xh, xl, ys, lane, yr);
                    else
                        symv_tiles<BD>(stage, xs, lane, yr);
                }
                __syncwarp();
                const int mn = m + 2 * total_warps;
                if (mn < items)
                {
                    if (lane == 0)
                    {
                        fence_proxy_async_smem();
                        bulk_load_stream(stage, inv + (size_t)mat_of(mn) * S, L::STAGE_BYTES, b, pol);
                    }
                    pending[s1 ? 1 : 0] = true;
                }
                const double scale = StoreTraits<Store>::SCALED ? mscale / xscale : 1.0;
                double d0 = 0.0, d1 = 0.0;
#pragma unroll
                for (int t = 0; t < BD; ++t)
                {
                    double zv;
                    if (ident)
                        zv = r64[t];
                    else
                        zv = StoreTraits<Store>::SCALED ? (double)yr[t] * scale : (double)yr[t];
                    out[t * 32 + lane] = zv;
                    d0 = fma(zv, r64[t], d0);
                    if (pr)
                        d1 = fma(zold[t], r64[t], d1);
                }
                // Fixed slots (no dynamic indexing, so part[] stays in registers).
                if (coarse)
                {
                    part[4] += d0;
                    part[5] += d1;
                }
                else if (m >= mas.first_iso_bank)
                {
                    part[2] += d0;
                    part[3] += d1;
                }
                else
                {
                    part[0] += d0;
                    part[1] += d1;
                }
            }
            if (!ok)
            {
                // Drain this warp's outstanding copies (bounded) before leaving.
                if (lane == 0)
                    mbar_drain(bar, pending, {phase0, phase1});
                __syncwarp();
            }
            return true;
        }

        // Barrier of the warps of team `team` (named barriers 1, 2, ...).
        template <int TEAM>
        __device__ __forceinline__ void team_sync(int team)
        {
            if (TEAM == 1)
                __syncwarp();
            else
                asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(TEAM * 32) : "memory");
        }

        // FP64 inverses: a team of BD warps per matrix, warp t of the team rows 32 t .. 32 t + 31 (a
        // lane's row needs no sum across lanes); its first warp also brings the input and forms the
        // dots. At 96 x 96 an SM works on three matrices and has three on their way. One warp per
        // matrix with transposed sums by shuffles (as FP32 below keeps: 64.6 us at 80^3 against 74.1 us
        // by rows) took 8,800 cycles per matrix, too long for the copies to keep going: 86.5 us for the
        // 8,322 matrices of the 61^3 mesh (310 MB), 54.1 us now, 48 us at the measured copy rate.
        template <int BD, int MODE>
        __device__ __forceinline__ bool mas_apply_rows(const MasView &mas, const double *__restrict__ r,
                                                       double *__restrict__ z0, PcgState *st, const PcgConfig &cfg,
                                                       Cta cta, bool early, double (&part)[APPLY_PARTS])
        {
            using L = ApplyLayout<BD, double>;
            constexpr int N = L::N, S = L::S;
            extern __shared__ __align__(128) unsigned char smem[];
            __shared__ int team_failed[L::TEAMS];
            const int w = warp_index(), lane = threadIdx.x & 31;
            const int team = w / BD, t = w - team * BD;
            unsigned char *base = smem + (size_t)team * L::TEAM_BYTES;
            double *xs = reinterpret_cast<double *>(base + 2 * L::STAGE_BYTES);
            double *ys = xs + N;
            uint64_t *bar = reinterpret_cast<uint64_t *>(base + 2 * L::STAGE_BYTES + L::XS_BYTES);
            const double *__restrict__ inv = static_cast<const double *>(mas.inv);
            const int banks = mas.banks;
            const int items = banks + mas.n_coarse_active;
            const int total_teams = cta.n * L::TEAMS;
            const int gt = cta.x * L::TEAMS + team;
            int *errp = st ? &st->error : nullptr;
            const bool pr = (MODE == 2) && cfg.polak_ribiere;
            const bool loader = t == 0 && lane == 0; // issues the team's copies
            auto mat_of = [&](int m) { return m < banks ? m : banks + mas.coarse_active[m - banks]; };
            auto in_of = [&](int m) -> const double * {
                return m < banks ? r + (size_t)m * N : mas.rc + (size_t)(mat_of(m) - banks) * N;
            };

            const uint64_t pol = l2_evict_first_policy(); // the inverses stream, the vectors stay
            bool pending[2] = {gt < items, gt + total_teams < items}; // copies issued and not consumed
            if (loader)
            {
                team_failed[team] = 0;
                mbar_init(&bar[0], 1);
                mbar_init(&bar[1], 1);
                fence_mbar_init();
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    if (pending[s])
                        bulk_load_stream(base + s * L::STAGE_BYTES, inv + (size_t)mat_of(gt + s * total_teams) * S,
                                         L::STAGE_BYTES, &bar[s], pol);
            }
            team_sync<BD>(team);
            // The first two inverses are on their way (no kernel of a solve writes them); now wait
            // for the predecessor (launched chained in a PCG iteration), or at the first coarse matrix.
            if (!early)
                pdl_wait();
            if (MODE != 0 && solve_done(st))
            {
                if (loader)
                    mbar_drain(bar, pending, {0u, 0u});
                return false;
            }
            uint32_t phase[2] = {0u, 0u};
            bool ok = true;
            double r_next[BD]; // first warp: input of the team's next item
            if (t == 0 && gt < items)
            {
                if (early && gt >= banks)
                    pdl_wait();
                const double *in = in_of(gt);
#pragma unroll
                for (int i = 0; i < BD; ++i)
                    r_next[i] = __ldcg(in + i * 32 + lane);
            }
            for (int m = gt, s = 0; m < items; m += total_teams, s ^= 1)
            {
                const bool coarse = m >= banks;
                const int mat = mat_of(m);
                double *out = coarse ? mas.zc + (size_t)(mat - banks) * N : z0 + (size_t)m * N;
                double r64[BD], zold[BD];
                if (t == 0)
                {
#pragma unroll
                    for (int i = 0; i < BD; ++i)
                    {
                        r64[i] = r_next[i];
                        xs[i * 32 + lane] = r64[i];
                    }
                    const int mnext = m + total_teams;
                    if (mnext < items)
                    {
                        if (early && mnext >= banks)
                            pdl_wait();
                        const double *in = in_of(mnext);
#pragma unroll
                        for (int i = 0; i < BD; ++i)
                            r_next[i] = __ldcg(in + i * 32 + lane);
                    }
                    if (pr)
#pragma unroll
                        for (int i = 0; i < BD; ++i)
                            zold[i] = out[i * 32 + lane];
                }
                // Coarse matrices of isolated rows are exactly the identity: z = r, unrounded.
                const bool ident = coarse && warp_uniform(mas.identity[mat - banks]);
                if (!mbar_wait_bounded(&bar[s], s ? phase[1] : phase[0], errp, cfg.wait_limit) && lane == 0)
                    team_failed[team] = 1;
                team_sync<BD>(team); // x complete; every warp has seen the copy or given up
                if (team_failed[team])
                {
                    ok = false;
                    break;
                }
                pending[s] = false;
                if (s)
                    phase[1] ^= 1u;
                else
                    phase[0] ^= 1u;
                if (!ident)
                    ys[t * 32 + lane] =
                        symv_row<BD>(reinterpret_cast<const double *>(base + s * L::STAGE_BYTES), xs, t, lane);
                team_sync<BD>(team); // y complete; the team is done with the stage and with x
                const int mn = m + 2 * total_teams;
                if (mn < items)
                {
                    if (loader)
                    {
                        fence_proxy_async_smem();
                        bulk_load_stream(base + s * L::STAGE_BYTES, inv + (size_t)mat_of(mn) * S, L::STAGE_BYTES, &bar[s],
                                         pol);
                    }
                    pending[s] = true;
                }
                if (t != 0)
                    continue;
                double d0 = 0.0, d1 = 0.0;
#pragma unroll
                for (int i = 0; i < BD; ++i)
                {
                    const double zv = ident ? r64[i] : ys[i * 32 + lane];
                    out[i * 32 + lane] = zv;
                    d0 = fma(zv, r64[i], d0);
                    if (pr)
                        d1 = fma(zold[i], r64[i], d1);
                }
                // Fixed slots (no dynamic indexing, so part[] stays in registers).
                if (coarse)
                {
                    part[4] += d0;
                    part[5] += d1;
                }
                else if (m >= mas.first_iso_bank)
                {
                    part[2] += d0;
                    part[3] += d1;
                }
                else
                {
                    part[0] += d0;
                    part[1] += d1;
                }
            }
            if (!ok && loader)
                mbar_drain(bar, pending, phase); // the outstanding copies (bounded) before leaving
            return true;
        }

        // early: the predecessor in the stream is k_coarse_levels, which lets this kernel start once its
        // own predecessor (the producer of r) has completed. The level-0 matrices then go ahead while the
        // coarse levels are summed, and pdl_wait() comes before the first coarse input. r, rc and st->done are
        // read past L1 (__ldcg): their producers were not waited for by this grid itself.
        // (One after the other, an iteration took 53.8 us at 44^3 in binary16, 49.7 us at 70^3 scalar FP64
        // and 180.5 us at 80^3, now 47.5, 44.0 and 172.7 us.)
        template <int BD, class Store, int MODE>
        __device__ __forceinline__ void mas_apply_body(const MasView &mas, const double *__restrict__ r,
                                                       double *__restrict__ z0, PcgState *st, const ReduceBuf &red,
                                                       const PcgConfig &cfg, Cta cta, bool prefetch_first, bool early)
        {
            if (!prefetch_first && MODE != 0)
            {
                pdl_wait();
                if (st->done)
                    return;
            }
            using L = ApplyLayout<BD, Store>;
            constexpr int THREADS = L::WARPS * 32;
            double part[APPLY_PARTS];
#pragma unroll
            for (int i = 0; i < APPLY_PARTS; ++i)
                part[i] = 0.0;
            bool ran;
            if constexpr (L::ROWS)
                ran = mas_apply_rows<BD, MODE>(mas, r, z0, st, cfg, cta, early, part);
            else
                ran = mas_apply_warps<BD, Store, MODE>(mas, r, z0, st, cfg, cta, early, part);
            // Every thread waits for the coarse levels before it leaves or releases the successor: this
            // kernel's end stands for theirs.
            if (early)
                pdl_wait();
            if (!ran)
                return;
            pdl_release(); // this warp's items are done: the successor may start launching
            if (MODE == 0)
                return;
            // Isolated rows: z = (1 + L) z0, so their r.z is (1 + L) r.z0 -- r.z0 is in the
            // level-0 sums, the coarse levels add L r.z0.
            const double Lc = (double)cfg.level_num;
            // (The dots with the previous z are wanted, and formed, for Polak-Ribiere's beta only.)
            if (MODE == 2 && cfg.polak_ribiere)
            {
                double tot[APPLY_PARTS];
                if (grid_reduce<APPLY_PARTS, THREADS, L::TEAMS * 32>(part, red.rz_parts, &st->counter[4], tot, cta) &&
                    threadIdx.x == 0)
                {
                    st->rz_coarse = tot[4] + Lc * tot[2];
                    st->rzx_coarse = tot[5] + Lc * tot[3];
                    pcg_finalize(st, cfg, MODE, tot[0] + tot[2] + st->rz_coarse, tot[1] + tot[3] + st->rzx_coarse);
                }
                return;
            }
            double rz[3] = {part[0], part[2], part[4]}, tot[3];
            if (grid_reduce<3, THREADS, L::TEAMS * 32>(rz, red.rz_parts, &st->counter[4], tot, cta) && threadIdx.x == 0)
            {
                st->rz_coarse = tot[2] + Lc * tot[1];
                st->rzx_coarse = 0.0;
                pcg_finalize(st, cfg, MODE, tot[0] + tot[1] + st->rz_coarse, 0.0);
            }
        }

        template <int BD, class Store, int MODE>
        __global__ void __launch_bounds__(ApplyLayout<BD, Store>::WARPS * 32)
            k_mas_apply(MasView mas, const double *__restrict__ r, double *__restrict__ z0, PcgState *st,
                        ReduceBuf red, PcgConfig cfg, int early)
        {
            mas_apply_body<BD, Store, MODE>(mas, r, z0, st, red, cfg, native_cta(), true, early != 0);
        }

        // The apply of every system of a batch (MODE 1: initial, 2: iteration) in one launch.
        template <int BD, class Store, int MODE>
        __global__ void __launch_bounds__(ApplyLayout<BD, Store>::WARPS * 32) k_mas_apply_batch(BatchView v)
        {
            const int4 e = batch_entry(v, BPH_APPLY);
            const BatchSystem &sy = v.sys[e.x];
            const Cta cta{e.y, e.z};
            const MasView mas = sy.mas;
            const ReduceBuf red = sy.red;
            const PcgConfig cfg = sy.cfg;
            mas_apply_body<BD, Store, MODE>(mas, sy.r, sy.z, sy.st, red, cfg, cta, false, false);
        }

        // ---- G right-hand sides at once (binary16 inverses only): the B operand's eight columns
        // hold the hi / lo splits of the G = RHS_GROUP vectors, so one pass over an inverse and the
        // same 36 MMAs serve all of them; every lane of a fragment quad holds a different
        // right-hand side of the result. Vectors are interleaved (value e of right-hand side g at
        // e * G + g). Per-right-hand-side dots and PCG steps; st[G] is the group record.
        template <int BD>
        struct ApplyLayoutG
        {
            static constexpr int N = 32 * BD;
            static constexpr int G = RHS_GROUP;
            static constexpr int S = (2 * BD) * (2 * BD - 1) / 2 * 256 + 2 * BD * 192;
            static constexpr int STAGE_BYTES = S * 2;
            static constexpr int XS_BYTES = 8 * G * N; // hi, lo (binary16) and the FP32 result rows
            static constexpr int WARP_BYTES = 2 * STAGE_BYTES + XS_BYTES + 16;
            static constexpr int SMEM_LIMIT = 232448 - 1024;
            static constexpr int W0 = SMEM_LIMIT / WARP_BYTES;
            static constexpr int WARPS = W0 > 16 ? 16 : W0;
            static_assert(STAGE_BYTES % 16 == 0, "bulk copies need 16-byte multiples");
            static_assert(2 * G == 8, "the B operand has eight columns: G hi / lo pairs");
        };

        // XS, YS: strides (values) between consecutive right-hand sides in xh / xl and in ys.
        template <int BD, int XS = 32 * BD, int YS = 32 * BD>
        __device__ __forceinline__ void symv_mma16_g(const __half *M, const __half *xh, const __half *xl, float *ys,
                                                     int lane)
        {
            constexpr int NS = 2 * BD, NB = NS * (NS - 1) / 2;
            const int g = lane >> 2, q = lane & 3;
            const int c = lane >> 3, rr = lane & 7;
            // B column n = g: right-hand side g / 2, hi (even) or lo (odd).
            const __half *xsrc = ((g & 1) ? xl : xh) + (g >> 1) * XS;
            uint32_t bf[NS][2];
#pragma unroll
            for (int S = 0; S < NS; ++S)
            {
                bf[S][0] = *reinterpret_cast<const uint32_t *>(xsrc + 16 * S + 2 * q);
                bf[S][1] = *reinterpret_cast<const uint32_t *>(xsrc + 16 * S + 2 * q + 8);
            }
            float d[NS][4];
#pragma unroll
            for (int R = 0; R < NS; ++R)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    d[R][i] = 0.f;
            const uint32_t mbase = smem_addr(M);
            const int ct = (c == 1) ? 2 : (c == 2 ? 1 : c);
            const uint32_t row_off = (uint32_t)(rr * 16);
#pragma unroll
            for (int R = 0; R < NS; ++R)
#pragma unroll
                for (int S = R + 1; S < NS; ++S)
                {
                    const uint32_t blk = mbase + (uint32_t)((R * (2 * NS - R - 1) / 2 + (S - R - 1)) * 512);
                    uint32_t a[4];
                    ldsm_x4(a, blk + c * 128 + row_off);
                    mma_16816(d[R], a, bf[S][0], bf[S][1]);
                    ldsm_x4_trans(a, blk + ct * 128 + row_off);
                    mma_16816(d[S], a, bf[R][0], bf[R][1]);
                }
            const int cd = (c == 1) ? 1 : (c == 3 ? 2 : 0);
#pragma unroll
            for (int R = 0; R < NS; ++R)
            {
                const uint32_t blk = mbase + (uint32_t)((NB * 256 + R * 192) * 2);
                uint32_t a[4];
                ldsm_x4_trans(a, blk + cd * 128 + row_off);
                a[2] = ldsm_x1(blk + 128 + row_off);
                mma_16816(d[R], a, bf[R][0], bf[R][1]);
            }
            // Columns 2q, 2q + 1 of rows g, g + 8 of each block row: right-hand side q.
#pragma unroll
            for (int R = 0; R < NS; ++R)
            {
                ys[q * YS + 16 * R + g] = d[R][0] + d[R][1];
                ys[q * YS + 16 * R + g + 8] = d[R][2] + d[R][3];
            }
            __syncwarp();
        }

        template <int BD, int MODE>
        __global__ void __launch_bounds__(ApplyLayoutG<BD>::WARPS * 32)
            k_mas_apply_g(MasView mas, const double *__restrict__ r, double *__restrict__ z0, PcgState *st,
                          ReduceBuf red, PcgConfig cfg)
        {
            using L = ApplyLayoutG<BD>;
            constexpr int N = L::N, S = L::S, WARPS = L::WARPS, G = L::G;
            constexpr int THREADS = WARPS * 32;
            PcgState *grp = st + G;
            if (grp->done)
                return;
            extern __shared__ __align__(128) unsigned char smem[];
            const int w = warp_index(), lane = threadIdx.x & 31;
            unsigned char *base = smem + (size_t)w * L::WARP_BYTES;
            __half *stage0 = reinterpret_cast<__half *>(base);
            __half *stage1 = reinterpret_cast<__half *>(base + L::STAGE_BYTES);
            __half *xh = reinterpret_cast<__half *>(base + 2 * L::STAGE_BYTES);
            __half *xl = xh + G * N;
            float *ys = reinterpret_cast<float *>(base + 2 * L::STAGE_BYTES + 4 * G * N);
            uint64_t *bar = reinterpret_cast<uint64_t *>(base + 2 * L::STAGE_BYTES + L::XS_BYTES);
            const __half *__restrict__ inv = static_cast<const __half *>(mas.inv);
            const int banks = mas.banks;
            const int items = banks + mas.n_coarse_active;
            const int total_warps = gridDim.x * WARPS;
            const int gw = blockIdx.x * WARPS + w;
            auto mat_of = [&](int m) { return m < banks ? m : banks + mas.coarse_active[m - banks]; };
            auto in_of = [&](int m) -> const double * {
                return m < banks ? r + (size_t)m * N * G : mas.rc + (size_t)(mat_of(m) - banks) * N * G;
            };
            const uint64_t pol = l2_evict_first_policy();
            if (lane == 0)
            {
                mbar_init(&bar[0], 1);
                mbar_init(&bar[1], 1);
                fence_mbar_init();
            }
            __syncwarp();
            if (lane == 0)
            {
                if (gw < items)
                    bulk_load_stream(stage0, inv + (size_t)mat_of(gw) * S, L::STAGE_BYTES, &bar[0], pol);
                if (gw + total_warps < items)
                    bulk_load_stream(stage1, inv + (size_t)mat_of(gw + total_warps) * S, L::STAGE_BYTES, &bar[1],
                                     pol);
            }
            bool pending[2] = {gw < items, gw + total_warps < items};
            double part[3 * G]; // per right-hand side: coupled banks, isolated banks, coarse
#pragma unroll
            for (int i = 0; i < 3 * G; ++i)
                part[i] = 0.0;
            uint32_t phase0 = 0, phase1 = 0;
            bool ok = true;
            int k = 0;
            for (int m = gw; m < items; m += total_warps, ++k)
            {
                const bool s1 = (k & 1) != 0;
                __half *stage = s1 ? stage1 : stage0;
                uint64_t *b = s1 ? &bar[1] : &bar[0];
                const bool coarse = m >= banks;
                const int mat = mat_of(m);
                const double *in = in_of(m);
                double *out = coarse ? mas.zc + (size_t)(mat - banks) * N * G : z0 + (size_t)m * N * G;
                double r64[BD][G];
#pragma unroll
                for (int t = 0; t < BD; ++t)
#pragma unroll
                    for (int h = 0; h < G / 2; ++h)
                    {
                        const double2 v = *reinterpret_cast<const double2 *>(in + (t * 32 + lane) * G + 2 * h);
                        r64[t][2 * h] = v.x;
                        r64[t][2 * h + 1] = v.y;
                    }
                double xscale[G];
#pragma unroll
                for (int gg = 0; gg < G; ++gg)
                {
                    double amax = 0.0;
#pragma unroll
                    for (int t = 0; t < BD; ++t)
                        amax = fmax(amax, fabs(r64[t][gg]));
#pragma unroll
                    for (int o = 16; o >= 1; o >>= 1)
                        amax = fmax(amax, __shfl_xor_sync(FULL, amax, o));
                    xscale[gg] = (amax > 0.0 && isfinite(amax)) ? ldexp(1.0, 14 - ilogb(amax)) : 1.0;
#pragma unroll
                    for (int t = 0; t < BD; ++t)
                    {
                        const float v = (float)(r64[t][gg] * xscale[gg]);
                        const __half h = __float2half_rn(v);
                        xh[gg * N + t * 32 + lane] = h;
                        xl[gg * N + t * 32 + lane] = __float2half_rn(v - __half2float(h));
                    }
                }
                __syncwarp();
                if (!mbar_wait_bounded(b, s1 ? phase1 : phase0, &grp->error, cfg.wait_limit))
                {
                    ok = false;
                    break;
                }
                pending[s1 ? 1 : 0] = false;
                if (s1)
                    phase1 ^= 1u;
                else
                    phase0 ^= 1u;
                const bool ident = coarse && warp_uniform(mas.identity[mat - banks]);
                if (!ident)
                    symv_mma16_g<BD>(stage, xh, xl, ys, lane);
                __syncwarp();
                const int mn = m + 2 * total_warps;
                if (mn < items)
                {
                    if (lane == 0)
                    {
                        fence_proxy_async_smem();
                        bulk_load_stream(stage, inv + (size_t)mat_of(mn) * S, L::STAGE_BYTES, b, pol);
                    }
                    pending[s1 ? 1 : 0] = true;
                }
                const double mscale = mas.inv_scale[mat];
                const int slot = coarse ? 2 : ((m >= mas.first_iso_bank) ? 1 : 0);
#pragma unroll
                for (int t = 0; t < BD; ++t)
                {
                    double zv[G];
#pragma unroll
                    for (int gg = 0; gg < G; ++gg)
                    {
                        zv[gg] = ident ? r64[t][gg] : (double)ys[gg * N + t * 32 + lane] * (mscale / xscale[gg]);
                        const double d = zv[gg] * r64[t][gg];
                        if (slot == 0)
                            part[gg] += d;
                        else if (slot == 1)
                            part[G + gg] += d;
                        else
                            part[2 * G + gg] += d;
                    }
#pragma unroll
                    for (int h = 0; h < G / 2; ++h)
                        *reinterpret_cast<double2 *>(out + (t * 32 + lane) * G + 2 * h) =
                            make_double2(zv[2 * h], zv[2 * h + 1]);
                }
                __syncwarp();
            }
            if (!ok)
            {
                if (lane == 0)
                    mbar_drain(bar, pending, {phase0, phase1});
                __syncwarp();
            }
            double tot[3 * G];
            if (grid_reduce<3 * G, THREADS>(part, red.rz_parts, &grp->counter[4], tot) && threadIdx.x == 0)
            {
                const double Lc = (double)cfg.level_num;
                int all_done = 1;
#pragma unroll
                for (int gg = 0; gg < G; ++gg)
                {
                    PcgState *sg = st + gg;
                    if (!sg->done)
                    {
                        sg->rz_coarse = tot[2 * G + gg] + Lc * tot[G + gg];
                        pcg_finalize(sg, cfg, MODE, tot[gg] + tot[G + gg] + sg->rz_coarse, 0.0);
                        if (sg->error)
                            grp->error = sg->error;
                    }
                    all_done &= sg->done ? 1 : 0;
                }
                grp->iter = MODE == 1 ? 0 : grp->iter + 1;
                if (all_done || grp->error)
                    grp->done = 1;
            }
        }

        // ---- RHS_WIDE (16) right-hand sides at once (block size 3, binary16 inverses): the B operand
        // of each m16n8k16 holds four right-hand sides' hi / lo splits, so each inverse is multiplied in
        // four n-tiles (symv_mma16_g per tile) and read from memory once for all sixteen. Lane l loads,
        // splits and stores right-hand side g = l % 16 (values e = 2 t + l / 16 of the matrix's 96), so
        // every load and store of the interleaved vectors is 128 B per 16 lanes. xh / xl and ys use
        // padded strides per right-hand side (100 halves, 97 floats) that spread the 16 lanes' words
        // over the shared-memory banks.
        struct ApplyLayoutW
        {
            static constexpr int BD = 3, N = 96, G = RHS_WIDE;
            static constexpr int XS = N + 4, YS = N + 1;
            static constexpr int S = (2 * BD) * (2 * BD - 1) / 2 * 256 + 2 * BD * 192;
            static constexpr int STAGE_BYTES = S * 2;
            static constexpr int XS_BYTES = 2 * 2 * G * XS + 4 * G * YS; // hi, lo, FP32 result
            static constexpr int WARP_BYTES = 2 * STAGE_BYTES + XS_BYTES + 16;
            static constexpr int SMEM_LIMIT = 232448 - 2048; // static shared memory: the grid sum's groups
            static constexpr int W0 = SMEM_LIMIT / WARP_BYTES;
            static constexpr int WARPS = W0 > 16 ? 16 : W0;
            static_assert(STAGE_BYTES % 16 == 0 && WARP_BYTES % 16 == 0 && XS_BYTES % 8 == 0, "alignment");
            static_assert((WARPS + 2) * 3 * G * 8 <= WARP_BYTES, "the final sums reuse the first warp's area");
        };

        template <int MODE>
        __global__ void __launch_bounds__(ApplyLayoutW::WARPS * 32)
            k_mas_apply_w(MasView mas, const double *__restrict__ r, double *__restrict__ z0, PcgState *st,
                          ReduceBuf red, PcgConfig cfg)
        {
            using L = ApplyLayoutW;
            constexpr int N = L::N, S = L::S, WARPS = L::WARPS, G = L::G, XS = L::XS, YS = L::YS;
            constexpr int THREADS = WARPS * 32;
            constexpr int VW = N / 2; // values of a matrix per lane (two lanes per right-hand side)
            PcgState *grp = st + G;
            if (grp->done)
                return;
            extern __shared__ __align__(128) unsigned char smem[];
            const int w = warp_index(), lane = threadIdx.x & 31;
            unsigned char *base = smem + (size_t)w * L::WARP_BYTES;
            __half *stage0 = reinterpret_cast<__half *>(base);
            __half *stage1 = reinterpret_cast<__half *>(base + L::STAGE_BYTES);
            __half *xh = reinterpret_cast<__half *>(base + 2 * L::STAGE_BYTES);
            __half *xl = xh + G * XS;
            float *ys = reinterpret_cast<float *>(base + 2 * L::STAGE_BYTES + 4 * G * XS);
            uint64_t *bar = reinterpret_cast<uint64_t *>(base + 2 * L::STAGE_BYTES + L::XS_BYTES);
            const __half *__restrict__ inv = static_cast<const __half *>(mas.inv);
            const int banks = mas.banks;
            const int items = banks + mas.n_coarse_active;
            const int total_warps = gridDim.x * WARPS;
            const int gw = blockIdx.x * WARPS + w;
            auto mat_of = [&](int m) { return m < banks ? m : banks + mas.coarse_active[m - banks]; };
            auto in_of = [&](int m) -> const double * {
                return m < banks ? r + (size_t)m * N * G : mas.rc + (size_t)(mat_of(m) - banks) * N * G;
            };
            const uint64_t pol = l2_evict_first_policy();
            if (lane == 0)
            {
                mbar_init(&bar[0], 1);
                mbar_init(&bar[1], 1);
                fence_mbar_init();
            }
            __syncwarp();
            if (lane == 0)
            {
                if (gw < items)
                    bulk_load_stream(stage0, inv + (size_t)mat_of(gw) * S, L::STAGE_BYTES, &bar[0], pol);
                if (gw + total_warps < items)
                    bulk_load_stream(stage1, inv + (size_t)mat_of(gw + total_warps) * S, L::STAGE_BYTES, &bar[1],
                                     pol);
            }
            bool pending[2] = {gw < items, gw + total_warps < items};
            const int g = lane & (G - 1), half = lane >> 4;
            double part[3] = {0.0, 0.0, 0.0}; // this lane's right-hand side: coupled, isolated, coarse
            uint32_t phase0 = 0, phase1 = 0;
            bool ok = true;
            int k = 0;
            for (int m = gw; m < items; m += total_warps, ++k)
            {
                const bool s1 = (k & 1) != 0;
                __half *stage = s1 ? stage1 : stage0;
                uint64_t *b = s1 ? &bar[1] : &bar[0];
                const bool coarse = m >= banks;
                const int mat = mat_of(m);
                const double *in = in_of(m);
                double *out = coarse ? mas.zc + (size_t)(mat - banks) * N * G : z0 + (size_t)m * N * G;
                double r64[VW];
#pragma unroll
                for (int t = 0; t < VW; ++t)
                    r64[t] = in[(2 * t + half) * G + g];
                double amax = 0.0;
#pragma unroll
                for (int t = 0; t < VW; ++t)
                    amax = fmax(amax, fabs(r64[t]));
                amax = fmax(amax, __shfl_xor_sync(FULL, amax, 16));
                const double xscale = (amax > 0.0 && isfinite(amax)) ? ldexp(1.0, 14 - ilogb(amax)) : 1.0;
#pragma unroll
                for (int t = 0; t < VW; ++t)
                {
                    const float v = (float)(r64[t] * xscale);
                    const __half h = __float2half_rn(v);
                    xh[g * XS + 2 * t + half] = h;
                    xl[g * XS + 2 * t + half] = __float2half_rn(v - __half2float(h));
                }
                __syncwarp();
                if (!mbar_wait_bounded(b, s1 ? phase1 : phase0, &grp->error, cfg.wait_limit))
                {
                    ok = false;
                    break;
                }
                pending[s1 ? 1 : 0] = false;
                if (s1)
                    phase1 ^= 1u;
                else
                    phase0 ^= 1u;
                const bool ident = coarse && warp_uniform(mas.identity[mat - banks]);
                if (!ident)
#pragma unroll
                    for (int nt = 0; nt < G / 4; ++nt)
                        symv_mma16_g<3, XS, YS>(stage, xh + 4 * nt * XS, xl + 4 * nt * XS, ys + 4 * nt * YS, lane);
                __syncwarp();
                const int mn = m + 2 * total_warps;
                if (mn < items)
                {
                    if (lane == 0)
                    {
                        fence_proxy_async_smem();
                        bulk_load_stream(stage, inv + (size_t)mat_of(mn) * S, L::STAGE_BYTES, b, pol);
                    }
                    pending[s1 ? 1 : 0] = true;
                }
                const double sc = mas.inv_scale[mat] / xscale;
                double d = 0.0;
#pragma unroll
                for (int t = 0; t < VW; ++t)
                {
                    const int e = 2 * t + half;
                    const double zv = ident ? r64[t] : (double)ys[g * YS + e] * sc;
                    out[e * G + g] = zv;
                    d = fma(zv, r64[t], d);
                }
                if (coarse)
                    part[2] += d;
                else if (m >= mas.first_iso_bank)
                    part[1] += d;
                else
                    part[0] += d;
                __syncwarp();
            }
            if (!ok)
            {
                if (lane == 0)
                    mbar_drain(bar, pending, {phase0, phase1});
                __syncwarp();
            }
            // Every warp is past its last stage (no copy in flight): the first warp's area holds the
            // per-warp sums, the CTA's sums and the totals.
            __syncthreads();
            double *wsum = reinterpret_cast<double *>(smem);
            double *cta = wsum + WARPS * 3 * G, *tot = cta + 3 * G;
#pragma unroll
            for (int i = 0; i < 3; ++i)
                part[i] += __shfl_xor_sync(FULL, part[i], 16);
            if (lane < G)
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    wsum[w * 3 * G + i * G + lane] = part[i];
            __syncthreads();
            if (threadIdx.x < 3 * G)
            {
                double s = 0.0;
                for (int ww = 0; ww < WARPS; ++ww)
                    s += wsum[ww * 3 * G + threadIdx.x];
                cta[threadIdx.x] = s;
            }
            if (grid_reduce_cta<3 * G, THREADS>(cta, red.rz_parts, &grp->counter[4], tot) && threadIdx.x == 0)
            {
                const double Lc = (double)cfg.level_num;
                int all_done = 1;
                for (int gg = 0; gg < G; ++gg)
                {
                    PcgState *sg = st + gg;
                    if (!sg->done)
                    {
                        sg->rz_coarse = tot[2 * G + gg] + Lc * tot[G + gg];
                        pcg_finalize(sg, cfg, MODE, tot[gg] + tot[G + gg] + sg->rz_coarse, 0.0);
                        if (sg->error)
                            grp->error = sg->error;
                    }
                    all_done &= sg->done ? 1 : 0;
                }
                grp->iter = MODE == 1 ? 0 : grp->iter + 1;
                if (all_done || grp->error)
                    grp->done = 1;
            }
        }

        // ---- Sixteen right-hand sides on the fifth-generation tensor cores (tcgen05) ------------
        // Inverse storage "tc" (built from the mma16 storage, the same binary16 values): the full
        // 96 x 96 matrix in 16 x 16 tiles, tile (i, s) (rows 16 i .., columns 16 s ..) at byte
        // s * TC_SLAB_G + i * 512, each tile the four 8 x 8 core matrices [rows 0-7 | cols 0-7],
        // [rows 0-7 | cols 8-15], [rows 8-15 | cols 0-7], [rows 8-15 | cols 8-15] of 16-byte rows:
        // the canonical no-swizzle K-major operand layout with 128 bytes between the two K halves of
        // a core pair and 256 bytes between 8-row groups. Column slab s is the A operand of one K = 16
        // step; in shared memory the slabs are TC_SLAB_S apart with rows 96-127 zero (M = 128).
        // The B operand is the item's 16 right-hand sides split into binary16 hi and lo parts
        // (N = 32: columns g and 16 + g), D = A B^T accumulates in FP32 in tensor memory.
        constexpr int TC_N = 96, TC_G = RHS_WIDE, TC_THREADS = 128;
        constexpr int TC_SLAB_G = 6 * 512;          // bytes of a column slab in global memory
        constexpr int TC_SLAB_S = 8 * 512;          // in shared memory (M = 128 rows)
        constexpr int TC_MAT_BYTES = 6 * TC_SLAB_G; // 18432 bytes per matrix

        __host__ __device__ constexpr int tc_offset(int row, int col)
        {
            return (col >> 4) * TC_SLAB_G + (row >> 4) * 512 + ((row >> 3) & 1) * 256 + ((col >> 3) & 1) * 128 +
                   (row & 7) * 16 + (col & 7) * 2;
        }

        // B operand element (n, k): K steps 1 KB apart, 8-column groups 256 bytes apart.
        __device__ __forceinline__ int tc_b_offset(int n, int k)
        {
            return (k >> 4) * 1024 + (n >> 3) * 256 + ((k >> 3) & 1) * 128 + (n & 7) * 16 + (k & 7) * 2;
        }

        struct TcLayout
        {
            static constexpr int A_BYTES = 6 * TC_SLAB_S;     // one stage of A
            static constexpr int X_BYTES = TC_N * TC_G * 8;   // one stage of the FP64 input block
            static constexpr int B_BYTES = 6 * 1024;
            static constexpr int OFF_X = 2 * A_BYTES;
            static constexpr int OFF_B = OFF_X + 2 * X_BYTES;
            static constexpr int OFF_AMAX = OFF_B + B_BYTES;  // [8][16] doubles
            static constexpr int OFF_XSC = OFF_AMAX + 8 * TC_G * 8;
            static constexpr int OFF_WSUM = OFF_XSC + TC_G * 8; // [4 warps][3][16] doubles
            static constexpr int OFF_BAR = OFF_WSUM + 4 * 3 * TC_G * 8;
            static constexpr int BYTES = OFF_BAR + 64;
            static_assert(OFF_X % 1024 == 0 && OFF_B % 128 == 0 && OFF_BAR % 16 == 0, "alignment");
        };

        // mma16 -> tc storage, one CTA per matrix.
        __global__ void __launch_bounds__(256) k_inv_to_tc(const __half *__restrict__ inv, __half *__restrict__ out)
        {
            constexpr int S16 = 6 * 5 / 2 * 256 + 6 * 192;
            const __half *src = inv + (size_t)blockIdx.x * S16;
            unsigned char *dst = reinterpret_cast<unsigned char *>(out) + (size_t)blockIdx.x * TC_MAT_BYTES;
            for (int e = threadIdx.x; e < TC_N * TC_N; e += blockDim.x)
            {
                const int row = e / TC_N, col = e - row * TC_N;
                *reinterpret_cast<__half *>(dst + tc_offset(row, col)) = src[mma16_index(3, row, col)];
            }
        }

        // The sixteen-right-hand-side MAS apply on tcgen05 (same work items, scales, outputs, dots
        // and PCG steps as k_mas_apply_w). One CTA of four warps per item at a time, items strided
        // over the grid; per item the inverse (six slab copies) and the 96 x 16 FP64 input block
        // arrive by bulk copies on one mbarrier, two items ahead. The four warps split the input into
        // binary16 hi / lo (per-column power-of-two scale), thread 0 issues six MMAs and commits them
        // to an mbarrier, and warps 0-2 read rows 0-95 of the accumulator (tcgen05.ld), combine hi +
        // lo, scale to FP64, store z and add the dots. Every wait is bounded (MAS_ERR_TIMEOUT).
        template <int MODE>
        __global__ void __launch_bounds__(TC_THREADS) k_mas_apply_tc(MasView mas, const __half *__restrict__ inv_tc,
                                                                     const double *__restrict__ r,
                                                                     double *__restrict__ z0, PcgState *st,
                                                                     ReduceBuf red, PcgConfig cfg)
        {
            using L = TcLayout;
            constexpr int N = TC_N, G = TC_G;
            PcgState *grp = st + G;
            if (grp->done)
                return;
            extern __shared__ __align__(1024) unsigned char smem[];
            const int tid = threadIdx.x, w = warp_index(), lane = tid & 31;
            unsigned char *sA = smem, *sX = smem + L::OFF_X, *sB = smem + L::OFF_B;
            double *amax_s = reinterpret_cast<double *>(smem + L::OFF_AMAX);
            double *xsc_s = reinterpret_cast<double *>(smem + L::OFF_XSC);
            double *wsum = reinterpret_cast<double *>(smem + L::OFF_WSUM);
            uint64_t *tma_bar = reinterpret_cast<uint64_t *>(smem + L::OFF_BAR); // [2]
            uint64_t *mma_bar = tma_bar + 2;
            uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tma_bar + 3);
            const int banks = mas.banks, items = banks + mas.n_coarse_active;
            auto mat_of = [&](int m) { return m < banks ? m : banks + mas.coarse_active[m - banks]; };
            auto in_of = [&](int m) -> const double * {
                return m < banks ? r + (size_t)m * N * G : mas.rc + (size_t)(mat_of(m) - banks) * N * G;
            };
            const uint64_t pol = l2_evict_first_policy();
            if (tid == 0)
            {
                mbar_init(&tma_bar[0], 1);
                mbar_init(&tma_bar[1], 1);
                mbar_init(mma_bar, 1);
                fence_mbar_init();
            }
            if (w == 0)
                tmem_alloc(tmem_slot, 32);
            // Rows 96-127 of every slab of both A stages: zero (the bulk copies fill rows 0-95).
            for (int i = tid; i < 2 * 6 * 64; i += TC_THREADS)
            {
                const int stg = i / 384, rem = i - stg * 384, slab = rem >> 6, q = rem & 63;
                reinterpret_cast<uint4 *>(sA + stg * L::A_BYTES + slab * TC_SLAB_S + 6 * 512)[q] = make_uint4(0, 0, 0, 0);
            }
            for (int i = tid; i < 4 * 3 * G; i += TC_THREADS)
                wsum[i] = 0.0;
            fence_proxy_async_smem();
            tc_fence_before_sync();
            __syncthreads();
            tc_fence_after_sync();
            const uint32_t taddr = *tmem_slot;
            const int m0 = blockIdx.x, stride = gridDim.x;
            // Thread 0: the inverse and the input block of item m into stage stg.
            auto issue = [&](int m, int stg) {
                const unsigned char *src = reinterpret_cast<const unsigned char *>(inv_tc) + (size_t)mat_of(m) * TC_MAT_BYTES;
                mbar_arrive_expect_tx(&tma_bar[stg], TC_MAT_BYTES + L::X_BYTES);
#pragma unroll 1
                for (int s = 0; s < 6; ++s)
                    bulk_copy_g2s_hint(sA + stg * L::A_BYTES + s * TC_SLAB_S, src + s * TC_SLAB_G, TC_SLAB_G,
                                       &tma_bar[stg], pol);
                bulk_copy_g2s(sX + stg * L::X_BYTES, in_of(m), L::X_BYTES, &tma_bar[stg]);
            };
            bool pending[2] = {m0 < items, m0 + stride < items};
            if (tid == 0)
            {
                if (pending[0])
                    issue(m0, 0);
                if (pending[1])
                    issue(m0 + stride, 1);
            }
            uint32_t tphase[2] = {0u, 0u}, mphase = 0u;
            bool mma_pending = false, ok = true;
            const uint32_t idesc = tc_idesc_f16_f32(128, 32);
            double dsum[G];
#pragma unroll
            for (int gg = 0; gg < G; ++gg)
                dsum[gg] = 0.0;
            int cat = 0; // dots of coupled banks, isolated banks, coarse matrices
            // This warp's running dots into its slots of category c (each category once per CTA:
            // items increase, and the categories with them).
            auto flush = [&](int c) {
#pragma unroll
                for (int gg = 0; gg < G; ++gg)
                {
                    const double v = warp_sum(dsum[gg]);
                    if (lane == 0)
                        wsum[(w * 3 + c) * G + gg] = v;
                    dsum[gg] = 0.0;
                }
            };
            const int g = tid & (G - 1), rg = tid >> 4; // input split: column g, rows 12 rg .. 12 rg + 11
            int k = 0;
            for (int m = m0; m < items; m += stride, ++k)
            {
                const int stg = k & 1;
                const bool wok = mbar_wait_bounded(&tma_bar[stg], tphase[stg], &grp->error, cfg.wait_limit);
                if (!__syncthreads_and(wok))
                {
                    ok = false;
                    break;
                }
                pending[stg] = false;
                tphase[stg] ^= 1u;
                const bool coarse = m >= banks;
                const int mat = mat_of(m);
                const int mcat = coarse ? 2 : (m >= mas.first_iso_bank ? 1 : 0);
                if (mcat != cat)
                {
                    flush(cat);
                    cat = mcat;
                }
                const double *x = reinterpret_cast<const double *>(sX + stg * L::X_BYTES);
                const bool ident = coarse && warp_uniform(mas.identity[mat - banks]);
                double xv[12], am = 0.0;
#pragma unroll
                for (int i = 0; i < 12; ++i)
                {
                    xv[i] = x[(rg * 12 + i) * G + g];
                    am = fmax(am, fabs(xv[i]));
                }
                amax_s[rg * G + g] = am;
                __syncthreads();
                double amx = 0.0;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    amx = fmax(amx, amax_s[q * G + g]);
                const double xscale = (amx > 0.0 && isfinite(amx)) ? ldexp(1.0, 14 - ilogb(amx)) : 1.0;
                if (rg == 0)
                    xsc_s[g] = mas.inv_scale[mat] / xscale; // column g's factor back to matrix values
                if (!ident)
                {
                    // Row pairs (kk, kk + 1) are adjacent in the operand layout: one 32-bit store
                    // per pair and part.
#pragma unroll
                    for (int i = 0; i < 12; i += 2)
                    {
                        const int kk = rg * 12 + i;
                        const float v0 = (float)(xv[i] * xscale), v1 = (float)(xv[i + 1] * xscale);
                        const __half h0 = __float2half_rn(v0), h1 = __float2half_rn(v1);
                        *reinterpret_cast<__half2 *>(sB + tc_b_offset(g, kk)) = __halves2half2(h0, h1);
                        *reinterpret_cast<__half2 *>(sB + tc_b_offset(G + g, kk)) =
                            __halves2half2(__float2half_rn(v0 - __half2float(h0)), __float2half_rn(v1 - __half2float(h1)));
                    }
                    fence_proxy_async_smem();
                }
                tc_fence_before_sync();
                __syncthreads();
                if (!ident)
                {
                    if (tid == 0)
                    {
                        tc_fence_after_sync();
                        const unsigned char *a = sA + stg * L::A_BYTES;
#pragma unroll
                        for (int s = 0; s < 6; ++s)
                            tc_mma_f16(taddr, tc_smem_desc(a + s * TC_SLAB_S, 128, 256), tc_smem_desc(sB + s * 1024, 128, 256),
                                       idesc, s > 0);
                        tc_commit(mma_bar);
                    }
                    mma_pending = true;
                    const bool mok = mbar_wait_bounded(mma_bar, mphase, &grp->error, cfg.wait_limit);
                    if (!__syncthreads_and(mok))
                    {
                        ok = false;
                        break;
                    }
                    mma_pending = false;
                    mphase ^= 1u;
                    tc_fence_after_sync();
                }
                if (w < 3)
                {
                    const int row = 32 * w + lane;
                    double *out = (coarse ? mas.zc + (size_t)(mat - banks) * N * G : z0 + (size_t)m * N * G) + (size_t)row * G;
                    const double *xr = x + row * G;
                    float hi[16], lo[16];
                    if (!ident)
                    {
                        const uint32_t ta = taddr + ((uint32_t)(32 * w) << 16);
                        tc_ld16(ta, hi);
                        tc_ld16(ta + 16, lo);
                        tc_wait_ld();
                    }
#pragma unroll
                    for (int gg = 0; gg < G; gg += 2)
                    {
                        double zv[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                        {
                            const double xin = xr[gg + h];
                            zv[h] = ident ? xin : (double)(hi[gg + h] + lo[gg + h]) * xsc_s[gg + h];
                            dsum[gg + h] = fma(zv[h], xin, dsum[gg + h]);
                        }
                        *reinterpret_cast<double2 *>(out + gg) = make_double2(zv[0], zv[1]);
                    }
                }
                tc_fence_before_sync();
                __syncthreads(); // accumulator read, the stage's A and X free
                const int mn = m + 2 * stride;
                pending[stg] = mn < items;
                if (tid == 0 && mn < items)
                    issue(mn, stg);
            }
            if (!ok && tid == 0)
            {
                // Leave nothing in flight: the MMAs and the bulk copies (bounded, default limit).
                if (mma_pending)
                    for (long long i = 0; i < MBAR_SPIN_LIMIT; ++i)
                        if (mbar_try_wait(mma_bar, mphase))
                            break;
                mbar_drain(tma_bar, pending, {tphase[0], tphase[1]});
            }
            flush(cat);
            tc_fence_before_sync();
            __syncthreads();
            if (w == 0)
            {
                tc_fence_after_sync();
                tmem_dealloc(taddr, 32);
            }
            // CTA sums (warps in order) into the first warp's slots, then the grid sum.
            double *cta = amax_s; // free now: 3 G doubles
            if (tid < 3 * G)
            {
                double s = 0.0;
                for (int ww = 0; ww < 4; ++ww)
                    s += wsum[ww * 3 * G + tid];
                cta[tid] = s;
            }
            __shared__ double totals[3 * G];
            if (grid_reduce_cta<3 * G, TC_THREADS>(cta, red.rz_parts, &grp->counter[4], totals) && tid == 0)
            {
                const double Lc = (double)cfg.level_num;
                int all_done = 1;
                for (int gg = 0; gg < G; ++gg)
                {
                    PcgState *sg = st + gg;
                    if (!sg->done)
                    {
                        sg->rz_coarse = totals[2 * G + gg] + Lc * totals[G + gg];
                        pcg_finalize(sg, cfg, MODE, totals[gg] + totals[G + gg] + sg->rz_coarse, 0.0);
                        if (sg->error)
                            grp->error = sg->error;
                    }
                    all_done &= sg->done ? 1 : 0;
                }
                grp->iter = MODE == 1 ? 0 : grp->iter + 1;
                if (all_done || grp->error)
                    grp->done = 1;
            }
        }

        // Coarse levels above the first from its components rc (level 0 of the coarse vector).
        // Each real node of level l sums its (at most 32) children of level l - 1 in a warp
        // (lane = child, in increasing order; deterministic). With three or more levels one CTA
        // (32 warps) per level-2 node computes its level-1 children (a warp each) and then itself
        // from them, so both levels take one round; a fourth level is summed by the last CTA to
        // finish (atomic ticket).
        constexpr int LEVEL_THREADS = 1024;

        // The lane's child of node i of level l, as a node of rc (-1: none).
        __device__ __forceinline__ int kid_node(const MasView &mas, int l, int i)
        {
            const int b = mas.kid_ptr[l][i], e = mas.kid_ptr[l][i + 1], lane = threadIdx.x & 31;
            return b + lane < e ? mas.coff[l - 1] + mas.kids[b + lane] : -1;
        }

        template <int BD>
        __device__ __forceinline__ void kid_sum(const MasView &mas, int node, bool cg, double (&v)[BD])
        {
#pragma unroll
            for (int c = 0; c < BD; ++c)
            {
                v[c] = 0.0;
                if (node >= 0)
                    v[c] = cg ? __ldcg(mas.rc + (size_t)node * BD + c) : mas.rc[(size_t)node * BD + c];
            }
#pragma unroll
            for (int c = 0; c < BD; ++c)
                v[c] = warp_sum(v[c]);
        }

        // The children's indices, three loads each waiting for the one before, are not written during a
        // solve and come before the wait; after it, the apply that follows may start on the level-0
        // matrices (mas_apply_body).
        template <int BD>
        __device__ __forceinline__ void coarse_levels_body(const MasView &mas, const PcgState *st, Cta cta)
        {
            constexpr int W = LEVEL_THREADS / 32;
            const int w = warp_index(), lane = threadIdx.x & 31;
            __shared__ double part[W][BD];
            __shared__ int is_last;
            if (mas.level_num == 2)
            {
                const int i = cta.x * W + w;
                const int node = i < mas.real_count[1] ? kid_node(mas, 1, i) : -1;
                pdl_wait();
                pdl_release();
                if ((st && st->done) || i >= mas.real_count[1])
                    return;
                double v[BD];
                kid_sum<BD>(mas, node, false, v);
                if (lane == 0)
#pragma unroll
                    for (int c = 0; c < BD; ++c)
                        mas.rc[((size_t)mas.coff[1] + i) * BD + c] = v[c];
                return;
            }
            // Level-2 node j = cta.x; warp w: its w-th level-1 child.
            const int j = cta.x;
            const int kb = warp_uniform(mas.kid_ptr[2][j]), ke = warp_uniform(mas.kid_ptr[2][j + 1]);
            const int i = kb + w < ke ? mas.kids[kb + w] : -1;
            const int node = i >= 0 ? kid_node(mas, 1, i) : -1;
            const int node3 = mas.level_num > 3 && w < mas.real_count[3] ? kid_node(mas, 3, w) : -1;
            pdl_wait();
            pdl_release();
            if (st && st->done)
                return;
            if (kb + w < ke)
            {
                double v[BD];
                kid_sum<BD>(mas, node, false, v);
                if (lane == 0)
#pragma unroll
                    for (int c = 0; c < BD; ++c)
                    {
                        mas.rc[((size_t)mas.coff[1] + i) * BD + c] = v[c];
                        part[w][c] = v[c];
                    }
            }
            __syncthreads();
            if (w == 0)
            {
#pragma unroll
                for (int c = 0; c < BD; ++c)
                {
                    const double t = warp_sum(kb + lane < ke ? part[lane][c] : 0.0);
                    if (lane == 0)
                        mas.rc[((size_t)mas.coff[2] + j) * BD + c] = t;
                }
            }
            if (mas.level_num <= 3)
                return;
            __syncthreads();
            if (threadIdx.x == 0)
            {
                __threadfence(); // cumulative: orders this CTA's stores (seen at the barrier) first
                is_last = atomicAdd(mas.ticket, 1u) == (unsigned)cta.n - 1;
            }
            __syncthreads();
            if (!warp_uniform(is_last))
                return;
            __threadfence();
            for (int k = w; k < mas.real_count[3]; k += W)
            {
                double v[BD];
                kid_sum<BD>(mas, k == w ? node3 : kid_node(mas, 3, k), true, v);
                if (lane == 0)
#pragma unroll
                    for (int c = 0; c < BD; ++c)
                        mas.rc[((size_t)mas.coff[3] + k) * BD + c] = v[c];
            }
            if (threadIdx.x == 0)
                *mas.ticket = 0u;
        }

        template <int BD>
        __global__ void __launch_bounds__(LEVEL_THREADS) k_coarse_levels(MasView mas, const PcgState *st)
        {
            coarse_levels_body<BD>(mas, st, native_cta());
        }

        template <int BD>
        __global__ void __launch_bounds__(LEVEL_THREADS) k_coarse_levels_batch(BatchView v)
        {
            const int4 e = batch_entry(v, BPH_COARSE);
            const BatchSystem &sy = v.sys[e.x];
            const Cta cta{e.y, e.z};
            const MasView mas = sy.mas;
            coarse_levels_body<BD>(mas, sy.st, cta);
        }

        // The coarse levels for nodes of NC components (the wide groups: 3 components x 16 right-hand
        // sides): a thread per component of a node, whose 32 children's values, consecutive over the
        // threads, are all on their way at once and are added in warp_sum's order (the bits of
        // k_coarse_levels). Level 1 over the device, the few nodes above it in the last CTA to finish. A
        // warp per node and eight components at a time, two warp sums in a row per value, took 40 us
        // at 40^3 in three CTAs, now 16 us (both with about 6 us of the timing events).
        constexpr int LEVEL_C_NODES = 4; // nodes of a CTA at a time

        template <int NC>
        __device__ __forceinline__ void kid_sums(const MasView &mas, int l, int i0, int count,
                                                 int (&kid)[LEVEL_C_NODES][32])
        {
            __syncthreads(); // the previous nodes' indices are done with; their sums are written
            for (int q = threadIdx.x; q < LEVEL_C_NODES * 32; q += LEVEL_C_NODES * NC)
            {
                const int i = i0 + q / 32;
                int node = -1;
                if (i < count)
                {
                    const int b = mas.kid_ptr[l][i], e = mas.kid_ptr[l][i + 1];
                    if (b + q % 32 < e)
                        node = mas.coff[l - 1] + mas.kids[b + q % 32];
                }
                kid[q / 32][q % 32] = node;
            }
            __syncthreads();
            const int k = threadIdx.x / NC, c = threadIdx.x - k * NC;
            if (i0 + k >= count)
                return;
            double v[32];
#pragma unroll
            for (int q = 0; q < 32; ++q)
            {
                const int node = kid[k][q];
                v[q] = node >= 0 ? __ldcg(mas.rc + (size_t)node * NC + c) : 0.0;
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1)
#pragma unroll
                for (int q = 0; q < o; ++q)
                    v[q] += v[q + o];
            mas.rc[((size_t)mas.coff[l] + i0 + k) * NC + c] = v[0];
        }

        template <int NC>
        __global__ void __launch_bounds__(LEVEL_C_NODES *NC) k_coarse_levels_c(MasView mas, const PcgState *grp)
        {
            if (grp && grp->done)
                return;
            __shared__ int kid[LEVEL_C_NODES][32];
            __shared__ int is_last;
            kid_sums<NC>(mas, 1, blockIdx.x * LEVEL_C_NODES, mas.real_count[1], kid);
            if (mas.level_num <= 2)
                return;
            __syncthreads();
            if (threadIdx.x == 0)
            {
                __threadfence(); // cumulative: orders this CTA's stores (seen at the barrier) first
                is_last = atomicAdd(mas.ticket, 1u) == gridDim.x - 1;
            }
            __syncthreads();
            if (!warp_uniform(is_last))
                return;
            __threadfence();
            for (int l = 2; l < mas.level_num && l <= 3; ++l)
                for (int i0 = 0; i0 < mas.real_count[l]; i0 += LEVEL_C_NODES)
                    kid_sums<NC>(mas, l, i0, mas.real_count[l], kid);
            if (threadIdx.x == 0)
                *mas.ticket = 0u;
        }

        // Level-0 restriction of r (initial residual, true-residual iterations, plain applies).
        // With period > 0 it runs only on iterations st->iter + 1 that are multiples of period.
        template <int BD>
        __device__ __forceinline__ void restrict_body(int banks, const double *__restrict__ r,
                                                      const int *__restrict__ lcco0, const int *__restrict__ cco0_base,
                                                      double *rc, const PcgState *st, int period, Cta cta)
        {
            pdl_wait();
            if (st && st->done)
                return;
            if (st && period > 0 && (st->iter + 1) % period != 0)
                return;
            const int lane = threadIdx.x & 31;
            const int bank = cta.x * 8 + warp_index();
            if (bank >= banks)
                return;
            const long long b0 = (long long)bank * 32 * BD;
            double reg[BD];
#pragma unroll
            for (int t = 0; t < BD; ++t)
                reg[t] = r[b0 + t * 32 + lane];
            bank_restrict<BD>(reg, bank, lcco0, cco0_base, rc);
        }

        template <int BD>
        __global__ void __launch_bounds__(256) k_restrict(int banks, const double *__restrict__ r,
                                                          const int *__restrict__ lcco0,
                                                          const int *__restrict__ cco0_base, double *rc,
                                                          const PcgState *st, int period)
        {
            restrict_body<BD>(banks, r, lcco0, cco0_base, rc, st, period, native_cta());
        }

        template <int BD>
        __global__ void __launch_bounds__(256) k_restrict_batch(BatchView v, int period)
        {
            const int4 e = batch_entry(v, BPH_RESTRICT);
            const BatchSystem &sy = v.sys[e.x];
            const Cta cta{e.y, e.z};
            restrict_body<BD>(sy.mas.first_iso_bank, sy.r, sy.mas.lcco0, sy.mas.cco0_base, sy.mas.rc, sy.st, period,
                              cta);
        }

        template <int BD>
        __global__ void k_prolong(MasView mas, const double *__restrict__ z0, double *__restrict__ z)
        {
            const long long len = (long long)mas.banks * 32 * BD;
            for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len;
                 i += (long long)gridDim.x * blockDim.x)
            {
                const long long node = i / BD;
                const int comp = (int)(i % BD);
                if ((node >> 5) >= mas.first_iso_bank)
                {
                    z[i] = (1.0 + mas.level_num) * z0[i];
                    continue;
                }
                const int4 cs = mas.cslot[node];
                double v = z0[i];
                if (cs.x >= 0)
                    v += mas.zc[(size_t)cs.x * BD + comp];
                if (cs.y >= 0)
                    v += mas.zc[(size_t)cs.y * BD + comp];
                if (cs.z >= 0)
                    v += mas.zc[(size_t)cs.z * BD + comp];
                if (cs.w >= 0)
                    v += mas.zc[(size_t)cs.w * BD + comp];
                z[i] = v;
            }
        }

        template <int BD, class Store>
        void prepare_variant()
        {
            using L = ApplyLayout<BD, Store>;
            const int smem = L::SMEM;
            cuda_check(cudaFuncSetAttribute(k_mas_apply<BD, Store, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            smem),
                       "apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply<BD, Store, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            smem),
                       "apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply<BD, Store, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            smem),
                       "apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply_batch<BD, Store, 1>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                       "apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply_batch<BD, Store, 2>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                       "apply smem attribute");
        }

        template <int BD, class Store, int MODE>
        void apply_launch_mode(const MasView &mas, const double *r, double *z, PcgState *st, ReduceBuf red,
                               PcgConfig cfg, bool after_levels, cudaStream_t s)
        {
            using L = ApplyLayout<BD, Store>;
            const size_t smem = L::SMEM;
            const int grid = mas_apply_grid(mas);
            if (MODE != 0 && grid > red.capacity)
                throw Error(ERR_INVALID, "[MAS] reduction scratch too small");
            // Chained in the PCG loop only: the kernel reads inverses before pdl_wait(), and a plain
            // apply may follow the kernels that write them.
            launch_chained(MODE != 0 && chained_launch(), k_mas_apply<BD, Store, MODE>, grid, L::WARPS * 32, smem, s,
                           mas, r, z, st, red, cfg, (int)(MODE != 0 && after_levels));
        }

        template <int BD, class Store>
        void apply_launch(const MasView &mas, const double *r, double *z, PcgState *st, ReduceBuf red, PcgConfig cfg,
                          int mode, bool after_levels, cudaStream_t s)
        {
            if (mode == 0)
                apply_launch_mode<BD, Store, 0>(mas, r, z, st, red, cfg, after_levels, s);
            else if (mode == 1)
                apply_launch_mode<BD, Store, 1>(mas, r, z, st, red, cfg, after_levels, s);
            else
                apply_launch_mode<BD, Store, 2>(mas, r, z, st, red, cfg, after_levels, s);
        }

        // Calls f.template operator()<BD, Store>() for the block size and storage type.
        template <class F>
        auto dispatch(int bd, int storage, F &&f)
        {
            switch (storage)
            {
            case STORE_F64:
                return bd == 1 ? f.template operator()<1, double>()
                               : (bd == 2 ? f.template operator()<2, double>() : f.template operator()<3, double>());
            case STORE_F16:
                return bd == 1 ? f.template operator()<1, __half>()
                               : (bd == 2 ? f.template operator()<2, __half>() : f.template operator()<3, __half>());
            default:
                return bd == 1 ? f.template operator()<1, float>()
                               : (bd == 2 ? f.template operator()<2, float>() : f.template operator()<3, float>());
            }
        }

        template <class F>
        auto dispatch_bd(int bd, F &&f)
        {
            return bd == 1 ? f.template operator()<1>() : (bd == 2 ? f.template operator()<2>() : f.template operator()<3>());
        }
    } // namespace

    int device_sm_count()
    {
        // Per host thread: batched solves run handles on several threads at once.
        static thread_local int cached_dev = -1, cached = 148;
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev != cached_dev)
        {
            int v = 0;
            if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0)
                cached = v;
            cached_dev = dev;
        }
        return cached;
    }

    void prepare_kernels(int bd, int storage)
    {
        device_sm_count();
        dispatch(bd, storage, [&]<int BD, class Store>() { prepare_variant<BD, Store>(); });
    }

    int restrict_grid(const MasView &mas)
    {
        if (mas.first_iso_bank <= 0 || mas.level_num <= 0)
            return 0;
        return (mas.first_iso_bank + 7) / 8;
    }

    int coarse_levels_grid(const MasView &mas)
    {
        if (mas.level_num <= 1 || mas.real_count[1] <= 0)
            return 0;
        const int grid = mas.level_num == 2 ? (mas.real_count[1] + LEVEL_THREADS / 32 - 1) / (LEVEL_THREADS / 32)
                                            : mas.real_count[2];
        return grid > 0 ? grid : 0;
    }

    // At least apply_items_per_warp() items per warp or team of warps (1 by default: the most CTAs, the lowest
    // latency for a lone solve). In batches of small systems more items per warp measured
    // faster: a warp's two-stage copy pipeline runs past its start-up latency, and fewer SMs are
    // held by one system's apply while other systems' kernels run.
    int mas_apply_grid(const MasView &mas)
    {
        return dispatch(mas.bd, mas.storage, [&]<int BD, class Store>() {
            using L = ApplyLayout<BD, Store>;
            const int sms = device_sm_count();
            const int items = mas.banks + mas.n_coarse_active;
            const int per_cta = L::TEAMS * apply_items_per_warp();
            int grid = (items + per_cta - 1) / per_cta;
            if (grid > sms)
                grid = sms;
            return grid < 1 ? 1 : grid;
        });
    }

    void launch_restrict_batch(const BatchView &v, int bd, int total, int period, cudaStream_t s)
    {
        if (total <= 0)
            return;
        dispatch_bd(bd, [&]<int BD>() {
            launch_chained(chained_launch(), k_restrict_batch<BD>, total, 256, 0, s, v, period);
        });
        cuda_check(cudaGetLastError(), "batched restrict launch");
    }

    void launch_coarse_levels_batch(const BatchView &v, int bd, int total, cudaStream_t s)
    {
        if (total <= 0)
            return;
        dispatch_bd(bd, [&]<int BD>() {
            launch_chained(chained_launch(), k_coarse_levels_batch<BD>, total, LEVEL_THREADS, 0, s, v);
        });
        cuda_check(cudaGetLastError(), "batched coarse levels launch");
    }

    void launch_mas_apply_batch(const BatchView &v, int bd, int storage, int total, int mode, cudaStream_t s)
    {
        if (mode != 1 && mode != 2)
            throw Error(ERR_INVALID, "[MAS] internal: batched applies are the initial and the iteration apply");
        if (total <= 0)
            return;
        dispatch(bd, storage, [&]<int BD, class Store>() {
            using L = ApplyLayout<BD, Store>;
            const size_t smem = L::SMEM;
            if (mode == 1)
                launch_chained(chained_launch(), k_mas_apply_batch<BD, Store, 1>, total, L::WARPS * 32, smem, s, v);
            else
                launch_chained(chained_launch(), k_mas_apply_batch<BD, Store, 2>, total, L::WARPS * 32, smem, s, v);
        });
        cuda_check(cudaGetLastError(), "batched apply launch");
    }

    int launch_restrict(const MasView &mas, const double *r, const PcgState *st, int period, cudaStream_t s)
    {
        const int grid = restrict_grid(mas);
        if (grid <= 0)
            return 0;
        dispatch_bd(mas.bd, [&]<int BD>() {
            launch_chained(chained_launch(), k_restrict<BD>, grid, 256, 0, s, mas.first_iso_bank, r, mas.lcco0,
                           mas.cco0_base, mas.rc, st, period);
        });
        return 1;
    }

    int launch_coarse_levels(const MasView &mas, const PcgState *st, cudaStream_t s)
    {
        const int grid = coarse_levels_grid(mas);
        if (grid <= 0)
            return 0;
        dispatch_bd(mas.bd,
                    [&]<int BD>() { launch_chained(chained_launch(), k_coarse_levels<BD>, grid, LEVEL_THREADS, 0, s, mas, st); });
        return 1;
    }

    void prepare_kernels_g(int bd)
    {
        dispatch_bd(bd, [&]<int BD>() {
            using L = ApplyLayoutG<BD>;
            const int smem = L::WARPS * L::WARP_BYTES;
            cuda_check(cudaFuncSetAttribute(k_mas_apply_g<BD, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                       "apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply_g<BD, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                       "apply smem attribute");
        });
        if (bd == 3)
        {
            const int smem = ApplyLayoutW::WARPS * ApplyLayoutW::WARP_BYTES;
            cuda_check(cudaFuncSetAttribute(k_mas_apply_w<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                       "wide apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply_w<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                       "wide apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply_tc<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            TcLayout::BYTES),
                       "tcgen05 apply smem attribute");
            cuda_check(cudaFuncSetAttribute(k_mas_apply_tc<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            TcLayout::BYTES),
                       "tcgen05 apply smem attribute");
        }
    }

    void launch_mas_apply_g(const MasView &mas, const double *r, double *z, PcgState *st, ReduceBuf red, PcgConfig cfg,
                            int mode, cudaStream_t s)
    {
        if (mas.storage != STORE_F16)
            throw Error(ERR_INVALID, "[MAS] several right-hand sides at once need precision fp16");
        dispatch_bd(mas.bd, [&]<int BD>() {
            using L = ApplyLayoutG<BD>;
            const int items = mas.banks + mas.n_coarse_active;
            int grid = (items + L::WARPS - 1) / L::WARPS;
            const int sms = device_sm_count();
            grid = grid > sms ? sms : (grid < 1 ? 1 : grid);
            if (grid * 3 * RHS_GROUP > red.capacity * 6)
                throw Error(ERR_INVALID, "[MAS] reduction scratch too small");
            const size_t smem = (size_t)L::WARPS * L::WARP_BYTES;
            if (mode == 1)
                k_mas_apply_g<BD, 1><<<grid, L::WARPS * 32, smem, s>>>(mas, r, z, st, red, cfg);
            else
                k_mas_apply_g<BD, 2><<<grid, L::WARPS * 32, smem, s>>>(mas, r, z, st, red, cfg);
        });
        cuda_check(cudaGetLastError(), "multi apply launch");
    }

    int launch_coarse_levels_g(const MasView &mas, cudaStream_t s)
    {
        if (mas.level_num <= 1 || mas.real_count[1] <= 0)
            return 0;
        const int grid = mas.level_num == 2 ? (mas.real_count[1] + LEVEL_THREADS / 32 - 1) / (LEVEL_THREADS / 32)
                                            : mas.real_count[2];
        if (grid <= 0)
            return 0;
        dispatch_bd(mas.bd, [&]<int BD>() {
            k_coarse_levels<BD * RHS_GROUP><<<grid, LEVEL_THREADS, 0, s>>>(mas, nullptr);
        });
        cuda_check(cudaGetLastError(), "multi coarse levels launch");
        return 1;
    }

    int launch_coarse_levels_w(const MasView &mas, const PcgState *grp, cudaStream_t s)
    {
        if (mas.level_num <= 1 || mas.real_count[1] <= 0)
            return 0;
        const int grid = (mas.real_count[1] + LEVEL_C_NODES - 1) / LEVEL_C_NODES;
        k_coarse_levels_c<3 * RHS_WIDE><<<grid, LEVEL_C_NODES * 3 * RHS_WIDE, 0, s>>>(mas, grp);
        cuda_check(cudaGetLastError(), "wide coarse levels launch");
        return 1;
    }

    void launch_mas_apply_w(const MasView &mas, const double *r, double *z, PcgState *st, ReduceBuf red,
                            PcgConfig cfg, int mode, cudaStream_t s)
    {
        using L = ApplyLayoutW;
        if (mas.bd != 3 || mas.storage != STORE_F16)
            throw Error(ERR_INVALID, "[MAS] sixteen right-hand sides need block_dim 3 and fp16 inverses");
        const int items = mas.banks + mas.n_coarse_active;
        int grid = (items + L::WARPS - 1) / L::WARPS;
        const int sms = device_sm_count();
        grid = grid > sms ? sms : (grid < 1 ? 1 : grid);
        if (grid > red.capacity)
            throw Error(ERR_INVALID, "[MAS] reduction scratch too small");
        const size_t smem = (size_t)L::WARPS * L::WARP_BYTES;
        if (mode == 1)
            k_mas_apply_w<1><<<grid, L::WARPS * 32, smem, s>>>(mas, r, z, st, red, cfg);
        else
            k_mas_apply_w<2><<<grid, L::WARPS * 32, smem, s>>>(mas, r, z, st, red, cfg);
        cuda_check(cudaGetLastError(), "wide apply launch");
    }

    size_t tc_storage_bytes(const MasView &mas) { return (size_t)(mas.banks + mas.total_coarse) * TC_MAT_BYTES; }

    void launch_inv_to_tc(const MasView &mas, void *out, cudaStream_t s)
    {
        if (mas.bd != 3 || mas.storage != STORE_F16)
            throw Error(ERR_INVALID, "[MAS] the tcgen05 apply needs block_dim 3 and fp16 inverses");
        const int mats = mas.banks + mas.total_coarse;
        if (mats > 0)
            k_inv_to_tc<<<mats, 256, 0, s>>>(static_cast<const __half *>(mas.inv), static_cast<__half *>(out));
        cuda_check(cudaGetLastError(), "tc storage launch");
    }

    void launch_mas_apply_tc(const MasView &mas, const void *inv_tc_v, const double *r, double *z, PcgState *st,
                             ReduceBuf red, PcgConfig cfg, int mode, cudaStream_t s)
    {
        const __half *inv_tc = static_cast<const __half *>(inv_tc_v);
        if (mas.bd != 3 || mas.storage != STORE_F16 || !inv_tc)
            throw Error(ERR_INVALID, "[MAS] the tcgen05 apply needs block_dim 3, fp16 inverses and the tc storage");
        const int items = mas.banks + mas.n_coarse_active;
        int grid = 2 * device_sm_count(); // two CTAs per SM (83 KB of shared memory each)
        grid = grid > items ? items : grid;
        grid = grid > red.capacity ? red.capacity : grid;
        grid = grid < 1 ? 1 : grid;
        const size_t smem = TcLayout::BYTES;
        if (mode == 1)
            k_mas_apply_tc<1><<<grid, TC_THREADS, smem, s>>>(mas, inv_tc, r, z, st, red, cfg);
        else
            k_mas_apply_tc<2><<<grid, TC_THREADS, smem, s>>>(mas, inv_tc, r, z, st, red, cfg);
        cuda_check(cudaGetLastError(), "tcgen05 apply launch");
    }

    void launch_mas_apply(const MasView &mas, const double *r, double *z, PcgState *st, ReduceBuf red, PcgConfig cfg,
                          int mode, bool after_levels, cudaStream_t s)
    {
        dispatch(mas.bd, mas.storage, [&]<int BD, class Store>() {
            apply_launch<BD, Store>(mas, r, z, st, red, cfg, mode, after_levels, s);
        });
    }

    void launch_prolong(const MasView &mas, const double *z0, double *z, cudaStream_t s)
    {
        const long long len = (long long)mas.banks * 32 * mas.bd;
        long long g = (len + 255) / 256;
        if (g > 148 * 16)
            g = 148 * 16;
        if (g < 1)
            g = 1;
        dispatch_bd(mas.bd, [&]<int BD>() { k_prolong<BD><<<(int)g, 256, 0, s>>>(mas, z0, z); });
        cuda_check(cudaGetLastError(), "prolong launch");
    }
} // namespace pmas
