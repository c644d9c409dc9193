// The whole PCG solve of one system in one launch (sm_100a), for systems whose subdomain inverses fit
// in the shared memory of all SMs, or nearly. The iteration kernels of such a system are bound by
// latency: launch, first loads and grid reduction, five times per iteration.
//
// Every CTA (one per SM) owns a fixed set of work items for the whole solve: MAS subdomains (banks,
// with their 32 block rows of the matrix and of x, r, p) and coarse matrices. It keeps in shared
// memory the vectors of its rows, its inverses (those that do not fit pass through a ring of bulk
// copies, on their way while the CTA does something else) and as many of its matrix rows as fit. Only p
// (gathered by the SpMV), the coarse vectors and the dot products pass through global memory, so an
// iteration is four grid barriers:
//
//   y = A p, p.y  | A |  r -= alpha y, r.r, level-0 restriction | B |  coarse sums and matrices | C |
//   beta, x += alpha p, p = z + beta p  | D |
//
// and the level-0 inverses are applied between the arrival at barrier B and the wait. On iterations
// that recompute the true residual a fifth barrier follows the update of x.
//
// The arithmetic and its order are those of the iteration kernels, so the iterates have the same bits:
// every per-bank dot is the warp sum the kernels form, and the totals are added in the order of their
// two-stage reductions (8 banks per CTA for p.Ap and r.r; the apply's teams -- item m belongs to
// team m mod (grid * teams per CTA) -- for r.z). Each CTA computes all totals and the scalar step
// itself.
//
// Measured: persist_max_banks below. An iteration at 20^3 is some 29,000 cycles: four barriers of 2,400 (148
// CTAs), 3,500 for the SpMV (one round of gathers from L2), 4,500 for the totals and the scalar step,
// 5,000 for the coarse levels.

#include <algorithm>
#include <climits>

#include "mas_apply.cuh"

namespace pmas
{
    namespace
    {
        constexpr int PS_THREADS = 384;
        constexpr int PS_WARPS = PS_THREADS / 32;

        // Per-warp scratch of the apply: the binary16 hi / lo input and 32 result rows, or the FP32 input.
        template <int BD, class Store>
        constexpr size_t PS_SCRATCH = StoreTraits<Store>::SCALED ? 128 * BD + 128
                                                                 : (std::is_same_v<Store, float> ? 128 * BD : 0);

        struct PersistArgs
        {
            BankedView A;
            MasView mas;
            PcgConfig cfg;
            PcgState *st;
            double *x, *r;
            double *pg, *xg; // p, and x of the last true residual, as the SpMV gathers them
            const double *b;
            double *dots;  // per-bank and per-team dots (persist_dots_size)
            unsigned *bar; // arrivals at the grid barriers of this launch (zero at the start)
            int items;     // banks + active coarse matrices
            int teams;     // teams of the apply: its grid * its teams per CTA
            int vgrid;     // the apply's grid
            int busy;      // teams with work
            int max_items; // most items of a CTA
            int slots, ring, batch; // shared-memory slots for inverses, how many of them are refilled, and how
                                    // many at a time
            int a_bytes;   // shared memory for matrix rows (and the lists of the coarse sums)
            int deep_nodes; // nodes of the coarse levels above the first
            int staged;     // shared memory of the staged dots (doubles)
            int first;      // start the solve (otherwise go on from st, x, r, p)
            int iters;      // iterations of this launch at most
            int period;     // true-residual period (0: never)
            int polls;      // limit of a grid barrier's wait
        };

        // Shared-memory record of one work item. Coarse matrices use r (input) and yz (output) only.
        template <int BD>
        struct alignas(16) ItemRec
        {
            double x[32 * BD], r[32 * BD], p[32 * BD];
            double yz[32 * BD]; // A p, then z
            ushort4 cslot[32]; // coarse nodes per level, 0xFFFF: none
            int len[32];
            signed char key[32];
            const double *avals; // matrix rows: values and columns
            const int *acols;
            double scale;
            int m, mat;      // work item and matrix
            int ident;       // the inverse is exactly the identity
            int resident;    // 1 + offset of the rows' copy in shared memory, 0: none
            int width, base; // bank: slots per row, first component; coarse matrix above the first level:
                             // end of its level in `deep`, and the offset of a coarse node there
        };

        struct PsShared
        {
            PcgState st;
            double red[16];
            double tot[3][16]; // r.z by class, in parts
            uint64_t bar, ring_bar[2];
            int deep_top, deep_lo, deep_hi; // coarse levels above the first: highest level this CTA needs,
                                            // its range of level-1 nodes
            int began; // every CTA had its SM in time
        };

        __device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p)
        {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
            return v;
        }

        __device__ __forceinline__ void red_release_gpu(unsigned *p, unsigned v)
        {
            asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
        }

        // Grid barrier: arrive, then wait, for `limit` polls (some 0.5 us each) after the first. Monotonic arrival
        // count (no reset inside a launch); its top bit (PERSIST_ABORT) tells every CTA that one gave up. A
        // wait that runs out sets it too, and it is the only record of that: the others may be past the
        // barrier by then, and through with the solve.
        __device__ __forceinline__ void ps_arrive(unsigned *bar)
        {
            __syncthreads();
            if (threadIdx.x == 0)
                red_release_gpu(bar, 1u);
        }

        __device__ __forceinline__ bool ps_wait(unsigned *bar, unsigned &target, int limit)
        {
            target += gridDim.x;
            bool gave_up = false;
            if (threadIdx.x == 0)
            {
                unsigned v = ld_acquire_gpu(bar);
#pragma unroll 1
                for (int left = limit; v < target && left > 0; --left)
                    v = ld_acquire_gpu(bar); // the abort bit ends the wait too
                gave_up = v < target || (v & PERSIST_ABORT);
                if (gave_up)
                    atomicOr(bar, PERSIST_ABORT);
            }
            return !__syncthreads_or(gave_up);
        }

        // The first barrier of a launch also finds out whether every CTA has an SM. The launch is a plain one:
        // a cooperative one waits, holding up the launches of every other stream as well, until the whole
        // device is free, and a kernel of another library may keep one SM for long. So a CTA that has waited
        // for `ARRIVE_POLLS` (some 0.1 ms) calls the launch off. That and the last arrival are decided by the
        // same word, so either all go on, each with its SM, or all leave, having changed nothing that
        // counts (PERSIST_LATE tells the host). 20^3 beside a one-CTA kernel of 200 ms: 199 ms for a
        // cooperative launch and 189 ms for a small kernel of a third stream; now 2.6 and 0.07 ms.
        constexpr int ARRIVE_POLLS = 256;

        __device__ __forceinline__ bool ps_begin(unsigned *bar, unsigned &target)
        {
            ps_arrive(bar);
            target += gridDim.x;
            bool leave = false;
            if (threadIdx.x == 0)
            {
                unsigned v = ld_acquire_gpu(bar);
#pragma unroll 1
                for (int i = 0; i < ARRIVE_POLLS && v < target; ++i)
                    v = ld_acquire_gpu(bar); // the abort bit ends the wait too
                // (At most one round per arrival: only those change the word while v < target.)
#pragma unroll 1
                while (v < target)
                {
                    const unsigned seen = atomicCAS(bar, v, v | PERSIST_ABORT | PERSIST_LATE);
                    if (seen == v)
                        break;
                    v = seen;
                }
                leave = (ld_acquire_gpu(bar) & PERSIST_ABORT) != 0;
            }
            return !__syncthreads_or(leave);
        }

        __device__ __forceinline__ bool ps_barrier(unsigned *bar, unsigned &target, int limit)
        {
            ps_arrive(bar);
            return ps_wait(bar, target, limit);
        }

        // Global dots (written before the last grid barrier) into shared memory, 16 bytes per thread and
        // step: every CTA reads the same lines at the same time, so the number of requests counts. `eights`
        // of them with one double of padding after every eight, `groups` with one after every GROUP (the
        // threads that add a group each then hit different banks), the others as they are (GROUP 0: eights
        // only). Counts even.
        template <int GROUP>
        __device__ __forceinline__ void stage_dots(const double *src, unsigned eights, unsigned groups, unsigned count,
                                                   double *dst)
        {
            constexpr unsigned STEP = PS_THREADS * 2, U = 3;
            const unsigned shift = eights / 8, tail = eights + groups, tail_shift = shift + groups / (GROUP ? GROUP : 1);
            auto put = [&](unsigned i, double d) {
                if constexpr (GROUP == 0)
                    dst[i + i / 8] = d;
                else
                    dst[i + (i < eights ? i / 8 : (i < tail ? shift + (i - eights) / GROUP : tail_shift))] = d;
            };
#pragma unroll 1
            for (unsigned i0 = threadIdx.x * 2; i0 < count; i0 += U * STEP)
            {
                double2 d[U];
#pragma unroll
                for (unsigned u = 0; u < U; ++u)
                    d[u] = __ldcg(reinterpret_cast<const double2 *>(src + min(i0 + u * STEP, count - 2)));
#pragma unroll
                for (unsigned u = 0; u < U; ++u)
                    if (i0 + u * STEP < count)
                    {
                        put(i0 + u * STEP, d[u].x);
                        put(i0 + u * STEP + 1, d[u].y);
                    }
            }
        }

        // Sum of staged per-bank dots in the order of the SpMV's and update_xr's two-stage reduction (8
        // banks per CTA, 256 threads in the last CTA). Every thread must call it; `sh` (8 doubles) holds
        // the warp sums after the caller's next barrier, bank_total adds them.
        __device__ __forceinline__ void bank_dots_stage(const double *dots, int banks, double *sh, int w)
        {
            if (w >= 8)
                return;
            const int groups = (banks + 7) / 8;
            double s = 0.0;
            for (int g = threadIdx.x; g < groups; g += 256)
            {
                double t = 0.0;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    t += dots[g * 9 + i];
                s += t;
            }
            s = warp_sum(s);
            if ((threadIdx.x & 31) == 0)
                sh[w] = s;
        }

        __device__ __forceinline__ double bank_total(const double *sh)
        {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w)
                t += sh[w];
            return t;
        }

        // The gathered vectors (p, and x on true-residual iterations) hold a node's values in 32 bytes at
        // block_dim 3, so that one 32-byte load brings them.
        template <int BD>
        constexpr int GATHER_STRIDE = BD == 3 ? 4 : BD;

        template <int BD>
        __device__ __forceinline__ void gather_node(const double *v, int node, double (&x)[BD])
        {
            const double *q = v + node * GATHER_STRIDE<BD>;
            if constexpr (BD == 3)
            {
                double pad;
                asm volatile("ld.global.cg.v4.f64 {%0, %1, %2, %3}, [%4];"
                             : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(pad)
                             : "l"(q)
                             : "memory");
            }
            else if constexpr (BD == 2)
            {
                const double2 t = __ldcg(reinterpret_cast<const double2 *>(q));
                x[0] = t.x;
                x[1] = t.y;
            }
            else
                x[0] = __ldcg(q);
        }

        // One bank's rows of y = A v by one warp (lane = block row). v was written by other CTAs before
        // the last grid barrier. RES: the rows are in shared memory, so only the gathers of v take
        // time: U of them in flight. Otherwise everything comes from L2. Slots past a row's end hold
        // column 0 and zero values, which add zero.
        template <int BD, int U, bool RES>
        __device__ __forceinline__ void bank_rows(const double *vp, const int *cp, int len, int width, const double *v,
                                                  int lane, double (&acc)[BD])
        {
            constexpr int BS = BD * BD, PAIRS = BS / 2;
            cp += lane;
            vp += lane * 2;
            auto load_block = [&](int k, double(&q)[BS]) {
                const double *blk = vp + k * 32 * BS;
#pragma unroll
                for (int i = 0; i < PAIRS; ++i)
                {
                    const double2 *s = reinterpret_cast<const double2 *>(blk + i * 64);
                    const double2 t = RES ? *s : __ldg(s);
                    q[2 * i] = t.x;
                    q[2 * i + 1] = t.y;
                }
                if (BS & 1)
                    q[BS - 1] = RES ? blk[PAIRS * 64 - lane] : __ldg(blk + PAIRS * 64 - lane);
            };
            int cn[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                cn[u] = u < width ? (RES ? cp[u * 32] : __ldg(cp + u * 32)) : 0;
#pragma unroll 1
            for (int k0 = 0; k0 < width; k0 += U)
            {
                double xc[U][BD], m[RES ? 2 : U][BS];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    gather_node<BD>(v, cn[u], xc[u]);
                if (!RES)
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        load_block(min(k0 + u, width - 1), m[RES ? 0 : u]);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    cn[u] = k0 + U + u < width ? (RES ? cp[(k0 + U + u) * 32] : __ldg(cp + (k0 + U + u) * 32)) : 0;
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int j = 0; j < BD; ++j)
                        xc[u][j] = k0 + u < len ? xc[u][j] : 0.0;
                if (RES)
                    load_block(k0, m[0]);
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    if (RES && u + 1 < U)
                        load_block(min(k0 + u + 1, width - 1), m[RES ? (u + 1) & 1 : 0]);
#pragma unroll
                    for (int i = 0; i < BD; ++i)
#pragma unroll
                        for (int j = 0; j < BD; ++j)
                            acc[i] = fma(m[RES ? u & 1 : u][i * BD + j], xc[u][j], acc[i]);
                }
            }
        }

        // Row 32 t + lane of y = M x for one mma16 matrix in shared memory: block rows 2 t and 2 t + 1 of
        // symv_mma16, each block row's products in the same order (block columns left to right, then
        // the diagonal block).
        template <int BD>
        __device__ __forceinline__ float symv_mma16_rows(const __half *M, const __half *xh, const __half *xl, float *ys,
                                                         int t, int lane)
        {
            constexpr int NS = 2 * BD, NB = NS * (NS - 1) / 2;
            const int g = lane >> 2, q = lane & 3;
            const int c = lane >> 3, rr = lane & 7;
            const __half *xsrc = (g == 0) ? xh : xl;
            const uint32_t mbase = smem_addr(M) + (uint32_t)(rr * 16);
            const int ct = (c == 1) ? 2 : (c == 2 ? 1 : c);
            const int cd = (c == 1) ? 1 : (c == 3 ? 2 : 0);
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int R = 2 * t + h;
                float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < NS; ++i)
                {
                    const int S = i < NS - 1 ? (i < R ? i : i + 1) : R; // the diagonal block last
                    const uint32_t b0 = g < 2 ? *reinterpret_cast<const uint32_t *>(xsrc + 16 * S + 2 * q) : 0u;
                    const uint32_t b1 = g < 2 ? *reinterpret_cast<const uint32_t *>(xsrc + 16 * S + 2 * q + 8) : 0u;
                    uint32_t a[4];
                    if (i == NS - 1)
                    {
                        const uint32_t blk = mbase + (uint32_t)((NB * 256 + R * 192) * 2);
                        ldsm_x4_trans(a, blk + cd * 128);
                        a[2] = ldsm_x1(blk + 128);
                    }
                    else
                    {
                        const int lo = S < R ? S : R, hi = S < R ? R : S;
                        const uint32_t blk = mbase + (uint32_t)((lo * (2 * NS - lo - 1) / 2 + (hi - lo - 1)) * 512);
                        if (S > R)
                            ldsm_x4(a, blk + c * 128);
                        else
                            ldsm_x4_trans(a, blk + ct * 128);
                    }
                    mma_16816(d, a, b0, b1);
                }
                if (q == 0)
                {
                    ys[16 * h + g] = d[0] + d[1];
                    ys[16 * h + g + 8] = d[2] + d[3];
                }
            }
            __syncwarp();
            return ys[lane];
        }

        // Rows 32 t .. 32 t + 31 of z = M r for one work item by one warp. The item's record, its inverse M and
        // the warp's scratch are given as offsets in shared memory (as pointers they would be read through
        // generic addresses in a function of its own).
        template <int BD, class Store>
        __device__ __noinline__ void apply_rows(unsigned rec_at, unsigned inv_at, unsigned scratch_at, int t, int lane,
                                                int banks, double *zc)
        {
            using L = ApplyLayout<BD, Store>;
            using Real = typename L::Real;
            constexpr int N = L::N;
            extern __shared__ __align__(128) unsigned char smem[];
            ItemRec<BD> &it = *reinterpret_cast<ItemRec<BD> *>(smem + rec_at);
            const Store *M = reinterpret_cast<const Store *>(smem + inv_at);
            unsigned char *scratch = smem + scratch_at;
            const int e = t * 32 + lane;
            double zv;
            if constexpr (L::MMA)
            {
                __half *xh = reinterpret_cast<__half *>(scratch), *xl = xh + N;
                double rv[BD];
#pragma unroll
                for (int i = 0; i < BD; ++i)
                    rv[i] = it.r[i * 32 + lane];
                const double xscale = half_scale<BD>(rv);
#pragma unroll
                for (int i = 0; i < BD; ++i)
                {
                    const float f = (float)(rv[i] * xscale);
                    const __half h = __float2half_rn(f);
                    xh[i * 32 + lane] = h;
                    xl[i * 32 + lane] = __float2half_rn(f - __half2float(h));
                }
                __syncwarp();
                zv = (double)symv_mma16_rows<BD>(M, xh, xl, reinterpret_cast<float *>(xl + N), t, lane) *
                     (it.scale / xscale);
            }
            else if constexpr (std::is_same_v<Real, double>)
                zv = symv_row<BD>(M, it.r, t, lane);
            else
            {
                float *xs = reinterpret_cast<float *>(scratch);
#pragma unroll
                for (int i = 0; i < BD; ++i)
                    xs[i * 32 + lane] = (float)it.r[i * 32 + lane];
                __syncwarp();
                zv = (double)symv_row<BD>(M, xs, t, lane);
            }
            if (it.ident)
                zv = it.r[e];
            it.yz[e] = zv;
            if (it.m >= banks)
                zc[(size_t)(it.mat - banks) * N + e] = zv;
            __syncwarp(); // the scratch is read
        }

        template <int BD, class Store>
        __global__ void __launch_bounds__(PS_THREADS, 1) k_pcg_persistent(const __grid_constant__ PersistArgs a)
        {
            using L = ApplyLayout<BD, Store>;
            using Rec = ItemRec<BD>;
            constexpr int N = L::N, BS = BD * BD;
            extern __shared__ __align__(128) unsigned char smem[];
            __shared__ PsShared sh;
            const int tid = threadIdx.x, w = warp_index(), lane = tid & 31;
            const MasView &mas = a.mas;
            const int banks = mas.banks;

            // ---- The CTA's items, banks first. With a team per item (single): a contiguous share of the banks
            // (neighbours gather from one another) and every gridDim.x-th coarse matrix, from the last CTA
            // down. Otherwise every gridDim.x-th team from the CTA's index on, item j = (k, i) in increasing
            // order (item m = blockIdx.x + i * gridDim.x + k * teams).
            const int G = (int)gridDim.x, back = G - 1 - (int)blockIdx.x;
            const bool single = a.busy == a.items;
            const int b0 = single ? (int)((long long)blockIdx.x * banks / G) : (int)blockIdx.x;
            int nb, ni, nv; // banks, items, teams
            if (single)
            {
                nb = (int)((long long)(blockIdx.x + 1) * banks / G) - b0;
                nv = ni = nb + (a.items - banks - back + G - 1) / G;
            }
            else
            {
                nv = (a.busy - b0 + G - 1) / G;
                nb = ni = 0;
#pragma unroll 1
                for (int k = b0; k < a.items; k += a.teams)
                {
                    ni += min(nv, (a.items - k + G - 1) / G);
                    nb += max(0, min(nv, (banks - k + G - 1) / G));
                }
            }

            // ---- Shared memory.
            Rec *rec = reinterpret_cast<Rec *>(smem);
            unsigned char *at = smem + (size_t)a.max_items * sizeof(Rec);
            const unsigned scratch_at = (unsigned)(at - smem) + (unsigned)w * PS_SCRATCH<BD, Store>;
            at += (size_t)PS_WARPS * PS_SCRATCH<BD, Store>;
            double *vpart = reinterpret_cast<double *>(at); // 3 * vgrid partials of the apply's dots
            at += (size_t)((3 * a.vgrid + 1) & ~1) * sizeof(double);
            double *deep = reinterpret_cast<double *>(at); // coarse sums above the first level
            at += (size_t)((a.deep_nodes * BD + 1) & ~1) * sizeof(double);
            double *staged = reinterpret_cast<double *>(at); // dots of every CTA
            at += (size_t)a.staged * sizeof(double);
            unsigned short *kids = reinterpret_cast<unsigned short *>(at); // children of the nodes of `deep`
            at += (size_t)a.deep_nodes * 64;
            unsigned char *slots = at; // the inverses
            unsigned char *a_rows = slots + (size_t)a.slots * L::STAGE_BYTES;
            const unsigned char *inv = static_cast<const unsigned char *>(mas.inv);
            // Inverse slots: the coarse matrices and the first `kept` banks keep theirs. Where the other
            // banks' do not fit, they pass through the last slots in batches (at most one round of the
            // CTA's warps), batch g (counted over the launch) through buffer g mod `buffers`.
            const int per = a.batch;
            const int buffers = ni <= a.slots ? 0 : a.ring / per;
            const int kept = buffers ? a.slots - a.ring - (ni - nb) : nb;
            const int batches = (nb - kept + per - 1) / per;
            unsigned char *ring = slots + (size_t)(a.slots - a.ring) * L::STAGE_BYTES;
            // Slot of a kept item: coarse ones first.
            auto slot_of = [&](int j) { return slots + (size_t)(j < nb ? ni - nb + j : j - nb) * L::STAGE_BYTES; };
            auto load_batch = [&](int g) {
                const int first = kept + g % batches * per, n = min(per, nb - first);
                uint64_t *bar = &sh.ring_bar[g % buffers];
                mbar_arrive_expect_tx(bar, (uint32_t)(n * L::STAGE_BYTES));
                for (int i = 0; i < n; ++i)
                    bulk_copy_g2s(ring + (size_t)(g % buffers * per + i) * L::STAGE_BYTES,
                                  inv + (size_t)rec[first + i].mat * L::STAGE_BYTES, L::STAGE_BYTES, bar);
            };

            double *dot_pap = a.dots;
            const int bank_pad = (banks + 7) & ~7, team_pad = (a.busy + 1) & ~1;
            const int extras = a.items - mas.first_iso_bank, first_extra = mas.first_iso_bank % a.teams;
            double *dot_bb = a.dots + bank_pad, *dot_rr = a.dots + 2 * bank_pad, *dot_rz = a.dots + 3 * bank_pad;

            // ---- Load the CTA's part of the system.
            if (tid == 0)
            {
                sh.deep_top = sh.deep_lo = sh.deep_hi = 0;
                mbar_init(&sh.bar, 1);
                mbar_init(&sh.ring_bar[0], 1);
                mbar_init(&sh.ring_bar[1], 1);
                fence_mbar_init();
                unsigned *z = reinterpret_cast<unsigned *>(&sh.st);
                const unsigned *src = reinterpret_cast<const unsigned *>(a.st);
#pragma unroll 1
                for (int i = 0; i < (int)(sizeof(PcgState) / sizeof(unsigned)); ++i)
                    z[i] = a.first ? 0u : src[i];
            }
#pragma unroll 1
            for (int j = w; j < ni; j += PS_WARPS)
            {
                Rec &it = rec[j];
                const int m = single ? (j < nb ? b0 + j : banks + back + (j - nb) * G) : b0 + j % nv * G + j / nv * a.teams;
                if (lane == 0)
                {
                    it.m = m;
                    it.mat = m < banks ? m : banks + mas.coarse_active[m - banks];
                    it.scale = StoreTraits<Store>::SCALED ? mas.inv_scale[it.mat] : 1.0;
                    it.ident = m >= banks ? mas.identity[it.mat - banks] : 0;
                }
                if (m >= banks)
                    continue;
                it.len[lane] = a.A.rowlen[m * 32 + lane];
                it.key[lane] = m < mas.first_iso_bank ? (signed char)mas.lcco0[m * 32 + lane] : -1;
                const int4 cs = mas.cslot[m * 32 + lane];
                it.cslot[lane] = make_ushort4((unsigned short)cs.x, (unsigned short)cs.y, (unsigned short)cs.z,
                                              (unsigned short)cs.w);
#pragma unroll 1
                for (int e = lane; e < N; e += 32)
                {
                    const size_t q = (size_t)m * N + e;
                    const size_t g = (size_t)(m * 32 + e / BD) * GATHER_STRIDE<BD> + e % BD;
                    it.x[e] = a.x[q];
                    it.p[e] = a.first ? 0.0 : a.pg[g];
                    it.r[e] = a.first ? 0.0 : a.r[q];
                    a.xg[g] = it.x[e];
                }
                if (lane == 0)
                {
                    const long long s0 = a.A.slice[m];
                    it.width = (int)(a.A.slice[m + 1] - s0);
                    it.base = m < mas.first_iso_bank ? mas.cco0_base[m] : 0;
                    it.avals = a.A.vals + s0 * 32 * BS;
                    it.acols = a.A.cols + s0 * 32;
                    it.resident = 0;
                }
            }
            __syncthreads();
            if (tid == 0)
            {
                // The inverses, and the matrix rows that fit, by bulk copies on one barrier.
                int used = 0;
#pragma unroll 1
                for (int j = 0; j < nb; ++j)
                {
                    const int bytes = rec[j].width * 32 * (BS * 8 + 4);
                    if (bytes > 0 && used + bytes <= a.a_bytes)
                    {
                        rec[j].resident = 1 + used;
                        used += bytes;
                    }
                }
                mbar_arrive_expect_tx(&sh.bar, (uint32_t)(used + (kept + ni - nb) * L::STAGE_BYTES));
#pragma unroll 1
                for (int g = 0; g < buffers; ++g)
                    load_batch(g);
#pragma unroll 1
                for (int j = 0; j < ni; ++j)
                {
                    if (j < kept || j >= nb)
                        bulk_copy_g2s(slot_of(j), inv + (size_t)rec[j].mat * L::STAGE_BYTES, L::STAGE_BYTES, &sh.bar);
                    if (j >= nb || !rec[j].resident)
                        continue;
                    const uint32_t vb = (uint32_t)rec[j].width * 32 * BS * 8, cb = (uint32_t)rec[j].width * 32 * 4;
                    unsigned char *to = a_rows + rec[j].resident - 1;
                    bulk_copy_g2s(to, rec[j].avals, vb, &sh.bar);
                    bulk_copy_g2s(to + vb, rec[j].acols, cb, &sh.bar);
                }
                // The coarse sums above the first level that this CTA's coarse matrices take.
#pragma unroll 1
                for (int j = nb; j < ni; ++j)
                {
                    const int g0 = (rec[j].mat - banks) * 32; // first coarse node of the matrix
                    int l = 0, below = 0;                     // its level, and the level's first node in `deep`
#pragma unroll 1
                    while (l + 1 < mas.level_num && g0 >= mas.coff[l + 1])
                    {
                        below += l > 0 ? mas.real_count[l] : 0;
                        ++l;
                    }
                    rec[j].base = l > 0 ? below - mas.coff[l] : 0;
                    rec[j].width = l > 0 ? below + mas.real_count[l] : 0;
                    if (l > 0)
                    {
                        const int f = l == 1 ? g0 - mas.coff[1] : 0;
                        const int e = l == 1 ? min(f + 32, mas.real_count[1]) : mas.real_count[1];
                        sh.deep_lo = sh.deep_top == 0 ? f : min(sh.deep_lo, f);
                        sh.deep_hi = max(sh.deep_hi, e);
                        sh.deep_top = max(sh.deep_top, l);
                    }
                }
            }
            __syncthreads();
            // Without its inverses and rows the CTA must not go on: it tells the others and leaves.
            bool ok = __syncthreads_and(mbar_wait_bounded(&sh.bar, 0u, nullptr, a.cfg.wait_limit)) != 0;
            if (!ok && tid == 0)
                atomicOr(a.bar, PERSIST_ABORT);
            unsigned target = 0;
            int batch = 0; // batches multiplied in this launch
            bool gave_up = false; // a wait for a batch ran out
            const int deep_top = warp_uniform(sh.deep_top), deep_lo = warp_uniform(sh.deep_lo),
                      deep_hi = warp_uniform(sh.deep_hi);
            {
                int to = 0; // the level's first node
#pragma unroll 1
                for (int l = 1; l <= deep_top; to += mas.real_count[l], ++l)
#pragma unroll 1
                    for (int i = (l == 1 ? deep_lo : 0) + w; i < (l == 1 ? deep_hi : mas.real_count[l]); i += PS_WARPS)
                    {
                        const int kb = mas.kid_ptr[l][i], ke = mas.kid_ptr[l][i + 1];
                        kids[(to + i) * 32 + lane] = kb + lane < ke ? (unsigned short)mas.kids[kb + lane] : 0xFFFF;
                    }
            }
            // x is where the first residual gathers it once every CTA is past this barrier (which also
            // orders the table above).
            ok = ps_begin(a.bar, target) && ok;
            if (tid == 0)
                sh.began = ok; // (kept here, not in a register through the loop)

#pragma unroll 1
            for (int n = a.first ? -1 : 0; ok; ++n)
            {
                const bool init = n < 0;
                // ---- y = A p and p.y, or (start, and true-residual iterations after their x update)
                // r = b - A x with r.r.
                bool residual = init;
#pragma unroll 1
                for (;;)
                {
                    const double *v = residual ? a.xg : a.pg;
#pragma unroll 1
                    for (int j = w; j < nb; j += PS_WARPS)
                    {
                        Rec &it = rec[j];
                        double acc[BD], part = 0.0, bb = 0.0;
#pragma unroll
                        for (int i = 0; i < BD; ++i)
                            acc[i] = 0.0;
                        const int width = warp_uniform(it.width), copy = warp_uniform(it.resident);
                        if (copy)
                            bank_rows<BD, BD == 3 ? 15 : 9, true>(
                                reinterpret_cast<const double *>(a_rows + copy - 1),
                                reinterpret_cast<const int *>(a_rows + copy - 1 + width * 32 * BS * 8), it.len[lane], width, v,
                                lane, acc);
                        else
                            bank_rows<BD, BD == 3 ? 5 : 8, false>(it.avals, it.acols, it.len[lane], width, v, lane, acc);
#pragma unroll
                        for (int i = 0; i < BD; ++i)
                        {
                            const int e = lane * BD + i;
                            if (residual)
                            {
                                const double bv = a.b[(size_t)it.m * N + e];
                                acc[i] = bv - acc[i];
                                it.r[e] = acc[i];
                                bb = fma(bv, bv, bb);
                            }
                            else
                                it.yz[e] = acc[i];
                            part = fma(acc[i], residual ? acc[i] : it.p[e], part);
                        }
                        part = warp_sum(part);
                        if (init)
                            bb = warp_sum(bb);
                        if (lane == 0)
                        {
                            (residual ? dot_rr : dot_pap)[it.m] = part;
                            if (init)
                                dot_bb[it.m] = bb;
                        }
                    }
                    if (residual)
                        break;
                    if (!(ok = ps_barrier(a.bar, target, a.polls)))
                        break;
                    stage_dots<0>(dot_pap, bank_pad, 0, bank_pad, staged);
                    __syncthreads();
                    bank_dots_stage(staged, banks, sh.red, w);
                    __syncthreads();
                    const double pap = bank_total(sh.red);
                    const double alpha = (fabs(pap) < 1e-20) ? 0.0 : sh.st.rz / pap;
                    residual = a.period > 0 && (warp_uniform(sh.st.iter) + 1) % a.period == 0;
                    if (tid == 0)
                    {
                        sh.st.pAp = pap;
                        sh.st.alpha = alpha;
                    }
#pragma unroll 1
                    for (int j = w; j < nb; j += PS_WARPS)
                    {
                        Rec &it = rec[j];
                        double part = 0.0;
#pragma unroll
                        for (int t = 0; t < BD; ++t)
                        {
                            const int e = t * 32 + lane;
                            if (residual)
                            {
                                const double xn = fma(alpha, it.p[e], it.x[e]);
                                it.x[e] = xn;
                                a.xg[(it.m * 32 + e / BD) * GATHER_STRIDE<BD> + e % BD] = xn;
                            }
                            else
                            {
                                const double rv = fma(-alpha, it.yz[e], it.r[e]);
                                it.r[e] = rv;
                                part = fma(rv, rv, part);
                            }
                        }
                        if (residual)
                            continue;
                        part = warp_sum(part);
                        if (lane == 0)
                            dot_rr[it.m] = part;
                    }
                    if (!residual)
                        break;
                    if (!(ok = ps_barrier(a.bar, target, a.polls)))
                        break;
                }
                if (!ok)
                    break;
                // ---- Level-0 restriction of r (a warp's own banks).
                __syncwarp();
#pragma unroll 1
                for (int j = w; j < nb; j += PS_WARPS)
                {
                    Rec &it = rec[j];
                    if (warp_uniform(it.m) >= mas.first_iso_bank)
                        continue;
                    double rv[BD];
#pragma unroll
                    for (int i = 0; i < BD; ++i)
                        rv[i] = it.r[lane * BD + i];
                    warp_segment_store<BD>(rv, it.key[lane], it.base, mas.rc);
                }
                ps_arrive(a.bar);

                // ---- The MAS apply, 32 rows of one matrix per warp. The subdomain matrices need this CTA's
                // r only; the coarse ones every CTA's.
#pragma unroll 1
                for (int part = 0; part < 2; ++part)
                {
                    if (part == 1)
                    {
                        if (!(ok = ps_wait(a.bar, target, a.polls)) || nb == ni)
                            break;
                        // Coarse levels above the first, four nodes per warp: eight lanes per node, four of its
                        // children each, added in the order of the warp sums of k_coarse_levels (children 16
                        // apart first, then 8, 4, 2, 1; absent ones are zero).
                        int from = 0, to = 0; // first node of the level below and of the level
#pragma unroll 1
                        for (int l = 1; l <= deep_top; ++l)
                        {
                            const int hi = l == 1 ? deep_hi : mas.real_count[l];
#pragma unroll 1
                            for (int i = (l == 1 ? deep_lo : 0) + w * 4; i < hi; i += PS_WARPS * 4)
                            {
                                const int node = i + (lane >> 3), s8 = lane & 7;
                                double t[4][BD];
#pragma unroll
                                for (int h = 0; h < 4; ++h)
                                {
                                    const int q = node < hi ? kids[(to + node) * 32 + s8 + 8 * h] : 0xFFFF;
                                    const int at = (q == 0xFFFF ? 0 : (l == 1 ? mas.coff[0] : from) + q) * BD;
#pragma unroll
                                    for (int c = 0; c < BD; ++c)
                                    {
                                        const double v = l == 1 ? __ldcg(mas.rc + at + c) : deep[at + c];
                                        t[h][c] = q == 0xFFFF ? 0.0 : v;
                                    }
                                }
#pragma unroll
                                for (int c = 0; c < BD; ++c)
                                {
                                    double v = (t[0][c] + t[2][c]) + (t[1][c] + t[3][c]);
#pragma unroll
                                    for (int o = 4; o >= 1; o >>= 1)
                                        v += __shfl_xor_sync(FULL, v, o);
                                    if (s8 == 0 && node < hi)
                                        deep[(to + node) * BD + c] = v;
                                }
                            }
                            __syncthreads();
                            from = to;
                            to += mas.real_count[l];
                        }
                        // The coarse inputs.
#pragma unroll 1
                        for (int q = tid; q < (ni - nb) * N; q += PS_THREADS)
                        {
                            Rec &it = rec[nb + q / N];
                            const int e = q % N, node = (it.mat - banks) * 32 + e / BD + it.base;
                            it.r[e] = node < it.width ? deep[node * BD + e % BD]
                                                      : __ldcg(mas.rc + (size_t)(it.mat - banks) * N + e);
                        }
                        __syncthreads();
                    }
                    // 32 rows of one matrix per warp: the kept ones, then (part 0) batch by batch.
                    const int j0 = part ? nb : 0, tasks = (part ? ni - nb : kept) * BD;
#pragma unroll 1
                    for (int k = w; k < tasks; k += PS_WARPS)
                        apply_rows<BD, Store>((j0 + k / BD) * (unsigned)sizeof(Rec), (unsigned)(slot_of(j0 + k / BD) - smem), scratch_at,
                                              k % BD, lane, banks, mas.zc);
                    const int end = part || buffers == 0 ? 0 : batches;
#pragma unroll 1
                    for (int done = 0; done < end; ++done, ++batch)
                    {
                        const int j = kept + done * per + w / BD;
                        if (!mbar_wait_bounded(&sh.ring_bar[batch % buffers], (uint32_t)(batch / buffers) & 1u, nullptr,
                                               a.cfg.wait_limit))
                            gave_up = true;
                        if (w / BD < per && j < nb)
                            apply_rows<BD, Store>(
                                j * (unsigned)sizeof(Rec),
                                (unsigned)(ring - smem) + (unsigned)(batch % buffers * per + w / BD) * L::STAGE_BYTES,
                                scratch_at, w % BD, lane, banks, mas.zc);
                        // Every warp is done with the batch: its buffer takes the batch `buffers` on.
                        if (__syncthreads_or(gave_up))
                            break;
                        if (tid == 0)
                        {
                            fence_proxy_async_smem();
                            load_batch(batch + buffers);
                        }
                    }
                }
                if (!ok)
                    break;
                if (__syncthreads_or(gave_up) && tid == 0)
                    atomicOr(a.bar, PERSIST_ABORT); // barrier C below tells every CTA
                // ---- r.z per team: its coupled banks in order, then the warp sum. A team has at most one item
                // beyond them (an isolated bank or a coarse matrix): its dot on its own, by item.
#pragma unroll 1
                for (int v = w; v < nv; v += PS_WARPS)
                {
                    double c = 0.0, beyond = 0.0;
                    int extra = -1;
#pragma unroll 1
                    for (int j = v; j < ni; j += nv)
                    {
                        const Rec &it = rec[j];
                        double d = 0.0;
#pragma unroll
                        for (int t = 0; t < BD; ++t)
                            d = fma(it.yz[t * 32 + lane], it.r[t * 32 + lane], d);
                        const int m = warp_uniform(it.m);
                        if (m < mas.first_iso_bank)
                            c += d;
                        else
                        {
                            beyond = d;
                            extra = m - mas.first_iso_bank;
                        }
                    }
                    c = warp_sum(c);
                    beyond = warp_sum(beyond);
                    if (lane == 0)
                    {
                        dot_rz[rec[v].m] = c;
                        if (extra >= 0)
                            dot_rz[team_pad + extra] = beyond;
                    }
                }
                if (!(ok = ps_barrier(a.bar, target, a.polls)))
                    break;
                // ---- Totals and the scalar step, in every CTA. The coarse corrections of the warp's first
                // rows of p are on their way meanwhile.
                double zc_next[4];
                ushort4 slot_next;
                auto coarse_of = [&](int k) {
                    const Rec &it = rec[k / BD];
                    const int e = (k % BD) * 32 + lane;
                    const double *zc = mas.zc + e % BD;
                    slot_next = it.cslot[e / BD];
                    auto value = [&](unsigned short q) { return __ldcg(zc + (q == 0xFFFF ? 0 : q) * BD); };
                    zc_next[0] = value(slot_next.x);
                    zc_next[1] = value(slot_next.y);
                    zc_next[2] = value(slot_next.z);
                    zc_next[3] = value(slot_next.w);
                };
                if (w < nb * BD)
                    coarse_of(w);
                if (init)
                {
                    stage_dots<0>(dot_bb, bank_pad, 0, bank_pad, staged);
                    __syncthreads();
                    bank_dots_stage(staged, banks, sh.red + 8, w);
                    __syncthreads();
                }
                double *staged_rz = staged + bank_pad / 8 * 9;
                stage_dots<L::TEAMS>(dot_rr, bank_pad, team_pad, bank_pad + team_pad + ((extras + 1) & ~1), staged);
                __syncthreads();
                bank_dots_stage(staged, banks, sh.red, w);
                for (int i = tid; i < 3 * a.vgrid; i += PS_THREADS)
                {
                    // Class i / vgrid of apply CTA c: its teams' dots in order.
                    const int cls = i < a.vgrid ? 0 : (i < 2 * a.vgrid ? 1 : 2), c = i - cls * a.vgrid;
                    double t = 0.0;
                    if (cls == 0)
                    {
                        const double *q = staged_rz + c * (L::TEAMS + 1);
#pragma unroll
                        for (int k = 0; k < L::TEAMS; ++k)
                            t += c * L::TEAMS + k < a.busy ? q[k] : 0.0;
                    }
                    else
                    {
                        // The items beyond the coupled banks: team first_iso_bank mod teams has the first.
                        const double *q = staged_rz + team_pad + team_pad / L::TEAMS;
                        const int lo = cls == 1 ? 0 : banks - mas.first_iso_bank;
                        const int hi = cls == 1 ? banks - mas.first_iso_bank : extras;
                        const int x0 = c * L::TEAMS - first_extra;
                        if ((x0 + L::TEAMS > lo && x0 < hi) || (x0 < 0 && x0 + a.teams < hi))
#pragma unroll
                            for (int k = 0; k < L::TEAMS; ++k)
                            {
                                const int x = x0 + k < 0 ? x0 + k + a.teams : x0 + k;
                                t += x >= lo && x < hi ? q[x] : 0.0;
                            }
                    }
                    vpart[i] = t;
                }
                __syncthreads();
                // The last apply CTA's sum: TEAMS * 32 threads stride over the CTAs, a warp sum each 32,
                // added in order (by thread 0 below).
                const int rounds = min(L::TEAMS, (a.vgrid + 31) / 32);
#pragma unroll 1
                for (int k = w; k < 3 * rounds; k += PS_WARPS)
                {
                    const int cls = k % 3, r = k / 3;
                    double t = 0.0;
#pragma unroll 1
                    for (int c = r * 32 + lane; c < a.vgrid; c += L::TEAMS * 32)
                        t += vpart[cls * a.vgrid + c];
                    t = warp_sum(t);
                    if (lane == 0)
                        sh.tot[cls][r] = t;
                }
                __syncthreads();
                if (tid == 0)
                {
                    sh.st.rr = bank_total(sh.red);
                    if (init)
                        sh.st.rr0 = bank_total(sh.red + 8);
                    const double Lc = (double)a.cfg.level_num;
                    double tot[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
                    for (int r = 0; r < rounds; ++r)
#pragma unroll
                        for (int i = 0; i < 3; ++i)
                            tot[i] += sh.tot[i][r];
                    sh.st.rz_coarse = tot[2] + Lc * tot[1];
                    sh.st.rzx_coarse = 0.0;
                    pcg_finalize(&sh.st, a.cfg, init ? 1 : 2, tot[0] + tot[1] + sh.st.rz_coarse, 0.0);
                }
                __syncthreads();
                // ---- x += alpha p (unless the true residual's update did it) and p = z + beta p.
                const bool pdo = !warp_uniform(sh.st.done), xdo = !residual;
                const double alpha = sh.st.alpha, beta = sh.st.beta;
                const double iso_scale = 1.0 + mas.level_num;
#pragma unroll 1
                for (int k = w; k < nb * BD; k += PS_WARPS)
                {
                    Rec &it = rec[k / BD];
                    const int e = (k % BD) * 32 + lane;
                    const double po = it.p[e];
                    if (xdo)
                        it.x[e] = fma(alpha, po, it.x[e]);
                    if (!pdo)
                        continue;
                    double v = it.yz[e];
                    if (it.m < mas.first_iso_bank)
                    {
                        if (k != w)
                            coarse_of(k);
                        v += slot_next.x != 0xFFFF ? zc_next[0] : 0.0;
                        v += slot_next.y != 0xFFFF ? zc_next[1] : 0.0;
                        v += slot_next.z != 0xFFFF ? zc_next[2] : 0.0;
                        v += slot_next.w != 0xFFFF ? zc_next[3] : 0.0;
                    }
                    else
                        v = iso_scale * v;
                    const double pn = init ? v : fma(beta, po, v);
                    it.p[e] = pn;
                    a.pg[(it.m * 32 + e / BD) * GATHER_STRIDE<BD> + e % BD] = pn;
                }
                if (!pdo || n + 1 == a.iters)
                    break;
                ok = ps_barrier(a.bar, target, a.polls);
            }

            // ---- Out: x, r, the state (as they were where the launch did not begin); no copy may be in flight
            // when the CTA leaves.
            __syncthreads();
#pragma unroll 1
            for (int j = w; sh.began && j < nb; j += PS_WARPS)
#pragma unroll 1
                for (int e = lane; e < N; e += 32)
                {
                    a.x[(size_t)rec[j].m * N + e] = rec[j].x[e];
                    a.r[(size_t)rec[j].m * N + e] = rec[j].r[e];
                }
            if (tid == 0)
            {
#pragma unroll 1
                for (long long i = 0; i < MBAR_SPIN_LIMIT; ++i)
                    if (mbar_try_wait(&sh.bar, 0u))
                        break;
#pragma unroll 1
                for (int g = batch; g < batch + buffers; ++g)
#pragma unroll 1
                    for (long long i = 0; i < MBAR_SPIN_LIMIT; ++i)
                        if (mbar_try_wait(&sh.ring_bar[g % buffers], (uint32_t)(g / buffers) & 1u))
                            break;
                if (sh.began && blockIdx.x == 0)
                    *a.st = sh.st;
            }
        }

        constexpr size_t PS_SMEM = 232448 - 1024; // dynamic shared memory beside the static part
        static_assert(sizeof(PsShared) <= 1024, "static shared memory of the persistent solve");

        // Banks up to which one launch is the faster way: beyond, an SM's 12 warps are busy with products for
        // longer than the iteration kernels' launches cost. With 148 SMs of 12 warps the time rises by steps:
        // every 1,776 banks one more round of products, every 148 one more bank on an SM. us per iteration, one launch /
        // iteration kernels, on both sides of each line: 3 x 3 blocks FP32 35.1 / 39.2 at 1,716 banks and
        // 42.7 / 39.7 at 1,855, binary16 36.5 / 35.9 at 1,855, 37.1 / 37.7 at 2,000 (29.5 / 35.4 at 1,716); 2 x 2
        // FP64 27.5 / 29.2 at 1,718 and 30.4 / 29.3 at 1,871, FP32 27.6 / 27.7 at 2,220 and 31.3 / 28.0 at 2,275,
        // binary16 26.9 / 27.4 at 2,275, 27.9 / 27.8 at 2,395 and 28.9 / 28.1 at 2,519; scalar FP64 23.1 / 24.9
        // at 3,042, 23.6 / 26.5 at 3,456 and 28.6 / 26.5 at 3,680, FP32 29.2 / 29.4 at 4,921 and 32.2 / 29.0 at 5,200,
        // binary16 28.4 / 28.8 at 5,200 and 30.1 / 28.1 at 5,488. (3 x 3 FP64: 38.5 / 39.9 at 1,350, where
        // the plan below still finds room for the inverses; for a cube of 1,341 banks it does not.)
        template <int BD, class Store>
        constexpr int persist_max_banks()
        {
            if (std::is_same_v<Store, double>)
                return BD == 3 ? 1400 : (BD == 2 ? 1776 : 3200);
            if (std::is_same_v<Store, float>)
                return BD == 3 ? 1776 : (BD == 2 ? 2220 : 4930);
            return BD == 3 ? 1900 : (BD == 2 ? 2300 : PERSIST_MAX_BANKS);
        }

        template <int BD, class Store>
        PersistPlan plan_variant(const MasView &mas)
        {
            using L = ApplyLayout<BD, Store>;
            PersistPlan pl;
            const int sms = device_sm_count();
            const int items = mas.banks + mas.n_coarse_active;
            // The dots are summed as the iteration kernels do for one bank per warp of update_xr.
            if (mas.level_num < 1 || mas.banks < 1 || mas.banks > persist_max_banks<BD, Store>() ||
                update_xr_grid(mas) != (mas.banks + 7) / 8)
                return pl;
            pl.vgrid = mas_apply_grid(mas);
            pl.teams = pl.vgrid * L::TEAMS;
            pl.busy = pl.teams < items ? pl.teams : items;
            pl.grid = pl.busy < sms ? pl.busy : sms;
            // The most items of a CTA (k_pcg_persistent's two divisions of the items).
            const int nv = (pl.busy + pl.grid - 1) / pl.grid;
            if (pl.busy == items)
                for (int c = 0; c < pl.grid; ++c)
                    pl.max_items =
                        std::max(pl.max_items, (int)((long long)(c + 1) * mas.banks / pl.grid) -
                                                   (int)((long long)c * mas.banks / pl.grid) +
                                                   (mas.n_coarse_active - (pl.grid - 1 - c) + pl.grid - 1) / pl.grid);
            else
                for (int k = 0; k < items; k += pl.teams)
                    pl.max_items += std::min(nv, (items - k + pl.grid - 1) / pl.grid);
            pl.deep_nodes = mas.real_count[1] + mas.real_count[2] + mas.real_count[3];
            const int extras = items - mas.first_iso_bank, team_dots = pl.busy + extras + 3;
            pl.staged = (mas.banks + 7) / 8 * 9 + team_dots + team_dots / L::TEAMS + 2;
            pl.staged += pl.staged & 1;
            if (pl.deep_nodes < 0 || pl.deep_nodes > 1024 || mas.total_coarse * 32 >= 0xFFFF || extras > pl.teams)
                return pl;
            const size_t fixed = pl.max_items * sizeof(ItemRec<BD>) + (size_t)PS_WARPS * PS_SCRATCH<BD, Store> +
                                 (size_t)((3 * pl.vgrid + 1) & ~1) * sizeof(double) +
                                 (size_t)((pl.deep_nodes * BD + 1) & ~1) * sizeof(double) +
                                 (size_t)pl.staged * sizeof(double) + (size_t)pl.deep_nodes * 64;
            if (fixed > PS_SMEM)
                return pl;
            const size_t room = PS_SMEM - fixed;
            pl.slots = (int)std::min(room / L::STAGE_BYTES, (size_t)pl.max_items);
            pl.batch = 1;
            if (pl.slots < pl.max_items)
            {
                // Two buffers, each at most one round of the warps.
                const int coarse = (mas.n_coarse_active + pl.grid - 1) / pl.grid + 1; // no CTA has more
                pl.batch = std::min(PS_WARPS / BD, (pl.slots - coarse) / 2);
                if (pl.batch < 1)
                    return pl;
                pl.ring = 2 * pl.batch;
                const int rounds = (pl.max_items - (pl.slots - pl.ring) + pl.batch - 1) / pl.batch;
                if (rounds > 7)
                    return pl;
            }
            pl.a_bytes = (int)((room - (size_t)pl.slots * L::STAGE_BYTES) / 16 * 16);
            pl.smem = fixed + (size_t)pl.slots * L::STAGE_BYTES + pl.a_bytes;
            pl.ok = true;
            return pl;
        }

        template <class F>
        auto dispatch_variant(int bd, int storage, F &&f)
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
    } // namespace

    // Where one launch is the faster path: up to persist_max_banks, with inverses, vectors and coarse lists in
    // shared memory, or the inverses through the ring in at most 7 batches per apply. us per solve_device,
    // iteration kernels -> one launch: 8^3 FP64 1,210 -> 650, 20^3 binary16 1,870 -> 940, 31^3 FP64 2,950 ->
    // 2,710, 37^3 FP32 3,240 -> 2,820, 300^2 plane FP64 3,680 -> 3,240.
    PersistPlan persist_plan(const MasView &mas)
    {
        return dispatch_variant(mas.bd, mas.storage, [&]<int BD, class Store>() { return plan_variant<BD, Store>(mas); });
    }

    size_t persist_dots_size(const MasView &mas, const PersistPlan &pl)
    {
        return 3 * (size_t)((mas.banks + 7) & ~7) + (size_t)pl.busy + (mas.banks + mas.n_coarse_active - mas.first_iso_bank) + 4;
    }

    size_t persist_gather_size(const MasView &mas)
    {
        return 2 * (size_t)mas.banks * 32 * (mas.bd == 3 ? 4 : mas.bd);
    }

    bool prepare_persistent(int bd, int storage)
    {
        return dispatch_variant(bd, storage, [&]<int BD, class Store>() {
            int per_sm = 0;
            if (cudaFuncSetAttribute(k_pcg_persistent<BD, Store>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)PS_SMEM) != cudaSuccess ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pcg_persistent<BD, Store>, PS_THREADS,
                                                              PS_SMEM) != cudaSuccess ||
                per_sm < 1)
            {
                cudaGetLastError();
                return false;
            }
            return true;
        });
    }

    void launch_pcg_persistent(const BankedView &A, const MasView &mas, const PcgConfig &cfg, const PersistPlan &pl,
                               PcgState *st, double *x, double *r, double *gather, const double *b, double *dots,
                               unsigned *bar, int first, int iters, int period, cudaStream_t s)
    {
        PersistArgs a{};
        a.A = A;
        a.mas = mas;
        a.cfg = cfg;
        a.st = st;
        a.x = x;
        a.r = r;
        a.pg = gather;
        a.xg = gather + persist_gather_size(mas) / 2;
        a.b = b;
        a.dots = dots;
        a.bar = bar;
        a.items = mas.banks + mas.n_coarse_active;
        a.teams = pl.teams;
        a.vgrid = pl.vgrid;
        a.busy = pl.busy;
        a.max_items = pl.max_items;
        a.slots = pl.slots;
        a.ring = pl.ring;
        a.batch = pl.batch;
        a.a_bytes = pl.a_bytes;
        a.deep_nodes = pl.deep_nodes;
        a.staged = pl.staged;
        a.first = first;
        a.iters = iters;
        a.period = period;
        a.polls = (int)std::min<long long>(cfg.wait_limit, INT_MAX);
        cuda_check(cudaMemsetAsync(bar, 0, sizeof(unsigned), s), "barrier reset");
        dispatch_variant(mas.bd, mas.storage, [&]<int BD, class Store>() {
            k_pcg_persistent<BD, Store><<<pl.grid, PS_THREADS, pl.smem, s>>>(a);
            cuda_check(cudaGetLastError(), "persistent solve launch");
        });
    }
} // namespace pmas
