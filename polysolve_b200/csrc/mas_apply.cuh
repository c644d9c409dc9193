// Device parts of the MAS apply that several kernels share (sm_100a): the symmetric products of one
// stored subdomain inverse with one vector, the reference's per-iteration scalar work, and the
// shared-memory shape of the streaming apply.
#pragma once

#include <type_traits>

#include "mas_common.cuh"

namespace pmas
{
    namespace
    {
        // Row 32 t + lane of y = M x for one tile-packed symmetric matrix in shared memory, by one warp.
        // Left of the diagonal the lane takes its column of the mirrored tiles, one product (and, over
        // the tiles, one running sum) per row r of a tile, added up as a tree over r; right of it its
        // own row, four partial sums by column modulo 4 per tile (16-byte reads). The order of the
        // additions is fixed by the matrix alone.
        template <int T, class Real>
        __device__ __forceinline__ Real symv_row(const Real *__restrict__ M, const Real *__restrict__ xs, int t, int lane)
        {
            constexpr int VEC = 16 / (int)sizeof(Real), UNITS = 32 / VEC;
            // Opaque to the compiler: the swizzled offsets are formed here (two integer operations each)
            // instead of being kept, and spilled, across the caller's loop.
            asm volatile("" : "+r"(lane));
            M += t * (t - 1) / 2 * 1024 + t * 528; // column tile t
            Real c[32];
#pragma unroll
            for (int r = 0; r < 32; ++r)
                c[r] = Real(0);
            const int u = lane / VEC, o = lane % VEC;
#pragma unroll 1
            for (int I = 0; I < t; ++I, M += 1024)
#pragma unroll
                for (int r = 0; r < 32; ++r)
                    c[r] = fma(M[r * 32 + (u ^ (r & (UNITS - 1))) * VEC + o], xs[32 * I + r], c[r]);
            Real y;
            {
                const Real *xj = xs + 32 * t;
                const int own = lane * (lane + 1) / 2;
                Real a0 = 0, a1 = 0;
#pragma unroll
                for (int j = 0; j < 32; ++j)
                {
                    const Real v = M[j >= lane ? j * (j + 1) / 2 + lane : own + j];
                    const Real x = xj[j];
                    if (j & 1)
                        a1 = fma(j >= lane ? v : Real(0), x, a1);
                    else
                        a0 = fma(j >= lane ? v : Real(0), x, a0);
                    c[j] = fma(j < lane ? v : Real(0), x, c[j]);
                }
#pragma unroll
                for (int s = 16; s >= 1; s >>= 1)
#pragma unroll
                    for (int i = 0; i < s; ++i)
                        c[i] += c[i + s];
                y = (a0 + a1) + c[0];
            }
            M += 528 + t * 1024; // tile (t, t + 1)
#pragma unroll 1
            for (int J = t + 1; J < T; ++J)
            {
                const Real *xj = xs + 32 * J;
                Real a[4] = {Real(0), Real(0), Real(0), Real(0)};
#pragma unroll
                for (int q = 0; q < UNITS; ++q)
                {
                    const Real *p = M + lane * 32 + (q ^ (lane & (UNITS - 1))) * VEC;
                    if constexpr (VEC == 2)
                    {
                        const double2 v = *reinterpret_cast<const double2 *>(p);
                        const double2 x = *reinterpret_cast<const double2 *>(xj + q * VEC);
                        a[(q & 1) * 2] = fma(v.x, x.x, a[(q & 1) * 2]);
                        a[(q & 1) * 2 + 1] = fma(v.y, x.y, a[(q & 1) * 2 + 1]);
                    }
                    else
                    {
                        const float4 v = *reinterpret_cast<const float4 *>(p);
                        const float4 x = *reinterpret_cast<const float4 *>(xj + q * VEC);
                        a[0] = fma(v.x, x.x, a[0]);
                        a[1] = fma(v.y, x.y, a[1]);
                        a[2] = fma(v.z, x.z, a[2]);
                        a[3] = fma(v.w, x.w, a[3]);
                    }
                }
                y += (a[0] + a[1]) + (a[2] + a[3]);
                M += J * 1024 + 528; // tile (t, J + 1)
            }
            return y;
        }

        // Lane l receives sum over lanes of c[l]; c is destroyed. 31 shuffles.
        __device__ __forceinline__ float transpose_sum32(float (&c)[32], int lane)
        {
#pragma unroll
            for (int s = 16; s >= 1; s >>= 1)
            {
                const bool upper = (lane & s) != 0;
#pragma unroll
                for (int i = 0; i < s; ++i)
                {
                    const float send = upper ? c[i] : c[i + s];
                    const float keep = upper ? c[i + s] : c[i];
                    c[i] = keep + __shfl_xor_sync(FULL, send, s);
                }
            }
            return c[0];
        }

        // Column tile J of y = M x for one tile-packed FP32 symmetric matrix (shared memory): adds the
        // row contributions of tiles (I, J), I <= J, to yr[I] and the transposed contributions
        // (rows of tile J) to yr[J]. Lane l owns rows 32 t + l.
        template <int T>
        __device__ __forceinline__ void symv_column(const float *__restrict__ M, const float *__restrict__ xs, int lane,
                                                    int J, float (&yr)[T])
        {
            int off = 0;
#pragma unroll
            for (int jj = 0; jj < T; ++jj)
                if (jj < J)
                    off += jj * 1024 + 528;
            float cy[32];
#pragma unroll
            for (int j = 0; j < 32; ++j)
                cy[j] = 0.f;
#pragma unroll
            for (int I = 0; I < T; ++I)
            {
                if (I >= J)
                    break;
                const float *tile = M + off + I * 1024 + lane * 32;
                const float xI = xs[32 * I + lane];
                float a0 = 0, a1 = 0, a2 = 0, a3 = 0;
#pragma unroll
                for (int j4 = 0; j4 < 8; ++j4)
                {
                    const float4 v = *reinterpret_cast<const float4 *>(tile + (j4 ^ (lane & 7)) * 4);
                    const float4 xv = *reinterpret_cast<const float4 *>(xs + 32 * J + 4 * j4);
                    a0 = fma(v.x, xv.x, a0);
                    a1 = fma(v.y, xv.y, a1);
                    a2 = fma(v.z, xv.z, a2);
                    a3 = fma(v.w, xv.w, a3);
                    cy[4 * j4 + 0] = fma(v.x, xI, cy[4 * j4 + 0]);
                    cy[4 * j4 + 1] = fma(v.y, xI, cy[4 * j4 + 1]);
                    cy[4 * j4 + 2] = fma(v.z, xI, cy[4 * j4 + 2]);
                    cy[4 * j4 + 3] = fma(v.w, xI, cy[4 * j4 + 3]);
                }
                yr[I] += (a0 + a1) + (a2 + a3);
            }
            // Diagonal tile, upper triangle by columns.
            const float *dt = M + off + J * 1024;
            const float xJ = xs[32 * J + lane];
            float a0 = 0, a1 = 0;
#pragma unroll
            for (int j = 0; j < 32; ++j)
            {
                const float v = (lane <= j) ? dt[j * (j + 1) / 2 + lane] : 0.f;
                const float xj = xs[32 * J + j];
                if (j & 1)
                    a1 = fma(v, xj, a1);
                else
                    a0 = fma(v, xj, a0);
                cy[j] = fma((lane < j) ? v : 0.f, xJ, cy[j]);
            }
            yr[J] += (a0 + a1) + transpose_sum32(cy, lane);
        }

        // y = M x by one warp (all column tiles).
        template <int T>
        __device__ __forceinline__ void symv_tiles(const float *__restrict__ M, const float *__restrict__ xs, int lane,
                                                   float (&yr)[T])
        {
#pragma unroll
            for (int t = 0; t < T; ++t)
                yr[t] = 0.f;
#pragma unroll
            for (int J = 0; J < T; ++J)
                symv_column<T>(M, xs, lane, J, yr);
        }

        // ---- Binary16 (mma16 layout): warp tensor-core products, m16n8k16, FP32 accumulation. ----
        __device__ __forceinline__ void ldsm_x4(uint32_t (&a)[4], uint32_t addr)
        {
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                         : "r"(addr));
        }
        __device__ __forceinline__ void ldsm_x4_trans(uint32_t (&a)[4], uint32_t addr)
        {
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                         : "r"(addr));
        }
        __device__ __forceinline__ uint32_t ldsm_x1(uint32_t addr)
        {
            uint32_t a;
            asm volatile("ldmatrix.sync.aligned.m8n8.x1.shared.b16 {%0}, [%1];" : "=r"(a) : "r"(addr));
            return a;
        }
        __device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
        {
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                         "{%8, %9}, {%0, %1, %2, %3};"
                         : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                         : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
        }

        // y = M x for one mma16 matrix in shared memory, by one warp. x enters as two binary16
        // columns (xh + xl = x scaled, ~22 significant bits), the B operand's columns 0 and 1; the
        // FP32 products of column 0 and 1 are added back. Each 16 x 16 block above the diagonal
        // is used twice: as stored for its block row and, loaded transposed, for its block
        // column. The result goes through ys (shared, N floats): lane l gets rows 32 t + l.
        template <int BD>
        __device__ __forceinline__ void symv_mma16(const __half *M, const __half *xh, const __half *xl, float *ys,
                                                   int lane, float (&yr)[BD])
        {
            constexpr int NS = 2 * BD, NB = NS * (NS - 1) / 2;
            const int g = lane >> 2, q = lane & 3;
            const int c = lane >> 3, rr = lane & 7; // ldmatrix: lanes 8c..8c+7 give the rows of core c
            uint32_t bf[NS][2];
            const __half *xsrc = (g == 0) ? xh : xl;
#pragma unroll
            for (int S = 0; S < NS; ++S)
            {
                bf[S][0] = g < 2 ? *reinterpret_cast<const uint32_t *>(xsrc + 16 * S + 2 * q) : 0u;
                bf[S][1] = g < 2 ? *reinterpret_cast<const uint32_t *>(xsrc + 16 * S + 2 * q + 8) : 0u;
            }
            float d[NS][4];
#pragma unroll
            for (int R = 0; R < NS; ++R)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    d[R][i] = 0.f;
            const uint32_t mbase = smem_addr(M);
            const int ct = (c == 1) ? 2 : (c == 2 ? 1 : c); // fragment c of a transposed block
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
            // Diagonal blocks [[D0, C], [C^T, D1]]: transposed loads of (D0, C, -, D1) give
            // fragments 0, 1, 3 (D0, D1 are symmetric); fragment 2 (C) is a plain load.
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
            if (q == 0)
#pragma unroll
                for (int R = 0; R < NS; ++R)
                {
                    ys[16 * R + g] = d[R][0] + d[R][1];
                    ys[16 * R + g + 8] = d[R][2] + d[R][3];
                }
            __syncwarp();
#pragma unroll
            for (int t = 0; t < BD; ++t)
                yr[t] = ys[t * 32 + lane];
        }

        // The power of two that brings the warp's largest |v| to [2^14, 2^15) (1 for all zeros, or where it
        // is not finite): the scale of the binary16 split. Only the exponent counts, so a 32-bit warp
        // maximum of the high words finds it; denormal and non-finite maxima take the general way.
        template <int BD>
        __device__ __forceinline__ double half_scale(const double (&v)[BD])
        {
            unsigned hi = 0;
#pragma unroll
            for (int i = 0; i < BD; ++i)
                hi = max(hi, (unsigned)__double2hiint(v[i]) & 0x7FFFFFFFu);
            const unsigned e = __reduce_max_sync(FULL, hi) >> 20; // biased exponent
            if (e >= 14 && e < 2047)
                return __hiloint2double((int)((2060u - e) << 20), 0); // 2^(14 - (e - 1023))
            double amax = 0.0;
#pragma unroll
            for (int i = 0; i < BD; ++i)
                amax = fmax(amax, fabs(v[i]));
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1)
                amax = fmax(amax, __shfl_xor_sync(FULL, amax, o));
            return (amax > 0.0 && isfinite(amax)) ? ldexp(1.0, 14 - ilogb(amax)) : 1.0;
        }

        // The reference's per-iteration scalar work and convergence test (MASSolver.cu:505,
        // 526-583), run by the last CTA of the apply. rz = r . z, rzcross = r . z_old (Polak-Ribiere).
        __device__ void pcg_finalize(PcgState *st, const PcgConfig &cfg, int mode, double rz, double rzcross)
        {
            if (st->error == ERR_TIMEOUT)
            {
                // A bounded wait gave up in this apply: z is incomplete, stop the solve here.
                st->done = 1;
                return;
            }
            if (mode == 1)
            {
                st->rz = rz;
                st->rz0 = rz;
                st->iter = 0;
                if (isnan(rz) || !isfinite(rz))
                {
                    st->error = ERR_NONFINITE;
                    st->done = 1;
                }
                return;
            }
            // Iteration number from the device state, so a captured chunk of iterations replays.
            const int iter = st->iter + 1;
            const double rz_old = st->rz;
            st->rz_old = rz_old;
            st->rz = rz;
            st->rzold_cross = rzcross;
            st->iter = iter;
            bool conv = false;
            if (iter % cfg.check_period == 0)
            {
                const double rel2 = cfg.rel_tol * cfg.rel_tol, abs2 = cfg.abs_tol * cfg.abs_tol;
                if (cfg.use_prec_norm)
                {
                    st->res_norm = sqrt(rz);
                    if (rz <= rel2 * st->rz0 || rz <= abs2)
                    {
                        st->status = (rz <= abs2) ? 2 : 1;
                        conv = true;
                    }
                }
                else
                {
                    const double rr = st->rr;
                    st->res_norm = sqrt(rr);
                    if (rr <= rel2 * st->rr0 || rr <= abs2)
                    {
                        st->status = (rr <= abs2) ? 2 : 1;
                        conv = true;
                    }
                }
            }
            if (conv)
                st->done = 1;
            else if (cfg.polak_ribiere)
            {
                const double beta = (fabs(rz_old) < 1e-20) ? 0.0 : (rz - rzcross) / rz_old;
                st->beta = beta > 0.0 ? beta : 0.0;
            }
            else
                st->beta = (fabs(rz_old) < 1e-20) ? 0.0 : rz / rz_old;
            if (iter == cfg.max_iter)
            {
                st->status = 3;
                st->done = 1;
            }
        }

        // Shared-memory shape of the streaming apply. A team of warps multiplies one matrix at a time:
        // one warp per 32 rows in FP64, else one warp. Two stages per team, as many teams as fit, at
        // most 16.
        template <int BD, class Store>
        struct ApplyLayout
        {
            using Real = typename StoreTraits<Store>::Real;
            static constexpr int N = 32 * BD;
            static constexpr bool MMA = StoreTraits<Store>::SCALED; // binary16: mma16 layout
            static constexpr int S = MMA ? (2 * BD) * (2 * BD - 1) / 2 * 256 + 2 * BD * 192 : N * (N + 1) / 2;
            static constexpr int STAGE_BYTES = S * (int)sizeof(Store);
            static constexpr bool ROWS = std::is_same_v<Store, double>;
            // x and y of FP64; x of FP32; binary16 hi / lo columns plus the FP32 result rows.
            static constexpr int XS_BYTES = ROWS ? 16 * N : (MMA ? 8 * N : 4 * N);
            static constexpr int TEAM = ROWS ? BD : 1; // warps per matrix
            static constexpr int TEAM_BYTES = 2 * STAGE_BYTES + XS_BYTES + 16;
            static constexpr int SMEM_LIMIT = 232448 - 1536; // leave room for static shared memory
            static constexpr int FIT = SMEM_LIMIT / TEAM_BYTES;
            static constexpr int TEAMS = FIT > 16 ? 16 : FIT;
            static constexpr int WARPS = TEAMS * TEAM;
            static constexpr int SMEM = TEAMS * TEAM_BYTES;
            static_assert(STAGE_BYTES % 16 == 0 && XS_BYTES % 16 == 0, "bulk copies need 16-byte multiples");
        };
    } // namespace
} // namespace pmas
