// Register-sliding FP32 step kernel: the FP32 performance path.
//
// Work decomposition: a strip of 128 computed columns (4 per lane) whose middle 112 are its
// output slides down a segment of rows, two rows per round (one in the fused form). A producer and a consumer warp
// share the round and meet at one named barrier (or, in the fused form, one warp does it all);
// x-neighbours come from warp shuffles (radius 1) or a shared-memory row (radius 4), and the
// y-direction order-8 stencils (D8_y o D8_y of the passive current, radius 8) read shared-memory
// rings of the rows held per lane.
//
// For row k:
//   stage A (row k)     lap, grad phi, mu_p, mu_a, zeta*lap*grad phi from phi rows k-1..k+1   (producer)
//   J1_y   (row k-4)    -D8_y mu_p + mag xi_y                      mu_p ring, rows k-8..k     (producer)
//   DY8    (row k-8)    D8_y J1_y                                  J1_y ring                  (producer)
//   J2     (row k-1)    -Tj mu_a + J_c                             mu_a partials, rows k-2..k (consumer)
//   divTj  (row k-2)    Tj . J2                                    J2 partials, rows k-3..k-1 (consumer)
//   output (row k-8)    J1_x = -D8_x mu_p + mag xi_x, DX8 = D8_x J1_x (row exchange),
//                       div J = DX8 + DY8 + divTj (delayed 6 rows), compensated update.       (consumer)
//
// Bound by the FP32 and integer pipes and what latency 16 warps leave uncovered: 186 issue slots per output
// site, 62 % of the issue slots and 54 % of the shared-memory pipe in use. All arithmetic runs on packed
// pairs of columns, with the constants read as pairs from the constant bank; odd x offsets of D8, whose
// pairs are not aligned, are differenced as scalars. Two rows per round share each D8_y window: 8 row
// reads per ring for two rows instead of 15, no mirrored ring rows, half the barriers. The phi rows are
// plain 16-byte loads, one row ahead, with an L2 prefetch. us per step at 4096^2, f32c, T = 0.05 and T = 0,
// 4 pairs per CTA: 132 and 98 (one row per round, mirrored rings: 138 and 109; bulk copies, scalar x
// stencils and per-row ring selects: 183 and 144). Other splits measured there at T = 0.05 against 138: rings
// as register windows 164 (spills at 16 warps per SM), the Tjhung chain moved to the producer 148, three
// warps per strip 174, producer and consumer two rounds apart on split barriers 133 (119 at T = 0, and half
// the CTAs fit in the one-pair form).
//
// Requirements (checked by step_f32_sliding_supported): ncols % 4 == 0 and
// ncols >= 112 (one strip's output width); any nrows >= 1.
//
// Arithmetic per site follows the same separable operators as the tile kernel
// (amb_step_tile.cuh); the noise is the shared Philox definition (amb_common.cuh),
// one Philox4x32-10 call per lane per row and component, so the result does
// not depend on the strip or segment decomposition.
#include "amb_kernels.h"
#include "amb_quad.cuh"
#include "amb_step_tile.cuh"

#include <cstdint>
#include <cstring>
#include <type_traits>

namespace amb
{
    namespace sliding
    {
        constexpr int kCols = 128;              // columns computed per warp (4 per lane)
        constexpr int kHalo = 8;                // mu_p halo on each side
        constexpr int kOut = kCols - 2 * kHalo; // 112 output columns per warp
        constexpr int kDelay = 6;               // rounds from divTj of a row to its output
        constexpr int kMupRing = 10;            // fused form: mu_p rows k-9..k (mirrored)
        constexpr int kJ1Ring = 9;              // fused form: J1_y rows k-12..k-4, the 9 rows of one D8_y (mirrored)

        constexpr int kPairMup = 16;  // mu_p rows k-8..k+1 in use and the two the producer fills meanwhile
        constexpr int kPairJ1 = 8;    // J1_y rows k-12..k-5 (rows k-4, k-3 replace the oldest two once they are read)

        // What a warp pair shares. A round takes two rows, so the rings advance by two rows and a window is
        // four row pairs, each contiguous.
        struct __align__(16) PairSmem
        {
            float mup[kPairMup][kCols];   // row r at (r - 1) mod 16
            float j1y[kPairJ1][kCols];    // row r at (r - 1) mod 8 (producer only)
            float hand[2][2][4][kCols];   // producer -> consumer, by round and row: mu_a(k), J_c,y(k), J_c,x(k), DY8(k-8)
            float dtj[kDelay][kCols];     // divTj rows k-8..k-3 (consumer only)
            float xch[2][2][kCols];       // J1_x row exchange of the consumer's lanes
        };

        // Shared memory of one warp that runs every stage of its strip (the fused form). The y rings are
        // written in two places, N rows apart, so that a window of rows is contiguous wherever it starts:
        // its rows are constant offsets from one base.
        struct __align__(16) WarpSmem
        {
            float mup[2 * kMupRing][kCols];
            float j1y[2 * kJ1Ring][kCols];
            float dtj[kDelay][kCols];
            float xch[2][kCols];
        };

        // Rows are read one round ahead of use, which covers the L2's latency; the DRAM's is covered by a
        // prefetch into the L2 some rows earlier (4096^2, one row per round: 136.6 us with it, 146.1 without).
        constexpr int kPrefetch = 4;
        __device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

        struct Task
        {
            int c0;        // strip origin: output columns [c0, c0 + 112)
            int store_lo;  // first column this strip stores (overlapping last strip)
            int r0, r1;    // output rows [r0, r1)
        };

        using Coef = QuadCoef;

        // Four normals of this lane's quad (global quad at column gcol) for one row and component.
        template <int NOISE, class K>
        __device__ __forceinline__ Quad normals(const StepParams& p, const K& k, const float* __restrict__ injected,
                                                int grow, int gcol, int comp)
        {
            if constexpr (NOISE == NOISE_PHILOX)
            {
                U4 ctr{uint32_t(gcol) >> 2, uint32_t(grow), uint32_t(uint64_t(p.step)),
                       (uint32_t(uint64_t(p.step) >> 32) << 1) | uint32_t(comp)};
                U4 q = philox4x32_10_rk(ctr, k.m.rk0, k.m.rk1);
                float2 zc, zs;  // (r cos, r sin) of the draws (x, y) and (z, w)
                box_muller_f32x2(make_uint2(q.x, q.z), make_uint2(q.y, q.w), zc, zs);
                return {make_float2(zc.x, zs.x), make_float2(zc.y, zs.y)};
            }
            else if constexpr (NOISE == NOISE_INJECTED)
                return load_quad(injected + (size_t)comp * p.ny * p.nx + (size_t)grow * p.nx + gcol);
            else
                return zero_quad();
        }

        __device__ __forceinline__ void pair_sync(int id)
        {
            asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
        }

        __device__ __forceinline__ Task make_task(int task, int nstrips, int seg_h, int ny, int nx)
        {
            Task t;
            int strip = task % nstrips, seg = task / nstrips;
            int c0 = strip * kOut;
            t.store_lo = c0;
            if (c0 + kOut > nx) c0 = nx - kOut;  // last strip overlaps its neighbour; stores only its own part
            t.c0 = c0;
            t.r0 = seg * seg_h;
            t.r1 = min(t.r0 + seg_h, ny);
            return t;
        }

        // The lane's four columns of the phi rows from r0 - 9 on, one row fetched ahead, with the row sums
        // and differences of stage A's three rows carried from row to row.
        struct Local
        {
            const float *base, *row;
            int grow, ny, nx, gcol, ecol, lane;
            float4 next;  // row after the newest taken
            float edge;   // lanes 0 and 31: the column beyond the strip
            Quad um, f, Am, A0, Dm, D0;

            __device__ __forceinline__ void fetch()
            {
                next = *reinterpret_cast<const float4*>(row + gcol);
                prefetch_l2((grow + kPrefetch < ny ? row + (size_t)kPrefetch * nx : base) + gcol);
                if (lane == 0 || lane == 31) edge = row[ecol];
                row += nx;
                if (++grow == ny)
                {
                    grow = 0;
                    row = base;
                }
            }
            __device__ __forceinline__ Quad take(Quad& A, Quad& D)
            {
                float l = __shfl_up_sync(0xffffffffu, next.w, 1), r = __shfl_down_sync(0xffffffffu, next.x, 1);
                if (lane == 0) l = edge;
                if (lane == 31) r = edge;
                const Quad v = quad(next);
                A = nsum(l, v, r);
                D = ndiff(l, v, r);
                return v;
            }
            __device__ __forceinline__ Local(const float* phi, int ny_, int nx_, const Task& t, int lane_)
                : base(phi), ny(ny_), nx(nx_), lane(lane_), edge(0.f)
            {
                gcol = wrap_index(t.c0 - 8 + 4 * lane, nx);
                ecol = wrap_index(lane == 0 ? t.c0 - 9 : t.c0 - 8 + kCols, nx);
                grow = wrap_index(t.r0 - 9, ny);
                row = phi + (size_t)grow * nx;
                fetch();
                um = take(Am, Dm);
                fetch();
                f = take(A0, D0);
                fetch();
            }
            // mu_p, mu_a and J_c of the next row
            template <class K>
            __device__ __forceinline__ void step(const K& k, Quad& mup, Quad& mua, Quad& jcy, Quad& jcx)
            {
                Quad Ap, Dp;
                const Quad dn = take(Ap, Dp);
                fetch();
                Quad l = k.s.lA * (Am + Ap);
                l = fma4(k.s.lB, um + dn, l);
                l = fma4(k.s.lC, A0, l);
                const Quad lap = fma4(k.s.lD, f, l);
                const Quad gx = fma4(k.s.gxb, D0, k.s.gxa * (Dm + Dp));
                const Quad gy = fma4(k.s.gyb, dn - um, k.s.gya * (Ap - Am));
                mup = fma4(k.m.nkappa, lap, fma4(fma4(k.m.c, f, k.m.b), f, k.m.a) * f);
                mua = k.m.lambda * fma4(gy, gy, gx * gx);
                const Quad zl = k.m.zeta * lap;
                jcy = zl * gy;
                jcx = zl * gx;
                um = f; f = dn;
                Am = A0; A0 = Ap;
                Dm = D0; D0 = Dp;
            }
        };

        // J1_y and DY8 of one lane's columns from the mu_p and J1_y rings.
        struct Passive
        {
            float *mup, *j1y;  // this lane's columns of ring position 0
            int wb = 0;        // position of mu_p row k-8 in round k: (k - 1) mod 10
            int jb = 0;        // position of J1_y row k-12

            __device__ __forceinline__ float* put_mup(Quad v)  // row k; returns the window's row k-8
            {
                float* w = mup + wb * kCols;
                store_quad(w + 8 * kCols, v);
                store_quad(w + (wb >= 2 ? 8 - kMupRing : 8 + kMupRing) * kCols, v);
                wb = wb + 1 == kMupRing ? 0 : wb + 1;
                return w;
            }
            __device__ __forceinline__ float* put_j1y(Quad v)  // row k-4; returns the window's row k-12
            {
                float* w = j1y + jb * kCols;
                store_quad(w + 8 * kCols, v);
                store_quad(w + (jb >= 1 ? 8 - kJ1Ring : 8 + kJ1Ring) * kCols, v);
                jb = jb + 1 == kJ1Ring ? 0 : jb + 1;
                return w;
            }
            // D8 along y at the centre of the nine rows from w on; the newest is `last`
            static __device__ __forceinline__ Quad d8y(const float2 (&c)[4], const float* w, Quad last)
            {
                Quad s = c[0] * (load_quad(w + 5 * kCols) - load_quad(w + 3 * kCols));
                s = fma4(c[1], load_quad(w + 6 * kCols) - load_quad(w + 2 * kCols), s);
                s = fma4(c[2], load_quad(w + 7 * kCols) - load_quad(w + kCols), s);
                return fma4(c[3], last - load_quad(w), s);
            }
        };

        // J2 and its Tjhung divergence down the rows: step k takes mu_a(k), J_c(k) and gives divTj(k-2).
        struct Active
        {
            Quad sxm0, sxm1, dxm0, dxm1, sxj0, sxj1, dxj0, dxj1, jcy, jcx;
            __device__ __forceinline__ Active()
            {
                sxm0 = sxm1 = dxm0 = dxm1 = sxj0 = sxj1 = dxj0 = dxj1 = jcy = jcx = zero_quad();
            }
            template <class K>
            __device__ __forceinline__ Quad step(const K& k, Quad mua, Quad ncy, Quad ncx)
            {
                const float ml = __shfl_up_sync(0xffffffffu, mua.b.y, 1), mr = __shfl_down_sync(0xffffffffu, mua.a.x, 1);
                const Quad sx = fma4(k.s.p1, nsum(ml, mua, mr), k.s.p3 * mua), dx = ndiff(ml, mua, mr);
                const Quad j2y = fma4(k.s.ndy, sx - sxm0, jcy);
                const Quad j2x = fma4(k.s.jx3, dxm1, fma4(k.s.jx1, dx + dxm0, jcx));
                sxm0 = sxm1; sxm1 = sx;
                dxm0 = dxm1; dxm1 = dx;
                jcy = ncy; jcx = ncx;
                const float yl = __shfl_up_sync(0xffffffffu, j2y.b.y, 1), yr = __shfl_down_sync(0xffffffffu, j2y.a.x, 1);
                const float xl = __shfl_up_sync(0xffffffffu, j2x.b.y, 1), xr = __shfl_down_sync(0xffffffffu, j2x.a.x, 1);
                const Quad sj = fma4(k.s.p1, nsum(yl, j2y, yr), k.s.p3 * j2y), dj = ndiff(xl, j2x, xr);
                Quad v = k.s.tx1 * (dxj0 + dj);
                v = fma4(k.s.tx3, dxj1, v);
                v = fma4(k.s.dyInv, sj - sxj0, v);
                sxj0 = sxj1; sxj1 = sj;
                dxj0 = dxj1; dxj1 = dj;
                return v;
            }
        };

        // J1_x, DX8, the update and the stores of the output rows, R rows at a time.
        template <int COMP, int NOISE, int R>
        struct Output
        {
            const float* phi_in;
            float* phi_out;
            __nv_bfloat16* residual;
            const float* injected;
            float* xch;       // this lane's columns of the warp's exchange rows, two sets of R
            int ny, nx, gcol, grow, last, flip = 0;
            int left, right;  // offsets of the neighbouring quads in a shared row (within it at its ends)
            bool store;
            float4 fnext[R];  // phi and residual of the next output rows
            uint2 rnext[R];

            // Output rows don't wrap; a row past the segment's last is computed from rows in range and not stored.
            __device__ __forceinline__ int at(int j) const { return min(grow + j, ny - 1); }
            __device__ __forceinline__ void ahead()
            {
#pragma unroll
                for (int j = 0; j < R; ++j)
                {
                    const int r = at(j);
                    const size_t i = (size_t)r * nx + gcol;
                    fnext[j] = *reinterpret_cast<const float4*>(phi_in + i);
                    if constexpr (COMP == COMP_BF16)
                    {
                        rnext[j] = *reinterpret_cast<const uint2*>(residual + i);
                        prefetch_l2(residual + (r + kPrefetch < ny ? i + (size_t)kPrefetch * nx : i));
                    }
                }
            }
            __device__ __forceinline__ Output(const float* in, float* out, __nv_bfloat16* res, const float* inj, float* x,
                                              int ny_, int nx_, const Task& t, int lane)
                : phi_in(in), phi_out(out), residual(res), injected(inj), xch(x + 4 * lane), ny(ny_), nx(nx_), grow(t.r0),
                  last(t.r1)
            {
                const int scol = t.c0 - 8 + 4 * lane;
                gcol = wrap_index(scol, nx);
                store = lane >= 2 && lane < 30 && scol >= t.store_lo && scol < nx;
                left = lane == 0 ? 0 : -4;
                right = lane == 31 ? 0 : 4;
            }
            // rows grow .. grow + R - 1, given their consecutive mu_p rows (this lane's columns of shared rows),
            // divTj and DY8
            template <class K>
            __device__ __forceinline__ void rows(const StepParams& p, const K& k, const float* mup, const Quad (&dtj)[R],
                                                 const Quad (&dy8)[R])
            {
                float* e = xch + flip * R * kCols;
                flip ^= 1;
                Quad j1x[R], f[R];
                uint2 rv[R];
#pragma unroll
                for (int j = 0; j < R; ++j)
                {
                    const float* m = mup + j * kCols;
                    const Quad xi = normals<NOISE>(p, k, injected, at(j), gcol, 1);
                    j1x[j] = fma4(k.m.mag, xi, d8x(k.s.nx8, load_quad(m + left), load_quad(m), load_quad(m + right)));
                    store_quad(e + j * kCols, j1x[j]);
                    f[j] = quad(fnext[j]);
                    if constexpr (COMP == COMP_BF16) rv[j] = rnext[j];
                }
                const int row = grow;
                grow += R;
                ahead();
                __syncwarp();  // the other set is rewritten only after the next round's
#pragma unroll
                for (int j = 0; j < R; ++j)
                {
                    const Quad div = d8x(k.s.px8, load_quad(e + j * kCols + left), j1x[j], load_quad(e + j * kCols + right))
                                   + (dtj[j] + dy8[j]);
                    const size_t gi = (size_t)(row + j) * nx + gcol;
                    const bool st = store && (j == 0 || row + j < last);
                    if constexpr (COMP == COMP_BF16)
                    {
                        const Quad rr{make_float2(__uint_as_float(rv[j].x << 16), __uint_as_float(rv[j].x & 0xffff0000u)),
                                      make_float2(__uint_as_float(rv[j].y << 16), __uint_as_float(rv[j].y & 0xffff0000u))};
                        const Quad F = fma4(k.s.dt, div, rr);
                        const Quad nf = f[j] - F;
                        const Quad nr = (nf - f[j]) + F;
                        if (st)
                        {
                            store_quad(phi_out + gi, nf);
                            __nv_bfloat162 lo = __floats2bfloat162_rn(nr.a.x, nr.a.y),
                                           hi = __floats2bfloat162_rn(nr.b.x, nr.b.y);
                            uint2 w;
                            w.x = *reinterpret_cast<uint32_t*>(&lo);
                            w.y = *reinterpret_cast<uint32_t*>(&hi);
                            *reinterpret_cast<uint2*>(residual + gi) = w;
                        }
                    }
                    else if (st)
                        store_quad(phi_out + gi, fma4(k.s.ndt, div, f[j]));
                }
            }
        };

        // The windows of a round that takes rows k and k+1: rows w[0..7] = r-8..r-1 of a ring before its rows r = n0
        // and r+1 = n1; D8 along y centred on rows r-4 and r-3.
        template <int N>
        __device__ __forceinline__ void d8y_two(const float2 (&c)[4], const float* ring, int row, Quad n0, Quad n1, Quad& d0,
                                                Quad& d1)
        {
            Quad w[8];
#pragma unroll
            for (int p = 0; p < 4; ++p)
            {
                const float* q = ring + ((row + 2 * p) & (N - 1)) * kCols;
                w[2 * p] = load_quad(q);
                w[2 * p + 1] = load_quad(q + kCols);
            }
            d0 = c[0] * (w[5] - w[3]);
            d0 = fma4(c[1], w[6] - w[2], d0);
            d0 = fma4(c[2], w[7] - w[1], d0);
            d0 = fma4(c[3], n0 - w[0], d0);
            d1 = c[0] * (w[6] - w[4]);
            d1 = fma4(c[1], w[7] - w[3], d1);
            d1 = fma4(c[2], n0 - w[2], d1);
            d1 = fma4(c[3], n1 - w[1], d1);
        }

        // Producer warp: stage A, the mu_p ring, J1_y with its noise, and DY8, two rows per round: round q takes
        // rows k = 2q + 1 and k + 1. Rows 1..6 feed no divTj row that an output reads, rows 1..8 no J1_y row and
        // rows 1..16 no DY8 row: their rounds run the body without those parts (the first three without a hand-off).
        template <int NOISE, class K>
        __device__ __forceinline__ void producer(PairSmem& sm, const float* __restrict__ phi_in, const StepParams& p,
                                                 const K& k, const float* __restrict__ injected, const Task& t,
                                                 int lane, int bar_id)
        {
            const int rounds = (t.r1 - t.r0 + 17) / 2;
            Local loc(phi_in, p.ny, p.nx, t, lane);
            float *mup = &sm.mup[0][4 * lane], *j1y = &sm.j1y[0][4 * lane], *hands = &sm.hand[0][0][0][4 * lane];
            int nrow = wrap_index(t.r0 - 4, p.ny);  // global row of the next J1_y row
            const auto draw = [&]() {
                const Quad z = normals<NOISE>(p, k, injected, nrow, loc.gcol, 0);
                nrow = nrow + 1 == p.ny ? 0 : nrow + 1;
                return z;
            };
            const auto round = [&](int q, auto hand_tag, auto j1_tag, auto dy_tag) {
                constexpr bool HAND = decltype(hand_tag)::value, J1 = decltype(j1_tag)::value, DY = decltype(dy_tag)::value;
                float* hand = hands + (q & 1) * 8 * kCols;
                Quad m[2];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                {
                    Quad mua, jcy, jcx;
                    loc.step(k, m[i], mua, jcy, jcx);
                    store_quad(mup + ((2 * q + i) & (kPairMup - 1)) * kCols, m[i]);
                    if constexpr (HAND)
                    {
                        store_quad(hand + 4 * i * kCols, mua);
                        store_quad(hand + (4 * i + 1) * kCols, jcy);
                        store_quad(hand + (4 * i + 2) * kCols, jcx);
                    }
                }
                if constexpr (J1)
                {
                    const Quad x0 = draw(), x1 = draw();
                    Quad s0, s1;
                    d8y_two<kPairMup>(k.s.ny8, mup, 2 * q - 8, m[0], m[1], s0, s1);
                    const Quad j0 = fma4(k.m.mag, x0, s0), j1 = fma4(k.m.mag, x1, s1);
                    if constexpr (DY)
                    {
                        Quad d0, d1;
                        d8y_two<kPairJ1>(k.s.py8, j1y, 2 * q + 4, j0, j1, d0, d1);
                        store_quad(hand + 3 * kCols, d0);
                        store_quad(hand + 7 * kCols, d1);
                    }
                    float* o = j1y + ((2 * q + 4) & (kPairJ1 - 1)) * kCols;  // where rows k-12, k-11 were
                    store_quad(o, j0);
                    store_quad(o + kCols, j1);
                }
                if constexpr (HAND) pair_sync(bar_id);
            };
            using F = std::false_type;
            using T = std::true_type;
            int q = 0;
#pragma unroll 1
            for (; q < 3; ++q) round(q, F{}, F{}, F{});
            round(q++, T{}, F{}, F{});
#pragma unroll 1
            for (; q < 8; ++q) round(q, T{}, T{}, F{});
#pragma unroll 1
            for (; q < rounds; ++q) round(q, T{}, T{}, T{});
        }

        // Consumer warp: the Tjhung chain from row 7 on (divTj of the first output row takes mu_a from row 7), the
        // output rows k-8 and k-7 from round 8 on. A segment of an odd height computes one row more than it stores.
        template <int COMP, int NOISE, class K>
        __device__ __forceinline__ void consumer(PairSmem& sm, const float* __restrict__ phi_in,
                                                 float* __restrict__ phi_out, __nv_bfloat16* residual, const StepParams& p,
                                                 const K& k, const float* __restrict__ injected, const Task& t, int lane,
                                                 int bar_id)
        {
            const int rounds = (t.r1 - t.r0 + 17) / 2;
            Active act;
            Output<COMP, NOISE, 2> out(phi_in, phi_out, residual, injected, &sm.xch[0][0][0], p.ny, p.nx, t, lane);
            const float* hands = &sm.hand[0][0][0][4 * lane];
            float* delay = &sm.dtj[0][4 * lane];
            const auto tjhung = [&](const float* hand, Quad (&old)[2]) {  // divTj into the ring, six rows older ones out
#pragma unroll
                for (int i = 0; i < 2; ++i, hand += 4 * kCols)
                {
                    const Quad v = act.step(k, load_quad(hand), load_quad(hand + kCols), load_quad(hand + 2 * kCols));
                    old[i] = load_quad(delay + i * kCols);
                    store_quad(delay + i * kCols, v);
                }
                delay = delay == &sm.dtj[kDelay - 2][4 * lane] ? &sm.dtj[0][4 * lane] : delay + 2 * kCols;
            };
            Quad dtj[2];
#pragma unroll 1
            for (int q = 3; q < 8; ++q)
            {
                pair_sync(bar_id);
                tjhung(hands + (q & 1) * 8 * kCols, dtj);
            }
            out.ahead();
#pragma unroll 1
            for (int q = 8; q < rounds; ++q)
            {
                const float* hand = hands + (q & 1) * 8 * kCols;
                pair_sync(bar_id);
                tjhung(hand, dtj);
                const Quad dy8[2] = {load_quad(hand + 3 * kCols), load_quad(hand + 7 * kCols)};
                out.rows(p, k, &sm.mup[(2 * q - 8) & (kPairMup - 1)][4 * lane], dtj, dy8);
            }
        }

        // One warp runs every stage of its strip: the producer's and the consumer's work of each round in
        // one instruction stream, with no hand-off buffers and no barrier between warps. The same
        // operations in the same order as the warp pair, so the same bits.
        template <int COMP, int NOISE, class K>
        __device__ __forceinline__ void fused_strip(WarpSmem& sm, const float* __restrict__ phi_in,
                                                    float* __restrict__ phi_out, __nv_bfloat16* residual,
                                                    const StepParams& p, const K& k,
                                                    const float* __restrict__ injected, const Task& t, int lane)
        {
            const int total = t.r1 - t.r0 + 16;
            Local loc(phi_in, p.ny, p.nx, t, lane);
            Passive pas{&sm.mup[0][4 * lane], &sm.j1y[0][4 * lane]};
            Active act;
            Output<COMP, NOISE, 1> out(phi_in, phi_out, residual, injected, &sm.xch[0][0], p.ny, p.nx, t, lane);
            float* delay = &sm.dtj[0][4 * lane];
            Quad xi = zero_quad();
            int nrow = 0;
            const auto draw = [&]() {
                xi = normals<NOISE>(p, k, injected, nrow, loc.gcol, 0);
                nrow = nrow + 1 == p.ny ? 0 : nrow + 1;
            };
            const auto round = [&](auto j1_tag, auto out_tag) {
                constexpr bool J1 = decltype(j1_tag)::value, OUT = decltype(out_tag)::value;
                Quad mup, mua, jcy, jcx, dy8[1];
                loc.step(k, mup, mua, jcy, jcx);
                const float* w = pas.put_mup(mup);
                if constexpr (J1)
                {
                    const Quad x = xi;
                    draw();
                    const Quad j1y = fma4(k.m.mag, x, Passive::d8y(k.s.ny8, w, mup));
                    const float* v = pas.put_j1y(j1y);
                    if constexpr (OUT) dy8[0] = Passive::d8y(k.s.py8, v, j1y);
                }
                const Quad v = act.step(k, mua, jcy, jcx);
                const Quad dtj[1] = {load_quad(delay)};
                store_quad(delay, v);
                delay = delay == &sm.dtj[kDelay - 1][4 * lane] ? &sm.dtj[0][4 * lane] : delay + kCols;
                // row k-8's neighbour columns: other lanes wrote them rounds ago (out.rows synchronises each round)
                if constexpr (OUT) out.rows(p, k, w, dtj, dy8);
                else __syncwarp();
            };
            using F = std::false_type;
            using T = std::true_type;
#pragma unroll 1
            for (int kl = 1; kl <= 8; ++kl) round(F{}, F{});
            nrow = wrap_index(t.r0 - 4, p.ny);
            draw();
#pragma unroll 1
            for (int kl = 9; kl <= 16; ++kl) round(T{}, F{});
            out.ahead();
#pragma unroll 1
            for (int kl = 17; kl <= total; ++kl) round(T{}, T{});
        }

        template <int COMP, int NOISE, int WARPS>
        __global__ void __launch_bounds__(32 * WARPS)
        sliding_fused_kernel(const float* __restrict__ phi_in, float* __restrict__ phi_out, __nv_bfloat16* residual,
                             const StepParams p, const Coef k, const float* __restrict__ injected, int seg_h,
                             int nstrips, int ntasks)
        {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
            const int task = blockIdx.x * WARPS + warp;
            if (task >= ntasks) return;
            WarpSmem& sm = reinterpret_cast<WarpSmem*>(smem_raw)[warp];
            const Task t = make_task(task, nstrips, seg_h, p.ny, p.nx);
            fused_strip<COMP, NOISE>(sm, phi_in, phi_out, residual, p, k, injected, t, lane);
        }

        template <int COMP, int NOISE, int PAIRS>
        __global__ void __launch_bounds__(64 * PAIRS)
        sliding_kernel(const float* __restrict__ phi_in, float* __restrict__ phi_out, __nv_bfloat16* residual,
                       const StepParams p, const Coef k, const float* __restrict__ injected, int seg_h, int nstrips,
                       int ntasks)
        {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            const int pair = threadIdx.x >> 6, role = (threadIdx.x >> 5) & 1, lane = threadIdx.x & 31;
            const int task = blockIdx.x * PAIRS + pair;
            if (task >= ntasks) return;  // both warps of the pair leave together
            PairSmem& sm = reinterpret_cast<PairSmem*>(smem_raw)[pair];
            const Task t = make_task(task, nstrips, seg_h, p.ny, p.nx);
            if (role == 0)
                producer<NOISE>(sm, phi_in, p, k, injected, t, lane, 1 + pair);
            else
                consumer<COMP, NOISE>(sm, phi_in, phi_out, residual, p, k, injected, t, lane, 1 + pair);
        }
    }

    namespace sliding
    {
        // Batched form: one warp pair (FUSED: one warp) per task of a task table that spans many replicas of
        // different sizes and parameters; the step index comes from device memory so that a captured CUDA
        // graph of several steps can be replayed. The replica's coefficients are copied from their table into
        // shared memory at the start of the task and read from there, where each read costs an instruction and
        // a wavefront; with one stencil for all replicas (SAME) only the model's are, and the stencil's, most
        // of the reads, come from the constant bank as in the single-field kernel (32 replicas of 128 to 1024
        // rows and columns, 6.5 M sites: 76.9 us per step, 85.2 with all coefficients in shared memory).
        // 8 one-pair CTAs per SM: at most 128 registers.
        template <int COMP, int NOISE, bool FUSED, bool SAME>
        __global__ void __launch_bounds__(FUSED ? 32 : 64, FUSED ? 9 : 8)
        sliding_ensemble_kernel(const EnsembleReplica* __restrict__ reps, const Coef* __restrict__ coefs,
                                const QuadStencil stencil, const EnsembleTask* __restrict__ tasks, int parity,
                                const int64_t* __restrict__ step_counter, int step_offset)
        {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            using Smem = typename std::conditional<FUSED, WarpSmem, PairSmem>::type;
            constexpr int NT = FUSED ? 32 : 64;
            const int lane = threadIdx.x & 31;
            Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
            const EnsembleTask bt = tasks[blockIdx.x];
            const EnsembleReplica& rd = reps[bt.replica];
            StepParams p = rd.p;
            p.step = *step_counter + step_offset;
            Coef* kc = reinterpret_cast<Coef*>(smem_raw + sizeof(Smem));
            {
                constexpr int skip = SAME ? int(sizeof(QuadStencil) / 4) : 0;
                const uint32_t* src = reinterpret_cast<const uint32_t*>(coefs + bt.replica);
                uint32_t* dst = reinterpret_cast<uint32_t*>(kc);
                for (int i = skip + threadIdx.x; i < int(sizeof(Coef) / 4); i += NT) dst[i] = src[i];
            }
            if constexpr (FUSED) __syncwarp();
            else __syncthreads();
            Task t;
            int c0 = bt.strip * kOut;
            t.store_lo = c0;
            if (c0 + kOut > p.nx) c0 = p.nx - kOut;
            t.c0 = c0;
            t.r0 = bt.r0;
            t.r1 = bt.r1;
            const QuadCoefParts k{SAME ? stencil : kc->s, kc->m};
            const float* in = rd.phi[parity];
            float* out = rd.phi[parity ^ 1];
            if constexpr (FUSED) fused_strip<COMP, NOISE>(sm, in, out, rd.residual, p, k, nullptr, t, lane);
            else if (threadIdx.x < 32) producer<NOISE>(sm, in, p, k, nullptr, t, lane, 1);
            else consumer<COMP, NOISE>(sm, in, out, rd.residual, p, k, nullptr, t, lane, 1);
        }
    }

    bool step_f32_sliding_supported(int ny, int nx, int variant)
    {
        (void)variant;
        return ny >= 1 && nx >= sliding::kOut && nx % 4 == 0;
    }

    namespace
    {
        // Rows of one segment that minimise waves x (rows + pipeline fill), given how many
        // warp pairs the device keeps resident. Fill rounds cost about 10 full rows.
        int choose_seg_h(int ny, int nx, int resident_pairs)
        {
            const int nstrips = (nx + sliding::kOut - 1) / sliding::kOut;
            double best = 1e300;
            int best_h = ny;
            for (int nsegs = 1; nsegs <= ny; ++nsegs)
            {
                int h = (ny + nsegs - 1) / nsegs;
                if (h < 16 && nsegs > 1) break;
                long long tasks = (long long)nstrips * ((ny + h - 1) / h);
                long long waves = (tasks + resident_pairs - 1) / resident_pairs;
                double cost = double(waves) * (h + 10);
                if (cost < best - 1e-9)
                {
                    best = cost;
                    best_h = h;
                }
            }
            return best_h;
        }

        template <int COMP, int NOISE, int WPB>
        cudaError_t launch_variant(const float* phi_in, float* phi_out, __nv_bfloat16* comp, const StepParams& p,
                                   const float* injected, int seg_h, cudaStream_t stream)
        {
            using namespace sliding;
            const size_t smem = sizeof(PairSmem) * WPB;
            auto kern = sliding_kernel<COMP, NOISE, WPB>;
            static int resident_pairs = 0;  // per kernel variant; the process drives one device type
            if (resident_pairs == 0)
            {
                cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
                if (e != cudaSuccess) return e;
                int dev = 0, sms = 0, blocks = 0;
                if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
                if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
                if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, 64 * WPB, smem)) != cudaSuccess)
                    return e;
                resident_pairs = blocks * WPB * sms > 0 ? blocks * WPB * sms : WPB;
            }
            if (seg_h <= 0) seg_h = choose_seg_h(p.ny, p.nx, resident_pairs);
            const int nstrips = (p.nx + kOut - 1) / kOut;
            const int nsegs = (p.ny + seg_h - 1) / seg_h;
            const int ntasks = nstrips * nsegs;
            const Coef k(p);
            kern<<<(ntasks + WPB - 1) / WPB, 64 * WPB, smem, stream>>>(phi_in, phi_out, comp, p, k, injected, seg_h,
                                                                       nstrips, ntasks);
            return cudaGetLastError();
        }

        template <int COMP, int NOISE, int WARPS>
        cudaError_t launch_fused(const float* phi_in, float* phi_out, __nv_bfloat16* comp, const StepParams& p,
                                 const float* injected, int seg_h, cudaStream_t stream)
        {
            using namespace sliding;
            const size_t smem = sizeof(WarpSmem) * WARPS;
            auto kern = sliding_fused_kernel<COMP, NOISE, WARPS>;
            static int resident = 0;  // per kernel variant; the process drives one device type
            if (resident == 0)
            {
                cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
                if (e != cudaSuccess) return e;
                int dev = 0, sms = 0, blocks = 0;
                if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
                if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
                if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, 32 * WARPS, smem)) != cudaSuccess)
                    return e;
                resident = blocks * WARPS * sms > 0 ? blocks * WARPS * sms : WARPS;
            }
            if (seg_h <= 0) seg_h = choose_seg_h(p.ny, p.nx, resident);
            const int nstrips = (p.nx + kOut - 1) / kOut;
            const int nsegs = (p.ny + seg_h - 1) / seg_h;
            const int ntasks = nstrips * nsegs;
            const Coef k(p);
            kern<<<(ntasks + WARPS - 1) / WARPS, 32 * WARPS, smem, stream>>>(phi_in, phi_out, comp, p, k, injected,
                                                                            seg_h, nstrips, ntasks);
            return cudaGetLastError();
        }

        template <int COMP, int WARPS>
        cudaError_t by_noise_fused(const float* phi_in, float* phi_out, __nv_bfloat16* comp, const StepParams& p,
                                   int noise_mode, const float* injected, int seg_h, cudaStream_t stream)
        {
            switch (noise_mode)
            {
            case NOISE_PHILOX: return launch_fused<COMP, NOISE_PHILOX, WARPS>(phi_in, phi_out, comp, p, injected, seg_h, stream);
            case NOISE_INJECTED: return launch_fused<COMP, NOISE_INJECTED, WARPS>(phi_in, phi_out, comp, p, injected, seg_h, stream);
            default: return launch_fused<COMP, NOISE_OFF, WARPS>(phi_in, phi_out, comp, p, injected, seg_h, stream);
            }
        }

        template <int COMP, int WPB>
        cudaError_t by_noise(const float* phi_in, float* phi_out, __nv_bfloat16* comp, const StepParams& p,
                             int noise_mode, const float* injected, int seg_h, cudaStream_t stream)
        {
            switch (noise_mode)
            {
            case NOISE_PHILOX: return launch_variant<COMP, NOISE_PHILOX, WPB>(phi_in, phi_out, comp, p, injected, seg_h, stream);
            case NOISE_INJECTED: return launch_variant<COMP, NOISE_INJECTED, WPB>(phi_in, phi_out, comp, p, injected, seg_h, stream);
            default: return launch_variant<COMP, NOISE_OFF, WPB>(phi_in, phi_out, comp, p, injected, seg_h, stream);
            }
        }
    }

    // variant: 0 = defaults; otherwise (seg_h << 4) | fused (8) | code, code 1 -> 1, 2 -> 2, 3 -> 4 warp
    // pairs (fused: warps) per CTA.
    cudaError_t launch_step_f32_sliding(const float* phi_in, float* phi_out, __nv_bfloat16* comp, int comp_mode,
                                        const StepParams& p, int noise_mode, const float* injected, int variant,
                                        cudaStream_t stream)
    {
        if (!step_f32_sliding_supported(p.ny, p.nx, variant)) return cudaErrorNotSupported;
        int seg_h = variant >> 4;
        int wpb = variant & 7;
        if (variant & 8)
        {
            if (comp_mode == COMP_BF16)
            {
                if (wpb == 1) return by_noise_fused<COMP_BF16, 1>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
                if (wpb == 2) return by_noise_fused<COMP_BF16, 2>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
                return by_noise_fused<COMP_BF16, 4>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
            }
            if (wpb == 1) return by_noise_fused<COMP_NONE, 1>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
            if (wpb == 2) return by_noise_fused<COMP_NONE, 2>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
            return by_noise_fused<COMP_NONE, 4>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
        }
        if (wpb == 0) wpb = 2;  // faster than 1 from 1000 x 1700 to 4096^2, by 3 to 12 %
        if (comp_mode == COMP_BF16)
        {
            if (wpb == 1) return by_noise<COMP_BF16, 1>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
            if (wpb == 3) return by_noise<COMP_BF16, 4>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
            return by_noise<COMP_BF16, 2>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
        }
        if (wpb == 1) return by_noise<COMP_NONE, 1>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
        if (wpb == 3) return by_noise<COMP_NONE, 4>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
        return by_noise<COMP_NONE, 2>(phi_in, phi_out, comp, p, noise_mode, injected, seg_h, stream);
    }
}

namespace amb
{
    size_t sliding_coef_bytes() { return sizeof(sliding::Coef); }

    namespace
    {
        // A pair's (or, fused, a warp's) shared memory plus its replica's coefficient block.
        template <bool FUSED>
        constexpr size_t ensemble_smem_bytes()
        {
            return (FUSED ? sizeof(sliding::WarpSmem) : sizeof(sliding::PairSmem)) + sizeof(sliding::Coef);
        }

        template <int COMP, int NOISE, bool FUSED, bool SAME>
        cudaError_t ensemble_launch(const EnsembleReplica* reps, const sliding::Coef* coefs, const QuadStencil& stencil,
                                    const EnsembleTask* tasks, int ntasks, int parity, const int64_t* step_counter,
                                    int step_offset, cudaStream_t stream)
        {
            auto kern = sliding::sliding_ensemble_kernel<COMP, NOISE, FUSED, SAME>;
            constexpr size_t smem = ensemble_smem_bytes<FUSED>();
            static bool configured = false;
            if (!configured)
            {
                cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
                if (e != cudaSuccess) return e;
                configured = true;
            }
            kern<<<ntasks, FUSED ? 32 : 64, smem, stream>>>(reps, coefs, stencil, tasks, parity, step_counter, step_offset);
            return cudaGetLastError();
        }

        template <bool FUSED>
        cudaError_t ensemble_resident(int* out)
        {
            auto kern = sliding::sliding_ensemble_kernel<COMP_BF16, NOISE_PHILOX, FUSED, true>;
            constexpr size_t smem = ensemble_smem_bytes<FUSED>();
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            int dev = 0, sms = 0, blocks = 0;
            if (e == cudaSuccess) e = cudaGetDevice(&dev);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, FUSED ? 32 : 64, smem);
            if (e == cudaSuccess) *out = blocks * sms > 0 ? blocks * sms : 1;
            return e;
        }
    }

    void sliding_make_coef(const StepParams& p, void* out)
    {
        sliding::Coef k(p);
        std::memcpy(out, &k, sizeof(k));
    }

    bool sliding_same_stencil(const void* coefs, int n)
    {
        const auto* k = static_cast<const sliding::Coef*>(coefs);
        for (int r = 1; r < n; ++r)
            if (std::memcmp(&k[r].s, &k[0].s, sizeof(QuadStencil)) != 0) return false;
        return true;
    }

    cudaError_t ensemble_resident_pairs(int* out, bool fused)
    {
        return fused ? ensemble_resident<true>(out) : ensemble_resident<false>(out);
    }

    cudaError_t launch_sliding_ensemble(const EnsembleReplica* reps, const void* coefs, const void* shared_coef,
                                        const EnsembleTask* tasks, int ntasks, int parity, const int64_t* step_counter,
                                        int step_offset, int comp_mode, int noise_mode, bool fused, cudaStream_t stream)
    {
        if (ntasks <= 0) return cudaSuccess;
        const auto* table = static_cast<const sliding::Coef*>(coefs);
        QuadStencil st{};
        if (shared_coef) st = static_cast<const sliding::Coef*>(shared_coef)->s;
        const auto go = [&](auto comp, auto noise) {
            constexpr int C = decltype(comp)::value, N = decltype(noise)::value;
            const auto run = [&](auto f, auto s) {
                return ensemble_launch<C, N, decltype(f)::value, decltype(s)::value>(reps, table, st, tasks, ntasks, parity,
                                                                                     step_counter, step_offset, stream);
            };
            if (fused) return shared_coef ? run(std::true_type{}, std::true_type{}) : run(std::true_type{}, std::false_type{});
            return shared_coef ? run(std::false_type{}, std::true_type{}) : run(std::false_type{}, std::false_type{});
        };
        using Bf16 = std::integral_constant<int, COMP_BF16>;
        using None = std::integral_constant<int, COMP_NONE>;
        using Philox = std::integral_constant<int, NOISE_PHILOX>;
        using Off = std::integral_constant<int, NOISE_OFF>;
        const bool noise = noise_mode == NOISE_PHILOX;
        if (comp_mode == COMP_BF16) return noise ? go(Bf16{}, Philox{}) : go(Bf16{}, Off{});
        return noise ? go(None{}, Philox{}) : go(None{}, Off{});
    }
}
