// FP64 steps of small grids: one tile per SM, many steps in one cooperative launch.
//
// The three-phase kernel (amb_step_phase.cuh) executes the fewest FP64 operations, but each of its
// phases ends in a grid barrier and starts with L2 latency, about 4 us whatever the grid. Here a CTA
// recomputes its tile's halo (for a 14 x 32 tile 1.5 times the operations) and a step has one barrier. The
// FP64 pipe takes 64 cycles per warp instruction and sub-partition, full warp or not, so every stage
// is a list of work items packed into whole warps, dealt out to the warps in turn: the full stage A
// on the middle, mu_p alone on the four arms, J1_y, J1_x and J2 side by side, the three terms of
// div J side by side. An item is a column and a run of rows whose row sums are carried. The noise is
// drawn into the arrays that J1 replaces, for the next step while the barrier completes.
//
// us per step at T = 0.05, this kernel and the three-phase kernel: 64^2 6.0 (12.5), 48 x 100 7.2 (12.7),
// 128^2 9.3 (13.2), 200 x 300 18.4 (20.1).
#pragma once

#include "amb_step_phase.cuh"

namespace amb
{
    namespace dtile
    {
        // Threads per CTA. 512 for the lowest time of one run. A CTA of 256 leaves half an SM's registers to a CTA of
        // another run, so that runs on several streams share the GPU, where a tile's lists are short enough for
        // eight warps. us per step of one run, and per step and run with eight at once, 256 threads (512; one launch
        // per step of the tile kernel): 64^2 6.0 and 3.7 (6.0 and 6.1; 47.7 and 6.4), 96^2 7.5 and 4.9 (7.1 and 7.1;
        // 47.7 and 6.3), 128^2 9.3 and 6.9 (8.9 and 9.0; 47.7 and 6.4), 200^2 16.6 and 12.9 (14.5 and 14.5; 47.7 and
        // 13.7). 512 threads on 64 registers each, two CTAs per SM: 128^2 9.4 and 7.3, 64^2 6.6 and 4.2.
        constexpr int kThreads = 512, kThreadsSmall = 256;
        constexpr double kSitesSmall = 110;  // most sites per SM for the small CTA

        struct Shape
        {
            int ty, tx;  // output rows and columns of a tile, tx a multiple of 4
            __host__ __device__ size_t doubles() const
            {
                return size_t(ty + 18) * (tx + 18) + size_t(ty + 16) * (tx + 16) + size_t(ty + 4) * (tx + 4)
                       + 2 * size_t(ty + 2) * (tx + 2) + size_t(ty + 8) * tx + size_t(ty) * (tx + 8) + size_t(ty) * tx;
            }
        };

        struct Arrays  // rows and columns from -9, -8, -2, -1; J1_y rows from -4, J1_x columns from -4
        {
            double *phi, *mup, *mua, *j2y, *j2x, *j1y, *j1x, *dx8;
            int pw, mw, aw, cw, xw;
            __device__ __forceinline__ Arrays(double* s, const Shape& t)
            {
                pw = t.tx + 18;
                mw = t.tx + 16;
                aw = t.tx + 4;
                cw = t.tx + 2;
                xw = t.tx + 8;
                phi = s;
                mup = phi + (t.ty + 18) * pw;
                mua = mup + (t.ty + 16) * mw;
                j2y = mua + (t.ty + 4) * aw;
                j2x = j2y + (t.ty + 2) * cw;
                j1y = j2x + (t.ty + 2) * cw;
                j1x = j1y + (t.ty + 8) * t.tx;
                dx8 = j1x + t.ty * xw;
            }
        };

        // Deals the items of one list, W columns times the runs of L rows in H, to the CTA's warps; lists
        // given to the same Deal follow one another. f(column, first row, last row + 1).
        template <int NT>
        struct Deal
        {
            int next = 0;
            template <typename F>
            __device__ __forceinline__ void operator()(int W, int H, int L, F&& f)
            {
                const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = NT / 32;
                const int n = W * ((H + L - 1) / L), chunks = (n + 31) >> 5;
                for (int c = (warp - next) & (warps - 1); c < chunks; c += warps)
                {
                    const int item = c * 32 + lane;
                    if (item < n)
                    {
                        const int g = item / W, j = item - g * W;
                        f(j, g * L, min(g * L + L, H));
                    }
                }
                next = (next + chunks) & (warps - 1);
            }
        };

        // xi of the tile's J1_y and J1_x into their arrays, one Philox call per quad of columns where the
        // quad is one of the noise's.
        template <int NT>
        __device__ __forceinline__ void draw(const Arrays& a, const Shape& t, const StepParams& p, int noise_mode,
                                             const double* injected, int r0, int c0)
        {
            if (noise_mode == NOISE_OFF) return;
            const int ny = p.ny, nx = p.nx, qy = t.tx / 4, qx = qy + 2, n1 = qy * (t.ty + 8), n = n1 + qx * t.ty;
            for (int e = threadIdx.x; e < n; e += NT)
            {
                const int comp = e >= n1, k = comp ? e - n1 : e, w = comp ? qx : qy;
                const int i = k / w, j = k - i * w;
                const int row = wrap_index(comp ? r0 + i : r0 + i - 4, ny), u = c0 + 4 * j - (comp ? 4 : 0);
                if (u >= nx + (comp ? 4 : 0)) continue;  // no site of the grid reads it
                double* out = comp ? a.j1x + i * a.xw + 4 * j : a.j1y + i * t.tx + 4 * j;
                const int g = wrap_index(u, nx);
                if (noise_mode == NOISE_PHILOX && (g & 3) == 0 && g + 4 <= nx)
                {
                    float z[4];
                    noise_quad(p.seed, p.step, row, g, comp, z);
#pragma unroll
                    for (int q = 0; q < 4; ++q) out[q] = phase::widen(z[q]);
                }
                else
                    for (int q = 0; q < 4; ++q)
                    {
                        const int col = wrap_index(u + q, nx);
                        out[q] = noise_mode == NOISE_PHILOX
                                     ? phase::widen(noise_normal(p.seed, p.step, row, col, comp))
                                     : injected[comp * size_t(ny) * nx + size_t(row) * nx + col];
                    }
            }
        }

        // Where site e of the tile with its halo lies in the field.
        __device__ __forceinline__ size_t halo_site(const Arrays& a, int e, int ny, int nx, int r0, int c0)
        {
            const int i = e / a.pw, j = e - i * a.pw;
            return size_t(wrap_index(r0 + i - 9, ny)) * nx + wrap_index(c0 + j - 9, nx);
        }

        // One step of the CTA's tile: halo load, stages, update. first: where this thread's first four sites lie,
        // formed once for all steps (the division and the wrap-arounds delayed the loads of each).
        template <int NT>
        __device__ __forceinline__ void step(const Arrays& a, const Shape& t, const phase::Coef& k, const double* in,
                                             double* out, int ny, int nx, int noise_mode, int r0, int c0,
                                             const size_t (&first)[4])
        {
            const int ty = t.ty, tx = t.tx, sites = (ty + 18) * a.pw;
            for (int e = threadIdx.x; e < sites; e += 4 * NT)
            {
                double v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                {
                    const int f = e + q * NT;
                    if (f < sites) v[q] = __ldcg(in + (e < NT ? first[q] : halo_site(a, f, ny, nx, r0, c0)));
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (e + q * NT < sites) a.phi[e + q * NT] = v[q];
            }
            __syncthreads();

            // about one item per thread: runs as long as that allows
            const auto run = [](int sites) { return max(1, sites / NT); };

            // ---- stage A. walk(column, rows, f): f(row, site) down a run, tile coordinates
            const auto walk = [&](int j, int lo, int hi, auto&& f) {
                const double* s = a.phi + (lo + 8) * a.pw + j + 9;
                double um = s[0], Am = kadd(s[-1], s[1], k), Dm = ksub(s[1], s[-1], k);
                s += a.pw;
                double m = s[0], A0 = kadd(s[-1], s[1], k), D0 = ksub(s[1], s[-1], k);
                for (int i = lo; i < hi; ++i)
                {
                    s += a.pw;
                    const double dn = s[0], Ap = kadd(s[-1], s[1], k), Dp = ksub(s[1], s[-1], k);
                    f(i, canon_site_a(um, m, dn, Am, A0, Ap, Dm, D0, Dp, k));
                    um = m; m = dn;
                    Am = A0; A0 = Ap;
                    Dm = D0; D0 = Dp;
                }
            };
            const auto only_mup = [&](int j, int lo, int hi) {  // the unused terms are dead code
                walk(j, lo, hi, [&](int i, const SiteA<double>& s) { a.mup[(i + 8) * a.mw + j + 8] = s.mup; });
            };
            {
                Deal<NT> deal;
                deal(tx + 4, ty + 4, run((tx + 4) * (ty + 4)), [&](int jj, int g0, int g1) {
                    const int j = jj - 2;
                    walk(j, g0 - 2, g1 - 2, [&](int i, const SiteA<double>& s) {
                        a.mup[(i + 8) * a.mw + j + 8] = s.mup;
                        a.mua[(i + 2) * a.aw + j + 2] = s.mua;
                        if (i >= -1 && i <= ty && j >= -1 && j <= tx)
                        {
                            a.j2y[(i + 1) * a.cw + j + 1] = s.jcy;
                            a.j2x[(i + 1) * a.cw + j + 1] = s.jcx;
                        }
                    });
                });
                const int l6 = min(3, run(12 * tx));  // runs of the six rows above and below
                deal(2 * tx, 6, l6, [&](int jj, int g0, int g1) {
                    const bool below = jj >= tx;
                    const int base = below ? ty + 2 : -8;
                    only_mup(below ? jj - tx : jj, base + g0, base + g1);
                });
                deal(12, ty, run(12 * ty), [&](int jj, int g0, int g1) { only_mup(jj < 6 ? jj - 8 : tx + jj - 4, g0, g1); });
            }
            __syncthreads();

            // ---- stage B: J1_y, J1_x (over their noise), J2 (over J_c)
            {
                Deal<NT> deal;
                const bool noisy = noise_mode != NOISE_OFF;
                deal(tx + 2, ty + 2, run((tx + 2) * (ty + 2)), [&](int j, int g0, int g1) {
                    const double* s = a.mua + g0 * a.aw + j + 1;  // row g0 - 2 of the tile
                    const auto smooth = [&] { return canon_smooth(s[-1], s[0], s[1], k); };
                    const auto diff = [&] { return ksub(s[1], s[-1], k); };
                    double sm = smooth(), dm = diff();
                    s += a.aw;
                    double s0 = g1 - g0 > 1 ? smooth() : 0.0, d0 = diff();
                    for (int i = g0; i < g1; ++i)
                    {
                        s += a.aw;
                        const double sp = smooth(), dp = diff();
                        const int e = i * a.cw + j;
                        a.j2y[e] = canon_j2y(sm, sp, a.j2y[e], k);
                        a.j2x[e] = canon_j2x(dm, d0, dp, a.j2x[e], k);
                        sm = s0; s0 = sp;
                        dm = d0; d0 = dp;
                    }
                });
                deal(tx, ty + 8, 1, [&](int j, int g, int) {
                    const double* c = a.mup + (g + 4) * a.mw + j + 8;
                    const int L = a.mw, e = g * tx + j;
                    a.j1y[e] = rfma(k.mag, noisy ? a.j1y[e] : 0.0, canon_d8(k.ny8, c[-L], c[L], c[-2 * L], c[2 * L], c[-3 * L], c[3 * L],
                                                           c[-4 * L], c[4 * L], k));
                });
                deal(tx + 8, ty, 1, [&](int j, int g, int) {
                    const double* c = a.mup + (g + 8) * a.mw + j + 4;
                    const int e = g * a.xw + j;
                    a.j1x[e] = rfma(k.mag, noisy ? a.j1x[e] : 0.0, canon_d8(k.nx8, c[-1], c[1], c[-2], c[2], c[-3], c[3], c[-4], c[4], k));
                });
            }
            __syncthreads();

            // ---- stage C: the three terms of div J (divTj over mu_a, DY8 over mu_p), then the update
            {
                Deal<NT> deal;
                deal(tx, ty, run(tx * ty), [&](int j, int g0, int g1) {
                    const double *y = a.j2y + g0 * a.cw + j + 1, *x = a.j2x + g0 * a.cw + j + 1;
                    const auto smooth = [&] { return canon_smooth(y[-1], y[0], y[1], k); };
                    const auto diff = [&] { return ksub(x[1], x[-1], k); };
                    double sm = smooth(), dm = diff();
                    y += a.cw;
                    x += a.cw;
                    double s0 = g1 - g0 > 1 ? smooth() : 0.0, d0 = diff();
                    for (int i = g0; i < g1; ++i)
                    {
                        y += a.cw;
                        x += a.cw;
                        const double sp = smooth(), dp = diff();
                        a.mua[i * tx + j] = canon_divtj(sm, sp, dm, d0, dp, k);
                        sm = s0; s0 = sp;
                        dm = d0; d0 = dp;
                    }
                });
                deal(tx, ty, 1, [&](int j, int g, int) {
                    const double* c = a.j1y + (g + 4) * tx + j;
                    a.mup[g * tx + j] = canon_d8(k.py8, c[-tx], c[tx], c[-2 * tx], c[2 * tx], c[-3 * tx], c[3 * tx], c[-4 * tx],
                                                 c[4 * tx], k);
                });
                deal(tx, ty, 1, [&](int j, int g, int) {
                    const double* c = a.j1x + g * a.xw + j + 4;
                    a.dx8[g * tx + j] = canon_d8(k.px8, c[-1], c[1], c[-2], c[2], c[-3], c[3], c[-4], c[4], k);
                });
            }
            __syncthreads();
            for (int e = threadIdx.x; e < tx * ty; e += NT)
            {
                const int i = e / tx, j = e - i * tx, gr = r0 + i, gc = c0 + j;
                if (gr < ny && gc < nx)
                    out[size_t(gr) * nx + gc] = canon_update(a.phi[(i + 9) * a.pw + j + 9], a.dx8[e], a.mua[e], a.mup[e], k);
            }
            __syncthreads();
        }

        // nsteps steps; each CTA owns one tile; step s reads buf[s % 2] and writes buf[(s + 1) % 2]. If the grid
        // barrier gives up, the CTA fills its share of both buffers with NaN (caught by the finite check).
        template <int NT>
        __global__ void __launch_bounds__(NT, kThreads / NT)
        step_dtile_kernel(double* buf0, double* buf1, unsigned* count, const StepParams p0, const phase::Coef coef,
                          const Shape t, int noise_mode, const double* injected, int nsteps)
        {
            extern __shared__ __align__(16) double smem_d[];
            __shared__ int ok;
            __shared__ __align__(16) unsigned char coef_smem[sizeof(phase::Coef)];
            for (int i = threadIdx.x; i < int(sizeof(phase::Coef) / 4); i += NT)
                reinterpret_cast<uint32_t*>(coef_smem)[i] = reinterpret_cast<const uint32_t*>(&coef)[i];
            __syncthreads();
            const phase::Coef& k = *reinterpret_cast<const phase::Coef*>(coef_smem);
            const Arrays a(smem_d, t);
            const int ny = p0.ny, nx = p0.nx, across = (nx + t.tx - 1) / t.tx;
            const int r0 = int(blockIdx.x) / across * t.ty, c0 = int(blockIdx.x) % across * t.tx;
            const size_t plane = size_t(ny) * nx;
            StepParams p = p0;
            const auto noise_of = [&](int s) { return injected ? injected + size_t(s) * 2 * plane : nullptr; };
            size_t first[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) first[q] = halo_site(a, threadIdx.x + q * NT, ny, nx, r0, c0);
            draw<NT>(a, t, p, noise_mode, noise_of(0), r0, c0);
            unsigned target = 0;
            for (int s = 0; s < nsteps; ++s)
            {
                step<NT>(a, t, k, (s & 1) ? buf1 : buf0, (s & 1) ? buf0 : buf1, ny, nx, noise_mode, r0, c0, first);
                if (s + 1 == nsteps) break;
                target += gridDim.x;
                if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
                p.step = p0.step + s + 1;
                draw<NT>(a, t, p, noise_mode, noise_of(s + 1), r0, c0);
                if (threadIdx.x == 0)
                {
                    int done = 0;
                    for (int i = 0; i < phase::kBarrierSpin && !done; ++i)
                    {
                        unsigned v;
                        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                        done = int(v - target) >= 0;
                    }
                    ok = done;
                }
                __syncthreads();
                if (!ok)
                {
                    const double nan = __longlong_as_double(0x7ff8000000000000ll);
                    for (size_t i = blockIdx.x * size_t(NT) + threadIdx.x; i < plane; i += size_t(gridDim.x) * NT)
                        buf0[i] = buf1[i] = nan;
                    return;
                }
            }
        }
    }
}
