// FP32 step, shared-memory tile form on packed column quads.
//
// One CTA produces a TY x TX tile of phi(t + dt) from a (TY + 18) x (TX + 24) tile of phi(t). The
// stages run out of shared memory with one thread per quad of columns (and, in stage A, a run of
// rows whose row sums are carried), the arithmetic packed in pairs: the same operations in the same
// order as every FP32 kernel (amb_canon.cuh), so the same bits. Any grid size: a quad that does not
// lie inside one row of the grid, and every quad of a grid whose rows are not whole quads, is read,
// drawn and written by column.
//
// Small grids are bound by latency: a grid barrier (1.25 us), the L2 latency of the halo and three
// block barriers, between stages of a few hundred issue slots. One tile per SM whose height makes the
// tile count match the SMs is therefore best where it fits (256^2: 7 or 14 rows, 3.4 us per step;
// two or three tiles per SM 4.8 and 6.6), several CTAs of 256 threads otherwise. us per step, f32c,
// T = 0.05, autotuned, this kernel and the one-column-per-thread tile kernel before it: 256^2 3.5 (6.3; 3.4 on
// all SMs' threads), 512^2 5.8 (8.7), 768^2 9.1 (15.4), 1024^2 16.3 (24.6), 250 x 333 4.5 (6.7); from 1536^2 on the
// sliding kernel, with less halo work, is the faster (28.7 there).
//
// The noise of a step depends on no field, so it is drawn into the arrays that J1 later replaces:
// before the tile's halo has arrived, and in the persistent form while the grid barrier completes.
#pragma once

#include "amb_quad.cuh"
#include "amb_step_tile.cuh"

namespace amb
{
    namespace quadtile
    {
        // Widths (columns) of the shared arrays and their first column relative to the tile; rows from
        // -9 (phi), -8 (mu_p), -2 (mu_a), -1 (J2), -4 (J1_y), 0 (J1_x).
        template <int TX>
        struct Geom
        {
            static constexpr int PW = TX + 24, P0 = 12;  // phi
            static constexpr int MW = TX + 16, M0 = 8;   // mu_p
            static constexpr int AW = TX + 8, A0 = 4;    // mu_a, J2, J1_x
            __host__ __device__ static constexpr int floats(int ty)
            {
                return (ty + 18) * PW + (ty + 16) * MW + (ty + 4) * AW + 2 * (ty + 2) * AW + (ty + 8) * TX + ty * AW;
            }
        };

        template <int TX>
        struct Arrays
        {
            using G = Geom<TX>;
            float *phi, *mup, *mua, *j2y, *j2x, *j1y, *j1x;
            __device__ __forceinline__ Arrays(float* s, int ty)
            {
                phi = s;
                mup = phi + (ty + 18) * G::PW;
                mua = mup + (ty + 16) * G::MW;
                j2y = mua + (ty + 4) * G::AW;
                j2x = j2y + (ty + 2) * G::AW;
                j1y = j2x + (ty + 2) * G::AW;
                j1x = j1y + (ty + 8) * TX;
            }
        };

        // One launch's constants: the grid, the constants of the arithmetic, the noise.
        struct Launch
        {
            int ny, nx, ty, noise_mode;
            bool vec;  // rows are whole 16-byte quads
            QuadCoef k;
        };

        // xi of the tile's J1_y and J1_x quads into their arrays.
        template <int TX, int NT>
        __device__ __forceinline__ void draw(const Arrays<TX>& a, const Launch& p, int64_t step, const float* injected,
                                             int r0, int c0)
        {
            using G = Geom<TX>;
            constexpr int QY = TX / 4, QX = G::AW / 4;
            if (p.noise_mode == NOISE_OFF) return;
            const int ny = p.ny, nx = p.nx, n1 = QY * (p.ty + 8), n = n1 + QX * p.ty;
            for (int t = threadIdx.x; t < n; t += NT)
            {
                const int comp = t >= n1, e = comp ? t - n1 : t;
                const int i = comp ? e / QX : e / QY, j = comp ? e - i * QX : e - i * QY;
                const int row = wrap_index(comp ? r0 + i : r0 + i - 4, ny);
                const int u = c0 + 4 * j - (comp ? G::A0 : 0), g = wrap_index(u, nx);
                if (u >= nx + (comp ? 4 : 0)) continue;  // no site of the grid reads it
                float* out = comp ? a.j1x + i * G::AW + 4 * j : a.j1y + i * TX + 4 * j;
                if (p.noise_mode == NOISE_INJECTED)
                {
                    for (int q = 0; q < 4; ++q)
                        out[q] = injected[comp * size_t(ny) * nx + size_t(row) * nx + wrap_index(u + q, nx)];
                    continue;
                }
                const auto quad_at = [&](int col) {  // the normals of the noise quad that holds column col
                    const U4 ctr{uint32_t(col) >> 2, uint32_t(row), uint32_t(uint64_t(step)),
                                 (uint32_t(uint64_t(step) >> 32) << 1) | uint32_t(comp)};
                    const U4 q = philox4x32_10_rk(ctr, p.k.m.rk0, p.k.m.rk1);
                    float2 zc, zs;
                    box_muller_f32x2(make_uint2(q.x, q.z), make_uint2(q.y, q.w), zc, zs);
                    return make_float4(zc.x, zs.x, zc.y, zs.y);
                };
                float4 z = quad_at(g);
                if ((g & 3) == 0 && g + 4 <= nx) *reinterpret_cast<float4*>(out) = z;
                else  // across the end of a row: the columns of two or three noise quads
                    for (int q = 0, held = g >> 2; q < 4; ++q)
                    {
                        const int col = wrap_index(u + q, nx);
                        if (col >> 2 != held)
                        {
                            z = quad_at(col);
                            held = col >> 2;
                        }
                        out[q] = (col & 2) ? ((col & 1) ? z.w : z.z) : ((col & 1) ? z.y : z.x);
                    }
            }
        }

        __device__ __forceinline__ void cp_async16(float* dst, const float* src)
        {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src)
                         : "memory");
        }

        // phi(t) with its halo, through L2 only (other CTAs of a persistent launch wrote it): asynchronous
        // 16-byte copies, or loads by column. Complete after wait_field().
        template <int TX, int NT>
        __device__ __forceinline__ void load_field(const Arrays<TX>& a, const Launch& p, const float* in, int r0, int c0)
        {
            using G = Geom<TX>;
            const int ny = p.ny, nx = p.nx, rows = p.ty + 18;
            if (p.vec)
            {
                constexpr int W = G::PW / 4;
                for (int t = threadIdx.x; t < rows * W; t += NT)
                {
                    const int i = t / W, j = t - i * W;
                    const int gr = wrap_index(r0 + i - 9, ny), gc = wrap_index(c0 + 4 * j - G::P0, nx);
                    cp_async16(a.phi + i * G::PW + 4 * j, in + size_t(gr) * nx + gc);
                }
            }
            else
            {
                // A thread walks down a run of rows of one column, so that a site costs a load, a store and a step of
                // the row (index arithmetic per site instead: 250 x 333 5.06 us per step, 4.57 so; 683 x 1801 29.6 and
                // 27.2). Aligned quads shifted between lanes were slower (6.1), as were other batches than 8 rows.
                constexpr int W = G::PW, NG = NT / W, B = 8;
                const int run = (rows + NG - 1) / NG, j = threadIdx.x % W, g = threadIdx.x / W;
                const int hi = g < NG ? min(rows, (g + 1) * run) : 0;
                int gr = wrap_index(r0 + g * run - 9, ny);
                const float* col = in + wrap_index(c0 + j - G::P0, nx);
                for (int i = g * run; i < hi; i += B)
                {
                    float v[B];  // all loads of a batch before its stores
#pragma unroll
                    for (int q = 0; q < B; ++q)
                    {
                        if (i + q < hi) v[q] = __ldcg(col + size_t(gr) * nx);
                        gr = gr + 1 == ny ? 0 : gr + 1;
                    }
#pragma unroll
                    for (int q = 0; q < B; ++q)
                        if (i + q < hi) a.phi[(i + q) * W + j] = v[q];
                }
            }
        }
        __device__ __forceinline__ void wait_field()
        {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }

        // One step of the tile whose phi and noise are in shared memory.
        template <int TX, int COMP, int NT>
        __device__ __forceinline__ void step(const Arrays<TX>& a, const Launch& p, float* out, __nv_bfloat16* comp, int r0,
                                             int c0)
        {
            using G = Geom<TX>;
            const QuadCoef& k = p.k;
            const int ty = p.ty, tid = threadIdx.x;

            // ---- stage A: mu_p on the plus-shaped region, mu_a and J_c on its middle; each thread walks
            // down a run of rows of one quad column
            {
                constexpr int W = G::MW / 4, NG = NT / W;
                const int run = (ty + 16 + NG - 1) / NG, j = tid % W, g = tid / W, q = j - 2;
                const bool mid = q >= 0 && q < TX / 4, near = q >= -1 && q <= TX / 4;
                const int lo = max(g * run - 8, mid ? -8 : near ? -2 : 0);
                const int hi = min(g * run - 8 + run, mid ? ty + 8 : near ? ty + 2 : ty);
                if (g < NG && lo < hi)
                {
                    const float* s = a.phi + (lo + 8) * G::PW + 4 * q + G::P0;  // row lo - 1
                    Quad um = load_quad(s);
                    Quad Am = nsum(s[-1], um, s[4]), Dm = ndiff(s[-1], um, s[4]);
                    s += G::PW;
                    Quad f = load_quad(s);
                    Quad A0 = nsum(s[-1], f, s[4]), D0 = ndiff(s[-1], f, s[4]);
                    float* m = a.mup + (lo + 8) * G::MW + 4 * q + G::M0;
                    int e = (lo + 2) * G::AW + 4 * q + G::A0;
                    for (int i = lo; i < hi; ++i)
                    {
                        s += G::PW;
                        const Quad dn = load_quad(s);
                        const Quad Ap = nsum(s[-1], dn, s[4]), Dp = ndiff(s[-1], dn, s[4]);
                        Quad l = k.s.lA * (Am + Ap);
                        l = fma4(k.s.lB, um + dn, l);
                        l = fma4(k.s.lC, A0, l);
                        const Quad lap = fma4(k.s.lD, f, l);
                        store_quad(m, fma4(k.m.nkappa, lap, fma4(fma4(k.m.c, f, k.m.b), f, k.m.a) * f));
                        if (near && i >= -2 && i < ty + 2)
                        {
                            const Quad gx = fma4(k.s.gxb, D0, k.s.gxa * (Dm + Dp));
                            const Quad gy = fma4(k.s.gyb, dn - um, k.s.gya * (Ap - Am));
                            store_quad(a.mua + e, k.m.lambda * fma4(gy, gy, gx * gx));
                            if (i >= -1 && i < ty + 1)
                            {
                                const Quad zl = k.m.zeta * lap;
                                store_quad(a.j2y + e - G::AW, zl * gy);
                                store_quad(a.j2x + e - G::AW, zl * gx);
                            }
                        }
                        um = f; f = dn;
                        Am = A0; A0 = Ap;
                        Dm = D0; D0 = Dp;
                        m += G::MW;
                        e += G::AW;
                    }
                }
            }
            __syncthreads();

            // ---- stage B: J1_y, J1_x (over their noise) and J2 (over J_c)
            {
                constexpr int QY = TX / 4, QX = G::AW / 4;
                const int n1 = QY * (ty + 8), n2 = n1 + QX * ty, n3 = n2 + QX * (ty + 2);
                const bool noisy = p.noise_mode != NOISE_OFF;
                for (int t = tid; t < n3; t += NT)
                {
                    if (t < n1)
                    {
                        const int i = t / QY, j = t - i * QY;  // row i - 4
                        const float* c = a.mup + (i + 4) * G::MW + 4 * j + G::M0;
                        constexpr int L = G::MW;
                        Quad s = k.s.ny8[0] * (load_quad(c + L) - load_quad(c - L));
                        s = fma4(k.s.ny8[1], load_quad(c + 2 * L) - load_quad(c - 2 * L), s);
                        s = fma4(k.s.ny8[2], load_quad(c + 3 * L) - load_quad(c - 3 * L), s);
                        s = fma4(k.s.ny8[3], load_quad(c + 4 * L) - load_quad(c - 4 * L), s);
                        float* e = a.j1y + i * TX + 4 * j;
                        store_quad(e, fma4(k.m.mag, noisy ? load_quad(e) : zero_quad(), s));
                    }
                    else if (t < n2)
                    {
                        const int i = (t - n1) / QX, j = t - n1 - i * QX;
                        const float* c = a.mup + (i + 8) * G::MW + 4 * j - G::A0 + G::M0;
                        const Quad s = d8x(k.s.nx8, load_quad(c - 4), load_quad(c), load_quad(c + 4));
                        float* e = a.j1x + i * G::AW + 4 * j;
                        store_quad(e, fma4(k.m.mag, noisy ? load_quad(e) : zero_quad(), s));
                    }
                    else
                    {
                        const int i = (t - n2) / QX, j = t - n2 - i * QX;  // row i - 1
                        // the outermost quads matter in their inner columns only; their outer neighbour is not read
                        const int l = j == 0 ? 0 : -1, r = j == QX - 1 ? 3 : 4;
                        const float* u = a.mua + i * G::AW + 4 * j;
                        const float *m = u + G::AW, *d = m + G::AW;
                        const Quad uq = load_quad(u), mq = load_quad(m), dq = load_quad(d);
                        const Quad su = fma4(k.s.p1, nsum(u[l], uq, u[r]), k.s.p3 * uq);
                        const Quad sd = fma4(k.s.p1, nsum(d[l], dq, d[r]), k.s.p3 * dq);
                        const Quad du = ndiff(u[l], uq, u[r]), dm = ndiff(m[l], mq, m[r]), dd = ndiff(d[l], dq, d[r]);
                        const int e = i * G::AW + 4 * j;
                        store_quad(a.j2y + e, fma4(k.s.ndy, sd - su, load_quad(a.j2y + e)));
                        store_quad(a.j2x + e, fma4(k.s.jx3, dm, fma4(k.s.jx1, dd + du, load_quad(a.j2x + e))));
                    }
                }
            }
            __syncthreads();

            // ---- stage C: div J and the update
            constexpr int Q = TX / 4;
            for (int t = tid; t < Q * ty; t += NT)
            {
                const int i = t / Q, j = t - i * Q;
                const int gr = r0 + i, gc = c0 + 4 * j;
                if (gr >= p.ny || gc >= p.nx) continue;
                const float* y0 = a.j2y + i * G::AW + 4 * j + G::A0;  // row i - 1
                const float* y2 = y0 + 2 * G::AW;
                const float* x0 = a.j2x + i * G::AW + 4 * j + G::A0;
                const float *x1 = x0 + G::AW, *x2 = x1 + G::AW;
                const Quad yu = load_quad(y0), yd = load_quad(y2);
                const Quad su = fma4(k.s.p1, nsum(y0[-1], yu, y0[4]), k.s.p3 * yu);
                const Quad sd = fma4(k.s.p1, nsum(y2[-1], yd, y2[4]), k.s.p3 * yd);
                const Quad du = ndiff(x0[-1], load_quad(x0), x0[4]), dm = ndiff(x1[-1], load_quad(x1), x1[4]),
                           dd = ndiff(x2[-1], load_quad(x2), x2[4]);
                Quad tj = k.s.tx1 * (du + dd);
                tj = fma4(k.s.tx3, dm, tj);
                tj = fma4(k.s.dyInv, sd - su, tj);
                const float* cy = a.j1y + (i + 4) * TX + 4 * j;
                Quad s = k.s.py8[0] * (load_quad(cy + TX) - load_quad(cy - TX));
                s = fma4(k.s.py8[1], load_quad(cy + 2 * TX) - load_quad(cy - 2 * TX), s);
                s = fma4(k.s.py8[2], load_quad(cy + 3 * TX) - load_quad(cy - 3 * TX), s);
                s = fma4(k.s.py8[3], load_quad(cy + 4 * TX) - load_quad(cy - 4 * TX), s);
                const float* cx = a.j1x + i * G::AW + 4 * j + G::A0;
                const Quad div = d8x(k.s.px8, load_quad(cx - 4), load_quad(cx), load_quad(cx + 4)) + (tj + s);
                const Quad f = load_quad(a.phi + (i + 9) * G::PW + 4 * j + G::P0);
                const size_t gi = size_t(gr) * p.nx + gc;
                if constexpr (COMP == COMP_BF16)
                {
                    Quad rr;
                    if (p.vec)
                    {
                        const uint2 v = *reinterpret_cast<const uint2*>(comp + gi);
                        rr = {make_float2(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u)),
                              make_float2(__uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u))};
                    }
                    else
                    {
                        float v[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = gc + q < p.nx ? __bfloat162float(comp[gi + q]) : 0.f;
                        rr = {make_float2(v[0], v[1]), make_float2(v[2], v[3])};
                    }
                    const Quad F = fma4(k.s.dt, div, rr);
                    const Quad nf = f - F;
                    const Quad nr = (nf - f) + F;
                    if (p.vec)
                    {
                        store_quad(out + gi, nf);
                        __nv_bfloat162 lo = __floats2bfloat162_rn(nr.a.x, nr.a.y), hi = __floats2bfloat162_rn(nr.b.x, nr.b.y);
                        uint2 w;
                        w.x = *reinterpret_cast<uint32_t*>(&lo);
                        w.y = *reinterpret_cast<uint32_t*>(&hi);
                        *reinterpret_cast<uint2*>(comp + gi) = w;
                    }
                    else
                    {
                        const float4 v = vec(nf), w = vec(nr);
                        const float nv[4] = {v.x, v.y, v.z, v.w}, nw[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (gc + q < p.nx)
                            {
                                out[gi + q] = nv[q];
                                comp[gi + q] = __float2bfloat16_rn(nw[q]);
                            }
                    }
                }
                else
                {
                    const Quad nf = fma4(k.s.ndt, div, f);
                    if (p.vec) store_quad(out + gi, nf);
                    else
                    {
                        const float4 v = vec(nf);
                        const float nv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (gc + q < p.nx) out[gi + q] = nv[q];
                    }
                }
            }
        }

        // One step, one tile per CTA.
        template <int TX, int COMP, int NT>
        __global__ void __launch_bounds__(NT, 512 / NT)
        step_quad_kernel(const float* in, float* out, __nv_bfloat16* comp, const Launch p, int64_t step_index,
                         const float* injected)
        {
            extern __shared__ __align__(16) float smem_f[];
            const Arrays<TX> a(smem_f, p.ty);
            const int tx = (p.nx + TX - 1) / TX, r0 = int(blockIdx.x) / tx * p.ty, c0 = int(blockIdx.x) % tx * TX;
            load_field<TX, NT>(a, p, in, r0, c0);
            draw<TX, NT>(a, p, step_index, injected, r0, c0);
            wait_field();
            step<TX, COMP, NT>(a, p, out, comp, r0, c0);
        }

        // nsteps steps in one cooperative launch: each CTA owns tiles blockIdx.x, + gridDim.x, ...; step s
        // reads buf[s % 2] and writes buf[(s + 1) % 2]. A bounded grid barrier separates the steps, and
        // the next step's noise of the CTA's first tile is drawn between arriving and waiting. If the
        // barrier gives up, the CTA fills its share of both buffers with NaN (caught by the finite check).
        template <int TX, int COMP, int NT>
        __global__ void __launch_bounds__(NT, 512 / NT)
        step_quad_persistent_kernel(float* buf0, float* buf1, __nv_bfloat16* comp, const Launch p, int64_t step0,
                                    const float* injected, int nsteps, unsigned* count)
        {
            extern __shared__ __align__(16) float smem_f[];
            __shared__ int ok;
            const Arrays<TX> a(smem_f, p.ty);
            const int tx = (p.nx + TX - 1) / TX, ntiles = tx * ((p.ny + p.ty - 1) / p.ty);
            const size_t plane = size_t(p.ny) * p.nx;
            const auto noise_of = [&](int s) { return injected ? injected + size_t(s) * 2 * plane : nullptr; };
            const int first = blockIdx.x;
            draw<TX, NT>(a, p, step0, noise_of(0), first / tx * p.ty, first % tx * TX);
            unsigned target = 0;
            for (int s = 0; s < nsteps; ++s)
            {
                const float* in = (s & 1) ? buf1 : buf0;
                float* out = (s & 1) ? buf0 : buf1;
                for (int tile = first; tile < ntiles; tile += gridDim.x)
                {
                    const int r0 = tile / tx * p.ty, c0 = tile % tx * TX;
                    load_field<TX, NT>(a, p, in, r0, c0);
                    if (tile != first) draw<TX, NT>(a, p, step0 + s, noise_of(s), r0, c0);
                    wait_field();
                    step<TX, COMP, NT>(a, p, out, comp, r0, c0);
                    __syncthreads();
                }
                if (s + 1 == nsteps) break;
                target += gridDim.x;
                if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
                draw<TX, NT>(a, p, step0 + s + 1, noise_of(s + 1), first / tx * p.ty, first % tx * TX);
                if (threadIdx.x == 0)
                {
                    int done = 0;
                    for (int i = 0; i < (1 << 21) && !done; ++i)
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
                    const float nan = __int_as_float(0x7fc00000);
                    for (size_t i = blockIdx.x * size_t(NT) + threadIdx.x; i < plane; i += size_t(gridDim.x) * NT)
                        buf0[i] = buf1[i] = nan;
                    return;
                }
            }
        }
    }
}
