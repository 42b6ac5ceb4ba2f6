// Explicit-Euler step in three grid-wide phases, many steps in one cooperative launch.
//
// The FP64 pipe is what binds the FP64 step on sm_103a: one warp instruction per 64 cycles and SM
// sub-partition (2 lanes per clock and SM), issued back to back by a single warp, at the same cost
// for a partial warp. Memory, registers, integer and FP32 work are free beside it, so this form
// spends them to leave no redundant FP64 operation: nothing is recomputed in halos. A site's step
// is 80 operations in the canonical order (amb_canon.cuh), where the fused tile kernel executes 118
// (halo sites, row sums recomputed per site).
//   phase 1  mu_p, mu_a, J_c           from phi (3 x 3)
//   phase 2  J1 = -D8 mu_p + mag xi    (y and x), J2 = -Tj mu_a + J_c
//   phase 3  div J and the update
// The planes between the phases live in a caller's workspace (L2 for small grids) and are read
// through L2 (ld.global.cg: other SMs wrote them in the same launch). A bounded grid barrier
// separates the phases (1.25 us for 152 CTAs).
//
// Work split: one warp marches down a run of rows of a 32-column block, keeping the row sums (and,
// for the y derivatives, a ring of rows) in registers. The rows of all blocks form one list that is
// cut evenly over all warps of the grid, so every sub-partition gets the same share to within one
// row (grids too small for that run as one tile per SM, amb_step_dtile.cuh).
//
// Measured, us per step at T = 0.05 (tile kernel before): 256^2 19.9 (47.8), 350^2 30.0 (48.7), 512^2 52.5 (94.5),
// 701 x 907 102 (222), 2048^2 597 (1177), 4096^2 2415 (4673), the last 6.9 Gsite/s or 88 % of the
// FP64 pipe for the 80 operations. Small grids are bound by the three barriers and the L2 latency
// behind each.
//
// Grids whose planes exceed the workspace are walked in bands of rows; a band recomputes the 8
// (4 for J1) rows of its neighbours on each side.
#pragma once

#include "amb_canon.cuh"
#include "amb_step_tile.cuh"

namespace amb
{
    namespace phase
    {
        constexpr int kPlanes = 8;         // mu_p, mu_a, J_c,y, J_c,x, J1_y, J1_x, J2_y, J2_x
        constexpr int kBandHalo = 8;       // rows of mu_p needed above and below a band
        constexpr size_t kHeader = 256;    // bytes before the planes: the barrier's arrival counter
        // One CTA per SM of 16 warps, all that 128 registers allow: four per sub-partition hide the L2
        // latency of the first loads of a row (4096^2: 2417 us per step; 12 warps 2522, 8 warps 2918).
        constexpr int kThreads = 512;
        constexpr int kBarrierSpin = 1 << 21;  // about 1 s of polling at L2 latency

        // The constants with every addition and product written as a fused multiply-add of three register
        // operands: a + b = fma(a, 1, b) and a b = fma(a, b, -0) round and sign exactly as the plain forms.
        // On sm_103a that instruction takes 64 cycles of a sub-partition's FP64 pipe where an add, a
        // multiply or a fused one with a constant-bank operand takes 76 (measured back to back), so the
        // constants are read from shared memory into registers and `one` and `nzero` come from there too.
        struct Coef : Canon<double>
        {
            double one, nzero;
            __host__ explicit Coef(const StepParams& p) : Canon<double>(p), one(1.0), nzero(-0.0) {}
        };
        __device__ __forceinline__ double kadd(double a, double b, const Coef& k) { return __fma_rn(a, k.one, b); }
        __device__ __forceinline__ double ksub(double a, double b, const Coef& k) { return __fma_rn(-b, k.one, a); }
        __device__ __forceinline__ double kmul(double a, double b, const Coef& k) { return __fma_rn(a, b, k.nzero); }

        // The planes of one workspace, all of `rows` rows. whole: they hold the full periodic grid;
        // otherwise plane row i is grid row base + i (not wrapped).
        template <typename Real>
        struct Planes
        {
            Real *mup, *mua, *jcy, *jcx, *j1y, *j1x, *j2y, *j2x;
            __host__ __device__ Planes(void* ws, size_t sites)
            {
                Real* p = reinterpret_cast<Real*>(static_cast<char*>(ws) + kHeader);
                mup = p;
                mua = p + sites;
                jcy = p + 2 * sites;
                jcx = p + 3 * sites;
                j1y = p + 4 * sites;
                j1x = p + 5 * sites;
                j2y = p + 6 * sites;
                j2x = p + 7 * sites;
            }
        };

        struct Band
        {
            int base;
            bool whole;
            int ny, nx;
            __device__ __forceinline__ size_t row(int r) const  // offset of grid row r in a plane
            {
                return size_t(whole ? wrap_index(r, ny) : r - base) * nx;
            }
        };

        // Grid-wide barrier of a cooperative launch (every CTA resident): release-add one arrival, poll
        // with acquire loads. Bounded: false if the arrivals did not come. The comparison is modular,
        // so the count may wrap.
        __device__ __forceinline__ bool barrier(unsigned* count, unsigned target, int* ok)
        {
            __syncthreads();
            if (threadIdx.x == 0)
            {
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
                int done = 0;
                for (int i = 0; i < kBarrierSpin && !done; ++i)
                {
                    unsigned v;
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                    done = int(v - target) >= 0;
                }
                *ok = done;
            }
            __syncthreads();
            return *ok != 0;
        }

        // FP32 normal widened to FP64 by bit arithmetic: the conversion instruction would take a slot
        // of the FP64 pipe. Exact for every normal number and zero (subnormals take the instruction).
        __device__ __forceinline__ double widen(float z)
        {
            const uint32_t b = __float_as_uint(z), m = b & 0x7fffffffu;
            if (m != 0 && m < 0x00800000u) return double(z);
            const uint32_t hi = (b & 0x80000000u) | (m == 0 ? 0u : (m >> 3) + 0x38000000u);
            return __hiloint2double(int(hi), int(b << 29));
        }

        // The run of this warp in a list of `groups` columns of `rows` rows each, cut evenly over all
        // warps; f(group, first, last) is called with row ranges [first, last) inside one group.
        template <typename F>
        __device__ __forceinline__ void for_runs(int groups, int rows, F&& f)
        {
            const unsigned warps = gridDim.x * (blockDim.x >> 5);
            const unsigned w = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // neighbours on other SMs
            const unsigned long long total = (unsigned long long)groups * rows;
            unsigned long long lo, hi;
            if (total <= warps)
            {
                lo = w;
                hi = w < total ? w + 1 : w;
            }
            else
            {
                lo = total * w / warps;
                hi = total * (w + 1) / warps;
            }
            while (lo < hi)
            {
                const int g = int(lo / rows), a = int(lo - (unsigned long long)g * rows);
                const int b = hi - lo < (unsigned long long)(rows - a) ? a + int(hi - lo) : rows;
                f(g, a, b);
                lo += b - a;
            }
        }

        // ---- phase 1: rows [r0, r0 + n) of mu_p, mu_a, J_c
        template <typename Real>
        __device__ __forceinline__ void local_terms(const Real* in, const Planes<Real>& w, const Band& bd,
                                                    const Coef& k, int r0, int n)
        {
            const int lane = threadIdx.x & 31, nx = bd.nx, ny = bd.ny;
            for_runs((nx + 31) >> 5, n, [&](int blk, int a, int b) {
                const int c = blk * 32 + lane;
                const bool act = c < nx;
                const int c0 = act ? c : nx - 1, cl = wrap_index(c0 - 1, nx), cr = wrap_index(c0 + 1, nx);
                Real l, m, r;
                const auto load = [&](int row) {
                    const Real* p = in + size_t(wrap_index(row, ny)) * nx;
                    l = __ldcg(p + cl);
                    m = __ldcg(p + c0);
                    r = __ldcg(p + cr);
                };
                load(r0 + a - 1);
                Real Am = kadd(l, r, k), Dm = ksub(r, l, k), um = m;
                load(r0 + a);
                Real A0 = kadd(l, r, k), D0 = ksub(r, l, k), f = m;
                load(r0 + a + 1);
                for (int i = a; i < b; ++i)
                {
                    const Real Ap = kadd(l, r, k), Dp = ksub(r, l, k), dn = m;
                    if (i + 1 < b) load(r0 + i + 2);
                    const SiteA<Real> s = canon_site_a(um, f, dn, Am, A0, Ap, Dm, D0, Dp, k);
                    if (act)
                    {
                        const size_t e = bd.row(r0 + i) + c;
                        w.mup[e] = s.mup;
                        w.mua[e] = s.mua;
                        w.jcy[e] = s.jcy;
                        w.jcx[e] = s.jcx;
                    }
                    um = f;
                    f = dn;
                    Am = A0;
                    A0 = Ap;
                    Dm = D0;
                    D0 = Dp;
                }
            });
        }

        // ---- phase 2: rows [r0, r0 + n) of J1_y, J1_x and J2 (three independent work items per
        // column block, so that small grids spread over three times as many warps)
        template <typename Real>
        __device__ __forceinline__ void fluxes(const Planes<Real>& w, const Band& bd, const Coef& k,
                                               const StepParams& p, int noise_mode, const Real* injected, int r0, int n)
        {
            const int lane = threadIdx.x & 31, nx = bd.nx, ny = bd.ny;
            const int nblk = (nx + 31) >> 5;
            const size_t plane = size_t(ny) * nx;
            const auto xi = [&](int row, int c, int comp) -> Real {
                if (noise_mode == NOISE_OFF) return Real(0);
                const int gr = wrap_index(row, ny);
                if (noise_mode == NOISE_INJECTED) return injected[comp * plane + size_t(gr) * nx + c];
                return widen(noise_normal(p.seed, p.step, gr, c, comp));
            };
            for_runs(3 * nblk, n, [&](int g, int a, int b) {
                const int role = g / nblk, c = (g - role * nblk) * 32 + lane;
                const bool act = c < nx;
                const int c0 = act ? c : nx - 1;
                if (role == 0)
                {
                    const auto at = [&](int row) { return __ldcg(w.mup + bd.row(row) + c0); };
                    Real m[9];  // rows i - 4 .. i + 4
#pragma unroll
                    for (int j = 0; j < 9; ++j) m[j] = at(r0 + a - 4 + j);
                    for (int i = a; i < b; ++i)
                    {
                        const Real nxt = i + 1 < b ? at(r0 + i + 5) : m[8];
                        const Real v = rfma(k.mag, xi(r0 + i, c0, 0),
                                            canon_d8(k.ny8, m[3], m[5], m[2], m[6], m[1], m[7], m[0], m[8], k));
                        if (act) w.j1y[bd.row(r0 + i) + c] = v;
#pragma unroll
                        for (int j = 0; j < 8; ++j) m[j] = m[j + 1];
                        m[8] = nxt;
                    }
                }
                else if (role == 1)
                {
                    int cm[4], cp[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        cm[j] = wrap_index(c0 - 1 - j, nx);
                        cp[j] = wrap_index(c0 + 1 + j, nx);
                    }
                    for (int i = a; i < b; ++i)
                    {
                        const size_t e = bd.row(r0 + i);
                        const Real* q = w.mup + e;
                        Real m[4], pl[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                        {
                            m[j] = __ldcg(q + cm[j]);
                            pl[j] = __ldcg(q + cp[j]);
                        }
                        const Real v = rfma(k.mag, xi(r0 + i, c0, 1),
                                            canon_d8(k.nx8, m[0], pl[0], m[1], pl[1], m[2], pl[2], m[3], pl[3], k));
                        if (act) w.j1x[e + c] = v;
                    }
                }
                else
                {
                    const int cl = wrap_index(c0 - 1, nx), cr = wrap_index(c0 + 1, nx);
                    Real l, m, r;
                    const auto load = [&](int row) {
                        const Real* q = w.mua + bd.row(row);
                        l = __ldcg(q + cl);
                        m = __ldcg(q + c0);
                        r = __ldcg(q + cr);
                    };
                    load(r0 + a - 1);
                    Real sm = canon_smooth(l, m, r, k), dm = ksub(r, l, k);
                    load(r0 + a);
                    Real s0 = canon_smooth(l, m, r, k), d0 = ksub(r, l, k);
                    load(r0 + a + 1);
                    for (int i = a; i < b; ++i)
                    {
                        const size_t e = bd.row(r0 + i);
                        const Real cy = __ldcg(w.jcy + e + c0), cx = __ldcg(w.jcx + e + c0);
                        const Real sp = canon_smooth(l, m, r, k), dp = ksub(r, l, k);
                        if (i + 1 < b) load(r0 + i + 2);
                        const Real y = canon_j2y(sm, sp, cy, k), x = canon_j2x(dm, d0, dp, cx, k);
                        if (act)
                        {
                            w.j2y[e + c] = y;
                            w.j2x[e + c] = x;
                        }
                        sm = s0;
                        s0 = sp;
                        dm = d0;
                        d0 = dp;
                    }
                }
            });
        }

        // ---- phase 3: rows [r0, r0 + n): div J and the update
        template <typename Real>
        __device__ __forceinline__ void update(const Real* in, Real* out, const Planes<Real>& w, const Band& bd,
                                               const Coef& k, int r0, int n)
        {
            const int lane = threadIdx.x & 31, nx = bd.nx;
            for_runs((nx + 31) >> 5, n, [&](int blk, int a, int b) {
                const int c = blk * 32 + lane;
                const bool act = c < nx;
                const int c0 = act ? c : nx - 1;
                int cm[4], cp[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    cm[j] = wrap_index(c0 - 1 - j, nx);
                    cp[j] = wrap_index(c0 + 1 + j, nx);
                }
                Real jy[9];  // J1_y rows i - 4 .. i + 4
#pragma unroll
                for (int j = 0; j < 9; ++j) jy[j] = __ldcg(w.j1y + bd.row(r0 + a - 4 + j) + c0);
                Real yl, ym, yr, xl, xr;
                const auto load = [&](int row) {
                    const size_t e = bd.row(row);
                    yl = __ldcg(w.j2y + e + cm[0]);
                    ym = __ldcg(w.j2y + e + c0);
                    yr = __ldcg(w.j2y + e + cp[0]);
                    xl = __ldcg(w.j2x + e + cm[0]);
                    xr = __ldcg(w.j2x + e + cp[0]);
                };
                load(r0 + a - 1);
                Real sm = canon_smooth(yl, ym, yr, k), dm = ksub(xr, xl, k);
                load(r0 + a);
                Real s0 = canon_smooth(yl, ym, yr, k), d0 = ksub(xr, xl, k);
                load(r0 + a + 1);
                for (int i = a; i < b; ++i)
                {
                    const size_t e = bd.row(r0 + i), gi = size_t(r0 + i) * nx;
                    const Real* q = w.j1x + e;
                    Real m[4], pl[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        m[j] = __ldcg(q + cm[j]);
                        pl[j] = __ldcg(q + cp[j]);
                    }
                    const Real f = __ldcg(in + gi + c0);
                    const Real nxt = i + 1 < b ? __ldcg(w.j1y + bd.row(r0 + i + 5) + c0) : jy[8];
                    const Real sp = canon_smooth(yl, ym, yr, k), dp = ksub(xr, xl, k);
                    if (i + 1 < b) load(r0 + i + 2);
                    const Real divtj = canon_divtj(sm, sp, dm, d0, dp, k);
                    const Real dy8 = canon_d8(k.py8, jy[3], jy[5], jy[2], jy[6], jy[1], jy[7], jy[0], jy[8], k);
                    const Real dx8 = canon_d8(k.px8, m[0], pl[0], m[1], pl[1], m[2], pl[2], m[3], pl[3], k);
                    if (act) out[gi + c] = canon_update(f, dx8, divtj, dy8, k);
#pragma unroll
                    for (int j = 0; j < 8; ++j) jy[j] = jy[j + 1];
                    jy[8] = nxt;
                    sm = s0;
                    s0 = sp;
                    dm = d0;
                    d0 = dp;
                }
            });
        }

        // nsteps steps; step s reads buf[s % 2] and writes buf[(s + 1) % 2]. band: output rows per band
        // (ny: the planes hold the whole grid). If a barrier gives up, the CTA fills its share of both
        // buffers with NaN (caught by the finite check) and leaves.
        template <typename Real>
        __global__ void __launch_bounds__(kThreads, 1)
        step_phase_kernel(Real* buf0, Real* buf1, void* ws, const StepParams p0, const Coef coef, int noise_mode,
                          const Real* injected, int nsteps, int band)
        {
            __shared__ int ok;
            __shared__ __align__(16) unsigned char coef_smem[sizeof(Coef)];
            for (int i = threadIdx.x; i < int(sizeof(Coef) / 4); i += blockDim.x)
                reinterpret_cast<uint32_t*>(coef_smem)[i] = reinterpret_cast<const uint32_t*>(&coef)[i];
            __syncthreads();
            const Coef& k = *reinterpret_cast<const Coef*>(coef_smem);
            const int ny = p0.ny, nx = p0.nx;
            const bool whole = band >= ny;
            const size_t sites = size_t(nx) * (whole ? ny : band + 2 * kBandHalo);
            const Planes<Real> w(ws, sites);
            unsigned* count = static_cast<unsigned*>(ws);
            unsigned target = 0;
            StepParams p = p0;
            const int h1 = whole ? 0 : kBandHalo, h2 = whole ? 0 : kBandHalo / 2;
            bool good = true;
            for (int s = 0; s < nsteps && good; ++s)
            {
                const Real* in = (s & 1) ? buf1 : buf0;
                Real* out = (s & 1) ? buf0 : buf1;
                p.step = p0.step + s;
                const Real* inj = injected ? injected + size_t(s) * 2 * ny * nx : nullptr;
                for (int r0 = 0; r0 < ny && good; r0 += band)
                {
                    const int n = min(band, ny - r0);
                    const Band bd{r0 - h1, whole, ny, nx};
                    local_terms(in, w, bd, k, r0 - h1, n + 2 * h1);
                    good = barrier(count, target += gridDim.x, &ok);
                    if (!good) break;
                    fluxes(w, bd, k, p, noise_mode, inj, r0 - h2, n + 2 * h2);
                    good = barrier(count, target += gridDim.x, &ok);
                    if (!good) break;
                    // the next band's phase 1 writes planes that this phase does not read
                    update(in, out, w, bd, k, r0, n);
                }
                if (good && s + 1 < nsteps) good = barrier(count, target += gridDim.x, &ok);
            }
            if (!good)
            {
                const Real nan = Real(__int_as_float(0x7fc00000));
                const size_t total = size_t(ny) * nx;
                for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x)
                    buf0[i] = buf1[i] = nan;
            }
        }
    }
}
