// Learned coarse stepper kernels (no reference counterpart): 5x5 circular
// convolutions as BF16 implicit GEMMs on the tcgen05 tensor cores with FP32
// accumulation in TMEM, for both inference and training, plus the
// mass-conserving fixed-point update that applies the predicted flux.
//
// Activation layout ("chunk planes"): bf16 [batch][C/8][nrows][ncols][8], i.e.
// for each group of 8 channels a plane of 16-byte sites. One 16-byte site row
// is one row of a tensor-core core matrix, so a tap shift of one site along x
// is a 16-byte move of the operand start address.
//
// Forward / data-gradient kernel (conv_fwd_kernel): one CTA owns a 128-site
// window of up to 16 output rows and stages all of its input rows (the rows plus
// a 2-row halo above and below, periodic wrap in both axes) in shared memory, one
// bulk copy per (row, channel chunk) for the in-range sites and, in the first and
// last windows, plain copies of the 2 periodically wrapped sites on each side by
// the epilogue warps; one mbarrier per row. Each staged input row, shifted by one of the
// five x taps, is the A operand (M = 128 sites, K-major, LBO = one channel-chunk
// plane, SBO = 8 sites) of ONE MMA per 16 input channels whose B operand stacks
// the five y taps along N (N = 5 x Cout): its five N slices are the contributions
// of that input row to the five output rows it touches, whose FP32 accumulators
// sit side by side in TMEM (zeroed first). One 128 x 160 x 16 MMA thus replaces
// five 128 x 32 x 16 ones and the A tile is read from shared memory once instead
// of five times. Rows at the edges of the CTA's range issue only the slices of
// the output rows they own. Warp 0 stages rows, as soon as the barriers exist, while warp 1 allocates TMEM
// and warps 2-9 zero it. One elected thread of warp 1 then issues the MMAs and commits one mbarrier per
// finished output row, warps 2-9 run the epilogue (bias, GELU, its derivative, or FP32 output).
// Six layers (5 -> 32 -> ... -> 2) at 512^2: 60 us in a graph, at 128^2 29.4 (79 and 36 with the MMAs issued under
// lane == 0, the rows requested once all warps were ready and half a row's channels per epilogue warp): 0.42 us
// of MMAs per staged row, 1.3 us before the first and 0.7 after the last. All
// layers in one cooperative launch, with flags between neighbouring tiles, took longer than the launches that it
// saved. The data gradient of a circular convolution is the forward convolution with the kernel flipped and
// the channel roles swapped, so the same kernel serves it with the
// GELU-derivative epilogue.
//
// Weight-gradient kernel (conv_wgrad_kernel): dW[ky][kx][ci][co] = sum over sites and rows of
// X[ci][row j + ky - 2][site + kx - 2] dZ[co][row j][site]. A block of 16/(Cin/8) X rows is stacked along
// M ((row, ci), 128 rows) and all dZ rows within two of them along N ((chunk, row, channel), up to 384), so ONE
// instruction per x tap and 16 sites accumulates every (X row, dZ row) pair, of which the diagonals
// ky = X row - dZ row are the taps: the other pairs (3 of 8) are not read. Both operands MN-major. Against
// five y taps as separate 128 x 32 instructions, each of which reads the whole A tile (33 of its 41 cycles),
// this takes a third of the tensor time. A persistent CTA works through its row blocks (double-buffered bulk
// copies) and keeps its x taps' accumulators in TMEM over chains of kChain blocks; after each chain the epilogue
// warps add the diagonals to FP32 sums in their registers, while the next blocks arrive. It writes one partial;
// a second kernel reduces the partials in a fixed order (deterministic gradients). The same CTAs sum dZ
// over the sites while it is staged (bias gradients).
// The tensor core truncates each addition to an accumulator, so a chain's error grows with its length. Largest
// error over the largest gradient, values of mean 0.5, 32 x 32 channels, chains of 4 / 8 / 16 blocks / all blocks of
// the CTA: 16 x 128^2 sites 0.6e-6 / 1.1e-6 / 2.0e-6 / 2.4e-6, 16 x 512^2 0.7e-6 / 1.2e-6 / 2.2e-6 / 45e-6 (partials of
// eight rows, before the CTAs were persistent: 1.7e-6 and 3.9e-6).
// Measured for 16 x 128^2 sites, 32 x 32 channels: 26.7 us and 3.6 us for the reduction (one chain 26.0; one
// 128 x 32 instruction per tap, 256 partials: 80 and 17); 16 x 512^2, both: 520 us (one chain 513). 9 us of the 26.7 are
// instructions, the rest the copies, which the copy engine takes one by one (dZ rows that follow one another
// in memory go as one), and the epilogue.
#include "amb_gb300.h"
#include "amb_kernels.h"
#include "amb_tc.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>

namespace
{
    using namespace amb::tc;

    constexpr int kTile = 128;              // output sites per tile (one row window)
    constexpr int kSites = kTile + 4;       // staged input sites per row (halo 2 on each side)
    constexpr int kRowPlane = kSites * 16;  // bytes of one channel chunk of one staged row
    constexpr int kThreads = 192;           // wgrad: warp 0 loads, warp 1 issues MMAs, warps 2-5 epilogue
    constexpr int kFwdThreads = 320;        // forward: warp 0 loads, warp 1 issues MMAs, warps 2-9 epilogue
    constexpr int kMaxFwdRows = 16;         // forward: most output rows per CTA (all inputs staged at once)
    constexpr uint32_t kSmemLimit = 227u * 1024u;
    constexpr int kTaps = 25;

    enum Epilogue
    {
        EPI_GELU = 0,      // out = bf16(gelu(acc + bias)), pre = bf16(acc + bias)
        EPI_F32 = 1,       // out_f32 = acc + bias (first `cout` channels)
        EPI_GELU_BWD = 2,  // out = bf16(acc * gelu'(gate))
    };

    struct FwdArgs
    {
        const uint16_t* in;     // [batch][cin/8][nrows][ncols][8]
        const uint16_t* wimg;   // [5 kx][cin/8][5 (4 - ky)][npad][8] (B operand image, K-major)
        const float* bias;      // [npad] or null
        uint16_t* out;          // [batch][npad/8][nrows][ncols][8]
        uint16_t* pre;          // optional, same layout as out
        const uint16_t* gate;   // EPI_GELU_BWD: same layout as out
        float* out_f32;         // [batch][cout][nrows][ncols]
        int batch, nrows, ncols, cin_chunks, npad, cout, epilogue, rows_per_cta;
        int* error;
    };

    struct WgradArgs
    {
        const uint16_t* x;   // [batch][cin/8][nrows][ncols][8]
        const uint16_t* dz;  // [batch][npad/8][nrows][ncols][8]
        float* partial;      // [CTA][x tap of the CTA][5 ky][cin][npad]
        float* bias;         // [CTA of group 0][npad], or null
        int batch, nrows, ncols;
        int first[6];        // first CTA of each x-tap group
        int* error;
    };

    __host__ __device__ constexpr uint32_t align128(uint32_t x) { return (x + 127u) & ~127u; }

    __host__ __device__ inline uint32_t fwd_weight_bytes(int cc, int npad) { return uint32_t(kTaps) * cc * npad * 16u; }
    __host__ __device__ inline uint32_t fwd_rows_offset(int cc, int npad) { return align128(fwd_weight_bytes(cc, npad)); }
    __host__ __device__ inline uint32_t fwd_bar_offset(int cc, int npad, int rows)
    {
        return fwd_rows_offset(cc, npad) + uint32_t(rows + 4) * cc * kRowPlane;
    }
    // barriers: full[rows + 4], accf[rows], zero, wbar, done; then the TMEM slot and abort flag
    __host__ __device__ inline uint32_t fwd_smem_bytes(int cc, int npad, int rows)
    {
        return fwd_bar_offset(cc, npad, rows) + uint32_t(2 * rows + 4 + 3) * 8u + 16u;
    }
    // TMEM columns: one npad-wide accumulator per output row, rounded up to a power of two
    __host__ __device__ inline uint32_t fwd_tmem_cols(int npad, int rows)
    {
        uint32_t need = uint32_t(npad * rows), c = 32;
        while (c < need) c <<= 1;
        return c;
    }

    // Row blocks (of eight instructions each) that an accumulator takes before it is added to the FP32 sums.
    constexpr int kChain = 8;

    // wgrad geometry for Cin = 8 CC and NPAD gradient channels
    template <int CC, int NPAD>
    struct Wg
    {
        static constexpr int CIN = 8 * CC, NQ = NPAD / 8;
        static constexpr int XR = 16 / CC;           // X rows of a block: M = 128 = (row, ci)
        static constexpr int ZR = XR + 4;            // dZ rows of a block: N = (row, co)
        static constexpr int COLS = ZR * NPAD;       // TMEM columns of one x tap
        static constexpr int KPC = 512 / COLS;       // x taps per CTA
        static constexpr int GROUPS = (5 + KPC - 1) / KPC;
        static constexpr uint32_t XB = (uint32_t(XR) * CC * kRowPlane + 127u) & ~127u;
        static constexpr uint32_t STAGE = XB + uint32_t(ZR) * NQ * kTile * 16u;
        static constexpr int ROW = NPAD + 4;         // floats of an accumulator row in shared memory
        static constexpr uint32_t ACC = 128u * ROW * 4u;  // one tap of all accumulator rows
        static constexpr int NST = 2 * STAGE + ACC + 1024u <= kSmemLimit ? 2 : 1;
        static constexpr uint32_t BARS = NST * STAGE;
        static constexpr uint32_t ACCS = BARS + 128u + 4u * 32u * 4u;
        static constexpr uint32_t SMEM = ACCS + ACC;
        static constexpr int PART = KPC * 5 * CIN * NPAD;  // floats of one CTA's partial
        static constexpr int SUMS = (CIN * NPAD + 511) / 512;  // quads of a tap's gradients per epilogue thread
        static_assert(SMEM <= kSmemLimit, "shared memory");
    };

    __device__ __forceinline__ void give_up(int* error, volatile int* abort, int code)
    {
        *abort = 1;
        if (error) atomicExch(error, code);
    }

    __device__ __forceinline__ int wrap_row(int r, int n)
    {
        r %= n;
        return r < 0 ? r + n : r;
    }

    // GELU in its tanh form (Hendrycks and Gimpel): 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))),
    // with the hardware tanh approximation (relative error about 2^-11, below the bf16 rounding
    // of the stored activations; end-state statistics of long learned runs are unchanged by it).
    constexpr float kGeluC0 = 0.7978845608028654f;  // sqrt(2 / pi)
    constexpr float kGeluC1 = 0.044715f;

    __device__ __forceinline__ float tanh_hw(float u)
    {
        float t;
        asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
        return t;
    }

    __device__ __forceinline__ float gelu_f(float z)
    {
        const float t = tanh_hw(kGeluC0 * z * (1.f + kGeluC1 * z * z));
        return 0.5f * z * (1.f + t);
    }

    __device__ __forceinline__ float gelu_grad_f(float z)
    {
        const float z2 = z * z;
        const float t = tanh_hw(kGeluC0 * z * (1.f + kGeluC1 * z2));
        return 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * kGeluC0 * (1.f + 3.f * kGeluC1 * z2);
    }

    __device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
    {
        __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&h);
    }

    __device__ __forceinline__ void unpack_bf16x8(const uint4& u, float (&f)[8])
    {
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        }
    }

    // ================================================================ self-test
    // One CTA: D (128 x n) = A (128 x k) * B (n x k)^T from row-major inputs, with A
    // and B staged in the K-major or MN-major core-matrix layout. Layout constants:
    //   K-major  A: SBO = 128 (8-row groups along M), LBO = 16 * 128 (K chunks)
    //   MN-major A: LBO = 128 (8-row K groups),       SBO = (k / 8) * 128 (M groups)
    //   (B likewise with n in place of 128.)
    __global__ void __launch_bounds__(128) tc_selftest_kernel(const uint16_t* __restrict__ A,
                                                              const uint16_t* __restrict__ B, float* __restrict__ D,
                                                              int n, int k, int a_mn, int b_mn, int* error)
    {
        extern __shared__ __align__(1024) uint8_t smem[];
        uint8_t* sa = smem;             // 64 KB region (A uses at most 16 KB)
        uint8_t* sb = smem + 65536;     // 32 KB region (B uses at most 4 KB)
        uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 98304);
        uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 98304 + 64);
        volatile int* abort = reinterpret_cast<volatile int*>(smem + 98304 + 128);
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

        // zero both regions, then scatter the operands
        for (int i = tid; i < 98304 / 16; i += 128) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        for (int idx = tid; idx < 128 * k; idx += 128)
        {
            int m = idx / k, kk = idx % k;
            uint32_t off = a_mn ? (m / 8) * (k / 8) * 128 + (kk / 8) * 128 + (kk % 8) * 16 + (m % 8) * 2
                                : (kk / 8) * 16 * 128 + (m / 8) * 128 + (m % 8) * 16 + (kk % 8) * 2;
            *reinterpret_cast<uint16_t*>(sa + off) = A[idx];
        }
        for (int idx = tid; idx < n * k; idx += 128)
        {
            int r = idx / k, kk = idx % k;
            uint32_t off = b_mn ? (r / 8) * (k / 8) * 128 + (kk / 8) * 128 + (kk % 8) * 16 + (r % 8) * 2
                                : (kk / 8) * (n / 8) * 128 + (r / 8) * 128 + (r % 8) * 16 + (kk % 8) * 2;
            *reinterpret_cast<uint16_t*>(sb + off) = B[idx];
        }
        if (tid == 0)
        {
            mbar_init(bar, 1);
            *abort = 0;
            fence_mbar_init();
        }
        fence_proxy_async();
        if (warp == 0)
        {
            tmem_alloc(tslot, 32);
            tmem_relinquish();
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const uint32_t tbase = *tslot;

        if (tid == 0)
        {
            const uint32_t idesc = idesc_bf16(128, n, a_mn != 0, b_mn != 0);
            const uint32_t a0 = smem_u32(sa), b0 = smem_u32(sb);
            for (int ks = 0; ks < k / 16; ++ks)
            {
                uint64_t ad = a_mn ? smem_desc(a0 + 2 * ks * 128, 128, (k / 8) * 128)
                                   : smem_desc(a0 + 2 * ks * 16 * 128, 16 * 128, 128);
                uint64_t bd = b_mn ? smem_desc(b0 + 2 * ks * 128, 128, (k / 8) * 128)
                                   : smem_desc(b0 + 2 * ks * (n / 8) * 128, (n / 8) * 128, 128);
                mma_bf16(tbase, ad, bd, idesc, ks > 0 ? 1u : 0u);
            }
            mma_commit(bar);
        }
        bool ok = mbar_wait(bar, 0, nullptr);
        ok = __all_sync(0xffffffffu, ok);
        if (ok)
        {
            tc_fence_after();
            float v[32];
            const uint32_t taddr = tbase + (uint32_t(warp * 32) << 16);
            if (n == 32) tmem_ld32(taddr, v);
            else tmem_ld16(taddr, v);
            tmem_wait_ld();
            const int m = warp * 32 + lane;
#pragma unroll
            for (int c = 0; c < 32; ++c)
                if (c < n) D[m * n + c] = v[c];
        }
        else if (lane == 0)
            give_up(error, abort, 1);
        tc_fence_before();
        __syncthreads();
        if (warp == 0)
        {
            tc_fence_after();
            tmem_dealloc(tbase, 32);
        }
    }

    // The epilogue of output rows first, first + 2, .. of one lane quarter: `lanes` is the TMEM address of the
    // quarter, `site` the lane's site in the tile's first row. A warp reads a whole row's channels at once, so
    // the waits for the accumulators and for TMEM, which the MMAs keep busy, come once for 32 channels, and two
    // rows are under way (a half row of 16 channels per warp: 68.3 us per forward at 512^2, 65.6 so). False if
    // a wait gave up.
    template <int NPAD, int EPI>
    __device__ __forceinline__ bool epilogue_rows(const FwdArgs& a, uint64_t* accf, const volatile int* abort, uint32_t lanes,
                                                  int first, int nout, int b, size_t site)
    {
        constexpr int NQ = NPAD / 8;
        const size_t plane = size_t(a.nrows) * a.ncols;
        float bias[NPAD];
#pragma unroll
        for (int e = 0; e < NPAD; ++e) bias[e] = EPI != EPI_GELU_BWD && a.bias ? a.bias[e] : 0.f;
        for (int j = first; j < nout; j += 2)
        {
            const size_t at = site + size_t(j) * a.ncols;
            uint4 gate[NQ];
            if constexpr (EPI == EPI_GELU_BWD)
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    gate[q] = *reinterpret_cast<const uint4*>(a.gate + ((size_t(b) * NQ + q) * plane + at) * 8);
            if (!__all_sync(0xffffffffu, mbar_wait(&accf[j], 0, abort))) return false;
            tc_fence_after();
            float v[32];
            if constexpr (NPAD == 32) tmem_ld32(lanes + uint32_t(j * NPAD), v);
            else tmem_ld16(lanes + uint32_t(j * NPAD), v);
            tmem_wait_ld();
            if constexpr (EPI == EPI_F32)
            {
#pragma unroll
                for (int e = 0; e < NPAD; ++e)
                    if (e < a.cout) a.out_f32[(size_t(b) * a.cout + e) * plane + at] = v[e] + bias[e];
            }
            else
            {
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                {
                    const size_t off = ((size_t(b) * NQ + q) * plane + at) * 8;
                    float o[8];
                    if constexpr (EPI == EPI_GELU)
                    {
                        float z[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                        {
                            z[e] = v[8 * q + e] + bias[8 * q + e];
                            o[e] = gelu_f(z[e]);
                        }
                        if (a.pre)
                            *reinterpret_cast<uint4*>(a.pre + off) =
                                make_uint4(pack_bf16x2(z[0], z[1]), pack_bf16x2(z[2], z[3]), pack_bf16x2(z[4], z[5]),
                                           pack_bf16x2(z[6], z[7]));
                    }
                    else
                    {
                        float g[8];
                        unpack_bf16x8(gate[q], g);
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] = v[8 * q + e] * gelu_grad_f(g[e]);
                    }
                    *reinterpret_cast<uint4*>(a.out + off) = make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]),
                                                                        pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
                }
            }
        }
        return true;
    }

    // ============================================================== forward
    // CC = input channel chunks (2 or 4) and NPAD = output channels, compile-time constants so that the
    // MMA issue loop unrolls and every descriptor is a base plus a constant.
    template <int CC, int NPAD>
    __global__ void __launch_bounds__(kFwdThreads, 1) conv_fwd_kernel(const FwdArgs a)
    {
        extern __shared__ __align__(1024) uint8_t smem[];
        constexpr int cc = CC, npad = NPAD;
        const int R = a.rows_per_cta;
        const uint32_t wbytes = fwd_weight_bytes(cc, npad);
        const uint32_t slot_bytes = uint32_t(cc) * kRowPlane;
        const uint32_t tcols = fwd_tmem_cols(npad, R);
        uint8_t* wsm = smem;
        uint8_t* rows = smem + fwd_rows_offset(cc, npad);
        uint64_t* full = reinterpret_cast<uint64_t*>(smem + fwd_bar_offset(cc, npad, R));
        uint64_t* accf = full + R + 4;
        uint64_t* zbar = accf + R;
        uint64_t* wbar = zbar + 1;
        uint64_t* done = wbar + 1;
        uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
        volatile int* abort = reinterpret_cast<volatile int*>(tslot + 1);

        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int nwin = a.ncols / kTile;
        const int ngroups = (a.nrows + R - 1) / R;
        int t = blockIdx.x;
        const int cw = t % nwin;
        t /= nwin;
        const int rg = t % ngroups;
        const int b = t / ngroups;
        const int c0 = cw * kTile;
        const int r0 = rg * R;
        const int nout = min(R, a.nrows - r0);
        const int nin = nout + 4;

        const int left = c0 == 0 ? 2 : 0, right = c0 + kTile == a.ncols ? 2 : 0;  // wrapped sites
        if (warp == 0)
        {
            // a row completes with its bulk copies and one arrival per wrapped site (below)
            for (int i = lane; i < R + 4; i += 32) mbar_init(&full[i], 1 + cc * (left + right));
            if (lane < R) mbar_init(&accf[lane], 1);
            if (lane == 0)
            {
                mbar_init(zbar, 256);
                mbar_init(wbar, 1);
                mbar_init(done, 1);
                *abort = 0;
            }
            fence_mbar_init();
            asm volatile("bar.arrive 1, 320;" ::: "memory");  // the others need the barriers, this warp nothing of theirs
            // The operand image and every input row of this CTA at once, one mbarrier per row, in the order the MMAs consume them. The window's sites c0-2 .. c0+129 of each
            // (row, channel chunk): the in-range run by ONE bulk copy here; where the window wraps round the
            // periodic row (first and last windows, 2 sites each side) the epilogue warps copy the wrapped
            // 16-byte sites before their first wait (one mbarrier arrival each). The copies of a lane issue one
            // after another, those of a warp's lanes closer together.
            const int run = kSites - left - right;
            if (lane == 0)
            {
                mbar_expect_tx(wbar, wbytes);
                bulk_g2s(wsm, a.wimg, wbytes, wbar);
            }
            for (int i = lane; i < nin; i += 32) mbar_expect_tx(&full[i], uint32_t(cc * run) * 16u);
            __syncwarp();
            for (int it = lane; it < nin * cc; it += 32)
            {
                const int i = it / cc, q = it % cc;
                const int row = wrap_row(r0 - 2 + i, a.nrows);
                const uint16_t* src = a.in + (size_t(b * cc + q) * a.nrows + row) * size_t(a.ncols) * 8;
                bulk_g2s(rows + i * slot_bytes + q * kRowPlane + left * 16, src + size_t(c0 - 2 + left) * 8,
                         uint32_t(run) * 16u, &full[i]);
            }
        }
        else
        {
            if (warp == 1)
            {
                tmem_alloc(tslot, tcols);
                tmem_relinquish();
            }
            tc_fence_before();
            asm volatile("bar.sync 1, 320;" ::: "memory");
            tc_fence_after();
        }
        const uint32_t tbase = warp ? *tslot : 0u;

        if (warp == 0)
        {
            if (lane == 0)
            {
                // no copy may still be in flight when the CTA exits
                mbar_wait(wbar, 0, nullptr);
                for (int i = 0; i < nin; ++i) mbar_wait(&full[i], 0, nullptr);
            }
        }
        else if (warp == 1)
        {
            if (elect_one())
            {
                const uint32_t wsa = smem_u32(wsm), rsa = smem_u32(rows);
                constexpr uint32_t kblock = 5u * npad * 16u;  // one (x tap, channel chunk) block of the image
                bool ok = mbar_wait(wbar, 0, abort) && mbar_wait(zbar, 0, abort) && mbar_wait(&full[0], 0, abort);
                tc_fence_after();
                bool issued_any = false;
                // The tensor core holds few MMAs in its queue, so what the issuing thread does between rows must
                // be short: rows unrolled by 4, so that descriptors are ready ahead, and the next row's barrier
                // read while MMAs are queued (512^2, six layers: 65.6 us with neither, 63.1 and 60.0).
#pragma unroll 4
                for (int i = 0; ok && i < nin; ++i)
                {
                    // slice s of this row's MMA feeds output row i - 4 + s (y tap 4 - s)
                    const int s_lo = i < 4 ? 4 - i : 0;
                    const int s_hi = nout + 3 - i < 4 ? nout + 3 - i : 4;
                    const uint32_t idesc = idesc_bf16(128, npad * (s_hi - s_lo + 1), false, false);
                    const uint32_t d = tbase + uint32_t((i - 4 + s_lo) * npad);
                    // base descriptors of this row; every MMA adds (byte offset >> 4) to the start
                    // address field (addresses stay below 256 KiB, so the 14-bit field never carries)
                    const uint64_t a0 = smem_desc(rsa + i * slot_bytes, kRowPlane, 128);
                    const uint64_t b0 = smem_desc(wsa + uint32_t(s_lo * npad * 16), kblock, 128);
                    constexpr uint64_t bstep = kblock >> 4;
                    bool next = true;
#pragma unroll
                    for (int kx = 0; kx < 5; ++kx)
                    {
#pragma unroll
                        for (int ks = 0; ks < cc / 2; ++ks)
                            mma_bf16(d, a0 + uint64_t((2 * ks * kRowPlane + kx * 16) >> 4),
                                     b0 + uint64_t(kx * cc + 2 * ks) * bstep, idesc, 1u);
                        if (kx == 2 && i + 1 < nin) next = mbar_try_wait(&full[i + 1], 0);
                    }
                    issued_any = true;
                    if (i >= 4) mma_commit(&accf[i - 4]);  // output row i - 4 has all five y taps
                    ok = next || mbar_wait(&full[i + 1], 0, abort);
                }
                if (!ok) give_up(a.error, abort, 2);
                if (issued_any)
                {
                    mma_commit(done);
                    mbar_wait(done, 0, nullptr);
                }
            }
        }
        else
        {
            // warps 2-9: lane quarter (warp % 4) of the tile, every other output row from (warp - 2) / 4 on
            const int q4 = warp & 3;  // the TMEM lane quarter this warp may access
            const int half = (warp - 2) >> 2;
            // zero this warp's half of the accumulator columns in its lane quarter
            const uint32_t lanes = uint32_t(q4 * 32) << 16;
            for (uint32_t c = half * (tcols / 2); c < (half + 1) * (tcols / 2); c += 16)
                tmem_st16_zero(tbase + lanes + c);
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(zbar);
            {
                // the wrapped sites of the staged rows (see warp 0): 16-byte plain copies, made
                // visible to the async proxy, one arrival on the row's mbarrier each
                const int per_chunk = left + right, per_row = cc * per_chunk;
                for (int it = int(threadIdx.x) - 64; it < nin * per_row; it += kFwdThreads - 64)
                {
                    const int i = it / per_row, rem = it - i * per_row;
                    const int q = rem / per_chunk, s = rem - q * per_chunk;
                    const bool at_left = s < left;
                    const int wsite = at_left ? s : kSites - right + (s - left);  // site in the window
                    const int gcol = at_left ? a.ncols - 2 + s : s - left;        // its periodic column
                    const int row = wrap_row(r0 - 2 + i, a.nrows);
                    const uint4 v = *reinterpret_cast<const uint4*>(
                        a.in + ((size_t(b * cc + q) * a.nrows + row) * size_t(a.ncols) + gcol) * 8);
                    *reinterpret_cast<uint4*>(rows + i * slot_bytes + q * kRowPlane + wsite * 16) = v;
                    fence_proxy_async();
                    mbar_arrive(&full[i]);
                }
            }
            const size_t site = size_t(r0) * a.ncols + c0 + q4 * 32 + lane;
            const bool ok = a.epilogue == EPI_GELU  ? epilogue_rows<NPAD, EPI_GELU>(a, accf, abort, tbase + lanes, half, nout, b, site)
                            : a.epilogue == EPI_F32 ? epilogue_rows<NPAD, EPI_F32>(a, accf, abort, tbase + lanes, half, nout, b, site)
                                                    : epilogue_rows<NPAD, EPI_GELU_BWD>(a, accf, abort, tbase + lanes, half, nout, b, site);
            if (!ok && lane == 0) give_up(a.error, abort, 3);
        }

        tc_fence_before();
        __syncthreads();
        if (warp == 1)
        {
            tc_fence_after();
            tmem_dealloc(tbase, tcols);
        }
    }

    // =========================================================== weight grad
    template <int CC, int NPAD>
    __global__ void __launch_bounds__(kThreads, 1) conv_wgrad_kernel(const WgradArgs a)
    {
        using G = Wg<CC, NPAD>;
        extern __shared__ __align__(1024) uint8_t smem[];
        uint64_t* full = reinterpret_cast<uint64_t*>(smem + G::BARS);
        uint64_t* empty = full + 2;
        uint64_t* done = empty + 2;
        uint64_t* drained = done + 1;
        uint32_t* tslot = reinterpret_cast<uint32_t*>(drained + 1);
        volatile int* abort = reinterpret_cast<volatile int*>(tslot + 1);
        float* bsum = reinterpret_cast<float*>(smem + G::BARS + 128);

        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        int group = 0;
        while (int(blockIdx.x) >= a.first[group + 1]) ++group;
        const int kx0 = group * G::KPC, nkx = min(G::KPC, 5 - kx0);
        const int cta = blockIdx.x - a.first[group], nctas = a.first[group + 1] - a.first[group];
        // Row blocks: those of XR rows first, then, where the rows are no multiple of it, each image's last, whose
        // missing X rows are zeros. Those are chains of their own, of which only the rows there are count: a zero row
        // times an infinite gradient is no zero.
        const int nwin = a.ncols / kTile, nblk = a.nrows / G::XR, rest = a.nrows - nblk * G::XR;
        const int whole = a.batch * nwin * nblk, total = whole + (rest ? a.batch * nwin : 0);
        const auto dealt = [&](int n) { return cta < n ? int(unsigned(n - cta + nctas - 1) / unsigned(nctas)) : 0; };
        const int mine = dealt(total), mine_whole = dealt(whole);  // row blocks of this CTA

        struct Block
        {
            int b, c0, r0, rows, left, right;  // image, first column, first X row, X rows, wrapped sites
        };
        const auto block = [&](int i) {
            const bool full = i < mine_whole;
            const unsigned t = cta + i * nctas - (full ? 0 : whole), n = full ? nblk : 1, u = t / n, v = u / unsigned(nwin);
            Block k;
            k.rows = full ? G::XR : rest;
            k.r0 = int(full ? t - u * n : nblk) * G::XR;
            k.c0 = int(u - v * nwin) * kTile;
            k.b = int(v);
            k.left = k.c0 == 0 ? 2 : 0;
            k.right = k.c0 + kTile == a.ncols ? 2 : 0;
            return k;
        };
        // The last block of a chain, given the blocks that the chain has before it.
        const auto ends = [&](int i, int before) { return before == kChain - 1 || i == mine_whole - 1 || i == mine - 1; };

        if (threadIdx.x == 0)
        {
            for (int i = 0; i < G::NST; ++i)
            {
                mbar_init(&full[i], 1 + 4);   // the loader and the four helper warps
                mbar_init(&empty[i], 1 + 4);  // the MMAs' completion and the helper warps
            }
            mbar_init(done, 1);     // the MMAs of a chain
            mbar_init(drained, 4);  // the epilogue warps have read its accumulators
            *abort = 0;
            fence_mbar_init();
        }
        if (warp == 0)
        {
            tmem_alloc(tslot, 512);
            tmem_relinquish();
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const uint32_t tbase = *tslot;

        if (warp == 0)
        {
            {
                // the copies of a block spread over the warp's lanes: one thread takes about 120 cycles to issue
                // each, the copy engine 75 per 2 KB and 148 per 8 KB
                int issued = 0;
                bool ok = true;
                for (int i = 0; i < mine; ++i)
                {
                    const int st = i % G::NST;
                    if (i >= G::NST)
                        ok = __all_sync(0xffffffffu, mbar_wait(&empty[st], (i / G::NST - 1) & 1, abort));
                    if (!ok) break;
                    const Block k = block(i);
                    const int lo = k.c0 - 2 + k.left, run = kSites - k.left - k.right;
                    uint8_t* xs = smem + st * G::STAGE;
                    uint8_t* zs = xs + G::XB;
                    if (lane == 0)
                        mbar_expect_tx(&full[st], uint32_t(k.rows * CC * run) * 16u + uint32_t(G::ZR * G::NQ) * kTile * 16u);
                    __syncwarp();
                    const int nxc = k.rows * CC;
                    for (int c = lane; c < nxc; c += 32)
                        bulk_g2s(xs + c * kRowPlane + k.left * 16,
                                 a.x + ((size_t(k.b * CC + c % CC) * a.nrows + k.r0 + c / CC) * size_t(a.ncols) + lo) * 8,
                                 uint32_t(run) * 16u, &full[st]);
                    // dZ rows r0 - 2 .. r0 + XR + 1, a chunk's rows one after the other: one copy per row, or, where
                    // the window is the whole row, one per run of rows up to the image's end
                    const bool runs = a.ncols == kTile && a.nrows >= G::ZR;
                    const int z0 = wrap_row(k.r0 - 2, a.nrows), n0 = runs ? min(G::ZR, a.nrows - z0) : 1;
                    const int per = runs ? (n0 < G::ZR ? 2 : 1) : G::ZR;
                    for (int c = lane; c < G::NQ * per; c += 32)
                    {
                        const int q = c / per, e = c - q * per;
                        const int r = runs ? e * n0 : e, n = runs ? (e ? G::ZR - n0 : n0) : 1;
                        bulk_g2s(zs + (q * G::ZR + r) * (kTile * 16),
                                 a.dz + ((size_t(k.b * G::NQ + q) * a.nrows + wrap_row(k.r0 - 2 + r, a.nrows))
                                             * size_t(a.ncols) + k.c0) * 8,
                                 uint32_t(n) * kTile * 16u, &full[st]);
                    }
                    __syncwarp();
                    ++issued;
                }
                if (!ok && lane == 0) give_up(a.error, abort, 4);
                // no copy may still be in flight when the CTA exits (the last of each stage completes last)
                for (int i = max(0, issued - G::NST); i < issued; ++i)
                    mbar_wait(&full[i % G::NST], (i / G::NST) & 1, nullptr);
            }
        }
        else if (warp == 1)
        {
            if (elect_one())
            {
                constexpr int N0 = G::COLS < 256 ? G::COLS : 256, N1 = G::COLS - N0;
                const uint32_t id0 = idesc_bf16(128, N0, true, true), id1 = idesc_bf16(128, N1 > 0 ? N1 : 16, true, true);
                const uint32_t sa = smem_u32(smem);
                bool ok = true, open = false;
                int chains = 0, before = 0;  // chains committed, blocks of the next one; open: it has instructions issued
                for (int i = 0; ok && i < mine; ++i)
                {
                    const int st = i % G::NST;
                    if (!mbar_wait(&full[st], (i / G::NST) & 1, abort) ||
                        (before == 0 && chains > 0 && !mbar_wait(drained, (chains - 1) & 1, abort)))
                    {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const bool first = before == 0;
                    const uint32_t xa = sa + st * G::STAGE, za = xa + G::XB;
                    for (int kxi = 0; kxi < nkx; ++kxi)
#pragma unroll
                        for (int ks = 0; ks < kTile / 16; ++ks)
                        {
                            const uint64_t ad = smem_desc(xa + uint32_t(ks * 16 + kx0 + kxi) * 16u, 128, kRowPlane);
                            const uint32_t d = tbase + uint32_t(kxi * G::COLS), acc = first && ks == 0 ? 0u : 1u;
                            mma_bf16(d, ad, smem_desc(za + ks * 256, 128, kTile * 16), id0, acc);
                            if constexpr (N1 > 0)
                                mma_bf16(d + N0, ad, smem_desc(za + (N0 / 8) * (kTile * 16) + ks * 256, 128, kTile * 16),
                                         id1, acc);
                        }
                    mma_commit(&empty[st]);
                    open = !ends(i, before++);
                    if (!open)
                    {
                        mma_commit(done);
                        ++chains;
                        before = 0;
                    }
                }
                if (!ok) give_up(a.error, abort, 5);
                if (open)
                {
                    mma_commit(done);
                    ++chains;
                }
                if (chains > 0 && !mbar_wait(done, (chains - 1) & 1, nullptr)) give_up(a.error, abort, 6);
            }
        }
        else
        {
            const int t = int(threadIdx.x) - 64;
            const bool bias = a.bias != nullptr && group == 0;
            float bs[G::NQ][8];
#pragma unroll
            for (int q = 0; q < G::NQ; ++q)
#pragma unroll
                for (int e = 0; e < 8; ++e) bs[q][e] = 0.f;
            bool ok = true;
            // ahead of the MMAs: the wrapped sites of a stage's X rows, zeros in the rows past the image
            const auto prepare = [&](int i) {
                const int st = i % G::NST;
                if (i >= G::NST) ok = __all_sync(0xffffffffu, ok && mbar_wait(&empty[st], (i / G::NST - 1) & 1, abort));
                if (!ok) return;
                const Block k = block(i);
                uint8_t* xs = smem + st * G::STAGE;
                const int per_chunk = k.left + k.right, per_row = CC * per_chunk;
                for (int it = t; it < k.rows * per_row; it += 128)
                {
                    const int r = it / per_row, rem = it - r * per_row;
                    const int q = rem / per_chunk, s = rem - q * per_chunk;
                    const bool at_left = s < k.left;
                    const int wsite = at_left ? s : kSites - k.right + (s - k.left);
                    const int gcol = at_left ? a.ncols - 2 + s : s - k.left;
                    *reinterpret_cast<uint4*>(xs + (r * CC + q) * kRowPlane + wsite * 16) = *reinterpret_cast<const uint4*>(
                        a.x + ((size_t(k.b * CC + q) * a.nrows + k.r0 + r) * size_t(a.ncols) + gcol) * 8);
                }
                for (int it = t; it < (G::XR - k.rows) * CC * kSites; it += 128)
                    *reinterpret_cast<uint4*>(xs + k.rows * CC * kRowPlane + it * 16) = make_uint4(0, 0, 0, 0);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[st]);
            };
            const auto finish = [&](int i) {
                const int st = i % G::NST;
                if (bias)
                {
                    ok = __all_sync(0xffffffffu, ok && mbar_wait(&full[st], (i / G::NST) & 1, abort));
                    if (!ok) return;
                    const Block k = block(i);
                    const uint8_t* zs = smem + st * G::STAGE + G::XB;
                    for (int r = 2; r < 2 + k.rows; ++r)  // the dZ rows with the block's X rows' numbers
#pragma unroll
                        for (int q = 0; q < G::NQ; ++q)
                        {
                            float v[8];
                            unpack_bf16x8(*reinterpret_cast<const uint4*>(zs + (q * G::ZR + r) * (kTile * 16) + t * 16), v);
#pragma unroll
                            for (int e = 0; e < 8; ++e) bs[q][e] += v[e];
                        }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[st]);
            };
            // A finished chain: the diagonals of its accumulators, summed over the X rows of a block through shared
            // memory and added to the thread's share of the gradients. The lane's accumulator row is X row xr,
            // channel ci; tap ky is dZ row xr - ky + 4 of the block. All four warps come here for every chain,
            // whatever their waits gave, so that the block barriers match.
            float4 sum[G::KPC][5][G::SUMS];
#pragma unroll
            for (int kxi = 0; kxi < G::KPC; ++kxi)
#pragma unroll
                for (int ky = 0; ky < 5; ++ky)
#pragma unroll
                    for (int f = 0; f < G::SUMS; ++f) sum[kxi][ky][f] = make_float4(0.f, 0.f, 0.f, 0.f);
            float* acc = reinterpret_cast<float*>(smem + G::ACCS);
            const auto sync4 = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
            const int q4 = warp & 3;
            const uint32_t lanes = uint32_t(q4 * 32) << 16;
            const auto load = [&](int kxi, int zr, float (&v)[32]) {  // the NPAD channels of dZ row zr
#pragma unroll
                for (int q = 0; q < G::NQ; ++q)
                    tmem_ld8(tbase + lanes + uint32_t(kxi * G::COLS + (q * G::ZR + zr) * 8), v + 8 * q);
                tmem_wait_ld();
            };
            const auto drain = [&](int chain, auto whole_blocks) {
                ok = __all_sync(0xffffffffu, ok && mbar_wait(done, chain & 1, abort));
                if (!ok && lane == 0) give_up(a.error, abort, 8);
                tc_fence_after();
#pragma unroll
                for (int kxi = 0; kxi < G::KPC; ++kxi)
                {
                    if (kxi >= nkx) continue;
#pragma unroll
                    for (int ky = 0; ky < 5; ++ky)
                    {
                        float v[32];
                        load(kxi, q4 * (G::XR / 4) - ky + 4, v);
                        if constexpr (CC == 2)  // two X rows per warp: the upper lanes' dZ row is the next one
                        {
                            float w[32];
                            load(kxi, 2 * q4 - ky + 5, w);
#pragma unroll
                            for (int n = 0; n < NPAD; ++n) v[n] = lane < 16 ? v[n] : w[n];
                        }
                        if constexpr (!decltype(whole_blocks)::value)
                        {
                            const bool counts = (q4 * 32 + lane) / G::CIN < rest;  // not a row past the image
#pragma unroll
                            for (int n = 0; n < NPAD; ++n) v[n] = counts ? v[n] : 0.f;
                        }
                        sync4();  // the tap before is read
                        float* row = acc + (q4 * 32 + lane) * G::ROW;
#pragma unroll
                        for (int n = 0; n < NPAD; n += 4)
                            *reinterpret_cast<float4*>(row + n) = make_float4(v[n], v[n + 1], v[n + 2], v[n + 3]);
                        sync4();
#pragma unroll
                        for (int f = 0; f < G::SUMS; ++f)
                        {
                            const int e = t + f * 128, ci = e / (NPAD / 4), n = e % (NPAD / 4) * 4;
                            if (G::CIN * NPAD % 512 != 0 && ci >= G::CIN) continue;
                            float4 s = *reinterpret_cast<const float4*>(acc + ci * G::ROW + n);
#pragma unroll
                            for (int xr = 1; xr < G::XR; ++xr)
                            {
                                const float4 u = *reinterpret_cast<const float4*>(acc + (xr * G::CIN + ci) * G::ROW + n);
                                s.x += u.x; s.y += u.y; s.z += u.z; s.w += u.w;
                            }
                            float4& g = sum[kxi][ky][f];
                            g.x += s.x; g.y += s.y; g.z += s.z; g.w += s.w;
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(drained);
            };
            int chain = 0, before = 0;
            for (int i = 0; i < mine + G::NST - 1; ++i)
            {
                const int j = i - (G::NST - 1);
                if (i < mine && ok) prepare(i);
                if (j >= 0 && ok) finish(j);
                if (!ok && lane == 0) give_up(a.error, abort, 7);
                if (j < 0 || !ends(j, before++)) continue;
                if (j < mine_whole) drain(chain++, std::true_type{});
                else drain(chain++, std::false_type{});
                before = 0;
            }
            float* part = a.partial + size_t(blockIdx.x) * G::PART;
#pragma unroll
            for (int kxi = 0; kxi < G::KPC; ++kxi)
#pragma unroll
                for (int ky = 0; ky < 5; ++ky)
#pragma unroll
                    for (int f = 0; f < G::SUMS; ++f)
                    {
                        const int e = t + f * 128;
                        if (kxi < nkx && e < G::CIN * NPAD / 4)
                            *reinterpret_cast<float4*>(part + size_t((kxi * 5 + ky) * G::CIN) * NPAD + e * 4) = sum[kxi][ky][f];
                    }
            if (bias)
            {
#pragma unroll
                for (int q = 0; q < G::NQ; ++q)
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                    {
                        float v = bs[q][e];
#pragma unroll
                        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                        if (lane == 0) bsum[(warp - 2) * 32 + q * 8 + e] = v;
                    }
                sync4();
                if (t < NPAD) a.bias[size_t(cta) * NPAD + t] = ((bsum[t] + bsum[32 + t]) + bsum[64 + t]) + bsum[96 + t];
            }
        }

        tc_fence_before();
        __syncthreads();
        if (warp == 0)
        {
            tc_fence_after();
            tmem_dealloc(tbase, 512);
        }
    }

    struct WgradReduceArgs
    {
        const float* partial;
        const float* bias_partial;
        int first[6];          // CTAs of each x-tap group
        int kpc, cin, npad;
        float* dw;             // [25][cin][npad], or null
        float* gw;             // [cout][cin_used][5][5], or null
        float* gb;             // [npad], or null
        int cout, cin_used;
    };

    // Sum of the CTAs' partials, four channels per thread, eight slices of the CTAs per element added in a
    // fixed order; the last block sums the bias partials.
    __global__ void __launch_bounds__(256) wgrad_reduce_kernel(const WgradReduceArgs a)
    {
        __shared__ float4 sums[8][32];
        const int el = threadIdx.x & 31, slice = threadIdx.x >> 5;
        const int n4 = a.npad / 4, total = 25 * a.cin * n4;
        const int e = blockIdx.x * 32 + el;
        if (blockIdx.x * 32 >= total)  // the bias block
        {
            float s = 0.f;
            if (el < a.npad)
                for (int c = slice; c < a.first[1]; c += 8) s += a.bias_partial[size_t(c) * a.npad + el];
            sums[slice][el].x = s;
            __syncthreads();
            if (slice == 0 && el < a.npad)
            {
                float v = sums[0][el].x;
                for (int i = 1; i < 8; ++i) v += sums[i][el].x;
                a.gb[el] = v;
            }
            return;
        }
        const int tap = e / (a.cin * n4), ci = e / n4 - tap * a.cin, n = e % n4;
        const int ky = tap / 5, kx = tap - ky * 5, g = kx / a.kpc;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e < total)
        {
            const size_t part = size_t(a.kpc) * 5 * a.cin * a.npad;
            const float* p = a.partial + ((size_t(kx - g * a.kpc) * 5 + ky) * a.cin + ci) * a.npad + n * 4;
            for (int c = a.first[g] + slice; c < a.first[g + 1]; c += 8)
            {
                const float4 v = *reinterpret_cast<const float4*>(p + size_t(c) * part);
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
        }
        sums[slice][el] = s;
        __syncthreads();
        if (slice != 0 || e >= total) return;
        for (int i = 1; i < 8; ++i)
        {
            const float4 v = sums[i][el];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        const float v[4] = {s.x, s.y, s.z, s.w};
        if (a.dw)  // a caller's array, aligned to its floats only
            for (int q = 0; q < 4; ++q) a.dw[(size_t(tap) * a.cin + ci) * a.npad + n * 4 + q] = v[q];
        if (a.gw && ci < a.cin_used)
            for (int q = 0; q < 4; ++q)
                if (n * 4 + q < a.cout) a.gw[(size_t(n * 4 + q) * a.cin_used + ci) * 25 + tap] = v[q];
    }

    // Operand images of the layers' weights w [cout][cin][5][5], one layer per blockIdx.y: the forward
    // convolution's [5 kx][cin_pad/8][5 (4 - ky)][npad][8] and, with the kernel flipped and the channel roles
    // swapped, the data gradient's [5 kx][npad/8][5 (4 - ky)][cin_pad][8], zero in the padding.
    constexpr int kImageLayers = 8;
    struct ImageArgs
    {
        struct Layer
        {
            const float* w;
            __nv_bfloat16 *img, *dimg;
            int cout, cin, cin_pad, npad;
        } layer[kImageLayers];
    };

    __global__ void weight_images_kernel(const __grid_constant__ ImageArgs args)
    {
        const ImageArgs::Layer& a = args.layer[blockIdx.y];
        const int n = 25 * a.cin_pad * a.npad;
        for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 2 * n; t += gridDim.x * blockDim.x)
        {
            const bool fwd = t < n;
            if (!(fwd ? a.img : a.dimg)) continue;
            const int k = fwd ? a.cin_pad : a.npad, m = fwd ? a.npad : a.cin_pad;  // channels along K, along N
            int e = fwd ? t : t - n;
            const int e0 = e % 8;
            e /= 8;
            const int row = e % m;
            e /= m;
            const int s = e % 5;
            e /= 5;
            const int kc = (e % (k / 8)) * 8 + e0, kx = e / (k / 8);
            const int co = fwd ? row : kc, ci = fwd ? kc : row;
            float v = 0.f;
            if (co < a.cout && ci < a.cin)
                v = a.w[((size_t(co) * a.cin + ci) * 5 + (fwd ? 4 - s : s)) * 5 + (fwd ? kx : 4 - kx)];
            (fwd ? a.img : a.dimg)[fwd ? t : t - n] = __float2bfloat16_rn(v);
        }
    }

    // FP32 planes [batch][c][plane] as bf16 chunk planes [batch][npad/8][plane][8], zero from channel c on.
    __global__ void chunk_kernel(const float* __restrict__ x, int c, int npad, size_t plane, size_t n, uint4* __restrict__ out)
    {
        for (size_t t = blockIdx.x * size_t(blockDim.x) + threadIdx.x; t < n; t += size_t(gridDim.x) * blockDim.x)
        {
            const size_t s = t % plane, r = t / plane;
            const int q = int(r % (npad / 8));
            const float* p = x + (r / (npad / 8)) * c * plane + s;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 8 * q + e < c ? p[(8 * q + e) * plane] : 0.f;
            out[t] = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                pack_bf16x2(v[6], v[7]));
        }
    }

    // ================================================== learned-step helpers
    // Network input planes from the field and per-sample parameters: channel 0 =
    // bf16(phi), 1 = 256 (phi - bf16(phi)) (the rounding remainder, so phi is
    // carried to ~16 significant bits), 2 = zeta / 4, 3 = lambda, 4 = 10 T, 5-15 = 0.
    __global__ void learned_input_kernel(const float* __restrict__ phi, const float* __restrict__ params, int batch,
                                         int nrows, int ncols, uint16_t* __restrict__ x)
    {
        const size_t plane = size_t(nrows) * ncols;
        const size_t n = size_t(batch) * plane;
        for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        {
            const int b = int(i / plane);
            const size_t s = i - size_t(b) * plane;
            const float f = phi[i];
            const __nv_bfloat16 hi = __float2bfloat16_rn(f);
            const float lo = (f - __bfloat162float(hi)) * 256.f;
            const float* pr = params + 3 * b;
            uint4 c0 = make_uint4(pack_bf16x2(__bfloat162float(hi), lo), pack_bf16x2(pr[0] * 0.25f, pr[1]),
                                  pack_bf16x2(pr[2] * 10.f, 0.f), 0u);
            reinterpret_cast<uint4*>(x)[(size_t(b) * 2 + 0) * plane + s] = c0;
            reinterpret_cast<uint4*>(x)[(size_t(b) * 2 + 1) * plane + s] = make_uint4(0, 0, 0, 0);
        }
    }

    // Two standard normals per site for the macro-step noise flux, Philox keyed
    // (seed, *step, site, component).
    __global__ void learned_noise_kernel(float* __restrict__ xi, int nrows, int ncols, uint64_t seed,
                                         const int64_t* __restrict__ step)
    {
        const int64_t st = *step;
        const size_t plane = size_t(nrows) * ncols;
        for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < plane; i += size_t(gridDim.x) * blockDim.x)
        {
            const int r = int(i / ncols), c = int(i - size_t(r) * ncols);
            xi[i] = amb::noise_normal(seed, st, r, c, 0);
            xi[plane + i] = amb::noise_normal(seed, st, r, c, 1);
        }
    }

    // The rfft2 spectra of two real white-noise fields of unit variance per site, drawn directly:
    // out[comp][r][k] at out + comp * n + r * rs + k * ks (complex64; k < ncols/2 + 1). Off the
    // self-conjugate columns (k = 0 and, for even ncols, k = ncols/2) each mode is a complex
    // normal with E|z|^2 = nrows ncols; in those columns mode r is the conjugate of mode
    // nrows - r, and the self-conjugate modes (r = 0, r = nrows/2) are real with the same
    // variance. One Philox call per (r, k) (keyed by the lower of r and nrows - r in those
    // columns) gives both components.
    __device__ __forceinline__ void spectral_noise_mode(uint64_t seed, int64_t st, int r, int k, int nrows, int ncols,
                                                        float2& vy, float2& vx)
    {
        const float s_half = sqrtf(0.5f * float(nrows) * float(ncols));
        const float s_full = sqrtf(float(nrows) * float(ncols));
        const bool herm = k == 0 || (ncols % 2 == 0 && k == ncols / 2);
        int rr = r;
        bool conj = false;
        if (herm && r > nrows / 2)
        {
            rr = nrows - r;
            conj = true;
        }
        const amb::U4 b = amb::noise_bits(seed, st, rr, 4 * k, 0);
        const float2 z0 = amb::box_muller_f32(b.x, b.y), z1 = amb::box_muller_f32(b.z, b.w);
        vy = make_float2(z0.x * s_half, z0.y * s_half);
        vx = make_float2(z1.x * s_half, z1.y * s_half);
        if (herm && (rr == 0 || (nrows % 2 == 0 && rr == nrows / 2)))
        {
            vy = make_float2(z0.x * s_full, 0.f);
            vx = make_float2(z1.x * s_full, 0.f);
        }
        if (conj)
        {
            vy.y = -vy.y;
            vx.y = -vx.y;
        }
    }

    __global__ void learned_noise_spectral_kernel(float2* __restrict__ out, int nrows, int ncols, int64_t rs,
                                                  int64_t ks, int64_t n, uint64_t seed,
                                                  const int64_t* __restrict__ step)
    {
        const int nk = ncols / 2 + 1;
        const int64_t st = *step;
        const int64_t total = int64_t(nrows) * nk;
        for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < total;
             i += int64_t(gridDim.x) * blockDim.x)
        {
            const int r = int(i / nk), k = int(i - int64_t(r) * nk);
            float2 vy, vx;
            spectral_noise_mode(seed, st, r, k, nrows, ncols, vy, vx);
            out[int64_t(r) * rs + int64_t(k) * ks] = vy;
            out[n + int64_t(r) * rs + int64_t(k) * ks] = vx;
        }
    }

    // The spectral combine with the noise spectrum drawn in place (the draw of
    // learned_noise_spectral_kernel for the same seed and step): the spectra are dense in
    // memory with row stride rs and column stride ks, one of them 1.
    __global__ void spectral_combine_noise_kernel(const float2* __restrict__ phi_hat, const float2* __restrict__ my,
                                                  const float2* __restrict__ mx, const float2* __restrict__ ny_,
                                                  const float2* __restrict__ nx_, float noise_mag, int nrows,
                                                  int ncols, int64_t rs, int64_t ks, uint64_t seed,
                                                  const int64_t* __restrict__ step, float2* __restrict__ out_y,
                                                  float2* __restrict__ out_x)
    {
        const int64_t n = int64_t(nrows) * (ncols / 2 + 1);
        const int64_t st = *step;
        for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        {
            int r, k;
            if (n <= INT32_MAX)  // 32-bit division (a 64-bit one costs several times the instructions)
            {
                const int ii = int(i);
                if (ks == 1)
                {
                    r = ii / int(rs);
                    k = ii - r * int(rs);
                }
                else
                {
                    k = ii / int(ks);
                    r = ii - k * int(ks);
                }
            }
            else if (ks == 1)
            {
                r = int(i / rs);
                k = int(i - int64_t(r) * rs);
            }
            else
            {
                k = int(i / ks);
                r = int(i - int64_t(k) * ks);
            }
            float2 u, v;
            spectral_noise_mode(seed, st, r, k, nrows, ncols, u, v);
            const float2 p = phi_hat[i], a = my[i], b = mx[i], c = ny_[i], d = nx_[i];
            float2 y = make_float2(p.x * a.x - p.y * a.y, p.x * a.y + p.y * a.x);
            float2 x = make_float2(p.x * b.x - p.y * b.y, p.x * b.y + p.y * b.x);
            y.x += noise_mag * (u.x * c.x - u.y * c.y);
            y.y += noise_mag * (u.x * c.y + u.y * c.x);
            x.x += noise_mag * (v.x * d.x - v.y * d.y);
            x.y += noise_mag * (v.x * d.y + v.y * d.x);
            out_y[i] = y;
            out_x[i] = x;
        }
    }

    // Face weights of the order-8 central derivative written as a difference of face sums:
    // D8 f(j) = F(j + 1/2) - F(j - 1/2) with F(j + 1/2) = sum_e w_e f(j + e), e = -3..4,
    // w_e = sum of c_d over d >= max(e, 1 - e), c = (4/5, -1/5, 4/105, -1/280) (the sum in
    // double, in increasing d, then rounded to float).
    constexpr double kC1 = 4.0 / 5.0, kC2 = -1.0 / 5.0, kC3 = 4.0 / 105.0, kC4 = -1.0 / 280.0;

    __device__ __forceinline__ float d8_face_weight(int e)
    {
        const int d0 = e > 1 - e ? e : 1 - e;
        return d0 == 1 ? float(kC1 + kC2 + kC3 + kC4)
                       : d0 == 2 ? float(kC2 + kC3 + kC4) : d0 == 3 ? float(kC3 + kC4) : float(kC4);
    }

    // Integer face increment through the face after site (r, c) along the axis (dr, dc), in
    // FP32 with explicitly rounded operations, so the two sites sharing the face compute the
    // same integer.
    __device__ __forceinline__ long long face_q(const float* __restrict__ f, const float* __restrict__ extra,
                                                const float* __restrict__ xi, float noise_mag, float scale, int r,
                                                int c, int dr, int dc, int nrows, int ncols)
    {
        const size_t k = size_t(r) * ncols + c;
        float v = f[k];
        if (extra) v = __fadd_rn(v, extra[k]);
        if (xi)
        {
            float s = 0.f;
#pragma unroll
            for (int e = -3; e <= 4; ++e)
            {
                int rr = r + dr * e, cc = c + dc * e;
                rr = rr < 0 ? rr + nrows : (rr >= nrows ? rr - nrows : rr);
                cc = cc < 0 ? cc + ncols : (cc >= ncols ? cc - ncols : cc);
                s = __fadd_rn(s, __fmul_rn(d8_face_weight(e), xi[size_t(rr) * ncols + cc]));
            }
            v = __fadd_rn(v, __fmul_rn(noise_mag, s));
        }
        float q = __fmul_rn(scale, v);
        q = q > 1e9f ? 1e9f : (q < -1e9f ? -1e9f : q);
        return (long long)__float2int_rn(q);  // |q| <= 1e9 < 2^31: the same value as a 64-bit conversion
    }

    // One site's new fixed-point value from its four face increments, with the checks that fail a span.
    __device__ __forceinline__ int updated_q(int q0, long long dq, bool finite, long long bound, bool* bad)
    {
        long long q = (long long)q0 - dq;
        if (!finite || q > bound || q < -bound)
        {
            *bad = true;
            q = q > bound ? bound : (q < -bound ? -bound : q);
        }
        return int32_t(q);
    }

    // q * 2^-24 rounded once to FP32: rounding q to FP32 and scaling by a power of two gives the same value
    // (|q| <= 2e9, so the scaled value is a normal number or zero)
    __device__ __forceinline__ float field_of(int q) { return __fmul_rn(__int2float_rn(q), 1.0f / 16777216.0f); }

    // Channel chunk 0 of the next network input, as learned_input_kernel forms it.
    __device__ __forceinline__ uint4 input_chunk(float f, float p0, float p1, float p2)
    {
        const __nv_bfloat16 hi = __float2bfloat16_rn(f);
        const float lo = (f - __bfloat162float(hi)) * 256.f;
        return make_uint4(pack_bf16x2(__bfloat162float(hi), lo), pack_bf16x2(p0 * 0.25f, p1), pack_bf16x2(p2 * 10.f, 0.f), 0u);
    }

    // phi_q -= sum of integer face increments (each face computed identically by the two
    // sites that share it, so the sum over all sites is unchanged: exact conservation).
    __global__ void learned_update_kernel(const float* __restrict__ flux, const float* __restrict__ extra,
                                          const float* __restrict__ xi, int nrows, int ncols, float scale_y,
                                          float scale_x, float noise_mag, int32_t* __restrict__ phi_q,
                                          float* __restrict__ phi_f, long long bound, int* __restrict__ flag,
                                          int64_t* __restrict__ advance, const float* __restrict__ params,
                                          uint4* __restrict__ x_next)
    {
        // the next macro step's noise key (nothing in this launch reads it)
        if (advance && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *advance += 1;
        const size_t plane = size_t(nrows) * ncols;
        const float* fy = flux;
        const float* fx = flux + plane;
        const float* ey = extra;
        const float* ex = extra ? extra + plane : nullptr;
        const float* xy = xi;
        const float* xx = xi ? xi + plane : nullptr;
        // rows by blockIdx.y (grid-stride), columns by blockIdx.x and the thread: no division per site
        const int c = blockIdx.x * blockDim.x + threadIdx.x;
        if (c >= ncols) return;
        const int cm = c == 0 ? ncols - 1 : c - 1;
        for (int r = blockIdx.y; r < nrows; r += gridDim.y)
        {
            const size_t i = size_t(r) * ncols + c;
            const int rm = r == 0 ? nrows - 1 : r - 1;
            long long dq = face_q(fx, ex, xx, noise_mag, scale_x, r, c, 0, 1, nrows, ncols) -
                           face_q(fx, ex, xx, noise_mag, scale_x, r, cm, 0, 1, nrows, ncols) +
                           face_q(fy, ey, xy, noise_mag, scale_y, r, c, 1, 0, nrows, ncols) -
                           face_q(fy, ey, xy, noise_mag, scale_y, rm, c, 1, 0, nrows, ncols);
            bool bad = false;
            const bool finite = isfinite(fx[i]) && isfinite(fy[i]) && (!extra || (isfinite(ex[i]) && isfinite(ey[i])));
            const int q = updated_q(phi_q[i], dq, finite, bound, &bad);
            if (bad) atomicOr(flag, 1);
            phi_q[i] = q;
            const float f = field_of(q);
            phi_f[i] = f;
            if (x_next) x_next[i] = input_chunk(f, params[0], params[1], params[2]);
        }
    }

    // The same on four columns per thread, for rows of whole aligned 16-byte quads and no per-site noise: a quarter of
    // the threads, 13 faces instead of 16 and wide accesses (a macro step at
    // 512^2: 82.6 -> 79.2 us, at 768^2 156.4 -> 147.7).
    __global__ void learned_update_quad_kernel(const float* __restrict__ flux, const float* __restrict__ extra, int nrows,
                                               int ncols, float scale_y, float scale_x, int32_t* __restrict__ phi_q,
                                               float* __restrict__ phi_f, long long bound, int* __restrict__ flag,
                                               int64_t* __restrict__ advance, const float* __restrict__ params,
                                               uint4* __restrict__ x_next)
    {
        if (advance && blockIdx.x == 0 && threadIdx.x == 0) *advance += 1;
        const size_t plane = size_t(nrows) * ncols;
        const int quads = ncols / 4;
        const size_t n = size_t(nrows) * quads;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const auto load = [](const float* p, size_t i) { return *reinterpret_cast<const float4*>(p + i); };
        const auto face = [&](float f, float e, float scale) {
            const float q = __fmul_rn(scale, extra ? __fadd_rn(f, e) : f);
            return (long long)__float2int_rn(q > 1e9f ? 1e9f : (q < -1e9f ? -1e9f : q));
        };
        for (size_t t = blockIdx.x * size_t(blockDim.x) + threadIdx.x; t < n; t += size_t(gridDim.x) * blockDim.x)
        {
            const int r = int(t / quads), c = int(t - size_t(r) * quads) * 4;
            const size_t row = size_t(r) * ncols, up = size_t(r == 0 ? nrows - 1 : r - 1) * ncols;
            const size_t left = row + (c == 0 ? ncols - 1 : c - 1);
            const float4 fy = load(flux, row + c), fx = load(flux + plane, row + c), fu = load(flux, up + c);
            const float4 ey = extra ? load(extra, row + c) : zero, ex = extra ? load(extra + plane, row + c) : zero,
                         eu = extra ? load(extra, up + c) : zero;
            const float fl = flux[plane + left], el = extra ? extra[plane + left] : 0.f;
            const int4 q0 = *reinterpret_cast<const int4*>(phi_q + row + c);
            const float vy[4] = {fy.x, fy.y, fy.z, fy.w}, vx[4] = {fx.x, fx.y, fx.z, fx.w}, vu[4] = {fu.x, fu.y, fu.z, fu.w};
            const float wy[4] = {ey.x, ey.y, ey.z, ey.w}, wx[4] = {ex.x, ex.y, ex.z, ex.w}, wu[4] = {eu.x, eu.y, eu.z, eu.w};
            const int qs[4] = {q0.x, q0.y, q0.z, q0.w};
            long long before = face(fl, el, scale_x);
            int q[4];
            float f[4];
            bool bad = false;
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                const long long here = face(vx[k], wx[k], scale_x);
                const long long dq = here - before + face(vy[k], wy[k], scale_y) - face(vu[k], wu[k], scale_y);
                before = here;
                const bool finite = isfinite(vx[k]) && isfinite(vy[k]) && isfinite(wx[k]) && isfinite(wy[k]);
                q[k] = updated_q(qs[k], dq, finite, bound, &bad);
                f[k] = field_of(q[k]);
            }
            if (bad) atomicOr(flag, 1);
            *reinterpret_cast<int4*>(phi_q + row + c) = make_int4(q[0], q[1], q[2], q[3]);
            *reinterpret_cast<float4*>(phi_f + row + c) = make_float4(f[0], f[1], f[2], f[3]);
            if (x_next)
            {
                const float p0 = params[0], p1 = params[1], p2 = params[2];
#pragma unroll
                for (int k = 0; k < 4; ++k) x_next[row + c + k] = input_chunk(f[k], p0, p1, p2);
            }
        }
    }

    // out_c = phi_hat * m_c + noise_mag * xi_hat_c * n_c for c = y, x (complex rfft2 spectra,
    // [ny][nx/2+1] each; xi_hat may be null).
    __global__ void spectral_combine_kernel(const float2* __restrict__ phi_hat, const float2* __restrict__ xi_hat,
                                            const float2* __restrict__ my, const float2* __restrict__ mx,
                                            const float2* __restrict__ ny_, const float2* __restrict__ nx_,
                                            float noise_mag, size_t n, float2* __restrict__ out_y,
                                            float2* __restrict__ out_x)
    {
        for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        {
            const float2 p = phi_hat[i], a = my[i], b = mx[i];
            float2 y = make_float2(p.x * a.x - p.y * a.y, p.x * a.y + p.y * a.x);
            float2 x = make_float2(p.x * b.x - p.y * b.y, p.x * b.y + p.y * b.x);
            if (xi_hat)
            {
                const float2 u = xi_hat[i], v = xi_hat[n + i], c = ny_[i], d = nx_[i];
                y.x += noise_mag * (u.x * c.x - u.y * c.y);
                y.y += noise_mag * (u.x * c.y + u.y * c.x);
                x.x += noise_mag * (v.x * d.x - v.y * d.y);
                x.y += noise_mag * (v.x * d.y + v.y * d.x);
            }
            out_y[i] = y;
            out_x[i] = x;
        }
    }

    int g_sms = 0;
    std::once_flag g_sms_once;

    int sm_count()
    {
        std::call_once(g_sms_once, [] {
            int dev = 0;
            cudaGetDevice(&dev);
            if (cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || g_sms < 1)
                g_sms = 148;
        });
        return g_sms;
    }

    // Rows per CTA for the forward kernel: every CTA stages all its input rows at once, so
    // shared memory and TMEM per CTA grow with the rows (at most kMaxFwdRows); one CTA per
    // SM (320 threads at ~150 registers); cost = waves x (rows + about three row times of
    // pipeline fill).
    int choose_fwd_rows(int batch, int nrows, int nwin, int cc, int npad)
    {
        const int sms = sm_count();
        int best = 1;
        double best_cost = 1e30;
        for (int r = 1; r <= kMaxFwdRows && r <= nrows; ++r)
        {
            if (fwd_smem_bytes(cc, npad, r) > kSmemLimit || npad * r > 512) break;
            const long long grid = (long long)batch * nwin * ((nrows + r - 1) / r);
            const long long waves = (grid + sms - 1) / sms;
            const double cost = double(waves) * (r + 3);
            if (cost < best_cost - 1e-9)
            {
                best_cost = cost;
                best = r;
            }
        }
        return best;
    }

    // Raises a kernel's dynamic shared-memory limit once per device (so that later
    // launches, e.g. inside a stream capture, make no attribute calls).
    std::mutex g_attr_mutex;
    int g_attr_selftest[64], g_attr_fwd[4][64], g_attr_wgrad[4][64];

    cudaError_t set_smem_attr(const void* fn, uint32_t bytes, int (&done)[64])
    {
        std::lock_guard<std::mutex> lock(g_attr_mutex);
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
        if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = 1;
        return e;
    }

    bool valid_geometry(int batch, int nrows, int ncols)
    {
        return batch >= 1 && nrows >= 3 && ncols >= kTile && ncols % kTile == 0 &&
               (long long)batch * nrows * ncols < (1ll << 31);
    }

    int fail_invalid(const char* what)
    {
        amb::set_last_error(what);
        return AMB_ERR_INVALID;
    }

    int fail_cuda(const char* what, cudaError_t e)
    {
        amb::set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
        return AMB_ERR_CUDA;
    }
}

// ============================================================= C ABI

extern "C" int amb_tc_selftest(const void* a, const void* b, float* d, int n, int k, int a_mn_major, int b_mn_major,
                               int* error, void* stream)
{
    if (!a || !b || !d || (n != 16 && n != 32) || k < 16 || k > 64 || k % 16 != 0)
        return fail_invalid("amb_tc_selftest: n must be 16 or 32, k in {16, 32, 48, 64}");
    const uint32_t smem = 98304 + 256;
    cudaError_t e = set_smem_attr(reinterpret_cast<const void*>(tc_selftest_kernel), smem, g_attr_selftest);
    if (e == cudaSuccess)
    {
        tc_selftest_kernel<<<1, 128, smem, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const uint16_t*>(a), static_cast<const uint16_t*>(b), d, n, k, a_mn_major, b_mn_major, error);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_tc_selftest", e);
}

extern "C" int amb_conv5x5_forward(const void* in, int batch, int nrows, int ncols, int cin, const void* wimg,
                                   const float* bias, int npad, int cout, int epilogue, void* out, void* pre,
                                   const void* gate, float* out_f32, int* error, void* stream)
{
    if (!in || !wimg || !valid_geometry(batch, nrows, ncols) || (cin != 16 && cin != 32) ||
        (npad != 16 && npad != 32) || epilogue < 0 || epilogue > 2)
        return fail_invalid("amb_conv5x5_forward: need ncols % 128 == 0, nrows >= 3, cin and npad in {16, 32}");
    if (epilogue == EPI_F32 && (!out_f32 || cout < 1 || cout > npad))
        return fail_invalid("amb_conv5x5_forward: FP32 epilogue needs out_f32 and 1 <= cout <= npad");
    if (epilogue != EPI_F32 && !out) return fail_invalid("amb_conv5x5_forward: bf16 epilogue needs out");
    if (epilogue == EPI_GELU_BWD && !gate) return fail_invalid("amb_conv5x5_forward: GELU' epilogue needs gate");
    const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!al16(in) || !al16(wimg) || (out && !al16(out)) || (pre && !al16(pre)) || (gate && !al16(gate)))
        return fail_invalid("amb_conv5x5_forward: bf16 buffers must be 16-byte aligned");

    FwdArgs a{};
    a.in = static_cast<const uint16_t*>(in);
    a.wimg = static_cast<const uint16_t*>(wimg);
    a.bias = bias;
    a.out = static_cast<uint16_t*>(out);
    a.pre = static_cast<uint16_t*>(pre);
    a.gate = static_cast<const uint16_t*>(gate);
    a.out_f32 = out_f32;
    a.batch = batch;
    a.nrows = nrows;
    a.ncols = ncols;
    a.cin_chunks = cin / 8;
    a.npad = npad;
    a.cout = epilogue == EPI_F32 ? cout : npad;
    a.epilogue = epilogue;
    const int nwin = ncols / kTile;
    a.rows_per_cta = choose_fwd_rows(batch, nrows, nwin, a.cin_chunks, npad);
    a.error = error;
    const uint32_t smem = fwd_smem_bytes(a.cin_chunks, npad, a.rows_per_cta);
    const int which = (a.cin_chunks == 4 ? 0 : 2) + (npad == 32 ? 0 : 1);
    using Kernel = void (*)(FwdArgs);
    constexpr Kernel kernels[4] = {conv_fwd_kernel<4, 32>, conv_fwd_kernel<4, 16>, conv_fwd_kernel<2, 32>,
                                   conv_fwd_kernel<2, 16>};
    const Kernel kern = kernels[which];
    cudaError_t e = set_smem_attr(reinterpret_cast<const void*>(kern), kSmemLimit, g_attr_fwd[which]);
    if (e == cudaSuccess)
    {
        const long long grid = (long long)batch * nwin * ((nrows + a.rows_per_cta - 1) / a.rows_per_cta);
        kern<<<unsigned(grid), kFwdThreads, smem, static_cast<cudaStream_t>(stream)>>>(a);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_conv5x5_forward", e);
}

namespace
{
    struct WgradPlan
    {
        int first[6] = {};
        int groups = 0, kpc = 0, part = 0;
        size_t bytes(int npad) const { return (size_t(first[groups]) * part + size_t(first[1]) * npad) * sizeof(float); }
    };

    // CTAs per x-tap group in proportion to its taps, one CTA per SM, no more than there are row blocks.
    template <int CC, int NPAD>
    WgradPlan wgrad_plan_of(int batch, int nrows, int ncols)
    {
        using G = Wg<CC, NPAD>;
        WgradPlan p;
        p.groups = G::GROUPS;
        p.kpc = G::KPC;
        p.part = G::PART;
        const long long blocks = (long long)batch * (ncols / kTile) * ((nrows + G::XR - 1) / G::XR);
        for (int g = 0; g < G::GROUPS; ++g)
        {
            const int taps = std::min(G::KPC, 5 - g * G::KPC);
            p.first[g + 1] = p.first[g] + int(std::min<long long>(blocks, std::max(1, sm_count() * taps / 5)));
        }
        for (int g = G::GROUPS; g < 5; ++g) p.first[g + 1] = p.first[g];
        return p;
    }

    WgradPlan wgrad_plan(int batch, int nrows, int ncols, int cin, int npad)
    {
        if (cin == 32) return npad == 32 ? wgrad_plan_of<4, 32>(batch, nrows, ncols) : wgrad_plan_of<4, 16>(batch, nrows, ncols);
        return npad == 32 ? wgrad_plan_of<2, 32>(batch, nrows, ncols) : wgrad_plan_of<2, 16>(batch, nrows, ncols);
    }

    template <int CC, int NPAD>
    cudaError_t launch_wgrad(const WgradArgs& a, int grid, int (&attr)[64], cudaStream_t s)
    {
        auto kern = conv_wgrad_kernel<CC, NPAD>;
        cudaError_t e = set_smem_attr(reinterpret_cast<const void*>(kern), Wg<CC, NPAD>::SMEM, attr);
        if (e != cudaSuccess) return e;
        kern<<<grid, kThreads, Wg<CC, NPAD>::SMEM, s>>>(a);
        return cudaGetLastError();
    }

    int param_grads(const char* name, const void* x, const void* dz, int batch, int nrows, int ncols, int cin, int npad,
                    int cin_used, int cout, float* dw, float* gw, float* gb, float* scratch, size_t scratch_bytes,
                    int* error, void* stream)
    {
        if (!x || !dz || !scratch || !valid_geometry(batch, nrows, ncols) || (cin != 16 && cin != 32) ||
            (npad != 16 && npad != 32) || cin_used < 1 || cin_used > cin || cout < 1 || cout > npad)
            return fail_invalid("weight gradient: need ncols % 128 == 0, nrows >= 3, cin and npad in {16, 32}");
        const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
        if (!al16(x) || !al16(dz) || !al16(scratch))
            return fail_invalid("weight gradient: x, dz and scratch must be 16-byte aligned");
        const WgradPlan plan = wgrad_plan(batch, nrows, ncols, cin, npad);
        if (scratch_bytes < plan.bytes(npad))
            return fail_invalid("weight gradient: scratch too small (see amb_conv5x5_wgrad_scratch_bytes)");
        WgradArgs a{};
        a.x = static_cast<const uint16_t*>(x);
        a.dz = static_cast<const uint16_t*>(dz);
        a.partial = scratch;
        a.bias = gb ? scratch + size_t(plan.first[plan.groups]) * plan.part : nullptr;
        a.batch = batch;
        a.nrows = nrows;
        a.ncols = ncols;
        std::copy(plan.first, plan.first + 6, a.first);
        a.error = error;
        auto s = static_cast<cudaStream_t>(stream);
        const int grid = plan.first[plan.groups];
        cudaError_t e = cin == 32 ? (npad == 32 ? launch_wgrad<4, 32>(a, grid, g_attr_wgrad[0], s)
                                                : launch_wgrad<4, 16>(a, grid, g_attr_wgrad[1], s))
                                  : (npad == 32 ? launch_wgrad<2, 32>(a, grid, g_attr_wgrad[2], s)
                                                : launch_wgrad<2, 16>(a, grid, g_attr_wgrad[3], s));
        if (e == cudaSuccess)
        {
            WgradReduceArgs r{};
            r.partial = a.partial;
            r.bias_partial = a.bias;
            std::copy(plan.first, plan.first + 6, r.first);
            r.kpc = plan.kpc;
            r.cin = cin;
            r.npad = npad;
            r.dw = dw;
            r.gw = gw;
            r.gb = gb;
            r.cout = cout;
            r.cin_used = cin_used;
            const int total = 25 * cin * npad / 4;
            wgrad_reduce_kernel<<<(total + 31) / 32 + (gb ? 1 : 0), 256, 0, s>>>(r);
            e = cudaGetLastError();
        }
        return e == cudaSuccess ? AMB_OK : fail_cuda(name, e);
    }
}

extern "C" size_t amb_conv5x5_wgrad_scratch_bytes(int batch, int nrows, int ncols, int cin, int npad)
{
    if (!valid_geometry(batch, nrows, ncols)) return 0;
    return wgrad_plan(batch, nrows, ncols, cin, npad).bytes(npad);
}

extern "C" int amb_conv5x5_wgrad(const void* x, const void* dz, int batch, int nrows, int ncols, int cin, int npad,
                                 float* dw, float* scratch, size_t scratch_bytes, int* error, void* stream)
{
    if (!dw) return fail_invalid("amb_conv5x5_wgrad: dw must not be NULL");
    return param_grads("amb_conv5x5_wgrad", x, dz, batch, nrows, ncols, cin, npad, cin, npad, dw, nullptr, nullptr,
                       scratch, scratch_bytes, error, stream);
}

extern "C" int amb_conv5x5_param_grads(const void* x, const void* dz, int batch, int nrows, int ncols, int cin, int npad,
                                       int cin_used, int cout, float* gw, float* gb, float* scratch, size_t scratch_bytes,
                                       int* error, void* stream)
{
    if (!gw) return fail_invalid("amb_conv5x5_param_grads: gw must not be NULL");
    return param_grads("amb_conv5x5_param_grads", x, dz, batch, nrows, ncols, cin, npad, cin_used, cout, nullptr, gw, gb,
                       scratch, scratch_bytes, error, stream);
}

extern "C" int amb_conv5x5_stack_images(int layers, const float* const* w, const int* cout, const int* cin,
                                        const int* cin_pad, const int* npad, void* const* img, void* const* dimg,
                                        void* stream)
{
    if (layers < 1 || !w || !cout || !cin || !cin_pad || !npad || !img || !dimg)
        return fail_invalid("amb_conv5x5_images: bad arguments");
    cudaError_t e = cudaSuccess;
    for (int l0 = 0; l0 < layers && e == cudaSuccess; l0 += kImageLayers)
    {
        ImageArgs a{};
        const int count = std::min(kImageLayers, layers - l0);
        int most = 0;
        for (int i = 0; i < count; ++i)
        {
            const int l = l0 + i;
            if (!w[l] || (!img[l] && !dimg[l]) || cin[l] < 1 || cout[l] < 1 || cin[l] > cin_pad[l] || cout[l] > npad[l] ||
                cin_pad[l] % 8 || npad[l] % 8)
                return fail_invalid("amb_conv5x5_images: bad arguments");
            a.layer[i] = {w[l], static_cast<__nv_bfloat16*>(img[l]), static_cast<__nv_bfloat16*>(dimg[l]), cout[l], cin[l],
                          cin_pad[l], npad[l]};
            most = std::max(most, 2 * 25 * cin_pad[l] * npad[l]);
        }
        weight_images_kernel<<<dim3((most + 255) / 256, count), 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_conv5x5_images", e);
}

extern "C" int amb_conv5x5_images(const float* w, int cout, int cin, int cin_pad, int npad, void* img, void* dimg,
                                  void* stream)
{
    return amb_conv5x5_stack_images(1, &w, &cout, &cin, &cin_pad, &npad, &img, &dimg, stream);
}

extern "C" int amb_conv5x5_stack_forward(const void* in, int batch, int nrows, int ncols, int layers, const int* cin,
                                         const int* npad, int cout, const void* const* wimg, const float* const* bias,
                                         void* const* out, void* const* pre, float* out_f32, int* error, void* stream)
{
    if (layers < 1 || !cin || !npad || !wimg || !bias || !out || !pre)
        return fail_invalid("amb_conv5x5_stack_forward: bad arguments");
    for (int l = 0; l < layers; ++l)
    {
        if (l && cin[l] != npad[l - 1])
            return fail_invalid("amb_conv5x5_stack_forward: each layer's cin must be the npad before it");
        const bool last = l == layers - 1;
        const int rc = amb_conv5x5_forward(l ? out[l - 1] : in, batch, nrows, ncols, cin[l], wimg[l], bias[l], npad[l],
                                           last ? cout : npad[l], last ? EPI_F32 : EPI_GELU, last ? nullptr : out[l],
                                           last ? nullptr : pre[l], nullptr, last ? out_f32 : nullptr, error, stream);
        if (rc != AMB_OK) return rc;
    }
    return AMB_OK;
}

extern "C" int amb_conv5x5_stack_backward(const float* dout, int batch, int nrows, int ncols, int layers, const int* cin,
                                          const int* cin_used, const int* npad, const int* cout, const void* const* x,
                                          const void* const* pre, const void* const* dimg, void* dz0, void* dz1,
                                          float* const* gw, float* const* gb, float* scratch, size_t scratch_bytes,
                                          int* error, void* stream)
{
    if (!dout || layers < 1 || !cin || !cin_used || !npad || !cout || !x || !pre || !dimg || !dz0 || (layers > 1 && !dz1) ||
        !gw || !gb || !valid_geometry(batch, nrows, ncols) || (npad[layers - 1] != 16 && npad[layers - 1] != 32) ||
        cout[layers - 1] < 1 || cout[layers - 1] > npad[layers - 1] || (reinterpret_cast<uintptr_t>(dz0) & 15))
        return fail_invalid("amb_conv5x5_stack_backward: bad arguments");
    const size_t plane = size_t(nrows) * ncols, n = plane * batch * (npad[layers - 1] / 8);
    const int grid = int(std::min<size_t>((n + 255) / 256, size_t(sm_count()) * 16));
    chunk_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(dout, cout[layers - 1], npad[layers - 1], plane, n,
                                                                      static_cast<uint4*>(dz0));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail_cuda("amb_conv5x5_stack_backward", e);
    void *dz = dz0, *prev = dz1;
    for (int l = layers - 1; l >= 0; --l)
    {
        int rc = amb_conv5x5_param_grads(x[l], dz, batch, nrows, ncols, cin[l], npad[l], cin_used[l], cout[l], gw[l], gb[l],
                                         scratch, scratch_bytes, error, stream);
        if (rc == AMB_OK && l > 0)
            rc = amb_conv5x5_forward(dz, batch, nrows, ncols, npad[l], dimg[l], nullptr, cin[l], cin[l], EPI_GELU_BWD, prev,
                                     nullptr, pre[l - 1], nullptr, error, stream);
        if (rc != AMB_OK) return rc;
        std::swap(dz, prev);
    }
    return AMB_OK;
}

extern "C" int amb_learned_input(const float* phi, const float* params, int batch, int nrows, int ncols, void* x,
                                 void* stream)
{
    if (!phi || !params || !x || !valid_geometry(batch, nrows, ncols))
        return fail_invalid("amb_learned_input: bad arguments");
    const size_t n = size_t(batch) * nrows * ncols;
    const int grid = int(std::min<size_t>((n + 255) / 256, size_t(sm_count()) * 16));
    learned_input_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(phi, params, batch, nrows, ncols,
                                                                            static_cast<uint16_t*>(x));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_learned_input", e);
}

extern "C" int amb_learned_noise(int nrows, int ncols, uint64_t seed, const int64_t* step, float* xi, void* stream)
{
    if (!step || !xi || nrows < 1 || ncols < 1) return fail_invalid("amb_learned_noise: bad arguments");
    const size_t n = size_t(nrows) * ncols;
    const int grid = int(std::min<size_t>((n + 255) / 256, size_t(sm_count()) * 16));
    learned_noise_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(xi, nrows, ncols, seed, step);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_learned_noise", e);
}

static int learned_update_launch(const float* flux, const float* extra, int nrows, int ncols, double dt_macro,
                                 double dx, double dy, const float* xi, double noise_mag, int32_t* phi_q, float* phi_f,
                                 double bound, int* flag, int64_t* step_to_advance, const float* params, void* x_next,
                                 void* stream)
{
    auto s = static_cast<cudaStream_t>(stream);
    const dim3 grid((ncols + 255) / 256, std::min(nrows, 65535));
    const double fix = 16777216.0;
    const double qb = std::min(bound * fix, 2.0e9);
    const bool noisy = xi && noise_mag > 0;
    const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!noisy && ncols % 4 == 0 && al16(flux) && al16(extra) && al16(phi_q) && al16(phi_f))
    {
        const size_t quads = size_t(nrows) * (ncols / 4);
        const int blocks = int(std::min<size_t>((quads + 127) / 128, size_t(sm_count()) * 16));
        learned_update_quad_kernel<<<blocks, 128, 0, s>>>(flux, extra, nrows, ncols, float(dt_macro / dy * fix),
                                                          float(dt_macro / dx * fix), phi_q, phi_f, (long long)qb, flag,
                                                          step_to_advance, params, static_cast<uint4*>(x_next));
    }
    else
        learned_update_kernel<<<grid, 256, 0, s>>>(flux, extra, noisy ? xi : nullptr, nrows, ncols,
                                               float(dt_macro / dy * fix), float(dt_macro / dx * fix),
                                               noisy ? float(noise_mag) : 0.f, phi_q, phi_f, (long long)qb, flag,
                                               step_to_advance, params, static_cast<uint4*>(x_next));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_learned_update", e);
}

static bool learned_update_args_ok(const float* flux, const int32_t* phi_q, const float* phi_f, const int* flag,
                                   int nrows, int ncols, double dt_macro, double dx, double dy, double noise_mag,
                                   double bound)
{
    return flux && phi_q && phi_f && flag && nrows >= 1 && ncols >= 1 && dt_macro > 0 && dx > 0 && dy > 0 &&
           noise_mag >= 0 && bound > 0;
}

extern "C" int amb_learned_update(const float* flux, const float* extra, int nrows, int ncols, double dt_macro,
                                  double dx, double dy, const float* xi, double noise_mag, int32_t* phi_q,
                                  float* phi_f, double bound, int* flag, int64_t* step_to_advance, void* stream)
{
    if (!learned_update_args_ok(flux, phi_q, phi_f, flag, nrows, ncols, dt_macro, dx, dy, noise_mag, bound))
        return fail_invalid("amb_learned_update: bad arguments");
    return learned_update_launch(flux, extra, nrows, ncols, dt_macro, dx, dy, xi, noise_mag, phi_q, phi_f, bound,
                                 flag, step_to_advance, nullptr, nullptr, stream);
}

extern "C" int amb_learned_update_input(const float* flux, const float* extra, int nrows, int ncols, double dt_macro,
                                        double dx, double dy, const float* xi, double noise_mag, int32_t* phi_q,
                                        float* phi_f, double bound, int* flag, int64_t* step_to_advance,
                                        const float* params, void* x_next, void* stream)
{
    if (!learned_update_args_ok(flux, phi_q, phi_f, flag, nrows, ncols, dt_macro, dx, dy, noise_mag, bound) ||
        !params || !x_next || (reinterpret_cast<uintptr_t>(x_next) & 15) != 0)
        return fail_invalid("amb_learned_update_input: bad arguments");
    return learned_update_launch(flux, extra, nrows, ncols, dt_macro, dx, dy, xi, noise_mag, phi_q, phi_f, bound,
                                 flag, step_to_advance, params, x_next, stream);
}

extern "C" int amb_learned_spectral_combine(const void* phi_hat, const void* xi_hat, const void* my, const void* mx,
                                            const void* ny, const void* nx, double noise_mag, int64_t n,
                                            void* out_y, void* out_x, void* stream)
{
    if (!phi_hat || !my || !mx || !out_y || !out_x || n < 1 || (xi_hat && (!ny || !nx)))
        return fail_invalid("amb_learned_spectral_combine: bad arguments");
    const int grid = int(std::min<int64_t>((n + 255) / 256, int64_t(sm_count()) * 8));
    spectral_combine_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const float2*>(phi_hat), static_cast<const float2*>(xi_hat), static_cast<const float2*>(my),
        static_cast<const float2*>(mx), static_cast<const float2*>(ny), static_cast<const float2*>(nx),
        float(noise_mag), size_t(n), static_cast<float2*>(out_y), static_cast<float2*>(out_x));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_learned_spectral_combine", e);
}

extern "C" int amb_learned_noise_spectral(int nrows, int ncols, uint64_t seed, const int64_t* step, void* out,
                                          int64_t row_stride, int64_t col_stride, void* stream)
{
    if (!step || !out || nrows < 1 || ncols < 2 || row_stride < 1 || col_stride < 1)
        return fail_invalid("amb_learned_noise_spectral: bad arguments");
    const int64_t n = int64_t(nrows) * (ncols / 2 + 1);
    const int grid = int(std::min<int64_t>((n + 255) / 256, int64_t(sm_count()) * 8));
    learned_noise_spectral_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<float2*>(out), nrows, ncols, row_stride, col_stride, n, seed ^ 0x5bd1e995a5a5a5a5ull, step);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_learned_noise_spectral", e);
}

extern "C" int amb_learned_spectral_combine_noise(const void* phi_hat, const void* my, const void* mx, const void* ny,
                                                  const void* nx, double noise_mag, int nrows, int ncols,
                                                  int64_t row_stride, int64_t col_stride, uint64_t seed,
                                                  const int64_t* step, void* out_y, void* out_x, void* stream)
{
    const int64_t nk = ncols / 2 + 1;
    const bool row_major = col_stride == 1 && row_stride == nk;
    const bool col_major = row_stride == 1 && col_stride == nrows;
    if (!phi_hat || !my || !mx || !ny || !nx || !step || !out_y || !out_x || nrows < 1 || ncols < 2 ||
        !(row_major || col_major))
        return fail_invalid("amb_learned_spectral_combine_noise: bad arguments (spectra must be dense)");
    const int64_t n = int64_t(nrows) * nk;
    const int grid = int(std::min<int64_t>((n + 255) / 256, int64_t(sm_count()) * 8));
    spectral_combine_noise_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const float2*>(phi_hat), static_cast<const float2*>(my), static_cast<const float2*>(mx),
        static_cast<const float2*>(ny), static_cast<const float2*>(nx), float(noise_mag), nrows, ncols, row_stride,
        col_stride, seed ^ 0x5bd1e995a5a5a5a5ull, step, static_cast<float2*>(out_y), static_cast<float2*>(out_x));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AMB_OK : fail_cuda("amb_learned_spectral_combine_noise", e);
}
