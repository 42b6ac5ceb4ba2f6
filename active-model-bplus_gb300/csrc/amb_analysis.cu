// Field analysis on the device: radial binning of a power spectrum (structure
// factor S(k)) and periodic connected-component labelling (droplet count).
//
// S(k) follows the reference's analysis notebook (examples/structureFactor.ipynb,
// cells 5-7): phi_q = FFT2(phi - phi0) dx dy, |phi_q|^2 averaged over the modes whose
// |k| falls in each bin, bins given by np.digitize(|k|, edges, right=True), i.e.
// bin l holds edges[l-1] < |k| <= edges[l]. The FFT itself is a library call made
// by the caller (cuFFT through torch.fft); this file does the binning.
//
// Droplets: 4-connected components of {phi > threshold} on the periodic grid, by
// union-find with atomic hooking of the larger root onto the smaller (a standard
// GPU connected-components scheme): first inside tiles of 16 x 64 sites in shared memory,
// then across the tiles' borders, then full path compression. Labels are the
// smallest linear index in each component; background sites get -1.
#include "amb_gb300.h"
#include "amb_kernels.h"

#include <cuda_runtime.h>

namespace
{
    constexpr int kBinRows = 4;        // rows a warp walks down its columns: few, so that 1024^2 fills the SMs
    constexpr int kBinEdges = 2048;    // most edges binned in shared memory

    // The exact bin of k: l with edges[l-1] < k <= edges[l] (np.digitize right=True; nedges if beyond), from
    // a guess a few bins away.
    __device__ __forceinline__ int exact_bin(double k, const double* __restrict__ edges, int nedges, int l)
    {
        while (l < nedges && edges[l] < k) ++l;
        while (l > 0 && !(edges[l - 1] < k)) --l;
        return l;
    }

    // The same by halving.
    template <typename Real>
    __device__ __forceinline__ int find_bin(Real k, const Real* __restrict__ edges, int nedges)
    {
        int l = 0;
        for (int hi = nedges; l < hi;)
        {
            const int mid = (l + hi) >> 1;
            if (edges[mid] < k) l = mid + 1;
            else hi = mid;
        }
        return l;
    }

    // What the binning kernel reads, with element strides rs, cs:
    // POWER   a full power spectrum [ny][nx];
    // HALF    an rfft2 spectrum [ny][nx/2 + 1]: |scale z|^2, the mirrored half counted through a weight of
    //         two (|k| of a mode and its mirror are the same bits);
    // PACKED  (ny even) the complex transform Z [ny/2][nx] of the field's even rows + i odd rows, half the
    //         work of a real transform of the field: with E, O the transforms of the even and odd
    //         rows, E = (Z(k) + conj Z(-k)) / 2 and O = (Z(k) - conj Z(-k)) / 2i, the field's modes are
    //         E + w O at row k and E - w O at row k + ny/2, w = exp(-2 pi i k / ny).
    enum Spectrum { POWER, HALF, PACKED };
    //
    // A warp takes 32 columns and walks down rows. Along a row |k| is monotonic, so the lanes of a bin are
    // neighbours: each run is summed by shuffles and its last lane adds it to the block's shared histogram
    // (lanes adding by themselves queue up on one address: 44 us). From row to row a lane's bin moves by
    // steps; it is found in FP32, whose error is below 2e-7 k, and within 1e-6 k of an edge decided in FP64
    // as the definition has it, so the FP64 pipe (64 cycles per warp instruction) sees one square root
    // per thousand modes instead of a square root, the products of |k| and nine comparisons for each.
    // 1024^2: 35 us, the packed transform's unpacking included, on top of 87 us for the transform (one
    // thread and two global atomics per mode, all in FP64: 94 us, after 172 us of complex transform
    // and 28 us of elementwise passes).
    // Past kBinEdges edges each mode's bin is found by halving in FP64: at 1024^2 a call takes 350 us with 2100
    // edges, 359 with 4096, 615 with 100000 (walking there from the first edge: 804, 1271, 23500).
    template <Spectrum MODE>
    __global__ void __launch_bounds__(256)
    radial_bin_kernel(const double* __restrict__ in, int ny, int nx, int64_t rs, int64_t cs, double scale, double dx,
                      double dy, const double* __restrict__ edges, int nedges, bool shared, double* __restrict__ sum,
                      unsigned long long* __restrict__ count)
    {
        extern __shared__ __align__(16) unsigned char raw[];
        double* hs = reinterpret_cast<double*>(raw);
        unsigned* hc = reinterpret_cast<unsigned*>(hs + (shared ? nedges : 0));
        float* ef = reinterpret_cast<float*>(hc + (shared ? nedges : 0));
        constexpr int SUB = MODE == PACKED ? 2 : 1;  // modes a lane forms per row
        __shared__ double ky2s[8][SUB][kBinRows];
        __shared__ float ky2f[8][SUB][kBinRows];
        __shared__ double2 tw[8][kBinRows];
        if (shared)
            for (int l = threadIdx.x; l < nedges; l += 256)
            {
                hs[l] = 0;
                hc[l] = 0;
                ef[l] = float(edges[l]);
            }
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int cols = MODE == POWER ? nx : nx / 2 + 1, nrows = ny / SUB, across = (cols + 31) / 32;
        const long long task = (long long)blockIdx.x * 8 + warp;
        const int c = int(task % across) * 32 + lane;
        const long long row0 = task / across * kBinRows;
        // 2 pi f / (n d) of a frequency index in numpy's fftfreq order, squared
        const auto k2 = [](int i, int n, double d) {
            const double k = 6.283185307179586 * (double(i < (n + 1) / 2 ? i : i - n) * (1.0 / (double(n) * d)));
            return k * k;
        };
        if (lane < kBinRows && row0 + lane < nrows)
        {
            const int r = int(row0) + lane;
            for (int h = 0; h < SUB; ++h)
            {
                ky2s[warp][h][lane] = k2(r + h * nrows, ny, dy);
                ky2f[warp][h][lane] = float(ky2s[warp][h][lane]);
            }
            if constexpr (MODE == PACKED) sincospi(-2.0 * r / ny, &tw[warp][lane].y, &tw[warp][lane].x);
        }
        __syncthreads();
        if (row0 < nrows)
        {
            const bool act = c < cols;
            const double kx2 = k2(act ? c : 0, nx, dx);
            const float kx2f = float(kx2);
            const unsigned ones = __ballot_sync(0xffffffffu, MODE == POWER || c == 0 || 2 * c == nx);  // weight one
            const bool twice = !((ones >> lane) & 1);
            const int rows = min(kBinRows, int(nrows - row0));
            int bins[SUB];
#pragma unroll
            for (int h = 0; h < SUB; ++h) bins[h] = -1;
            for (int i = 0; i < rows; ++i)
            {
                double vs[SUB];
                if constexpr (MODE == PACKED)
                {
                    const int r = int(row0) + i, rm = r == 0 ? 0 : nrows - r, cm = c == 0 ? 0 : nx - c;
                    double2 z = make_double2(0, 0), m = z;
                    if (act)
                    {
                        z = *reinterpret_cast<const double2*>(in + 2 * (r * rs + c * cs));
                        m = *reinterpret_cast<const double2*>(in + 2 * (rm * rs + cm * cs));
                    }
                    const double ex = z.x + m.x, ey = z.y - m.y, ox = z.y + m.y, oy = m.x - z.x;  // 2 E, 2 O
                    const double2 w = tw[warp][i];
                    const double px = w.x * ox - w.y * oy, py = w.x * oy + w.y * ox;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                    {
                        const double re = (h ? ex - px : ex + px) * (0.5 * scale), im = (h ? ey - py : ey + py) * (0.5 * scale);
                        vs[h] = re * re + im * im;
                    }
                }
                else if constexpr (MODE == HALF)
                {
                    vs[0] = 0;
                    if (act)
                    {
                        const double2 z = *reinterpret_cast<const double2*>(in + 2 * ((row0 + i) * rs + c * cs));
                        const double re = z.x * scale, im = z.y * scale;
                        vs[0] = re * re + im * im;
                    }
                }
                else
                    vs[0] = act ? in[(row0 + i) * rs + c * cs] : 0;
#pragma unroll
                for (int h = 0; h < SUB; ++h)
                {
                    double v = act ? (twice ? vs[h] + vs[h] : vs[h]) : 0;
                    int l = bins[h];
                    if (act)
                    {
                        const float k = sqrtf(kx2f + ky2f[warp][h][i]);
                        if (shared && k > 1e-18f && k < 1e18f)
                        {
                            if (l < 0) l = find_bin(k, ef, nedges);
                            else
                            {
                                while (l < nedges && ef[l] < k) ++l;
                                while (l > 0 && !(ef[l - 1] < k)) --l;
                            }
                            const float tol = 1e-6f * k;
                            if ((l < nedges && !(fabsf(ef[l] - k) > tol)) || (l > 0 && !(fabsf(ef[l - 1] - k) > tol)))
                                l = exact_bin(sqrt(kx2 + ky2s[warp][h][i]), edges, nedges, l);
                        }
                        else  // more edges than shared memory takes, or out of FP32's range
                            l = find_bin(sqrt(kx2 + ky2s[warp][h][i]), edges, nedges);
                        bins[h] = l;
                    }
                    const int bin = act ? l : -1;
                    const int before = __shfl_up_sync(0xffffffffu, bin, 1);
                    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || before != bin);
                    const int head = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
#pragma unroll
                    for (int d = 1; d < 32; d *= 2)
                    {
                        const double up = __shfl_up_sync(0xffffffffu, v, d);
                        if (lane - d >= head) v += up;
                    }
                    const bool last = lane == 31 || ((heads >> (lane + 1)) & 1);
                    if (act && last && bin < nedges)
                    {
                        const unsigned run = (0xffffffffu >> (31 - lane)) & (0xffffffffu << head);
                        const unsigned n = 2 * __popc(run) - __popc(run & ones);
                        if (shared)
                        {
                            atomicAdd(&hs[bin], v);
                            atomicAdd(&hc[bin], n);
                        }
                        else
                        {
                            atomicAdd(&sum[bin], v);
                            atomicAdd(&count[bin], (unsigned long long)n);
                        }
                    }
                }
            }
        }
        if (!shared) return;
        __syncthreads();
        for (int l = threadIdx.x; l < nedges; l += 256)
            if (hc[l])
            {
                atomicAdd(&sum[l], hs[l]);
                atomicAdd(&count[l], (unsigned long long)hc[l]);
            }
    }

    // ----------------------------------------------------------- components

    __device__ __forceinline__ int find_root(const int* __restrict__ parent, int i)
    {
        while (true)
        {
            int p = parent[i];
            if (p == i) return i;
            i = p;
        }
    }

    // Union of two foreground roots: hook the larger index under the smaller with atomicCAS
    // (retry while another thread moved the root).
    __device__ void unite(int* parent, int a, int b)
    {
        while (true)
        {
            a = find_root(parent, a);
            b = find_root(parent, b);
            if (a == b) return;
            if (a > b)
            {
                int t = a;
                a = b;
                b = t;
            }
            int old = atomicCAS(&parent[b], b, a);
            if (old == b) return;
            b = old;
        }
    }

    // One thread per site of a block's tile. 1024^2: tiles 14, borders 6, compression 5 us (unions of all
    // neighbours in global memory: 62, with 11 for a compression that counted by one atomic per root).
    constexpr int kTileC = 64, kTileR = 16;

    // Components inside each tile by union-find in shared memory; parent gets the global index of the
    // tile component's smallest site (tile order and global order agree), -1 for background.
    template <typename Real>
    __global__ void __launch_bounds__(kTileC * kTileR)
    ccl_tiles(const Real* __restrict__ f, int ny, int nx, int tiles_x, double threshold, int* __restrict__ parent)
    {
        __shared__ int local[kTileC * kTileR];
        const int t = threadIdx.x, lr = t / kTileC, lc = t % kTileC;
        const int r0 = int(blockIdx.x) / tiles_x * kTileR, c0 = int(blockIdx.x) % tiles_x * kTileC;
        const int r = r0 + lr, c = c0 + lc;
        const bool inside = r < ny && c < nx;
        const bool fg = inside && double(f[size_t(r) * nx + c]) > threshold;
        local[t] = fg ? t : -1;
        __syncthreads();
        // runs along the row first: the leftmost site of the run, from the warp's ballot
        const unsigned ballot = __ballot_sync(0xffffffffu, fg);
        const int lane = t & 31;
        if (fg)
        {
            const unsigned gaps = ~ballot & ((1u << lane) - 1);  // background to the left in the warp
            local[t] = t - lane + (gaps ? 32 - __clz(gaps) : 0);
        }
        __syncthreads();
        if (fg && lane == 0 && lc > 0 && local[t - 1] >= 0) unite(local, t - 1, t);  // across the warp's boundary
        // one union per run that starts above: where the pair to the left is not joined already
        if (fg && lr > 0 && local[t - kTileC] >= 0 && !(lane > 0 && local[t - 1] >= 0 && local[t - kTileC - 1] >= 0))
            unite(local, t - kTileC, t);
        __syncthreads();
        if (inside)
        {
            int g = -1;
            if (fg)
            {
                const int root = find_root(local, t);
                g = (r0 + root / kTileC) * nx + c0 + root % kTileC;
            }
            parent[size_t(r) * nx + c] = g;
        }
    }

    // Unions across the tiles' left and upper borders (with the periodic neighbours).
    __global__ void ccl_borders(int ny, int nx, int tiles_x, int tiles_y, int* parent)
    {
        const int nv = tiles_x * ny, nh = tiles_y * nx;
        for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nv + nh; e += gridDim.x * blockDim.x)
        {
            int i, j;
            if (e < nv)
            {
                const int r = e / tiles_x, c = (e - r * tiles_x) * kTileC;
                i = r * nx + c;
                j = r * nx + (c == 0 ? nx - 1 : c - 1);
            }
            else
            {
                const int tr = (e - nv) / nx, c = e - nv - tr * nx, r = tr * kTileR;
                i = r * nx + c;
                j = (r == 0 ? ny - 1 : r - 1) * nx + c;
            }
            if (parent[i] >= 0 && parent[j] >= 0) unite(parent, i, j);
        }
    }

    // Every site's root, and the number of roots (one atomic per warp).
    __global__ void ccl_compress(int n, int* parent, int* __restrict__ ncomp)
    {
        int roots = 0;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        {
            if (parent[i] < 0) continue;
            int root = find_root(parent, i);
            if (root == i) ++roots;
            parent[i] = root;
        }
        roots = __reduce_add_sync(0xffffffffu, roots);
        if ((threadIdx.x & 31) == 0 && roots) atomicAdd(ncomp, roots);
    }

    int grid_for(size_t n)
    {
        size_t g = (n + 255) / 256;
        return int(g > 152 * 16 ? 152 * 16 : (g == 0 ? 1 : g));
    }
}

namespace
{
    template <Spectrum MODE>
    int radial(const char* name, const double* in, int ny, int nx, int64_t rs, int64_t cs, double scale, double dx,
               double dy, const double* edges, int nedges, double* sum, unsigned long long* count, cudaStream_t s)
    {
        cudaError_t e = cudaMemsetAsync(sum, 0, sizeof(double) * nedges, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, sizeof(unsigned long long) * nedges, s);
        if (e == cudaSuccess)
        {
            const int across = ((MODE == POWER ? nx : nx / 2 + 1) + 31) / 32, rows = MODE == PACKED ? ny / 2 : ny;
            const long long tasks = (long long)across * ((rows + kBinRows - 1) / kBinRows);
            const bool shared = nedges <= kBinEdges;
            const size_t smem = shared ? size_t(nedges) * 16 : 0;
            radial_bin_kernel<MODE><<<unsigned((tasks + 7) / 8), 256, smem, s>>>(in, ny, nx, rs, cs, scale, dx, dy, edges,
                                                                              nedges, shared, sum, count);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) return AMB_OK;
        amb::set_last_error(std::string(name) + ": " + cudaGetErrorString(e));
        return AMB_ERR_CUDA;
    }
}

extern "C" int amb_radial_spectrum(const double* power, int nrows, int ncols, double dx, double dy,
                                   const double* edges, int nedges, double* sum, unsigned long long* count,
                                   void* stream)
{
    if (!power || !edges || !sum || !count || nrows < 1 || ncols < 1 || nedges < 1 || !(dx > 0) || !(dy > 0))
    {
        amb::set_last_error("amb_radial_spectrum: bad arguments");
        return AMB_ERR_INVALID;
    }
    return radial<POWER>("amb_radial_spectrum", power, nrows, ncols, ncols, 1, 1.0, dx, dy, edges, nedges, sum, count,
                         static_cast<cudaStream_t>(stream));
}

extern "C" int amb_radial_rfft(const void* spectrum, int nrows, int ncols, int64_t row_stride, int64_t col_stride,
                               int packed, double scale, double dx, double dy, const double* edges, int nedges,
                               double* sum, unsigned long long* count, void* stream)
{
    if (!spectrum || !edges || !sum || !count || nrows < 1 || ncols < 1 || nedges < 1 || !(dx > 0) || !(dy > 0)
        || row_stride < 1 || col_stride < 1 || (reinterpret_cast<uintptr_t>(spectrum) & 15) || (packed && nrows % 2))
    {
        amb::set_last_error("amb_radial_rfft: bad arguments");
        return AMB_ERR_INVALID;
    }
    const auto s = static_cast<cudaStream_t>(stream);
    const auto* in = static_cast<const double*>(spectrum);
    return packed ? radial<PACKED>("amb_radial_rfft", in, nrows, ncols, row_stride, col_stride, scale, dx, dy, edges,
                                   nedges, sum, count, s)
                  : radial<HALF>("amb_radial_rfft", in, nrows, ncols, row_stride, col_stride, scale, dx, dy, edges,
                                 nedges, sum, count, s);
}

namespace
{
    template <typename Real>
    int label_impl(const Real* field, int nrows, int ncols, double threshold, int* labels, int* ncomp, void* stream)
    {
        if (!field || !labels || !ncomp || nrows < 1 || ncols < 1 || int64_t(nrows) * ncols > (int64_t(1) << 31) - 1)
        {
            amb::set_last_error("amb_label_components: bad arguments (grid must have < 2^31 sites)");
            return AMB_ERR_INVALID;
        }
        auto s = static_cast<cudaStream_t>(stream);
        const int n = nrows * ncols;
        cudaError_t e = cudaMemsetAsync(ncomp, 0, sizeof(int), s);
        if (e == cudaSuccess)
        {
            const int tx = (ncols + kTileC - 1) / kTileC, ty = (nrows + kTileR - 1) / kTileR;
            ccl_tiles<Real><<<tx * ty, kTileC * kTileR, 0, s>>>(field, nrows, ncols, tx, threshold, labels);
            ccl_borders<<<grid_for(size_t(tx) * nrows + size_t(ty) * ncols), 256, 0, s>>>(nrows, ncols, tx, ty, labels);
            ccl_compress<<<grid_for(n), 256, 0, s>>>(n, labels, ncomp);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess)
        {
            amb::set_last_error(std::string("amb_label_components: ") + cudaGetErrorString(e));
            return AMB_ERR_CUDA;
        }
        return AMB_OK;
    }
}

extern "C" int amb_label_components_f64(const double* field, int nrows, int ncols, double threshold, int* labels,
                                        int* ncomp, void* stream)
{
    return label_impl(field, nrows, ncols, threshold, labels, ncomp, stream);
}

extern "C" int amb_label_components_f32(const float* field, int nrows, int ncols, double threshold, int* labels,
                                        int* ncomp, void* stream)
{
    return label_impl(field, nrows, ncols, threshold, labels, ncomp, stream);
}
