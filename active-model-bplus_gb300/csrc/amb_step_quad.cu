// Launchers of the FP32 quad tile kernel (amb_step_quad.cuh): one launch per step, or cooperative
// launches of many steps.
#include "amb_kernels.h"
#include "amb_step_quad.cuh"

#include <algorithm>
#include <mutex>

namespace amb
{
    namespace
    {
        using quadtile::Geom;
        using quadtile::Launch;

        constexpr int kMaxRows = 64;

        // Resident CTAs of a kernel at a given tile height, per device; raises the kernel's shared-memory
        // limit the first time.
        struct Residency
        {
            std::mutex mutex;
            int of[16][kMaxRows + 1] = {};
            cudaError_t get(const void* kernel, int nt, int ty, size_t smem, size_t smem_max, int* out)
            {
                int dev = 0, sms = 0, blocks = 0;
                cudaError_t e = cudaGetDevice(&dev);
                if (e != cudaSuccess) return e;
                std::lock_guard<std::mutex> lock(mutex);
                int* slot = dev < 16 ? &of[dev][ty] : nullptr;
                if (slot && *slot)
                {
                    *out = *slot;
                    return cudaSuccess;
                }
                if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_max))) != cudaSuccess)
                    return e;
                if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
                if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, nt, smem)) != cudaSuccess) return e;
                if (blocks < 1) return cudaErrorNotSupported;
                *out = blocks * sms;
                if (slot) *slot = *out;
                return cudaSuccess;
            }
        };

        template <int TX, int COMP, int NT>
        cudaError_t run(float* a, float* b, __nv_bfloat16* comp, const Launch& l, int64_t step0, const float* injected,
                        int nsteps, bool persistent, unsigned* count, cudaStream_t stream)
        {
            const size_t smem = size_t(Geom<TX>::floats(l.ty)) * 4, most = size_t(Geom<TX>::floats(kMaxRows)) * 4;
            const long long tiles = (long long)((l.nx + TX - 1) / TX) * ((l.ny + l.ty - 1) / l.ty);
            if (tiles > 0x7fffffffll) return cudaErrorInvalidValue;
            const int ntiles = int(tiles);
            int resident = 0;
            if (!persistent)
            {
                static Residency residency;
                auto kern = quadtile::step_quad_kernel<TX, COMP, NT>;
                cudaError_t e = residency.get(reinterpret_cast<const void*>(kern), NT, l.ty, smem, most, &resident);
                if (e != cudaSuccess) return e;
                kern<<<ntiles, NT, smem, stream>>>(a, b, comp, l, step0, injected);
                return cudaGetLastError();
            }
            static Residency residency;
            auto kern = quadtile::step_quad_persistent_kernel<TX, COMP, NT>;
            cudaError_t e = residency.get(reinterpret_cast<const void*>(kern), NT, l.ty, smem, most, &resident);
            if (e != cudaSuccess) return e;
            if ((e = cudaMemsetAsync(count, 0, sizeof(unsigned), stream)) != cudaSuccess) return e;
            Launch ll = l;
            void* args[] = {&a, &b, &comp, &ll, &step0, &injected, &nsteps, &count};
            return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(ntiles < resident ? ntiles : resident),
                                               dim3(NT), args, smem, stream);
        }

        template <int TX, int COMP>
        cudaError_t by_threads(int threads, float* a, float* b, __nv_bfloat16* comp, const Launch& l, int64_t step0,
                               const float* injected, int nsteps, bool persistent, unsigned* count, cudaStream_t stream)
        {
            return threads == 256 ? run<TX, COMP, 256>(a, b, comp, l, step0, injected, nsteps, persistent, count, stream)
                                  : run<TX, COMP, 512>(a, b, comp, l, step0, injected, nsteps, persistent, count, stream);
        }
    }

    cudaError_t launch_step_quad(float* a, float* b, __nv_bfloat16* comp, const StepParams& p, int noise_mode,
                                 const float* injected, int nsteps, const QuadTile& tile, unsigned* count,
                                 cudaStream_t stream)
    {
        const auto al = [](const void* q, uintptr_t n) { return (reinterpret_cast<uintptr_t>(q) & (n - 1)) == 0; };
        const Launch l{p.ny, p.nx, tile.rows < 1 ? 1 : tile.rows > kMaxRows ? kMaxRows : tile.rows, noise_mode,
                       p.nx % 4 == 0 && al(a, 16) && al(b, 16) && al(comp, 8), QuadCoef(p)};
        const bool persistent = count != nullptr;
        const auto go = [&](float* in, float* out, int64_t step, const float* inj, int n) {
            if (tile.cols64)
                return comp ? by_threads<64, COMP_BF16>(tile.threads, in, out, comp, l, step, inj, n, persistent, count, stream)
                            : by_threads<64, COMP_NONE>(tile.threads, in, out, comp, l, step, inj, n, persistent, count, stream);
            return comp ? by_threads<32, COMP_BF16>(tile.threads, in, out, comp, l, step, inj, n, persistent, count, stream)
                        : by_threads<32, COMP_NONE>(tile.threads, in, out, comp, l, step, inj, n, persistent, count, stream);
        };
        // A persistent launch takes at most some 10 ms of steps, so that a long run stays a queue of launches, between
        // which other streams' kernels that need whole SMs get their turn. A step takes 2.5 us however small the grid,
        // and 15.5 ps per site (1024^2).
        const double step_seconds = std::max(2.5e-6, double(p.ny) * p.nx * 15.5e-12);
        const int most = persistent ? int(std::max(1.0, 0.01 / step_seconds)) : 1;
        for (int s = 0, n; s < nsteps; s += n)
        {
            n = std::min(most, nsteps - s);
            const float* inj = injected ? injected + size_t(s) * 2 * p.ny * p.nx : nullptr;
            cudaError_t e = go(s & 1 ? b : a, s & 1 ? a : b, p.step + s, inj, n);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
}
