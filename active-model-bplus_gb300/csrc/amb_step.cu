// Launchers for the FP64 shared-memory tile step kernel (amb_step_tile.cuh): one launch per step, or
// (small grids) one cooperative launch for many steps with a grid barrier between them.
#include "amb_kernels.h"
#include "amb_step_tile.cuh"

namespace amb
{
    namespace
    {
        // Output tiles of TY rows x 32 columns, TY = 32 or 28.
        template <int NT, int TY>
        cudaError_t launch_tile(const double* phi_in, double* phi_out, const StepParams& p, int noise_mode,
                                const double* injected, cudaStream_t stream)
        {
            constexpr int TX = 32;
            using G = TileGeom<TY, TX>;
            constexpr size_t smem = G::template smem_bytes<double>();
            auto kern = step_tile_kernel<double, TY, TX, NT>;
            static bool configured = false;  // attribute is per-function; setting it twice is harmless
            if (!configured)
            {
                cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
                if (e != cudaSuccess) return e;
                configured = true;
            }
            dim3 grid((p.nx + TX - 1) / TX, (p.ny + TY - 1) / TY);
            kern<<<grid, NT, smem, stream>>>(phi_in, phi_out, p, Canon<double>(p), noise_mode, injected);
            return cudaGetLastError();
        }

        // All nsteps in one cooperative launch (grid = the resident CTAs, at most one per tile).
        // The grid barrier's arrival counter and error word come from the stream-ordered allocator
        // (cudaMallocAsync), so concurrent launches on other streams never share them.
        template <int NT, int TY>
        cudaError_t launch_tile_persistent(double* buf0, double* buf1, const StepParams& p, int noise_mode,
                                           const double* injected, int nsteps, cudaStream_t stream)
        {
            constexpr int TX = 32;
            using G = TileGeom<TY, TX>;
            constexpr size_t smem = G::template smem_bytes<double>();
            auto kern = step_tile_persistent_kernel<double, TY, TX, NT>;
            static int resident = 0;  // co-resident CTAs on this device type
            if (resident == 0)
            {
                cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
                if (e != cudaSuccess) return e;
                int dev = 0, sms = 0, blocks = 0, coop = 0;
                if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
                if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev)) != cudaSuccess) return e;
                if (!coop) return cudaErrorNotSupported;
                if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
                if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, NT, smem)) != cudaSuccess) return e;
                resident = blocks * sms;
                if (resident < 1) return cudaErrorNotSupported;
            }
            const int ntiles = ((p.nx + TX - 1) / TX) * ((p.ny + TY - 1) / TY);
            const int grid = ntiles < resident ? ntiles : resident;
            void* ws = nullptr;
            cudaError_t e = cudaMallocAsync(&ws, 2 * sizeof(unsigned), stream);
            if (e != cudaSuccess) return e;
            e = cudaMemsetAsync(ws, 0, 2 * sizeof(unsigned), stream);
            unsigned* count = static_cast<unsigned*>(ws);
            int* error = reinterpret_cast<int*>(count + 1);
            const Canon<double> k(p);
            StepParams pp = p;
            if (e == cudaSuccess)
            {
                void* args[] = {&buf0, &buf1, &pp, const_cast<Canon<double>*>(&k), &noise_mode,
                                const_cast<double**>(&injected), &nsteps, &count, &error};
                e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(grid), dim3(NT), args, smem,
                                                stream);
            }
            const cudaError_t ef = cudaFreeAsync(ws, stream);
            return e != cudaSuccess ? e : ef;
        }

        template <int TY>
        cudaError_t by_threads(const double* phi_in, double* phi_out, const StepParams& p, int noise_mode,
                               const double* injected, int groups, cudaStream_t stream)
        {
            if (groups == 4) return launch_tile<1024, TY>(phi_in, phi_out, p, noise_mode, injected, stream);
            if (groups == 2) return launch_tile<512, TY>(phi_in, phi_out, p, noise_mode, injected, stream);
            return launch_tile<256, TY>(phi_in, phi_out, p, noise_mode, injected, stream);
        }

        template <int TY>
        cudaError_t by_threads_persistent(double* a, double* b, const StepParams& p, int noise_mode,
                                          const double* injected, int nsteps, int groups, cudaStream_t stream)
        {
            if (groups == 4) return launch_tile_persistent<1024, TY>(a, b, p, noise_mode, injected, nsteps, stream);
            if (groups == 2) return launch_tile_persistent<512, TY>(a, b, p, noise_mode, injected, nsteps, stream);
            return launch_tile_persistent<256, TY>(a, b, p, noise_mode, injected, nsteps, stream);
        }
    }

    cudaError_t launch_step_tile(const double* phi_in, double* phi_out, const StepParams& p, int noise_mode,
                                 const double* injected, int groups, bool rows28, cudaStream_t stream)
    {
        return rows28 ? by_threads<28>(phi_in, phi_out, p, noise_mode, injected, groups, stream)
                      : by_threads<32>(phi_in, phi_out, p, noise_mode, injected, groups, stream);
    }

    cudaError_t launch_steps_tile_persistent(double* a, double* b, const StepParams& p, int noise_mode,
                                             const double* injected, int nsteps, int groups, bool rows28,
                                             cudaStream_t stream)
    {
        return rows28 ? by_threads_persistent<28>(a, b, p, noise_mode, injected, nsteps, groups, stream)
                      : by_threads_persistent<32>(a, b, p, noise_mode, injected, nsteps, groups, stream);
    }
}
