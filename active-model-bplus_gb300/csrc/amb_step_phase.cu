// Launcher of the three-phase step kernel (amb_step_phase.cuh).
#include "amb_kernels.h"
#include "amb_step_phase.cuh"

#include <algorithm>
#include <mutex>

namespace amb
{
    namespace
    {
        // Largest planes workspace. A band of at most this many bytes keeps the recomputed rows of a
        // band boundary (16 of phase 1, 8 of phase 2) below 1 % of the band at 4096 columns.
        constexpr size_t kWorkspaceCap = size_t(256) << 20;
        // Sites x steps of one launch, about half a second of FP64 work, so that a long run stays a
        // queue of launches.
        constexpr double kLaunchWork = 4e9;

        template <typename Real>
        size_t workspace_bytes(int ny, int nx, int* band)
        {
            const size_t row = size_t(nx) * sizeof(Real) * phase::kPlanes;
            if (row * ny <= kWorkspaceCap)
            {
                *band = ny;
                return phase::kHeader + row * ny;
            }
            // at least as many rows as a band recomputes, whatever that takes
            const size_t fit = kWorkspaceCap / row;
            const size_t rows = std::max<size_t>(fit, 3 * 2 * phase::kBandHalo);
            if (rows >= size_t(ny))
            {
                *band = ny;
                return phase::kHeader + row * ny;
            }
            const int nb = int((size_t(ny) + rows - 2 * phase::kBandHalo - 1) / (rows - 2 * phase::kBandHalo));
            *band = (ny + nb - 1) / nb;  // even bands
            return phase::kHeader + row * (*band + 2 * phase::kBandHalo);
        }
    }

    size_t step_phase_workspace(int ny, int nx)
    {
        int band;
        return workspace_bytes<double>(ny, nx, &band);
    }

    cudaError_t launch_steps_phase(double* a, double* b, const StepParams& p, int noise_mode, const double* injected,
                                   int nsteps, void* workspace, cudaStream_t stream)
    {
        static std::mutex mutex;
        static int sms_of[64];
        int dev = 0, sms = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        {
            std::lock_guard<std::mutex> lock(mutex);
            if (dev < 64 && sms_of[dev]) sms = sms_of[dev];
            else
            {
                int coop = 0;
                if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev)) != cudaSuccess) return e;
                if (!coop) return cudaErrorNotSupported;
                if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
                if (dev < 64) sms_of[dev] = sms;
            }
        }
        int band = 0;
        workspace_bytes<double>(p.ny, p.nx, &band);
        const phase::Coef k(p);
        const int chunk = int(std::max(1.0, std::min(double(nsteps), kLaunchWork / (double(p.ny) * p.nx))));
        for (int done = 0; done < nsteps;)
        {
            const int n = std::min(chunk, nsteps - done);
            if ((e = cudaMemsetAsync(workspace, 0, phase::kHeader, stream)) != cudaSuccess) return e;
            StepParams pp = p;
            pp.step = p.step + done;
            const double* inj = injected ? injected + size_t(done) * 2 * p.ny * p.nx : nullptr;
            double* in = (done & 1) ? b : a;
            double* out = (done & 1) ? a : b;
            int m = n;
            void* args[] = {&in, &out, &workspace, &pp, const_cast<phase::Coef*>(&k), &noise_mode, &inj, &m, &band};
            e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(phase::step_phase_kernel<double>), dim3(sms),
                                            dim3(phase::kThreads), args, 0, stream);
            if (e != cudaSuccess) return e;
            done += n;
        }
        return cudaSuccess;
    }
}
