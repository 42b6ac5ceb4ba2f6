// Launcher of the FP64 step kernels: one tile per SM for small grids (amb_step_dtile.cuh), three
// grid-wide phases for the others (amb_step_phase.cuh).
#include "amb_kernels.h"
#include "amb_step_dtile.cuh"
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
        // A band has at least 48 rows, which for long rows are more than that; past this (700000 columns) the grid is
        // left to the tile kernel.
        constexpr size_t kWorkspaceMost = size_t(2) << 30;
        // Longest launch in seconds, and the steps that fit: a long run stays a queue of launches, between which
        // another stream's kernels find the SMs free (300000 steps of 64^2 in 180 launches: 6.0 us per step, as in
        // one). A step takes 6 us (tiles) or 12 us (phases) however small the grid, and 145 ps per site where the FP64
        // pipe binds.
        constexpr double kLaunchSeconds = 0.01;
        int steps_per_launch(int ny, int nx, bool tiles)
        {
            const double step = std::max(tiles ? 6e-6 : 12e-6, double(ny) * nx * 145e-12);
            return int(std::max(1.0, kLaunchSeconds / step));
        }
        constexpr size_t kTileSmem = size_t(200) << 10;

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

    namespace
    {
        // FP64 warp instructions of one step of a tile, as its lists are packed (runs of about one item per
        // thread), plus what the barriers and the halo load cost beside them.
        double tile_cost(int ty, int tx, int threads)
        {
            const auto list = [=](int w, int h, double per_site, double per_run) {
                const int l = std::max(1, w * h / threads), items = w * ((h + l - 1) / l);
                return double((items + 31) / 32) * (l * per_site + per_run);
            };
            return list(tx + 4, ty + 4, 25, 4) + list(2 * tx, 6, 11, 2) + list(12, ty, 11, 2) + list(tx + 2, ty + 2, 9, 8)
                   + list(tx, ty + 8, 9, 0) + list(tx + 8, ty, 9, 0) + list(tx, ty, 9, 8) + 2 * list(tx, ty, 8, 0)
                   + list(tx, ty, 3, 0);
        }

        // The tile shape that spreads a grid over the SMs, one tile each, at the least cost (64^2: 4 x 8, 6.0 us;
        // 1 x 64 12.3). False above 400 sites per SM, where the halo costs more than two grid barriers (us per
        // step, tiles and phases: 128^2 9.3 and 13.2, 200 x 300 18.4 and 20.1, 256^2 19.9 and 20.0, 350^2 35.8
        // and 29.5).
        bool tile_shape(int ny, int nx, int sms, dtile::Shape* best, int* threads)
        {
            double least = 1e300;
            *threads = double(ny) * nx > dtile::kSitesSmall * sms ? dtile::kThreads : dtile::kThreadsSmall;
            if (double(ny) * nx > 400.0 * sms) return false;
            for (int tx : {8, 12, 16, 24, 32, 48})
            {
                const int across = (nx + tx - 1) / tx, down = sms / across;
                if (down < 1) continue;
                const dtile::Shape t{std::max(1, (ny + down - 1) / down), tx};
                if (t.doubles() * sizeof(double) > kTileSmem) continue;
                const double cost = tile_cost(t.ty, t.tx, *threads);
                if (cost < least)
                {
                    least = cost;
                    *best = t;
                }
            }
            return least < 1e300;
        }
    }

    size_t step_phase_workspace(int ny, int nx)
    {
        int band;
        const size_t bytes = workspace_bytes<double>(ny, nx, &band);
        return bytes <= kWorkspaceMost ? bytes : 0;
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
        dtile::Shape tile{};
        int threads = 0;
        const bool small = tile_shape(p.ny, p.nx, sms, &tile, &threads);
        const void* dtile_kernel = threads == dtile::kThreads
                                       ? reinterpret_cast<const void*>(dtile::step_dtile_kernel<dtile::kThreads>)
                                       : reinterpret_cast<const void*>(dtile::step_dtile_kernel<dtile::kThreadsSmall>);
        if (small)
        {
            static std::mutex attr_mutex;
            static bool configured[2][64];
            bool* done = configured[threads == dtile::kThreads];
            std::lock_guard<std::mutex> lock(attr_mutex);
            if (dev >= 64 || !done[dev])
            {
                e = cudaFuncSetAttribute(dtile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTileSmem));
                if (e != cudaSuccess) return e;
                if (dev < 64) done[dev] = true;
            }
        }
        int band = 0;
        workspace_bytes<double>(p.ny, p.nx, &band);
        const phase::Coef k(p);
        const int chunk = steps_per_launch(p.ny, p.nx, small);
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
            if (small)
            {
                const int tiles = ((p.ny + tile.ty - 1) / tile.ty) * ((p.nx + tile.tx - 1) / tile.tx);
                unsigned* count = static_cast<unsigned*>(workspace);
                void* args[] = {&in, &out, &count, &pp, const_cast<phase::Coef*>(&k), &tile, &noise_mode, &inj, &m};
                e = cudaLaunchCooperativeKernel(dtile_kernel, dim3(tiles), dim3(threads), args, tile.doubles() * sizeof(double), stream);
                if (e != cudaSuccess) return e;
                done += n;
                continue;
            }
            void* args[] = {&in, &out, &workspace, &pp, const_cast<phase::Coef*>(&k), &noise_mode, &inj, &m, &band};
            e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(phase::step_phase_kernel<double>), dim3(sms),
                                            dim3(phase::kThreads), args, 0, stream);
            if (e != cudaSuccess) return e;
            done += n;
        }
        return cudaSuccess;
    }
}
