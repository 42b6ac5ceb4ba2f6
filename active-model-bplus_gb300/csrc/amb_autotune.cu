// Measured choice of the FP32 step kernel and its launch shape for one grid shape
// (no reference counterpart; the reference launches fixed 8 x 8 blocks).
//
// Candidates: the tile kernel with 256 or 512 threads per CTA, 32 or 64 output columns and the
// heights that put a whole number of tiles on each SM, launched once per step or once for all steps
// (persistent, grid barrier between steps), and the warp-pair sliding
// kernel with 1, 2 or 4 pairs per CTA (or, fused, one single warp per CTA) and the row-segment
// heights that put a whole number of tasks on each SM (plus the occupancy model's own choice). All candidates
// give bitwise the same field. Each is timed with CUDA events over a few steps on
// scratch buffers of the same shape; the fastest few are timed again and the best, or a nearly as fast one
// that leaves more of the GPU to runs on other streams (kSparing), is kept in a process-wide cache keyed by (device, nrows, ncols, compensated,
// noise), which AMB_KERNEL_AUTO consults. The kernels do the same work whatever the
// field values, so zero-filled scratch fields time the real workload.
#include "amb_gb300.h"
#include "amb_kernels.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

namespace
{
    using Key = std::tuple<int, int, int, int, int>;  // device, nrows, ncols, compensated, noise
    struct Entry
    {
        amb_kernel_config config;
        double us_per_step;
    };
    // A persistent launch on at most a quarter, or else half, of the GPU's threads is taken where it is at most this
    // much slower than the fastest: runs of small grids on several streams then advance at once. us per step and run,
    // one run and eight at once, f32c, T = 0.05: 128^2 3.0 and 0.85 (the fastest shape: 2.9 and 2.8), 64^2 2.95 and
    // 0.47 (3.0 and 1.5), 256^2 3.7 and 2.1 (3.4 and 3.2); from 250 x 333 on no such shape comes near the fastest.
    constexpr double kSparing = 1.08;

    std::map<Key, Entry> g_cache;
    std::mutex g_mutex;

    struct Scratch
    {
        float* a = nullptr;
        float* b = nullptr;
        uint16_t* r = nullptr;
        void* ws = nullptr;
        ~Scratch()
        {
            if (ws) cudaFree(ws);
            if (a) cudaFree(a);
            if (b) cudaFree(b);
            if (r) cudaFree(r);
        }
    };

    int key_device()
    {
        int d = 0;
        cudaGetDevice(&d);
        return d;
    }
}

namespace amb
{
    bool autotune_lookup(int nrows, int ncols, int compensated, int noise, amb_kernel_config* out)
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto it = g_cache.find(Key{key_device(), nrows, ncols, compensated ? 1 : 0, noise ? 1 : 0});
        if (it == g_cache.end()) return false;
        *out = it->second.config;
        return true;
    }
}

extern "C" int amb_autotune_f32(const amb_stencil* stencil, const amb_model* model, int nrows, int ncols,
                                int compensated, int probe_steps, void* stream, amb_kernel_config* best,
                                double* us_per_step)
{
    if (!stencil || !model || !best || nrows < 1 || ncols < 1 || probe_steps < 1 || probe_steps > 1000)
    {
        amb::set_last_error("amb_autotune_f32: bad arguments (probe_steps in [1, 1000])");
        return AMB_ERR_INVALID;
    }
    const int noise = model->temperature > 0 ? 1 : 0;
    const Key key{key_device(), nrows, ncols, compensated ? 1 : 0, noise};
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto it = g_cache.find(key);
        if (it != g_cache.end())
        {
            *best = it->second.config;
            if (us_per_step) *us_per_step = it->second.us_per_step;
            return AMB_OK;
        }
    }
    const size_t n = size_t(nrows) * ncols;
    Scratch s;
    cudaError_t e = cudaMalloc(&s.a, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&s.b, n * sizeof(float));
    if (e == cudaSuccess && compensated) e = cudaMalloc(&s.r, n * sizeof(uint16_t));
    const size_t ws_bytes = amb_step_workspace_bytes(AMB_F32, nrows, ncols);
    if (e == cudaSuccess) e = cudaMalloc(&s.ws, ws_bytes);
    if (e == cudaSuccess) e = cudaMemset(s.a, 0, n * sizeof(float));
    if (e == cudaSuccess && compensated) e = cudaMemset(s.r, 0, n * sizeof(uint16_t));
    if (e != cudaSuccess)
    {
        amb::set_last_error(std::string("amb_autotune_f32: ") + cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? AMB_ERR_NOMEM : AMB_ERR_CUDA;
    }

    std::vector<amb_kernel_config> cands;
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, key_device());
    // Tile heights that put m tiles on each SM (and the default 32 rows), for both tile widths.
    for (int cols : {32, 64})
    {
        const int across = (ncols + cols - 1) / cols, wide = cols == 64 ? AMB_FLAG_TILE_COLS_64 : 0;
        std::vector<int> rows{std::min(32, nrows)};
        for (int m : {1, 2, 3, 4, 6})
        {
            const int down = std::max(1, std::min(nrows, sms * m / across));
            const int h = (nrows + down - 1) / down;
            if (h <= 64) rows.push_back(h);
        }
        std::sort(rows.begin(), rows.end());
        rows.erase(std::unique(rows.begin(), rows.end()), rows.end());
        for (int h : rows)
            for (int groups : {1, 2})
                for (int flags : {0, AMB_FLAG_PERSISTENT}) cands.push_back({AMB_KERNEL_TILE, h, groups, flags | wide});
        for (int part : {2, 4})  // on a half and a quarter of the SMs' threads
        {
            const int h = (nrows + std::max(1, 2 * sms / part / across) - 1) / std::max(1, 2 * sms / part / across);
            if (h <= 64) cands.push_back({AMB_KERNEL_TILE, h, 1, AMB_FLAG_PERSISTENT | wide});
        }
    }
    if (ncols >= 112 && ncols % 4 == 0)
    {
        // Segment heights that put m tasks on each SM: a task costs its rows plus about eight rows of
        // pipeline fill, so the best height is one whose task count just fills the SMs, with as many
        // resident tasks as pay for their fill (1536^2: 24 rows, 30.8 us; 16 and 32 rows 37). Heights are even:
        // a warp pair takes two rows per round.
        const int strips = (ncols + 111) / 112;
        const auto rows_for = [&](int m) {
            const int segs = std::max(1, std::min(nrows, sms * m / strips));
            return ((nrows + segs - 1) / segs + 1) & ~1;
        };
        const auto add = [&](std::initializer_list<int> ms, int pairs, int flags) {
            std::vector<int> rows{0};
            for (int m : ms) rows.push_back(rows_for(m));
            std::sort(rows.begin(), rows.end());
            rows.erase(std::unique(rows.begin(), rows.end()), rows.end());
            for (int h : rows) cands.push_back({AMB_KERNEL_SLIDING, h, pairs, flags});
        };
        for (int pairs : {1, 2, 4}) add({2, 3, 4, 5, 6, 7, 8, 16}, pairs, 0);
        add({6, 8, 10, 12}, 1, AMB_FLAG_FUSED);
    }

    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    auto time_one = [&](const amb_kernel_config& c, float* ms) -> int {
        int in_spare = 0;
        int rc = amb_step_f32_ws(stencil, model, 1, nrows, ncols, s.a, s.b, s.r, 0, 2, nullptr, &c, s.ws, ws_bytes, stream,
                                 &in_spare);
        if (rc) return rc;
        cudaEventRecord(t0, static_cast<cudaStream_t>(stream));
        rc = amb_step_f32_ws(stencil, model, 1, nrows, ncols, s.a, s.b, s.r, 2, probe_steps, nullptr, &c, s.ws, ws_bytes,
                             stream, &in_spare);
        if (rc) return rc;
        cudaEventRecord(t1, static_cast<cudaStream_t>(stream));
        if (cudaEventSynchronize(t1) != cudaSuccess) return AMB_ERR_CUDA;
        cudaEventElapsedTime(ms, t0, t1);
        return AMB_OK;
    };

    std::vector<std::pair<float, int>> times;
    int rc = AMB_OK;
    std::pair<float, int> chosen{0.f, 0};
    // How much of the GPU's threads (two CTAs of 256 per SM, by registers) a persistent launch holds on to.
    const auto share = [&](const amb_kernel_config& c) {
        if (c.kernel != AMB_KERNEL_TILE || !(c.flags & AMB_FLAG_PERSISTENT)) return 1.0;
        const int cols = c.flags & AMB_FLAG_TILE_COLS_64 ? 64 : 32;
        const double ctas = double((ncols + cols - 1) / cols) * ((nrows + c.seg_rows - 1) / c.seg_rows);
        return std::min(1.0, ctas * c.pairs_per_cta / (2.0 * sms));
    };
    for (size_t i = 0; i < cands.size() && rc == AMB_OK; ++i)
    {
        float ms = 0.f;
        rc = time_one(cands[i], &ms);
        if (rc == AMB_OK) times.push_back({ms, int(i)});
    }
    if (rc == AMB_OK)
    {
        std::sort(times.begin(), times.end());
        // second round for the leaders, over all and among those that leave half or three quarters of the GPU to
        // others: keep each one's fastest time
        std::vector<size_t> leaders;
        for (double most : {1.0, 0.5, 0.25})
        {
            const size_t count = most == 1.0 ? 4 : 2;
            for (size_t j = 0, taken = 0; j < times.size() && taken < count; ++j)
                if (times[j].first > 1.25f * times[0].first) break;  // out of reach, whatever the timing's noise
                else if (share(cands[times[j].second]) <= most)
                {
                    ++taken;
                    if (std::find(leaders.begin(), leaders.end(), j) == leaders.end()) leaders.push_back(j);
                }
        }
        const bool sparing = share(cands[times[leaders.back()].second]) <= 0.5;  // then twice: the choice is close
        for (int again = 0; again < (sparing ? 2 : 1); ++again)
            for (size_t j : leaders)
            {
                float ms = 0.f;
                if (rc == AMB_OK) rc = time_one(cands[times[j].second], &ms);
                if (rc == AMB_OK) times[j].first = std::min(times[j].first, ms);
            }
        float fastest = times[leaders[0]].first;
        for (size_t j : leaders) fastest = std::min(fastest, times[j].first);
        const auto pick = [&](double most) {
            const std::pair<float, int>* best = nullptr;
            for (size_t j : leaders)
                if (share(cands[times[j].second]) <= most && (!best || times[j].first < best->first)) best = &times[j];
            return best;
        };
        for (double most : {0.25, 0.5, 1.0})
        {
            const auto* p = pick(most);
            if (!p || p->first > kSparing * fastest) continue;
            chosen = *p;
            break;
        }
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    if (rc != AMB_OK) return rc;
    *best = cands[chosen.second];
    const double us = 1000.0 * chosen.first / probe_steps;
    if (us_per_step) *us_per_step = us;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        g_cache[key] = Entry{*best, us};
    }
    return AMB_OK;
}
