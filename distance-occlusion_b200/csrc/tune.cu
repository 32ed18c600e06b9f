// tune.cu -- the launch-configuration table and the autotuner that fills it.
//
// Every kernel family here has launch parameters that change speed but never
// results (all kernels are exact for any of them): cells per lane of the row
// sweeps, the blocks of Danielsson, the engine of FastSweep 3D, rows per CTA of
// the JumpFlood passes, threads per CTA of the EDT line passes, the CTA shape of
// the batched kernel.  The table maps (family, size bucket = ceil(log2 of the row
// or line length)) to a value per device; 0 means "not tuned", and launchers then
// use their built-in rules.  dol_autotune measures each candidate on synthetic
// problems of the caller's shape (CUDA events, best of three runs): the first
// candidate is what an untuned launch does, and stays unless another is faster by
// more than kTuneNoise; dol_tune_set pins a value by hand.
#include <float.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "dol_b200.h"
#include "gen.cuh"
#include "kernels.h"

namespace dolk {

constexpr int kTuneDevices = 16;
constexpr int kTuneBuckets = 16;
constexpr float kTuneNoise = 0.97f;   // a candidate's time over the best so far, to replace it
static int g_tune[kTuneDevices][kTuneKinds][kTuneBuckets];
static std::mutex g_tune_mu;

static int bucket_of(int w)
{
    int b = 0;
    while (b < kTuneBuckets - 1 && (1 << b) < w) b++;
    return b;
}

static int cur_dev()
{
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return d >= 0 && d < kTuneDevices ? d : 0;
}

int tune_get(int kind, int w)
{
    if (kind < 0 || kind >= kTuneKinds) return 0;
    std::lock_guard<std::mutex> lock(g_tune_mu);
    return g_tune[cur_dev()][kind][bucket_of(w)];
}

void tune_put(int kind, int w, int value)
{
    if (kind < 0 || kind >= kTuneKinds) return;
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tune[cur_dev()][kind][bucket_of(w)] = value;
}

// test hooks of the bounded waits (kernels.h); process-wide, read at launch
static WaitHooks g_wait_hooks = {-1, 1u << 22};

WaitHooks wait_hooks()
{
    std::lock_guard<std::mutex> lock(g_tune_mu);
    return g_wait_hooks;
}

// candidate values per family, the built-in rule first: 0, or the value that means
// the same (Danielsson and FastSweep 2D 1, FastSweep 3D a positive one where the
// rule takes the columns, JumpFlood 3D 8, the batch 4, the EDT 512)
static std::vector<int> candidates(int kind, int w, int h, int d)
{
    switch (kind) {
        case kTuneDan2:
        case kTuneDan3: return {1, 2, 4, 8};   // cells per lane of a block's rows
        case kTuneFs2: return {1, 4, 8};       // cells per lane
        case kTuneFs3: {   // streaming columns, then the anti-diagonal wavefront (negative)
            std::vector<int> c;
            // (any positive value: the cells per thread of the slices that take over on little scratch)
            for (int most : {128, 256})
                for (int s : {1, 2, 4, 8})
                    if (c.empty() && (w + s - 1) / s <= most) c.push_back(s);
            if (fastsweep3_by_slices(w, h, d)) c.insert(c.begin(), 0);
            for (int s : {1, 2, 4, 8})
                if ((w + s - 1) / s <= 256) c.push_back(-s);
            return c;
        }
        case kTuneJfa2: return {0, 2, 4, 8, 16};   // one launch (up to 2^22 cells), or a launch per pass
        case kTuneJfa3: return {8, 2, 4, 16, -2, -4, -8, -16};   // z walk, then one thread per cell
        case kTuneBatch: return {4, 8};
        case kTuneEdt: return {512, 256};
        case kTuneDanRows: return {0, 4, 8, 16, kDanSerial};
        case kTuneDanSlices: return {0, 1, 4, 16, 64};
    }
    return {};
}

}  // namespace dolk

using namespace dolk;

// the batched kernel: a 256-image + 4-volume batch of the synthetic polygon /
// sphere generator, each CTA shape in turn
static dol_status tune_batch(cudaStream_t st)
{
    const int n2 = 256, n3 = 4, n = n2 + n3;
    std::vector<dol_batch_item> items(n);
    long long words = 0, dbytes = 0, cells = 0;
    dol_status s = dol_gen_batch(n2, n3, 13u, items.data(), &words, &dbytes, &cells, nullptr, st);
    if (s != DOL_OK) return s;
    void *dm = nullptr, *dd = nullptr, *df = nullptr, *ws = nullptr;
    const size_t wsb = dol_batch_workspace_size(n);
    if (cudaMalloc(&dm, words * 4) != cudaSuccess || cudaMalloc(&dd, dbytes) != cudaSuccess ||
        cudaMalloc(&df, cells * 4) != cudaSuccess || cudaMalloc(&ws, wsb) != cudaSuccess) {
        cudaGetLastError();
        for (void* p : {dm, dd, df, ws})
            if (p) cudaFree(p);
        return (dol_status)set_error(DOL_ERR_NO_MEMORY, "autotune scratch allocation failed");
    }
    s = dol_gen_batch(n2, n3, 13u, items.data(), nullptr, nullptr, nullptr, static_cast<uint32_t*>(dm), st);
    if (s == DOL_OK) s = dol_batch_prepare(n, items.data(), ws, wsb, st);
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    int best_v = 4;
    float best_t = FLT_MAX;
    for (int v : candidates(kTuneBatch, 1024, 1, 1)) {
        if (s != DOL_OK) break;
        tune_put(kTuneBatch, 1024, v);
        s = dol_batch_run(n, static_cast<uint32_t*>(dm), dd, static_cast<float*>(df), ws, st);
        float t_best = FLT_MAX;
        for (int rep = 0; rep < 3 && s == DOL_OK; rep++) {
            cudaEventRecord(a, st);
            s = dol_batch_run(n, static_cast<uint32_t*>(dm), dd, static_cast<float*>(df), ws, st);
            cudaEventRecord(b, st);
            cudaEventSynchronize(b);
            float t = 0.0f;
            cudaEventElapsedTime(&t, a, b);
            if (t < t_best) t_best = t;
        }
        if (t_best < kTuneNoise * best_t) {
            best_t = t_best;
            best_v = v;
        }
    }
    tune_put(kTuneBatch, 1024, best_v);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaStreamSynchronize(st);
    for (void* p : {dm, dd, df, ws})
        if (p) cudaFree(p);
    return s;
}

extern "C" {

DOL_API int dol_tune_get(int kind, int w) { return tune_get(kind, w); }

DOL_API void dol_test_wait_hooks(int stall_sweep, unsigned limit)
{
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_wait_hooks.stall_sweep = stall_sweep >= 0 && stall_sweep < 8 ? stall_sweep : -1;
    g_wait_hooks.limit = limit ? limit : 1u << 22;
}

DOL_API void dol_tune_set(int kind, int w, int value) { tune_put(kind, w, value); }

DOL_API dol_status dol_autotune(int kind, int w, int h, int d, void* stream)
{
    if (kind < 0 || kind >= kTuneKinds) return (dol_status)set_error(DOL_ERR_INVALID_ARG, "unknown tuning family %d", kind);
    if (w < 1 || h < 1 || d < 1) return (dol_status)set_error(DOL_ERR_INVALID_ARG, "empty shape");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (kind == kTuneBatch) return tune_batch(st);
    const bool vol = kind == kTuneDan3 || kind == kTuneFs3 || kind == kTuneJfa3 || kind == kTuneEdt ||
                     ((kind == kTuneDanRows && d > 1) || kind == kTuneDanSlices);
    // a bounded synthetic problem of the caller's row / line shape
    int tw = w, th = h, td = vol ? d : 1;
    if (kind == kTuneFs2) th = h < 256 ? h : 256;
    if (kind == kTuneFs3 || kind == kTuneDan3 || ((kind == kTuneDanRows || kind == kTuneDanSlices) && vol)) {
        // these are bound by their dependency chains, so the ranking changes with
        // rows and slices: the caller's shape up to 2^25 cells, beyond that rows
        // and slices halved in turn
        while ((long long)tw * th * td > (1LL << 25) && (th > 64 || td > 64)) {
            if (th >= td)
                th = (th + 1) / 2;
            else
                td = (td + 1) / 2;
        }
    }
    if (kind == kTuneJfa2 && (long long)tw * th > (1LL << 22)) th = (int)((1LL << 22) / tw > 0 ? (1LL << 22) / tw : 1);
    if (kind == kTuneEdt) {
        // the EDT's line kernels are what the value picks, and their cost per
        // CTA depends on the y and z line lengths: narrow the volume along x
        // (independent column tiles) before shortening the lines
        while ((long long)tw * th * td > (1LL << 26) && tw > 64) tw = ((tw / 2 + 15) / 16) * 16;
    }
    if (kind == kTuneJfa3 || kind == kTuneEdt) {
        while ((long long)tw * th * td > (1LL << 26) && td > 1) td = (td + 1) / 2;
    }
    const long long cells = (long long)tw * th * td;
    const size_t mwords = (size_t)((tw + 31) / 32) * th * td;

    void *dm = nullptr, *dl = nullptr, *tmp = nullptr, *ws = nullptr;
    const size_t cell_bytes = vol ? 6 : 4;
    const bool dan = kind == kTuneDan2 || kind == kTuneDan3 || kind == kTuneDanRows || kind == kTuneDanSlices;
    // (sized for every candidate, whatever value is set now)
    size_t ws_bytes = kind == kTuneEdt   ? edt_workspace_bytes(3, tw, th, td)
                      : dan              ? dan_blocks_workspace_bytes(vol ? 3 : 2, tw, th, td, 1)
                      : kind == kTuneFs3 ? std::max(fastsweep3_columns_most(tw, th, td), fastsweep3_workspace_bytes_min(tw, th, td))
                                         : 0;
    // an image's cost depends on its content: noise, and points
    const int contents = vol ? 1 : 2;
    bool ok = cudaMallocAsync(&dm, contents * mwords * 4, st) == cudaSuccess &&
              cudaMallocAsync(&dl, (size_t)cells * (kind == kTuneEdt ? 4 : cell_bytes), st) == cudaSuccess &&
              cudaMallocAsync(&tmp, jumpflood_workspace_bytes(vol ? 3 : 2, tw, th, td), st) == cudaSuccess &&
              cudaMallocAsync(&ws, ws_bytes + 256, st) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        for (void* p : {dm, dl, tmp, ws})
            if (p) cudaFreeAsync(p, st);
        return (dol_status)set_error(DOL_ERR_NO_MEMORY, "autotune scratch allocation failed");
    }
    std::vector<uint32_t> hm(contents > 1 ? mwords : 0, 0u);
    if (kind == kTuneEdt) {
        dol_gen_value_noise_3d(tw, th, td, 16, 3u, static_cast<uint32_t*>(dm), st);
    } else if (vol) {
        // solids sized to the volume: on a scatter of single seeds candidates rank
        // differently (FastSweep 3D wavefronts, Danielsson's cells per lane)
        const int m = std::min(tw, std::min(th, td));
        dol_gen_shapes_3d(tw, th, td, 32, 32, std::max(1, 4 * m / 256), std::max(2, 40 * m / 256), 5u,
                          static_cast<uint32_t*>(dm), st);
    } else {
        dol_gen_value_noise_3d(tw, th, 1, 32, 3u, static_cast<uint32_t*>(dm), st);
        uint32_t seed = 77;
        const int points = (int)std::max(8LL, cells / 10000);
        for (int i = 0; i < points; i++) {
            seed = lcg_next(seed);
            const int x = lcg_scale(seed, tw);
            seed = lcg_next(seed);
            const int y = lcg_scale(seed, th);
            hm[(size_t)y * ((tw + 31) / 32) + (x >> 5)] |= 1u << (x & 31);
        }
        cudaMemcpyAsync(static_cast<uint32_t*>(dm) + mwords, hm.data(), mwords * 4, cudaMemcpyHostToDevice, st);
    }
    int* err = nullptr;
    cudaMallocAsync((void**)&err, sizeof(int), st);

    auto run_one = [&](const uint32_t* mask) {
        const int dim = vol ? 3 : 2;
        switch (kind) {
            case kTuneDan2:
            case kTuneDan3:   // through the entry path: block schedule or serial engine
                launch_init_border(dim, mask, dl, tw, th, td, st);
                run_danielsson(dim, dl, tw, th, td, 2, true, ws, ws_bytes, err, st);
                break;
            case kTuneFs2:
                launch_init_border(2, mask, dl, tw, th, 1, st);
                launch_fastsweep_2d(dl, tw, th, 2, st);
                break;
            case kTuneFs3:
                launch_init_border(3, mask, dl, tw, th, td, st);
                launch_fastsweep_3d(dl, tw, th, td, 2, ws, ws_bytes, err, st);
                break;
            case kTuneJfa2:
            case kTuneJfa3:
                launch_init_border(dim, mask, dl, tw, th, td, st);
                launch_jumpflood(dim, dl, tmp, tw, th, td, 2, true, err, 0, st);
                break;
            case kTuneEdt:
                launch_edt_mask(3, mask, static_cast<float*>(dl), tw, th, td, DOL_EDT_SIGNED, ws,
                                ws_bytes, err, st);
                break;
            case kTuneDanRows:
            case kTuneDanSlices:
                launch_init_border(dim, mask, dl, tw, th, td, st);
                run_danielsson(dim, dl, tw, th, td, 2, true, ws, ws_bytes, err, st);
                break;
            case kTuneBatch:
                break;
        }
    };
    auto run_once = [&]() {
        for (int c = 0; c < contents; c++) run_one(static_cast<uint32_t*>(dm) + c * mwords);
    };

    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    float best_t = FLT_MAX;
    const int saved = tune_get(kind, w);
    int best_v = saved;
    // a narrowed synthetic volume looks its value up under its own width:
    // give it each candidate too, and put its entry back afterwards
    const bool other_key = bucket_of(tw) != bucket_of(w);
    const int saved_tw = tune_get(kind, tw);
    for (int v : candidates(kind, tw, th, td)) {
        tune_put(kind, w, v);
        if (other_key) tune_put(kind, tw, v);
        run_once();   // warm-up
        float t_best = FLT_MAX;
        for (int rep = 0; rep < 3; rep++) {
            cudaEventRecord(a, st);
            run_once();
            cudaEventRecord(b, st);
            cudaEventSynchronize(b);
            float t = 0.0f;
            cudaEventElapsedTime(&t, a, b);
            if (t < t_best) t_best = t;
        }
        if (t_best < kTuneNoise * best_t) {
            best_t = t_best;
            best_v = v;
        }
    }
    tune_put(kind, w, best_v);
    if (other_key) tune_put(kind, tw, saved_tw);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    for (void* p : {dm, dl, tmp, ws, (void*)err})
        if (p) cudaFreeAsync(p, st);
    cudaStreamSynchronize(st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (dol_status)set_error(DOL_ERR_CUDA, "autotune: %s", cudaGetErrorString(e));
    return DOL_OK;
}

}  // extern "C"
