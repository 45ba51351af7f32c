// A CPU stand-in for the CUDA runtime and for librcabf's kernel launchers, so
// that the host code (geometry.cpp, api.cpp, server.cpp) plans, checks sizes
// and dispatches on a machine without a GPU.  Device memory is host memory;
// launches compute nothing: they are written to a log, one line each, and
// checked as the device would (a kernel function's shared-memory limit).
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "geometry.h"
#include "launchers.h"
#include "plan.h"

namespace {
std::mutex g_mu;
std::string g_log;
std::map<std::vector<int>, size_t> g_smem;   // kernel function -> its dynamic shared-memory limit
std::set<std::vector<int>> g_loaded;         // kernel functions launched so far
std::atomic<int> g_pending{0};               // host functions enqueued and not yet returned
int g_copies = 1;

void note(const std::string &s)
{
    std::lock_guard<std::mutex> lk(g_mu);
    g_log += s + "\n";
}
}  // namespace

extern "C" {

// ---- control, for the tests ----
void fake_set_copies(int on) { g_copies = on; }   // 0: host-buffer calls on pointers that hold nothing
void fake_take_log(char *buf, size_t len)
{
    std::lock_guard<std::mutex> lk(g_mu);
    snprintf(buf, len, "%s", g_log.c_str());
    g_log.clear();
}

// ---- CUDA runtime ----
cudaError_t cudaMalloc(void **p, size_t n) { return (*p = aligned_alloc(256, (n + 255) / 256 * 256 + 256)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (g_copies) memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaLaunchHostFunc(cudaStream_t, cudaHostFn_t fn, void *p)
{
    ++g_pending;
    std::thread([fn, p] {
        std::this_thread::sleep_for(std::chrono::milliseconds(20));
        fn(p);
        --g_pending;
    }).detach();
    return cudaSuccess;
}

}  // extern "C"

namespace rcabf {

static cudaError_t set_limit(std::vector<int> f, size_t smem)   // cudaFuncSetAttribute: the value given, up or down
{
    std::lock_guard<std::mutex> lk(g_mu);
    g_smem[f] = smem;
    return cudaSuccess;
}

// One launch of a fused kernel function: refused above its limit.
static cudaError_t launch(const char *name, std::vector<int> f, size_t smem, const FusedParams &p)
{
    std::string s = name;
    for (size_t i = 1; i < f.size(); ++i) s += " " + std::to_string(f[i]);
    {
        std::lock_guard<std::mutex> lk(g_mu);
        const auto it = g_smem.find(f);
        if (smem > (it == g_smem.end() ? 48 * 1024 : it->second)) return cudaErrorInvalidValue;
        if (!g_loaded.insert(f).second) f.clear();
    }
    // the first launch of a function may load its module, which waits for all
    // work in flight, host functions too (here 3 s at most)
    for (int i = 0; !f.empty() && g_pending.load() > 0; ++i) {
        if (i == 3000) return cudaErrorLaunchTimeout;
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
    }
    s += " jobs " + std::to_string(p.n_jobs);
    const FusedJob &J = p.jobs[0];   // what sets the order of its sums
    s += " order " + std::to_string(J.tu) + "," + std::to_string(J.tv) + "," + std::to_string(J.tz) + "," +
         std::to_string(J.n_sym) + "," + std::to_string(J.mirror) + "," + std::to_string(J.n_split) + "," +
         std::to_string(J.split_rx);
    s += " frames";
    for (int j = 0; j < p.n_jobs; ++j) s += " " + std::to_string(p.jobs[j].n_frame);
    note(s);
    return cudaSuccess;
}

cudaError_t launch_ingest(const IngestParams &, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_prep(PrepParams &, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_range(const RangeParams &, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_mask(const DevGeom &, float *, int, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_fma_probe(float *, int, int, cudaStream_t) { return cudaSuccess; }

cudaError_t launch_fused(int mode, int kind, int fb, int store, const FusedParams &p, int, size_t smem, cudaStream_t)
{
    return launch("fused", {0, mode, kind, fb, store}, smem, p);
}
cudaError_t prepare_fused(int mode, int kind, int fb, int store, size_t smem)
{
    return set_limit({0, mode, kind, fb, store}, smem);
}
int fused_occupancy(int, int, int, int, size_t) { return 2; }

cudaError_t launch_fused_vb(int kind, int d, int fb, int store, const FusedParams &p, int, size_t smem, cudaStream_t)
{
    return launch("vb", {2, kind, d, fb, store}, smem, p);
}
cudaError_t prepare_fused_vb(int kind, int d, int fb, int store, size_t smem)
{
    return set_limit({2, kind, d, fb, store}, smem);
}
int fused_vb_occupancy(int, int, int, int, size_t) { return 4; }

cudaError_t launch_fused_vbs(int kind, int d, int fb, int deg, const FusedParams &p, int, size_t smem, cudaStream_t)
{
    return launch("vbs", {1, kind, d, fb, deg}, smem, p);
}
cudaError_t prepare_fused_vbs(int kind, int d, int fb, int deg, size_t smem)
{
    return set_limit({1, kind, d, fb, deg}, smem);
}
int fused_vbs_occupancy(int, int, int, int, size_t) { return 3; }
cudaError_t launch_vbs_reduce(float2 *, const float2 *, int64_t, int, int, cudaStream_t) { return cudaSuccess; }

cudaError_t launch_fused_tc(int kind, int split, int bf16, const FusedJob &job, int fb, int rows, int64_t, unsigned long long *,
                            int, cudaStream_t)
{
    note("tc " + std::to_string(kind) + " " + std::to_string(split) + " " + std::to_string(bf16) + " " +
         std::to_string(fb) + " rows " + std::to_string(rows) + " of " + std::to_string(job.n_sample));
    return cudaSuccess;
}
int tc_max_frames_per_block(int split) { return split ? 208 : 232; }
int tc_tmem_columns(int, int) { return 512; }
size_t tc_launch_smem(int) { return 116 * 1024; }

cudaError_t launch_ref_das(int kind, const PlainParams &p, cudaStream_t)
{
    note("ref " + std::to_string(kind) + " frames " + std::to_string(p.n_frame));
    return cudaSuccess;
}
cudaError_t launch_plain(int, int, const PlainParams &, cudaStream_t)
{
    note("plain");
    return cudaSuccess;
}

cudaError_t noalloc_region(void **ws, unsigned long long **err)
{
    static unsigned long long e;
    *ws = (void *)256;
    *err = &e;
    return cudaSuccess;
}

// reference-compatible tables, to the rounding of these formulas
cudaError_t launch_ref_tables(const RefTableParams &p, cudaStream_t)
{
    *p.ratio_out = p.fd / p.fs;
    for (int64_t k = 0; k < p.n_rxkey; ++k) p.apod_sum[k] = 0.0f;
    for (int r = 0; r < p.n_ele; ++r)
        for (int64_t k = 0; k < p.n_rxkey; ++k) {
            const float z = p.rx_key_z[k], ap = std::fabs(p.rx_key_u[k] - p.ele_u[r]);
            const bool valid = ap < z / p.fnumber;
            p.rx_tab[r * p.n_rxkey + k] =
                make_float4(std::hypot(ap, z - p.ele_z[r]) * p.inv_c, valid ? 1.0f : 0.0f, valid ? 1.0f : 0.0f, 0.0f);
        }
    for (int t = 0; t < p.n_tx; ++t)
        for (int64_t k = 0; k < p.n_txkey; ++k)
            p.tx_tab[t * p.n_txkey + k] =
                make_float4((std::hypot(p.tx_key_v[k] - p.vs_v[t], p.tx_key_z[k] - p.vs_z[t]) - p.min_dist[t]) * p.inv_c,
                            1.0f, p.tx_key_z[k], 0.0f);
    return cudaSuccess;
}

}  // namespace rcabf
