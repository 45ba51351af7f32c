// Auxiliary kernels of librcabf: channel-data ingest, per-tile window range
// tables, the apodisation-sum mask, and an FP32 FMA throughput probe.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "das_kernels.cuh"
#include "launchers.h"

namespace rcabf {

// ------------------------------------------------------------------------
// Ingest: caller layout [frame][tx][ele][sample] (any rcabf_iq_dtype) ->
// slabs [tx][ele][frame block][sample][frame in block] in the storage type.
// One block moves 64 samples x FB frames of one (tx, ele) through shared
// memory so that both the reads (along samples) and the writes (along
// sample-major, frame-minor rows) are coalesced.
// ------------------------------------------------------------------------
template <int STORE> __device__ __forceinline__ typename StoreT<STORE>::T from_f2(float2 v);
template <> __device__ __forceinline__ float2 from_f2<ST_F32>(float2 v) { return v; }
template <> __device__ __forceinline__ __half2 from_f2<ST_F16>(float2 v) { return __float22half2_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat162 from_f2<ST_BF16>(float2 v) { return __float22bfloat162_rn(v); }

constexpr int INGEST_NS = 64;
constexpr int INGEST_FCHUNK = 64;    // frames of a block one CTA moves
constexpr int INGEST_MAX_FB = 256;

// grid.y = frame block x chunk of up to INGEST_FCHUNK of its frames
template <int STORE, int IQ>
__global__ void __launch_bounds__(256) ingest_kernel(const IngestParams p)
{
    using T = typename StoreT<STORE>::T;
    __shared__ float2 tile[INGEST_FCHUNK][INGEST_NS + 1];
    const int n_base = blockIdx.x * INGEST_NS;
    const int n_chunk = (p.fb + INGEST_FCHUNK - 1) / INGEST_FCHUNK;
    const int fb = blockIdx.y / n_chunk;
    const int f0 = (blockIdx.y % n_chunk) * INGEST_FCHUNK;   // first frame of the chunk within the block
    const int te = blockIdx.z;
    const int tx = te / p.n_ele, ele = te % p.n_ele;
    const int FB = p.fb;
    const int FC = min(INGEST_FCHUNK, FB - f0);              // frames of this chunk
    for (int i = threadIdx.x; i < FC * INGEST_NS; i += blockDim.x) {
        const int fi = i / INGEST_NS, nl = i % INGEST_NS;
        const int64_t f = (int64_t)fb * FB + f0 + fi;
        const int n = n_base + nl;
        float2 v = make_float2(0.f, 0.f);
        if (f < p.n_frame && n < p.n_sample)
            v = load_iq<IQ>(p.iq, ((f * p.n_tx + tx) * (int64_t)p.n_ele + ele) * p.n_sample + n);
        tile[fi][nl] = v;
    }
    __syncthreads();
    T *slab = reinterpret_cast<T *>(reinterpret_cast<char *>(p.S) +
                                    (((int64_t)tx * p.n_ele + ele) * p.n_fb + fb) * p.slab_bytes);
    const int n_rows = max(p.n_rows, p.n_sample);
    T *slab2 = p.S2 == nullptr ? nullptr
                               : reinterpret_cast<T *>(reinterpret_cast<char *>(p.S2) +
                                                       (((int64_t)tx * p.n_ele + ele) * p.n_fb + fb) * p.slab_bytes);
    for (int i = threadIdx.x; i < FC * INGEST_NS; i += blockDim.x) {
        const int nl = i / FC, fi = i % FC;
        const int n = n_base + nl;
        if (n < n_rows) {
            const float2 v = tile[fi][nl];
            slab[(int64_t)n * FB + f0 + fi] = from_f2<STORE>(v);   // zeros past the record
            if (slab2) slab2[(int64_t)n * FB + f0 + fi] = from_f2<STORE>(make_float2(-v.y, v.x));
        }
    }
}

template <int STORE>
static cudaError_t launch_ingest_store(const IngestParams &p, cudaStream_t st)
{
    const int n_chunk = (p.fb + INGEST_FCHUNK - 1) / INGEST_FCHUNK;
    dim3 grid((std::max(p.n_rows, p.n_sample) + INGEST_NS - 1) / INGEST_NS, p.n_fb * n_chunk, p.n_tx * p.n_ele);
    switch (p.iq_dtype) {
    case 0: ingest_kernel<STORE, 0><<<grid, 256, 0, st>>>(p); break;
    case 1: ingest_kernel<STORE, 1><<<grid, 256, 0, st>>>(p); break;
    case 2: ingest_kernel<STORE, 2><<<grid, 256, 0, st>>>(p); break;
    case 3: ingest_kernel<STORE, 3><<<grid, 256, 0, st>>>(p); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_ingest(const IngestParams &p, int store, cudaStream_t st)
{
    if (p.fb < 1 || p.fb > INGEST_MAX_FB || (int64_t)p.n_fb * ((p.fb + INGEST_FCHUNK - 1) / INGEST_FCHUNK) > 65535 ||
        p.n_tx * p.n_ele > 65535)
        return cudaErrorInvalidValue;
    switch (store) {
    case ST_F32: return launch_ingest_store<ST_F32>(p, st);
    case ST_F16: return launch_ingest_store<ST_F16>(p, st);
    case ST_BF16: return launch_ingest_store<ST_BF16>(p, st);
    default: return cudaErrorInvalidValue;
    }
}

// ------------------------------------------------------------------------
// Window range tables: (min, max) of the table delay over each tile's keys,
// valid entries only.  tab is [rows][n_a * n_z]; out is [rows][tiles_a][tiles_z].
// ------------------------------------------------------------------------
__global__ void range_kernel(const RangeParams p)
{
    const int64_t n_out = (int64_t)p.rows * p.tiles_a * p.tiles_z;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_out) return;
    const int tzi = (int)(i % p.tiles_z);
    const int tai = (int)((i / p.tiles_z) % p.tiles_a);
    const int64_t row = i / ((int64_t)p.tiles_z * p.tiles_a);
    float lo = __int_as_float(0x7f800000), hi = -lo;
    for (int a = 0; a < p.ta; ++a) {
        const int64_t ia = (int64_t)tai * p.ta + a;
        if (ia >= p.n_a) break;
        for (int z = 0; z < p.tz; ++z) {
            const int64_t iz = (int64_t)tzi * p.tz + z;
            if (iz >= p.n_z) break;
            const float4 e = p.tab[row * p.n_a * p.n_z + ia * p.n_z + iz];
            bool ok = true;
            if (p.is_rx) ok = (p.mode == MODE_EXACT) ? (e.w > 0.0f) : (e.z != 0.0f);
            if (ok) { lo = fminf(lo, e.x); hi = fmaxf(hi, e.x); }
        }
    }
    p.out[i] = make_float2(lo, hi);
}

cudaError_t launch_range(const RangeParams &p, cudaStream_t st)
{
    const int64_t n = (int64_t)p.rows * p.tiles_a * p.tiles_z;
    if (n <= 0) return cudaSuccess;
    range_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(p);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------
// Mask: sum over receive elements of the apodisation, for every insonified
// (pixel, tx) (RCA.cu:247-250, 301-304), summed over transmits when
// compounding (RCA.m:696).
// ------------------------------------------------------------------------
__global__ void mask_kernel(const DevGeom g, float *mask, int compound, int accumulate)
{
    const int64_t n_vox = g.n_z * g.n_u * g.n_v;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_vox) return;
    const int64_t iz = v % g.n_z, iu = (v / g.n_z) % g.n_u, iv = v / (g.n_z * g.n_u);
    const int64_t rxkey = iu * g.n_z + iz, txkey = iv * g.n_z + iz;
    const int64_t pix = iz * g.s_z + iu * g.s_u + iv * g.s_v;
    const float a = g.apod_sum[rxkey];
    float total = 0.0f;
    for (int tx = 0; tx < g.n_tx; ++tx) {
        bool cone = true;   // with no cone table the transmit mask is off: every table entry is inside
        if (g.cone_u) {
            const float4 t = g.tx_tab[(int64_t)tx * g.n_v * g.n_z + txkey];
            cone = ((g.mode == MODE_EXACT) ? t.w : t.y) != 0.0f &&
                   g.cone_u[(int64_t)tx * g.n_u * g.n_z + rxkey] != 0;
        }
        const float m = cone ? a : 0.0f;
        if (compound) {
            total = __fadd_rn(total, m);
        } else {
            float *o = mask + (int64_t)tx * g.n_pix + pix;
            *o = accumulate ? *o + m : m;
        }
    }
    if (compound) mask[pix] = accumulate ? mask[pix] + total : total;
}

cudaError_t launch_mask(const DevGeom &g, float *mask, int compound, int accumulate, cudaStream_t st)
{
    const int64_t n = g.n_z * g.n_u * g.n_v;
    mask_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, mask, compound, accumulate);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------
// Everything the streaming kernel needs before it starts, in one launch of
// independent blocks: channel data -> FP32 slab rows (rounded through the
// storage type, in the layout they are staged in: das_common.cuh's frame
// pairs as (re, re, im, im), padded rows, zero rows past the record), the two
// window range tables, and a zeroed work counter.  A call on a
// small grid is bound by launches and by the range kernel's few threads
// (10-17 us each for one thread per table entry on the 64 x 64 x 128 grid);
// here 16 lanes share an entry and all parts run at once.
// ------------------------------------------------------------------------
constexpr int PREP_THREADS = 256;
constexpr int RANGE_LANES = 16;

template <int STORE, int IQ>
__device__ __forceinline__ void prep_ingest(const IngestParams &p, int64_t i)
{
    const int rows = p.n_rows;
    const int n = (int)(i % rows);
    const int64_t q = i / rows;                       // (tx, ele), frame block
    const int fb = (int)(q % p.n_fb);
    const int64_t te = q / p.n_fb;
    if (te >= (int64_t)p.slab_tx * p.slab_ele) return;
    const int FB = p.fb;
    char *row = reinterpret_cast<char *>(p.S) + (te * p.n_fb + fb) * p.slab_bytes + (int64_t)n * vbs_row_bytes(FB);
    const int64_t f0 = (int64_t)fb * FB;
    const int tx = (int)(te / p.slab_ele), ele = (int)(te % p.slab_ele);
    const unsigned sh = p.n_sym == 4 ? 2 : p.n_sym == 2 ? 1 : 0;
    auto sample = [&](int64_t f) {   // copy f mod n_sym of frame f / n_sym
        const int64_t fr = f >> sh;
        if (n >= p.n_sample || fr >= p.n_frame) return make_float2(0.f, 0.f);
        const int m = vbs_mirrored(p.mirror, (int)f & (p.n_sym - 1));
        const int t = m & VBS_MIRROR_V ? p.n_tx - 1 - tx : tx, e = m & VBS_MIRROR_U ? p.n_ele - 1 - ele : ele;
        return to_f2(from_f2<STORE>(load_iq<IQ>(p.iq, ((fr * p.n_tx + t) * p.n_ele + e) * p.n_sample + n)));
    };
    if (FB == 1) {
        *reinterpret_cast<float2 *>(row) = sample(f0);
        return;
    }
#pragma unroll 4
    for (int k = 0; k < FB; k += 2) {
        const float2 a = sample(f0 + k), b = sample(f0 + k + 1);
        *reinterpret_cast<float4 *>(row + 8 * k) = make_float4(a.x, b.x, a.y, b.y);
    }
}

// one table entry per RANGE_LANES lanes
__device__ __forceinline__ void prep_range(const RangeParams &p, int64_t i, int lane)
{
    const int64_t n_out = p.rows * p.tiles_a * p.tiles_z;
    float lo = __int_as_float(0x7f800000), hi = -lo;
    if (i < n_out) {
        const int tzi = (int)(i % p.tiles_z);
        const int tai = (int)((i / p.tiles_z) % p.tiles_a);
        const float4 *tab = p.tab + i / ((int64_t)p.tiles_z * p.tiles_a) * p.n_a * p.n_z;
        const int nz = (int)min((int64_t)p.tz, p.n_z - (int64_t)tzi * p.tz);
        const int na = (int)min((int64_t)p.ta, p.n_lim - (int64_t)tai * p.ta);
        for (int k = lane; k < na * nz; k += RANGE_LANES) {
            const float4 e = __ldg(&tab[((int64_t)tai * p.ta + k / nz) * p.n_z + (int64_t)tzi * p.tz + k % nz]);
            if (!p.is_rx || e.w > 0.0f) { lo = fminf(lo, e.x); hi = fmaxf(hi, e.x); }
        }
    }
#pragma unroll
    for (int d = RANGE_LANES / 2; d > 0; d >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    if (lane == 0 && i < n_out) p.out[i] = make_float2(lo, hi);
}

template <int STORE, int IQ>
__global__ void __launch_bounds__(PREP_THREADS) prep_kernel(const __grid_constant__ PrepParams p)
{
    int64_t b = blockIdx.x;
    if (b == 0 && threadIdx.x == 0) *p.counter = 0u;
    if (b < p.blocks_rx + p.blocks_tx) {
        const bool rx = b < p.blocks_rx;
        if (!rx) b -= p.blocks_rx;
        prep_range(rx ? p.rx : p.tx, (b * PREP_THREADS + threadIdx.x) / RANGE_LANES, threadIdx.x % RANGE_LANES);
        return;
    }
    b -= p.blocks_rx + p.blocks_tx;
    prep_ingest<STORE, IQ>(p.ingest, b * PREP_THREADS + threadIdx.x);
}

template <int STORE>
static void launch_prep_store(const PrepParams &p, unsigned blocks, cudaStream_t st)
{
    switch (p.ingest.iq_dtype) {
    case 0: prep_kernel<STORE, 0><<<blocks, PREP_THREADS, 0, st>>>(p); break;
    case 1: prep_kernel<STORE, 1><<<blocks, PREP_THREADS, 0, st>>>(p); break;
    case 2: prep_kernel<STORE, 2><<<blocks, PREP_THREADS, 0, st>>>(p); break;
    default: prep_kernel<STORE, 3><<<blocks, PREP_THREADS, 0, st>>>(p); break;
    }
}

cudaError_t launch_prep(PrepParams &p, int store, cudaStream_t st)
{
    auto blocks = [](int64_t n) { return (n + PREP_THREADS - 1) / PREP_THREADS; };
    p.blocks_rx = blocks(p.rx.rows * p.rx.tiles_a * p.rx.tiles_z * RANGE_LANES);
    p.blocks_tx = blocks(p.tx.rows * p.tx.tiles_a * p.tx.tiles_z * RANGE_LANES);
    const int64_t n = p.blocks_rx + p.blocks_tx +
                      blocks((int64_t)p.ingest.slab_tx * p.ingest.slab_ele * p.ingest.n_fb * p.ingest.n_rows);
    if (n > INT32_MAX || p.ingest.iq_dtype < 0 || p.ingest.iq_dtype > 3) return cudaErrorInvalidValue;
    switch (store) {
    case ST_F32: launch_prep_store<ST_F32>(p, (unsigned)n, st); break;
    case ST_F16: launch_prep_store<ST_F16>(p, (unsigned)n, st); break;
    case ST_BF16: launch_prep_store<ST_BF16>(p, (unsigned)n, st); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------------------
// out[f][pix] (+)= sum over splits of part[split][f][pix], in split order:
// the transmit ranges of a grid too small to fill the GPU with whole items.
__global__ void __launch_bounds__(256) vbs_reduce_kernel(float2 *__restrict__ out, const float2 *__restrict__ part,
                                                         int64_t n, int n_split, int accumulate)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 a = part[i];
    for (int s = 1; s < n_split; ++s) {
        const float2 b = part[(int64_t)s * n + i];
        a.x += b.x;
        a.y += b.y;
    }
    if (accumulate) {
        const float2 q = out[i];
        a.x += q.x;
        a.y += q.y;
    }
    out[i] = a;
}

cudaError_t launch_vbs_reduce(float2 *out, const float2 *partial, int64_t n, int n_split, int accumulate,
                              cudaStream_t st)
{
    vbs_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, partial, n, n_split, accumulate);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------
// FP32 FMA throughput probe: 8 independent FMA chains per thread.
// ------------------------------------------------------------------------
__global__ void __launch_bounds__(256) fma_probe_kernel(float *out, int iters, float b, float c)
{
    float a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = (float)(threadIdx.x + k) * 1e-3f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int u = 0; u < 16; ++u)
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] = fmaf(a[k], b, c);
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += a[k];
    if (s == 12345.678f) out[threadIdx.x] = s;  // keeps the chains live
}

cudaError_t launch_fma_probe(float *out, int blocks, int iters, cudaStream_t st)
{
    fma_probe_kernel<<<blocks, 256, 0, st>>>(out, iters, 0.999999f, 1e-6f);
    return cudaGetLastError();
}

}  // namespace rcabf
