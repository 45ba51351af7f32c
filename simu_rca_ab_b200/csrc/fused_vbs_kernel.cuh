// Persistent delay-and-sum kernel for few frames (sm_100a, EXACT tables,
// rectilinear grids): register accumulators, sample windows streamed by bulk
// copies several (tx, rx) steps ahead.
//
// A thread owns 4 voxels along v (the transmit-steering axis) and the
// FB frames of a block, as in the tensor-memory variant (fused_vb_kernel.cuh),
// whose arithmetic it keeps operation for operation: the two give the same
// bits.  With few frames per block the per-step work around the frame sums
// sets the pace, and this kernel is built around that:
//   - one elected warp scans the steps 32 at a time, drops the ones whose
//     window is empty for the tile, and issues the others' windows as bulk
//     copies (cp.async.bulk, one per step: the ingest writes slabs as FP32
//     rows already padded to the shared-memory stride) in chunks of up to
//     `krec` steps, three chunks in flight; no thread copies rows, converts
//     samples or computes windows, and there is no CTA barrier in the loop
//     (a full / empty mbarrier pair per chunk);
//   - the weights of voxel pairs are formed with packed FP32 operations
//     (fma.rn.f32x2: the scalar chain on each half);
//   - work items are handed out by an atomic counter, deepest tiles first
//     (the f-number leaves shallow tiles with few active steps, so a fixed
//     assignment leaves SMs idle at the end), and the scan runs on into the
//     next item while the current one is computed.
//
// Measured (B200, against the barrier-per-step kernels it replaced): 8 frames,
// 128 x 128 x 256, two orientations 257 -> 158 ms; 4 frames of a 256-element probe
// 361 -> 202 ms; 20 frames, 97 x 95 x 159 47.3 -> 28.5 ms; one frame, 64 x 64 x 128
// 9.38 -> 0.88 ms; one frame, 32 x 32 x 64, 4 transmits 455 -> 87 us.
// What bounds it: the FMA pipe with the shared-memory loads that feed it, and
// fixed latencies (8 frames: FMA pipe 58 % busy at 8 and at 12 warps per SM alike,
// issue slots 49 %; one frame: 49 % and 52 %).
// Grids centred on the probe and symmetric transmits: the voxels of half the u
// (v) axis carry their mirror images as further frames (VBS_MIRROR_*).
//
// D = 1, 2: the four voxels share TAPS + D staged rows (weights shifted to each
// voxel's first row, zeros elsewhere): one 16-byte load feeds 16 FMAs.
// D = 3, 4: pairs of voxels share TAPS + D - 2 rows, where the steering step
// spreads the four over more than two rows but a pair over at most two.
// D = 0: every voxel reads its own TAPS rows: single frames without mirrored
// copies, whose two FMAs per row leave the loads cheap, and wider spreads.
#pragma once

#include "das_common.cuh"
#include "poly_weights.cuh"
#include "tc_common.cuh"

namespace rcabf {

// Chunks of steps in flight, and most steps of a chunk.
constexpr int VS_STAGES = 3;
constexpr int VS_MAXREC = VBS_MAX_RECORDS;
constexpr int VS_THREADS = VB_THREADS_HOST;
constexpr int VS_WARPS = VS_THREADS / 32;
// 1.5 x 2^23: adding it rounding down leaves floor(x) in the low mantissa
// bits for |x| < 2^22 (the planner bounds the record length by VBS_MAX_SAMPLES)
constexpr float VS_MAGIC = 12582912.0f;
constexpr int VS_MAGIC_BITS = 0x4B400000;

// One step of a chunk: staged rows [lo, lo + count) of (tx, rx); the top bits
// of `count` hold the step's place m among the steps its slab serves.
struct __align__(16) VsRec {
    int32_t lo, count, tx, rx;
};
constexpr int VS_M_SHIFT = 28;
// One chunk: n records of work item `item` (-1: no more items), `last` the
// item's last chunk.
struct __align__(16) VsChunkInfo {
    int32_t item, n, last, pad;
};

// Bulk copy global -> shared, completion counted in bytes on an mbarrier
// (both addresses 16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Work item -> frame block, ranges of transmits and elements, and tile.  Tiles in depth-slowest
// order, deepest first.
struct VsItem {
    int job, fb, split, tu, tv, tz, tx0, n_tx, rx0, n_rx;
};
__device__ __forceinline__ VsItem vs_item(const FusedParams &prm, int item)
{
    VsItem w;
    w.job = 0;
    while (w.job + 1 < prm.n_jobs && prm.jobs[w.job + 1].item_begin <= item) ++w.job;
    const FusedJob &J = prm.jobs[w.job];
    uint32_t r = (uint32_t)(item - J.item_begin);
    w.tu = (int)(r % (uint32_t)J.tiles_u);
    r /= (uint32_t)J.tiles_u;
    w.tv = (int)(r % (uint32_t)J.tiles_v);
    r /= (uint32_t)J.tiles_v;
    w.split = (int)(r % (uint32_t)J.n_split);
    r /= (uint32_t)J.n_split;
    w.fb = (int)(r % (uint32_t)J.n_fb);
    w.tz = J.tiles_z - 1 - (int)(r / (uint32_t)J.n_fb);
    const int nst = J.n_split / J.split_rx, t = w.split / J.split_rx, e = w.split - t * J.split_rx;
    w.tx0 = (int)((int64_t)t * J.g.n_tx / nst);
    w.n_tx = (int)((int64_t)(t + 1) * J.g.n_tx / nst) - w.tx0;
    w.rx0 = (int)((int64_t)e * J.g.n_ele / J.split_rx);
    w.n_rx = (int)((int64_t)(e + 1) * J.g.n_ele / J.split_rx) - w.rx0;
    return w;
}

// A thread's first voxel (depth, receive axis, steering axis), and how many of
// its four lie on the grid's part that is computed.
struct __align__(16) VsVoxel {
    int iz, iu, iv, n;
};
__device__ __forceinline__ VsVoxel vs_voxel(const FusedJob &J, const VsItem &w, int tid)
{
    VsVoxel x;
    const unsigned q = (unsigned)tid / (unsigned)J.tu;
    x.iu = w.tu * J.tu + tid - (int)q * J.tu;
    x.iv = (w.tv * J.tv + (int)(q % (unsigned)J.tv)) * VB_BLOCK;
    x.iz = w.tz * J.tz + (int)(q / (unsigned)J.tv);
    const int rem = J.nv_t - x.iv;
    x.n = !(x.iz < J.g.n_z && x.iu < J.nu_t) || rem <= 0 ? 0 : rem >= VB_BLOCK ? VB_BLOCK : rem;
    return x;
}

// Scan state of a CTA, uniform over the scanning warp: the item scanned, the
// one after it (fetched ahead), its steps, the first step of the next batch
// of 32, the rotation of its step order, and the lanes of the current batch
// whose step is still to be issued.
struct VsScan {
    int item, next, steps, base, rot;
    unsigned mask;
    VsItem it;
};

template <int KIND, int FB, int DEG, int D>
__global__ void __launch_bounds__(VS_THREADS, vbs_min_ctas(FB)) fused_vbs_kernel(const __grid_constant__ FusedParams prm)
{
    static_assert(VB_BLOCK == 4, "weights are formed for two pairs of voxels");
    static_assert(FB == 1 || FB % 2 == 0, "frames are processed in pairs");
    static_assert(FB >= 2 || D == 0, "single frames: each voxel reads its own rows");
    using KT = KindTraits<KIND>;
    constexpr int VB = VB_BLOCK;
    constexpr int TAPS = KT::TAPS;
    constexpr int DS = D >= 3 ? D - 2 : D;       // shift rows of a group of voxels
    constexpr int GV = D >= 3 ? 2 : VB_BLOCK;    // its voxels
    constexpr int R = TAPS + DS;                 // rows it reads (D = 0: per voxel)
    constexpr int STRIDE = vbs_row_bytes(FB);
    constexpr int NP = FB == 1 ? 1 : FB / 2;     // frame pairs
    constexpr bool OWN = FB <= 4 || D >= 3;      // (4: a block one frame's mirrored copies fill)

    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full[VS_STAGES], empty[VS_STAGES];
    __shared__ VsRec recs[VS_STAGES][VS_MAXREC];
    __shared__ VsChunkInfo info[VS_STAGES];
    __shared__ VsScan scan_s;
    __shared__ VsItem item_s[VS_WARPS];          // per warp: the item it works on
    __shared__ VsVoxel vox_s[FB < 8 ? VS_THREADS : 1];   // per thread: its voxels
    __shared__ float4 tx_s[3][VS_THREADS];       // per thread: its voxels' index part and phasor of the transmit
    __shared__ float4 e_s[2][VS_THREADS];        // per thread: receive table entries of this and the next record
    __shared__ float4 scan_rng[32];              // per lane: receive, transmit table ranges of the next batch
    __shared__ int scan_lo[32], scan_cnt[32];    // per lane: window of its step of the current batch
    __shared__ volatile int abort_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t slot_bytes = (uint32_t)vbs_slot_bytes(FB, prm.wmax);
    const int krec = prm.krec;
    const uint32_t zero_rows = VS_STAGES * (unsigned)krec * slot_bytes;   // offset of TAPS rows of zeros behind the chunks
    {
        unsigned dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (krec < 1 || krec > VS_MAXREC || dyn < zero_rows + TAPS * STRIDE) {
            if (tid == 0) atomicAdd(prm.err_count, 1ull);
            return;
        }
    }
    if (tid == 0) {
        for (int i = 0; i < VS_STAGES; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], VS_WARPS);
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (D == 0)
        for (int i = tid; i < TAPS * STRIDE / 4; i += VS_THREADS) reinterpret_cast<float *>(smem + zero_rows)[i] = 0.f;
    __syncthreads();
    volatile int *abort = &abort_s;
    const uint32_t sbase = smem_u32(smem);

    // ---------------- the scan (warp 0) ----------------
    // Its state lives in shared memory between chunks: in registers it would
    // cost every warp of the CTA the same registers.
    // per lane: step position p of the item -> (tx, rx)
    auto step_of = [&](const VsScan &k, int p, int &tx, int &rx) {
        int e = p + k.rot;
        if (e >= k.steps) e -= k.steps;
        const int t = e / k.it.n_rx;
        rx = k.it.rx0 + e - t * k.it.n_rx;
        tx = k.it.tx0 + t;
    };
    // starts the copy of the table ranges of batch `base`
    auto fetch_ranges = [&](const VsScan &k) {
        const int p = k.base + lane;
        if (p < k.steps) {
            const FusedJob &J = prm.jobs[k.it.job];
            int tx, rx;
            step_of(k, p, tx, rx);
            cp_async<8>(&scan_rng[lane].x, &J.rx_range[((int64_t)rx * J.tiles_u + k.it.tu) * J.tiles_z + k.it.tz]);
            cp_async<8>(&scan_rng[lane].z, &J.tx_range[((int64_t)tx * J.tiles_v + k.it.tv) * J.tiles_z + k.it.tz]);
        }
        cp_async_commit();
    };
    // takes the next item: its scan starts at its first step
    auto scan_item = [&](VsScan &k, int item) {
        k.item = item < (int)prm.n_items ? item : -1;
        k.mask = 0;
        k.base = k.steps = 0;
        if (k.item < 0) return;
        k.next = 0;
        if (lane == 0) k.next = (int)atomicAdd(prm.counter, 1u);   // needed when this item's scan ends
        k.next = __shfl_sync(0xffffffffu, k.next, 0);
        k.it = vs_item(prm, k.item);
        const FusedJob &J = prm.jobs[k.it.job];
        k.steps = k.it.n_tx * k.it.n_rx;
        // transmit order rotated per tile: a hash of the tile picks the
        // quarter of the transmits the item starts from, so that CTAs of an
        // SM do not run their steps in lock step; whole transmits, so a
        // per-transmit item (n_tx = 1) is complete
        const uint32_t tile = (uint32_t)(k.it.tz + J.tiles_z * (k.it.tu + J.tiles_u * k.it.tv));
        const int t0 = k.it.n_tx >= 4 ? (int)(((tile * 0x9E3779B1u) >> 30) * (uint32_t)k.it.n_tx / 4u) : 0;
        k.rot = t0 * k.it.n_rx;
        fetch_ranges(k);
    };
    // fills stage st with the next chunk
    auto issue = [&](int st) {
        VsScan k = scan_s;
        __syncwarp();
        int n = 0, last = 0;
        uint32_t bytes = 0;
        const int item = k.item;
        if (item >= 0) {
            const FusedJob &J = prm.jobs[k.it.job];
            const int n_ele = J.g.n_ele;
            const char *S = reinterpret_cast<const char *>(J.S);
            const uint32_t slot0 = sbase + (uint32_t)(st * krec) * slot_bytes;
            int lo = scan_lo[lane], cnt = scan_cnt[lane];   // this lane's step of the batch before base
            while (n < krec) {
                int tx, rx;
                if (k.mask == 0) {
                    if (k.base >= k.steps) { last = 1; break; }
                    // windows of batch `base`, from the ranges copied ahead
                    cp_async_wait<0>();
                    bool act = false;
                    lo = cnt = 0;
                    if (k.base + lane < k.steps) {
                        step_of(k, k.base + lane, tx, rx);
                        const float4 q = scan_rng[lane];
                        if (q.x <= q.y && q.z <= q.w) {
                            const float ab = ab_value(J.g, tx, rx), fmax_n = (float)J.n_sample;
                            float lo_f = __fadd_rn(__fadd_rn(q.z, q.x), ab);
                            float hi_f = __fadd_rn(__fadd_rn(q.w, q.y), ab);
                            lo_f = fminf(fmaxf(floorf(lo_f), -1.0f), fmax_n);
                            hi_f = fminf(fmaxf(floorf(hi_f), -1.0f), fmax_n);
                            lo = max((int)lo_f - KT::LO, 0);
                            const int hi = min((int)hi_f - KT::LO + TAPS - 1, J.n_sample - 2);
                            if (hi >= lo) {
                                if (FB == 1) lo &= ~1;   // 8-byte rows: keep the copy 16-byte aligned
                                cnt = hi + DS - lo + 1;   // + shift rows
                                act = cnt <= prm.wmax;
                                if (!act) atomicAdd(prm.err_count, 1ull);   // never expected: the planner bounds the window
                            }
                        }
                    }
                    k.mask = __ballot_sync(0xffffffffu, act);
                    scan_lo[lane] = lo;
                    scan_cnt[lane] = cnt;
                    k.base += 32;
                    fetch_ranges(k);
                    continue;
                }
                const int rank = __popc(k.mask & ((1u << lane) - 1u));
                const bool mine = ((k.mask >> lane) & 1u) && rank < krec - n;
                if (mine) {
                    const int slot = n + rank;
                    step_of(k, k.base - 32 + lane, tx, rx);
                    int m = 0, slab = tx * n_ele + rx;
                    if (J.compact) {
                        const bool mu = (J.mirror & VBS_MIRROR_U) && rx > n_ele - 1 - rx;
                        const bool mv = (J.mirror & VBS_MIRROR_V) && tx > J.g.n_tx - 1 - tx;
                        slab = (mv ? J.g.n_tx - 1 - tx : tx) * (J.mirror & VBS_MIRROR_U ? (n_ele + 1) / 2 : n_ele) +
                               (mu ? n_ele - 1 - rx : rx);
                        m = J.n_sym == 4 ? (mu ? 1 : 0) | (mv ? 2 : 0) : mu || mv ? 1 : 0;
                    }
                    recs[st][slot] = VsRec{lo, cnt | m << VS_M_SHIFT, tx, rx};
                    const uint32_t b = ((uint32_t)(cnt * STRIDE) + 15u) & ~15u;
                    bulk_load(slot0 + (uint32_t)slot * slot_bytes,
                              S + ((int64_t)slab * J.n_fb + k.it.fb) * J.slab_bytes + (int64_t)lo * STRIDE, b, &full[st]);
                    bytes += b;
                }
                const unsigned took = __ballot_sync(0xffffffffu, mine);
                n += __popc(took);
                k.mask &= ~took;
            }
        }
        bytes = __reduce_add_sync(0xffffffffu, bytes);
        if (last) scan_item(k, k.next);
        __syncwarp();   // the lanes' records before lane 0's arrival
        if (lane == 0) {
            info[st] = VsChunkInfo{item, n, last, 0};
            scan_s = k;
            mbar_arrive_expect_tx(&full[st], bytes);
        }
        __syncwarp();
    };

    if (warp == 0) {
        int first = 0;
        if (lane == 0) first = (int)atomicAdd(prm.counter, 1u);
        VsScan k{};
        scan_item(k, __shfl_sync(0xffffffffu, first, 0));
        if (lane == 0) scan_s = k;
        __syncwarp();
        issue(0);
        issue(1);
    }

    // ---------------- state of the item being computed ----------------
    // (what the frame sums do not need is kept in shared memory, or with 8
    // frames worked out again: registers decide how many CTAs share an SM)
    int cur = -1, cur_tx = -1, n_pair = 0;
    int cur_m = 0;                            // the accumulators' slot s holds copy s ^ cur_m
    const float4 *rxp = nullptr;              // receive table entry of element 0, and the elements' stride
    int rx_stride = 0;
    float lim = 0.f;                          // sample indices at or past it leave the record
    int ab_job = -1;                          // the item's job, where it has an aberration law
    bool have_e = false;                      // the next record's table entry is on its way
    int e_buf = 0;
    unsigned cone_bits = 0;
    // FB = 1: (re, im) of voxel v in are[v][0]; else frames 2p, 2p + 1 of
    // voxel v: re in are[v][p], im in aim[v][p]
    float2 are[VB][NP], aim[VB][FB == 1 ? 1 : NP];

    // starts the copy of the receive table entry of element rx
    auto fetch_e = [&](int rx) {
        cp_async<16>(&e_s[e_buf][tid], rxp + (int64_t)rx * rx_stride);
        cp_async_commit();
        e_buf ^= 1;
    };

    for (uint32_t c = 0;; ++c) {
        const int st = (int)(c % VS_STAGES);
        if (!__all_sync(0xffffffffu, mbar_wait(&full[st], (c / VS_STAGES) & 1u, abort))) break;
        const VsChunkInfo ck = info[st];
        if (ck.item < 0) break;
        if (ck.item != cur) {
            cur = ck.item;
            cur_tx = -1;
            cur_m = 0;
            const VsItem ci = vs_item(prm, cur);
            const FusedJob &J = prm.jobs[ci.job];
            const VsVoxel x = vs_voxel(J, ci, tid);
            if constexpr (FB < 8) {   // many short items: decoded once
                vox_s[tid] = x;
                __syncwarp();
                if (lane == 0) item_s[warp] = ci;
                __syncwarp();
            }
            rxp = J.g.rx_tab + (x.n > 0 ? (int64_t)x.iu * J.g.n_z + x.iz : 0);   // off the grid: any entry, never used
            rx_stride = (int)(J.g.n_u * J.g.n_z);
            lim = (float)(J.n_sample - 1 - KT::HI);
            ab_job = J.g.ab != nullptr ? ci.job : -1;
            n_pair = FB == 1 ? 1 : (min(FB, J.n_vf - ci.fb * FB) + 1) / 2;
#pragma unroll
            for (int v = 0; v < VB; ++v)
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    are[v][p] = make_float2(0.f, 0.f);
                    if constexpr (FB > 1) aim[v][p] = make_float2(0.f, 0.f);
                }
        }
        const uint32_t slot0 = (uint32_t)(st * krec) * slot_bytes;   // offset in smem
        if (!have_e && ck.n > 0) fetch_e(recs[st][0].rx);
        for (int i = 0; i < ck.n; ++i) {
            VsRec h = recs[st][i];
            const int m = (int)((unsigned)h.count >> VS_M_SHIFT);
            h.count &= (1 << VS_M_SHIFT) - 1;
            cp_async_wait<0>();
            const float4 e = e_s[e_buf ^ 1][tid];
            if (i + 1 < ck.n) fetch_e(recs[st][i + 1].rx);
            if (h.tx != cur_tx) {
                cur_tx = h.tx;
                cone_bits = 0;
                const VsItem ci = FB < 8 ? item_s[warp] : vs_item(prm, cur);
                const DevGeom &g = prm.jobs[ci.job].g;
                const VsVoxel x = FB < 8 ? vox_s[tid] : vs_voxel(prm.jobs[ci.job], ci, tid);
                if (x.n > 0) {
                    const float4 *txrow = g.tx_tab + (int64_t)h.tx * (g.n_v * g.n_z) + x.iz;
                    const bool cu = g.cone_u == nullptr ||
                                    g.cone_u[(int64_t)h.tx * rx_stride + (int64_t)x.iu * g.n_z + x.iz] != 0;
                    float4 t[VB];
                    // (kept in shared memory, not in 12 registers across the frame sums)
#pragma unroll
                    for (int v = 0; v < VB; ++v) {
                        // voxels past the grid: the last one's entry, never in cone_bits
                        t[v] = __ldg(&txrow[(int64_t)(x.iv + min(v, x.n - 1)) * g.n_z]);
                        if (cu && v < x.n && t[v].w != 0.0f) cone_bits |= 1u << v;
                    }
                    tx_s[0][tid] = make_float4(t[0].x, t[1].x, t[2].x, t[3].x);
                    tx_s[1][tid] = make_float4(t[0].y, t[1].y, t[2].y, t[3].y);
                    tx_s[2][tid] = make_float4(t[0].z, t[1].z, t[2].z, t[3].z);
                }
            }
            if constexpr (FB >= 2) {
                if (m != cur_m) {   // half-way through the elements (transmits): the copies' slots swap
                    if ((m ^ cur_m) & 1) {
#pragma unroll
                        for (int v = 0; v < VB; ++v)
#pragma unroll
                            for (int p = 0; p < NP; ++p) {
                                are[v][p] = make_float2(are[v][p].y, are[v][p].x);
                                aim[v][p] = make_float2(aim[v][p].y, aim[v][p].x);
                            }
                    }
                    if constexpr (FB >= 4) {
                        if ((m ^ cur_m) & 2) {
#pragma unroll
                            for (int v = 0; v < VB; ++v)
#pragma unroll
                                for (int p = 0; p < NP; p += 2) {
                                    const float2 r = are[v][p], q = aim[v][p];
                                    are[v][p] = are[v][p + 1];
                                    aim[v][p] = aim[v][p + 1];
                                    are[v][p + 1] = r;
                                    aim[v][p + 1] = q;
                                }
                        }
                    }
                    cur_m = m;
                }
            }
            if (cone_bits == 0 || !(e.w > 0.0f)) continue;

            // ---- sample index of each voxel: floor and fraction ----
            float2 fl[2], dd[2];
            float rd[VB];
            bool ok[VB];
            float ab = 0.0f;
            if (ab_job >= 0) ab = ab_value(prm.jobs[ab_job].g, h.tx, h.rx);
            float base = 3.0e38f;
            const float4 ti = tx_s[0][tid];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float2 idx = __fadd2_rn(j ? make_float2(ti.z, ti.w) : make_float2(ti.x, ti.y), make_float2(e.x, e.x));
                idx = __fadd2_rn(idx, make_float2(ab, ab));
                rd[2 * j] = __fadd_rd(idx.x, VS_MAGIC);
                rd[2 * j + 1] = __fadd_rd(idx.y, VS_MAGIC);
                fl[j] = make_float2(rd[2 * j] - VS_MAGIC, rd[2 * j + 1] - VS_MAGIC);
                dd[j] = make_float2(idx.x - fl[j].x, idx.y - fl[j].y);
                ok[2 * j] = ((cone_bits >> (2 * j)) & 1u) && fl[j].x >= (float)KT::LO && fl[j].x < lim;
                ok[2 * j + 1] = ((cone_bits >> (2 * j + 1)) & 1u) && fl[j].y >= (float)KT::LO && fl[j].y < lim;
                if (ok[2 * j]) base = fminf(base, fl[j].x);
                if (ok[2 * j + 1]) base = fminf(base, fl[j].y);
            }
            if (!(base < 2.0e38f)) continue;

            // ---- phasor P = apod exp(j phase_tx) exp(j phase_rx) exp(j phase_ab) ----
            float2 Px[2], Py[2];
            const float4 tr = tx_s[1][tid], tq = tx_s[2][tid];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float2 txr = j ? make_float2(tr.z, tr.w) : make_float2(tr.x, tr.y);
                const float2 txq = j ? make_float2(tq.z, tq.w) : make_float2(tq.x, tq.y);
                const float2 ey = make_float2(e.y, e.y), ez = make_float2(e.z, e.z);
                const float2 nq = make_float2(-txq.x, -txq.y);
                Px[j] = __ffma2_rn(txr, ey, __fmul2_rn(nq, ez));
                Py[j] = __ffma2_rn(txr, ez, __fmul2_rn(txq, ey));
            }
            if (ab_job >= 0) {
                const float2 abp = ab_phasor(prm.jobs[ab_job].g, h.tx, h.rx);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 qx = Px[j], qy = Py[j];
                    const float2 ax = make_float2(abp.x, abp.x), ay = make_float2(abp.y, abp.y);
                    Px[j] = __ffma2_rn(qx, ax, __fmul2_rn(make_float2(-qy.x, -qy.y), ay));
                    Py[j] = __ffma2_rn(qx, ay, __fmul2_rn(qy, ax));
                }
            }

            if constexpr (D == 0) {
                // each voxel's own rows; a voxel without a contribution reads
                // the rows of zeros and adds exact zeros
                float2 w[2][TAPS];
#pragma unroll
                for (int j = 0; j < 2; ++j) poly_weights2<KIND, DEG>(dd[j], w[j]);
                const uint32_t slot = slot0 + (uint32_t)i * slot_bytes;
                uint32_t a[VB];
                bool bad = false;
#pragma unroll
                for (int v = 0; v < VB; ++v) {
                    const int row = __float_as_int(rd[v]) - VS_MAGIC_BITS - KT::LO - h.lo;
                    const bool in = (unsigned)row <= (unsigned)(h.count - TAPS);
                    bad = bad || (ok[v] && !in);
                    a[v] = ok[v] && in ? slot + (uint32_t)(row * STRIDE) : zero_rows;
                }
                if (bad) atomicAdd(prm.err_count, 1ull);   // never expected: window bound violated
                auto wt = [&](int v, int k) { return v & 1 ? w[v >> 1][k].y : w[v >> 1][k].x; };
                if constexpr (FB == 1) {
                    float2 tv[VB];   // interpolated sample
#pragma unroll
                    for (int v = 0; v < VB; ++v) {
                        tv[v] = make_float2(0.f, 0.f);
#pragma unroll
                        for (int k = 0; k < TAPS; ++k) {
                            const float2 x = *reinterpret_cast<const float2 *>(smem + a[v] + k * STRIDE);
                            tv[v].x = fmaf(wt(v, k), x.x, tv[v].x);
                            tv[v].y = fmaf(wt(v, k), x.y, tv[v].y);
                        }
                    }
#pragma unroll
                    for (int v = 0; v < VB; ++v) {
                        const float px = v & 1 ? Px[v >> 1].y : Px[v >> 1].x, py = v & 1 ? Py[v >> 1].y : Py[v >> 1].x;
                        float2 &q = are[v][0];
                        q.x = fmaf(px, tv[v].x, fmaf(-py, tv[v].y, q.x));
                        q.y = fmaf(px, tv[v].y, fmaf(py, tv[v].x, q.y));
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        if (p < n_pair) {
#pragma unroll
                            for (int v = 0; v < VB; ++v) {
                                const float px = v & 1 ? Px[v >> 1].y : Px[v >> 1].x;
                                const float py = v & 1 ? Py[v >> 1].y : Py[v >> 1].x;
                                float2 tre = make_float2(0.f, 0.f), tim = tre;
#pragma unroll
                                for (int k = 0; k < TAPS; ++k) {
                                    const float4 x = *reinterpret_cast<const float4 *>(smem + a[v] + k * STRIDE + p * 16);
                                    const float2 w2 = make_float2(wt(v, k), wt(v, k));
                                    tre = __ffma2_rn(w2, make_float2(x.x, x.y), tre);
                                    tim = __ffma2_rn(w2, make_float2(x.z, x.w), tim);
                                }
                                are[v][p] = __ffma2_rn(make_float2(px, px), tre,
                                                       __ffma2_rn(make_float2(-py, -py), tim, are[v][p]));
                                aim[v][p] = __ffma2_rn(make_float2(px, px), tim,
                                                       __ffma2_rn(make_float2(py, py), tre, aim[v][p]));
                            }
                        }
                    }
                }
            } else {
                // groups of GV voxels share rows from their lowest first one.
                // Weights are shifted to each voxel's first row; rows 0 .. DS-1
                // and TAPS .. R-1 are taken by some of a group's voxels only.
                // OWN: the others leave them out (and a voxel without a
                // contribution leaves its sums alone), so that a NaN or
                // infinite sample reaches no voxel whose taps do not touch it,
                // as in the one-voxel kernel that single frames and wide
                // spreads ran on.  Otherwise they add zero times the row, as
                // the tensor-memory kernel does (leaving them out measured
                // 11 % on 8 frames, 10 % on one).
#pragma unroll
                for (int v0 = 0; v0 < VB; v0 += GV) {
                    float gb = base;
                    if constexpr (GV < VB) {
                        gb = 3.0e38f;
#pragma unroll
                        for (int v = v0; v < v0 + GV; ++v)
                            if (ok[v]) gb = fminf(gb, v & 1 ? fl[v >> 1].y : fl[v >> 1].x);
                    }
                    const bool some = GV == VB || gb < 2.0e38f;
                    const int row = __float_as_int(gb + VS_MAGIC) - VS_MAGIC_BITS - KT::LO - h.lo;
                    const bool in = row >= 0 && row + R <= h.count;
                    if (some && !in) {
                        atomicAdd(prm.err_count, 1ull);   // never expected: window bound violated
#pragma unroll
                        for (int v = v0; v < v0 + GV; ++v) ok[v] = false;
                    }
                    const int row0 = some && in ? row : 0;   // (0: any staged row, not added)
                    float ws[GV][R];
                    bool s1[GV], s2[GV];
#pragma unroll
                    for (int j = 0; j < GV / 2; ++j) {
                        float2 w[TAPS];
                        poly_weights2<KIND, DEG>(dd[v0 / 2 + j], w);
#pragma unroll
                        for (int h2 = 0; h2 < 2; ++h2) {
                            const int q = 2 * j + h2, v = v0 + q;
                            const float sh = (h2 ? fl[v0 / 2 + j].y : fl[v0 / 2 + j].x) - gb;   // rows of shift
                            if (ok[v] && sh > (float)DS + 0.5f) { atomicAdd(prm.err_count, 1ull); ok[v] = false; }
                            s1[q] = sh > 0.5f;
                            s2[q] = DS >= 2 && sh > 1.5f;
#pragma unroll
                            for (int k = 0; k < R; ++k) {
                                auto wt = [&](int i) {   // OWN: rows the voxel leaves out may carry any weight
                                    const int c = i < 0 ? 0 : i < TAPS ? i : TAPS - 1;
                                    return OWN || c == i ? (h2 ? w[c].y : w[c].x) : 0.0f;
                                };
                                float a = wt(k);
                                if (s1[q]) a = wt(k - 1);
                                if constexpr (DS >= 2) { if (s2[q]) a = wt(k - 2); }
                                ws[q][k] = a;
                            }
                        }
                    }
                    auto uses = [&](int q, int k) {   // whether the group's voxel q adds row k
                        if (!OWN || (k >= DS && k < TAPS)) return true;
                        if constexpr (DS == 1) return k == 0 ? !s1[q] : s1[q];
                        else return k == 0 ? !s1[q] : k == 1 ? !s2[q] : k == TAPS ? s1[q] : s2[q];
                    };
                    float px[GV], py[GV];
#pragma unroll
                    for (int q = 0; q < GV; ++q) {
                        const int v = v0 + q;
                        const bool use = OWN || ok[v];
                        px[q] = use ? (v & 1 ? Px[v >> 1].y : Px[v >> 1].x) : 0.0f;
                        py[q] = use ? (v & 1 ? Py[v >> 1].y : Py[v >> 1].x) : 0.0f;
                    }
                    const uint32_t a0 = slot0 + (uint32_t)i * slot_bytes + (uint32_t)(row0 * STRIDE);
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        if (p < n_pair) {
                            float2 tre[GV], tim[GV];
#pragma unroll
                            for (int q = 0; q < GV; ++q) { tre[q] = make_float2(0.f, 0.f); tim[q] = tre[q]; }
#pragma unroll
                            for (int k = 0; k < R; ++k) {
                                const float4 x = *reinterpret_cast<const float4 *>(smem + a0 + k * STRIDE + p * 16);
#pragma unroll
                                for (int q = 0; q < GV; ++q) {
                                    const float2 w2 = make_float2(ws[q][k], ws[q][k]);
                                    if (uses(q, k)) {
                                        tre[q] = __ffma2_rn(w2, make_float2(x.x, x.y), tre[q]);
                                        tim[q] = __ffma2_rn(w2, make_float2(x.z, x.w), tim[q]);
                                    }
                                }
                            }
#pragma unroll
                            for (int q = 0; q < GV; ++q) {
                                const int v = v0 + q;
                                if (OWN && !ok[v]) continue;
                                const float2 p2 = make_float2(px[q], px[q]);
                                are[v][p] = __ffma2_rn(p2, tre[q], __ffma2_rn(make_float2(-py[q], -py[q]), tim[q], are[v][p]));
                                aim[v][p] = __ffma2_rn(p2, tim[q], __ffma2_rn(make_float2(py[q], py[q]), tre[q], aim[v][p]));
                            }
                        }
                    }
                }
            }
        }
        have_e = false;
        if (ck.last) {
            const VsItem ci = FB < 8 ? item_s[warp] : vs_item(prm, cur);
            const FusedJob &J = prm.jobs[ci.job];
            const DevGeom &g = J.g;
            const VsVoxel x = FB < 8 ? vox_s[tid] : vs_voxel(J, ci, tid);
            // the item's outputs: the volume (or the transmit's own, when not
            // compounded), or this transmit range's part of it
            cur = -1;
            float2 *out = J.out;
            int64_t stride = g.n_pix;
            bool add = J.accumulate != 0;
            if (!J.compound) {
                stride = (int64_t)g.n_tx * g.n_pix;
            } else if (J.n_split > 1) {
                out = J.partial + (int64_t)ci.split * J.n_frame * g.n_pix;
                add = false;
            }
#pragma unroll
            for (int f = 0; f < FB; ++f) {
                const int vf = ci.fb * FB + f;
                if (vf >= J.n_vf) continue;
                const int fr = J.n_sym == 1 ? vf : vf / J.n_sym;
                const int m = vbs_mirrored(J.mirror, (vf - fr * J.n_sym) ^ cur_m);
                const int ou = m & VBS_MIRROR_U ? (int)g.n_u - 1 - x.iu : x.iu;
                if ((m & VBS_MIRROR_U) && ou == x.iu) continue;   // the middle column: the unmirrored copy writes it
                // not compounded: copy m of transmit tx0 is the mirrored transmit's
                const int64_t off = J.compound ? 0
                                               : (int64_t)(m & VBS_MIRROR_V ? g.n_tx - 1 - ci.tx0 : ci.tx0) * g.n_pix;
                float2 *o0 = out + (int64_t)fr * stride + off + x.iz * g.s_z + ou * g.s_u;
#pragma unroll
                for (int v = 0; v < VB; ++v) {
                    const int iv = x.iv + v, ov = m & VBS_MIRROR_V ? (int)g.n_v - 1 - iv : iv;
                    if (v < x.n && !((m & VBS_MIRROR_V) && ov == iv)) {
                        float2 a;
                        if constexpr (FB == 1) a = are[v][0];
                        else a = f & 1 ? make_float2(are[v][f >> 1].y, aim[v][f >> 1].y)
                                       : make_float2(are[v][f >> 1].x, aim[v][f >> 1].x);
                        float2 *o = o0 + ov * g.s_v;
                        if (add) { float2 q = *o; q.x += a.x; q.y += a.y; *o = q; }
                        else *o = a;
                    }
                }
            }
        }
        else {
            // the next chunk's first table entry, when the chunk has landed
            const uint32_t nc = c + 1;
            const int ns = (int)(nc % VS_STAGES);
            if (__all_sync(0xffffffffu, mbar_test_wait(&full[ns], (nc / VS_STAGES) & 1u))) {
                have_e = info[ns].n > 0;
                if (have_e) fetch_e(recs[ns][0].rx);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[st]);
        if (warp == 0) {
            // refill the stage of the chunk before this one: the other warps
            // had the whole of this chunk to leave it
            if (c >= 1 && !__all_sync(0xffffffffu, mbar_wait(&empty[(c - 1) % VS_STAGES], ((c - 1) / VS_STAGES) & 1u, abort)))
                break;
            issue((int)((c + 2) % VS_STAGES));
        }
    }
    if (abort_s) {
        // a wait ran out: count it, and leave only when the copies this CTA
        // issued have landed (each wait bounded)
        if (tid == 0) {
            atomicAdd(prm.err_count, 1ull);
            int none = 0;
            for (int i = 0; i < VS_STAGES; ++i)
                for (uint32_t ph = 0; ph < 2; ++ph) mbar_wait(&full[i], ph, &none, 100000000ull);
        }
    }
}

}  // namespace rcabf
