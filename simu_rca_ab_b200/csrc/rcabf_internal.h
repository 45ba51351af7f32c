// Internal structures shared by the host code and the CUDA kernels of librcabf.
//
// Data layout in HBM (one geometry):
//   rx_tab  float4 [n_ele][n_rxkey]   rx key = iu * n_z + iz (u = receive axis)
//             EXACT      : {irx, ar, ai, apod}   irx = fs * tau_rx (samples, FP64-built),
//                                                (ar, ai) = apod * exp(+j 2 pi fd/fs irx)
//             REF_COMPAT : {delay_rx (s), apod, valid, 0}   reference FP32 arithmetic
//   tx_tab  float4 [n_tx][n_txkey]    tx key = iv * n_z + iz (v = transmit steering axis)
//             EXACT      : {itx, pr, pi, cone_v}  itx = fs * (tau_tx + t0),
//                                                 (pr, pi) = exp(+j 2 pi (fd/fs itx - 2 fd z / c))
//             REF_COMPAT : {delay_tx (s), cone_v, z (m, FP32), 0}
//   cone_u  uint8  [n_tx][n_rxkey]    transmit-cone test along the receive axis (or NULL)
//   apod_sum float [n_rxkey]          sum over elements of the apodisation (the reference's mask)
//   ab      float  [n_ele] or [n_tx][n_ele]  receive aberration delay (EXACT: samples, REF: s)
//   ab_ph   float2 same shape             EXACT only: exp(+j 2 pi fd ab)
// Channel data after ingest (workspace):
//   S       [tx][ele][frame block][sample][frame in block], storage type
//           (complex64, half2 or bf16x2), each (tx, ele, block) slab padded to 16 B.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define RCABF_HD __host__ __device__
#else
#define RCABF_HD
#endif

namespace rcabf {

enum Mode : int { MODE_EXACT = 0, MODE_REF = 1 };

// Interpolation kernels as compile-time kinds.  TAPS taps on samples
// n0 - LO .. n0 - LO + TAPS - 1; a sample index n0 is usable when
// LO <= n0 < n_sample - 1 - HI (the reference's rule, RCA.cu:233-243, 323).
enum Kind : int { K_QUAD3 = 0, K_REF6 = 1, K_LANCZOS2 = 2, K_LANCZOS3 = 3, K_LANCZOS4 = 4 };

template <int KIND> struct KindTraits;
template <> struct KindTraits<K_QUAD3>    { static constexpr int TAPS = 3, LO = 1, HI = 1, WIN = 0; };
template <> struct KindTraits<K_REF6>     { static constexpr int TAPS = 6, LO = 2, HI = 3, WIN = 2; };
template <> struct KindTraits<K_LANCZOS2> { static constexpr int TAPS = 4, LO = 1, HI = 2, WIN = 2; };
template <> struct KindTraits<K_LANCZOS3> { static constexpr int TAPS = 6, LO = 2, HI = 3, WIN = 3; };
template <> struct KindTraits<K_LANCZOS4> { static constexpr int TAPS = 8, LO = 3, HI = 4, WIN = 4; };

inline RCABF_HD int kind_lo(int k) { return k == K_QUAD3 ? 1 : k == K_LANCZOS2 ? 1 : k == K_LANCZOS4 ? 3 : 2; }
inline RCABF_HD int kind_hi(int k) { return k == K_QUAD3 ? 1 : k == K_LANCZOS2 ? 2 : k == K_LANCZOS4 ? 4 : 3; }
inline RCABF_HD int kind_taps(int k) { return k == K_QUAD3 ? 3 : k == K_LANCZOS2 ? 4 : k == K_LANCZOS4 ? 8 : 6; }

enum Store : int { ST_F32 = 0, ST_F16 = 1, ST_BF16 = 2 };
inline RCABF_HD int store_bytes(int st) { return st == ST_F32 ? 8 : 4; }

// Scalars the REF_COMPAT arithmetic needs, exactly as the reference kernel
// holds them (RCA.cu:121-125, 164, 372).
struct RefScalars {
    float fs, fd, t0, inv_c, ratio;  // ratio = fdividef(fd, fs)
};

// Device view of one geometry.
struct DevGeom {
    const float4 *rx_tab;
    const float4 *tx_tab;
    const uint8_t *cone_u;     // NULL when the transmit mask is off
    const float *apod_sum;
    const float *ab;           // NULL when no aberration law
    const float2 *ab_ph;       // EXACT only
    const float *wtab;         // EXACT windowed-sinc kinds: polyphase weight table (WT_Q x 16 floats)
    int32_t ab_per_tx;
    int32_t mode;
    int32_t n_ele, n_tx;
    int64_t n_z, n_u, n_v;     // tile space: rx key = iu*n_z+iz, tx key = iv*n_z+iz
    int64_t s_z, s_u, s_v;     // output pixel index strides
    int64_t n_pix;
    RefScalars ref;
};

// One acquisition inside a fused launch.
struct FusedJob {
    DevGeom g;
    const void *S;             // ingested channel data
    int64_t slab_bytes;        // bytes of one (tx, ele, block) slab
    const float2 *rx_range;    // [n_ele][tiles_u][tiles_z] (min, max) table delay per tile
    const float2 *tx_range;    // [n_tx][tiles_v][tiles_z]
    float2 *out;               // [frame][compound ? 1 : n_tx][pix]
    int64_t item_begin;        // first work item of this job
    int32_t n_fb, n_frame, n_sample;
    int32_t compound, accumulate;
    int32_t tiles_z, tiles_u, tiles_v;
    int32_t tu, tv, tz;        // tile shape, tu*tv*tz = blockDim.x
    // streaming kernel: tile-space extents (halved along a mirrored axis), the
    // copies of a frame a block holds (1, 2 or 4: see VBS_MIRROR_*), frames x copies
    int32_t nu_t, nv_t;
    int32_t n_sym, mirror, n_vf, compact;
    // streaming kernel: ranges of steps, an item each: n_split / split_rx ranges
    // of transmits (n_tx when not compounded) x split_rx ranges of elements
    int32_t n_split, split_rx;
    float2 *partial;           // its sums per range [n_split][frame][pix] when compounded and n_split > 1
};

// Tensor-core kernel (fused_tc_kernel.cuh): voxel tiles of 128 voxels, tu
// (receive axis) x tv (steering axis) x 1 depth, with windows of at most
// TC_MAX_ROWS sample rows per (tx, rx) step; TC_TILE_U x TC_TILE_V is the
// preferred shape.
constexpr int TC_TILE_U = 4, TC_TILE_V = 32, TC_MAX_ROWS = 32;

constexpr int MAX_JOBS = 24;
constexpr int REF_MAX_FRAMES = 4;             // the per-transmit REF_COMPAT kernel: most frames, and
constexpr size_t REF_MAX_BYTES = 2ull << 30;  // most bytes of transmit sums
constexpr int FUSED_THREADS = 256;
constexpr int FUSED_STAGES = 3;
constexpr int VB_BLOCK = 4;          // voxels per thread along v in the voxel-blocked kernel
constexpr int VB_THREADS_HOST = 128; // its CTA size
constexpr int VB_STAGE_REGS = 2;     // 16-byte staging chunks a thread holds (FP16/BF16 slabs)
constexpr int VB_TM_MIN_BLOCKS = 4;  // launch-bounds hint with the accumulators in tensor memory (128 registers, no spills)
// tensor-memory columns a CTA of the voxel-blocked kernel allocates: 16 per
// frame pair, a power of two >= 32
constexpr RCABF_HD int vb_tmem_cols_host(int fb) { return fb * 8 <= 32 ? 32 : fb * 8; }

// Streaming voxel-blocked kernel (fused_vbs_kernel.cuh): steps per chunk at
// most, the longest record its floor() covers, FP32 slab rows in the layout
// they are staged in (frame pairs as (re, re, im, im), rows of 4 frames or
// more padded by 16 bytes so that 8 consecutive rows start in distinct banks).
// Mirror symmetry.  On a grid centred on the probe, the voxel at -u sees
// element E-1-r as the voxel at u sees element r, and with transmits steered
// symmetrically the voxel at -v sees transmit T-1-t as the voxel at v sees t:
// the same delays, weights, apodisation and phasors.  The streaming kernel then
// covers u >= 0 (v >= 0) only and carries the mirrored voxels as further
// "frames" of the block whose samples come from the mirrored element
// (transmit): the per-step work is shared by 2 or 4 times the frames.
// The steps (t, r), (t, E-1-r), (T-1-t, r), (T-1-t, E-1-r) read the same samples
// in another order of the copies, so one slab serves all of them where a block
// holds whole frames (`compact`): slot s of a row is copy s ^ m of step m of
// the four, and the kernel keeps its accumulators in slot order.
constexpr int VBS_MIRROR_U = 1, VBS_MIRROR_V = 2;
// copy s of a frame (s < n_sym) -> the axes it mirrors
constexpr RCABF_HD int vbs_mirrored(int mirror, int s)
{
    return mirror == (VBS_MIRROR_U | VBS_MIRROR_V) ? s : s ? mirror : 0;
}
// Degree of its weight polynomials: that of the storage where voxels share rows
// (d = 1, 2; the tensor-memory kernel's), the highest where pairs do or none.
constexpr RCABF_HD int vbs_weight_degree(int d, int store) { return (d == 1 || d == 2) && store != ST_F32 ? 6 : 8; }
constexpr int VBS_MAX_RECORDS = 8;
constexpr int VBS_MAX_SAMPLES = 1 << 21;
// CTAs per SM its registers are budgeted for: 2 x 4 x FB accumulators, the
// weights and the row in flight.  8 frames: three CTAs of 168 registers against
// two of 244: 28.9 against 32.3 ms (20 frames, 97 x 95 x 159), 201 against 222
// ms (4 frames, mirrored, 256 elements).  4 frames: three against four of 128
// registers: 0.90 against 1.00 ms (one frame, mirrored, 64 x 64 x 128).
constexpr RCABF_HD int vbs_min_ctas(int fb) { return fb >= 16 ? 2 : fb >= 4 ? 3 : 4; }
constexpr int VBS_PAD_ROWS = 2;      // zero rows past the record (shift rows)
constexpr RCABF_HD int vbs_row_bytes(int fb) { return fb <= 2 ? 8 * fb : 8 * fb + 16; }
constexpr RCABF_HD int vbs_slot_bytes(int fb, int wmax) { return (wmax * vbs_row_bytes(fb) + 15) / 16 * 16; }

struct FusedParams {
    FusedJob jobs[MAX_JOBS];
    int32_t n_jobs;
    int32_t wmax;               // rows per shared-memory stage
    int32_t row_words;          // shared-memory row stride (4-byte words)
    int32_t krec;               // streaming kernel: steps per chunk
    uint32_t *counter;          // streaming kernel: work items handed out (zero at launch)
    int64_t n_items;
    unsigned long long *err_count;
};

// Plain kernel: one launch per frame, thread per voxel, global gathers from
// the caller's [frame][tx][ele][sample] layout.
struct PlainParams {
    DevGeom g;
    const void *iq;
    int32_t iq_dtype;           // rcabf_iq_dtype
    int32_t n_sample;
    int64_t frame;
    int64_t n_frame;
    int32_t frames;             // per-channel, every frame in one launch: frames a thread takes
    int32_t compound, accumulate;
    int32_t per_channel;        // out is [element][frame][tx][pix]: one value per receive element
    float2 *out;
    unsigned long long *err_count;
};

}  // namespace rcabf
