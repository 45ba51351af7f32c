// Delay-and-sum of few frames in the reference's own single-precision
// arithmetic (REF_COMPAT tables): one thread per (voxel, transmit) and frame
// block, samples gathered from the caller's layout through L1.
//
// Each (voxel, transmit, element) costs some 300 instructions of sine, divide
// and sine-cosine evaluations that must be the reference's (ref_weights,
// setup_ref), against 24 for the samples of a frame, so the instruction issue
// rate bounds it.  The one-voxel fused kernel it replaces for few frames ran
// the transmits one after another and synchronised its 256 voxels at every
// step for the sake of the sample staging (one frame, 48 x 48 x 96 voxels, 16
// transmits, 64 elements, 6 taps: 7.5 ms, 3.5 here).  Here transmits run side by side,
// nothing synchronises, and the transmits' sums are added in the reference's
// order afterwards (launch_vbs_reduce): the same bits.
#pragma once

#include "das_common.cuh"
#include "plain_kernel.cuh"

namespace rcabf {

// blockIdx.y: transmit, blockIdx.z: frame block
template <int KIND, int IQ, int FB>
__global__ void __launch_bounds__(256) ref_das_kernel(const __grid_constant__ PlainParams prm)
{
    using KT = KindTraits<KIND>;
    const DevGeom &g = prm.g;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= g.n_z * g.n_u * g.n_v) return;
    const int tx = blockIdx.y;
    const int64_t f0 = (int64_t)blockIdx.z * FB;
    const int64_t iz = v % g.n_z, iu = (v / g.n_z) % g.n_u, iv = v / (g.n_z * g.n_u);
    const int64_t n_rxkey = g.n_u * g.n_z, rxkey = iu * g.n_z + iz;
    const float4 t = __ldg(&g.tx_tab[(int64_t)tx * (g.n_v * g.n_z) + iv * g.n_z + iz]);
    bool cone = t.y != 0.0f;
    if (g.cone_u != nullptr) cone = cone && g.cone_u[(int64_t)tx * n_rxkey + rxkey] != 0;
    float2 acc[FB];
#pragma unroll
    for (int f = 0; f < FB; ++f) acc[f] = make_float2(0.f, 0.f);
    if (cone) {
        const int64_t frame = (int64_t)g.n_tx * g.n_ele * prm.n_sample;
        const int64_t chan0 = (f0 * g.n_tx + tx) * (int64_t)g.n_ele;
        const float4 *rx = g.rx_tab + rxkey;
        for (int r = 0; r < g.n_ele; ++r, rx += n_rxkey) {
            const float4 e = __ldg(rx);
            if (e.z == 0.0f) continue;      // outside the aperture
            Setup<KIND> st;
            setup_ref<KIND>(t, e, ab_value(g, tx, r), g.ref, prm.n_sample, st);
            if (!st.ok) continue;
            const int64_t base = (chan0 + r) * prm.n_sample + st.n0 - KT::LO;
#pragma unroll
            for (int f = 0; f < FB; ++f) {
                if (FB > 1 && f0 + f >= prm.n_frame) break;
                float2 s;
#pragma unroll
                for (int j = 0; j < KT::TAPS; ++j) {
                    const float2 x = load_iq<IQ>(prm.iq, base + f * frame + j);
                    if (j == 0) {
                        s = make_float2(__fmul_rn(st.w[0], x.x), __fmul_rn(st.w[0], x.y));
                    } else {
                        s.x = __fadd_rn(s.x, __fmul_rn(st.w[j], x.x));
                        s.y = __fadd_rn(s.y, __fmul_rn(st.w[j], x.y));
                    }
                }
                const float cs = st.P.x, sn = st.P.y;   // RCA.cu:375-380
                float2 &a = acc[f];
                a.x = __fadd_rn(a.x, __fmul_rn(st.apod, __fadd_rn(__fmul_rn(s.x, cs), __fmul_rn(s.y, sn))));
                a.y = __fadd_rn(a.y, __fmul_rn(st.apod, __fadd_rn(__fmul_rn(-s.x, sn), __fmul_rn(s.y, cs))));
            }
        }
    }
    // [transmit][frame][voxel] sums to be added, or the transmit's own output
    const int64_t pix = iz * g.s_z + iu * g.s_u + iv * g.s_v;
#pragma unroll
    for (int f = 0; f < FB; ++f) {
        if (f0 + f >= prm.n_frame) break;
        if (prm.compound) {
            prm.out[((int64_t)tx * prm.n_frame + f0 + f) * g.n_pix + pix] = acc[f];
        } else {
            float2 *o = prm.out + ((f0 + f) * g.n_tx + tx) * g.n_pix + pix;
            if (prm.accumulate) { float2 q = *o; q.x += acc[f].x; q.y += acc[f].y; *o = q; }
            else *o = acc[f];
        }
    }
}

}  // namespace rcabf
