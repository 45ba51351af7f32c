// Fused + plain kernel instantiations for REF_COMPAT tables (the reference's
// quadratic and 6-tap kernels, complex64 storage).  Compiled with
// -fmad=false so that no product is fused into a following addition.
#include "fused_inst.cuh"
#include "ref_kernel.cuh"

namespace rcabf {

cudaError_t fused_entry_ref(int kind, int store, int fb, const FusedParams *p, int grid, size_t smem,
                            cudaStream_t st, int what, int *occ)
{
    if (store != ST_F32) return cudaErrorInvalidValue;
    if (kind == K_QUAD3) return fused_fb<MODE_REF, K_QUAD3, ST_F32>(fb, p, grid, smem, st, what, occ);
    if (kind == K_REF6) return fused_fb<MODE_REF, K_REF6, ST_F32>(fb, p, grid, smem, st, what, occ);
    return cudaErrorInvalidValue;
}

template <int KIND, int IQ>
static cudaError_t ref_das(const PlainParams &p, cudaStream_t st)
{
    const int64_t n = p.g.n_z * p.g.n_u * p.g.n_v;
    const int fb = p.n_frame >= 3 ? 4 : (int)p.n_frame;
    const dim3 grid((unsigned)((n + 255) / 256), (unsigned)p.g.n_tx, (unsigned)((p.n_frame + fb - 1) / fb));
    if (fb == 1) ref_das_kernel<KIND, IQ, 1><<<grid, 256, 0, st>>>(p);
    else if (fb == 2) ref_das_kernel<KIND, IQ, 2><<<grid, 256, 0, st>>>(p);
    else ref_das_kernel<KIND, IQ, 4><<<grid, 256, 0, st>>>(p);
    return cudaGetLastError();
}

template <int KIND>
static cudaError_t ref_das_iq(const PlainParams &p, cudaStream_t st)
{
    switch (p.iq_dtype) {
    case 0: return ref_das<KIND, 0>(p, st);
    case 1: return ref_das<KIND, 1>(p, st);
    case 2: return ref_das<KIND, 2>(p, st);
    case 3: return ref_das<KIND, 3>(p, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_ref_das(int kind, const PlainParams &p, cudaStream_t st)
{
    if (kind == K_QUAD3) return ref_das_iq<K_QUAD3>(p, st);
    if (kind == K_REF6) return ref_das_iq<K_REF6>(p, st);
    return cudaErrorInvalidValue;
}

cudaError_t plain_entry_ref(int kind, const PlainParams &p, cudaStream_t st)
{
    if (kind == K_QUAD3) return plain_iq<MODE_REF, K_QUAD3>(p, st);
    if (kind == K_REF6) return plain_iq<MODE_REF, K_REF6>(p, st);
    return cudaErrorInvalidValue;
}

}  // namespace rcabf
