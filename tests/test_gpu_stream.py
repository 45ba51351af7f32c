"""The streaming voxel-blocked kernel (register accumulators, the planner's
choice for few frames) against the FP64 oracle, on grids and frame counts at
the edges of its tiles: voxel blocks of 4 along the steering axis, tiles of
4 x 8 x 16 voxels, frame blocks of 1 to 8, frame pairs half empty, blocks that
share their sample rows (steering spread of at most 2 rows over a block) or
read their own, grids split by transmits, records whose ends the windows
cross.

Tolerance: the sample index is the FP32 sum of two FP32 table entries, three
roundings of at most 7.6e-6 samples each below index 256; white samples have an
RMS slope of pi / sqrt(3) per sample, so the index costs at most 4.2e-5 relative
RMS.  The polynomial weights add at most about sqrt(8 taps) x their error, 1.2e-6
(degree 8) or 7.9e-5 (degree 6, shared rows of FP16 / BF16 data).  Samples are
rounded to FP16 before either side reads them.
"""
import ctypes as C
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


from oracle import host as H


def _case(nz, nx, ny, span_deg, interp, receive_x=True, mask_tx=False, n_tx=3, n_ele=24, shift=0.0):
    from simu_rca_ab_b200 import workloads as W
    pitch = 0.3e-3
    X, Y, Z = W.make_grid(nx, ny, nz, 7.2e-3, 7.2e-3, 4e-3, 6e-3)
    pos, zero = W.rca_probe(n_ele, pitch), np.zeros(n_ele)
    th = np.deg2rad(np.linspace(-span_deg, span_deg, n_tx)) if n_tx > 1 else np.zeros(1)
    G = {"gridBfX": X + shift, "gridBfY": Y + shift, "gridBfZ": Z, "posEleX": pos if receive_x else zero,
         "posEleY": zero if receive_x else pos, "posEleZ": zero, "apertureX": 7e-3, "apertureY": 7e-3,
         "apertureZ": 0.0}
    T = {"thetaX": th * (not receive_x), "thetaY": th * receive_x, "flagReceiveX": receive_x}
    P = {"samplingFrequency": 15.6e6, "demodulationFrequency": 7.8e6, "speedOfSound": 1540.0,
         "startTime": -4e-6, "fnumber": 1.0}
    O = {"interpolation": interp[0], "lanczosOrder": interp[1], "flagMaskTransmit": mask_tx}
    return G, T, P, O, n_tx, n_ele


def _errcount():
    from simu_rca_ab_b200 import _lib as L
    n = C.c_int64()
    L.check(L.lib().rcabf_take_error_count(C.byref(n)))
    return n.value


CODE = {"quadratic": H.INTERP_QUAD3, "ref6": H.INTERP_REF6, "lanczos": H.INTERP_LANCZOS}


def _check(case, n_frame, ns, storage="float32", compound=True):
    """Relative RMS error of the planner's kernel against the FP64 oracle."""
    import torch
    from simu_rca_ab_b200 import _lib as L
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200 import workloads as W
    from simu_rca_ab_b200.params import normalize
    G, T, P, O, n_tx, n_ele = case
    g = torch.Generator(device="cuda").manual_seed(3)
    iq = torch.randn(n_frame, n_tx, n_ele, ns, dtype=torch.complex64, device="cuda", generator=g)
    if storage == "float16":
        iq = iq.to(torch.complex32)
    eng = B.default_engine()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        geom = eng.geometry(normalize(np.zeros(1, np.complex64), G, T, P, O))
        out, mask = eng.beamform(geom, iq, storage={"float32": L.STORE_F32, "float16": L.STORE_F16}[storage],
                                 compound=compound)
        dn = iq.to(torch.complex64).cpu().numpy()
        r = H.prepare(W.as_matlab(dn), G, T, P, {"flagMaskTransmit": O["flagMaskTransmit"]})
    f64, m64 = H.run_fp64(r, CODE[O["interpolation"]], O["lanczosOrder"], data=dn)
    c64, cm = H.compound(f64, m64, True) if compound else (f64, m64)
    ref = np.asarray(c64).reshape(out.shape)
    assert np.allclose(mask.cpu().numpy().ravel(), np.asarray(cm).ravel(), rtol=1e-5, atol=1e-6)
    assert _errcount() == 0
    return H.rel_rms(out.cpu().numpy(), ref)


TOL = {8: 4.6e-5, 6: 2.7e-4}
L4, L3, L2, Q, R6 = ("lanczos", 4), ("lanczos", 3), ("lanczos", 2), ("quadratic", 3), ("ref6", 3)


@pytest.mark.parametrize("storage", ["float32", "float16"])
@pytest.mark.parametrize("nz,nx,ny,span", [(33, 9, 21, 2.0), (16, 4, 8, 4.0), (17, 5, 9, 12.0), (1, 3, 2, 3.0),
                                            (17, 5, 11, 20.0), (18, 9, 6, 30.0)])
@pytest.mark.parametrize("n_frame", [1, 2, 3, 4, 5, 9])
def test_stream_kernel_vs_fp64(cuda, storage, nz, nx, ny, span, n_frame):
    # degree-6 weights: shared rows of half-precision data, more than one frame
    deg = 8 if storage == "float32" or n_frame == 1 else 6
    assert _check(_case(nz, nx, ny, span, L4), n_frame, 180, storage) < TOL[deg]


@pytest.mark.parametrize("interp", [L3, L2, Q, R6])
@pytest.mark.parametrize("receive_x,mask_tx,compound,shift", [(True, True, True, 0.0), (False, True, False, 0.0),
                                                              (False, False, True, 0.4e-3)])
def test_stream_kernel_interpolations_masks_and_outputs(cuda, interp, receive_x, mask_tx, compound, shift):
    for nf, ns in ((1, 150), (6, 97)):      # 97 samples: the record ends inside the grid
        case = _case(31, 12, 18, 3.0, interp, receive_x, mask_tx, n_tx=5, shift=shift)
        assert _check(case, nf, ns, compound=compound) < TOL[8]


@pytest.mark.parametrize("nx,ny,n_tx,n_ele", [(16, 32, 4, 24), (15, 31, 5, 25), (16, 5, 3, 24), (3, 32, 4, 25),
                                              (15, 31, 1, 24)])
@pytest.mark.parametrize("n_frame,compound,receive_x", [(1, True, True), (2, True, False), (3, False, True),
                                                        (5, True, True)])
def test_mirrored_grids(cuda, nx, ny, n_tx, n_ele, n_frame, compound, receive_x):
    """Grids centred on the probe, both axes or one mirrored, odd and even
    counts of columns, elements and transmits (the middle ones mirror
    themselves)."""
    if not receive_x:
        nx, ny = ny, nx
    case = _case(18, nx, ny, 3.0, L3, receive_x, True, n_tx=n_tx, n_ele=n_ele)
    assert _check(case, n_frame, 170, compound=compound) < TOL[8]


@pytest.mark.parametrize("shift,ny,span,n_frame", [(0.0, 31, 3.0, 1), (0.4e-3, 31, 3.0, 1), (0.0, 16, 14.0, 1),
                                                   (0.4e-3, 16, 14.0, 5), (0.0, 8, 30.0, 5)])
def test_a_bad_sample_stays_in_its_voxels(cuda, shift, ny, span, n_frame):
    """A NaN and an infinite sample of a single frame, or of a grid whose voxel
    blocks spread over more than two rows, reach the voxels whose taps touch
    them, and no others: the plain kernel's set."""
    import torch
    from simu_rca_ab_b200 import _lib as L
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200.params import normalize
    G, T, P, O, n_tx, n_ele = _case(18, 15, ny, span, L4, shift=shift)
    eng = B.default_engine()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        geom = eng.geometry(normalize(np.zeros(1, np.complex64), G, T, P, O))
    g = torch.Generator(device="cuda").manual_seed(5)
    iq = torch.randn(n_frame, n_tx, n_ele, 170, dtype=torch.complex64, device="cuda", generator=g)
    iq[0, 1, 7, 60] = float("nan")
    iq[-1, 0, 20, 95] = float("inf")
    out, _ = eng.beamform(geom, iq)
    ref, _ = eng.beamform(geom, iq, kernel=L.KERNEL_PLAIN)
    bad, want = ~torch.isfinite(out.real + out.imag), ~torch.isfinite(ref.real + ref.imag)
    assert torch.equal(bad, want) and 0 < int(want.sum()) < want.numel() // 2
    assert _errcount() == 0


@pytest.mark.parametrize("nz,nx,ny,span", [(6, 17, 33, 3.0), (5, 9, 16, 6.0), (9, 40, 20, 2.0)])
@pytest.mark.parametrize("n_frame", [1, 3, 16, 31])
def test_coarse_depths_and_full_16_frame_blocks(cuda, nz, nx, ny, span, n_frame):
    """Depths 13 to 24 samples apart (flat tiles), and frame counts that fill
    16-frame blocks (the tensor-memory kernel)."""
    assert _check(_case(nz, nx, ny, span, L4), n_frame, 180) < TOL[8]
