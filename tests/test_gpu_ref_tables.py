"""Few frames on reference-compatible tables: the per-(voxel, transmit) kernel
(the planner's choice) against the fused kernel by name, which the suite pins
to the reference's bits: identical bits."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_frame", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("interp", ["quadratic", "ref6"])
@pytest.mark.parametrize("receive_x,mask_tx,compound,ab,real", [
    (True, True, True, False, False), (False, True, False, False, True), (True, False, True, True, False)])
def test_per_transmit_kernel_gives_the_fused_kernels_bits(cuda, n_frame, interp, receive_x, mask_tx, compound, ab, real):
    import torch
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200 import workloads as W
    n, n_tx, ns = 24, 3, 140
    X, Y, Z = W.make_grid(9, 11, 29, 7.2e-3, 7.2e-3, 4e-3, 6e-3)
    pos, zero = W.rca_probe(n, 0.3e-3), np.zeros(n)
    th = np.deg2rad(np.linspace(-4, 4, n_tx))
    G = {"gridBfX": X, "gridBfY": Y, "gridBfZ": Z, "posEleX": pos if receive_x else zero,
         "posEleY": zero if receive_x else pos, "posEleZ": zero, "apertureX": 7e-3, "apertureY": 7e-3,
         "apertureZ": 0.0}
    T = {"thetaX": th * (not receive_x), "thetaY": th * receive_x, "flagReceiveX": receive_x}
    P = {"samplingFrequency": 15.6e6, "demodulationFrequency": 7.8e6, "speedOfSound": 1540.0, "startTime": -4e-6,
         "fnumber": 1.0}
    O = {"interpolation": interp, "tableMode": "ref_compat", "flagMaskTransmit": mask_tx, "flagCompounding": compound}
    if ab:
        O["abLawRx"] = np.linspace(-2e-8, 3e-8, n)
    g = torch.Generator(device="cuda").manual_seed(2)
    if real:
        iq = torch.randn(n_frame * n_tx, 1, n, 2 * ns, device="cuda", generator=g)
    else:
        iq = torch.randn(n_frame * n_tx, 1, n, ns, dtype=torch.complex64, device="cuda", generator=g)
    iq = iq.permute(3, 2, 1, 0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        a, ma = B.bf_rca(iq, G, T, P, O)
        b, mb = B.bf_rca(iq, G, T, P, {**O, "kernel": "fused_noblock"})
    assert float(b.abs().max()) > 0.0
    assert torch.equal(a, b) and torch.equal(ma, mb)
