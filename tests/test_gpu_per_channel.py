"""Per-channel output of every frame in one launch, where its threads take
ranges of several frames (the last one shorter), against one launch per frame:
identical bits."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depths,n_frame", [(1, 1), (17, 100), (40, 131), (3, 2053)])
@pytest.mark.parametrize("tables", ["exact", "ref_compat"])
def test_ranges_of_frames_give_the_per_frame_bits(cuda, depths, n_frame, tables):
    import torch
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200 import workloads as W
    w = W.get("c0", n_frame=1)
    g = w.groups[0]
    z = np.linspace(5e-3, 25e-3, depths).reshape(depths, 1, 1)
    G = dict(g.Geometry, gridBfX=np.zeros_like(z), gridBfY=np.zeros_like(z), gridBfZ=z)
    T = dict(g.Transmit, thetaX=g.Transmit["thetaX"][:5], thetaY=g.Transmit["thetaY"][:5])
    O = {"interpolation": "ref6", "tableMode": tables}
    gen = torch.Generator(device="cuda").manual_seed(1)
    iq = torch.randn(n_frame * 5, 1, w.n_ele, 300, dtype=torch.complex64, device="cuda", generator=gen).permute(3, 2, 1, 0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        a, ma = B.bf_rca_nosum(iq, G, T, w.Param, O)
        b, mb = B.bf_rca_nosum(iq, G, T, w.Param, {**O, "kernel": "plain"})
    assert torch.equal(a, b) and torch.equal(ma, mb)
