"""Per-channel output where a thread takes a range of several frames, the last
range shorter: the bits of one launch per frame.  (Smaller calls give every
thread one frame.)"""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depths,n_frame,frames", [(40, 701, 7), (40, 199, 2), (96, 1009, 16)])
@pytest.mark.parametrize("tables", ["exact", "ref_compat"])
def test_ranges_of_several_frames_give_the_per_frame_bits(cuda, depths, n_frame, frames, tables):
    import torch
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200 import workloads as W
    n_tx, ns = 5, 300
    w = W.get("c0", n_frame=1)
    # the launch's rule: four threads per resident one, at most 16 frames each
    threads = torch.cuda.get_device_properties(cuda).multi_processor_count * 8192
    assert min(16, depths * w.n_ele * n_tx * n_frame // threads) == frames and n_frame % frames == 1
    g = w.groups[0]
    z = np.linspace(5e-3, 25e-3, depths).reshape(depths, 1, 1)
    G = dict(g.Geometry, gridBfX=np.zeros_like(z), gridBfY=np.zeros_like(z), gridBfZ=z)
    T = dict(g.Transmit, thetaX=g.Transmit["thetaX"][:n_tx], thetaY=g.Transmit["thetaY"][:n_tx])
    O = {"interpolation": "ref6", "tableMode": tables}
    gen = torch.Generator(device="cuda").manual_seed(1)
    iq = torch.randn(n_frame * n_tx, 1, w.n_ele, ns, dtype=torch.complex64, device="cuda", generator=gen)
    iq = iq.permute(3, 2, 1, 0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        a, ma = B.bf_rca_nosum(iq, G, T, w.Param, O)
        b, mb = B.bf_rca_nosum(iq, G, T, w.Param, {**O, "kernel": "plain"})
    assert float(a.abs().max()) > 0.0
    assert torch.equal(a, b) and torch.equal(ma, mb)
