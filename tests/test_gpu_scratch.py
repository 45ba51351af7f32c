"""A call whose scratch memory cannot be allocated runs on the kernels that
stage the channel data in storage type, where these fit; otherwise, and for a
kernel by name, the allocation error is raised.

Tolerance: the kernels' weights differ by at most 7.9e-5 (degree-6 polynomials
of half-precision data; 1.2e-6 with degree 8 and with the tables' interpolation
1e-5), which white samples carry into the sums as sqrt(8 taps) times that."""
import warnings

import numpy as np
import pytest

from tests.host_runtime import acquisition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_frame,storage,tables", [(1, "float32", "exact"), (5, "float16", "exact"),
                                                     (2, "float32", "ref_compat")])
def test_call_without_room_for_its_scratch_runs_on_a_smaller_plan(cuda, monkeypatch, n_frame, storage, tables):
    import torch
    from oracle import host as H
    from simu_rca_ab_b200 import _lib as L
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200.params import normalize
    eng = B.Engine("cuda")
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        geom = eng.geometry(normalize(np.zeros(1, np.complex64), *acquisition(
            40, 32, 32, 2.0, tables=tables, interp=("ref6", 3) if tables == "ref_compat" else ("lanczos", 4))))
    g = torch.Generator(device="cuda").manual_seed(9)
    iq = torch.randn(n_frame, geom.n_tx, geom.n_ele, 180, dtype=torch.complex64, device="cuda", generator=g)
    st = L.STORE_F32
    if storage == "float16":
        iq, st = iq.to(torch.complex32), L.STORE_F16
    ref, ref_mask = (t.clone() for t in eng.beamform(geom, iq, storage=st))
    kw = dict(iq_dtype=L.IQ_C32 if storage == "float16" else L.IQ_C64, n_sample=180, n_frame=n_frame, compound=True,
              storage=st)
    out, mask = torch.full_like(ref, float("nan")), torch.full_like(ref_mask, float("nan"))
    a = eng.make_args(geom, iq, out=out, mask=mask, **kw)
    need, room = eng.workspace_bytes(geom, a), eng._workspace
    eng._ws.clear()

    def short(limit):
        def allocate(nbytes, stream_ptr):
            if nbytes > limit:
                raise torch.OutOfMemoryError("no room")
            return room(nbytes, stream_ptr)
        return allocate

    monkeypatch.setattr(eng, "_workspace", short(need - 1))
    eng.run(geom, a)
    torch.cuda.synchronize()
    assert (a.kernel, a.frames_per_block) == (L.KERNEL_AUTO, 0) and a.workspace_bytes < need
    assert H.rel_rms(out.cpu().numpy(), ref.cpu().numpy()) < (2.7e-4 if storage == "float16" else 4.6e-5)
    assert torch.equal(mask, ref_mask)
    monkeypatch.setattr(eng, "_workspace", short(1))
    with pytest.raises(torch.OutOfMemoryError):
        eng.run(geom, a)
    assert (a.kernel, a.frames_per_block) == (L.KERNEL_AUTO, 0)
    a.kernel = L.KERNEL_FUSED_NOBLOCK
    with pytest.raises(torch.OutOfMemoryError):
        eng.run(geom, a)
    eng.close()
