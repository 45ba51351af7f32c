"""Host-buffer calls cut into chunks, a last one of one frame among them, give
the bits of the call on device buffers: grids with and without mirror symmetry,
steep steering, reference tables, half-precision data."""
import warnings

import numpy as np
import pytest

from tests.host_runtime import acquisition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("span,shift,storage,tables", [
    (2.0, 1e-3, "float16", "exact"), (2.0, 0.0, "float16", "exact"), (20.0, 0.0, "float32", "exact"),
    (30.0, 1e-3, "float32", "exact"), (2.0, 0.0, "float32", "ref_compat")])
@pytest.mark.parametrize("n_frame,chunks", [(9, (0, 1, 8)), (20, (0, 8, 16)), (16, (0, 5))])
def test_chunked_host_call_gives_the_device_calls_bits(cuda, span, shift, storage, tables, n_frame, chunks):
    import torch
    from simu_rca_ab_b200 import _lib as L
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200.params import normalize
    ns, half = 180, storage == "float16"
    acq = acquisition(40, 17, 21, span, shift=shift, tables=tables, n_ele=8 if tables == "ref_compat" else 24,
                      interp=("ref6", 3) if tables == "ref_compat" else ("lanczos", 4))
    eng = B.default_engine()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        geom = eng.geometry(normalize(np.zeros(1, np.complex64), *acq))
    g = torch.Generator(device="cuda").manual_seed(4)
    iq = torch.randn(n_frame, geom.n_tx, geom.n_ele, ns, dtype=torch.complex64, device="cuda", generator=g)
    if half:
        iq = iq.to(torch.complex32)
    kw = dict(iq_dtype=L.IQ_C32 if half else L.IQ_C64, n_sample=ns, n_frame=n_frame, mask=None, compound=True,
              storage=L.STORE_F16 if half else L.STORE_F32)
    out = torch.empty((n_frame, 1, geom.n_pix), dtype=torch.complex64, device="cuda")
    eng.run(geom, eng.make_args(geom, iq, out=out, **kw))
    iq_h, ref = iq.cpu().pin_memory(), out.cpu()
    assert float(ref.abs().max()) > 0.0
    for chunk in chunks:
        out_h = torch.full(out.shape, float("nan"), dtype=torch.complex64).pin_memory()
        eng.run_host(geom, eng.make_args(geom, iq_h, out=out_h, host=True, **kw), frames_per_chunk=chunk)
        torch.cuda.synchronize()
        assert torch.equal(out_h, ref), chunk


@pytest.mark.parametrize("storage", ["float32", "float16"])
@pytest.mark.parametrize("shift,shape", [(0.0, (72, 96, 96)), (1e-3, (72, 96, 96)), (0.0, (40, 32, 32))])
@pytest.mark.parametrize("compound", [True, False])
def test_frame_blocks_asked_for_give_one_result(cuda, storage, shift, shape, compound):
    """Blocks of 2 to 16 frames, of which full ones of 16 run on the
    tensor-memory kernel on a large grid."""
    import torch
    from simu_rca_ab_b200 import _lib as L
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200.params import normalize
    eng = B.default_engine()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        geom = eng.geometry(normalize(np.zeros(1, np.complex64),
                                      *acquisition(*shape, 2.0, shift=shift, n_ele=8, n_tx=3)))
    g = torch.Generator(device="cuda").manual_seed(6)
    iq = torch.randn(16, geom.n_tx, geom.n_ele, 180, dtype=torch.complex64, device="cuda", generator=g)
    st = L.STORE_F32
    if storage == "float16":
        iq, st = iq.to(torch.complex32), L.STORE_F16
    outs = [eng.beamform(geom, iq, storage=st, compound=compound, frames_per_block=fb)[0].clone() for fb in (2, 4, 8, 16)]
    assert float(outs[0].abs().max()) > 0.0
    for o in outs[1:]:
        assert torch.equal(o, outs[0])


@pytest.mark.parametrize("fb,which", [(1, (0, 1, 2, 3, 4, 5)), (4, (0, 1)), (4, (2, 3, 4, 5)), (16, (2, 3, 4, 5))])
def test_batch_of_mixed_grids_gives_the_bits_of_each_alone(cuda, fb, which):
    """Mirrored and unmirrored grids, steering spreads that share rows, pairs or
    none, points: one batch, several kernels."""
    import torch
    from simu_rca_ab_b200 import _lib as L
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200.params import normalize
    eng = B.default_engine()
    kws = [dict(span=2.0), dict(span=2.0, shift=1e-3), dict(span=20.0), dict(span=30.0), dict(span=30.0, shift=1e-3),
           dict(span=2.0, points=True)]
    g = torch.Generator(device="cuda").manual_seed(7)
    geoms, args, wss, outs, refs, iqs = [], [], [], [], [], []
    for k in which:
        kw = dict(kws[k])
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            geom = eng.geometry(normalize(np.zeros(1, np.complex64), *acquisition(33, 9, 12, kw.pop("span"), **kw)))
        iq = torch.randn(3, geom.n_tx, geom.n_ele, 180, dtype=torch.complex64, device="cuda", generator=g)
        refs.append(eng.beamform(geom, iq, frames_per_block=fb)[0].clone())
        outs.append(torch.full_like(refs[-1], float("nan")))
        a = eng.make_args(geom, iq, iq_dtype=L.IQ_C64, n_sample=180, n_frame=3, out=outs[-1], mask=None, compound=True,
                          frames_per_block=fb)
        wss.append(torch.empty(max(256, eng.workspace_bytes(geom, a)), dtype=torch.uint8, device="cuda"))
        geoms.append(geom)
        args.append(a)
        iqs.append(iq)
    eng.run_batch(geoms, args, wss)
    torch.cuda.synchronize()
    for o, r in zip(outs, refs):
        assert torch.equal(o, r) and float(r.abs().max()) > 0.0


@pytest.mark.parametrize("n_frame,storage,tables,shift", [
    (16, "float32", "exact", 0.0), (16, "float32", "exact", 1e-3), (1, "float16", "exact", 0.0),
    (5, "float16", "exact", 1e-3), (2, "float32", "ref_compat", 0.0)])
def test_served_requests_share_a_launch_and_give_the_bits_of_each_alone(cuda, n_frame, storage, tables, shift):
    import torch
    from simu_rca_ab_b200 import _lib as L
    from simu_rca_ab_b200 import beamformer as B
    from simu_rca_ab_b200.params import normalize
    from simu_rca_ab_b200.server import Server
    eng = B.default_engine()
    half = storage == "float16"
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        geom = eng.geometry(normalize(np.zeros(1, np.complex64), *acquisition(
            40, 32, 32, 2.0, shift=shift, tables=tables, interp=("ref6", 3) if tables == "ref_compat" else ("lanczos", 4))))
    g = torch.Generator(device="cuda").manual_seed(8)
    kw = dict(iq_dtype=L.IQ_C32 if half else L.IQ_C64, n_sample=180, n_frame=n_frame,
              storage=L.STORE_F16 if half else L.STORE_F32)
    iqs = [torch.randn(n_frame, geom.n_tx, geom.n_ele, 180, dtype=torch.complex64, device="cuda", generator=g)
           for _ in range(3)]
    iqs = [q.to(torch.complex32) for q in iqs] if half else iqs
    refs = []
    for q in iqs:
        refs.append(torch.empty((n_frame, 1, geom.n_pix), dtype=torch.complex64, device="cuda"))
        eng.run(geom, eng.make_args(geom, q, out=refs[-1], mask=None, compound=True, **kw))
    torch.cuda.synchronize()
    outs = [torch.full_like(r, float("nan")) for r in refs]
    torch.cuda.synchronize()
    with Server(eng, 1 << 30, n_streams=2, batch_window_us=200_000) as srv:
        for t in [srv.submit_beamform(geom, q, o, **kw) for q, o in zip(iqs, outs)]:
            assert srv.wait(t, 60.0) == 0
        assert srv.stats().launches == 1
    for o, r in zip(outs, refs):
        assert torch.equal(o, r) and float(r.abs().max()) > 0.0
