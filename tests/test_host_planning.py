"""The host code of librcabf (planning, sizes, dispatch) on the CPU, with the
stand-in runtime of tests/host_runtime: which calls are accepted, with which
kernel, in which order of sums, and with how much scratch memory."""
import pytest

from simu_rca_ab_b200 import _lib as L
from tests.host_runtime import Host, acquisition, build


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    return build(tmp_path_factory.mktemp("host_runtime"))


@pytest.fixture
def host(built):
    return Host(built)


F32, F16, BF16 = L.STORE_F32, L.STORE_F16, L.STORE_BF16


# FP16 and BF16 data run one kernel function where voxels share rows (steering
# spread of at most 2 rows over a voxel block), all three storages where not
@pytest.mark.parametrize("span,stores", [(2.0, (F16, BF16, F16)), (2.0, (BF16, F32, F16, BF16)),
                                         (20.0, (F32, F16, F32)), (30.0, (F16, BF16, F32, F16))])
@pytest.mark.parametrize("n_frame", [2, 4, 8])
def test_shared_memory_limit_is_kept_per_kernel_function(built, span, stores, n_frame):
    """The windows that take the most shared memory, then those that take the
    least on other storages of the same kernel function, then the first again:
    the function's limit stays where the first ones need it."""
    acqs = [acquisition(33, 9, 11, span, shift=1e-3, depth=(4e-3, mm * 1e-3)) for mm in range(1, 13)]

    def plan(acq, store):   # (planning looks the limit up: in a copy of its own)
        h = Host(built)
        g = h.geometry(*acq)
        return h.plan(g, h.args(g, n_frame, 300, storage=store))

    plans = [plan(a, stores[0]) for a in acqs]
    variant = [(p["kernel"], p["row_shift"], p["frames_per_block"]) for p in plans]
    same = [i for i, v in enumerate(variant) if v == variant[0]]
    big, small = (f(same, key=lambda i: plans[i]["smem_bytes"]) for f in (max, min))
    assert variant[0][0] == "fused_voxel_blocked"
    assert plans[big]["smem_bytes"] > plans[small]["smem_bytes"]
    h = Host(built)
    g = {i: h.geometry(*acqs[i]) for i in (big, small)}
    for k, store in enumerate(stores):
        i = big if k in (0, len(stores) - 1) else small
        assert h.beamform(g[i], h.args(g[i], n_frame, 300, storage=store)) == 0, (k, store)


FRAMES_CHUNKS = [(n, c) for n in (2, 4, 9, 13, 16, 18, 20, 31, 36, 40) for c in (0, 1, 2, 3, 5, 7, 8)]


@pytest.mark.parametrize("tables,shift,nz,nx,ny,stores", [
    ("ref_compat", 0.0, 40, 24, 24, (F32,)), ("exact", 0.0, 40, 32, 32, (F32, F16)),
    ("exact", 1e-3, 40, 32, 32, (F32, F16)), ("exact", 0.0, 6, 17, 33, (F32, BF16))])
def test_host_buffer_call_fits_the_workspace_it_asks_for(host, tables, shift, nz, nx, ny, stores):
    """Every chunk of a host-buffer call, the shorter last one too, fits the
    scratch size the call reported, on grids with more voxels than channel
    samples; reference tables keep one kernel for all chunks."""
    g = host.geometry(*acquisition(nz, nx, ny, 2.0, shift=shift, n_ele=8, tables=tables,
                                   interp=("ref6", 3) if tables == "ref_compat" else ("lanczos", 4)))
    for n_frame, chunk in FRAMES_CHUNKS:
        for store in stores:
            for compound in (True, False):
                a = host.args(g, n_frame, 97, storage=store, compound=compound)
                host.log()
                assert host.beamform_host(g, a, chunk) == 0, (n_frame, chunk, store, compound)
                kernels = {line.split()[0] for line in host.log()}
                if tables == "ref_compat":
                    assert kernels == {"ref" if n_frame <= 4 else "fused"}, (n_frame, chunk)


def test_host_buffer_call_on_few_reference_frames_is_one_launch(host):
    """Up to 4 frames share the per-transmit kernel's work: one chunk."""
    g = host.geometry(*acquisition(20, 12, 12, 2.0, n_ele=8, tables="ref_compat", interp=("ref6", 3)))
    for n_frame in (1, 2, 3, 4):
        host.log()
        assert host.beamform_host(g, host.args(g, n_frame, 97), 0) == 0
        assert host.log() == [f"ref 1 frames {n_frame}"]


def _sums(line):
    """What the order and the terms of a launch's sums depend on: the kernel,
    its row sharing and weights, tile, mirrored axes and ranges."""
    w = line.split()
    k = w.index("order")
    return (w[0], w[1], w[2], w[4], w[k + 1])   # (w[3]: the frame block)


@pytest.mark.parametrize("shift", [0.0, 1e-3])
@pytest.mark.parametrize("nz,nx,ny,span", [(33, 9, 21, 2.0), (40, 32, 32, 2.0), (17, 5, 11, 20.0), (18, 9, 6, 30.0),
                                           (6, 17, 33, 3.0)])
@pytest.mark.parametrize("kernel", [L.KERNEL_AUTO, L.KERNEL_FUSED_TMEM, L.KERNEL_FUSED_REGS])
def test_chunks_of_a_host_buffer_call_sum_as_the_whole_call(host, shift, nz, nx, ny, span, kernel):
    """Each chunk, a last one of one frame too, runs the kernel, weights, tile
    and ranges of the call on device buffers."""
    g = host.geometry(*acquisition(nz, nx, ny, span, shift=shift))
    for n_frame, chunk in FRAMES_CHUNKS:
        for store, compound in ((F32, True), (F16, True), (BF16, False)):
            a = host.args(g, n_frame, 180, storage=store, compound=compound, kernel=kernel)
            host.log()
            status = host.beamform(g, a)
            whole = host.log()
            assert host.beamform_host(g, a, chunk) == status, (n_frame, chunk, store)
            chunks = host.log()
            if status == 0 and not whole[0].startswith("tc"):
                assert {_sums(c) for c in chunks} == {_sums(whole[0])}, (n_frame, chunk, store, compound)


@pytest.mark.parametrize("store", [F32, F16, BF16])
@pytest.mark.parametrize("nz,nx,ny", [(33, 9, 21), (40, 32, 32), (80, 48, 48), (6, 17, 33)])
@pytest.mark.parametrize("depth_mm", [3, 9, 20])
def test_full_16_frame_counts_take_16_frame_blocks_or_the_streaming_kernel(host, store, nz, nx, ny, depth_mm):
    """The tensor-memory kernel's blocks of 8 are slower than the streaming
    kernel: no call of 15 frames or more falls to them."""
    g = host.geometry(*acquisition(nz, nx, ny, 2.0, depth=(4e-3, depth_mm * 1e-3)))
    for n_frame in (15, 16, 27, 31):
        p = host.plan(g, host.args(g, n_frame, 700, storage=store))
        assert (p["kernel"], p["frames_per_block"]) in (("fused_voxel_blocked_tmem", 16), ("fused_voxel_blocked", 8)), p


@pytest.mark.parametrize("shift", [0.0, 1e-3])
@pytest.mark.parametrize("nz,nx,ny,depth_mm", [(33, 9, 21, 3), (40, 32, 32, 9), (96, 96, 96, 9), (6, 17, 33, 3)])
@pytest.mark.parametrize("store,compound", [(F32, True), (F16, True), (F32, False)])
def test_frame_blocks_asked_for(host, shift, nz, nx, ny, depth_mm, store, compound):
    """frames_per_block = 16 runs on the tensor-memory kernel as the call that
    leaves it open does, where its blocks are full, voxels share one shift row
    and the tiles fill the GPU, and every block size of a call sums in one order."""
    g = host.geometry(*acquisition(nz, nx, ny, 2.0, shift=shift, depth=(4e-3, depth_mm * 1e-3)))
    for n_frame in (2, 8, 9, 15, 16, 18, 27, 32):
        orders, kernel = set(), {}
        for fb in (0, 2, 4, 8, 16):
            host.log()
            a = host.args(g, n_frame, 700, storage=store, compound=compound, fb=fb)
            assert host.beamform(g, a) == 0
            words = host.log()[0].split()
            kernel[fb] = words[0], words[-1] if words[0] == "tc" else words[3]
            if fb and words[0] != "fused":
                order = words[words.index("order") + 1].split(",")
                orders.add(tuple(order if compound else order[:-2]))   # (ranges only split compounded sums)
        assert len(orders) == 1, (n_frame, orders)
        d = host.plan(g, host.args(g, n_frame, 700, storage=store, compound=compound))["row_shift"]
        if kernel[0] == ("vb", "16") and n_frame % 16 == 0 and d == 1 and nz * nx * ny > 512 * 1184:
            assert kernel[16] == kernel[0], (n_frame, kernel)


# (mirrored grids and others, steps of every steepness, points, one row)
BATCH = [dict(), dict(shift=1e-3), dict(span=20.0), dict(span=30.0), dict(span=30.0, shift=1e-3), dict(points=True),
         dict(ny=1), dict(nz=96, nx=96, ny=72)]


def _batch_geometry(host, kw):
    kw = {"nz": 33, "nx": 9, "ny": 12, "span": 2.0, **kw}
    return host.geometry(*acquisition(kw.pop("nz"), kw.pop("nx"), kw.pop("ny"), kw.pop("span"), **kw))


@pytest.mark.parametrize("fb,accepted", [
    (1, [set(range(len(BATCH)))]),                  # one voxel per thread, or the streaming kernel
    (4, [{0, 1, 7}, {2, 3, 4, 5, 6}]),              # shared rows; wider spreads and grids without a block
    (16, [{0, 1, 7}, {2, 3, 4, 5, 6}])])
def test_batches_take_mirrored_steep_and_other_grids_together(host, fb, accepted):
    """One batch of two or of all grids of a class, each job with the kernel and
    order of sums that it has alone; grids of different classes are refused."""
    gs = [_batch_geometry(host, kw) for kw in BATCH]
    args = [host.args(g, 16 if fb == 16 else 3, 180, fb=fb) for g in gs]
    alone = []
    for g, a in zip(gs, args):
        host.log()
        assert host.beamform(g, a) == 0
        alone.append(host.log()[0].split(" jobs")[0])
    for i in range(len(gs)):
        for k in range(len(gs)):
            ok = any({i, k} <= c for c in accepted)
            host.log()
            assert host.batch([gs[i], gs[k]], [args[i], args[k]]) == (0 if ok else L.ERR_UNSUPPORTED), (i, k)
            if ok:
                want = {alone[i], alone[k]}
                assert sorted(line.split(" jobs")[0] for line in host.log()) == sorted(want), (i, k)
    for c in accepted:
        host.log()
        assert host.batch([gs[i] for i in sorted(c)], [args[i] for i in sorted(c)]) == 0
        assert len(host.log()) == len({alone[i] for i in c})


def test_batch_of_tensor_core_calls_keeps_each_record_length(host):
    """Jobs with records of two lengths have slabs of two heights: a launch each."""
    g = _batch_geometry(host, {})
    args = [host.args(g, 40, ns, storage=F16, kernel=L.KERNEL_FUSED_TC, fb=40) for ns in (180, 180, 300)]
    assert host.batch([g] * 3, args) == 0
    assert [line.split("rows ")[1] for line in host.log()] == ["212 of 180", "212 of 180", "332 of 300"]


def _server(host, n_streams, batch_window_us):
    import ctypes as C
    cfg, srv = L.ServerConfig(), C.c_void_p()
    cfg.struct_size, cfg.hbm_budget_bytes = C.sizeof(cfg), 1 << 28
    cfg.n_streams, cfg.max_queue, cfg.max_batch, cfg.batch_window_us = n_streams, 16, 8, batch_window_us
    assert host.lib.rcabf_server_create(C.byref(cfg), C.byref(srv)) == 0
    return srv


SERVED = [(dict(), 16, F32), (dict(shift=1e-3), 16, F32), (dict(), 31, F32), (dict(), 1, F16), (dict(shift=1e-3), 1, BF16),
          (dict(), 1, F32), (dict(shift=1e-3), 5, F16), (dict(span=30.0), 3, F32), (dict(), 40, F16),
          (dict(tables="ref_compat", interp=("ref6", 3)), 1, F32), (dict(tables="ref_compat", interp=("ref6", 3)), 4, F32),
          (dict(tables="ref_compat", interp=("ref6", 3)), 6, F32), (dict(points=True), 2, F32)]


@pytest.mark.parametrize("kw,n_frame,store", SERVED)
def test_server_runs_equal_requests_in_one_launch_with_the_plan_each_has_alone(host, kw, n_frame, store):
    import ctypes as C
    g = _batch_geometry(host, kw)
    assert host.beamform(g, host.args(g, n_frame, 180, storage=store)) == 0
    alone = host.log()
    srv = _server(host, n_streams=1, batch_window_us=50_000)
    tickets = []
    for k in range(3):
        a, t = host.args(g, n_frame, 180, storage=store), C.c_uint64()
        a.out = (k + 2) << 20        # outputs of their own: requests on one output wait for each other
        assert host.lib.rcabf_server_submit(srv, g, C.byref(a), C.byref(t)) == 0
        tickets.append(t)
    st = C.c_int()
    for t in tickets:
        assert host.lib.rcabf_server_wait_for(srv, t, 20.0, C.byref(st)) == 0 and st.value == 0
    stats = L.ServerStats()
    stats.struct_size = C.sizeof(stats)
    one = not alone[0].startswith("tc")      # (tensor-core requests are launched one by one)
    assert host.lib.rcabf_server_get_stats(srv, C.byref(stats)) == 0 and stats.launches == (1 if one else 3)
    assert host.lib.rcabf_server_destroy(srv) == 0
    assert {line.split(" jobs")[0] for line in host.log()} == {line.split(" jobs")[0] for line in alone}


@pytest.mark.parametrize("kw", [dict(), dict(shift=1e-3), dict(span=20.0), dict(tables="ref_compat", interp=("ref6", 3))])
@pytest.mark.parametrize("kernel", [L.KERNEL_AUTO, L.KERNEL_FUSED_REGS])
def test_calls_whose_storage_type_slabs_fit_run_in_the_static_workspace(host, kw, kernel):
    """A plan with FP32 slabs, or with transmit sums, that exceeds the 64 MiB of
    the call without allocation gives way to one that fits: the tensor-memory
    kernel in the planner's frame blocks or smaller ones, or one voxel per thread."""
    import ctypes as C
    g = _batch_geometry(host, kw)
    ref = "tables" in kw
    if kernel == L.KERNEL_FUSED_REGS and (ref or "span" in kw):
        return
    limit, cut = 64 << 20, 0
    for n_frame in (1, 2, 3, 4, 5, 8, 9, 12, 17, 24):
        for store in (F32,) if ref else (F32, F16, BF16):
            for mb in (20, 40, 60, 63):   # storage-type slabs of about mb MB: one frame block of each size
                block = 1 << (n_frame - 1).bit_length()
                ns = int(mb * 1e6 / (5 * 24 * (block if block <= 16 else 16 * -(-n_frame // 16)) * (8 if store == F32 else 4)))
                fits = []
                for k in (L.KERNEL_FUSED_TMEM,) + (() if kernel == L.KERNEL_FUSED_REGS else (L.KERNEL_FUSED_NOBLOCK,)):
                    for fb in (min(block, 16), 0):
                        a, n = host.args(g, n_frame, ns, storage=store, kernel=k, fb=fb), C.c_size_t()
                        if host.lib.rcabf_beamform_workspace_size(g, C.byref(a), C.byref(n)) == 0:
                            fits.append(n.value <= limit)
                a = host.args(g, n_frame, ns, storage=store, kernel=kernel)
                n = C.c_size_t()
                if not any(fits) or host.lib.rcabf_beamform_workspace_size(g, C.byref(a), C.byref(n)) != 0:
                    continue
                assert host.lib.rcabf_beamform_noalloc(g, C.byref(a), None) == 0, (n_frame, store, mb)
                cut += n.value > limit
    assert cut > 0 or (ref and kernel == L.KERNEL_AUTO)


@pytest.mark.parametrize("kw,n_frame,want", [
    (dict(tables="ref_compat", interp=("ref6", 3)), 1, {("fused", "1")}),
    (dict(tables="ref_compat", interp=("ref6", 3)), 4, {("fused", "4")}),
    (dict(ny=21), 1, {("vbs", "2"), ("vbs", "4"), ("vbs", "8")}), (dict(shift=1e-3), 2, {("vbs", "2"), ("vbs", "4")})])
def test_autotuning_times_the_fused_kernel_and_blocks_of_mirrored_copies(host, kw, n_frame, want):
    import ctypes as C
    g = _batch_geometry(host, kw)
    r = L.TuneResult()
    r.struct_size = C.sizeof(r)
    host.log()
    assert host.lib.rcabf_autotune(g, C.byref(host.args(g, n_frame, 180)), None, 1, C.byref(r)) == 0
    assert want <= {(line.split()[0], line.split()[3]) for line in host.log()}


def test_server_launches_kernels_for_the_first_time_while_others_run(host):
    """The first launch of a kernel waits for the work in flight, whose completion
    takes the server's lock: the scheduler does not hold it meanwhile."""
    import ctypes as C
    g = _batch_geometry(host, {})
    srv = _server(host, n_streams=4, batch_window_us=0)
    tickets, st = [], C.c_int()
    for k, (n_frame, store) in enumerate([(1, F32), (2, F32), (5, F16), (16, F32), (40, F16), (9, BF16)]):
        a, t = host.args(g, n_frame, 180, storage=store), C.c_uint64()
        a.out = (k + 2) << 20
        assert host.lib.rcabf_server_submit(srv, g, C.byref(a), C.byref(t)) == 0
        tickets.append(t)
    for t in tickets:
        assert host.lib.rcabf_server_wait_for(srv, t, 30.0, C.byref(st)) == 0 and st.value == 0
    assert host.lib.rcabf_server_destroy(srv) == 0


def test_server_launch_takes_a_bounded_amount_of_work(host):
    """Requests share a launch up to 3e10 voxel x element x transmit x frame."""
    import ctypes as C
    g = host.geometry(*acquisition(64, 64, 64, 2.0))
    per = 64 ** 3 * 24 * 5 * 64
    assert 14 * per <= 3e10 < 15 * per
    srv, st, tickets = _server(host, n_streams=1, batch_window_us=50_000), C.c_int(), []
    a = host.args(g, 64, 60)
    for k in range(16):
        a.out, t = (k + 2) << 20, C.c_uint64()
        assert host.lib.rcabf_server_submit(srv, g, C.byref(a), C.byref(t)) == 0
        tickets.append(t)
    for t in tickets:
        assert host.lib.rcabf_server_wait_for(srv, t, 30.0, C.byref(st)) == 0 and st.value == 0
    jobs = [int(line.split(" jobs ")[1].split()[0]) for line in host.log()]
    assert sum(jobs) == 16 and max(jobs) * per <= 3e10 and max(jobs) > 1
    assert host.lib.rcabf_server_destroy(srv) == 0
