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
