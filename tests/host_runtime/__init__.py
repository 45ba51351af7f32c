"""librcabf's host code on the CPU: geometry.cpp, api.cpp and server.cpp built
with the stand-in runtime and launchers of fake_runtime.cpp."""
import ctypes as C
import shutil
import subprocess
import warnings
from pathlib import Path

import numpy as np

from simu_rca_ab_b200 import _lib as L
from simu_rca_ab_b200.build import CSRC, CUDA_HOME, HOST_CXX, INCLUDE

HERE = Path(__file__).resolve().parent
WS = C.c_void_p(1 << 20)     # a workspace, input and output address: never read


def build(out_dir) -> Path:
    lib = Path(out_dir) / "librcabf_host.so"
    src = [CSRC / n for n in ("api.cpp", "geometry.cpp", "server.cpp")] + [HERE / "fake_runtime.cpp"]
    # (-Bsymbolic: its own runtime, not the one PyTorch has loaded)
    flags = ["-O1", "-Wl,-Bsymbolic", "-std=c++17", "-fPIC", "-shared", "-I", str(CSRC), "-I", str(INCLUDE),
             "-I", f"{CUDA_HOME}/include"]
    subprocess.run([HOST_CXX, *flags, *map(str, src), "-o", str(lib), "-lpthread"], check=True)
    return lib


class Host:
    """A private copy of the built library: its own caches and log."""

    _copies = 0

    def __init__(self, lib: Path):
        Host._copies += 1
        own = lib.with_name(f"{lib.stem}_{Host._copies}.so")
        shutil.copy(lib, own)
        self.lib = C.CDLL(str(own))
        for name, (res, args) in L._SIGS.items():
            if hasattr(self.lib, name):
                getattr(self.lib, name).restype, getattr(self.lib, name).argtypes = res, args

    def geometry(self, G, T, P, O):
        from simu_rca_ab_b200.beamformer import _desc_from_acq
        from simu_rca_ab_b200.params import normalize
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            acq = normalize(np.zeros(1, np.complex64), G, T, P, O)
        d, keep = _desc_from_acq(acq)
        p = C.c_void_p()
        assert self.lib.rcabf_create_geometry(C.byref(d), None, C.byref(p)) == 0
        p.n_tx, p.n_ele, p.keep = acq.n_tx, acq.n_ele, keep
        return p

    def args(self, g, n_frame, n_sample, *, storage=L.STORE_F32, compound=True, fb=0, kernel=L.KERNEL_AUTO,
             workspace=1 << 60):
        a = L.BeamformArgs()
        a.struct_size = C.sizeof(L.BeamformArgs)
        a.iq_dtype = L.IQ_C64
        a.iq = a.out = a.workspace = WS.value
        a.n_sample, a.n_ch, a.n_tx, a.n_frame = n_sample, g.n_ele, g.n_tx, n_frame
        a.storage, a.compound, a.kernel, a.frames_per_block = storage, int(compound), kernel, fb
        a.workspace_bytes = workspace
        return a

    def plan(self, g, a):
        import json
        buf = C.create_string_buffer(1024)
        s = self.lib.rcabf_describe_plan(g, C.byref(a), buf, 1024)
        return json.loads(buf.value.decode()) if s == 0 else s

    def workspace(self, g, a):
        n = C.c_size_t()
        assert self.lib.rcabf_beamform_workspace_size(g, C.byref(a), C.byref(n)) == 0
        return n.value

    def beamform(self, g, a):
        return self.lib.rcabf_beamform(g, C.byref(a), None)

    def beamform_host(self, g, a, chunk):
        """The call with exactly the workspace it asks for."""
        n = C.c_size_t()
        s = self.lib.rcabf_beamform_host_workspace_size(g, C.byref(a), chunk, C.byref(n))
        if s != 0:
            return s
        a.workspace_bytes = n.value
        self.lib.fake_set_copies(0)
        try:
            return self.lib.rcabf_beamform_host(g, C.byref(a), chunk, None)
        finally:
            self.lib.fake_set_copies(1)

    def batch(self, gs, args):
        arr = (L.BeamformArgs * len(gs))(*args)
        return self.lib.rcabf_beamform_batch(len(gs), (C.c_void_p * len(gs))(*[g.value for g in gs]), arr, None)

    def log(self):
        """The launches since the last call, a line each."""
        buf = C.create_string_buffer(1 << 16)
        self.lib.fake_take_log(buf, 1 << 16)
        return buf.value.decode().splitlines()


def acquisition(nz, nx, ny, span_deg, *, n_tx=5, n_ele=24, shift=0.0, interp=("lanczos", 4), tables="exact",
                depth=(4e-3, 6e-3), points=False):
    """Geometry / Transmit / Param / Options of a small probe; `shift` moves the
    grid off the probe's centre (no mirror symmetry)."""
    from simu_rca_ab_b200 import workloads as W
    X, Y, Z = W.make_grid(nx, ny, nz, 7.2e-3, 7.2e-3, *depth)
    if points:
        rng = np.random.default_rng(0)
        X, Y, Z = (rng.uniform(lo, hi, (nz, 1, 1)) for lo, hi in ((-3e-3, 3e-3), (-3e-3, 3e-3), (4e-3, 8e-3)))
    pos, zero = W.rca_probe(n_ele, 0.3e-3), np.zeros(n_ele)
    th = np.deg2rad(np.linspace(-span_deg, span_deg, n_tx)) if n_tx > 1 else np.zeros(1)
    G = {"gridBfX": X + shift, "gridBfY": Y + shift, "gridBfZ": Z, "posEleX": pos, "posEleY": zero, "posEleZ": zero,
         "apertureX": 7e-3, "apertureY": 7e-3, "apertureZ": 0.0}
    T = {"thetaX": np.zeros(n_tx), "thetaY": th, "flagReceiveX": True}
    P = {"samplingFrequency": 15.6e6, "demodulationFrequency": 7.8e6, "speedOfSound": 1540.0, "startTime": -4e-6,
         "fnumber": 1.0}
    O = {"interpolation": interp[0], "lanczosOrder": interp[1], "flagMaskTransmit": False, "tableMode": tables}
    return G, T, P, O
