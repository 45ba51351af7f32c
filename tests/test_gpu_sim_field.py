"""The simulator's element field (rcabf_sim_element_field) against its model in
FP64, with and without attenuation strong enough to leave the series of
cosh / sinh, directivity arguments across the main lobe and past it, focused
and flat elevation, with and without a baffle.

Tolerance: k r stays below 200 rad and takes four FP32 roundings (r, k, their
product, the sum of the exponent), 1.2e-5 rad each; the beam expansion sums
terms of magnitude up to 2 to about 1 (a factor of 8 on FP32 rounding, 1e-6), and
near the edge of the main lobe sin(z) loses |z| / |sin z|.  Relative RMS over the
field: at most 1e-4.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GA = [0.187 + 0.275j, 0.288 - 1.954j, 0.187 - 0.275j, 0.288 + 1.954j]
GB = [4.558 - 25.59j, 8.598 - 7.924j, 4.558 + 25.59j, 8.598 + 7.924j]


def _flat(theta, k, width, baffle):
    z = 0.5 * np.sin(theta) * width * k
    with np.errstate(divide="ignore", invalid="ignore"):
        s = np.where(z == 0, 1.0, np.sin(z) / z)
    s = np.where(np.abs(z) < np.pi, s, 0.0)
    return s * np.cos(theta) if baffle else s


def _field(scat, ele, k, width, height, foc, baffle):
    out = 0
    kk = k[:, None, None]
    for q in range(ele.shape[0]):
        d = [scat[i][:, None] - ele[q, i][None, :] for i in range(3)]
        r = np.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        az, el = np.arcsin(d[0] / r) - ele[q, 3], np.arcsin(d[1] / r) - ele[q, 4]
        side = _flat(az, kk, width, baffle)
        if foc > 10:
            beam = _flat(el, kk, width, baffle)
        else:
            y = r * np.sin(el)
            al, be, ga = 1j * kk * (r - foc) / (2 * r * foc), -1j * kk * y / r, 1j * kk * y * y / (2 * r)
            beam = sum(A * np.sqrt(np.pi / (B / height ** 2 + al)) * np.exp(be ** 2 / (4 * (B / height ** 2 + al)) + ga)
                       for A, B in zip(GA, GB))
        out = out + np.exp(1j * kk * r) / r * side * beam
    return out


@pytest.mark.parametrize("attenuation", [0.0, 1e-3, 0.15])
@pytest.mark.parametrize("foc", [20e-3, 100.0])
@pytest.mark.parametrize("baffle,width", [(0, 0.27e-3), (1, 2.0e-3)])
def test_element_field_vs_fp64(cuda, attenuation, foc, baffle, width):
    import torch
    from simu_rca_ab_b200.simulator import _element_field
    rng = np.random.default_rng(4)
    n_s, n_e, n_q, n_f = 37, 19, 3, 23
    scat = np.stack([rng.uniform(-3e-3, 3e-3, n_s), rng.uniform(-3e-3, 3e-3, n_s), rng.uniform(2e-3, 5e-3, n_s)])
    scat = scat.astype(np.float32)
    ele = np.zeros((n_q, 5, n_e), np.float32)
    ele[:, 0] = np.linspace(-2e-3, 2e-3, n_e)
    ele[:, 1] = np.linspace(-1e-3, 1e-3, n_q)[:, None]
    k = (np.linspace(0, 3e4, n_f) * (1 + 1j * attenuation)).astype(np.complex64)
    trans = {"ElementWidth": width, "ElementHeight": 2e-3, "ElementElevationFocus": foc, "baffle": baffle,
             "lensCorrection": 0.0}
    dev = torch.device("cuda")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    out = _element_field(dev, t(scat), t(ele), t(k), trans, 1540.0, torch.cuda.current_stream().cuda_stream)
    ref = _field(scat.astype(np.float64), ele.astype(np.float64), k.astype(np.complex128), width, 2e-3, foc, baffle)
    err = np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err < 1e-4, err
