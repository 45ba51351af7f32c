"""Performance cases of the RCA beamformer and of the steps around it.

Each case is a call a user's program makes again and again on new channel
data, with the geometry (delay and apodisation tables) and the acquisition
parameters in hand:

  beamform  Engine.beamform on device-resident channel data (streaming use),
            one receive orientation or the row + column pair summed into one
            volume
  dropin    bf_rca(data, Geometry, Transmit, Param, Options), the reference
            wrapper's call, exact or reference-compatible tables
  nosum     bf_rca_nosum, one value per receive element (dataset producer)
  clutter   svd_clutter_filter of a beamformed ensemble
  simulate  sim_us_rca, the producer of the channel data

Channel data are band-limited speckle (a 2-cycle pulse at f0, demodulated)
with an attenuation along the record, common to the frames, plus a fluctuating
part and -30 dB of white noise.
"""
import math
import warnings

import numpy as np
import torch

from simu_rca_ab_b200 import _lib as L
from simu_rca_ab_b200 import workloads as W
from simu_rca_ab_b200.beamformer import bf_rca, bf_rca_nosum, default_engine
from simu_rca_ab_b200.clutter import keep_components, svd_clutter_filter
from simu_rca_ab_b200.params import normalize
from simu_rca_ab_b200.simulator import sim_plan, sim_us_rca

C = 1540.0
# interpolation -> (name, Lanczos order, taps before n0, taps)
INTERP = {"quad": ("quadratic", 3, 1, 3), "ref6": ("ref6", 3, 2, 6), "l2": ("lanczos", 2, 1, 4),
          "l3": ("lanczos", 3, 2, 6), "l4": ("lanczos", 4, 3, 8)}
STORAGE = {"float32": L.STORE_F32, "float16": L.STORE_F16, "bfloat16": L.STORE_BF16}
EXACT_UNITS = 1.2e9      # voxel.rx.tx.frame above which the 64-bit model takes too long


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def _bf(name, family="beamform", **kw):
    """A beamforming case: the 64+64 (0.3 mm) or larger (0.2 mm) RCA probe, a
    grid of nz x nx x ny voxels over the probe's field of view."""
    c = {"name": name, "family": family, "probe": 64, "n_tx": 16, "span_deg": 8.0, "n_frame": 1, "n_sample": 512,
         "nz": 128, "nx": 64, "ny": 64, "f0": 7.8e6, "fs": 15.6e6, "z0": 5e-3, "z_span": 20e-3, "fnumber": 1.5,
         "interp": "l3", "storage": "float32", "both": False, "receive_x": True, "mask_tx": False,
         "tables": "exact"}
    c.update(kw)
    return c


def listed():
    return [
        # a live view while the probe is positioned: one frame, few transmits, the smallest serving grid
        _bf("live frame", n_tx=4, nz=64, nx=32, ny=32),
        # one compounded volume of the 64+64 probe
        _bf("single volume"),
        # the reference wrapper's own call and defaults: quadratic interpolation, transmit cone mask, two frames
        _bf("drop-in defaults", family="dropin", n_tx=8, n_frame=2, nz=67, nx=61, ny=53, interp="quad", mask_tx=True),
        # the same call where a user needs the reference kernel's bits (its 6-tap interpolation)
        _bf("reference tables", family="dropin", nz=96, nx=48, ny=48, interp="ref6", tables="ref_compat"),
        # a short burst of volumes, row and column transmits compounded
        _bf("volume burst", probe=128, span_deg=10.0, n_frame=8, n_sample=1024, nz=256, nx=128, ny=128, z_span=25e-3,
            fnumber=1.2, interp="l4", both=True),
        # one request of a serving mix: a middle-sized grid, a frame count that fills no block
        _bf("serving request", probe=128, n_tx=8, span_deg=10.0, n_frame=20, n_sample=1024, nz=159, nx=95, ny=97,
            z_span=25e-3, receive_x=False),
        # the largest probe and record, few frames, half-precision channel data, the central depths of its volume
        _bf("large probe", probe=256, n_tx=32, span_deg=12.0, n_frame=4, n_sample=2048, nz=96, nx=256, ny=256, f0=5e6,
            fs=10e6, z0=20e-3, z_span=10e-3, fnumber=1.0, interp="l4", storage="float16"),
        # a Doppler ensemble
        _bf("doppler ensemble", probe=128, n_tx=11, span_deg=5.0, n_frame=200, n_sample=768, nz=160, nx=96, ny=96,
            z_span=25e-3, fnumber=1.2, interp="l4", storage="float16"),
        # a shorter ensemble on a smaller grid, bfloat16 channel data
        _bf("short ensemble", probe=128, n_tx=11, span_deg=5.0, n_frame=60, n_sample=768, nz=125, nx=61, ny=63,
            z_span=25e-3, fnumber=1.2, interp="l4", storage="bfloat16"),
        # the aberration data set's call: a line of 17 depths, every receive element, 100 frames
        _bf("per-channel line", family="nosum", n_frame=100, nz=17, nx=1, ny=1, mask_tx=True, interp="l3"),
        # the clutter filter of the Doppler ensemble
        {"name": "clutter filter", "family": "clutter", "n_frame": 200, "nz": 160, "nx": 96, "ny": 96, "lo": 0.1,
         "hi": 0.9, "kind": "band"},
        # simulated channel data of a small phantom
        {"name": "simulate", "family": "simulate", "n_ele": 64, "n_sub": 8, "n_tx": 16, "n_scat": 200, "n_frame": 2,
         "n_sample": 1024, "moving": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["beamform"] * 7 + ["dropin"] * 2 + ["nosum", "clutter", "simulate"])
    if family == "clutter":
        return {"family": family, "n_frame": _log_int(rng, 24, 200), "nz": rng.randint(48, 160),
                "nx": rng.randint(24, 96), "ny": rng.randint(24, 96), "lo": round(rng.uniform(0.04, 0.25), 3),
                "hi": round(rng.uniform(0.7, 1.0), 3), "kind": rng.choice(["band", "high"])}
    if family == "simulate":
        return {"family": family, "n_ele": rng.choice([32, 48, 64]), "n_sub": rng.randint(4, 8),
                "n_tx": rng.randint(1, 18), "n_scat": _log_int(rng, 20, 200), "n_frame": rng.randint(1, 2),
                "n_sample": rng.choice([512, 640, 1024]), "moving": rng.random() < 0.2}
    probe = rng.choice([64, 64, 128, 128, 192, 256])
    small = probe == 64
    ns = rng.choice([512, 600] if small else [768, 1000, 1024])
    if probe > 128:
        ns = rng.choice([1536, 2048])
    fs, f0 = (10e6, 5e6) if probe > 128 else (15.6e6, 7.8e6)
    z0 = round(rng.uniform(4e-3, 8e-3), 5)
    # the deepest voxel's round trip stays inside the record
    z_span = round(0.75 * ns / fs * C / 2 * rng.uniform(0.6, 0.9), 5)
    c = dict(family=family, probe=probe, n_tx=_log_int(rng, 1, 32), span_deg=round(rng.uniform(3.0, 12.0), 2),
             n_sample=ns, fs=fs, f0=f0, z0=z0, z_span=z_span, fnumber=round(rng.uniform(1.0, 2.0), 2),
             receive_x=rng.random() < 0.7)
    if family == "nosum":
        c.update(n_tx=_log_int(rng, 4, 32), n_frame=_log_int(rng, 10, 128), nz=rng.randint(5, 40), nx=1, ny=1,
                 mask_tx=rng.random() < 0.5, interp=rng.choice(["quad", "ref6", "l3"]), probe=rng.choice([64, 128]))
        c["n_sample"], c["fs"], c["f0"], c["z_span"] = 512, 15.6e6, 7.8e6, min(c["z_span"], 15e-3)
        return _drawn(c)
    c.update(nz=rng.randint(48, 192), nx=rng.randint(24, 128), ny=rng.randint(24, 128), mask_tx=rng.random() < 0.3,
             interp=rng.choice(["l3", "l3", "l4", "l4", "l2", "ref6", "quad"]))
    if family == "dropin":
        ref = rng.random() < 0.5
        c.update(n_frame=rng.randint(1, 4), tables="ref_compat" if ref else "exact",
                 interp=rng.choice(["quad", "ref6"]) if ref else c["interp"], n_tx=_log_int(rng, 1, 16))
        limit = 4e9
    else:
        nf = rng.choice([1, _log_int(rng, 1, 16), _log_int(rng, 1, 31), _log_int(rng, 32, 200)])
        c.update(n_frame=nf, storage=rng.choice(["float32", "float32", "float16", "bfloat16"]),
                 both=rng.random() < 0.25)
        limit = 8e9 if nf == 1 else 6e10
    while c["nz"] * c["nx"] * c["ny"] * probe * c["n_tx"] * c["n_frame"] * (2 if c.get("both") else 1) > limit:
        if c["n_tx"] > 4:
            c["n_tx"] -= max(1, c["n_tx"] // 4)
        else:
            k = rng.choice(["nx", "ny", "nz"])
            c[k] = max(9, int(c[k] * 0.8))
    return _drawn(c)


def _drawn(c):
    d = _bf("", **c)
    del d["name"]
    return d


# --------------------------------------------------------------------------
# Beamforming
# --------------------------------------------------------------------------
def _axes(case):
    """Lateral and depth coordinates (m) of the case's grid."""
    pitch = 0.3e-3 if case["probe"] == 64 else 0.2e-3
    lat = case["probe"] * pitch
    x = (np.arange(case["nx"]) - (case["nx"] - 1) / 2.0) * (lat / case["nx"])
    y = (np.arange(case["ny"]) - (case["ny"] - 1) / 2.0) * (lat / case["ny"])
    z = case["z0"] + np.arange(case["nz"]) * (case["z_span"] / case["nz"])
    return pitch, x, y, z


def _orientations(case):
    return [True, False] if case["both"] else [bool(case["receive_x"])]


def _angles(case):
    return np.deg2rad(np.linspace(-case["span_deg"], case["span_deg"], case["n_tx"])) if case["n_tx"] > 1 else np.zeros(1)


def _structs(case, receive_x):
    """The reference wrapper's Geometry, Transmit, Param and Options."""
    pitch, x, y, z = _axes(case)
    X, Z, Y = np.meshgrid(x, z, y)
    pos = W.rca_probe(case["probe"], pitch)
    zero, th = np.zeros(case["probe"]), _angles(case)
    ap = (case["probe"] - 1) * pitch
    G = {"gridBfX": X, "gridBfY": Y, "gridBfZ": Z, "posEleX": pos if receive_x else zero,
         "posEleY": zero if receive_x else pos, "posEleZ": zero, "apertureX": ap, "apertureY": ap, "apertureZ": 0.0}
    T = {"thetaX": np.zeros_like(th) if receive_x else th, "thetaY": th if receive_x else np.zeros_like(th),
         "flagReceiveX": receive_x}
    P = {"samplingFrequency": case["fs"], "demodulationFrequency": case["f0"], "speedOfSound": C,
         "startTime": -(2 * case["z0"] / C - 16 / case["fs"]), "fnumber": case["fnumber"]}
    name, order, _, _ = INTERP[case["interp"]]
    O = {"flagCompounding": True, "flagMaskTransmit": case["mask_tx"], "interpolation": name, "lanczosOrder": order,
         "storage": case["storage"], "tableMode": case["tables"]}
    return G, T, P, O


def _speckle(case, gen):
    """Channel data [frame][transmit][element][sample] complex64 on the GPU."""
    dev = gen.device
    shape = (case["n_tx"], case["probe"], case["n_sample"])
    sigma = 0.85 / case["f0"] * case["fs"]
    k = int(math.ceil(3 * sigma))
    env = [math.exp(-0.5 * (i / sigma) ** 2) for i in range(-k, k + 1)]
    norm = math.sqrt(sum(e * e for e in env))
    decay = torch.exp(-1.5 * torch.arange(shape[-1], device=dev) / shape[-1])

    def band(*lead):
        w = torch.randn(*lead, *shape[:-1], shape[-1] + 2 * k, dtype=torch.complex64, device=dev, generator=gen)
        out = torch.zeros(*lead, *shape, dtype=torch.complex64, device=dev)
        for i, e in enumerate(env):
            out.add_(w[..., i:i + shape[-1]], alpha=e / norm)
        return out.mul_(decay)

    tissue = band()
    data = torch.randn(case["n_frame"], *shape, dtype=torch.complex64, device=dev, generator=gen).mul_(0.03)
    data.add_(tissue)
    if case["n_frame"] > 1:      # a part of its own in each frame, made a few frames at a time
        for f in range(0, case["n_frame"], 16):
            data[f:f + 16].add_(band(min(16, case["n_frame"] - f)), alpha=0.1)
    return data


def _matlab(iq):
    """[frame][tx][element][sample] -> the reference's [samples, channels, 1, events] indexing."""
    f, t, e, s = iq.shape
    return iq.view(f * t, 1, e, s).permute(3, 2, 1, 0)


def _prepare_bf(case, gen):
    data = []
    for _ in _orientations(case):
        iq = _speckle(case, gen)
        if case["storage"] == "float16":
            iq = iq.to(torch.complex32)
        elif case["storage"] == "bfloat16":
            iq = torch.view_as_real(iq).to(torch.bfloat16)
        data.append(iq)
    structs = [_structs(case, rx) for rx in _orientations(case)]
    if case["family"] != "beamform":
        return {"case": case, "data": _matlab(data[0]), "structs": structs[0]}
    eng = default_engine()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        geoms = [eng.geometry(normalize(np.zeros(1, np.complex64), *s)) for s in structs]
    return {"case": case, "data": data, "engine": eng, "geoms": geoms}


def _run_bf(state):
    case = state["case"]
    if case["family"] != "beamform":
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            return (bf_rca if case["family"] == "dropin" else bf_rca_nosum)(state["data"], *state["structs"])
    eng, geoms, data = state["engine"], state["geoms"], state["data"]
    store = STORAGE[case["storage"]]
    dtype = {"float32": L.IQ_C64, "float16": L.IQ_C32, "bfloat16": L.IQ_BF16X2}[case["storage"]]
    if case["storage"] == "bfloat16":
        # pairs of bfloat16: the buffer's element count is twice the samples'
        out = torch.empty((case["n_frame"], 1, geoms[0].n_pix), dtype=torch.complex64, device=eng.device)
        mask = torch.empty((1, geoms[0].n_pix), dtype=torch.float32, device=eng.device)
        first = 0
    else:
        out, mask = eng.beamform(geoms[0], data[0], storage=store, iq_dtype=dtype)
        first = 1
    for k in range(first, len(geoms)):      # further orientations are added to the volume
        a = eng.make_args(geoms[k], data[k], iq_dtype=dtype, n_sample=case["n_sample"], n_frame=case["n_frame"],
                          out=out, mask=mask, compound=True, storage=store, accumulate=k > 0)
        eng.run(geoms[k], a)
    return out, mask


def _cone(vl, vz, half, p, z):
    """Whether (p, z) lies inside the transmit cone through the aperture's edges."""
    def angle(bx, cx, cz):
        abx, abz, acx, acz = bx - vl, -vz, cx - vl, cz - vz
        return np.arccos(np.clip((abx * acx + abz * acz) / np.sqrt((abx ** 2 + abz ** 2) * (acx ** 2 + acz ** 2)), -1, 1))
    whole = angle(-half, half, 0.0)
    return (angle(-half, p, z) <= whole) & (angle(half, p, z) <= whole)


def _weights(interp, d):
    """Interpolation weight of each tap at fractional offset d (float64)."""
    _, a, lo, taps = INTERP[interp]
    if interp == "quad":
        return [d * (d - 1) / 2, (1 - d) * (1 + d), d * (d + 1) / 2]
    a = 2 if interp == "ref6" else a      # the reference's 6 taps carry a sinc(x) sinc(x / 2) kernel
    return [torch.sinc(d + (lo - j)) * torch.sinc((d + (lo - j)) / a) for j in range(taps)]


def _exact_bf(case, seed):
    """Delay and sum in 64 bits: [frame][u][v][z] volumes (or per channel and
    transmit) and the apodisation sum."""
    if _units(case) > EXACT_UNITS:
        return None
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    state = _prepare_bf(case, gen)
    data = state["data"]
    if case["family"] != "beamform":
        d = data.permute(3, 2, 1, 0)
        data = [d.reshape(case["n_frame"], case["n_tx"], case["probe"], case["n_sample"])]
    data = [torch.view_as_complex(d.double()) if case["storage"] == "bfloat16" else d.to(torch.complex64).to(torch.complex128)
            for d in data]
    pitch, x, y, z = _axes(case)
    pos = W.rca_probe(case["probe"], pitch)
    ap = (case["probe"] - 1) * pitch
    fs, fd, t0, ns = case["fs"], case["f0"], -(2 * case["z0"] / C - 16 / case["fs"]), case["n_sample"]
    _, _, lo, taps = INTERP[case["interp"]]
    nosum = case["family"] == "nosum"
    F, T, E = case["n_frame"], case["n_tx"], case["probe"]
    dd = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    total, mask_total = None, None
    for rx, iq in zip(_orientations(case), data):
        u, v = (x, y) if rx else (y, x)
        th = _angles(case)
        vz = -10.0 / np.sqrt(1 + np.tan(th) ** 2)
        vv = vz * np.tan(th)      # the sources lie off the steering axis v; along u they are centred
        # distance to the nearest element as the wrapper pairs the positions
        md = np.sqrt((pos[None] - vv[:, None]) ** 2 + vz[:, None] ** 2).min(1)
        lat = np.abs(u[None, :, None] - pos[:, None, None])                       # [E, u, 1]
        apf = z / case["fnumber"]
        valid = lat < apf
        apod = dd(np.where(valid, 0.5 * (1 + np.cos(np.pi * lat / apf)), 0.0))    # [E, u, z]
        irx = dd(np.sqrt(lat ** 2 + z ** 2) / C * fs)
        asum = apod.sum(0)                                                        # [u, z]
        shape = (F, u.size, v.size, z.size)
        vol = None if nosum else torch.zeros(shape, dtype=torch.complex128, device=dev)
        per = torch.zeros((E, F, T) + shape[1:], dtype=torch.complex128, device=dev) if nosum else None
        mask = torch.zeros((T,) + shape[1:], dtype=torch.float64, device=dev)
        zz = dd(z)
        step = max(1, int(2e7 // (u.size * v.size * z.size)))
        for t in range(T):
            itx = dd(((np.sqrt((v[:, None] - vv[t]) ** 2 + (z[None] - vz[t]) ** 2) - md[t]) / C + t0) * fs)   # [v, z]
            cone = torch.ones(shape[1:], dtype=torch.bool, device=dev)
            if case["mask_tx"]:
                cone &= dd(_cone(0.0, vz[t], ap / 2, u[:, None], z[None]))[:, None, :]
                cone &= dd(_cone(vv[t], vz[t], ap / 2, v[:, None], z[None]))[None]
            mask[t] = torch.where(cone, asum[:, None, :].expand(shape[1:]), torch.zeros((), dtype=torch.float64, device=dev))
            for e0 in range(0, E, step):
                idx = irx[e0:e0 + step, :, None, :] + itx[None, None]             # [e, u, v, z]
                fl = idx.floor()
                ok = (fl >= lo) & (fl < ns - (taps - lo)) & (apod[e0:e0 + step] > 0)[:, :, None, :] & cone
                n0 = torch.where(ok, fl, torch.full_like(fl, lo)).long() - lo
                w = _weights(case["interp"], idx - fl)
                ph = 2 * math.pi * fd * (idx / fs - 2 * zz / C)
                g = torch.where(ok, apod[e0:e0 + step, :, None, :], torch.zeros((), dtype=torch.float64, device=dev))
                g = torch.polar(g, ph)
                ei = torch.arange(e0, min(E, e0 + step), device=dev)[:, None, None, None] * ns
                for f in range(F):
                    flat = iq[f, t].reshape(-1)
                    s = sum(wj * flat[ei + n0 + j] for j, wj in enumerate(w)) * g
                    if nosum:
                        per[e0:e0 + step, f, t] = s
                    else:
                        vol[f] += s.sum(0)
        res = per if nosum else vol
        mask = mask if nosum else mask.sum(0)
        if rx:      # -> x before y
            pass
        else:
            res = res.transpose(-3, -2)
            mask = mask.transpose(-3, -2)
        total = res if total is None else total + res
        mask_total = mask if mask_total is None else mask_total + mask
    # [.., x, y, z] -> pixel order z fastest, then x, then y
    total, mask_total = total.transpose(-3, -2), mask_total.transpose(-3, -2)
    if case["family"] == "beamform":
        return total.reshape(F, 1, -1), mask_total.reshape(1, -1)
    if nosum:      # [E, F, T, y, x, z] -> [z, x, y, T, F, E]
        return total.permute(5, 4, 3, 2, 1, 0), mask_total.permute(3, 2, 1, 0)
    return total[:, None].permute(4, 3, 2, 1, 0), mask_total[None].permute(3, 2, 1, 0)


def _units(case):
    return (case["nz"] * case["nx"] * case["ny"] * case["probe"] * case["n_tx"] * case["n_frame"]
            * (2 if case["both"] else 1))


def _work_bf(case):
    """Channel data read once and volumes written once; per voxel, element
    inside the f-number aperture, transmit and frame: one complex sample
    interpolated with real weights (4 per tap), rotated (6) and added (2)."""
    pitch, x, y, z = _axes(case)
    pos = W.rca_probe(case["probe"], pitch)
    n_pix = case["nz"] * case["nx"] * case["ny"]
    per_sample = 8 if case["storage"] == "float32" else 4
    taps = INTERP[case["interp"]][3]
    flops = nbytes = 0.0
    for rx in _orientations(case):
        u, nv = (x, case["ny"]) if rx else (y, case["nx"])
        active = int((np.abs(u[None, :, None] - pos[:, None, None]) < z / case["fnumber"]).sum())
        flops += (4.0 * taps + 8) * active * nv * case["n_tx"] * case["n_frame"]
        nbytes += per_sample * case["n_frame"] * case["n_tx"] * case["probe"] * case["n_sample"]
    if case["family"] == "nosum":
        nbytes += 8.0 * n_pix * case["n_frame"] * case["n_tx"] * case["probe"] + 4.0 * n_pix * case["n_tx"]
    else:
        nbytes += 8.0 * n_pix * case["n_frame"] + 4.0 * n_pix
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------------------
# Clutter filter
# --------------------------------------------------------------------------
def _prepare_clutter(case, gen):
    """An ensemble as bf_rca returns it: [Nz, Nx, Ny, frame], each frame's
    voxels contiguous; slowly moving tissue 40 dB above blood, and noise."""
    dev = gen.device
    n_t, n_pix = case["n_frame"], case["nz"] * case["nx"] * case["ny"]
    t = torch.arange(n_t, device=dev) / n_t
    rnd = lambda *s: torch.randn(*s, dtype=torch.complex64, device=dev, generator=gen)
    slow = torch.stack([torch.exp(2j * math.pi * f * t) for f in (0.0, 0.35, -0.4, 0.8, -0.9, 1.3)], 1)
    gain = torch.tensor([100.0, 40.0, 30.0, 10.0, 8.0, 3.0], device=dev)
    blood = torch.stack([torch.exp(2j * math.pi * f * t * n_t / 200) for f in (12.0, 19.0, 27.0, -15.0)], 1)
    x = (slow * gain).to(torch.complex64) @ rnd(6, n_pix)
    x += blood.to(torch.complex64) @ rnd(4, n_pix)
    for f in range(n_t):
        x[f] += 0.3 * rnd(n_pix)
    return {"case": case, "iq": x.view(n_t, case["ny"], case["nx"], case["nz"]).permute(3, 2, 1, 0)}


def _run_clutter(state):
    c = state["case"]
    return svd_clutter_filter(state["iq"], None, (c["lo"], c["hi"]), c["kind"])


def _exact_clutter(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    iq = _prepare_clutter(case, gen)["iq"]
    n_t = case["n_frame"]
    x = iq.permute(3, 2, 1, 0).reshape(n_t, -1)
    gram = torch.zeros((n_t, n_t), dtype=torch.complex128, device=x.device)
    for p in range(0, x.shape[1], 1 << 18):
        xs = x[:, p:p + (1 << 18)].to(torch.complex128)
        gram += xs.conj() @ xs.T
    ev, vec = torch.linalg.eigh(gram)
    ev, vec = ev.flip(0), vec.flip(1)
    keep = torch.from_numpy(keep_components(n_t, (case["lo"], case["hi"]), case["kind"])).to(x.device)
    v = vec[:, keep]
    proj = (v @ v.conj().T).conj()
    out = torch.empty(x.shape, dtype=torch.complex128, device=x.device)
    for p in range(0, x.shape[1], 1 << 18):
        out[:, p:p + (1 << 18)] = proj @ x[:, p:p + (1 << 18)].to(torch.complex128)
    return out.view(n_t, case["ny"], case["nx"], case["nz"]).permute(3, 2, 1, 0), ev


def _work_clutter(case):
    """The ensemble read and written; the Hermitian Gram (half of it) and the
    projection, 8 operations per complex multiply-add."""
    n_t, n_pix = case["n_frame"], case["nz"] * case["nx"] * case["ny"]
    return {"bytes": 16.0 * n_t * n_pix, "flops": 12.0 * n_t * n_t * n_pix}


# --------------------------------------------------------------------------
# Simulator
# --------------------------------------------------------------------------
def _prepare_sim(case, seed):
    """An RCA of n_ele + n_ele strips (n_sub sub-elements each), plane waves,
    point scatterers, static or moving between the events."""
    rng = np.random.default_rng(seed)
    n, q, f0 = case["n_ele"], case["n_sub"], 7.8e6
    pitch = 0.3e-3
    pos = W.rca_probe(n, pitch)
    strip = (np.arange(q) - (q - 1) / 2) * (n * pitch / q)
    tx, rx = np.zeros((n, 5, q)), np.zeros((n, 5, q))
    tx[:, 0, :], tx[:, 1, :] = strip[None], pos[:, None]
    rx[:, 0, :], rx[:, 1, :] = pos[:, None], strip[None]
    t = np.arange(0, 2 / f0, 1 / 250e6)
    ir = np.sin(2 * np.pi * f0 * t) * np.hanning(t.size)
    trans = lambda p: {"frequency": f0, "impulseResponse": ir, "lensCorrection": 0.0, "ElementPos": p,
                       "ElementHeight": 2e-3, "ElementWidth": 0.27e-3, "ElementElevationFocus": 20e-3, "baffle": 1}
    n_event, half = case["n_tx"] * case["n_frame"], n * pitch / 2
    base = np.stack([rng.uniform(-half, half, case["n_scat"]), rng.uniform(-half, half, case["n_scat"]),
                     rng.uniform(5e-3, 20e-3, case["n_scat"]), rng.rayleigh(1.0, case["n_scat"])], 1)
    scat = np.repeat(base[:, :, None], n_event, 2)
    if case["moving"]:
        scat[:, 2] += 2e-6 * np.arange(n_event)
    th = np.deg2rad(np.linspace(-8, 8, case["n_tx"])) if case["n_tx"] > 1 else np.zeros(1)
    TXSI = [{"pulseShape": np.sin(2 * np.pi * f0 * t), "Delay": (pos * np.sin(a) - (pos * np.sin(a)).min()) / C,
             "Apod": np.ones(n)} for a in th]
    RXSI = [{"samplingFrequency": 4 * f0, "demodFrequency": f0, "startTime": 0.0, "numelSample": case["n_sample"],
             "sampleMode": "NS200BW", "InputFilter": np.array([1.0]), "Apod": np.ones(n)} for _ in th]
    return ({"speedOfSound": C, "attenuation": 0.5, "scattererPos": scat}, trans(tx), trans(rx), TXSI, RXSI)


# 4-Gaussian beam expansion of the focused elevation aperture
_GA = [0.187 + 0.275j, 0.288 - 1.954j, 0.187 - 0.275j, 0.288 + 1.954j]
_GB = [4.558 - 25.59j, 8.598 - 7.924j, 4.558 + 25.59j, 8.598 + 7.924j]


def _field(r_scat, ele, k, trans):
    """Element field [f, s, e] in complex128 (the simulator's acoustic model)."""
    width, height, foc = trans["ElementWidth"], trans["ElementHeight"], trans["ElementElevationFocus"]
    kk = k[:, None, None]
    acc = 0
    for q in range(ele.shape[2]):
        d = [r_scat[:, i, None] - ele[None, :, i, q] for i in range(3)]
        r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        az = torch.asin(d[0] / r) - ele[None, :, 3, q]
        el = torch.asin(d[1] / r) - ele[None, :, 4, q]
        arg = kk * (0.5 * torch.sin(az) * width)
        side = torch.where(arg.abs() > 0, torch.sin(arg) / arg, torch.ones_like(arg))
        side = torch.where(arg.abs() < math.pi, side, torch.zeros_like(arg))
        side = side * torch.cos(az) if trans["baffle"] == 1 else side
        y = r * torch.sin(el)
        al, be, ga = 1j * kk * ((r - foc) / (2 * r * foc)), -1j * kk * (y / r), 1j * kk * (y * y / (2 * r))
        foc_sum = 0
        for A, B in zip(_GA, _GB):
            ag = B / height ** 2 + al
            foc_sum = foc_sum + A * torch.sqrt(math.pi / ag) * torch.exp(be * be / (4 * ag) + ga)
        acc = acc + torch.exp(1j * kk * r) / r * side * foc_sum
    return torch.nan_to_num(acc, nan=0.0)


def _exact_sim(case, seed):
    args = _prepare_sim(case, seed)
    p = sim_plan(*args)
    dev = torch.device("cuda")
    dd = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    cc = lambda a: dd(np.asarray(a, np.complex128))
    k, c, n_tx, n_fast, sub, numel = cc(p["k"]), p["c"], p["n_tx"], p["n_fast"], p["sub"], p["numel"]
    w = k.real * c
    txf, rxf = cc(np.conj(p["pulse"]) * np.conj(p["ir_tx"])), cc(p["ipf"] * p["ir_rx"])
    delay, apod, rapod = dd(p["delay"]), dd(p["apod"]), dd(p["rx_apod"])
    tx_ele, rx_ele = dd(p["pos_tx"]), dd(p["pos_rx"])
    scat = dd(p["scat"])
    n_out = 2 * min(-(-numel // sub), -(-(numel - 1) // sub))
    i = torch.arange(n_out, device=dev)
    ts = sub * (i // 2) + i % 2
    fi = torch.arange(p["n_freq"], device=dev)
    tw = torch.polar(torch.ones((), dtype=torch.float64, device=dev).expand(n_out, fi.numel()),
                     (2 * math.pi / n_fast) * ((ts[:, None] * fi[None]) % n_fast).double())
    raw = torch.zeros((p["n_event"], rx_ele.shape[0], n_out), dtype=torch.float64, device=dev)
    for f0 in range(0, p["n_event"], n_tx):
        groups = [[f0 + j] for j in range(n_tx)] if case["moving"] else [list(range(f0, f0 + n_tx))]
        for ev in groups:
            pos = scat[:, :3, ev[0]]
            spec = []
            for fs in torch.arange(p["n_freq"], device=dev).split(16):
                et = _field(pos, tx_ele, k[fs], p["tx"])                         # [f, s, e]
                er = _field(pos, rx_ele, k[fs], p["rx"])
                g = [e - f0 for e in ev]
                wt = torch.polar(apod[:, g].expand(fs.numel(), -1, -1), w[fs][:, None, None] * delay[:, g])
                tx = txf[fs][:, None, None] * (et @ wt) * scat[:, 3, ev][None]    # [f, s, g]
                spec.append(rxf[fs][:, None, None] * rapod[:, g] * (er.transpose(1, 2) @ tx))
            sp = torch.cat(spec).permute(2, 1, 0)                                 # [g, e', f]
            rf = (sp.real @ tw.real.T + sp.imag @ tw.imag.T) / n_fast
            rf[..., ts >= n_fast] = 0
            raw[ev] = rf
    return raw.permute(2, 1, 0).cpu().numpy()


def _work_sim(case):
    """Inputs and Raw once; about 400 operations per element-field term (its
    Green's function, directivities and four complex Gaussians), one complex
    multiply-add per field value and transmit, the inverse transform by FFT."""
    n_samp = case["n_sample"] + 128
    n_freq = n_samp // 2
    terms = 2.0 * n_freq * case["n_scat"] * case["n_ele"]
    groups = case["n_frame"] * (case["n_tx"] if case["moving"] else 1)
    flops = terms * groups * case["n_sub"] * 400 + terms * 8 * case["n_frame"] * case["n_tx"]
    flops += case["n_frame"] * case["n_tx"] * case["n_ele"] * 5.0 * n_samp * math.log2(n_samp)
    nbytes = 4.0 * case["n_frame"] * case["n_tx"] * (case["n_ele"] * case["n_sample"] + 4 * case["n_scat"])
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------------------
def prepare(case, seed):
    if case["family"] == "simulate":
        return {"case": case, "args": _prepare_sim(case, seed)}
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return _prepare_clutter(case, gen) if case["family"] == "clutter" else _prepare_bf(case, gen)


def run(state):
    family = state["case"]["family"]
    if family == "simulate":
        return sim_us_rca(*state["args"])
    return _run_clutter(state) if family == "clutter" else _run_bf(state)


def exact(case, seed):
    if case["family"] == "simulate":
        return _exact_sim(case, seed)
    return _exact_clutter(case, seed) if case["family"] == "clutter" else _exact_bf(case, seed)


def work(case):
    return {"simulate": _work_sim, "clutter": _work_clutter}.get(case["family"], _work_bf)(case)
