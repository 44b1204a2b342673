"""Performance cases: the reconstructions and OTFs that a user of this library runs.

A case is one pass through the public Python calls over the C ABI, from raw
images in host memory to the result in host memory, as an acquisition program
or a batch job makes it.  Kinds:

  frame   one 2D acquisition (3 directions x 3 phases), k0 searched
  live    consecutive 2D frames of one acquisition (Reconstructor.process_series), k0 kept from time 0
  volume  one 3D acquisition (3 directions x 5 phases), k0 searched
  series  consecutive 3D time points (process_series), k0 kept from time 0
  sheet   one deskewed light-sheet acquisition (1 direction x 5 phases), k0 searched
  batch   a mixed queue of 2D frames and 3D volumes (Server.run_batch)
  otf     makeotf on a bead stack

Inputs are seeded simulations made on the GPU: beads and filaments imaged with
a scalar widefield PSF under a sinusoidal pattern, Poisson noise on a camera
offset.  Stacks and results are page-locked (host_empty), as in a program that
cares for throughput; the smallest frame, the sheet and makeotf use plain
numpy memory.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn

DEV = "cuda"
F32 = np.float32
NPH = {"2d": 3, "3d": 5}
#: per pattern direction, rad
ANGLES = (-0.8043, -1.8555, 0.2388)
#: 2D: a value whose float32 bits end in zeros, so that kz = 0 (all there is in 2D) is kept
WIENER_2D = 0.00048828125
WIENER_3D = 0.001
DESKEW_DEG = 31.8
OTF_ARGS = ["-angle", "-0.8043", "-ls", "0.2035", "-xyres", "0.08", "-zres", "0.125", "-na", "1.42", "-nimm", "1.515",
            "-wavelength", "528", "-beaddiam", "0.1", "-fixorigin", "3", "20"]


def _f(v):
    return float(F32(v))


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a live preview on a cropped camera field: the smallest call, all latency
        {"name": "frame_128", "kind": "frame", "nx": 128, "ny": 128, "dtype": "u16", "pinned": False},
        # the ordinary 2D acquisition
        {"name": "frame_512", "kind": "frame", "nx": 512, "ny": 512, "dtype": "u16", "pinned": True},
        # a large 2D field already converted to float32 (flat-fielded elsewhere), not square
        {"name": "frame_1024x960_f32", "kind": "frame", "nx": 1024, "ny": 960, "dtype": "f32", "pinned": True},
        # a 2D time lapse replayed in one call
        {"name": "live_512_n16", "kind": "live", "nx": 512, "ny": 512, "n": 16, "dtype": "u16", "pinned": True},
        # a small ragged 3D crop, few sections, odd section count
        {"name": "volume_96x80x9_f32", "kind": "volume", "nx": 96, "ny": 80, "nz": 9, "dtype": "f32", "pinned": True},
        # the ordinary standalone volume
        {"name": "volume_256x32", "kind": "volume", "nx": 256, "ny": 256, "nz": 32, "dtype": "u16", "pinned": True},
        # a ragged crop of a large field
        {"name": "volume_640x384x30", "kind": "volume", "nx": 640, "ny": 384, "nz": 30, "dtype": "u16",
         "pinned": True},
        # the largest: a whole camera field, precision configuration
        {"name": "volume_1024x64", "kind": "volume", "nx": 1024, "ny": 1024, "nz": 64, "dtype": "u16",
         "pinned": True},
        # the benchmark's time series
        {"name": "series_512x48_n4", "kind": "series", "nx": 512, "ny": 512, "nz": 48, "n": 4, "dtype": "u16",
         "pinned": True},
        # light sheet: sheared sections, one pattern direction
        {"name": "sheet_256x192x40", "kind": "sheet", "nx": 256, "ny": 192, "nz": 40, "dtype": "u16",
         "pinned": False},
        # a queue of small jobs of several shapes
        {"name": "batch_mixed", "kind": "batch", "nx": 512, "ny": 512, "nz": 24, "frames": 12, "volumes": 4,
         "dtype": "u16", "pinned": True},
        # the OTF made once per objective and colour
        {"name": "otf_128x64", "kind": "otf", "nx": 128, "ny": 128, "nz": 64},
    ]


def _good(n, even=True):
    """The size nearest to n (from below) that factors into 2, 3, 5 and 7."""
    def ok(v):
        for p in (2, 3, 5, 7):
            while v % p == 0:
                v //= p
        return v == 1
    n = int(n)
    while n > 1 and (not ok(n) or (even and n % 2)):
        n -= 1
    return n


def _deskewed(nx, nz):
    """The width that deskewing gives sections of nx columns (any that covers them and transforms well)."""
    o = _optics(False)
    return _good(nx + nz * abs(math.cos(_f(DESKEW_DEG) * math.pi / 180.0)) * _f(o.dz) / _f(o.dxy), False)


def draw(rng):
    def size(lo, hi, even=True):
        return _good(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.99))), even)
    kind = rng.choice(["frame", "live", "volume", "volume", "series", "sheet", "batch", "otf"])
    dtype = rng.choice(["u16", "u16", "f32"])
    pinned = rng.random() < 0.7
    if kind == "frame":
        return {"kind": kind, "nx": size(128, 1024), "ny": size(128, 1024), "dtype": dtype, "pinned": pinned}
    if kind == "live":
        return {"kind": kind, "nx": size(128, 768), "ny": size(128, 768), "n": rng.randint(2, 24), "dtype": dtype,
                "pinned": pinned}
    if kind == "volume":
        return {"kind": kind, "nx": size(96, 640), "ny": size(80, 640), "nz": size(9, 64, False), "dtype": dtype,
                "pinned": pinned}
    if kind == "series":
        return {"kind": kind, "nx": size(96, 512), "ny": size(80, 512), "nz": size(9, 48, False),
                "n": rng.randint(2, 5), "dtype": dtype, "pinned": pinned}
    if kind == "sheet":
        nx, nz = size(160, 512), size(16, 60, False)
        while _deskewed(nx, nz) % 2:
            nx -= 2
        return {"kind": kind, "nx": nx, "ny": size(128, 512), "nz": nz, "dtype": dtype, "pinned": pinned}
    if kind == "batch":
        return {"kind": kind, "nx": size(192, 640), "ny": size(192, 640), "nz": size(9, 32, False),
                "frames": rng.randint(2, 16), "volumes": rng.randint(1, 5), "dtype": dtype, "pinned": pinned}
    n = size(96, 160)
    return {"kind": kind, "nx": n, "ny": n, "nz": size(24, 72, False)}


# ------------------------------------------------------------ acquisitions
def _optics(twod):
    return syn.Optics(nphases=NPH["2d" if twod else "3d"], angles=ANGLES)


@lru_cache(maxsize=4)
def _otf_pages(twod, dz):
    if twod:
        return syn.ra_otf(_optics(True), nx_psf=128, norders=2, twod=True)
    return syn.ra_otf(_optics(False), nx_psf=128, nz_psf=64, dz_psf=dz)


def _geometry(case):
    """What the acquisition is, in the units of its configuration."""
    twod = case["kind"] in ("frame", "live")
    sheet = case["kind"] == "sheet"
    o = _optics(twod)
    g = {"nx_raw": case["nx"], "nx": case["nx"], "ny": case["ny"], "nz": 1 if twod else case["nz"], "twod": twod,
         "ndirs": 1 if sheet else 3, "nph": o.nphases, "norders": o.nphases // 2 + 1, "dz": F32(o.dz), "shear": 0.0,
         "dzpsf": o.dz}
    extra = {}
    if twod:
        extra["wiener"] = WIENER_2D
    if sheet:
        rad = DESKEW_DEG * math.pi / 180.0
        ang = float(F32(DESKEW_DEG)) * math.pi / 180.0
        g["nx"] = _deskewed(g["nx_raw"], g["nz"])
        g["shear"] = F32(math.cos(ang) * float(F32(o.dz)) / float(F32(o.dxy)))
        g["dz"] = F32(float(F32(o.dz)) * abs(math.sin(ang)))
        g["dzpsf"] = round(o.dz * math.sin(rad), 6)
        extra.update(ndirs=1, k0angles="%.6f" % ANGLES[0], deskew=DESKEW_DEG)
    g["config"] = syn.config_text(o, twod=twod, extra=extra, dz_psf=g["dzpsf"])
    g["otf"] = _otf_pages(twod, g["dzpsf"])
    return g


def _simulate(g, seed, n=1):
    """n consecutive stacks (float32 on the GPU, [ndirs * nz * nph][ny][nx_raw]) of one drifting, bleaching scene."""
    o = _optics(g["twod"])
    nx, ny, nz, nph = g["nx"], g["ny"], g["nz"], g["nph"]
    dz = float(g["dz"])
    gen = torch.Generator(DEV).manual_seed(int(seed))

    def uni(*shape):
        return torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64)

    # beads: uniform positions, lognormal brightness; filaments: smooth random walks
    nb = max(60, int(0.5 * nx * ny * nz * o.dxy * o.dxy * dz))
    pos = uni(nb, 3)
    val = torch.exp(0.3 * torch.randn(nb, generator=gen, device=DEV, dtype=torch.float64))
    turn = torch.cumsum(0.3 * torch.randn(30, 200, generator=gen, device=DEV, dtype=torch.float64), 1)
    turn = turn + 2 * math.pi * uni(30, 1)
    step = 0.05 / o.dxy
    walk = torch.stack([torch.cumsum(step * torch.cos(turn), 1) / nx, torch.cumsum(step * torch.sin(turn), 1) / ny,
                        0.002 * torch.cumsum(uni(30, 200) - 0.5, 1)], -1) + uni(30, 1, 3)
    pos = torch.cat([pos, walk.reshape(-1, 3)])
    val = torch.cat([val, torch.full((30 * 200,), 0.3, device=DEV, dtype=torch.float64)])
    m1 = 0.5 + 0.4 * uni(g["ndirs"]).cpu().numpy()
    m2 = 0.4 + 0.4 * uni(g["ndirs"]).cpu().numpy()
    # the PSF's transform
    kx = torch.fft.fftfreq(nx, d=o.dxy, device=DEV, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, d=o.dxy, device=DEV, dtype=torch.float64)
    kr2 = ky[:, None] ** 2 + kx[None, :] ** 2
    pupil = (kr2 <= (o.na / o.lambda_em) ** 2).double()
    kz = torch.sqrt(torch.clamp((o.nimm / o.lambda_em) ** 2 - kr2, min=0))
    zs = torch.fft.fftfreq(nz, d=1.0 / nz, device=DEV, dtype=torch.float64) * dz
    psf = torch.empty(nz, ny, nx, device=DEV)
    for i in range(nz):
        psf[i] = torch.fft.ifft2(pupil * torch.exp(2j * math.pi * kz * zs[i])).abs().square().float()
    psf /= psf.sum()
    otf0 = torch.fft.fftn(psf)
    otf1 = torch.fft.fftn(psf * torch.cos(2 * math.pi * o.kz1() * zs).float()[:, None, None]) if nz > 1 else otf0
    x = (torch.arange(nx, device=DEV, dtype=torch.float64) * o.dxy)[None, :]
    y = (torch.arange(ny, device=DEV, dtype=torch.float64) * o.dxy)[:, None]
    shift = None
    if g["shear"]:  # section z of the raw stack starts at another x
        c = nx / 2.0 - g["nx_raw"] / 2.0 + float(g["shear"]) * (torch.arange(nz, device=DEV) - nz / 2.0)
        shift = torch.exp(2j * math.pi * torch.fft.fftfreq(nx, device=DEV)[None, :] * c[:, None])[:, None, :]
    stacks = []
    for t in range(n):
        scene = torch.zeros(nz * ny * nx, device=DEV, dtype=torch.float64)
        xi = torch.floor(torch.remainder(pos[:, 0] * nx + 0.2 * t, nx)).long().clamp(max=nx - 1)
        yi = torch.floor(torch.remainder(pos[:, 1], 1.0) * ny).long().clamp(max=ny - 1)
        zi = torch.floor(torch.remainder(pos[:, 2], 1.0) * nz).long().clamp(max=nz - 1)
        # whole counts: the order of the additions does not matter
        scene.index_add_(0, (zi * ny + yi) * nx + xi, torch.round(val * 1024 * 0.99 ** t))
        scene = scene.reshape(nz, ny, nx).float()

        def image(weight, otf):
            f = torch.fft.fftn(scene if weight is None else scene * weight) * otf
            im = torch.fft.ifftn(f).real
            return im if shift is None else torch.fft.ifft(torch.fft.fft(im, dim=2) * shift, dim=2).real

        base = image(None, otf0)
        raw = torch.empty(g["ndirs"], nz, nph, ny, g["nx_raw"], device=DEV)
        for d in range(g["ndirs"]):
            k = 1.0 / (2.0 * o.ls) if nz > 1 else 1.0 / o.ls
            arg = 2 * math.pi * k * (math.cos(ANGLES[d]) * x + math.sin(ANGLES[d]) * y)
            # order 1 moves with the focal plane in 3D; 2D has order 1 alone
            c1, s1 = image(torch.cos(arg).float(), otf1), image(torch.sin(arg).float(), otf1)
            c2, s2 = (image(torch.cos(2 * arg).float(), otf0), image(torch.sin(2 * arg).float(), otf0)) \
                if nz > 1 else (None, None)
            scale = 1000.0 * 0.99 ** t / (float(base.max()) * (1 + m1[d] + m2[d]))
            for p in range(nph):
                phi = 2 * math.pi * p / nph
                im = base + m1[d] * (math.cos(phi) * c1 - math.sin(phi) * s1)
                if nz > 1:
                    im = im + m2[d] * (math.cos(2 * phi) * c2 - math.sin(2 * phi) * s2)
                im = torch.poisson((im * scale).clamp(min=0), generator=gen) + 100.0
                raw[d, :, p] = im[:, :, :g["nx_raw"]]
        stacks.append(raw.reshape(-1, ny, g["nx_raw"]).clamp(max=32767))
    return stacks


def _host(shape, dtype, pinned):
    return sr.host_empty(shape, dtype) if pinned else np.zeros(shape, dtype)


def _to_host(stack, case):
    """A simulated stack in the host memory and type that the camera program has it in."""
    if case["dtype"] == "u16":
        a = _host(tuple(stack.shape), np.uint16, case["pinned"])
        torch.from_numpy(a.view(np.int16)).copy_(stack.to(torch.int16))
    else:
        a = _host(tuple(stack.shape), np.float32, case["pinned"])
        torch.from_numpy(a).copy_(stack)
    return a


def _bead_stack(case, seed):
    """Bead PSF sections on the GPU, float32 [nz * 5][ny][nx], phase fastest."""
    o = _optics(False)
    nx, ny, nz, nph = case["nx"], case["ny"], case["nz"], 5
    gen = torch.Generator(DEV).manual_seed(int(seed))
    off = (torch.rand(3, generator=gen, device=DEV).double() * 0.8 - 0.4).cpu().numpy()
    phase = 0.3
    psf = torch.from_numpy(syn.widefield_psf(nx, ny, nz, o)).to(DEV)
    fx, fy, fz = (torch.fft.fftfreq(n, device=DEV, dtype=torch.float64) for n in (nx, ny, nz))
    move = torch.exp(-2j * math.pi * (fx[None, None, :] * (nx // 2 + off[0]) + fy[None, :, None] * (ny // 2 + off[1]) +
                                      fz[:, None, None] * (nz // 2 + off[2])))
    zs = torch.fft.fftfreq(nz, d=1.0 / nz, device=DEV, dtype=torch.float64) * o.dz
    det0 = torch.fft.ifftn(torch.fft.fftn(psf) * move).real
    det1 = torch.fft.ifftn(torch.fft.fftn(psf * torch.cos(2 * math.pi * o.kz1() * zs)[:, None, None]) * move).real
    out = torch.empty(nz, nph, ny, nx, device=DEV, dtype=torch.float64)
    for p in range(nph):
        phi = 2 * math.pi * p / nph
        out[:, p] = det0 * (1 + 0.8 * math.cos(2 * phi + 2 * phase)) + 0.9 * math.cos(phi + phase) * det1
    out *= 1e5 / out.max()
    return (torch.poisson(out.clamp(min=0).float(), generator=gen) + 100.0).reshape(nz * nph, ny, nx)


# ------------------------------------------------------------------ passes
def _batch_parts(case):
    """(2D case, smaller 2D case, 3D case) of a batch."""
    two = {**case, "kind": "frame"}
    small = {**two, "nx": _good(case["nx"] * 3 / 4), "ny": _good(case["ny"] * 3 / 4)}
    vol = {**case, "kind": "volume", "nx": _good(case["nx"] / 2), "ny": _good(case["ny"] / 2)}
    return two, small, vol


def _out_shape(g):
    return (g["nz"], 2 * g["ny"], 2 * g["nx"])


def prepare(case, seed):
    sr.load_library()
    kind = case["kind"]
    if kind == "otf":
        return {"kind": kind, "psf": _bead_stack(case, seed).cpu().numpy()}
    if kind == "batch":
        parts = _batch_parts(case)
        geo = [_geometry(c) for c in parts]
        srv = sr.Server(workers=6, hbm_budget=60e9)
        cfg2 = srv.add_config(geo[0]["config"], geo[0]["otf"])
        cfg3 = srv.add_config(geo[2]["config"], geo[2]["otf"])
        items = []
        for i in range(case["frames"] + case["volumes"]):
            k = 2 if i * case["volumes"] // (case["frames"] + case["volumes"]) != \
                (i + 1) * case["volumes"] // (case["frames"] + case["volumes"]) else i % 2
            raw = _to_host(_simulate(geo[k], seed * 1000 + i)[0], parts[k])
            items.append((cfg3 if k == 2 else cfg2, raw, _host(_out_shape(geo[k]), np.float32, case["pinned"])))
        for cfg, g in ((cfg2, geo[0]), (cfg2, geo[1]), (cfg3, geo[2])):
            srv.reserve(cfg, g["nx"], g["ny"], g["ndirs"] * g["nph"] * g["nz"], 2)
        return {"kind": kind, "server": srv, "items": items}
    g = _geometry(case)
    n = case.get("n", 0)
    raws = [_to_host(s, case) for s in _simulate(g, seed, 1 + n)]
    r = sr.Reconstructor(g["nx_raw"], g["ny"], raws[0].shape[0], g["config"], g["otf"])
    outs = [_host(r.out_shape, np.float32, case["pinned"]) for _ in range(max(1, n))]
    if n:  # time 0 fits k0; the passes reconstruct the time points after it
        r.set_ntimes(1000)
        r.set_raw(raws[0])
        r.load_and_rescale(0, 0)
        r.set_cur_time(0)
        r.process()
    return {"kind": kind, "r": r, "raws": raws, "outs": outs, "n": n}


def run(state):
    if state["kind"] == "otf":
        return sr.make_otf(state["psf"], OTF_ARGS)
    if state["kind"] == "batch":
        state["server"].run_batch(state["items"])
        return [out for _, _, out in state["items"]]
    r = state["r"]
    if state["n"]:
        r.process_series(state["raws"][1:], state["outs"], t0=1)
        return state["outs"]
    r.set_raw(state["raws"][0])
    r.load_and_rescale(0, 0)
    r.set_cur_time(0)
    r.process()
    out = r.result(state["outs"][0])
    k0, amps = r.fit()
    return {"volume": out, "k0": k0, "amps": amps}


def work(case):
    """Raw stack read and result written once; the transforms of a reconstruction at 5 n log2 n."""
    kind = case["kind"]
    if kind == "batch":
        two, small, vol = _batch_parts(case)
        w = {"bytes": 0.0, "flops": 0.0}
        nsmall = case["frames"] // 2
        for c, n in ((two, case["frames"] - nsmall), (small, nsmall), (vol, case["volumes"])):
            for k, v in work(c).items():
                w[k] += n * v
        return w
    if kind == "otf":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 4.0 * 5 * n + 3 * (case["nx"] // 2 + 1) * 2 * case["nz"] * 4.0,
                "flops": 5 * 2.5 * n * math.log2(n)}
    g = _geometry(case)
    n = g["nx"] * g["ny"] * g["nz"]
    images = g["ndirs"] * g["nph"]
    raw = images * g["nx_raw"] * g["ny"] * g["nz"] * (2.0 if case["dtype"] == "u16" else 4.0)
    # forward: real transforms of every image; back: one complex transform of the
    # doubled grid per direction and order, the bands filling half of x and y
    fwd = images * 2.5 * n * math.log2(n)
    back = (1 + g["ndirs"] * (g["norders"] - 1)) * 5.0 * 2 * n * math.log2(2 * n)
    reps = max(1, case.get("n", 0))
    return {"bytes": reps * (raw + 4.0 * 4 * n), "flops": reps * (fwd + back)}


# ------------------------------------------------------------- 64-bit values
def _parabola(a1, a2, a3):
    curve = (a3 + a1) - 2 * a2
    if curve == 0:
        return 0.0
    peak = -0.5 * (a3 - a1) / curve
    return 0.0 if abs(peak) > 1.5 else peak


class _Exact:
    """One acquisition's reconstruction in 64-bit torch.

    Everything is written on the full complex spectrum P_o(k) of order o of a
    direction, the transform of sum_j image_j exp(i j o phi).  Numbers whose
    rounding decides something (supports, plane counts, the angles and
    magnitudes that the search visits) are formed in float32, as the method
    defines them; all else is 64-bit.
    """

    def __init__(self, g, twod_wiener):
        self.g = g
        o = _optics(g["twod"])
        self.nx, self.ny, self.nz = g["nx"], g["ny"], g["nz"]
        self.nd, self.nph, self.no = g["ndirs"], g["nph"], g["norders"]
        self.dxy, dz = F32(o.dxy), g["dz"]
        na, nimm, wave = F32(o.na), F32(o.nimm), o.wave_nm
        self.wiener = F32(twod_wiener)
        # the flag that drops kz = 0 also reads the low half of the Wiener constant's bits
        self.nokz0 = int(np.array([self.wiener], np.float32).view(np.uint32)[0]) & 0xFFFF != 0
        self.dkx, self.dky = F32(1) / (F32(self.nx) * self.dxy), F32(1) / (F32(self.ny) * self.dxy)
        dkz = F32(1) / (F32(self.nz) * dz)
        pages = g["otf"]
        if g["twod"]:
            self.nzotf, self.nrotf, dkzotf = 1, pages.shape[2] // 2, F32(1)
        else:
            self.nzotf, self.nrotf = pages.shape[2] // 2, pages.shape[1]
            dkzotf = F32(1) / (F32(g["dzpsf"]) * F32(self.nzotf))
        self.dkr = F32(1) / (self.dxy * F32(self.nrotf - 1) * F32(2))
        self.kzscale = float(F32(dkz / dkzotf))
        c = torch.from_numpy(pages.astype(np.float64)).to(DEV).reshape(pages.shape[0], self.nrotf, self.nzotf, 2)
        c = torch.view_as_complex(c.contiguous())
        self.otf = [c[min(i, c.shape[0] - 1)] if i < c.shape[0] else c[0] for i in range(self.no)]
        cut = F32(float(na) * 2.0 / (wave * 0.001))
        self.cut = cut if float(cut) <= 1 / (2 * float(self.dxy)) else F32(1 / (2 * float(self.dxy)))
        lam = F32(F32(wave) / nimm / 1000.0)
        alpha = F32(math.asin(float(F32(na / nimm))))
        cosa = F32(math.cos(float(alpha)))
        zmax = max(self.nz // 2 - 1, 0)
        z = math.ceil((1.0 - float(cosa)) / float(lam) / float(dkz))
        self.zov = zmax if z > self.nz // 2 else z
        z0 = math.ceil(float(F32(F32(F32(1) - cosa) / lam) / dkz))
        zdc = [z0] * self.no
        zdc[-1] = int(1.3 * z0)
        for i in range(1, self.no - 1):
            zdc[i] = int(F32(F32(1) + lam / F32(0.88 * lam)) * F32(z0))
        self.zdc = [zmax if v >= self.nz // 2 else v for v in zdc]
        mag = F32(F32(1) / F32(o.ls))
        if self.nz > 1:
            mag = F32(mag / F32(self.nph // 2))
        ang = [F32(float("%.6f" % a)) for a in ANGLES[:self.nd]]
        self.guess = [(_f(mag * math.cos(float(a))), _f(mag * math.sin(float(a)))) for a in ang]
        self.fo2 = 2 if self.nz > 1 else 1
        # signed frequency indices of the full grid, the Nyquist one positive
        self.jx = torch.arange(self.nx, device=DEV)
        self.jx = torch.where(self.jx > self.nx // 2, self.jx - self.nx, self.jx)
        self.jy = torch.arange(self.ny, device=DEV)
        self.jy = torch.where(self.jy > self.ny // 2, self.jy - self.ny, self.jy)

    # ---- images -> spectra
    def load(self, raw):
        g, nx, ny, nz, nph = self.g, self.nx, self.ny, self.nz, self.nph
        insc = float(F32(1.0 / (nx * ny * nz * 4.0 * self.nd)))
        raw = raw.reshape(self.nd, nz, nph, ny, g["nx_raw"])
        fact = torch.tensor([_f(1.0 - _f(math.sin(_f((l + 0.5) / 10.0 * math.pi * 0.5)))) for l in range(10)],
                            device=DEV, dtype=torch.float64)
        ref = None
        self.P = []
        for d in range(self.nd):
            im = (raw[d].double() - 100.0) * insc
            if g["shear"]:
                im = self._deskew(im)
            sums = im.sum((2, 3))
            if d == 0:
                ref = sums[:, 0].clone()
            im = im * (ref[:, None] / sums)[:, :, None, None]
            diff = (im[..., -1, :] - im[..., 0, :]) / 2
            im[..., :10, :] += diff[..., None, :] * fact[:, None]
            im[..., ny - 10:, :] -= diff[..., None, :] * fact.flip(0)[:, None]
            diff = (im[..., -1] - im[..., 0]) / 2
            im[..., :10] += diff[..., None] * fact
            im[..., nx - 10:] -= diff[..., None] * fact.flip(0)
            row = []
            for o in range(self.no):
                w = torch.tensor([complex(_f(math.cos(j * o * _f(2 * math.pi / nph))),
                                          _f(math.sin(j * o * _f(2 * math.pi / nph)))) for j in range(nph)],
                                 device=DEV, dtype=torch.complex128)
                s = torch.zeros(nz, ny, nx, device=DEV, dtype=torch.complex128)
                for j in range(nph):
                    s += im[:, j] * w[j]
                row.append(torch.fft.fftn(s))
            self.P.append(row)

    def _deskew(self, im):
        g, nz = self.g, self.nz
        xo = np.arange(self.nx, dtype=np.float64)
        out = torch.zeros(nz, self.nph, self.ny, self.nx, device=DEV, dtype=torch.float64)
        nr = g["nx_raw"]
        for z in range(nz):
            xin = (xo - self.nx / 2.0 - float(g["shear"]) * (z - nz / 2.0) + nr / 2.0).astype(np.float32)
            m = (xin >= 0) & (xin < nr)
            i0 = np.floor(xin).astype(np.int64).clip(0, nr - 1)
            off = torch.from_numpy((xin - np.floor(xin)).astype(np.float64)).to(DEV)
            i0t = torch.from_numpy(i0).to(DEV)
            # the pixel after a row's last one is the next row's first
            flat = torch.cat([im[z].reshape(self.nph, -1),
                              torch.zeros(self.nph, 1, device=DEV, dtype=torch.float64)], 1)
            at = torch.arange(self.ny, device=DEV)[:, None] * nr + i0t[None, :]
            v = (1 - off) * flat[:, at] + off * flat[:, at + 1]
            out[z] = v * torch.from_numpy(m.astype(np.float64)).to(DEV)
        return out

    # ---- OTF of `order` at radii r2d [ny][nx] and planes z [n] -> [n][ny][nx]
    def _otf(self, order, r2d, z):
        kzi = z.double() * self.kzscale
        kzi = torch.where(kzi < 0, kzi + self.nzotf, kzi)
        iz = torch.floor(kzi).long()
        az = (kzi - iz)[:, None]
        t = self.otf[order].T  # [kz][kr]
        nxt = torch.where(iz == self.nzotf - 1, torch.zeros_like(iz), iz + 1)
        t = t[iz] * (1 - az) + t[nxt % self.nzotf] * az
        kri = r2d / float(self.dkr)
        ir = torch.floor(kri).long()
        ar = kri - ir
        last = self.nrotf - 1
        return t[:, ir.clamp(max=last)] * (1 - ar) + t[:, (ir + 1).clamp(max=last)] * ar

    def _rad(self, kx=0.0, ky=0.0):
        """Radii about (-kx, -ky): 64-bit, and as the method rounds them."""
        x = self.jx.double() * float(self.dkx) + kx
        y = self.jy.double() * float(self.dky) + ky
        r = torch.sqrt(y[:, None] ** 2 + x[None, :] ** 2)
        xf = self.jx.float() * float(self.dkx) + torch.tensor(kx, dtype=torch.float32, device=DEV)
        yf = self.jy.float() * float(self.dky) + torch.tensor(ky, dtype=torch.float32, device=DEV)
        return r, torch.sqrt(xf[None, :] * xf[None, :] + yf[:, None] * yf[:, None])

    # ---- the fit
    def _overlaps(self, d, o1, o2, k0):
        kx, ky = _f(F32(k0[0]) * F32(o2 - o1)), _f(F32(k0[1]) * F32(o2 - o1))
        f02 = 5.0 if self.nz > 1 else 1.0
        z = torch.arange(-self.zov, self.zov + 1, device=DEV)
        if self.nokz0:
            z = z[z != 0]
        otfcut = _f(0.006)
        cut = float(self.cut)
        r, rf = self._rad()
        xy = torch.zeros(self.ny, self.nx, device=DEV, dtype=torch.complex128)
        ov = []
        for a, b, sign in ((o1, o2, -1.0), (o2, o1, 1.0)):
            rs, rsf = self._rad(sign * kx, sign * ky)
            ok = ((rf <= cut) if sign < 0 else (rf < cut)) & (rsf <= cut)
            own, other = self._otf(a, r, z), self._otf(b, rs, z)
            f1, f2 = (1.0, f02) if sign < 0 else (f02, 1.0)
            ok = ok & (own.abs() * f1 > otfcut) & (other.abs() * f2 > otfcut)
            root = torch.sqrt(own.abs().square() + other.abs().square())
            w = torch.where(ok, other / torch.where(root > 0, root, torch.ones_like(root)), 0)
            # planes left out are zero: Parseval along z
            ov.append(torch.fft.ifft2(self.P[d][a][z % self.nz] * w) * (self.nx * self.ny))
        xy = (ov[0].conj() * ov[1]).sum(0) * self.nz
        return xy, float(ov[0].abs().square().sum() * self.nz)

    def _modamp(self, xy, sx, o1, o2, k):
        kx, ky = _f(F32(k[0]) * F32(o2 - o1)), _f(F32(k[1]) * F32(o2 - o1))
        ex = torch.exp(2j * math.pi * (torch.arange(self.nx, device=DEV).double() - 0.5 * self.nx) * kx *
                       float(self.dxy))
        ey = torch.exp(2j * math.pi * (torch.arange(self.ny, device=DEV).double() - 0.5 * self.ny) * ky *
                       float(self.dxy))
        return complex((ey @ (xy @ ex)).item()) / sx

    def _findk0(self, d):
        k0 = self.guess[d]
        xy, _ = self._overlaps(d, 0, self.fo2, k0)
        cc = torch.fft.fft2(xy.conj()).abs().square()
        at = int(torch.argmax(cc.reshape(-1)))
        iy, ix = divmod(at, self.nx)
        v = lambda yy, xx: float(cc[yy % self.ny, xx % self.nx])  # noqa: E731
        px = _parabola(v(iy, ix - 1), v(iy, ix), v(iy, ix + 1)) + ix
        py = _parabola(v(iy - 1, ix), v(iy, ix), v(iy + 1, ix)) + iy
        gx, gy = k0[0] / float(self.dkx), k0[1] / float(self.dky)
        px += self.nx * ((gx > px + self.nx // 2) - (gx < px - self.nx // 2))
        py += self.ny * ((gy > py + self.ny // 2) - (gy < py - self.ny // 2))
        return _f(px * float(self.dkx) / self.fo2), _f(py * float(self.dky) / self.fo2)

    def _search(self, d):
        k = self._findk0(d)
        mag = F32(math.sqrt(k[0] * k[0] + k[1] * k[1]))
        ang = F32(math.atan2(k[1], k[0]))

        def vec(a, m):
            return _f(m * F32(math.cos(float(a)))), _f(m * F32(math.sin(float(a))))

        xy, sx = self._overlaps(d, 0, self.fo2, vec(ang, mag))

        def amp2(a, m):
            v = self._modamp(xy, sx, 0, self.fo2, vec(a, m))
            return F32(v.real * v.real + v.imag * v.imag)

        def climb(f, start, step):
            x2, y2 = start, f(start)
            x3 = F32(start + step)
            y3 = f(x3)
            if not y3 > y2:  # the other way
                step, (x2, y2), (x3, y3) = F32(-step), (x3, y3), (x2, y2)
            x1, y1 = F32(0), F32(0)
            while y3 > y2:
                x1, y1, x2, y2 = x2, y2, x3, y3
                x3 = F32(x3 + step)
                y3 = f(x3)
            if x1 == x2 or x2 == x3 or x3 == x1:
                return F32(0)
            b1, b2 = F32(0.5) * (x1 + x2), F32(0.5) * (x2 + x3)
            s1, s2 = (y2 - y1) / (x2 - x1), (y3 - y2) / (x3 - x2)
            curve = (s2 - s1) / (b2 - b1)
            return F32(0) if curve == 0 else F32(b2 - s2 / curve)

        ang = climb(lambda a: amp2(a, mag), ang, F32(0.001))
        mag = climb(lambda m: amp2(ang, m), mag, F32(0.1 / (max(self.nx, self.ny) * float(self.dxy))))
        k = vec(ang, mag)
        amps = [complex(1)] + [0j] * (self.no - 1)
        amps[self.fo2] = self._modamp(xy, sx, 0, self.fo2, k)
        for o in range(1, self.no):
            if o != self.fo2:
                xy, sx = self._overlaps(d, 0, o, k)
                amps[o] = self._modamp(xy, sx, 0, o, k)
        return k, amps

    def fit(self, k0=None):
        """k0 searched, or kept: the amplitudes then at the given one."""
        self.k0, self.amps = [], []
        for d in range(self.nd):
            if k0 is None:
                k, amps = self._search(d)
            else:
                k, amps = k0[d], [complex(1)]
                for o in range(1, self.no):
                    xy, sx = self._overlaps(d, 0, o, k)
                    amps.append(self._modamp(xy, sx, 0, o, k))
            self.k0.append(k)
            self.amps.append(amps)

    # ---- Wiener filter and assembly
    def volume(self):
        nx, ny, nz, no = self.nx, self.ny, self.nz, self.no
        X, Y = 2 * nx, 2 * ny
        cut = float(self.cut)
        dkx, dky = F32(1.0 / (nx * float(self.dxy))), F32(1.0 / (ny * float(self.dxy)))
        dk = float(min(dkx, dky))
        supp_r = float(F32(10) * F32(dk))
        damped0 = not self.g["twod"]  # dampenOrder0 is set for 3D
        k0mag = _f(math.sqrt(self.k0[0][0] ** 2 + self.k0[0][1] ** 2))
        apocut, zapocut = cut + k0mag * (no - 1), self.zdc[1]
        a2 = [[abs(a) ** 2 for a in amps] for amps in self.amps]
        out = torch.zeros(nz, Y, X, device=DEV, dtype=torch.float64)

        def singular(r, rf, w, z, order):
            """The weight of a band near its centre."""
            if order == 0 and damped0:
                w = w * ((r / cut) ** 2 + (z.abs() / float(self.zdc[0])).abs()[:, None, None] ** 3)
            else:
                x = r / dk
                s = 1.0 / (1.0 + 20000.0 / (x ** 6 + 20.0))
                w = w * torch.where(rf <= supp_r, s, torch.ones_like(s))
            if order == 0 and self.nokz0:
                w = w * (z != 0).double()[:, None, None]
            return w

        jx, jy = torch.remainder(self.jx, X), torch.remainder(self.jy, Y)
        for order in range(no):
            z = torch.arange(-self.zdc[order], self.zdc[order] + 1, device=DEV)
            for d in range(self.nd):
                kx, ky = _f(F32(order) * F32(self.k0[d][0])), _f(F32(order) * F32(self.k0[d][1]))
                r, rf = self._rad()
                rabs, _ = self._rad(kx, ky)
                own = self._otf(order, r, z)
                damp = singular(r, rf, torch.ones(len(z), 1, 1, device=DEV, dtype=torch.float64), z, order)
                total = own.abs().square() * (a2[d][order] if order else 1.0) * damp
                for d2 in range(self.nd):
                    for o2 in range(-(no - 1), no):
                        if (d2, o2) == (d, order):
                            continue
                        sx = _f(F32(kx) - F32(F32(o2) * F32(self.k0[d2][0])))
                        sy = _f(F32(ky) - F32(F32(o2) * F32(self.k0[d2][1])))
                        r2, r2f = self._rad(sx, sy)
                        w = self._otf(abs(o2), r2, z).abs().square() * (a2[d2][abs(o2)] if o2 else 1.0)
                        total += torch.where(r2f < cut, singular(r2, r2f, w, z, abs(o2)), 0.0)
                scale = damp * own.conj() / (total + float(F32(self.wiener * self.wiener)))
                rho = (rabs / apocut) ** 2
                if zapocut > 0:
                    rho = rho + (z.abs() / float(zapocut))[:, None, None] ** 2
                scale = scale * (1 - torch.sqrt(rho).clamp(max=1.0))
                if order:
                    scale = scale * np.conj(self.amps[d][order])
                v = torch.where(rf <= cut, self.P[d][order][z % nz] * scale, 0)
                if order == 0:  # the half spectrum is scaled, the other half is its conjugate
                    neg = torch.nonzero(self.jx < 0).reshape(-1)
                    back = torch.remainder(-torch.arange(ny, device=DEV), ny)
                    v[:, :, neg] = v.flip(0)[:, back][:, :, nx - neg].conj()
                big = torch.zeros(nz, Y, X, device=DEV, dtype=torch.complex128)
                big[(z % nz)[:, None, None], jy[None, :, None], jx[None, None, :]] = v
                del v, total, scale, own
                big = torch.fft.ifftn(big) * float(nz * Y * X)
                if order == 0:
                    out += big.real
                    continue
                k0x, k0y = _f(F32(self.k0[d][0]) * F32(order)), _f(F32(self.k0[d][1]) * F32(order))
                px = (torch.arange(X, device=DEV).double() - nx) * (2 * math.pi * k0x * _f(self.dxy / F32(2)))
                py = (torch.arange(Y, device=DEV).double() - ny) * (2 * math.pi * k0y * _f(self.dxy / F32(2)))
                out += 2.0 * (big * torch.exp(1j * px)[None, None, :] * torch.exp(1j * py)[None, :, None]).real
        return out


def _exact_single(case, stack):
    g = _geometry(case)
    e = _Exact(g, WIENER_2D if g["twod"] else WIENER_3D)
    e.load(stack)
    e.fit()
    return e


def _exact_otf(psf, case):
    nx, ny, nz, nph, no = case["nx"], case["ny"], case["nz"], 5, 3
    p = psf.double().reshape(nz, nph, ny, nx)
    dr, dz, ls, ang, dia = _f(0.08), _f(0.125), _f(0.2035), _f(-0.8043), _f(0.1)
    x, y = torch.arange(nx, device=DEV), torch.arange(ny, device=DEV)
    edge = (x < 20)[None, :] | (x > nx - 20)[None, :] | (y < 20)[:, None] | (y > ny - 20)[:, None]
    bg = p[:, :, edge].mean(-1)
    fact = torch.tensor([_f(1.0 - math.sin((l + 0.5) / 10.0 * math.pi * 0.5)) for l in range(10)], device=DEV,
                        dtype=torch.float64)
    diff = (p[..., -1, :] - p[..., 0, :]) / 2
    p[..., :10, :] += diff[..., None, :] * fact[:, None]
    p[..., ny - 10:, :] -= diff[..., None, :] * fact.flip(0)[:, None]
    diff = (p[..., -1] - p[..., 0]) / 2
    p[..., :10] += diff[..., None] * fact
    p[..., nx - 10:] -= diff[..., None] * fact.flip(0)
    avg = p.mean(1)
    at = int(torch.argmax(avg.reshape(-1)))
    k, rest = divmod(at, ny * nx)
    i, j = divmod(rest, nx)
    v = lambda a, b, c: float(avg[a % nz, b % ny, c % nx])  # noqa: E731
    zc = k + _parabola(v(k - 1, i, j), v(k, i, j), v(k + 1, i, j))
    yc = i + _parabola(v(k, i - 1, j), v(k, i, j), v(k, i + 1, j))
    xc = j + _parabola(v(k, i, j - 1), v(k, i, j), v(k, i, j + 1))
    p -= bg[:, :, None, None]
    nxh = nx // 2 + 1

    def signed(n):
        s = torch.arange(n, device=DEV)
        return torch.where(s > n // 2, s - n, s).double()

    fz, fy, fx = signed(nz)[:, None, None], signed(ny)[None, :, None], \
        torch.arange(nxh, device=DEV).double()[None, None, :]
    rot = torch.exp(2j * math.pi * (zc / nz * fz + yc / ny * fy + xc / nx * fx))
    # radial bins as the method rounds them
    dkx, dky, dkr = F32(1) / (F32(nx) * F32(dr)), F32(1) / (F32(ny) * F32(dr)), F32(1) / (F32(min(nx, ny)) * F32(dr))
    kyf = (signed(ny).cpu().numpy().astype(np.float32) * dky)[:, None]
    kxf = (np.arange(nxh).astype(np.float32) * dkx)[None, :]
    rd = np.sqrt(kxf * kxf + kyf * kyf).astype(np.float32)
    bins = np.rint((rd / dkr).astype(np.float32)).astype(np.int64)
    inside = torch.from_numpy(rd < F32(F32(0.5) / F32(dr))).to(DEV)
    nb = min(nx, ny) // 2 + 1
    idx = torch.from_numpy(bins).to(DEV)[inside].clamp(max=nb - 1)
    cnt = torch.zeros(nb, device=DEV, dtype=torch.float64).index_add_(0, idx, torch.ones_like(idx).double())
    bands = []
    for b in range(nph):
        order = (b + 1) // 2
        w = [1.0 if b == 0 else math.cos(q * order * 2 * math.pi / nph) if b % 2 else
             math.sin(q * order * 2 * math.pi / nph) for q in range(nph)]
        s = sum(p[:, q] * _f(w[q] / nph) for q in range(nph))
        f = torch.fft.rfftn(s) * rot
        k0 = order / (no - 1) / ls
        kk = torch.sqrt((fz / (nz * dz)) ** 2 + (fy / (ny * dr) + k0 * math.sin(ang)) ** 2 +
                        (fx / (nx * dr) + k0 * math.cos(ang)) ** 2)
        a = dia * 0.5
        u = 2 * math.pi * a * torch.where(kk == 0, torch.ones_like(kk), kk)
        ratio = torch.where(kk == 0, torch.ones_like(kk), 3.0 / (u * u) * (torch.sin(u) / u - torch.cos(u)))
        f = f / ratio
        acc = torch.zeros(nz, nb, device=DEV, dtype=torch.complex128).index_add_(1, idx, f[:, inside])
        acc = (acc / cnt.clamp(min=1)).T.cpu().numpy()  # [kr][kz]
        acc[:, 0] = acc[:, 0].real
        for q in range(1, nz // 2 + 1):
            m = (acc[:, q] + np.conj(acc[:, nz - q])) / 2
            acc[:, q], acc[:, nz - q] = m, np.conj(m)
        acc[0, 1 if order == 0 else 0:] = acc[1, 1 if order == 0 else 0:]
        if b == 0:  # a straight line through kr = 3..20 replaces the first points
            k1, k2 = 3, 20
            sums = acc[:k2 + 1].real.sum(1)
            sums[0] = acc[0, 0].real
            mid, t = 0.5 * (k1 + k2), np.arange(k1, k2 + 1)
            slope = (sums[k1:] * (t - mid)).sum() / ((t - mid) ** 2).sum()
            for q in range(k1):
                acc[q, 0] = acc[q, 0].real - (sums[q] - (sums[k1:].mean() + (q - mid) * slope)) + 1j * acc[q, 0].imag
            norm = acc[0, 0].real
        bands.append(acc / norm)
    out = np.zeros((no, nxh, 2 * nz))
    for o in range(no):
        v = bands[0] if o == 0 else None
        if o:
            re, im = bands[2 * o - 1], bands[2 * o]
            phi = math.atan(np.abs(im).sum() / np.abs(re).sum())
            r0, i0 = re[nx // 4, 0].real, im[nx // 4, 0].real
            phi = phi + math.pi if r0 < 0 < i0 else math.pi - phi if r0 < 0 and i0 < 0 else -phi if r0 > 0 and i0 > 0 \
                else phi
            v = re * math.cos(phi) - im * math.sin(phi)
        out[o, :, 0::2], out[o, :, 1::2] = v.real, v.imag
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "otf":
        return _exact_otf(_bead_stack(case, seed), case)
    if kind == "batch":
        parts = _batch_parts(case)
        outs, total = [], case["frames"] + case["volumes"]
        for i in range(total):
            k = 2 if i * case["volumes"] // total != (i + 1) * case["volumes"] // total else i % 2
            outs.append(_exact_single(parts[k], _simulate(_geometry(parts[k]), seed * 1000 + i)[0]).volume())
        return outs
    g = _geometry(case)
    n = case.get("n", 0)
    stacks = _simulate(g, seed, 1 + n)
    e = _exact_single(case, stacks[0])
    if n:
        k0, outs = e.k0, []
        for s in stacks[1:]:
            e.load(s)
            e.fit(k0)
            outs.append(e.volume().cpu())
        return outs
    return {"volume": e.volume(), "k0": np.array(e.k0, np.float64), "amps": np.array(e.amps, np.complex128)}
