"""The work a program has this library do, as cases that can be timed.

A case is a dict of plain values; ``kind`` says which part of the path it is:

* ``frame``: one steered CONFIG frame -- a new STATE, then the render, as the
  steering loop does it -- without skipping, with the exact grid or with the
  learned one;
* ``ref``: one steered frame with the reference's own sampling;
* ``edit``: a transfer-function edit and the first frame under it (the new
  TF's skipping grid is built on the way);
* ``batch``: many views, TFs and sizes in one persistent launch, the
  requests entered anew as a server does;
* ``open``: a dataset opened -- upload, bricks, macrocells, corner-packed
  copies -- up to its first frame;
* ``histogram``, ``gradient``: the passes over a resident volume that LUT
  building and shading need;
* ``composite``: sort-last compositing of per-rank sub-images and the RGBA8
  rule;
* ``train``: one epoch of the learned predictor, forward and backward.

Volumes are sums of Gaussian blobs like the benchmark's (``synth``), made on
the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ivr_gb300 import api, synth
from ivr_gb300.state import orbit_state

DTYPES = {"u8": (255.0, np.uint8), "u16": (65535.0, np.uint16), "f32": (255.0, np.float32)}
REF_MODES = {"med": api.TF_MED, "seismic2": api.TF_SEISMIC2, "chem": api.TF_CHEM}


def listed():
    return [
        # a thumbnail of a small dataset while the user drags the camera: the
        # smallest call, where launches and host work count
        dict(name="frame_small", kind="frame", dtype="u8", nx=128, ny=128, nz=128, blobs=8, noise=0.05, zero=0.0,
             bricks=1, w=256, h=256, skip="grid", step=0.5, tf="ramp", rgba32=False),
        # the drop-in path with the reference's own semantics
        dict(name="ref_frame", kind="ref", dtype="u8", nx=128, ny=128, nz=128, blobs=8, noise=0.05, mode="seismic2",
             bricks=1, w=512, h=512),
        # the sorted-brick benchmark frame: 2x2x2 bricks, the FP32 frame too
        dict(name="frame_bricks", kind="frame", dtype="f32", nx=512, ny=512, nz=512, blobs=64, noise=0.02, zero=0.0,
             bricks=2, w=1024, h=1024, skip="grid", step=0.5, tf="ramp", rgba32=True),
        # the plain method on a ragged volume and window: what dense TFs and
        # the oracle comparison render
        dict(name="frame_plain", kind="frame", dtype="u16", nx=301, ny=260, nz=223, blobs=24, noise=0.02, zero=0.0,
             bricks=1, w=853, h=479, skip="none", step=0.5, tf="ramp", rgba32=True),
        # the headline frame: 1024^3 u16, full HD, learned skipping
        dict(name="frame_learned", kind="frame", dtype="u16", nx=1024, ny=1024, nz=1024, blobs=256, noise=0.0,
             zero=0.7, bricks=1, w=1920, h=1080, skip="learned", step=0.5, tf="knots", rgba32=False),
        # a TF edit under learned skipping and its first frame
        dict(name="edit_learned", kind="edit", dtype="u16", nx=512, ny=512, nz=512, blobs=128, noise=0.0, zero=0.7,
             bricks=1, w=1280, h=720, skip="learned", step=0.5, tf="knots", rgba32=False),
        # a server's batch of requests of mixed sizes
        dict(name="batch_mixed", kind="batch", dtype="f32", nx=512, ny=512, nz=512, blobs=64, noise=0.02, zero=0.0,
             bricks=2, frames=32, tfs=4, largest=1920),
        # a dataset opened, up to its first frame
        dict(name="open_volume", kind="open", dtype="f32", nx=384, ny=384, nz=384, blobs=32, noise=0.02, zero=0.0,
             bricks=2, w=1024, h=1024, skip="grid", step=0.5, tf="ramp", rgba32=False),
        # initvolluts' histogram over the whole 16-bit range
        dict(name="histogram_u16", kind="histogram", dtype="u16", nx=512, ny=512, nz=512, blobs=64, noise=0.0,
             zero=0.7),
        # the per-voxel gradient of a float volume
        dict(name="gradient_f32", kind="gradient", dtype="f32", nx=512, ny=512, nz=384, blobs=32, noise=0.02,
             zero=0.0),
        # eight ranks' sub-images of a full-HD frame composited and quantised
        dict(name="composite_hd", kind="composite", ranks=8, w=1920, h=1080),
        # one epoch of the predictor over 262,144 cells
        dict(name="train_epoch", kind="train", dtype="u16", nx=512, ny=512, nz=512, blobs=128, noise=0.0, zero=0.7,
             bricks=1, tfs=8, batch=8192),
    ]


def _spread(rng, lo, hi):
    """A size from lo to hi, even over its logarithm, odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _volume(rng, lo, hi):
    base = _spread(rng, lo, hi)
    sides = [max(8, min(hi, int(base * rng.uniform(0.6, 1.2)))) for _ in range(3)]
    return dict(dtype=rng.choice(["u8", "u16", "f32"]), nx=sides[0], ny=sides[1], nz=sides[2],
                blobs=rng.randint(6, 96), noise=rng.choice([0.0, 0.02, 0.05]), zero=rng.choice([0.0, 0.5, 0.7]))


def _window(rng, lo=96, hi=1920):
    w = _spread(rng, lo, hi)
    return dict(w=w, h=max(64, int(w * rng.uniform(0.5, 1.0))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["frame", "frame", "frame", "ref", "edit", "batch", "open", "histogram", "gradient",
                       "composite", "train"])
    if kind == "frame":
        c = dict(kind=kind, **_volume(rng, 64, 640), bricks=rng.choice([1, 2, 3]), **_window(rng),
                 skip=rng.choice(["none", "grid", "grid", "learned"]), step=round(rng.uniform(0.25, 1.0), 3),
                 tf=rng.choice(["ramp", "knots"]), rgba32=rng.random() < 0.4)
        if c["skip"] == "none":  # every lattice point of every ray: smaller windows
            c["w"], c["h"] = min(c["w"], 1024), min(c["h"], 768)
        return c
    if kind == "ref":
        c = _volume(rng, 32, 320)
        del c["zero"]
        return dict(kind=kind, **c, mode=rng.choice(sorted(REF_MODES)), bricks=rng.choice([1, 2]),
                    **_window(rng, 96, 1024))
    if kind == "edit":
        return dict(kind=kind, **_volume(rng, 64, 640), bricks=rng.choice([1, 2]), **_window(rng, 96, 1280),
                    skip=rng.choice(["grid", "learned"]), step=0.5, tf="knots", rgba32=False)
    if kind == "batch":
        return dict(kind=kind, **_volume(rng, 64, 512), bricks=rng.choice([1, 2]), frames=rng.randint(3, 40),
                    tfs=rng.randint(1, 4), largest=_spread(rng, 256, 1920))
    if kind == "open":
        return dict(kind=kind, **_volume(rng, 48, 512), bricks=rng.choice([1, 2, 3]), **_window(rng, 96, 1024),
                    skip="grid", step=0.5, tf="ramp", rgba32=False)
    if kind in ("histogram", "gradient"):
        return dict(kind=kind, **_volume(rng, 48, 512))
    if kind == "composite":
        return dict(kind=kind, ranks=rng.randint(2, 16), **_window(rng))
    c = _volume(rng, 96, 512)
    c["dtype"] = rng.choice(["u8", "u16", "f32"])
    return dict(kind="train", **c, bricks=rng.choice([1, 2]), tfs=rng.randint(2, 8),
                batch=rng.choice([1000, 2048, 4096, 8192]))


# ---- inputs -----------------------------------------------------------------
def _blobs(case, seed):
    """The case's volume on the GPU in its dtype's range, float32 (nz, ny, nx):
    blobs summed as one product of their separable factors."""
    rng = np.random.default_rng(seed)
    n = int(case["blobs"])
    centre, amp = rng.uniform(0.2, 0.8, (n, 3)), rng.uniform(0.3, 1.0, n)
    sigma = rng.uniform(0.03, 0.12, n) * min(1.0, (8.0 / n) ** (1.0 / 3.0))
    dims = (case["nx"], case["ny"], case["nz"])
    big = float(max(dims))
    f = []
    for a, m in enumerate(dims):
        x = (torch.arange(m, device="cuda", dtype=torch.float64) + 0.5) / big
        c = torch.tensor(centre[:, a] * (m / big), device="cuda")
        s = torch.tensor(sigma, device="cuda")
        f.append(torch.exp(-((x[None, :] - c[:, None]) ** 2) / (2 * s[:, None] ** 2)).float())
    f[2] = f[2] * torch.tensor(amp, device="cuda").float()[:, None]
    vol = torch.empty(dims[::-1], device="cuda")
    zx = (f[2][:, :, None] * f[0][:, None, :]).reshape(n, -1)  # [blob][z x]
    for y in range(0, dims[1], 64):
        part = f[1][:, y:y + 64].t() @ zx
        vol[:, y:y + 64, :] = part.reshape(-1, dims[2], dims[0]).transpose(0, 1)
    del zx
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    if case.get("noise", 0.0) > 0:
        vol += (torch.rand(vol.shape, generator=gen, device="cuda") * 2 - 1) * case["noise"]
    vol.clamp_(0.0, 1.0)
    if case.get("zero", 0.0) > 0:  # that share of the 16^3 cells exactly zero
        top = torch.nn.functional.max_pool3d(vol[None, None], 16, 16, ceil_mode=True).flatten()
        t = torch.sort(top)[0][min(top.numel() - 1, int(case["zero"] * top.numel()))]
        vol[vol <= t] = 0.0
    return vol.mul_(DTYPES[case["dtype"]][0])


def _host_volume(case, seed):
    v = _blobs(case, seed)
    if case["dtype"] == "f32":
        return v.cpu().numpy()
    v = v.round_()
    if case["dtype"] == "u8":
        return v.to(torch.uint8).cpu().numpy()
    return v.to(torch.int32).to(torch.int16).cpu().numpy().view(np.uint16)


def _scale(case):
    return 256.0 / 65536.0 if case["dtype"] == "u16" else 1.0


def _lut(case, seed):
    if case.get("tf", "knots") == "ramp":
        return synth.ramp_tf(256)
    return synth.knot_tf(seed, zero_first=True)[0]


def _camera(case, seed, w=None, h=None):
    rng = np.random.default_rng(seed + 17)
    return orbit_state(float(rng.uniform(0, 360)), float(rng.uniform(-60, 60)), w or case["w"], h or case["h"])


def _params(case):
    skip = {"none": api.SKIP_NONE, "grid": api.SKIP_GRID, "learned": api.SKIP_LEARNED}[case["skip"]]
    return api.config_params(step=case["step"], skip=skip)


class State:
    """What the program holds; its handles are freed with it."""

    def __init__(self, case):
        self.case = case
        self.ctx = api.Context(0)
        self.handles = []

    def keep(self, h):
        self.handles.append(h)
        return h

    def volume(self, host):
        v = self.keep(self.ctx.load_volume(host))
        b = int(self.case.get("bricks", 1))
        return v.bricks(b, b, b) if b > 1 else v

    def __del__(self):
        torch.cuda.synchronize()
        for h in self.handles:  # the volume before its predictor
            h.free()
        self.ctx.close()


def _predictor(s, epochs, tfs, seed, batch=8192):
    """A predictor and its training set: the cells of the volume under tfs TFs."""
    m = s.keep(s.ctx.mlp(seed))
    for t in range(tfs):
        tf = s.ctx.transfer_function().set_lut(synth.knot_tf(1000 + t, zero_first=True)[0], 0, _scale(s.case))
        m.add_samples(s.vol, tf)
        tf.free()
    if epochs:
        m.train(epochs, batch_rows=batch, lr=2e-3, wneg=16.0)
    return m


def _sub_images(case, seed):
    """Premultiplied sub-images, each empty outside its rectangle."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    h, w = case["h"], case["w"]
    sub = torch.rand((case["ranks"], h, w, 4), generator=gen, device="cuda")
    sub[..., :3] *= sub[..., 3:]
    rng = np.random.default_rng(seed)
    for k in range(case["ranks"]):
        y, x = int(rng.integers(0, h // 2)), int(rng.integers(0, w // 2))
        mask = torch.zeros((h, w, 1), device="cuda")
        mask[y:y + h * 2 // 3, x:x + w * 2 // 3] = 1.0
        sub[k] *= mask
    return sub


def prepare(case, seed):
    s = State(case)
    kind = case["kind"]
    if kind == "composite":
        shape = (case["h"], case["w"], 4)
        s.sub = _sub_images(case, seed)
        s.back = torch.zeros(shape, device="cuda")
        s.out8 = torch.empty(shape, dtype=torch.uint8, device="cuda")
        return s
    host = _host_volume(case, seed)
    if kind == "open":
        s.host = host
        s.tf = s.keep(s.ctx.transfer_function().set_lut(_lut(case, seed), 0, _scale(case)))
        s.view = s.keep(s.ctx.view())
    else:
        s.vol = s.volume(host)
    if kind in ("frame", "edit"):
        if case["skip"] == "learned":
            s.mlp = _predictor(s, 15, 8, 1)
            s.vol.set_mlp(s.mlp, s.mlp.calibrate(0.02)[0], certify=True)
        s.lut = _lut(case, seed)
        s.tf = s.keep(s.ctx.transfer_function().set_lut(s.lut, 0, _scale(case)))
        s.view = s.keep(s.ctx.view())
    if kind == "ref":
        s.tf = s.keep(s.ctx.transfer_function())
        s.tf.set_colormap(s.vol, api.CM_SEISMIC, REF_MODES[case["mode"]])
        s.view = s.keep(s.ctx.view())
        s.params = api.ref_params()
    if kind in ("frame", "edit", "open"):
        s.params = _params(case)
    if kind in ("frame", "edit", "ref", "open"):
        s.camera = _camera(case, seed)
        s.out8 = torch.empty((case["h"], case["w"], 4), dtype=torch.uint8, device="cuda")
        s.out32 = torch.empty((case["h"], case["w"], 4), device="cuda") if case.get("rgba32") else None
    if kind == "batch":
        sizes, rng = np.random.default_rng(5), np.random.default_rng(seed + 5)
        s.tfs = [s.keep(s.ctx.transfer_function().set_lut(synth.knot_tf(seed + t, zero_first=True)[0], 0, _scale(case)))
                 for t in range(case["tfs"])]
        s.batch = s.keep(s.ctx.batch(case["frames"]))
        s.frames, size = [], 0
        for k in range(case["frames"]):
            w, h = _batch_size(case, sizes)
            p = api.config_params(step=float(rng.uniform(0.25, 1.0)))
            s.frames.append((s.keep(s.ctx.view()), _camera(case, seed + 31 * k, w, h), p, s.tfs[k % len(s.tfs)], size))
            size += w * h * 4
        s.out8 = torch.empty(size, dtype=torch.uint8, device="cuda")
    if kind == "histogram":
        mn, mx = s.vol.minmax()
        s.bins = int(mx - mn + 1)
    if kind == "gradient":
        s.out32 = torch.empty((case["nz"], case["ny"], case["nx"], 4), device="cuda")
    if kind == "train":
        s.mlp = _predictor(s, 0, case["tfs"], seed)
    return s


def _batch_size(case, rng):
    share = [1.0, 0.5, 0.25, 0.125][int(rng.integers(0, 4))]
    w = max(64, int(case["largest"] * share))
    return w, max(64, w * 9 // 16)


# ---- one pass ---------------------------------------------------------------
def _ptr(t):
    return None if t is None else t.data_ptr()


def run(s):
    kind = s.case["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind in ("frame", "ref", "edit"):
        if kind == "edit":
            s.tf.set_lut(s.lut, 0, _scale(s.case))
        s.view.set(s.vol, s.camera, s.params)
        s.view.render(s.tf, _ptr(s.out32), s.out8.data_ptr(), stream)
        return {"rgba8": s.out8} if s.out32 is None else {"rgba32": s.out32, "rgba8": s.out8}
    if kind == "open":
        vol = s.ctx.load_volume(s.host)
        b = int(s.case["bricks"])
        if b > 1:
            vol.bricks(b, b, b)
        s.view.set(vol, s.camera, s.params)
        s.view.render(s.tf, None, s.out8.data_ptr(), stream)
        vol.free()
        return {"rgba8": s.out8}
    if kind == "batch":
        s.batch.clear()
        for view, camera, p, tf, off in s.frames:
            view.set(s.vol, camera, p)
            s.batch.add(view, tf, None, s.out8.data_ptr() + off)
        s.batch.render(True, stream)
        return {"rgba8": s.out8}
    if kind == "histogram":
        return {"hist": s.vol.histogram(s.bins)}
    if kind == "gradient":
        s.vol.gradient(s.out32.data_ptr(), stream)
        return {"gradient": s.out32}
    if kind == "composite":
        n, h, w = s.sub.shape[0], s.sub.shape[1], s.sub.shape[2]
        s.back.zero_()
        s.ctx.composite(s.back.data_ptr(), s.sub.data_ptr(), n, w, h, stream)
        s.ctx.quantize(s.back.data_ptr(), s.out8.data_ptr(), w * h * 4, stream)
        return {"rgba32": s.back, "rgba8": s.out8}
    losses = s.mlp.train(1, batch_rows=s.case["batch"], lr=2e-3, wneg=16.0)
    return {"losses": losses, "params": s.mlp.params()}


def _cells(case):
    n = 1
    for a in ("nx", "ny", "nz"):
        n *= (case[a] - 2) // 16 + 1
    return n


def work(case):
    """Bytes and operations of one pass that no method can do without."""
    kind = case["kind"]
    if kind == "composite":
        n = case["w"] * case["h"]
        return {"bytes": 16.0 * n * (case["ranks"] + 1) + 4.0 * n, "flops": 12.0 * n * case["ranks"]}
    vox = float(case["nx"]) * case["ny"] * case["nz"]
    esz = np.dtype(DTYPES[case["dtype"]][1]).itemsize
    if kind == "histogram":
        return {"bytes": vox * esz, "flops": 2.0 * vox}
    if kind == "gradient":
        return {"bytes": vox * (esz + 16.0), "flops": 15.0 * vox}
    if kind == "train":  # a row: 26-64-64-1 forward, twice that backward
        rows = _cells(case) * case["tfs"]
        return {"bytes": rows * (64.0 + 4.0), "flops": 6.0 * rows * (26 * 64 + 64 * 64 + 64)}
    # Frames: a box of side 2 seen from distance 5 with 30 degrees of field of
    # view: its mean silhouette (a quarter of its surface) covers about 0.84
    # of the window's height squared, and a ray's mean path in it is 4 V / S.
    # Of the lattice an opacity TF leaves about a tenth to sample.
    def frame(w, h, step):
        big = float(max(case["nx"], case["ny"], case["nz"]))
        x, y, z = (case[a] / big for a in ("nx", "ny", "nz"))
        face = x * y + y * z + z * x
        rays = min(1.0, 0.84 * face / 3.0 * h / w) * w * h
        samples = rays * (2.0 * x * y * z / face) * big / step
        kept = 1.0 if case.get("skip", "grid") == "none" else 0.1
        return w * h * (20.0 if case.get("rgba32") else 4.0) + kept * vox * esz, 40.0 * kept * samples
    if kind == "batch":
        rng = np.random.default_rng(5)
        got = []
        for _ in range(case["frames"]):
            w, h = _batch_size(case, rng)
            got.append(frame(w, h, 0.54))  # the harmonic mean of the steps
        return {"bytes": 0.1 * vox * esz + sum(g[0] - 0.1 * vox * esz for g in got), "flops": sum(g[1] for g in got)}
    if kind == "ref":  # at most 256 samples of a thousandth of the view axis
        n = float(case["w"]) * case["h"]
        return {"bytes": 4.0 * n + 0.2 * vox * esz, "flops": 40.0 * 256 * 0.6 * n}
    b, f = frame(case["w"], case["h"], case["step"])
    if kind == "open":
        b += vox * esz
    if kind == "edit":
        b += _cells(case) * 42.0
        f += 2.0 * _cells(case) * (26 * 64 + 64 * 64 + 64) if case["skip"] == "learned" else 0.0
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits ----------------------------------------------------
def _exact_frame(case, seed):
    """The CONFIG frame by definition: one lattice per ray over the box, the
    trilinear sample of every point, front-to-back until term_alpha."""
    st = _camera(case, seed)
    dims = (case["nx"], case["ny"], case["nz"])
    big = float(max(dims))
    vol = _blobs(case, seed)
    vol = (vol if case["dtype"] == "f32" else vol.round_()).double().reshape(-1)
    lut = torch.tensor(_lut(case, seed), device="cuda").double()
    f64 = dict(dtype=torch.float64, device="cuda")
    m = torch.tensor(list(st.mvm), **f64).reshape(4, 4).t()
    rot = m[:3, :3].t()
    orig = rot @ torch.tensor([-float(m[0, 3]), -float(m[1, 3]), 5.0], **f64)
    left, right, bottom, top = (float(v) for v in st.vv)
    w, h = case["w"], case["h"]
    u = left + (torch.arange(w, **f64) + 0.5) * ((right - left) / w)
    v = bottom + (torch.arange(h, **f64) + 0.5) * ((top - bottom) / h)
    vv, uu = torch.meshgrid(v, u, indexing="ij")
    d = torch.stack([uu, vv, torch.full_like(uu, -5.0)], -1).reshape(-1, 3) @ rot.t()
    half = torch.tensor([n / big for n in dims], **f64)
    a, b = (-half - orig) / d, (half - orig) / d
    t0 = torch.minimum(a, b).amax(1).clamp_min(0.0)
    t1 = torch.maximum(a, b).amin(1)
    dt = case["step"] * (2.0 / big) / d.norm(dim=1)
    acc = torch.zeros((w * h, 4), **f64)
    ray = torch.nonzero(t1 > t0).flatten()
    lim = torch.tensor([n - 1.0 for n in dims], **f64)
    i = 0
    while ray.numel():
        t = t0[ray] + i * dt[ray]
        live = t < t1[ray]
        ray, t = ray[live], t[live]
        p = ((orig + t[:, None] * d[ray]) + half) * (big / 2.0)
        p = torch.minimum(p.clamp_min(0.0), lim)
        c = torch.minimum(p.floor(), lim - 1.0)
        q = p - c
        c = c.long()
        at = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
        s = 0.0
        for k in range(8):
            e = [(k >> n) & 1 for n in range(3)]
            wgt = 1.0
            for n in range(3):
                wgt = wgt * (q[:, n] if e[n] else 1.0 - q[:, n])
            s = s + wgt * vol[at + (e[2] * dims[1] + e[1]) * dims[0] + e[0]]
        rgba = lut[(s * _scale(case)).long().clamp(0, lut.shape[0] - 1)]
        now = acc[ray]
        wgt = (1.0 - now[:, 3:]) * rgba[:, 3:]
        now = now + wgt * torch.cat([rgba[:, :3], torch.ones_like(wgt)], 1)
        acc[ray] = now
        ray = ray[now[:, 3] < 0.99]
        i += 1
    return {"rgba32": acc.reshape(h, w, 4), "rgba8": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "frame" and case["rgba32"]:
        points = case["w"] * case["h"] * max(case["nx"], case["ny"], case["nz"]) / case["step"]
        return _exact_frame(case, seed) if points < 4e9 else None
    if kind == "gradient":
        v = torch.from_numpy(_host_volume(case, seed).astype(np.float32)).cuda().double()
        g = []
        for axis in (2, 1, 0):
            n = v.shape[axis]
            hi = torch.arange(n, device="cuda").add(1).clamp_max(n - 1)
            lo = torch.arange(n, device="cuda").sub(1).clamp_min(0)
            g.append((v.index_select(axis, hi) - v.index_select(axis, lo)) / 2.0)
        g.append((g[0] ** 2 + g[1] ** 2 + g[2] ** 2).sqrt())
        return {"gradient": torch.stack(g, -1)}
    if kind == "composite":
        sub = _sub_images(case, seed)
        d = torch.zeros(sub.shape[1:], dtype=torch.float64, device="cuda")
        for k in range(sub.shape[0] - 1, -1, -1):
            src = sub[k].double()
            d = src + (1.0 - src[..., 3:]) * d
        return {"rgba32": d, "rgba8": None}
    return None
