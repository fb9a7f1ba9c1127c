"""The work that a user has this package do, as timed cases through its public entry points.

Seven kinds, over the sizes of the package's own benchmark, tests and example workloads:

  dropin  the reference's call loop (TimeStep, injectdata, extractdata; host wavelet and traces)
  step    3D time stepping on the device: forward, adjoint (linear for VTI) or with the imaging condition
  loop2d  a whole 2D shot in one call (WFD_Prop_Run: steps, source injection, receiver extraction)
  batch   several ginsu-cropped 3D shots advanced together (ShotBatch)
  born    a Born injection and an adjoint accumulation of one model space (V, VB, B or VEA)
  sep     the wavefield-separation imaging condition (FWI or RTM)
  codec   a saved wavefield through the learned codec, encode and decode

Grids are (nx, ny, nz), z fastest. Inputs are made on the GPU from the seed: layered velocities of
1500-4500 m/s with smooth perturbations, Gardner densities, a Q profile with an absorbing sponge,
smooth anisotropy and tilt, and band-limited wavefields. `exact` is the same arithmetic in float64
with plain torch.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as tf

DEV = "cuda"
C = [float(np.float32(c)) for c in (1225.0 / 1024.0, -245.0 / 3072.0, 49.0 / 5120.0, -5.0 / 7168.0)]
D = 10.0
IV = float(np.float32(1.0 / D))
MODELS = {"iso": ("V", "B", "DtOmegaInvQ"), "vti": ("V", "B", "DtOmegaInvQ", "Eps", "Eta", "F"),
          "tti": ("V", "B", "DtOmegaInvQ", "Eps", "Eta", "F", "SinTheta", "CosTheta", "SinPhi", "CosPhi")}
# bytes a cell of one time step cannot do without: each model and field array read once, the new
# field and the spatial derivative written once
STEP_BYTES = {("iso", 3): 28, ("vti", 3): 56, ("tti", 3): 72, ("iso", 2): 28, ("vti", 2): 56, ("tti", 2): 64}
STEP_FLOPS = {("iso", 3): 105, ("vti", 3): 240, ("tti", 3): 290, ("iso", 2): 75, ("vti", 2): 170, ("tti", 2): 300}


# ---- the cases -----------------------------------------------------------------------------------
def listed():
    return [
        # a quality-control or test-sized shot driven exactly as the reference is: launch latency
        dict(name="dropin iso 64", kind="dropin", phys="iso", nx=64, ny=60, nz=68, steps=4, nrec=15, fs=True),
        # the benchmark's default workload
        dict(name="step iso 512", kind="step", phys="iso", nx=512, ny=512, nz=512, steps=4, mode="forward", fs=True),
        # a cropped shot window: sizes as the acquisition gives them, nothing a multiple of anything
        dict(name="step iso odd", kind="step", phys="iso", nx=301, ny=203, nz=251, steps=4, mode="forward", fs=True),
        # the benchmark's anisotropic workloads
        dict(name="step vti 400", kind="step", phys="vti", nx=400, ny=400, nz=400, steps=2, mode="forward", fs=True),
        dict(name="step tti 400", kind="step", phys="tti", nx=400, ny=400, nz=400, steps=2, mode="forward", fs=True),
        # a cropped TTI window
        dict(name="step tti odd", kind="step", phys="tti", nx=203, ny=181, nz=251, steps=2, mode="forward", fs=True),
        # the benchmark's 2D shot, and the reference's own 2D benchmark grid in TTI
        dict(name="loop2d iso 501", kind="loop2d", phys="iso", nx=501, nz=501, nt=400, fs=True),
        dict(name="loop2d tti 1000x500", kind="loop2d", phys="tti", nx=1000, nz=500, nt=200, fs=True),
        # a batch of uneven ginsu windows, Iso and VTI mixed, as the batched benchmark cuts them
        dict(name="batch 8", kind="batch", shots=8, lo=96, hi=176, nz=200, steps=4, cut=5),
        # linearised modelling and migration in the full anisotropic model space
        dict(name="born vea tti", kind="born", phys="tti", nx=200, ny=180, nz=240, variant="VEA", fs=True),
        # full-waveform inversion's separated imaging condition
        dict(name="sep fwi iso", kind="sep", phys="iso", nx=160, ny=128, nz=300, cond="FWI", fs=True),
        # one saved snapshot into the codec and back
        dict(name="codec 512x256x400", kind="codec", nx=512, ny=256, nz=400),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "step", "step", "loop2d", "batch", "born", "sep", "codec"])
    even = rng.random() < 0.5  # half the depths a multiple of 4, the others as they come
    z = lambda lo, hi: 4 * max(1, _size(rng, lo, hi) // 4) if even else _size(rng, lo, hi)  # noqa: E731
    phys = rng.choice(["iso", "vti", "tti"])
    fs = rng.random() < 0.85
    if kind == "dropin":
        return dict(kind=kind, phys=phys, nx=_size(rng, 40, 200), ny=_size(rng, 40, 200), nz=z(40, 240),
                    steps=rng.randint(2, 6), nrec=rng.randint(4, 40), fs=fs)
    if kind == "step":
        return dict(kind=kind, phys=phys, nx=_size(rng, 64, 400), ny=_size(rng, 64, 400), nz=z(64, 400),
                    steps=rng.randint(2, 3), mode=rng.choice(["forward", "adjoint", "image"]), fs=fs)
    if kind == "loop2d":
        return dict(kind=kind, phys=phys, nx=_size(rng, 200, 2400), nz=z(150, 1200), nt=rng.randint(60, 300), fs=fs)
    if kind == "batch":
        lo = _size(rng, 48, 120)
        return dict(kind=kind, shots=rng.randint(2, 16), lo=lo, hi=lo + rng.randint(16, 90),
                    nz=4 * (_size(rng, 60, 280) // 4), steps=2 * rng.randint(1, 4), cut=rng.randint(0, 999))
    if kind == "born":
        variant = rng.choice(["V", "VB", "B"] if phys == "iso" else ["V", "VEA", "VEA"])
        return dict(kind=kind, phys=phys, nx=_size(rng, 48, 300), ny=_size(rng, 48, 300), nz=z(64, 300),
                    variant=variant, fs=fs)
    if kind == "sep":
        return dict(kind=kind, phys=phys, nx=_size(rng, 24, 220), ny=_size(rng, 24, 220), nz=z(64, 520),
                    cond=rng.choice(["FWI", "RTM"]), fs=fs)
    return dict(kind=kind, nx=_size(rng, 64, 512), ny=_size(rng, 64, 512), nz=z(64, 400))


def _shape(c):
    return (c["nx"], c["ny"], c["nz"]) if "ny" in c else (c["nx"], c["nz"])


def _windows(c):
    """The batch's shot windows: (nx, ny) and physics, cut as the survey's acquisition gives them."""
    r = np.random.default_rng(c["cut"])
    out = []
    for i in range(c["shots"]):
        nx, ny = (int(v) for v in r.integers(c["lo"], c["hi"] + 1, 2))
        out.append(((nx, ny, c["nz"]), "iso" if i % 2 == 0 else "vti"))
    return out


def work(c):
    k = c["kind"]
    if k == "batch":
        b = f = 0
        for (nx, ny, nz), ph in _windows(c):
            b += nx * ny * nz * STEP_BYTES[ph, 3] * c["steps"]
            f += nx * ny * nz * STEP_FLOPS[ph, 3] * c["steps"]
        return {"bytes": b, "flops": f}
    sh = _shape(c)
    n = int(np.prod(sh))
    if k in ("dropin", "step", "loop2d"):
        nd, nt = len(sh), c.get("steps") or c.get("nt")
        per = STEP_BYTES[c["phys"], nd]
        if c.get("mode") == "adjoint" and c["phys"] == "vti":
            per -= 8
        extra = 0 if c.get("mode") != "image" else n * (12 if c["phys"] == "iso" else 16)
        return {"bytes": n * per * nt + extra, "flops": n * STEP_FLOPS[c["phys"], nd] * nt}
    if k == "born":
        # injection then accumulation, each array once in each of the two calls
        per = {("iso", "V"): 24 + 24, ("iso", "VB"): 32 + 36, ("iso", "B"): 28 + 28,
               ("vti", "V"): 32 + 36, ("tti", "V"): 32 + 36, ("vti", "VEA"): 64 + 68, ("tti", "VEA"): 80 + 84}
        return {"bytes": n * per[c["phys"], c["variant"]], "flops": n * (40 if c["variant"] == "V" else 250)}
    if k == "sep":
        fields = 1 if c["phys"] == "iso" else 2
        return {"bytes": n * (8 * fields + 16), "flops": n * fields * 100}
    nb = int(np.prod([-(-s // 8) for s in sh]))
    return {"bytes": 8 * n + 2 * 97 * nb, "flops": nb * 4 * 2 * 512 * 32}


# ---- inputs --------------------------------------------------------------------------------------
def _up(low, shape):
    """Smooth field from a coarse grid (linear interpolation)."""
    mode = "trilinear" if len(shape) == 3 else "bilinear"
    return tf.interpolate(low[None, None], size=shape, mode=mode, align_corners=True)[0, 0]


def _noise(shape, cells, gen):
    low = [max(2, s // cells + 1) for s in shape]
    return _up(torch.rand(low, generator=gen, device=DEV) * 2 - 1, shape)


def _axis(v, axis, nd):
    return v.reshape([-1 if i == axis else 1 for i in range(nd)])


def _model(shape, phys, dt, fs, gen, nsponge=20):
    nd, nz = len(shape), shape[-1]
    layer = _axis((torch.arange(nz, device=DEV) * 8 // nz).float() / 7, nd - 1, nd)
    v = (1500 + 3000 * layer) * (1 + 0.05 * _noise(shape, 20, gen))
    m = {"V": v, "B": 1 / (0.31 * v.sqrt().sqrt()).clamp(1.0, 2.5)}
    q = 125 + 75 * _noise(shape, 32, gen)
    ks = None
    for a, s in enumerate(shape):
        i = torch.arange(s, device=DEV)
        k = (s - 1 - i) if (a == nd - 1 and fs) else torch.minimum(i, s - 1 - i)
        k = _axis(k, a, nd)
        ks = k if ks is None else torch.minimum(ks, k)
    w = (ks.float() / (nsponge - 1)).clamp(max=1.0)
    m["DtOmegaInvQ"] = (dt * 2 * math.pi * 5.0) / torch.exp(math.log(0.1) * (1 - w) + w * torch.log(q))
    del q, w, ks
    if phys != "iso":
        m["Eps"] = (0.2 * layer + 0.04 * (1 + _noise(shape, 20, gen))).clamp(0, 0.3)
        m["Eta"] = (0.1 * layer + 0.02 * (1 + _noise(shape, 20, gen))).clamp(0, 0.15)
        m["F"] = torch.full(shape, 0.85, device=DEV)
    if phys == "tti":
        th = math.pi / 8 * (1 + _noise(shape, 20, gen))
        m["SinTheta"], m["CosTheta"] = torch.sin(th), torch.cos(th)
        if nd == 3:
            ph = math.pi * (1 + _noise(shape, 20, gen))
            m["SinPhi"], m["CosPhi"] = torch.sin(ph), torch.cos(ph)
    return {k: t.float().contiguous() for k, t in m.items()}


def _wave(shape, gen):
    """A band-limited wavefield: about six cells a wavelength over a slower amplitude."""
    return (_noise(shape, 3, gen) * (1.2 + _noise(shape, 24, gen))).contiguous()


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _dt(nd):
    return 0.0005 if nd == 3 else 0.001


def _acquisition(shape, nrec, seed):
    """1-based (iu, ir, c) of an off-grid source (8 windowed-sinc points an axis) near the surface and
    of on-grid receivers at depth index 2: nrec an axis in 3D, every column in 2D."""
    r = np.random.default_rng(seed)
    nz, nd = shape[-1], len(shape)
    axes, w = [], []
    for a, s in enumerate(shape):
        pos = r.uniform(8.1, 11.9) if a == nd - 1 else s / 2 + r.uniform(-0.4, 0.4)
        i = np.arange(8) + int(pos) - 3
        axes.append(i)
        w.append(np.sinc(i - pos) * np.cos(np.pi * (i - pos) / 10) ** 2)
    grid = np.meshgrid(*axes, indexing="ij")
    c = np.ones([8] * nd)
    for a in range(nd):
        c = c * w[a].reshape([-1 if i == a else 1 for i in range(nd)])
    iu = np.ravel_multi_index([g.ravel() for g in grid], shape) + 1
    src = (iu.astype(np.int64), np.ones(iu.size, np.int64), c.ravel().astype(np.float32))
    if nd == 2:
        riu = 3 + np.arange(shape[0], dtype=np.int64) * nz
    else:
        xs, ys = (np.unique(np.round(np.linspace(5, s - 6, nrec)).astype(np.int64)) for s in shape[:2])
        riu = (3 + ys[None, :] * nz + xs[:, None] * nz * shape[1]).ravel()
    rec = (riu, np.arange(1, riu.size + 1), np.ones(riu.size, np.float32))
    return src, rec


def _wavelet(nt, dt, seed):
    f = 12.0 + (seed % 7) * 0.5
    t = dt * np.arange(nt) - min(1.2 / f, 0.4 * nt * dt)
    return ((1 - 2 * (np.pi * f * t) ** 2) * np.exp(-(np.pi * f * t) ** 2)).astype(np.float32)


def _points(p):
    from wavefd_b200.spacetime import SOURCEPOINT32
    a = np.zeros(p[0].size, SOURCEPOINT32)
    a["iu"], a["ir"], a["c"] = p
    return a


# ---- objects -------------------------------------------------------------------------------------
class _Owner:
    """Frees a propagator when its arrays are no longer held by anything."""

    def __init__(self, prop, free):
        self.prop, self.free = prop, free

    def __del__(self):
        torch.cuda.synchronize()
        self.free(self.prop)


class _Managed:
    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (ptr, False), "version": 3,
                                         "strides": None}


class _Object:
    """A propagator with its model loaded, and its arrays as device tensors."""

    def __init__(self, shape, phys, dt, fs, model, nthreads=None):
        from wavefd_b200 import props
        nd = len(shape)
        cls = getattr(props, "Prop%dDAco%sDenQ_DEO2_FDTD" % (nd, {"iso": "Iso", "vti": "VTI", "tti": "TTI"}[phys]))
        size = dict(nx=shape[0], nz=shape[-1], **({"ny": shape[1]} if nd == 3 else {}))
        self.props, self.shape, self.phys = props, shape, phys
        self.prop = cls(nsponge=20, dz=D, dy=D, dx=D, dt=dt, freesurface=fs, nthreads=nthreads, **size)
        self.owner = _Owner(self.prop, props.free)
        for k, t in model.items():
            self._array(k).copy_(t)
        self.cur = [self._array("PCur"), self._array("POld")]
        self.space = [self._array("PSpace")]
        self.mcur = []
        if phys != "iso":
            self.mcur = [self._array("MCur"), self._array("MOld")]
            self.space.append(self._array("MSpace"))
        self.n = 0  # time steps taken: the two pressure arrays change places at each
        torch.cuda.synchronize()
        self.prop.prefetch()

    def _array(self, name):
        p = getattr(self.prop.abi, "get" + name)(self.prop.p)
        return torch.as_tensor(_Managed(ctypes.cast(p, ctypes.c_void_p).value, self.shape, self.owner), device=DEV)

    def now(self, m=False):
        a = self.mcur if m else self.cur
        return a[self.n & 1], a[1 - (self.n & 1)]

    def outputs(self):
        out = dict(zip(("pcur", "pold"), self.now()))
        out["pspace"] = self.space[0]
        if self.mcur:
            out.update(zip(("mcur", "mold"), self.now(True)))
            out["mspace"] = self.space[1]
        return out


class _Table:
    def __init__(self, points, by_receiver):
        from wavefd_b200 import _lib
        from wavefd_b200.abi import SourcePoint32
        self.lib = _lib.library()
        self.t = self.lib.WFD_Points_Create(points.ctypes.data_as(ctypes.POINTER(SourcePoint32)), len(points),
                                            by_receiver)

    def __del__(self):
        if getattr(self, "t", None):
            self.lib.WFD_Points_Free(self.t)
            self.t = None


def _fields(c, seed, shape, phys, fs):
    """Model and wavefields of one object, in a fixed order of random draws."""
    gen = _gen(seed)
    model = _model(shape, phys, _dt(len(shape)), fs, gen)
    waves = [_wave(shape, gen) for _ in range(2 if phys == "iso" else 4)]
    return model, waves, gen


def _codec_weights():
    """Weights that code smooth blocks as training does, in closed form: each 4^3 sub-block by its 8
    lowest cosine products (as +- pairs, so that the leaky units act as 1.5 x), each 8^3 block by the 32
    lowest of the 64 combinations of those."""
    i = np.arange(8)
    half = np.linalg.qr(np.stack([np.ones(4), np.cos(np.pi * (np.arange(4) + 0.5) / 4)], 1))[0]  # 4 cells x 2
    two = np.kron(np.eye(2), half)  # 8 cells x (sub-block, feature)
    axis = np.linalg.qr(two.T @ np.stack([np.cos(np.pi * (i + 0.5) * f / 8) for f in range(4)], 1))[0]
    axis = axis.reshape(2, 2, 4)  # sub-block, feature, order
    phi = np.einsum("ai,bj,ck->abcijk", half, half, half).reshape(64, 8)  # cell, feature
    orders = sorted(((a, b, c) for a in range(4) for b in range(4) for c in range(4)), key=lambda o: (sum(o), o))[:32]
    comb = np.stack([np.einsum("si,tj,uk->stuijk", *(axis[:, :, o] for o in os)).reshape(8, 8) for os in orders])
    pair = np.array([1.0, -1.0])
    w1 = np.einsum("kf,p->fpk", phi, pair).reshape(16, 64)
    w2 = np.einsum("isf,p->isfp", comb, pair).reshape(32, 128) / 1.5
    w3 = np.einsum("isf,p->sfpi", comb, pair).reshape(128, 32)
    w4 = np.einsum("kf,p->kfp", phi, pair).reshape(64, 16) / 1.5
    return np.concatenate([w1.ravel(), np.zeros(16), w2.ravel(), np.zeros(32), w3.ravel(), np.zeros(128), w4.ravel(),
                           np.zeros(64)]).astype(np.float32)


def prepare(c, seed):
    k = c["kind"]
    if k == "codec":
        from wavefd_b200.codec import WavefieldCodec
        shape, gen = _shape(c), _gen(seed)
        codec = WavefieldCodec(seed=3)
        codec.params = _codec_weights()
        # a saved snapshot: 30 cells a wavelength, sharp around a few sources
        f = _noise(shape, 15, gen)
        for _ in range(3):
            x, y, z = (int(v) for v in (torch.rand(3, generator=gen, device=DEV).cpu() * torch.tensor(shape) * 0.7))
            b = f[x:x + 12, y:y + 12, z:z + 12]
            b += 3 * (torch.rand(b.shape, generator=gen, device=DEV) * 2 - 1)
        return dict(c=c, codec=codec, shape=shape, field=f.contiguous(), code=codec.empty_code(shape),
                    out=torch.empty(shape, device=DEV))
    if k == "batch":
        from wavefd_b200.batch import ShotBatch
        objs, traces, keep = [], [], []
        nt = 64 * c["steps"]
        for i, (shape, phys) in enumerate(_windows(c)):
            model, waves, _ = _fields(c, seed + 100 * i, shape, phys, True)
            o = _Object(shape, phys, _dt(3), True, model)
            for t, w in zip(o.cur + o.mcur, waves):
                t.copy_(w)
            objs.append(o)
        b = ShotBatch([o.prop for o in objs])
        b.owners = [o.owner for o in objs]  # the batch goes before its shots
        for i, o in enumerate(objs):
            src, rec = (_points(p) for p in _acquisition(o.shape, 12, seed + i))
            wav = torch.from_numpy(_wavelet(nt, _dt(3), seed + i)).to(DEV)
            traces.append(torch.zeros((len(rec), nt), device=DEV))
            b.set_acquisition(i, src, wav, rec, traces[-1], nt)
            keep.append(wav)
        return dict(c=c, b=b, objs=objs, traces=traces, keep=keep)
    shape, phys, fs = _shape(c), c["phys"], c["fs"]
    dt = _dt(len(shape))
    if k == "loop2d":
        model, _, _ = _fields(c, seed, shape, phys, fs)
        o = _Object(shape, phys, dt, fs, model)
        src, rec = (_points(p) for p in _acquisition(shape, 0, seed))
        return dict(c=c, o=o, src=_Table(src, 0), rec=_Table(rec, 1),
                    wav=torch.from_numpy(_wavelet(c["nt"], dt, seed)).to(DEV),
                    traces=torch.zeros((len(rec), c["nt"]), device=DEV), keep=(src, rec),
                    stream=torch.cuda.ExternalStream(o.prop.stream()))
    model, waves, gen = _fields(c, seed, shape, phys, fs)
    o = _Object(shape, phys, dt, fs, model, nthreads=8)
    for t, w in zip(o.cur + o.mcur, waves):
        t.copy_(w)
    s = dict(c=c, o=o)
    if k == "dropin":
        from wavefd_b200.spacetime import receiver_blocking, source_blocking
        src, rec = _acquisition(shape, c["nrec"], seed)
        s["src"], s["rec"] = source_blocking(_points(src), 8), receiver_blocking(_points(rec), 8)
        s["wav"] = _wavelet(c["steps"], dt, seed).reshape(1, -1)
        s["traces"] = np.zeros((rec[0].size, c["steps"]), np.float32)
        torch.cuda.synchronize()
        for it in range(2):  # a time loop's first steps: the arrays it asks for settle on the device
            s["o"].props.PCur(o.prop)
            o.props.propagateforward(o.prop)
            o.n += 1
        for t, w in zip(o.cur + o.mcur, waves):
            t.copy_(w)
    elif k in ("born", "sep") or c.get("mode") == "image":
        s.update(_extras(c, shape, phys, gen))
    torch.cuda.synchronize()
    return s


def _extras(c, shape, phys, gen):
    """Model perturbations or images, and the saved wavefields, of the Born and imaging calls."""
    s = {"wf": {}, "dm": {}, "img": {}}
    for key in ("pspace", "pold") if phys == "iso" else ("pspace", "mspace", "pold", "mold"):
        s["wf"][key] = _wave(shape, gen) * (1.0 if key.endswith("old") else 40.0)
    keys = {"V": ("v",), "VB": ("v", "b"), "B": ("b",), "VEA": ("v", "ϵ", "η")}[c.get("variant", "V")]
    for key in keys:
        s["dm"][key] = _noise(shape, 6, gen) * {"v": 40.0, "b": 0.03, "ϵ": 0.01, "η": 0.01}[key]
        s["img"][key] = torch.zeros(shape, device=DEV)
    return s


# ---- one pass ------------------------------------------------------------------------------------
def run(s):
    c = s["c"]
    k = c["kind"]
    if k == "codec":
        s["codec"].encode(s["field"], s["shape"], s["code"])
        s["codec"].decode(s["code"], s["shape"], s["out"])
        return s["out"]
    if k == "batch":
        s["b"].run(c["steps"], it0=1)
        for o in s["objs"]:
            o.n += c["steps"]
        return {"shots": [o.outputs() for o in s["objs"]], "traces": s["traces"]}
    o = s["o"]
    if k == "loop2d":
        with torch.cuda.stream(s["stream"]):
            for t in o.cur + o.mcur + [s["traces"]]:
                t.zero_()
        lib = s["src"].lib
        vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        rc = lib.WFD_Prop_Run(o.prop.p, c["nt"], 1, s["src"].t, vp(s["wav"]), s["rec"].t, vp(s["traces"]), c["nt"], 1)
        if rc:
            raise RuntimeError("WFD_Prop_Run: %d" % rc)
        o.n += c["nt"]
        return {**o.outputs(), "traces": s["traces"]}
    if k == "dropin":
        from wavefd_b200 import spacetime
        s["traces"][:] = 0
        for it in range(1, c["steps"] + 1):
            o.props.propagateforward(o.prop)
            o.n += 1
            pcur = o.props.PCur(o.prop)
            spacetime.injectdata(pcur, s["src"], s["wav"], it)
            spacetime.extractdata(s["traces"], pcur, it, s["rec"])
        return {**o.outputs(), "traces": s["traces"]}
    if k == "step":
        image = c["mode"] == "image"
        linear = c["mode"] != "forward" and c["phys"] == "vti"
        o.prop.step_async(c["steps"] - (1 if image else 0), linear=linear)
        out = {}
        if image:
            from wavefd_b200 import _lib
            vp = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
            _lib.check(_lib.library().WFD_Prop_TimeStepImage(
                o.prop.p, vp(s["img"]["v"]), vp(s["wf"]["pspace"]), vp(s["wf"].get("mspace")), int(linear)), "image")
            out["img"] = s["img"]["v"]
        o.n += c["steps"]
        return {**o.outputs(), **out}
    if k == "born":
        mt = getattr(o.props, o.prop.NAME + "_Model_" + c["variant"])()
        o.props.forwardBornInjection(o.prop, mt, s["dm"], s["wf"])
        o.props.adjointBornAccumulation(o.prop, mt, o.props.ImagingConditionStandard(), s["img"], s["wf"])
        out = {"img " + n: t for n, t in s["img"].items()}
        out["pcur"] = o.now()[0]
        if o.mcur:
            out["mcur"] = o.now(True)[0]
        return out
    mt = getattr(o.props, o.prop.NAME + "_Model_V")()
    cond = getattr(o.props, "ImagingConditionWaveFieldSeparation" + c["cond"])()
    o.props.adjointBornAccumulation(o.prop, mt, cond, s["img"], s["wf"])
    return s["img"]["v"]


# ---- the same in float64 -------------------------------------------------------------------------
class _Ops:
    """Staggered 8th-order derivatives with the free-surface images, on float64 tensors."""

    def __init__(self, shape, fs):
        self.shape, self.fs, self.nd = shape, fs, len(shape)
        r = torch.ones(shape, dtype=torch.bool, device=DEV)
        for a, n in enumerate(shape):
            i = torch.arange(n, device=DEV)
            ok = i < n - 4
            if not (a == self.nd - 1 and fs):
                ok &= i >= 4
            r &= _axis(ok, a, self.nd)
        self.r = r  # cells that are updated
        self.top = _axis(torch.arange(shape[-1], device=DEV) == 0, self.nd - 1, self.nd) if fs else None

    def _diff(self, f, a, plus):
        """Along axis a: sum c_k (f[i+k] - f[i+1-k]) (plus) or sum c_k (f[i+k-1] - f[i-k])."""
        n, z = self.shape[a], a == self.nd - 1
        if z and self.fs:
            top = -f[..., 1:5].flip(-1) if plus else f[..., 0:4].flip(-1)
            e, off = torch.cat([top, f], -1), 4
        else:
            e, off = f, 0
        out = torch.zeros(self.shape, dtype=torch.float64, device=DEV)
        lo = 0 if off else 4
        at = lambda d: e.narrow(a, lo + d + off, n - 4 - lo)  # noqa: E731
        o = out.narrow(a, lo, n - 4 - lo)
        for j in range(1, 5):
            hi, low = (j, 1 - j) if plus else (j - 1, -j)
            o += C[j - 1] * (at(hi) - at(low))
        return out * IV

    def grad(self, f):
        """D+ triple (or pair), zero outside, the lateral ones zero on the surface row."""
        out = []
        for a in range(self.nd):
            g = self._diff(f, a, True) * self.r
            if self.fs and a < self.nd - 1:
                g.masked_fill_(self.top, 0.0)
            out.append(g)
        return out

    def minus(self, f, a):
        g = self._diff(f, a, False) * self.r
        if self.fs:
            g.masked_fill_(self.top, 0.0)
        return g


def _sandwich(ops, m, P, M):
    """Pass 1 of the anisotropic steps: the vectors whose divergences drive p and m."""
    E, A, F, B = 1 + 2 * m["Eps"], m["Eta"], m["F"], m["B"]
    S = torch.sqrt(1 - A * A)
    dP, dM = ops.grad(P), ops.grad(M)
    if "SinTheta" in m and ops.nd == 3:
        u = [m["SinTheta"] * m["CosPhi"], m["SinTheta"] * m["SinPhi"], m["CosTheta"]]
        gP, gM = (sum(w * d for w, d in zip(u, g)) for g in (dP, dM))
        FE = B * F * A * S
        tP = -B * (2 * m["Eps"] + F * A * A) * gP + FE * gM
        tM = FE * gP + B * F * A * A * gM
        return [B * E * d + w * tP for d, w in zip(dP, u)], [B * (1 - F) * d + w * tM for d, w in zip(dM, u)]
    if "SinTheta" in m:
        s, co = m["SinTheta"], m["CosTheta"]
        dP, dM = ([co * g[0] - s * g[1], s * g[0] + co * g[1]] for g in (dP, dM))
    p = [B * E * d for d in dP[:-1]] + [B * (1 - F * A * A) * dP[-1] + B * F * A * S * dM[-1]]
    q = [B * (1 - F) * d for d in dM[:-1]] + [B * F * A * S * dP[-1] + B * (1 - F + F * A * A) * dM[-1]]
    if "SinTheta" in m:  # 2D: back to the grid's axes, the rotation inside the D- stencil
        p, q = ([co * t[0] + s * t[1], -s * t[0] + co * t[1]] for t in (p, q))
    return p, q


def _step64(ops, m, st, dt):
    """One step of st = {pcur, pold, pspace[, mcur, mold, mspace]} in place of the old fields."""
    k = dt * dt * m["V"] ** 2 / m["B"]
    if "mcur" in st:
        p, q = _sandwich(ops, m, st["pcur"], st["mcur"])
        L = {"p": sum(ops.minus(t, a) for a, t in enumerate(p)), "m": sum(ops.minus(t, a) for a, t in enumerate(q))}
        del p, q
    else:
        L = {"p": sum(ops.minus(m["B"] * t, a) for a, t in enumerate(ops.grad(st["pcur"])))}
    for f, lap in L.items():
        cur, old = st[f + "cur"], st[f + "old"]
        new = k * lap - m["DtOmegaInvQ"] * (cur - old) - old + 2 * cur
        st[f + "old"], st[f + "cur"] = cur, torch.where(ops.r, new, old)
        st[f + "space"] = lap


def _state(waves, shape):
    z = lambda: torch.zeros(shape, dtype=torch.float64, device=DEV)  # noqa: E731
    st = {}
    for f, i in (("p", 0), ("m", 2)):
        if i < len(waves):
            st[f + "cur"], st[f + "old"], st[f + "space"] = waves[i].double(), waves[i + 1].double(), z()
    return st


def _scatter(st, src, wav, it):
    iu = torch.from_numpy(src[0] - 1).to(DEV)
    st["pcur"] = st["pcur"].clone()
    st["pcur"].view(-1).index_add_(0, iu, torch.from_numpy(src[2]).to(DEV).double() * float(wav[it - 1]))


def _gather(st, rec):
    return st["pcur"].view(-1)[torch.from_numpy(rec[0] - 1).to(DEV)]


def _shot64(shape, phys, fs, model, waves, nt, ntr, src=None, rec=None, wav=None):
    dt = float(np.float32(_dt(len(shape))))
    ops = _Ops(shape, fs)
    m = {k: t.double() for k, t in model.items()}
    st = _state(waves, shape)
    tr = torch.zeros((rec[0].size, ntr), dtype=torch.float64, device=DEV) if rec is not None else None
    for it in range(1, nt + 1):
        _step64(ops, m, st, dt)
        if src is not None:
            _scatter(st, src, wav, it)
            tr[:, it - 1] = _gather(st, rec)
    return ops, m, st, tr


def _rotated(ops, m, f):
    """The Born gradient triple (rotated in TTI)."""
    d = ops.grad(f)
    if "SinTheta" not in m:
        return d
    st, ct, sp, cp = m["SinTheta"], m["CosTheta"], m["SinPhi"], m["CosPhi"]
    return [ct * cp * d[0] + ct * sp * d[1] - st * d[2], -sp * d[0] + cp * d[1],
            st * cp * d[0] + st * sp * d[1] + ct * d[2]]


def _divergence(ops, m, t):
    if "SinTheta" in m:
        st, ct, sp, cp = m["SinTheta"], m["CosTheta"], m["SinPhi"], m["CosPhi"]
        t = [ct * cp * t[0] - sp * t[1] + st * cp * t[2], ct * sp * t[0] + cp * t[1] + st * sp * t[2],
             -st * t[0] + ct * t[2]]
    return sum(ops.minus(x, a) for a, x in enumerate(t))


def _born64(c, shape, model, waves, ex):
    ops = _Ops(shape, c["fs"])
    m = {k: t.double() for k, t in model.items()}
    dm, wf = ({k: t.double() for k, t in ex[n].items()} for n in ("dm", "wf"))
    V, B, dt = m["V"], m["B"], float(np.float32(_dt(3)))
    w = [x.double() for x in waves]
    k2, aniso, var = dt * dt * V * V / B, c["phys"] != "iso", c["variant"]
    img, zero = {}, torch.zeros(shape, dtype=torch.float64, device=DEV)
    fv = 2 * B / V ** 3
    if not aniso:
        src = zero
        corr = wf["pspace"] * w[1]
        if "V" in var:
            src = src + wf["pspace"] * fv * dm["v"]
            img["v"] = fv * corr
        if "B" in var:
            g = ops.grad(wf["pold"])
            src = src - wf["pspace"] * dm["b"] / V ** 2 + sum(ops.minus(dm["b"] * d, a) for a, d in enumerate(g))
            img["b"] = -corr / V ** 2 - sum(a * b for a, b in zip(g, ops.grad(w[1])))
        out = {"pcur": w[0] + k2 * src}
    else:
        img["v"] = fv * (wf["pspace"] * w[1] + wf["mspace"] * w[3])
        sp, sm = fv * dm["v"] * wf["pspace"], fv * dm["v"] * wf["mspace"]
        if var == "VEA":
            A, F, dE, dA = m["Eta"], m["F"], dm["ϵ"], dm["η"]
            g, h = _rotated(ops, m, wf["pold"]), _rotated(ops, m, wf["mold"])
            x = B * F * (1 - 2 * A * A) / torch.sqrt(1 - A * A)
            sp = sp + _divergence(ops, m, [2 * B * dE * g[0], 2 * B * dE * g[1],
                                           -2 * B * F * A * dA * g[2] + dA * x * h[2]])
            sm = sm + _divergence(ops, m, [zero, zero, 2 * B * F * A * dA * h[2] + dA * x * g[2]])
            b, n = _rotated(ops, m, w[1]), _rotated(ops, m, w[3])
            img["ϵ"] = -2 * B * (g[0] * b[0] + g[1] * b[1])
            img["η"] = (2 * B * F * A * g[2] - x * h[2]) * b[2] - (2 * B * F * A * h[2] + x * g[2]) * n[2]
        out = {"pcur": w[0] + k2 * sp, "mcur": w[2] + k2 * sm}
    out.update({"img " + n: t for n, t in img.items()})
    return out


def _sep64(c, shape, model, waves, ex):
    """Up- and down-going parts by the sign of the vertical wavenumber, a column at a time."""
    n = 2 * shape[-1]
    drop = slice(n // 2 + 1, n)
    adj = slice(1, n // 2) if c["cond"] == "FWI" else drop
    acc = 0.0
    pairs = [("pspace", waves[1])] + ([("mspace", waves[3])] if c["phys"] != "iso" else [])
    for name, old in pairs:
        parts = []
        for f, cut in ((ex["wf"][name], drop), (old, adj)):
            s = torch.fft.ifft(f.double(), n=n, dim=-1)  # sign +1, scaled by 1/n
            s[..., cut] = 0
            parts.append(torch.fft.fft(s, dim=-1)[..., :shape[-1]])
            del s
        acc = acc + (parts[0].real * parts[1].real - parts[0].imag * parts[1].imag)
    return 2 * model["B"].double() / model["V"].double() ** 3 * acc


def exact(c, seed):
    k = c["kind"]
    if k == "codec":
        return None  # a learned code with 16-bit weights has no value of its own in 64 bits
    if k == "batch":
        shots, traces = [], []
        for i, (shape, phys) in enumerate(_windows(c)):
            model, waves, _ = _fields(c, seed + 100 * i, shape, phys, True)
            src, rec = _acquisition(shape, 12, seed + i)
            nt = 64 * c["steps"]
            _, _, st, tr = _shot64(shape, phys, True, model, waves, c["steps"], nt, src, rec,
                                   _wavelet(nt, _dt(3), seed + i))
            shots.append(st)
            traces.append(tr)
        return {"shots": shots, "traces": traces}
    shape, phys, fs = _shape(c), c["phys"], c["fs"]
    dt = _dt(len(shape))
    model, waves, gen = _fields(c, seed, shape, phys, fs)
    if k == "loop2d":
        waves = [torch.zeros(shape, device=DEV) for _ in waves]
        src, rec = _acquisition(shape, 0, seed)
        _, _, st, tr = _shot64(shape, phys, fs, model, waves, c["nt"], c["nt"], src, rec, _wavelet(c["nt"], dt, seed))
        return {**st, "traces": tr}
    if k == "dropin":
        src, rec = _acquisition(shape, c["nrec"], seed)
        _, _, st, tr = _shot64(shape, phys, fs, model, waves, c["steps"], c["steps"], src, rec,
                               _wavelet(c["steps"], dt, seed))
        return {**st, "traces": tr}
    if k == "step":
        image = c["mode"] == "image"
        _, m, st, _ = _shot64(shape, phys, fs, model, waves, c["steps"], 0)
        if c["mode"] != "forward" and phys == "vti":  # the linear step writes no spatial derivatives
            st["pspace"] = st["mspace"] = torch.zeros(shape, dtype=torch.float64, device=DEV)
        if image:
            ex = _extras(c, shape, phys, gen)
            a = ex["wf"]["pspace"].double() * st["pold"]
            if phys != "iso":
                a = a + ex["wf"]["mspace"].double() * st["mold"]
            st["img"] = 2 * m["B"] / m["V"] ** 3 * a
        return st
    ex = _extras(c, shape, phys, gen)
    return _born64(c, shape, model, waves, ex) if k == "born" else _sep64(c, shape, model, waves, ex)
