"""Performance cases: the calls that programs of this framework make, over the sizes they make
them at.

Every case is one pass through the public Python interface (`ds2d_b200.Elastic2D`,
`ds2d_b200.unet.UNet`, `ds2d_b200.api.bandpass_filter`):

  forward      background modelling of a few shots, records on the host
  rtm          elastic RTM (forward, reconstruction, adjoint, imaging), images on the host
  elsrtm       one reference-mode ELSRTM iteration (PML, boundary strips, Born sets, NCC source)
  ac_normal    L^T L of the acoustic Born pair, the operator of CG-LSRTM and of training pairs
  lsrtm        a few CG-LSRTM iterations
  unet_forward the preconditioner network applied to images
  unet_train   one training step of it (loss, gradients, Adam)
  bandpass     the band-pass filter of the two gradient images

Grids, shot counts and networks are those of the benchmark and the tests, or lie between them;
time axes are shortened so that a pass stays within seconds (the work per time step does not
depend on their length).  `exact` restates each call in plain FP64 torch.
"""
import math

import numpy as np
import torch

from ds2d_b200 import Elastic2D, ShotGeom
from ds2d_b200.api import bandpass_filter
from ds2d_b200.unet import UNet

DX, DT, F0 = 10.0, 0.0008, 15.0
COEF = (1225.0 / 1024.0, -245.0 / 3072.0, 49.0 / 5120.0, -5.0 / 7168.0)


# ---- the cases ----------------------------------------------------------------------------------
def listed():
    return [
        # forward modelling of one shot on the small layered grid with a PML: many short steps,
        # so launch latency counts
        dict(name="forward_251x101", kind="forward", boundary="pml", allnx=251, allnz=101, nx=251,
             pml=20, nt=2000, shots=1),
        # the smallest migration: two shots on a test-sized grid
        dict(name="rtm_64x32", kind="rtm", boundary="random", strips="f32", device=False, allnx=64,
             allnz=32, nx=48, pml=10, nt=200, shots=2, wmin=0),
        # elastic RTM with the random boundary, 60 shots on one GPU: the benchmark's headline
        dict(name="rtm_1201x401", kind="rtm", boundary="random", strips="f32", device=True,
             allnx=1201, allnz=401, nx=1201, pml=40, nt=250, shots=60, wmin=0),
        # shots with their own aperture windows in one batch
        dict(name="rtm_uneven_4001x401", kind="rtm", boundary="random", strips="f32", device=True,
             allnx=4001, allnz=401, nx=1500, pml=40, nt=150, shots=24, wmin=400),
        # reference-mode ELSRTM iteration on a small survey, half-precision strips
        dict(name="elsrtm_251x101", kind="elsrtm", strips="bf16", allnx=251, allnz=101, nx=251,
             pml=20, nt=500, shots=4),
        # reference-mode ELSRTM iteration at the benchmark's size
        dict(name="elsrtm_1201x401", kind="elsrtm", strips="f32", allnx=1201, allnz=401, nx=1201,
             pml=40, nt=400, shots=16),
        # CG-LSRTM on a test-sized survey
        dict(name="lsrtm_96x48", kind="lsrtm", allnx=96, allnz=48, nx=96, pml=12, nt=300, shots=8,
             iters=3),
        # the normal operator of CG-LSRTM on the application grid
        dict(name="ac_normal_2001x601", kind="ac_normal", boundary="random", strips="f32",
             allnx=2001, allnz=601, nx=2001, pml=20, nt=100, shots=16),
        # the same operator with the PML and BF16 boundary strips
        dict(name="ac_normal_pml_1001x301", kind="ac_normal", boundary="pml", strips="bf16",
             allnx=1001, allnz=301, nx=1001, pml=20, nt=200, shots=8),
        # the preconditioner network on one image of the application grid
        dict(name="unet_forward_2008x608", kind="unet_forward", base=32, n=1, h=2008, w=608),
        # a training step on the batch of crops that the training pipeline draws
        dict(name="unet_train_8x128x256", kind="unet_train", base=32, n=8, h=128, w=256),
        # the gradient filter at the end of an iteration, on the benchmark's grid
        dict(name="bandpass_1201x401", kind="bandpass", nx=1201, nz=401, z1=10, z2=60),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "rtm", "elsrtm", "lsrtm", "ac_normal", "unet_forward",
                       "unet_train", "bandpass"])
    if kind == "unet_forward":
        return dict(kind=kind, base=32, n=rng.randint(1, 3), h=8 * _log(rng, 6, 200),
                    w=8 * _log(rng, 6, 70))
    if kind == "unet_train":
        return dict(kind=kind, base=rng.choice([32, 32, 32, 64]), n=rng.randint(1, 8),
                    h=8 * _log(rng, 4, 24), w=8 * _log(rng, 4, 32))
    if kind == "bandpass":
        return dict(kind=kind, nx=_log(rng, 60, 1500), nz=_log(rng, 40, 600),
                    z1=rng.choice([0, 5, 12]), z2=rng.randint(20, 80))
    if kind == "lsrtm":
        nx = _log(rng, 60, 400)
        return dict(kind=kind, allnx=nx, allnz=_log(rng, 36, 160), nx=nx, pml=rng.randint(12, 24),
                    nt=rng.randint(150, 400), shots=rng.randint(2, 10), iters=rng.randint(2, 4))
    allnx, allnz = _log(rng, 90, 1300), _log(rng, 50, 420)
    nx = rng.choice([allnx, rng.randint(max(64, allnx // 2), allnx)])
    pml = rng.randint(10, 40)
    shots = _log(rng, 1, 20)
    nt = rng.randint(120, 500)
    cap = {"forward": 4.0e9, "rtm": 3.0e9, "elsrtm": 1.2e9, "ac_normal": 1.5e9}[kind]
    cells = (nx + 2 * pml) * (allnz + 2 * pml) * nt
    shots = max(1, min(shots, int(cap / cells)))
    c = dict(kind=kind, allnx=allnx, allnz=allnz, nx=nx, pml=pml, nt=nt, shots=shots)
    if kind == "forward":
        c.update(boundary=rng.choice(["pml", "random"]))
    elif kind == "rtm":
        c.update(boundary=rng.choice(["pml", "random", "random"]),
                 strips=rng.choice(["f32", "f16", "bf16"]), device=rng.random() < 0.5,
                 wmin=rng.choice([0, max(48, nx // 3)]))
    elif kind == "elsrtm":
        c.update(strips=rng.choice(["f32", "f16", "bf16"]), nt=max(nt, 300))
    else:
        c.update(boundary=rng.choice(["pml", "random"]), strips=rng.choice(["f32", "bf16"]))
    return c


# ---- inputs, from the seed alone ----------------------------------------------------------------
def _ricker(nt):
    t = np.arange(nt) * DT - int(1.0 / F0 / DT) * DT
    a = (math.pi * F0 * t) ** 2
    return (np.exp(-a) * (1.0 - 2.0 * a)).astype(np.float32)


def _velocity(nx, nz, rng, vtop, vbot, layers):
    """vtop..vbot with depth, `layers` dipping steps (0: continuous), a few Gaussian lenses."""
    x, z = np.arange(nx)[:, None] / nx, np.arange(nz)[None, :] / nz
    depth = np.clip(z + rng.uniform(-0.1, 0.1) * (x - 0.5), 0.0, 0.9999)
    if layers:
        depth = np.floor(depth * layers) / max(layers - 1, 1)
    v = vtop + (vbot - vtop) * depth
    for _ in range(4):
        cx, cz, r = rng.uniform(0.1, 0.9), rng.uniform(0.2, 0.9), rng.uniform(0.05, 0.15)
        v = v * (1.0 + rng.uniform(-0.06, 0.06) * np.exp(-((x - cx) ** 2 + (z - cz) ** 2) / (2 * r * r)))
    return np.clip(v, vtop, vbot).astype(np.float32)


def _reflectivity(nx, nz, rng):
    """Sparse spikes of 5 % of the cells, N(0, 0.05), none at the surface."""
    m = np.where(rng.random((nx, nz)) < 0.05, rng.normal(0.0, 0.05, (nx, nz)), 0.0)
    m[:, :4] = 0.0
    return m.astype(np.float32)


def _shots(c, rng, reach=None):
    """Shots along the surface with receivers two cells down on the window's columns (those
    within `reach` columns of the source, if given)."""
    allnx, pml, out = c["allnx"], c["pml"], []
    n = c["shots"]
    xs = np.linspace(0, allnx - 1, n).round().astype(int) if n > 1 else [allnx // 2]
    for sx in xs:
        w = c["nx"]
        if c.get("wmin"):
            w = int(rng.integers(c["wmin"], c["nx"] + 1))
        left = int(np.clip(sx - w // 2, 0, allnx - w))
        isx = pml + int(sx) - left
        cols = np.arange(pml, pml + w, dtype=np.int32)
        if reach:
            cols = cols[np.abs(cols - isx) <= reach]
        out.append(ShotGeom(win_left=left, isx=isx, isz=pml, igz=pml + 2, igx=cols, nx=w))
    return out


def _records(shots, nt, seed):
    """Records of a few hyperbolic events per shot, [sum ntr][nt] twice, on the GPU."""
    g = torch.Generator().manual_seed(seed)
    t = torch.arange(nt, device="cuda") * DT
    out = []
    for _ in range(2):
        rows = []
        for s in shots:
            off = torch.from_numpy(np.abs(s.igx.astype(np.float32) - s.isx)).cuda()[:, None] * DX
            rec = torch.zeros(len(s.igx), nt, device="cuda")
            for k in range(4):
                u = torch.rand(3, generator=g).tolist()
                t0 = 0.0 if k == 0 else u[0] * 0.7 * nt * DT
                v = 2000.0 + 2500.0 * u[1]
                a = (math.pi * F0 * (t - torch.sqrt(t0 * t0 + (off / v) ** 2) - 1.0 / F0)) ** 2
                rec += (0.3 + u[2]) * (1.0 if k == 0 else 0.4) * torch.exp(-a) * (1.0 - 2.0 * a)
            rows.append(rec)
        out.append(torch.cat(rows).contiguous())
    return out


def _acoustic(c):
    return c["kind"] in ("ac_normal", "lsrtm")


def _inputs(c, seed):
    """Everything the call reads: models, wavelet, shots, and images or records."""
    rng = np.random.default_rng(seed)
    i = {}
    if c["kind"] == "bandpass":
        for k in ("pp", "ps"):
            i[k] = rng.standard_normal((c["nx"], c["nz"])).astype(np.float32)
        return i
    if c["kind"].startswith("unet"):
        i["params"] = _params(c["base"], rng)
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (c["n"], c["h"], c["w"])
        x = torch.randn(shape, generator=g, device="cuda")
        i["x"] = x / x.pow(2).mean(dim=(1, 2), keepdim=True).sqrt()
        i["t"] = torch.randn(shape, generator=g, device="cuda")
        return i
    nx, nz, nt = c["allnx"], c["allnz"], c["nt"]
    i["wavelet"], i["seed"] = _ricker(nt), seed
    if c["kind"] == "forward":
        i["vp"] = _velocity(nx, nz, rng, 2500.0, 5500.0, 4)
        i["rho"] = (310.0 * i["vp"].astype(np.float64) ** 0.25).astype(np.float32)
    elif _acoustic(c):
        i["vp"] = _velocity(nx, nz, rng, 1800.0, 4500.0, 0)
        i["m"] = _reflectivity(nx, nz, rng)
    else:
        i["vp"] = _velocity(nx, nz, rng, 2000.0, 6000.0, 0)
    i["vs"] = np.zeros_like(i["vp"]) if _acoustic(c) else (i["vp"] / 1.73).astype(np.float32)
    # The NCC source divides by each trace's norm: receivers that the wavefield reaches within
    # the time axis.
    i["shots"] = _shots(c, rng, reach=nt // 10 if c["kind"] == "elsrtm" else None)
    if c["kind"] == "elsrtm":
        i["pp"], i["ps"] = (_reflectivity(nx, nz, rng) for _ in range(2))
    if c["kind"] in ("rtm", "elsrtm", "lsrtm"):
        i["rz"], i["rx"] = _records(i["shots"], nt, seed)
    return i


def _layers(base):
    """(cin, cout, kernel) of the network's convolutions in parameter order."""
    c = [base, 2 * base, 4 * base, 8 * base]
    out, prev = [], 1
    for l in range(4):
        out += [(prev, c[l], 3), (c[l], c[l], 3)]
        prev = c[l]
    for l in (2, 1, 0):
        out += [(prev + c[l], c[l], 3), (c[l], c[l], 3)]
        prev = c[l]
    return out + [(c[0], 1, 1)]


def _params(base, rng):
    """He-normal weights [k][k][cout][cin] and small biases, flat."""
    parts = []
    for ci, co, k in _layers(base):
        parts.append(rng.standard_normal(k * k * co * ci) * math.sqrt((2.0 if k == 3 else 1.0) / (ci * k * k)))
        parts.append(0.05 * rng.standard_normal(co))
    return np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    c, i = case, _inputs(case, seed)
    s = dict(case=c, i=i)
    if c["kind"] == "bandpass":
        return s
    if c["kind"].startswith("unet"):
        s["net"] = UNet(base=c["base"], max_n=c["n"], max_h=c["h"], max_w=c["w"])
        s["net"].set_params(i["params"])
        s["y"] = torch.empty_like(i["x"])
        return s
    e = Elastic2D(c["allnx"], c["allnz"], c["nx"], c["pml"], c["nt"], DX, DX, DT,
                  boundary=c.get("boundary", "random" if c["kind"] == "lsrtm" else "pml"),
                  strips=c.get("strips", "f32"), max_shots=c["shots"], max_ntr=c["nx"],
                  seed=i["seed"])
    e.set_models(i["vp"], i["vs"], i.get("rho"))
    e.set_wavelet(i["wavelet"])
    if c["kind"] == "elsrtm":
        e.set_image(i["pp"], i["ps"])
    if c["kind"] == "lsrtm" or (c["kind"] == "rtm" and not c["device"]):
        s["hz"], s["hx"] = i["rz"].cpu().numpy(), i["rx"].cpu().numpy()
    if c["kind"] == "ac_normal":
        s["m"] = torch.from_numpy(i["m"]).cuda()
        s["img"] = torch.zeros_like(s["m"])
    s["e"] = e
    return s


# ---- one pass -----------------------------------------------------------------------------------
def run(state):
    c, i, e = state["case"], state["i"], state.get("e")
    kind = c["kind"]
    if kind == "forward":
        return e.forward(i["shots"])
    if kind == "rtm":
        if c["device"]:
            e.rtm_device(i["shots"], i["rz"].data_ptr(), i["rx"].data_ptr())
        else:
            e.rtm(i["shots"], state["hz"], state["hx"])
        return e.read_images(which=("pp_grad", "ps_grad", "illumination"))
    if kind == "elsrtm":
        misfit = e.elsrtm_device(i["shots"], i["rz"].data_ptr(), i["rx"].data_ptr(), 1)
        images = e.read_images(which=("pp_grad", "ps_grad", "illumination", "b_pp", "b_ps"))
        return {"misfit": misfit, **images}
    if kind == "lsrtm":
        return e.lsrtm(i["shots"], state["hz"], state["hx"], c["iters"])
    if kind == "ac_normal":
        e.ac_normal_device(i["shots"], state["m"].data_ptr(), state["img"].data_ptr())
        return state["img"]
    if kind == "unet_forward":
        state["net"].forward(i["x"].data_ptr(), state["y"].data_ptr(), c["n"], c["h"], c["w"])
        return state["y"]
    if kind == "unet_train":
        loss, grads = state["net"].loss_grad(i["x"].data_ptr(), i["t"].data_ptr(), c["n"], c["h"],
                                             c["w"], want_grads=True)
        state["net"].adam_step(lr=1e-3)
        return {"loss": loss, "grads": grads}
    return bandpass_filter(i["pp"], i["ps"], c["z1"], c["z2"])


# ---- the work a pass cannot do without ----------------------------------------------------------
L2_BYTES = 126e6


def work(case):
    """Inputs read and outputs written once, plus, where the wavefields of the batch exceed the
    on-chip memory, each propagation's state read and written once per time step."""
    c, kind = case, case["kind"]
    if kind == "bandpass":
        n = c["nx"] * c["nz"]
        return dict(bytes=2 * 2 * 4 * n, flops=2 * 2 * 5 * n * math.log2(n))
    if kind.startswith("unet"):
        macs, nw = 0.0, 0
        px = [c["n"] * c["h"] * c["w"] / 4 ** l for l in (0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0)]
        for (ci, co, k), p in zip(_layers(c["base"]), px):
            macs += p * ci * co * k * k
            nw += k * k * ci * co + co
        if kind == "unet_forward":
            return dict(bytes=4 * (2 * px[0] + nw), flops=2 * macs)
        return dict(bytes=4 * (2 * px[0] + 7 * nw), flops=6 * macs)
    w = (c["wmin"] + c["nx"]) / 2 if c.get("wmin") else c["nx"]
    cells = c["shots"] * (w + 2 * c["pml"]) * (c["allnz"] + 2 * c["pml"])
    model = c["allnx"] * c["allnz"] * 4
    rec = c["shots"] * w * c["nt"] * 4 * 2
    # fields of one propagation, propagations, flops per cell and step of one propagation
    fields, props, fl = {"forward": (5, 1, 150), "rtm": (5, 3, 160), "elsrtm": (5, 6, 160),
                         "ac_normal": (3, 5, 70), "lsrtm": (3, 5, 70)}[kind]
    if kind == "lsrtm":
        props = 2 * c["iters"] + 3 * (c["iters"] + 1)
    state = 4 * fields * cells
    moved = 2 * state * props * c["nt"] if 2 * state > L2_BYTES else 0
    return dict(bytes=rec + 6 * model + moved, flops=fl * props * cells * c["nt"])


# ---- the same calls in FP64 ---------------------------------------------------------------------
def _diff(f, axis, ahead):
    """8-tap staggered difference along x (axis 1) or z (2): sum c_i (f[+i] - f[1-i]) (ahead) or
    sum c_i (f[i-1] - f[-i]); zero within 4 cells of the grid's edges."""
    out = torch.zeros_like(f)
    n = f.shape
    inner = out[:, 4:n[1] - 4, 4:n[2] - 4]

    def at(k):
        sx, sz = (k, 0) if axis == 1 else (0, k)
        return f[:, 4 + sx:n[1] - 4 + sx, 4 + sz:n[2] - 4 + sz]

    for j, cf in enumerate(COEF, 1):
        hi, lo = (j, 1 - j) if ahead else (j - 1, -j)
        inner.add_(at(hi) - at(lo), alpha=cf)
    return out


def _band_factor(seed, shot, nx, nz):
    """Random band: u in [0, 1) from SplitMix64 of (seed, shot, cell), factor 0.6 + 0.4 u."""
    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    with np.errstate(over="ignore"):
        h = mix(np.array([seed], np.uint64) ^ (np.array([0xD1B54A32D192ED03], np.uint64) * np.uint64(shot + 1)))
        key = (np.arange(nx, dtype=np.uint64)[:, None] << np.uint64(32)) | np.arange(nz, dtype=np.uint64)[None, :]
        u = (mix(h ^ key) >> np.uint64(40)).astype(np.float64) / 16777216.0
    return 0.6 + 0.4 * u


class _Scheme:
    """The staggered-grid scheme of a group of shots with one window width, FP64 on the GPU."""

    def __init__(self, c, i, shots, ids):
        self.c, self.i, self.shots = c, i, shots
        rbc = c.get("boundary", "random" if c["kind"] == "lsrtm" else "pml") == "random"
        P, nz, self.dt, self.dx = c["pml"], c["allnz"], float(np.float32(DT)), DX
        w = shots[0].nx
        self.P, self.w, self.nz, self.nt = P, w, nz, c["nt"]
        X, Z = w + 2 * P, nz + 2 * P
        jx, jz = np.clip(np.arange(X) - P, 0, w - 1), np.clip(np.arange(Z) - P, 0, nz - 1)
        band = np.ones((X, Z), bool)
        band[P:X - P, P:Z - P] = False

        def window(a, fill=None):
            return np.stack([(a if fill is None else fill)[np.ix_(s.win_left + jx, jz)] for s in shots]).astype(np.float64)

        vp, vs = window(i["vp"]), window(i["vs"])
        if rbc:
            f = np.stack([np.where(band, _band_factor(i["seed"], k, X, Z), 1.0) for k in ids])
            vp, vs = vp * f, vs * f
        rho = window(i["rho"]) if "rho" in i else np.full_like(vp, 2000.0)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        self.lam, self.mu = dev(rho * (vp ** 2 - 2 * vs ** 2)), dev(rho * vs ** 2)
        self.l2m, self.b = self.lam + 2 * self.mu, dev(1.0 / rho)
        self.kpp, self.kps = dev(-2 * vp ** 2 * rho), dev(-2 * vs ** 2 * rho)
        self.rbc = rbc
        if not rbc:
            k = math.log10(1000.0) * 5.0 * vp / (2.0 * P)
            prof = lambda n: np.maximum(np.maximum(P - np.arange(n), np.arange(n) - (n - P)), 0) / P
            hx = dev(k * prof(X)[None, :, None] ** 4 * self.dt * 0.5)
            hz = dev(k * prof(Z)[None, None, :] ** 4 * self.dt * 0.5)
            self.d1x, self.rx, self.d1z, self.rz = 1 - hx, 1 / (1 + hx), 1 - hz, 1 / (1 + hz)
        self.interior = (slice(None), slice(P, X - P), slice(P, Z - P))
        if "m" in i or "pp" in i:
            self.dmp = dev(window(i["m"] if "m" in i else i["pp"]))
            self.dms = dev(window(i["ps"])) if "ps" in i else torch.zeros_like(self.dmp)
        self.src = (torch.arange(len(shots), device="cuda"),
                    torch.tensor([s.isx for s in shots], device="cuda"),
                    torch.tensor([s.isz for s in shots], device="cuda"))
        sid = np.concatenate([np.full(len(s.igx), n) for n, s in enumerate(shots)])
        self.rec = (torch.from_numpy(sid).cuda(),
                    torch.from_numpy(np.concatenate([s.igx for s in shots]).astype(np.int64)).cuda(),
                    torch.tensor(np.concatenate([np.full(len(s.igx), s.igz) for s in shots]), device="cuda"))
        # Boundary strips: within 4 cells of the interior's edge, over the interior's extent.
        s = np.zeros((X, Z), bool)
        s[P:X - P, P - 4:P + 4] = s[P:X - P, Z - P - 4:Z - P + 4] = True
        s[P - 4:P + 4, P:Z - P] = s[X - P - 4:X - P + 4, P:Z - P] = True
        self.strip, self.outer = torch.from_numpy(s).cuda(), torch.from_numpy(s & band).cuda()
        self.shape = (len(shots), X, Z)

    def zeros(self, n):
        return [torch.zeros(self.shape, dtype=torch.float64, device="cuda") for _ in range(n)]

    def damp(self, parts, incs, x_then_z):
        """parts += incs with the split damping (x part, z part, ...); returns nothing."""
        for p, u, ax in zip(parts, incs, x_then_z):
            if self.rbc:
                p.add_(u)
            elif ax == "x":
                p.copy_((self.d1x * p + u) * self.rx)
            else:
                p.copy_((self.d1z * p + u) * self.rz)

    # -- elastic ------------------------------------------------------------------------------
    def field(self):
        """vx, vz, txx, tzz, txz and, with a PML, their x and z parts."""
        f = dict(zip(("vx", "vz", "txx", "tzz", "txz"), self.zeros(5)))
        if not self.rbc:
            f["split"] = self.zeros(10)
        return f

    def _apply(self, f, names, incs):
        if self.rbc:
            for k, n in enumerate(names):
                f[n].add_(incs[2 * k] + incs[2 * k + 1])
            return
        first = 0 if names[0] == "vx" else 4
        parts = f["split"][first:first + 2 * len(names)]
        self.damp(parts, incs, "xz" * len(names))
        for k, n in enumerate(names):
            f[n].copy_(parts[2 * k] + parts[2 * k + 1])

    def velocity(self, f, it=None, ov=None):
        txx, tzz, txz = f["txx"], f["tzz"], f["txz"]
        if ov is not None:
            txx, tzz, txz = txx + ov[0], tzz + ov[1], txz + ov[2]
        elif it is not None:
            txx, tzz = txx.clone(), tzz.clone()
            for t in (txx, tzz):
                t[self.src] += float(self.i["wavelet"][it])
        cb = self.b * (self.dt / self.dx)
        self._apply(f, ("vx", "vz"), (cb * _diff(txx, 1, True), cb * _diff(txz, 2, False),
                                      cb * _diff(txz, 1, False), cb * _diff(tzz, 2, True)))

    def stress(self, f):
        q = self.dt / self.dx
        xx, zz = q * _diff(f["vx"], 1, False), q * _diff(f["vz"], 2, False)
        zx, xz = q * _diff(f["vz"], 1, True), q * _diff(f["vx"], 2, True)
        self._apply(f, ("txx", "tzz", "txz"), (self.l2m * xx, self.lam * zz, self.lam * xx,
                                               self.l2m * zz, self.mu * zx, self.mu * xz))

    def born(self, f):
        """Born source of the velocities, on the interior."""
        out, s = self.zeros(3), self.interior
        P = -2 * self.l2m * self.dmp
        Q = P + 4 * self.mu * self.dms
        xx, zz = _diff(f["vx"], 1, False) / self.dx, _diff(f["vz"], 2, False) / self.dx
        sh = (_diff(f["vz"], 1, True) + _diff(f["vx"], 2, True)) / self.dx
        out[0][s] = (P * xx + Q * zz)[s]
        out[1][s] = (Q * xx + P * zz)[s]
        out[2][s] = (-2 * self.mu * self.dms * sh)[s]
        return out

    def reverse(self, f, strip=None, ov=None):
        """One step back on the interior (stress, then velocity); returns the strains."""
        s, q = self.interior, self.dt / self.dx
        vx, vz = f["vx"], f["vz"]
        if strip is not None:
            vx, vz = vx.clone(), vz.clone()
            vx[:, self.strip], vz[:, self.strip] = strip
        xx, zz = _diff(vx, 1, False), _diff(vz, 2, False)
        zx, xz = _diff(vz, 1, True), _diff(vx, 2, True)
        f["txx"][s] -= (q * (self.l2m * xx + self.lam * zz))[s]
        f["tzz"][s] -= (q * (self.lam * xx + self.l2m * zz))[s]
        f["txz"][s] -= (q * self.mu * (zx + xz))[s]
        if callable(ov):
            ov = ov()
        t = [f["txx"], f["tzz"], f["txz"]] if ov is None else [f[n] + o for n, o in zip(("txx", "tzz", "txz"), ov)]
        cb = self.b * q
        f["vx"][s] -= (cb * (_diff(t[0], 1, True) + _diff(t[2], 2, False)))[s]
        f["vz"][s] -= (cb * (_diff(t[2], 1, False) + _diff(t[1], 2, True)))[s]
        if strip is not None:
            o = self.outer[self.strip]
            f["vx"][:, self.outer], f["vz"][:, self.outer] = strip[0][:, o], strip[1][:, o]
        return [a / self.dx for a in (xx, zz, xz, zx)]

    def adjoint(self, a, rz, rx):
        """Modulus-free adjoint step: stresses of the injected velocities, then velocities."""
        q = self.dt / self.dx
        vx, vz = a["vx"].clone(), a["vz"].clone()
        vz[self.rec] += rz
        vx[self.rec] += rx
        xx, zz = -q * _diff(vx, 1, False), -q * _diff(vz, 2, False)
        zx, xz = -q * _diff(vz, 1, True), -q * _diff(vx, 2, True)
        if self.rbc:
            a["txx"].add_(xx), a["tzz"].add_(zz), a["txz"].add_(zx + xz)
        else:
            self.damp((a["txx"], a["tzz"]), (xx, zz), "xz")
            self.damp(a["split"][8:], (zx, xz), "xz")
            a["txz"].copy_(a["split"][8] + a["split"][9])
        cb = self.b * q
        m = self.mu * a["txz"]
        self._apply(a, ("vx", "vz"), (-cb * _diff(self.l2m * a["txx"] + self.lam * a["tzz"], 1, True),
                                      -cb * _diff(m, 2, False), -cb * _diff(m, 1, False),
                                      -cb * _diff(self.l2m * a["tzz"] + self.lam * a["txx"], 2, True)))

    def image(self, img, g, a):
        s = self.interior
        xx, zz, xz, zx = (v[s] for v in g)
        txx, tzz, txz = a["txx"][s], a["tzz"][s], a["txz"][s]
        img[0].add_(self.kpp[s] * (xx + zz) * (txx + tzz))
        img[1].add_(self.kps[s] * (-2 * (xx * tzz + zz * txx) + (xz + zx) * txz))

    def images(self, n):
        return [torch.zeros(len(self.shots), self.w, self.nz, dtype=torch.float64, device="cuda") for _ in range(n)]

    def place(self, imgs, full):
        for k, im in enumerate(imgs):
            for n, s in enumerate(self.shots):
                full[k, s.win_left:s.win_left + self.w] += im[n]

    def forward(self):
        f, out = self.field(), ([], [])
        for it in range(self.nt):
            self.velocity(f, it)
            out[0].append(f["vz"][self.rec]), out[1].append(f["vx"][self.rec])
            self.stress(f)
        return [torch.stack(o, 1) for o in out]

    def keep(self, f):
        return f["vx"][:, self.strip].clone(), f["vz"][:, self.strip].clone()

    def rtm(self, rz, rx, full):
        f, strips = self.field(), []
        for it in range(self.nt):
            self.velocity(f, it)
            self.stress(f)
            if not self.rbc:
                strips.append(self.keep(f))
        a, img = self.field(), self.images(3)
        for it in range(self.nt - 1, -1, -1):
            g = self.reverse(f, strips[it] if strips else None)
            self.adjoint(a, rz[:, it], rx[:, it])
            self.image(img[:2], g, a)
            img[2].add_((f["vx"] ** 2 + f["vz"] ** 2)[self.interior])
        self.place(img, full)

    def elsrtm(self, oz, ox, full):
        f, b1, b2, st, st1 = self.field(), self.field(), self.field(), [], []
        lz, lx = [], []
        for it in range(self.nt):
            self.velocity(f, it)
            self.stress(f)
            self.velocity(b1, ov=self.born(f))
            self.stress(b1)
            self.velocity(b2, ov=self.born(b1))
            self.stress(b2)
            lz.append(b1["vz"][self.rec] + b2["vz"][self.rec])
            lx.append(b1["vx"][self.rec] + b2["vx"][self.rec])
            st.append(self.keep(f)), st1.append(self.keep(b1))
        lz, lx = torch.stack(lz, 1), torch.stack(lx, 1)
        ntr = torch.tensor([len(s.igx) for s in self.shots], device="cuda")[self.rec[0]].double()
        res, mis = [], 0.0
        for d, o in ((lz, oz), (lx, ox)):
            dd, oo, do = ((u * v).sum(1, keepdim=True) for u, v in ((d, d), (o, o), (d, o)))
            res.append((do / dd * d - o) / (dd.sqrt() * oo.sqrt()))
            mis -= float((do[:, 0] / (dd[:, 0].sqrt() * oo[:, 0].sqrt()) / (2 * ntr)).sum())
        a, img = self.field(), self.images(5)
        for it in range(self.nt - 1, -1, -1):
            g = self.reverse(f, st[it])
            g1 = self.reverse(b1, st1[it], ov=lambda: self.born(f))
            self.adjoint(a, res[0][:, it], res[1][:, it])
            self.image(img[:2], g, a)
            img[2].add_((f["vx"] ** 2 + f["vz"] ** 2)[self.interior])
            self.image(img[3:], g1, a)
        self.place(img, full)
        return mis

    # -- acoustic Born pair -------------------------------------------------------------------
    def ac_state(self):
        return self.zeros(4)  # vx, vz and the two parts of s

    def ac_step(self, y, it=None, ov=None):
        q = self.dt / self.dx
        S = y[2] + y[3]
        if ov is not None:
            S = S + ov
        if it is not None:
            S[self.src] += float(self.i["wavelet"][it])
        self.damp(y[:2], (self.b * q * _diff(S, 1, True), self.b * q * _diff(S, 2, True)), "xz")
        dx, dz = _diff(y[0], 1, False), _diff(y[1], 2, False)
        self.damp(y[2:], (self.lam * q * dx, self.lam * q * dz), "xz")
        e = torch.zeros_like(S)
        e[self.interior] = (-2 * self.lam * (dx + dz) / self.dx)[self.interior]
        return e

    def ac_forward(self, m):
        """Records of L m."""
        mw = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
        for n, s in enumerate(self.shots):
            mw[n, self.P:self.P + self.w, self.P:self.P + self.nz] = m[s.win_left:s.win_left + self.w]
        bg, sc, rz, rx = self.ac_state(), self.ac_state(), [], []
        for it in range(self.nt):
            e = self.ac_step(bg, it) * mw
            self.ac_step(sc, ov=e)
            rz.append(sc[1][self.rec]), rx.append(sc[0][self.rec])
        return torch.stack(rz, 1), torch.stack(rx, 1)

    def ac_adjoint(self, rz, rx, grad):
        """grad += L^T (rz, rx), with the background's Born factors kept for every step."""
        bg, q = self.ac_state(), self.dt / self.dx
        es = [self.ac_step(bg, it)[self.interior].clone() for it in range(self.nt)]
        yx, yz, sx, sz = self.ac_state()
        img = self.images(1)[0]
        dec = lambda d, r: (1.0 if self.rbc else d * r)
        inv = lambda r: (1.0 if self.rbc else r)
        k = {} if self.rbc else dict(d1x=self.d1x, rx=self.rx, d1z=self.d1z, rz=self.rz)
        g = lambda n: k.get(n, 1.0)
        upd = torch.zeros(self.shape[1:], dtype=torch.float64, device="cuda")
        upd[4:-4, 4:-4] = 1.0
        for it in range(self.nt - 1, -1, -1):
            yx *= dec(g("d1x"), g("rx"))
            yz *= dec(g("d1z"), g("rz"))
            yz[self.rec] += rz[:, it]
            yx[self.rec] += rx[:, it]
            yx -= q * _diff(self.lam * sx * inv(g("rx")), 1, True)
            yz -= q * _diff(self.lam * sz * inv(g("rz")), 2, True)
            gs = -(_diff(self.b * q * yx * inv(g("rx")), 1, False) + _diff(self.b * q * yz * inv(g("rz")), 2, False))
            gs *= upd
            sx *= dec(g("d1x"), g("rx"))
            sz *= dec(g("d1z"), g("rz"))
            sx += gs
            sz += gs
            img += es[it] * gs[self.interior]
        self.place([img], grad[None])


def _groups(c, i):
    """Schemes of the shots, grouped by window width, with each group's shots and trace rows."""
    rows, n = [], 0
    for s in i["shots"]:
        rows.append(np.arange(n, n + len(s.igx)))
        n += len(s.igx)
    widths = {}
    for k, s in enumerate(i["shots"]):
        widths.setdefault(s.nx, []).append(k)
    for ids in widths.values():
        yield (_Scheme(c, i, [i["shots"][k] for k in ids], ids),
               torch.from_numpy(np.concatenate([rows[k] for k in ids])).cuda())


def _exact_unet(c, i):
    F = torch.nn.functional
    flat = torch.from_numpy(i["params"]).double().cuda().requires_grad_(c["kind"] == "unet_train")
    layers, off = [], 0
    for ci, co, k in _layers(c["base"]):
        w = flat[off:off + k * k * co * ci].view(k, k, co, ci).permute(2, 3, 0, 1)
        off += k * k * co * ci
        layers.append((w, flat[off:off + co], k // 2))
        off += co
    nxt = iter(layers)

    def conv(v, act=True):
        w, b, p = next(nxt)
        v = F.conv2d(v, w, b, padding=p)
        return v.relu() if act else v

    h, skips = i["x"].double()[:, None], []
    for l in range(4):
        h = conv(conv(h))
        if l < 3:
            skips.append(h)
            h = F.avg_pool2d(h, 2)
    for l in (2, 1, 0):
        h = conv(conv(torch.cat([F.interpolate(h, scale_factor=2, mode="nearest"), skips[l]], 1)))
    y = conv(h, act=False)[:, 0]
    if c["kind"] == "unet_forward":
        return y
    loss = (y - i["t"].double()).pow(2).mean()
    loss.backward()
    return {"loss": float(loss), "grads": flat.grad}


def _exact_bandpass(c, i):
    nx, nz = c["nx"], c["nz"]
    y, x = np.arange(nx)[:, None] - nx // 2, np.arange(nz)[None, :] - nz // 2
    d2 = (x ** 2 + (nz / nx * y) ** 2).astype(np.float64)
    k = np.exp(-d2 / (2.0 * c["z2"] ** 2))
    if c["z1"]:
        k = k - np.exp(-d2 / (2.0 * c["z1"] ** 2))
    k = np.maximum(k, 0.0)
    k /= k.max()
    hx, hz = nx // 2, nz // 2
    swapped = k.copy()  # quadrants exchanged; the last row / column of an odd size stay
    swapped[:2 * hx, :2 * hz] = np.roll(k[:2 * hx, :2 * hz], (hx, hz), (0, 1))
    out = []
    for name in ("pp", "ps"):
        g = np.fft.ifft2(swapped * np.fft.fft2(i[name].astype(np.float64)))
        out.append(g.real - g.imag)
    return tuple(out)


def exact(case, seed):
    c, i = case, _inputs(case, seed)
    kind = c["kind"]
    if kind == "bandpass":
        return _exact_bandpass(c, i)
    if kind.startswith("unet"):
        return _exact_unet(c, i)
    nx, nz = c["allnx"], c["allnz"]
    new = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")
    if "rz" in i:
        rz, rx = i["rz"].double(), i["rx"].double()
    ntr = sum(len(s.igx) for s in i["shots"])
    if kind == "forward":
        out = new(2, ntr, c["nt"])
        for sch, rows in _groups(c, i):
            out[0][rows], out[1][rows] = sch.forward()
        return tuple(out)
    if kind == "rtm":
        full = new(3, nx, nz)
        for sch, rows in _groups(c, i):
            sch.rtm(rz[rows], rx[rows], full)
        return dict(zip(("pp_grad", "ps_grad", "illumination"), full))
    if kind == "elsrtm":
        full, mis = new(5, nx, nz), 0.0
        for sch, rows in _groups(c, i):
            mis += sch.elsrtm(rz[rows], rx[rows], full)
        return {"misfit": mis, **dict(zip(("pp_grad", "ps_grad", "illumination", "b_pp", "b_ps"), full))}
    (sch, rows), = _groups(c, i)

    def transpose(dz, dx):
        g = new(nx, nz)
        sch.ac_adjoint(dz, dx, g)
        return g

    if kind == "ac_normal":
        return transpose(*sch.ac_forward(torch.from_numpy(i["m"]).double().cuda()))
    # CGLS from m = 0
    m, r = new(nx, nz), [rz.clone(), rx.clone()]
    norm = float(sum(v.square().sum() for v in r))
    s = transpose(*r)
    p, gamma, hist = s.clone(), float(s.square().sum()), []
    for _ in range(c["iters"]):
        w = sch.ac_forward(p)
        alpha = gamma / float(sum(v.square().sum() for v in w))
        m += alpha * p
        for v, u in zip(r, w):
            v -= alpha * u
        hist.append(math.sqrt(float(sum(v.square().sum() for v in r)) / norm))
        s = transpose(*r)
        old, gamma = gamma, float(s.square().sum())
        p = s + gamma / old * p
    return m, np.array(hist)
