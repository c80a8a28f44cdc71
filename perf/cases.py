"""The work a user of this framework has it do, as cases that can be timed.

Ocean cases advance a model through the time loop (``Model.run``), a batch of
models (``Batch.run``), or a coupler's loop of asynchronous transfers and
steps over the C ABI.  Closure cases call the tensor-core network: its
forward pass, its loss gradient, and a mixed-precision run with the network's
tendency applied.  Grids, levels and time steps are those of
``pcom_b200.synth`` (128 x 64 x 20 box, 1 and 0.25 degree global) or generic
ones of other sizes.

A case is a dict of plain values:
  kind   "run" | "coupled" | "ensemble" | "closure_run" | "forward" | "gradient"
  grid   a name of pcom_b200.synth, "basin" (flat, walls) or "globe"
         (periodic, with land; any size), with ni, nj, nk
  prec   "fp64" or "mixed";  steps: baroclinic steps of one pass

``exact`` gives the network's outputs and gradients in 64 bits.  An ocean
pass is some hundred dependent stencil operators per step, 120 barotropic
substeps among them, and has no short statement outside the model: its
outputs (FP64, or FP32 of the mixed form) have no value there.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from pcom_b200 import _lib as L
from pcom_b200.closure import Network
from pcom_b200.model import Batch, Model
from pcom_b200.synth import make_case

SIZES = {"tiny_bathy": (24, 14, 12), "box": (128, 64, 20), "global1": (360, 160, 30), "global025": (1440, 640, 30)}
LAYERS = ((16, 64), (64, 64), (64, 64), (64, 64), (64, 16))  # (in, out) channels of the closure network
# what a pass of the model leaves behind: state, tendencies, accumulators
FIELDS = ("tc", "sc", "uc", "vc", "wm", "am", "alpha", "auc", "avc", "act", "acs", "acr", "acu", "acv", "acw",
          "chc", "ubc", "vbc", "mch", "acch", "acssh")


def _grid(name, **kw):
    ni, nj, nk = SIZES[name]
    return dict(grid=name, ni=ni, nj=nj, nk=nk, **kw)


def listed():
    return [
        # one call for one step on a toy grid: what a call costs when the GPU has next to nothing to do
        dict(name="run_tiny", kind="run", prec="fp64", steps=1, **_grid("tiny_bathy")),
        # the regional box, a model day per call
        dict(name="run_box", kind="run", prec="fp64", steps=24, **_grid("box")),
        # an odd-sized global grid in mixed precision: ragged tiles everywhere
        dict(name="run_odd_mixed", kind="run", prec="mixed", steps=24, grid="globe", ni=211, nj=97, nk=23),
        # the headline configuration, a model day per call, in both precisions
        dict(name="run_global1", kind="run", prec="fp64", steps=24, **_grid("global1")),
        dict(name="run_global1_mixed", kind="run", prec="mixed", steps=24, **_grid("global1")),
        # the 0.25 degree model that produces the closure's training data
        dict(name="run_global025", kind="run", prec="fp64", steps=3, **_grid("global025")),
        # a coupled 1 degree run: forcing up and barotropic state down every step
        dict(name="coupled_global1", kind="coupled", prec="fp64", steps=6, **_grid("global1")),
        # ensemble members of the box and smaller basins, stepped together
        dict(name="ensemble", kind="ensemble", prec="fp64", steps=6, members=16, basins=8, **_grid("box")),
        # a closure run: eight mixed steps, then the network's tendency
        dict(name="closure_run", kind="closure_run", prec="mixed", steps=8, **_grid("global1")),
        # the network alone on the 1 degree grid: one inference, one gradient
        dict(name="forward_global1", kind="forward", ni=360, nj=160, nk=30),
        dict(name="gradient_global1", kind="gradient", ni=360, nj=160, nk=30),
        # training on a small odd region
        dict(name="gradient_region", kind="gradient", ni=131, nj=67, nk=12),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case of the same kinds: grids from toys to half a degree, odd sizes among them."""
    kind = rng.choice(("run", "run", "run", "coupled", "ensemble", "closure_run", "forward", "gradient"))
    nj = _log(rng, 12, 320)
    ni = int(nj * rng.uniform(1.2, 2.25))
    nk = rng.randint(8, 36)
    if kind in ("forward", "gradient"):
        return dict(kind=kind, ni=min(ni, 400), nj=min(nj, 180), nk=nk)
    if kind == "ensemble":
        return dict(kind=kind, prec="fp64", steps=rng.randint(1, 6), members=rng.randint(2, 16),
                    basins=rng.randint(0, 8), grid="basin", ni=min(ni, 160), nj=min(nj, 100), nk=nk)
    grid = rng.choice(("globe", "globe", "basin")) if nj <= 150 else "globe"
    prec = "mixed" if kind == "closure_run" else rng.choice(("fp64", "fp64", "mixed"))
    if kind == "closure_run":
        grid, ni, nj = "globe", min(ni, 400), min(nj, 180)
    return dict(kind=kind, prec=prec, steps=rng.randint(1, 8 if nj > 180 else 24), grid=grid, ni=ni, nj=nj, nk=nk)


# ------------------------------------------------------------------ inputs
def _globe(ni, nj, nk):
    """A periodic 78S-80N grid of any size with smooth random land."""
    c = make_case("basin", noise=0.0, glo_ni=ni, glo_nj=nj, nk=nk)
    rng = np.random.default_rng(1000 * ni + nj)
    lon = (np.arange(ni) + 0.5) * (360.0 / ni)
    lat = -78.0 + np.arange(nj) * (158.0 / (nj - 1))
    f = np.full((nj, ni), 0.6)
    for n in range(1, 7):
        for _ in range(3):
            a, b = rng.uniform(0, 2 * np.pi, 2)
            f += np.cos(n * np.deg2rad(lon) + a)[None, :] * np.cos(rng.integers(1, 7) * np.deg2rad(lat) + b)[:, None] / n
    depth = np.where(f > 0, 5500.0 * f / f.max(), 0.0)
    itn = np.where(depth > 0, np.clip(np.rint(depth / (4000.0 / nk)), 1, nk), 0).astype(np.int32)
    dt = 60 if ni <= 400 and nj <= 180 else 30 if ni <= 720 and nj <= 320 else 20
    tx = np.broadcast_to(0.1 * np.sin(3.0 * np.deg2rad(lat))[None, :, None], (12, nj, ni)).copy()
    sst = np.broadcast_to((2.0 + 26.0 * np.cos(np.deg2rad(lat)) ** 2)[None, :, None], (12, nj, ni)).copy()
    return dict(c, name="globe", lon=lon, lat=lat, itn=itn, dtbt=dt, dtbc=60 * dt, taux=tx, bct=sst)


def _ocean(case, seed, grid=None, size=None):
    grid = grid or case["grid"]
    ni, nj, nk = size or (case["ni"], case["nj"], case["nk"])
    if grid == "globe":
        c = _globe(ni, nj, nk)
    elif grid == "basin":
        c = make_case("basin", noise=0.0, glo_ni=ni, glo_nj=nj, nk=nk)
    else:
        c = make_case(grid, noise=0.0)
    # the members of an ensemble differ so; it leaves some columns to be mixed
    rng = np.random.default_rng(seed)
    pt = c["pt"] + 0.05 * rng.standard_normal(c["pt"].shape, dtype=np.float32)
    sa = c["sa"] + 0.01 * rng.standard_normal(c["sa"].shape, dtype=np.float32)
    return dict(c, pt=pt, sa=sa)


def _model(case, seed, **kw):
    return Model(_ocean(case, seed, **kw), flags=L.PCOM_PREC_MIXED if case["prec"] == "mixed" else L.PCOM_PREC_FP64)


class _Array:
    """A model's device array; a tensor made of it keeps the model."""

    def __init__(self, model, ptr, n, elem):
        self.model = model
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f%d" % elem, "data": (ptr, False), "version": 3}


def _view(m, name):
    p, n, e = C.c_void_p(), C.c_int64(), C.c_int32()
    L.check(m.lib.pcom_gpu_field_ptr(m.handle, name.encode(), C.byref(p), C.byref(n), C.byref(e)), name)
    return torch.as_tensor(_Array(m, p.value, n.value, e.value), device="cuda")


def _fields(m, names=FIELDS):
    return {f: _view(m, f) for f in names}


def _parameters(seed):
    rng = np.random.default_rng(seed)
    out = []
    for li, (k, n) in enumerate(LAYERS):
        real_k, real_n = (5 if li == 0 else k), (4 if li == 4 else n)
        w, b = np.zeros((9, n, k), np.float32), np.zeros(n, np.float32)
        w[:, :real_n, :real_k] = rng.standard_normal((9, real_n, real_k)) * np.sqrt(2.0 / (9 * real_k))
        b[:real_n] = 0.05 * rng.standard_normal(real_n)
        out += [w.reshape(-1), b]
    return np.concatenate(out)


def _images(case, seed):
    """Normalised features, targets and the wet mask of the level images."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nk, nj, ni = case["nk"], case["nj"], case["ni"]
    normal = lambda *s: torch.randn(s, generator=g, device="cuda")
    wet = torch.nn.functional.avg_pool2d(normal(1, 1, nj + 8, ni + 8), 9, 1)[0, 0] > -0.06
    x = torch.zeros((nk, nj, ni, 16), device="cuda")
    x[..., :5] = normal(nk, nj, ni, 5) * wet[None, :, :, None]
    mask = wet[None, :, :, None].expand(nk, nj, ni, 4).float().contiguous()
    return x.bfloat16(), normal(nk, nj, ni, 4) * mask, mask


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        net = Network(case["nj"], case["ni"], case["nk"])
        net.set_params(_parameters(seed))
        x, target, mask = _images(case, seed)
        y = torch.empty((case["nk"], case["nj"], case["ni"], 4), device="cuda")
        return dict(kind=kind, net=net, x=x, y=y, target=target, mask=mask, grad=np.empty(net.nparam, np.float32))
    if kind == "ensemble":
        models = [_model(case, 100 * seed + q) for q in range(case["members"])]
        for q in range(case["basins"]):
            ni, nj, nk = (max(12, int(v * s)) for v, s in zip((case["ni"], case["nj"], case["nk"]),
                                                              (0.5 + 0.06 * q, 0.9 - 0.05 * q, 1.0 - 0.02 * q)))
            models.append(_model(case, 100 * seed + 50 + q, grid="basin", size=(ni, nj, nk)))
        batch = Batch(models)
        batch.run(3)
        batch.autotune()
        return dict(kind=kind, models=models, batch=batch, steps=case["steps"])
    m = _model(case, seed)
    s = dict(kind=kind, model=m, steps=case["steps"])
    if kind == "coupled":
        m.run(3)
        forcing = m.int_bnd()
        s["frc"] = [_pinned(m.ni * m.nj) for _ in range(6)]
        for t, k in zip(s["frc"], ("taux", "tauy", "t", "s", "pa", "fw")):
            t.copy_(torch.from_numpy(forcing[k].reshape(-1)))
        s["back"] = [_pinned(m.ni * m.nj) for _ in range(3)]
        ptr = lambda t: C.cast(t.data_ptr(), L.dbl_p)
        s["forcing"] = L.Forcing(*[ptr(t) for t in s["frc"]])
        st = s["state"] = L.State()
        st.chc, st.ubc, st.vbc = (ptr(t) for t in s["back"])
        s["it"] = m.iter
    elif kind == "closure_run":
        m.run(3)
        s["it"] = m.iter
        net = s["net"] = Network(case["nj"], case["ni"], case["nk"])
        net.set_params(_parameters(seed))
        st = s["stats"] = L.CnnStats()
        st.in_mean[:] = [0.0, 0.0, 8.0, 35.0, 0.0]
        st.in_std[:] = [0.05, 0.05, 7.0, 0.1, 1e-6]
        st.out_std[:] = [1e-8, 1e-8, 3e-8, 0.0]
        st.out_gain[:] = [0.0, 0.0, 0.5, 0.5]
        st.out_clip = 3.0
        alpha = m.field("alpha")
        for k in range(case["nk"]):
            st.alpha_ref[k] = float(alpha[k].mean())
        npix = case["ni"] * case["nj"] * case["nk"]
        s["x"] = torch.zeros((npix, 16), dtype=torch.bfloat16, device="cuda")
        s["y"] = torch.zeros((npix, 4), device="cuda")
    return s


# ------------------------------------------------------------------ a pass
def run(s):
    kind = s["kind"]
    if kind == "forward":
        s["net"].forward(s["x"], s["y"])
        return s["y"]
    if kind == "gradient":
        net, loss = s["net"], C.c_double()
        if net.lib.pcom_cnn_gradient(net.h, s["x"].data_ptr(), s["target"].data_ptr(), s["mask"].data_ptr(), net.nimg,
                                     s["grad"].ctypes.data, C.byref(loss)) != 0:
            raise L.PcomError("pcom_cnn_gradient")
        return {"loss": loss.value, "grad": s["grad"]}
    if kind == "ensemble":
        s["batch"].run(s["steps"])
        two = (s["models"][0], s["models"][-1])
        return [_fields(m) for m in two] + [_fields(m, ("tc",)) for m in s["models"][1:-1]]
    m, lib = s["model"], s["model"].lib
    if kind == "run":
        m.run(s["steps"])
    elif kind == "coupled":
        for _ in range(s["steps"]):
            s["it"] += 1
            L.check(lib.pcom_gpu_set_forcing_async(m.handle, C.byref(s["forcing"])), "set_forcing_async")
            L.check(lib.pcom_gpu_step_async(m.handle, s["it"]), "step_async")
            L.check(lib.pcom_gpu_get_state_async(m.handle, C.byref(s["state"])), "get_state_async")
        m.sync()
        return dict(_fields(m), back=s["back"])
    else:
        for _ in range(s["steps"]):
            s["it"] += 1
            m.step_handle(s["it"])
        L.check(lib.pcom_gpu_cnn_features(m.handle, C.c_void_p(s["x"].data_ptr()), C.byref(s["stats"])), "features")
        m.sync()
        s["net"].forward(s["x"], s["y"])
        L.check(lib.pcom_gpu_cnn_apply(m.handle, C.c_void_p(s["y"].data_ptr()), C.byref(s["stats"]),
                                       float(s["steps"] * 3600)), "apply")
        m.sync()
        return dict(_fields(m), x=s["x"], y=s["y"])
    return _fields(m)


# ------------------------------------------------------- what a pass needs
def _step_work(ni, nj, nk, prec):
    n2, n3, e = ni * nj, ni * nj * nk, 4 if prec == "mixed" else 8
    # 3-D fields read once (T, S, u, v, four AB3 tendencies, am, km, kh, the
    # density derivatives, six accumulators) and written once (T, S, u, v,
    # two tendencies, am, alpha, w, the accumulators); the 2-D state,
    # coefficients and forcing once (120 substeps keep them on the chip)
    return 34 * e * n3 + 45 * 8 * n2, 1100 * n3 + 120 * 260 * n2


def _net_flops(npix, backward):
    fwd = 2 * 9 * (5 * 64 + 3 * 64 * 64 + 64 * 4) * npix
    return fwd if not backward else 3 * fwd - 2 * 9 * 5 * 64 * npix


def work(case):
    kind, ni, nj, nk = case["kind"], case["ni"], case["nj"], case["nk"]
    npix, par = ni * nj * nk, 4 * 121000
    if kind == "forward":
        return {"bytes": npix * (32 + 16) + par, "flops": _net_flops(npix, False)}
    if kind == "gradient":
        return {"bytes": npix * (32 + 16 + 16) + 2 * par, "flops": _net_flops(npix, True)}
    b, f = _step_work(ni, nj, nk, case["prec"])
    b, f = b * case["steps"], f * case["steps"]
    if kind == "ensemble":
        part = sum((0.5 + 0.06 * q) * (0.9 - 0.05 * q) for q in range(case["basins"]))
        b, f = b * (case["members"] + part), f * (case["members"] + part)
    if kind == "coupled":
        b += case["steps"] * 8 * 8 * ni * nj
    if kind == "closure_run":
        b, f = b + npix * 64, f + _net_flops(npix, False)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------ in 64 bits
def _conv64(x, w, b):
    """3x3 convolution of [n][H][W][C] images, zero rows beyond the edges, periodic in x."""
    n, h, wd, _ = x.shape
    x = torch.cat([x[:, :, -1:], x, x[:, :, :1]], 2)
    zero = torch.zeros_like(x[:, :1])
    x = torch.cat([zero, x, zero], 1)
    return b + sum(x[:, t // 3:t // 3 + h, t % 3:t % 3 + wd] @ w[t].T for t in range(9))


def exact(case, seed):
    if case["kind"] not in ("forward", "gradient"):
        return None
    x, target, mask = _images(case, seed)
    p = torch.from_numpy(_parameters(seed)).cuda().double()
    p.requires_grad_(case["kind"] == "gradient")
    total, loss, ys = mask.double().sum(), 0.0, []
    for q in range(case["nk"]):
        a, o = x[q:q + 1].double(), 0
        for li, (k, n) in enumerate(LAYERS):
            a = _conv64(a, p[o:o + 9 * n * k].view(9, n, k), p[o + 9 * n * k:o + 9 * n * k + n])
            o += 9 * n * k + n
            a = a if li == 4 else torch.relu(a)
        if case["kind"] == "forward":
            ys.append(a[..., :4])
            continue
        part = (mask[q].double() * (a[0, ..., :4] - target[q].double()) ** 2).sum() / total
        part.backward()
        loss += float(part)
    return torch.cat(ys) if ys else {"loss": loss, "grad": p.grad}
