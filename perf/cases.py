"""The calls whose speed matters to a user of the package, with their inputs.

``listed()`` gives the fixed cases and ``draw(rng)`` one more of the same
ranges.  ``prepare`` makes what a program holds before the call (plan,
weights, inputs on the GPU, from the seed alone), ``run`` is one pass through
the public entry points, ``work`` the bytes and operations the pass cannot do
without, and ``exact`` the result in 64 bits from plain torch.

Kinds of cases:

* ``pair3d``: direct and transpose projection of all views of a 3D scan
  (``Projector3D.forward`` / ``backward``), cone or parallel beam, closed-form
  cubic or tabulated footprint, a full circular orbit or irregular angles;
* ``view3d``: the same for one view, the closure an iterative program calls
  view by view (``Projector3D.single_view``);
* ``gates4d``: the data term of a gated scan and its gradient in one call
  (``Projector3D.wls_grad``);
* ``pair2d``: direct and transpose projection of a 2D scan (``Projector2D``),
  parallel, fan or Long-Fessler model;
* ``objective``: cost and gradient of the TV-regularised reconstruction
  (``recon.Objective``), 2D or 3D: what an iteration evaluates;
* ``conv``: one 3x3x3 convolution layer of the warm-start network through the
  C interface (``include/trtt_b200.h``), at a layer's channels: inference
  (``trtt_b200_conv3_forward``), or forward, input gradient and weight and bias
  gradients (``trtt_b200_conv3_wgrad``) as a training step calls them.  The
  whole network is no case: one BF16 rounding more or less in a layer travels
  through those behind it, to 1e-3 of the output.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

RSC, RSD = 1000.0, 1500.0  # source to isocentre, source to detector (mm)
SLOPE = 0.1                # leaky ReLU of the network

# the network's layers: channels of the first and the skip input, output channels
LAYERS = {"e1a": (16, 0, 16), "e1b": (16, 0, 16), "e2a": (16, 0, 32), "e2b": (32, 0, 32), "e3a": (32, 0, 64),
          "e3b": (64, 0, 64), "d2a": (64, 32, 32), "d1a": (32, 16, 16)}


def listed():
    return [
        # cone-beam scan of the bench workload: every iteration of a
        # reconstruction applies the pair to all views
        dict(name="cone_scan_256", kind="pair3d", mode="cone", nx=256, ny=256, nz=256, nu=512, nv=512,
             views=360, orbit="full", table=0, object="phantom", layout="columns", s_scl=1.0, d_scl=1.0),
        # cost and gradient on a dense iterate at the size the warm start is
        # trained and evaluated on (weighted data, TV)
        dict(name="cone_objective_128", kind="objective", mode="cone", nx=128, ny=128, nz=128, nu=256, nv=256,
             views=90, mu=5.0, eps=1e-2, weights=True, s_scl=1.0, d_scl=1.0),
        # irregular acquisition (gated or sparse angles) of a non-square
        # volume on an odd detector
        dict(name="cone_irregular", kind="pair3d", mode="cone", nx=100, ny=92, nz=75, nu=151, nv=133,
             views=61, orbit="irregular", table=0, object="phantom", layout="xyz", s_scl=1.1, d_scl=1.3),
        # tabulated footprint, the reference's default model
        dict(name="cone_table_128", kind="pair3d", mode="cone", nx=128, ny=128, nz=128, nu=256, nv=256,
             views=90, orbit="full", table=10001, object="phantom", layout="xyz", s_scl=1.0, d_scl=1.0),
        # parallel beam in 3D, half turn, odd sizes, dense object
        dict(name="parallel_scan_odd", kind="pair3d", mode="parallel", nx=97, ny=97, nz=83, nu=129, nv=141,
             views=75, orbit="half", table=0, object="iterate", layout="xyz", s_scl=1.0, d_scl=1.0),
        # one view at a time: the per-view closure of the operator layer
        dict(name="cone_one_view", kind="view3d", mode="cone", nx=128, ny=128, nz=128, nu=256, nv=256,
             views=90, view=17, table=0, object="phantom", s_scl=1.0, d_scl=1.0),
        # gated scan: 10 gates, 20 to 60 views each, all in one call
        dict(name="gates4d", kind="gates4d", nx=128, ny=128, nz=64, nu=256, nv=256, gates=10, vmin=20,
             vmax=60, weights=False, s_scl=1.0, d_scl=1.0),
        # 2D fan beam, 512^2 image, 720 views, 1024 cells
        dict(name="fan2d_512", kind="pair2d", mode="fan", nx=512, ny=512, nv=1024, views=720, table=0,
             object="phantom", s_scl=0.5, d_scl=0.5),
        # 2D parallel-beam reconstruction: cost and gradient of one iteration
        dict(name="parallel2d_objective", kind="objective", mode="parallel", nx=256, ny=256, nz=0, nu=0, nv=367,
             views=180, mu=1e-2, eps=1e-3, weights=False, s_scl=1.0, d_scl=1.0),
        # Long-Fessler separable footprints on the fan-beam scan
        dict(name="long_fessler_512", kind="pair2d", mode="lf", nx=512, ny=512, nv=1024, views=720, table=0,
             object="phantom", s_scl=0.5, d_scl=0.5),
        # warm-start network: the largest layer of an inference at 128^3 (the
        # decoder's concatenated input at full resolution), and a layer of a
        # training step at batch 2, half resolution
        dict(name="conv_infer_128", kind="conv", layer="d1a", train=False, batch=1, d=128, h=128, w=128),
        dict(name="conv_train_64", kind="conv", layer="e2b", train=True, batch=2, d=64, h=64, w=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair3d", "pair3d", "pair3d", "view3d", "gates4d", "pair2d", "pair2d", "objective",
                       "objective", "conv", "conv"])
    if kind in ("pair3d", "view3d", "gates4d") or (kind == "objective" and rng.random() < 0.5):
        n = _log_int(rng, 24, 176)
        square = rng.random() < 0.5
        nx = n + (n & 1) if square else n
        ny = nx if square else max(8, int(n * rng.uniform(0.7, 1.3)))
        nz = max(8, int(n * rng.uniform(0.4, 1.2)))
        nd = rng.uniform(1.4, 2.0)
        s_scl, d_scl = rng.uniform(0.5, 1.5), 1.0
        d_scl = s_scl * rng.choice([1.0, 1.0, rng.uniform(0.8, 1.5)])
        nu, nv = int(nz * nd * s_scl / d_scl) + 8, int(max(nx, ny) * nd * s_scl / d_scl) + 8
        if rng.random() < 0.5:
            nu, nv = (nu + 3) // 4 * 4, (nv + 3) // 4 * 4
        base = dict(nx=nx, ny=ny, nz=nz, nu=nu, nv=nv, s_scl=round(s_scl, 4), d_scl=round(d_scl, 4))
        mode = rng.choice(["cone", "cone", "parallel"])
        if kind == "gates4d":
            nt = rng.randint(2, 12)
            vmin = rng.randint(5, 20)
            cap = max(vmin + 1, int(1.2e9 / (nx * ny * nz * nt)))
            return dict(kind=kind, gates=nt, vmin=vmin, vmax=min(vmin + rng.randint(1, 40), cap),
                        weights=rng.random() < 0.5, **base)
        table = rng.choice([0, 0, 10001]) if kind != "objective" else 0
        cap = max(4, int((6e8 if table else 2.4e9) / (nx * ny * nz)))
        views = min(_log_int(rng, 12, 360), cap)
        if kind == "view3d":
            return dict(kind=kind, mode=mode, views=views, view=rng.randrange(views), table=table,
                        object=rng.choice(["phantom", "iterate"]), **base)
        if kind == "objective":
            return dict(kind=kind, mode=mode, views=views, mu=rng.choice([0.0, 1e-2, 5.0]), eps=1e-2,
                        weights=rng.random() < 0.5, **base)
        orbit = rng.choice(["full", "full", "half", "irregular"])
        if orbit == "full" and rng.random() < 0.6:
            views = max(4, views // 4 * 4)
        return dict(kind=kind, mode=mode, views=views, orbit=orbit, table=table,
                    object=rng.choice(["phantom", "iterate"]), layout=rng.choice(["xyz", "columns"]), **base)
    if kind in ("pair2d", "objective"):
        n = _log_int(rng, 48, 512)
        ny = n if rng.random() < 0.5 else max(16, int(n * rng.uniform(0.7, 1.3)))
        s_scl = round(rng.uniform(0.4, 1.2), 4)
        d_scl = round(s_scl * rng.choice([1.0, rng.uniform(0.7, 1.5)]), 4)
        nv = int(max(n, ny) * rng.uniform(1.3, 2.2) * s_scl / d_scl) + 4
        views = _log_int(rng, 24, 720)
        base = dict(nx=n, ny=ny, nv=nv, views=views, s_scl=s_scl, d_scl=d_scl)
        if kind == "objective":
            return dict(kind=kind, mode=rng.choice(["parallel", "fan"]), nz=0, nu=0, mu=1e-2, eps=1e-3,
                        weights=rng.random() < 0.5, **base)
        mode = rng.choice(["parallel", "fan", "fan", "lf"])
        return dict(kind=kind, mode=mode, table=0 if mode == "lf" else rng.choice([0, 10001]),
                    object=rng.choice(["phantom", "iterate"]), **base)
    d, h, w = (4 * rng.randint(5, 30) for _ in range(3))
    return dict(kind="conv", layer=rng.choice(sorted(LAYERS)), train=rng.random() < 0.5,
                batch=rng.randint(1, 2), d=d, h=h, w=w)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(case, seed, salt=0):
    return np.random.default_rng([int(seed), salt])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 7)


def _ellipsoids(nx, ny, nz, seed, shift=0.0):
    """Sum of 20 (10 in 2D: nz = 0) random ellipsoids, the first a large
    centred body, on the (nz, ny, nx) or (ny, nx) grid; float32 on the GPU."""
    rng = _rng(None, seed)
    flat = nz == 0
    def ax(n):
        return (torch.arange(n, device="cuda", dtype=torch.float32) - 0.5 * (n - 1)) / (0.5 * n)
    x, y = ax(nx)[None, None, :], ax(ny)[None, :, None]
    z = (ax(nz) if not flat else torch.zeros(1, device="cuda"))[:, None, None]
    vol = torch.zeros(max(nz, 1), ny, nx, device="cuda")
    for e in range(10 if flat else 20):
        r, phi = 0.55 * math.sqrt(rng.uniform()), rng.uniform(0, 2 * math.pi)
        c = [r * math.cos(phi), r * math.sin(phi), 0.0 if flat else rng.uniform(-0.5, 0.5)]
        a = rng.uniform(0.06, 0.3, size=3)
        if e == 0:
            c, a = [0.0, 0.0, 0.0], np.append(rng.uniform(0.85, 0.95, size=2), rng.uniform(1.1, 1.3))
        ang, val = rng.uniform(0, math.pi), rng.uniform()
        ca, sa = math.cos(ang), math.sin(ang)
        xr, yr = (x - c[0]) * ca + (y - c[1]) * sa, -(x - c[0]) * sa + (y - c[1]) * ca
        vol += val * ((xr / a[0]) ** 2 + (yr / a[1]) ** 2 + ((z - c[2] - shift) / a[2]) ** 2 <= 1.0)
    return vol[0] if flat else vol


def _object(case, seed, nz=None):
    """The phantom itself, or a dense positive iterate near it."""
    vol = _ellipsoids(case["nx"], case["ny"], case["nz"] if nz is None else nz, seed)
    if case.get("object", "iterate") == "iterate":
        vol = vol + 0.05 + 0.1 * torch.rand(vol.shape, device="cuda", generator=_gen(seed))
    return vol


def _residual(shape, seed):
    """Detector residuals: noise."""
    return torch.randn(shape, device="cuda", generator=_gen(seed + 1))


def _dome(shape, top, seed):
    """Detector data of the magnitude of the object's line integrals, 1% noise."""
    axes = [torch.linspace(-1, 1, n, device="cuda") for n in shape[1:]]
    r2 = axes[0] ** 2 if len(axes) == 1 else axes[0][:, None] ** 2 + axes[1][None, :] ** 2
    dome = top * (1.0 - r2).clamp(min=0.0)
    return (dome[None] + 0.01 * top * torch.randn(shape, device="cuda", generator=_gen(seed + 2))).contiguous()


def _theta(case, seed):
    n, orbit = case["views"], case.get("orbit", "full")
    if case["kind"] in ("pair2d", "objective") and case["mode"] == "parallel":
        orbit = "half"
    if orbit == "irregular":
        return np.sort(_rng(case, seed, 3).uniform(0.0, 2.0 * math.pi, n))
    return np.arange(n) * ((math.pi if orbit == "half" else 2.0 * math.pi) / n)


def _gates(case, seed):
    """(t_index, theta) of a gated scan: views per gate drawn uniformly,
    fractional gate index inside the gate, angles over the orbit."""
    rng = _rng(case, seed, 4)
    counts = rng.integers(case["vmin"], case["vmax"] + 1, case["gates"])
    t = np.concatenate([g + rng.uniform(0.0, 1.0, c) for g, c in enumerate(counts)])
    return t, np.sort(rng.uniform(0.0, 2.0 * math.pi, len(t)))


def _inputs(case, seed):
    """Everything random of a case, as GPU tensors and host arrays."""
    k = case["kind"]
    if k == "conv":
        c1, c2, co = LAYERS[case["layer"]]
        g = _gen(seed)

        def act(c, scale):
            """Padded channels-last BF16 activations (zero border)."""
            a = torch.zeros(case["batch"], case["d"] + 2, case["h"] + 2, case["w"] + 2, c, device="cuda")
            v = a[:, 1:-1, 1:-1, 1:-1]
            v.copy_(torch.nn.functional.leaky_relu(torch.randn(v.shape, device="cuda", generator=g), SLOPE) * scale)
            return a.bfloat16()

        w = torch.randn(co, 27, c1 + c2, device="cuda", generator=g) * math.sqrt(2.0 / (27 * (c1 + c2)))
        return {"x1": act(c1, 0.5), "x2": act(c2, 0.5) if c2 else None, "gy": act(co, 1e-3),
                "w": w.bfloat16().float(), "b": 0.02 * torch.randn(co, device="cuda", generator=g)}
    if k == "gates4d":
        t, theta = _gates(case, seed)
        vol = torch.stack([_ellipsoids(case["nx"], case["ny"], case["nz"], seed,
                                       0.15 * (1 - math.cos(2 * math.pi * g / case["gates"])))
                           for g in range(case["gates"])]) + 0.02
        shape = (len(t), case["nv"], case["nu"])
        d = {"vol": vol, "t": t, "theta": theta, "y": _dome(shape, 0.6 * case["nx"] * case["s_scl"], seed)}
        d["w"] = torch.exp(-0.02 * d["y"].clamp(min=0)) if case["weights"] else None
        return d
    two_d = k == "pair2d" or (k == "objective" and case["nz"] == 0)
    d = {"theta": _theta(case, seed), "vol": _object(case, seed, 0 if two_d else None)}
    shape = (case["views"], case["nv"]) if two_d else (case["views"], case["nv"], case["nu"])
    if k == "objective":
        d["y"] = _dome(shape, 0.6 * case["nx"] * case["s_scl"], seed)
        d["w"] = torch.exp(-0.02 * d["y"].clamp(min=0)) if case["weights"] else None
    else:
        d["y"] = _residual((1,) + shape[1:] if k == "view3d" else shape, seed)
    return d


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def _lf_params(case):
    from yoricktrtt_b200.dropin import LF2DParams
    return LF2DParams(pixelSize=case["d_scl"], pixelStep=case["d_scl"], voxelSize=case["s_scl"],
                      sourceDistance=RSC, detectorDistance=RSD - RSC, objectOffset1=0.0, objectOffset2=0.0,
                      objectDimension1=case["nx"], objectDimension2=case["ny"], detectorDimension=case["nv"])


def _projector(case, theta):
    from yoricktrtt_b200 import footprint, geometry as G
    from yoricktrtt_b200.projectors import Projector3D
    from yoricktrtt_b200.recon import Projector2D
    s, d = case["s_scl"], case["d_scl"]
    table = footprint.make_footprint(3, case["table"]) if case.get("table") else None
    if case["kind"] == "pair2d" or case.get("nz") == 0:
        if case["mode"] == "lf":
            return Projector2D(lf_params=_lf_params(case), beta=theta - math.pi / 2, offset=np.zeros(len(theta)))
        mode = G.TRTT_PARALLEL_BEAM if case["mode"] == "parallel" else G.TRTT_FAN_BEAM
        return Projector2D(G.circular_scan_2d(case["nx"], case["ny"], s, 3, case["nv"], d, len(theta), mode=mode,
                                              rsc=RSC, rsd=RSD, theta=theta), table)
    mode = G.TRTT_PARALLEL_BEAM if case.get("mode") == "parallel" else G.TRTT_CONE_BEAM
    return Projector3D(G.circular_scan_3d(case["nx"], case["ny"], case["nz"], s, 3, case["nu"], case["nv"], d, d,
                                          len(theta), mode=mode, rsc=RSC, rsd=RSD, theta=theta), table)


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _prepare_conv(case, s):
    """Packed weights, output and gradient buffers and scratch, as the network keeps them."""
    from yoricktrtt_b200 import _lib
    lib = _lib.load()
    c1, c2, co = LAYERS[case["layer"]]
    s["case"], s["grid"] = case, (case["batch"], case["d"], case["h"], case["w"])
    for key, tr in (("fw", 0), ("bw", 1)):
        s[key] = torch.empty(27 * co * (c1 + c2), dtype=torch.bfloat16, device="cuda")
        _lib.check(lib.trtt_b200_conv3_pack(_ptr(s["w"]), co, c1 + c2, tr, _ptr(s[key]), _stream()), "conv3_pack")
    s["y"] = torch.zeros_like(s["gy"])
    if case["train"]:
        s["dx1"], s["dx2"] = torch.zeros_like(s["x1"]), torch.zeros_like(s["x2"]) if c2 else None
        s["dw"], s["db"] = torch.zeros_like(s["w"]), torch.zeros_like(s["b"])
        s["nscratch"] = lib.trtt_b200_conv3_wgrad_scratch(co, c1 + c2, *s["grid"])
        s["scratch"] = torch.empty(s["nscratch"] // 4 + 1, device="cuda")
    return s


def _run_conv(s):
    from yoricktrtt_b200 import _lib
    lib = _lib.load()
    c1, c2, co = LAYERS[s["case"]["layer"]]
    _lib.check(lib.trtt_b200_conv3_forward(
        _ptr(s["x1"]), c1, _ptr(s["x2"]), c2, _ptr(s["fw"]), co, _ptr(s["b"]), 0, SLOPE, _ptr(s["y"]), None, 0, 0,
        None, *s["grid"], _stream()), "conv3_forward")
    if not s["case"]["train"]:
        return s["y"]
    _lib.check(lib.trtt_b200_conv3_forward(
        _ptr(s["gy"]), co, None, 0, _ptr(s["bw"]), c1 + c2, None, 3, 1.0, _ptr(s["dx1"]), _ptr(s["dx2"]), c1, 0,
        None, *s["grid"], _stream()), "conv3 input gradient")
    _lib.check(lib.trtt_b200_conv3_wgrad(
        _ptr(s["gy"]), co, _ptr(s["x1"]), c1, _ptr(s["x2"]), c2, _ptr(s["dw"]), _ptr(s["db"]), _ptr(s["scratch"]),
        s["nscratch"], *s["grid"], _stream()), "conv3_wgrad")
    return {k: s[k] for k in ("y", "dx1", "dx2", "dw", "db") if s[k] is not None}


def prepare(case, seed):
    inp = _inputs(case, seed)
    s = {"case": case}
    if case["kind"] == "conv":
        return _prepare_conv(case, inp)
    pr = s["pr"] = _projector(case, inp["theta"])
    s["y"] = inp["y"]
    if case["kind"] == "gates4d":
        pr.set_gates(case["gates"], inp["t"])
        s["vol"], s["w"] = inp["vol"].movedim(-3, -1).contiguous(), inp["w"]
    elif case["kind"] == "objective":
        from yoricktrtt_b200.recon import Objective
        s["vol"] = inp["vol"]
        s["obj"] = Objective(pr, inp["y"], inp["w"], mu=case["mu"], eps=case["eps"])
    else:
        s["vol"] = inp["vol"]
        if case.get("layout") == "columns":
            s["vol"] = inp["vol"].movedim(-3, -1).contiguous()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "conv":
        return _run_conv(state)
    pr, vol, y = state["pr"], state["vol"], state["y"]
    if kind == "pair3d":
        return {"sino": pr.forward(vol, layout=case["layout"]), "back": pr.backward(y, layout=case["layout"])}
    if kind == "view3d":
        op = pr.single_view(case["view"])
        return {"sino": op(vol, 0), "back": op(y, 1)}
    if kind == "gates4d":
        grad = torch.zeros_like(vol)
        cost = pr.wls_grad(vol, y, grad, state["w"])
        return {"cost": cost, "grad": grad}
    if kind == "pair2d":
        return {"sino": pr.forward(vol), "back": pr.backward(y)}
    f, g = state["obj"](vol)
    return {"f": f, "g": g}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    if case["kind"] == "conv":
        c1, c2, co = LAYERS[case["layer"]]
        vox = case["batch"] * case["d"] * case["h"] * case["w"]
        ci, wts = c1 + c2, 27 * (c1 + c2) * co
        flops = 2 * vox * wts
        if not case["train"]:
            return {"bytes": 2 * (vox * (ci + co) + wts), "flops": flops}
        # x, gy in, y, dx out; weights in, their gradients out
        return {"bytes": 2 * vox * (2 * ci + 2 * co) + 8 * wts, "flops": 3 * flops}
    # footprints of a cubic B-spline: 4 voxels wide, about 4 s magn / d + 1
    # cells; per voxel and view one cell edge costs about 10 operations and a
    # cell 2 more, per column, view and detector cell of its profile 2 per row
    two_d = case["kind"] == "pair2d" or case.get("nz") == 0
    mag = 1.0 if case.get("mode") == "parallel" else RSD / RSC
    cells = 4.0 * case["s_scl"] * mag / case["d_scl"] + 1.0
    views = 1 if case["kind"] == "view3d" else case.get("views")
    if case["kind"] == "gates4d":
        views = case["gates"] * (case["vmin"] + case["vmax"]) // 2
    if two_d:
        if case["mode"] == "lf":
            cells = 2.0 * case["s_scl"] * mag / case["d_scl"] + 1.0
        vox, det = case["nx"] * case["ny"], views * case["nv"]
        flops = 2 * vox * views * (20 + 12 * cells)
    else:
        cols = case["nx"] * case["ny"]
        vox, det = cols * case["nz"] * case.get("gates", 1), views * case["nu"] * case["nv"]
        span = min(case["nu"], case["nz"] * case["s_scl"] * mag / case["d_scl"] + cells)
        flops = 2 * cols * views * (case["nz"] * (12 + 12 * cells) + 2 * span * cells)
    if case["kind"] in ("objective", "gates4d"):  # iterate, data (and weights) in, gradient out
        nbytes = 4 * (2 * vox + det * (2 if case["weights"] else 1))
        flops += 4 * det + (60 * vox if case.get("mu") else 0)
    else:
        nbytes = 2 * 4 * (vox + det)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _prim(x):
    """Integral of the centred cubic B-spline up to x."""
    t = x.abs()
    a, b = (2.0 - t).clamp(min=0.0), (1.0 - t).clamp(min=0.0)
    g = (a ** 4 - 4.0 * b ** 4) / 24.0
    return torch.where(x <= 0, g, 1.0 - g)


def _table(m):
    """Cumulative table of the cubic B-spline: (cum, first abscissa, step)."""
    n = 9
    step = (n - 1) / (m - 1)
    x = np.arange(m) * step - 0.5 * (n - 1)
    t = np.abs(x)
    b = np.where(t < 1, 2.0 / 3.0 - t * t + 0.5 * t ** 3, np.where(t < 2, (2.0 - t) ** 3 / 6.0, 0.0))
    cum = np.concatenate([[0.0], np.cumsum(0.5 * step * (b[:-1] + b[1:]))])
    return torch.tensor(cum, device="cuda"), -0.5 * (n - 1), step


def _axis(c, h, n, right, L, table):
    """Cells and weights of footprints centred at c with scale h on n cells:
    (index, weight), each c.shape + (L,), weights 0 past the footprint."""
    hs = 2.0 * h
    lo = torch.floor(c - hs).clamp(0, n - 1)
    hi = (torch.floor(c + hs) + 1).clamp(0, right + 1)
    l = torch.arange(L + 1, device="cuda", dtype=torch.float64)
    if table is None:
        e = _prim(((lo - c) / h)[..., None] + l * (1.0 / h)[..., None])
    else:
        cum, x0, step = table
        inc = (1.0 / h) / step
        pos = (((lo - c) - h * x0) * inc)[..., None] + l * inc[..., None]
        e = cum[pos.clamp(0, len(cum) - 1).floor().long()]
    w = (e[..., 1:] - e[..., :-1]) * (l[:-1] < (hi - lo)[..., None])
    idx = (lo[..., None] + l[:-1]).clamp(max=n - 1).long()
    return idx, w


class _Exact3D:
    """One view's column footprints in 64 bits (circular orbit about z)."""

    def __init__(self, case):
        self.c = case
        self.par = case.get("mode") == "parallel"
        self.table = _table(case["table"]) if case.get("table") else None
        s = case["s_scl"]
        f = dict(device="cuda", dtype=torch.float64)
        self.X = ((torch.arange(case["nx"], **f) - 0.5 * (case["nx"] - 1)) * s)[None, :]
        self.Y = ((torch.arange(case["ny"], **f) - 0.5 * (case["ny"] - 1)) * s)[:, None]
        self.Z = (torch.arange(case["nz"], **f) - 0.5 * (case["nz"] - 1)) * s

    def chunks(self, theta):
        """Per run of columns: (columns, dense v weights, u cells, u weights x rho)."""
        c, s, d = self.c, self.c["s_scl"], self.c["d_scl"]
        phi = math.pi - theta
        xr = (math.cos(phi) * self.X - math.sin(phi) * self.Y).reshape(-1)
        yr = (math.sin(phi) * self.X + math.cos(phi) * self.Y).reshape(-1)
        h0 = s / d
        # the smallest distance of a voxel to the source bounds the magnification
        far = 0.5 * math.hypot(c["nx"], c["ny"]) * s
        mmax = 1.0 if self.par else RSD / (RSC - far)
        L = int(math.ceil(4.0 * h0 * mmax * 1.2)) + 2
        step = max(1, int(1.5e7 / (c["nz"] * L)))
        for a in range(0, xr.numel(), step):
            x, y = xr[a:a + step], yr[a:a + step]
            if self.par:
                vc, hv = y / d + 0.5 * c["nv"], torch.full_like(y, h0)
                uc = (self.Z / d + 0.5 * c["nu"])[None, :].expand(len(y), -1)
                hu, rho = torch.full_like(uc, h0), torch.full_like(uc, s ** 3)
            else:
                m = RSD / (x + RSC)
                vc = m * y / d + 0.5 * c["nv"]
                va = (vc - 0.5 * c["nv"]) * d
                dv = torch.sqrt(1.0 + va * va / RSD ** 2)
                hv = h0 * m * dv
                uc = m[:, None] * self.Z[None, :] / d + 0.5 * c["nu"]
                ua = (uc - 0.5 * c["nu"]) * d
                du = torch.sqrt(1.0 + ua * ua / (RSD ** 2 + va * va)[:, None])
                hu = h0 * m[:, None] * du
                rho = s ** 3 * (m * m * dv)[:, None] * du
            vi, vw = _axis(vc, hv, c["nv"], c["nv"] - 1, L, self.table)
            wv = torch.zeros(len(y), c["nv"], device="cuda", dtype=torch.float64).scatter_add_(1, vi, vw)
            ui, uw = _axis(uc, hu, c["nu"], c["nu"] - 1, L, self.table)
            yield slice(a, a + len(y)), wv, ui, uw * rho[..., None]

    def pair(self, theta, vol=None, y=None, out=None):
        """(projection of vol (columns, nz), out += transpose of y)."""
        c = self.c
        sino = None if vol is None else torch.zeros(c["nv"], c["nu"], device="cuda", dtype=torch.float64)
        for sl, wv, ui, uw in self.chunks(theta):
            n = wv.shape[0]
            if vol is not None:
                p = torch.zeros(n, c["nu"], device="cuda", dtype=torch.float64)
                p.scatter_add_(1, ui.reshape(n, -1), (uw * vol[sl][..., None]).reshape(n, -1))
                sino += wv.T @ p
            if y is not None:
                q = wv @ y
                out[sl] += (uw * torch.gather(q, 1, ui.reshape(n, -1)).view(uw.shape)).sum(-1)
        return sino


class _Exact2D:
    """One view's pixel footprints in 64 bits (parallel, fan, Long-Fessler)."""

    def __init__(self, case):
        self.c = case
        self.table = _table(case["table"]) if case.get("table") else None
        f = dict(device="cuda", dtype=torch.float64)
        s = case["s_scl"]
        self.X = ((torch.arange(case["nx"], **f) - 0.5 * (case["nx"] - 1)) * s)[None, :]
        self.Y = ((torch.arange(case["ny"], **f) - 0.5 * (case["ny"] - 1)) * s)[:, None]

    def cells(self, theta):
        c, s, d, nv = self.c, self.c["s_scl"], self.c["d_scl"], self.c["nv"]
        far = 0.5 * math.hypot(c["nx"], c["ny"]) * s
        mmax = 1.0 if c["mode"] == "parallel" else RSD / (RSC - far)
        L = int(math.ceil((4.0 if c["mode"] != "lf" else 2.0) * mmax * 1.2 * s / d)) + 3
        if c["mode"] == "lf":
            return self._lf(theta - math.pi / 2, L)
        phi = math.pi - theta
        yr = math.sin(phi) * self.X + math.cos(phi) * self.Y
        h0 = s / d
        if c["mode"] == "parallel":
            vc, h, rho = yr / d + 0.5 * nv, torch.full_like(yr, h0), torch.full_like(yr, s * s)
        else:
            m = RSD / (math.cos(phi) * self.X - math.sin(phi) * self.Y + RSC)
            vc = m * yr / d + 0.5 * nv
            dv = torch.sqrt(1.0 + ((vc - 0.5 * nv) * d) ** 2 / RSD ** 2)
            h, rho = h0 * m * dv, s * s * m * dv
        # the closed-form 2D model never reaches the last cell
        idx, w = _axis(vc, h, nv, nv - 1 if self.table else nv - 2, L, self.table)
        return idx, w * rho[..., None]

    def _lf(self, beta, L):
        c, s, d, nv = self.c, self.c["s_scl"], self.c["d_scl"], self.c["nv"]
        cb, sb = math.cos(beta), math.sin(beta)
        t = []
        for a in (-0.5, 0.5):
            for b in (-0.5, 0.5):
                x, y = self.X + a * s, self.Y + b * s
                t.append(RSD / d * (y * sb + x * cb) / (RSC - (y * cb - x * sb)) + 0.5 * (nv - 1))
        t = torch.stack(t, -1).sort(-1).values
        qx, qy = (self.X + RSC * sb).expand(t.shape[:-1]), (self.Y - RSC * cb).expand(t.shape[:-1])
        q = torch.where(qy.abs() > qx.abs(), qx / qy, qy / qx)
        amp = torch.sqrt(1.0 + q * q) * s * d

        def cum(p):
            t0, t1, t2, t3 = (t[..., i:i + 1] for i in range(4))
            up = torch.where(t1 > t0, (torch.minimum(p, t1) - t0).clamp(min=0) ** 2 / (2 * (t1 - t0)), 0.0)
            flat = (torch.minimum(p, t2) - t1).clamp(min=0)
            dn = torch.where(t3 > t2, ((t3 - t2) - (t3 - torch.minimum(p, t3)).clamp(min=0) ** 2 / (t3 - t2)) / 2, 0.0)
            return up + flat + torch.where(p > t2, dn, torch.zeros_like(dn))

        lo = torch.floor(t[..., :1] - 0.5)
        k = lo + torch.arange(L, device="cuda", dtype=torch.float64)
        w = (cum(k + 0.5) - cum(k - 0.5)) * amp[..., None]
        w = w * ((k >= 0) & (k <= nv - 1))
        return k.clamp(0, nv - 1).long(), w

    def pair(self, theta, vol=None, y=None, out=None):
        nv = self.c["nv"]
        idx, w = self.cells(theta)
        n = idx.shape[0]
        sino = None
        if vol is not None:
            p = torch.zeros(n, nv, device="cuda", dtype=torch.float64)
            sino = p.scatter_add_(1, idx.reshape(n, -1), (w * vol[..., None]).reshape(n, -1)).sum(0)
        if y is not None:
            out += (w * y[idx]).sum(-1)
        return sino


def _tv(x, mu, eps):
    """mu times the smoothed TV of the spline samples of x, and its gradient."""
    x = x.detach().requires_grad_(True)
    z = x
    for ax in range(x.dim()):
        n = x.shape[ax]
        if n > 1:
            zero = torch.zeros_like(z.narrow(ax, 0, 1))
            z = (2.0 / 3.0) * z + (torch.cat([zero, z.narrow(ax, 0, n - 1)], ax)
                                   + torch.cat([z.narrow(ax, 1, n - 1), zero], ax)) / 6.0
    s2 = torch.full_like(z, eps * eps)
    for ax in range(x.dim()):
        if x.shape[ax] > 1:
            diff = z.diff(dim=ax)
            s2 = s2 + torch.cat([diff, torch.zeros_like(z.narrow(ax, 0, 1))], ax) ** 2
    f = mu * (torch.sqrt(s2) - eps).sum()
    return float(f), torch.autograd.grad(f, x)[0]


def _exact_conv(case, inp):
    import torch.nn.functional as F

    def dense(a):  # padded channels-last -> (batch, c, d, h, w)
        return a[:, 1:-1, 1:-1, 1:-1].permute(0, 4, 1, 2, 3).double().contiguous()

    def padded(a):
        return F.pad(a.permute(0, 2, 3, 4, 1), (0, 0, 1, 1, 1, 1, 1, 1)).contiguous()

    c1, c2, co = LAYERS[case["layer"]]
    x = torch.cat([dense(inp[k]) for k in ("x1", "x2") if inp[k] is not None], 1).requires_grad_(case["train"])
    w = inp["w"].double().requires_grad_(case["train"])
    b = inp["b"].double().requires_grad_(case["train"])
    y = F.conv3d(x, w.permute(0, 2, 1).reshape(co, c1 + c2, 3, 3, 3), b, padding=1)
    out = padded(F.leaky_relu(y.detach(), SLOPE))
    if not case["train"]:
        return out
    y.backward(dense(inp["gy"]))  # the gradient given is that of the layer's linear output
    d = {"y": out, "dx1": padded(x.grad[:, :c1]), "dw": w.grad, "db": b.grad}
    if c2:
        d["dx2"] = padded(x.grad[:, c1:])
    return d


def exact(case, seed):
    inp = _inputs(case, seed)
    kind = case["kind"]
    if kind == "conv":
        return _exact_conv(case, inp)
    two_d = kind == "pair2d" or (kind == "objective" and case["nz"] == 0)
    E = _Exact2D(case) if two_d else _Exact3D(case)
    vol, theta = inp["vol"].double(), inp["theta"]
    y = inp["y"].double()
    if not two_d:
        vol = vol.movedim(-3, -1)  # (..., ny, nx, nz)
        vol = vol.reshape(vol.shape[:-3] + (-1, vol.shape[-1])).contiguous()
    if kind == "gates4d":
        w = 1.0 if inp["w"] is None else inp["w"].double()
        nt, out, cost = case["gates"], torch.zeros_like(vol), 0.0
        for v, t in enumerate(inp["t"]):
            g0, g1, pe = int(math.floor(t)) % nt, int(math.ceil(t)) % nt, t - math.floor(t)
            r = E.pair(theta[v], vol=(1.0 - pe) * vol[g0] + pe * vol[g1]) - y[v]
            wr = r * (1.0 if inp["w"] is None else w[v])
            cost += 0.5 * float((wr * r).sum())
            b = torch.zeros_like(vol[0])
            E.pair(theta[v], y=wr, out=b)
            out[g0] += (1.0 - pe) * b
            out[g1] += pe * b
        grad = out.view(nt, case["ny"], case["nx"], case["nz"])
        return {"cost": torch.tensor([cost], dtype=torch.float64), "grad": grad}
    out = torch.zeros_like(vol)
    views = [case["view"]] if kind == "view3d" else range(case["views"])
    sino, f = [], 0.0
    for n, v in enumerate(views):
        if kind == "objective":
            r = E.pair(theta[v], vol=vol) - y[v]
            wr = r if inp["w"] is None else r * inp["w"][v].double()
            f += 0.5 * float((wr * r).sum())
            E.pair(theta[v], y=wr, out=out)
        else:
            sino.append(E.pair(theta[v], vol=vol, y=y[n], out=out))
    if not two_d:
        out = out.view(case["ny"], case["nx"], case["nz"])
        if case.get("layout") != "columns":
            out = out.movedim(-1, -3).contiguous()
    if kind != "objective":
        return {"sino": torch.stack(sino), "back": out}
    if case["mu"] > 0:
        tv, gtv = _tv(inp["vol"].double(), case["mu"], case["eps"])
        f, out = f + tv, out + gtv
    return {"f": f, "g": out}
