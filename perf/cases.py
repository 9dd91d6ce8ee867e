"""The calls that users of this framework make, for timing and comparison.

Twelve listed cases over the framework's two halves: the lattice Boltzmann
solver (the reference's small, ordinary and large lattices in 2D and 3D, each
storage kind that a run uses in earnest, the drop-in that hands its whole
state over, and the ensemble that generates training data), and the
warm-start network (prediction, a training step's gradients, and one
convolution layer through the C entry points). draw() gives further cases
of the same ranges.

Every pass starts from the inputs in hand (the solver from InitUP's 100
draws or from the uploaded state, the network from its weights), so passes on
the same state give the same outputs. Flow cases run tens to hundreds of
iterations where a study runs thousands.
"""
import ctypes as C
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imexlb-1.0_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import imexlb as im  # noqa: E402
from imexlb import neural  # noqa: E402

PRECISION = {"fp64": im.FP64, "fp64fast": im.FP64_FAST, "fp32": im.FP32, "bf16": im.BF16,
             "fp16": im.FP16, "fix64": im.FIX64}
BYTES = {"fp64": 8, "fp64fast": 8, "fix64": 8, "fp32": 4, "bf16": 2, "fp16": 2}
GHOST = 3


def _flow(name, nx, ny, nz, d, re, u, precision, steps, interv=0, every=0, mass=False, dropin=False):
    c = dict(kind="flow", nx=nx, ny=ny, nz=nz, d=d, re=re, u=u, precision=precision, steps=steps,
             interv=interv, every=every, mass=mass, dropin=dropin)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a quick look at a small cylinder: kernels of a few microseconds, so launches and
        # the host path count; Monitor lines and the mass check as a run prints them
        _flow("cylinder_128x64_fp64", 128, 64, 0, 16.0, 40.0, 0.05, "fp64", 200, interv=50, mass=True),
        # the plain FP64 run that arbitrates the warm start: force sample every 20 iterations
        _flow("cylinder_1024x512_fp64", 1024, 512, 0, 40.0, 100.0, 0.05, "fp64", 200, every=20),
        # the warm-started run's storage on the same lattice
        _flow("cylinder_1024x512_fp16", 1024, 512, 0, 40.0, 100.0, 0.05, "fp16", 500, every=20),
        # the drop-in inside a host program: its whole state handed over, advanced with
        # Monitor lines, and handed back
        _flow("sphere_128x64x64_dropin", 128, 64, 64, 12.0, 100.0, 0.04, "fp64", 40, interv=20,
              dropin=True),
        # the drop-in's ordinary 3D size (the reference's input_3d.in)
        _flow("sphere_256x128x128_fp64", 256, 128, 128, 24.0, 100.0, 0.04, "fp64", 40, interv=20),
        # the same accuracy in fixed point
        _flow("sphere_256x128x128_fix64", 256, 128, 128, 24.0, 100.0, 0.04, "fix64", 100, interv=50),
        # single-precision storage with drag recorded along the way
        _flow("sphere_256x128x128_fp32", 256, 128, 128, 24.0, 100.0, 0.04, "fp32", 200, every=20),
        # the large lattice of the reduced-precision study, half storage
        _flow("sphere_512x256x256_fp16", 512, 256, 256, 48.0, 200.0, 0.04, "fp16", 150, every=50),
        # the data generator: uneven cylinder cases in one batch, a snapshot of each at the end
        dict(name="ensemble_24_fp32", kind="ensemble", cases=24, nx_lo=256, nx_hi=1024, table=7,
             precision="fp32", steps=500),
        # the prediction that warm-starts one run
        dict(name="net_predict_1", kind="net", n=1, h=128, w=256, train=False),
        # one training step's forward pass, loss and gradients at the training batch
        dict(name="net_train_16", kind="net", n=16, h=128, w=256, train=True),
        # the network's largest layer (upsampling) through the C entry points, both directions
        dict(name="conv_up_16x64x128x48", kind="conv", n=16, h=64, w=128, cin=48, cout=48, stride=1,
             upsample=1, relu=1),
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    k = rng.random()
    if k < 0.3:  # 2D flows, small to large, any storage
        nx = int(_log_uniform(rng, 96, 1500))
        ny = int(nx * rng.uniform(0.4, 0.6))
        d = round(rng.uniform(0.08, 0.2) * ny, 2)
        p = rng.choice(["fp64", "fp64", "fp64fast", "fix64", "fp32", "fp16", "bf16"])
        return _flow(None, nx, ny, 0, d, round(rng.uniform(40, 150), 1), 0.05, p,
                     rng.randrange(50, 300), interv=rng.choice([0, 0, 25]), every=rng.choice([0, 20, 20]),
                     mass=rng.random() < 0.3)
    if k < 0.6:  # 3D flows
        nx = int(_log_uniform(rng, 80, 400))
        ny, nz = int(nx * rng.uniform(0.45, 0.55)), int(nx * rng.uniform(0.45, 0.55))
        d = round(rng.uniform(0.12, 0.25) * min(ny, nz), 2)
        p = rng.choice(["fp64", "fix64", "fp32", "fp32", "fp16", "fp16", "bf16", "fp64fast"])
        most = {"fp64": 6e6, "fp64fast": 6e6, "fix64": 2e7, "fp32": 5e7, "fp16": 1.2e8, "bf16": 1.2e8}[p]
        steps = max(6, min(rng.randrange(20, 200), int(10 * most / (nx * ny * nz))))
        return _flow(None, nx, ny, nz, d, round(rng.uniform(40, 150), 1), 0.04, p, steps,
                     interv=rng.choice([0, 10]), every=rng.choice([0, 10, 20]),
                     mass=rng.random() < 0.2, dropin=rng.random() < 0.15 and nx < 150)
    if k < 0.7:  # ensembles
        return dict(kind="ensemble", cases=rng.randrange(3, 25), nx_lo=256, nx_hi=rng.choice([512, 768, 1024]),
                    table=rng.randrange(1000), precision=rng.choice(["fp32", "fp32", "fp16", "bf16"]),
                    steps=rng.randrange(100, 500))
    if k < 0.85:  # predictions and training steps
        return dict(kind="net", n=int(_log_uniform(rng, 1, 17)), h=4 * rng.randrange(8, 41),
                    w=4 * rng.randrange(16, 73), train=rng.random() < 0.6)
    # single layers
    return dict(kind="conv", n=int(_log_uniform(rng, 1, 17)), h=rng.randrange(13, 70), w=rng.randrange(25, 140),
                cin=rng.choice([16, 32, 48, 48, 64]), cout=rng.choice([16, 32, 48, 48, 64]),
                stride=rng.choice([1, 1, 2]), upsample=rng.choice([0, 0, 1]), relu=rng.choice([0, 1]))


# ---- solver -----------------------------------------------------------------

def _dim(c):
    return 3 if c["nz"] else 2


def _config(c, yoff=0.0):
    # the relaxation parameter that gives inlet speed u at this Reynolds number
    nu = c["u"] * c["d"] / c["re"]
    return im.make_config(_dim(c), c["nx"], c["ny"], c["nz"], charlength=c["d"] / c["nx"], xpos=0.25,
                          re=c["re"], ome=1.0 / (3.0 * nu + 0.5), yoff=yoff)


def _table(c):
    """The ensemble's cases: sizes, diameters, Reynolds numbers and offsets."""
    rng = np.random.default_rng(c["table"])
    out = []
    for _ in range(c["cases"]):
        nx = int(rng.integers(c["nx_lo"] // 32, c["nx_hi"] // 32 + 1)) * 32
        out.append((dict(nx=nx, ny=nx // 2, nz=0, d=float(rng.uniform(16, 48)),
                         re=float(rng.uniform(40, 200)), u=0.05), float(rng.uniform(-2, 2))))
    return out


def _draws(seed):
    return np.random.default_rng(seed).random(100)


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True)


def _prepare_flow(c, seed):
    cfg = _config(c)
    s = im.Solver(cfg, precision=PRECISION[c["precision"]])
    s.set_geometry(im.Setup(cfg, device=0, state=False))
    n, nq, dim = cfg.array_size, cfg.nq, cfg.dim
    st = dict(case=c, solver=s, rv=_draws(seed), p=_pinned(n), u=_pinned(n * dim))
    if c["dropin"]:
        # InitUP's fields and a zero f, fb, in the host program's own buffers
        setup = im.Setup(cfg, rv=st["rv"])
        st["in"] = [torch.zeros(n * nq, dtype=torch.float64).pin_memory() for _ in range(2)]
        st["in"] += [torch.from_numpy(setup.p).pin_memory(), torch.from_numpy(setup.u).pin_memory()]
        st["f"], st["fb"] = _pinned(n * nq), _pinned(n * nq)
    return st


def _run_flow(st):
    c, s = st["case"], st["solver"]
    if c["dropin"]:
        s.upload_ptr(*[t.data_ptr() for t in st["in"]])
    else:
        s.init_state(st["rv"])
    s.init_pdf()
    out = {}
    if c["every"]:
        log, out["force"] = s.step_observed(0, c["steps"], c["interv"], c["every"])
    else:
        log = s.step(0, c["steps"], c["interv"])
    if c["interv"]:
        out["umax"] = log
    if c["mass"]:
        out["drag"], out["mass"] = s.observe()
    f, fb = (st["f"], st["fb"]) if c["dropin"] else (None, None)
    s.download_ptr(f.data_ptr() if c["dropin"] else 0, fb.data_ptr() if c["dropin"] else 0,
                   st["p"].data_ptr(), st["u"].data_ptr())
    out["p"], out["u"] = st["p"], st["u"]
    if c["dropin"]:
        out["f"], out["fb"] = f, fb
    return out


SAMPLE_W, SAMPLE_H = 256, 128


def _prepare_ensemble(c, seed):
    solvers, rv = [], []
    for k, (one, yoff) in enumerate(_table(c)):
        cfg = _config(one, yoff)
        s = im.Solver(cfg, precision=PRECISION[c["precision"]])
        s.set_geometry(im.Setup(cfg, device=0, state=False))
        rv.append(_draws([seed, k]))
        s.init_state(rv[-1])
        s.init_pdf()
        s.step(0, 1)
        solvers.append(s)
    batch = im.Batch(solvers)
    batch.tune(trial=4)  # the launch shape, once per batch
    return dict(case=c, solvers=solvers, rv=rv, batch=batch)


def _run_ensemble(st):
    for s, rv in zip(st["solvers"], st["rv"]):
        s.init_state(rv)
        s.init_pdf()
        s.step(0, 1)
    st["batch"].step(st["case"]["steps"])
    return [s.sample(SAMPLE_W, SAMPLE_H) for s in st["solvers"]]


# ---- network ----------------------------------------------------------------

def _fields(n, h, w, seed):
    """Masks of one cylinder each, Reynolds numbers and smooth wakes behind them."""
    rng = np.random.default_rng(seed)
    col = lambda lo, hi: torch.tensor(rng.uniform(lo, hi, n), dtype=torch.float32, device="cuda").view(n, 1, 1)
    cx, cy, r, re = col(0.2 * w, 0.3 * w), col(0.45 * h, 0.55 * h), col(0.02 * w, 0.05 * w), col(40, 200)
    X = torch.arange(w, device="cuda", dtype=torch.float32).view(1, 1, w) - cx
    Y = torch.arange(h, device="cuda", dtype=torch.float32).view(1, h, 1) - cy
    rr = torch.sqrt(X * X + Y * Y)
    frac = torch.clamp(rr - r + 0.5, 0, 1)  # fluid fraction of the pixel
    wake = torch.exp(-Y * Y / (2 * r * r)) * torch.sigmoid(X / r) * torch.exp(-torch.relu(X) / (0.3 * w))
    ux = frac * (1 - 0.9 * wake)
    uy = frac * wake * torch.sin(X * 6.0 / r / 5.0) * (re / 400)
    p = 0.4 * torch.exp(-rr / (2 * r)) * torch.sign(-X)
    return frac, re, torch.stack([p, ux, uy], dim=-1).contiguous()


def _prepare_net(c, seed):
    frac, re, target = _fields(c["n"], c["h"], c["w"], seed)
    x = torch.zeros(c["n"], c["h"], c["w"], neural.CIN, device="cuda")
    x[..., 0] = frac
    x[..., 1] = re / 200.0
    return dict(case=c, net=neural.Net(seed=seed % (1 << 31)), x=x.to(torch.bfloat16), target=target)


def _run_net(st):
    net = st["net"]
    if not st["case"]["train"]:
        return net.forward(st["x"])
    y = net.forward(st["x"], keep=True)
    loss, dy = net.loss(y, st["target"])
    return [y, loss] + net.backward(dy)


def _conv_desc(c):
    up = 2 if c["upsample"] else 1
    return im.ConvDesc(c["n"], c["h"], c["w"], c["cin"], (up * c["h"] - 1) // c["stride"] + 1,
                       (up * c["w"] - 1) // c["stride"] + 1, c["cout"], 0, c["stride"], c["upsample"])


def _prepare_conv(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    d = _conv_desc(c)
    # activations behind a ReLU, as every layer but the first reads them
    x = torch.relu(rnd(c["n"], c["h"], c["w"], c["cin"])).to(torch.bfloat16)
    w = (rnd(c["cout"], 9 * c["cin"]) * (2.0 / (9 * c["cin"])) ** 0.5).to(torch.bfloat16)
    return dict(case=c, desc=d, x=x, w=w, b=0.1 * rnd(c["cout"]),
                dy=1e-3 * rnd(c["n"], d.hout, d.wout, c["cout"]))


def _run_conv(st):
    c, d = st["case"], st["desc"]
    L, p = im.lib(), neural._p

    def ok(rc):
        if rc:
            raise RuntimeError("convolution call failed (%d)" % rc)

    new = lambda shape, dt: torch.empty(shape, dtype=dt, device="cuda")
    up = 2 if c["upsample"] else 1
    y = new((c["n"], d.hout, d.wout, c["cout"]), torch.bfloat16)
    ok(L.imexlb_nn_conv_fwd(C.byref(d), p(st["x"]), p(st["w"]), p(st["b"]), c["relu"], p(y), None, None))
    dz = new(y.shape, torch.bfloat16)
    db = torch.zeros(c["cout"], device="cuda")
    ok(L.imexlb_nn_act_grad(p(st["dy"]), p(y) if c["relu"] else None, y.numel(), c["cout"], c["relu"],
                            p(dz), p(db), None))
    dw = torch.zeros((c["cout"], 9 * c["cin"]), device="cuda")
    ok(L.imexlb_nn_conv_bwd_weight(C.byref(d), p(st["x"]), p(dz), p(dw), None))
    dgrid = new((c["n"], up * c["h"], up * c["w"], c["cin"]), torch.float32)
    dx = new((c["n"], c["h"], c["w"], c["cin"]), torch.float32) if c["upsample"] else None
    wt = new((c["cin"], 9 * c["cout"]), torch.bfloat16)
    ok(L.imexlb_nn_conv_bwd_data(C.byref(d), p(dz), p(st["w"]), p(wt), p(dgrid), p(dx), None))
    return [y, dz, db, dw, dgrid] + ([dx] if c["upsample"] else [])


def prepare(case, seed):
    return {"flow": _prepare_flow, "ensemble": _prepare_ensemble, "net": _prepare_net,
            "conv": _prepare_conv}[case["kind"]](case, seed)


def run(state):
    return {"flow": _run_flow, "ensemble": _run_ensemble, "net": _run_net,
            "conv": _run_conv}[state["case"]["kind"]](state)


# ---- work -------------------------------------------------------------------

def _nodes(c):
    return (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1 if c["nz"] else 1)


def _conv_work(n, hin, win, cin, hout, wout, cout, up, passes, out_bytes=2):
    """One layer: bytes of its tensors and multiply-adds of `passes` GEMMs."""
    px = n * hout * wout
    b = n * hin * win * cin * 2 + px * cout * out_bytes + 9 * cin * cout * 2
    f = 2.0 * px * cout * 9 * cin * passes
    return b, f


def work(case):
    c = case
    if c["kind"] == "flow":
        # every iteration reads and writes each population once; the fields go back in FP64
        dim = _dim(c)
        q = 9 if dim == 2 else 27
        n = _nodes(c)
        b = c["steps"] * 2.0 * q * BYTES[c["precision"]] * n + 8.0 * (1 + dim) * n
        if c["dropin"]:
            b += 8.0 * n * (4 * q + 1 + dim)
        return {"bytes": b, "flops": c["steps"] * 12.0 * q * n}
    if c["kind"] == "ensemble":
        n = sum(_nodes(one) for one, _ in _table(c))
        return {"bytes": (c["steps"] + 1) * 18.0 * BYTES[c["precision"]] * n + c["cases"] * 16.0 * SAMPLE_W * SAMPLE_H,
                "flops": c["steps"] * 108.0 * n}
    if c["kind"] == "conv":
        d = _conv_desc(c)
        b, f = _conv_work(c["n"], c["h"], c["w"], c["cin"], d.hout, d.wout, c["cout"], c["upsample"], 3)
        px, up = c["n"] * d.hout * d.wout, 4 if c["upsample"] else 1
        # x, w and dy are read; y, dz, the gradients of x (on the stencil grid and summed) and w written
        b += px * c["cout"] * (4 + 2) + 9 * c["cin"] * c["cout"] * 4
        b += c["n"] * c["h"] * c["w"] * c["cin"] * 4 * (up + (1 if up > 1 else 0))
        return {"bytes": b, "flops": f}
    b = f = 0.0
    h, w = c["h"], c["w"]
    for i, (cin, cout, stride, up, _) in enumerate(neural.LAYERS):
        hg, wg = (2 * h, 2 * w) if up else (h, w)
        ho, wo = (hg - 1) // stride + 1, (wg - 1) // stride + 1
        last = i == len(neural.LAYERS) - 1
        lb, lf = _conv_work(c["n"], h, w, cin, ho, wo, cout, up, (3 if i else 2) if c["train"] else 1,
                            4 if last else 2)
        b, f = b + lb * (3 if c["train"] else 1), f + lf
        h, w = ho, wo
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits ----------------------------------------------

class _Exact:
    """The flow in torch float64 whole-array operations: BGK collision, periodic
    halo, wall / obstacle / inlet / outlet copies, pull, moments. Arrays are
    [.., Z, Y, X] with the ghost layers (2D: Z = 1)."""

    def __init__(self, c, yoff=0.0):
        self.dim = dim = _dim(c)
        self.L = [c["nx"] + 1, c["ny"] + 1] + ([c["nz"] + 1] if dim == 3 else [])
        nu = c["u"] * c["d"] / c["re"]
        self.ome = 1.0 / (3.0 * nu + 0.5)
        self.uu = c["re"] * ((2.0 - self.ome) / (6.0 * self.ome)) / (c["d"] / c["nx"] * c["nx"])
        G = GHOST
        self.P = P = [l + 2 * G for l in self.L]
        # velocities and weights in the reference's order
        if dim == 2:
            self.e = [(i, j, 0) for i in (-1, 0, 1) for j in (-1, 0, 1)]
            self.t = [4.0 * (1 - 0.75 * i * i) * (1 - 0.75 * j * j) / 9.0 for i, j, _ in self.e]
        else:
            self.e = [(i, j, k) for k in (-1, 0, 1) for i in (-1, 0, 1) for j in (-1, 0, 1)]
            self.t = [8.0 / 4.0 ** (abs(i) + abs(j) + abs(k)) / 27.0 for i, j, k in self.e]
        self.Q = len(self.e)
        shape = (P[2] if dim == 3 else 1, P[1], P[0])
        dev = "cuda"
        self.shape, self.N = shape, int(np.prod(shape))
        # nodes outside the obstacle are fluid; the periodic halo repeats them
        r = c["d"] / c["nx"] * c["nx"] * 0.5
        x = torch.arange(self.L[0], device=dev, dtype=torch.float64) - 0.25 * c["nx"]
        y = torch.arange(self.L[1], device=dev, dtype=torch.float64) - (c["ny"] / 2.0 + yoff)
        r2 = x[None, None, :] ** 2 + y[None, :, None] ** 2
        if dim == 3:
            z = torch.arange(self.L[2], device=dev, dtype=torch.float64) - c["nz"] / 2.0
            r2 = r2 + z[:, None, None] ** 2
        geo = torch.zeros(shape, dtype=torch.bool, device=dev)
        self.inner = (slice(G, -G) if dim == 3 else slice(None), slice(G, -G), slice(G, -G))
        geo[self.inner] = r2 > r * r
        self.fluid = geo[self.inner].clone()
        self.wrap(geo[None])
        self.geo = geo
        self._obstacle()

    def wrap(self, a):
        """Ghost layers from one period away, every dimension."""
        G = GHOST
        a[..., :G], a[..., -G:] = a[..., -2 * G:-G].clone(), a[..., G:2 * G].clone()
        a[..., :G, :], a[..., -G:, :] = a[..., -2 * G:-G, :].clone(), a[..., G:2 * G, :].clone()
        if self.dim == 3:
            a[..., :G, :, :], a[..., -G:, :, :] = a[..., -2 * G:-G, :, :].clone(), a[..., G:2 * G, :, :].clone()

    def _obstacle(self):
        """The obstacle cells the reference bounces: the first solid cell of each
        x-row with a fluid node at one of its probes; their copies, each
        from where its value comes; the links of the force sum."""
        dim, Q = self.dim, self.Q
        dy, dz = self.P[0], self.P[0] * self.P[1] if dim == 3 else 0
        geo = self.geo.reshape(-1).cpu().numpy()
        solid = np.zeros(self.shape, dtype=bool)
        solid[self.inner] = ~self.fluid.cpu().numpy()
        cand = np.flatnonzero(solid.reshape(-1))
        hit = np.zeros(cand.size, dtype=bool)
        for q, (ex, _, _) in enumerate(self.e):
            at = cand + ex + dy * (q * dim + 1) + dz * (q * dim + 2 if dim == 3 else 0)
            ok = ~hit & (at >= 0) & (at < self.N)
            hit[ok] = geo[at[ok]]
        cand = cand[hit]
        cells = np.sort(cand[np.unique(cand // dy, return_index=True)[1]])
        off = [ex + dy * ey + dz * ez for ex, ey, ez in self.e]
        origin = {}
        for cell in cells.tolist():
            for q in range(Q):
                s = (Q - 1 - q) * self.N + cell + 2 * off[q]
                origin[q * self.N + cell] = origin.get(s, s)
        as_index = lambda v: torch.tensor(np.fromiter(v, dtype=np.int64, count=len(origin)), device="cuda")
        self.user_to, self.user_from = as_index(origin.keys()), as_index(origin.values())
        # links x -> s = x + e from fluid to solid nodes
        a, b, q_of = [], [], []
        body = np.flatnonzero(solid.reshape(-1))
        fluid = np.zeros(self.shape, dtype=bool)
        fluid[self.inner] = self.fluid.cpu().numpy()
        fluid = fluid.reshape(-1)
        for q in range(Q):
            src = body - off[q]
            s = body[fluid[src]]
            a.append(q * self.N + s - off[q])
            b.append((Q - 1 - q) * self.N + s)
            q_of.append(np.full(s.size, q))
        dev = lambda v: torch.tensor(np.concatenate(v), device="cuda")
        self.link_a, self.link_b = dev(a), dev(b)
        self.link_e = torch.tensor(np.array(self.e, dtype=np.float64)[:, :dim], device="cuda")[dev(q_of)]

    def profile(self):
        n = self.L[-1] - 1
        v = torch.arange(self.L[-1], device="cuda", dtype=torch.float64)
        v = self.uu * 4.0 * v * (n - v) / float(n * n)
        return v.view(-1, 1, 1) if self.dim == 3 else v.view(1, -1, 1)

    def init(self, draws):
        r = 1.0 + (torch.tensor(draws, device="cuda") - 0.5) * 2.0 * 0.2
        ids = torch.arange(self.N, device="cuda").view(self.shape)[self.inner]
        self.u = [torch.zeros(self.fluid.shape, dtype=torch.float64, device="cuda") for _ in range(self.dim)]
        self.u[0] = self.profile() * r[ids % 100] * self.fluid
        self.p = torch.zeros_like(self.u[0])
        self.f = torch.zeros((self.Q,) + tuple(self.fluid.shape), dtype=torch.float64, device="cuda")
        self.fb = torch.zeros((self.Q,) + self.shape, dtype=torch.float64, device="cuda")
        usq = sum(v * v for v in self.u)
        for q in range(self.Q):
            self.f[q] = self.feq(q, usq) * self.fluid

    def feq(self, q, usq):
        e = self.e[q]
        eu = sum((v if s > 0 else -v) for s, v in zip(e, self.u) if s) if any(e[:self.dim]) else None
        s = -1.5 * usq
        if eu is not None:
            s = s + 3.0 * eu + 4.5 * eu * eu
        return self.t[q] * (3.0 * self.p + s)

    def step(self):
        G, dim, Q, L = GHOST, self.dim, self.Q, self.L
        usq = sum(v * v for v in self.u)
        fb = self.fb
        for q in range(Q):
            inner = fb[(q,) + self.inner]
            new = (1.0 - self.ome) * self.f[q] + self.ome * self.feq(q, usq)
            inner.copy_(torch.where(self.fluid, new, inner))
        for q in range(Q):
            self.wrap(fb[q:q + 1])
        # walls: low and high face of y (2D) / z (3D), bounced from two cells in
        span = lambda ax, shift: slice(G - 1 + shift, G + L[ax] + 1 + shift)
        for at, sign in ((G - 1, 1), (G + L[-1], -1)):
            for q, (ex, ey, ez) in enumerate(self.e):
                if (ez if dim == 3 else ey) != sign:
                    continue
                if dim == 3:
                    fb[q, at, span(1, 0), span(0, 0)] = fb[Q - 1 - q, at + 2 * sign, span(1, 2 * ey), span(0, 2 * ex)]
                else:
                    fb[q, 0, at, span(0, 0)] = fb[Q - 1 - q, 0, at + 2 * sign, span(0, 2 * ex)]
        flat = fb.view(-1)
        flat[self.user_to] = flat[self.user_from]
        # inlet and outlet columns
        fb[..., G - 1] = fb[..., G]
        ys = slice(G - 1, G + L[1] + 1)
        for q, (ex, ey, ez) in enumerate(self.e):
            if ex == -1:
                zs = (lambda s: slice(G - 1 + s, G + L[2] + 1 + s)) if dim == 3 else (lambda s: slice(None))
                y2 = slice(ys.start + ey, ys.stop + ey)
                fb[q, zs(0), ys, G + L[0]] = fb[q, zs(ez), y2, G + L[0] - 1].clone()
        # pull and moments
        p = torch.zeros_like(self.p)
        u = [torch.zeros_like(p) for _ in range(dim)]
        for q, e in enumerate(self.e):
            ix = [slice(G - s, G - s + l) for s, l in zip(e, L)]
            v = fb[(q, ix[2] if dim == 3 else 0, ix[1], ix[0])]
            v = (v if dim == 3 else v[None]) * self.fluid
            self.f[q] = v
            p += v
            for k in range(dim):
                if e[k]:
                    u[k] += e[k] * v
        self.p, self.u = p / 3.0, u
        self.u[0][..., 0] = self.profile()[..., 0] * self.fluid[..., 0]
        self.u[1][..., 0] = 0.0
        self.p[..., -1] = 0.0

    def umax(self):
        s = torch.sqrt(self.u[0] ** 2 + self.u[1] ** 2) * self.fluid
        s.view(-1)[torch.nonzero(self.fluid.view(-1))[0]] = 0.0  # Monitor leaves out the first fluid node
        return float(s.max())

    def force(self):
        flat = self.fb.view(-1)
        return ((flat[self.link_a] + flat[self.link_b])[:, None] * self.link_e).sum(0).cpu().numpy()

    def padded(self, parts):
        """Per-node values in the reference layout, ghost and solid cells zero."""
        out = torch.zeros(self.shape + (len(parts),), dtype=torch.float64, device="cuda")
        for k, v in enumerate(parts):
            out[self.inner + (k,)] = v * self.fluid
        return out

    def velocity(self):
        """u in the reference layout: the inlet profile is also set on the column's
        first ghost rows (one below, two above the lattice)."""
        out, G, L = self.padded(self.u), GHOST, self.L
        n = L[-1] - 1
        v = torch.arange(-1, L[-1] + 2, device="cuda", dtype=torch.float64)
        v = self.uu * 4.0 * v * (n - v) / float(n * n)
        for ax in range(1, self.dim):  # ghost rows of y, then of z
            for at in (-1, L[ax], L[ax] + 1):
                if self.dim == 2:
                    out[0, G + at, G, 0] = v[1 + at]
                elif ax == 1:
                    out[G - 1:G + L[2] + 2, G + at, G, 0] = v
                else:
                    out[G + at, G - 1:G + L[1] + 2, G, 0] = v[1 + at]
        return out


def _exact_flow(c, seed):
    x = _Exact(c)
    x.init(_draws(seed))
    umax, force = [], []
    for it in range(c["steps"]):
        if c["interv"] and it % c["interv"] == 0:
            umax.append(x.umax())
        x.step()
        if c["every"] and it % c["every"] == 0:
            force.append(x.force())
    out = {}
    if c["every"]:
        out["force"] = np.array(force)
    if c["interv"]:
        out["umax"] = np.array(umax)
    if c["mass"]:
        out["drag"], out["mass"] = x.force(), float(x.f.sum())
    out["p"], out["u"] = x.padded([x.p]).view(-1).cpu(), x.velocity().view(-1).cpu()
    if c["dropin"]:
        # fb's ghost corners repeat what the reference reads outside its arrays
        out["f"], out["fb"] = x.padded(list(x.f)).view(-1).cpu(), None
    return out


def _exact_ensemble(c, seed):
    outs = []
    for k, (one, yoff) in enumerate(_table(c)):
        x = _Exact(one, yoff)
        x.init(_draws([seed, k]))
        for _ in range(c["steps"] + 1):
            x.step()
        # bilinear between nodes at the pixel centres
        L0, L1 = x.L
        at = lambda n, L: torch.clamp((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * L / n - 0.5, 0, L - 1)
        X, Y = at(SAMPLE_W, L0), at(SAMPLE_H, L1)
        x0, y0 = torch.clamp(X.long(), max=L0 - 2), torch.clamp(Y.long(), max=L1 - 2)
        fx, fy = (X - x0)[None, :], (Y - y0)[:, None]
        planes = []
        for v in (x.fluid.double(), x.p, x.u[0], x.u[1]):
            g = lambda b, a: (v * x.fluid)[0][(y0 + b)[:, None], (x0 + a)[None, :]]
            planes.append((1 - fy) * ((1 - fx) * g(0, 0) + fx * g(0, 1)) + fy * ((1 - fx) * g(1, 0) + fx * g(1, 1)))
        outs.append(torch.stack(planes))
    return outs


def _conv64(x, w, b, stride, up):
    """3x3 convolution of NHWC float64 values (zero padding)."""
    cout, cin = w.shape[0], x.shape[-1]
    x = x.permute(0, 3, 1, 2)
    if up:
        x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
    return F.conv2d(x, w.view(cout, 3, 3, cin).permute(0, 3, 1, 2), b, stride=stride, padding=1).permute(0, 2, 3, 1)


def _half(v):
    return v.to(torch.bfloat16).double()


def _conv_grads64(x, w, dz, stride, up):
    """Gradients of _conv64: with respect to the stencil grid, x and w."""
    grid = x.repeat_interleave(2, 1).repeat_interleave(2, 2) if up else x
    grid, w = grid.clone().requires_grad_(True), w.clone().requires_grad_(True)
    _conv64(grid, w, None, stride, 0).backward(dz)
    g = grid.grad
    n, h, wd, ch = x.shape
    dx = g.view(n, h, 2, wd, 2, ch).sum((2, 4)) if up else g
    return g, dx, w.grad


def _exact_conv(c, seed):
    st = _prepare_conv(c, seed)
    x, w = st["x"].double(), st["w"].double()
    y = _conv64(x, w, st["b"].double(), c["stride"], c["upsample"])
    y = torch.relu(y) if c["relu"] else y
    dz = st["dy"].double() * (y > 0) if c["relu"] else st["dy"].double()
    g, dx, dw = _conv_grads64(x, w, _half(dz), c["stride"], c["upsample"])
    return [y, dz, dz.sum((0, 1, 2)), dw, g] + ([dx] if c["upsample"] else [])


def _exact_net(c, seed):
    """64-bit sums; activations and their gradients kept in bfloat16 between
    layers, as the network stores them."""
    st = _prepare_net(c, seed)
    net = st["net"]
    acts, n_layers = [st["x"].double()], len(neural.LAYERS)
    ws, bs = [w.double() for w in net.wb], [b.double() for b in net.b]
    for i, (_, _, stride, up, relu) in enumerate(neural.LAYERS):
        y = _conv64(acts[-1], ws[i], bs[i], stride, up)
        y = torch.relu(y) if relu else y
        acts.append(y if i == n_layers - 1 else _half(y))
    y = acts[-1]
    if not c["train"]:
        return y
    used = neural.USED
    diff = y[..., :used] - st["target"].double()
    count = diff.numel()
    dy = torch.zeros_like(y)
    dy[..., :used] = 2.0 * diff / count
    gw, gb = [None] * n_layers, [None] * n_layers
    for i in range(n_layers - 1, -1, -1):
        _, _, stride, up, relu = neural.LAYERS[i]
        g = dy * (acts[i + 1] > 0) if relu else dy
        gb[i] = g.sum((0, 1, 2))
        _, dy, gw[i] = _conv_grads64(acts[i], ws[i], _half(g), stride, up)
    return [y, (diff * diff).sum().view(1) / count] + gw + gb


def exact(case, seed):
    if case["kind"] == "flow" and case["steps"] * _nodes(case) > 6e9:
        return None
    with torch.no_grad() if case["kind"] in ("flow", "ensemble") else torch.enable_grad():
        return {"flow": _exact_flow, "ensemble": _exact_ensemble, "net": _exact_net,
                "conv": _exact_conv}[case["kind"]](case, seed)
