"""The workloads this framework is timed on, through its public entry points.

Kinds of case:

* ``steps``    a handler steps a channel and its four result fields come to the host
               (``create_handler``, ``run_steps``, ``sync_results``, the result getters);
* ``run``      a handler's whole life cycle: ``initialize``, ``start``, ``block_until_finished``, results,
               with a frame of results every ``frame`` steps;
* ``steady``   the steady-state loop: steps with the residual taken every ``k`` steps (``run_to_residual``);
* ``batch``    many uneven porous channels advanced together (``Batch.run``, ``Batch.result``);
* ``nn_forward`` / ``nn_train``  the warm-start operator: one inference, one training step.

Channels start from rest, as the solver always does, and go on from pass to pass (``run`` starts anew).
Geometries: "open" (walls only), "circle" (walls and a disk of radius H/8 at W/4), "porous" (walls and
disks of radius 3 to 11 in a jittered grid), "scenario-circle" (the solver's own circle scenario).
"""
import math

import numpy as np
import torch

import portlbm_gb300 as plbm

# value size in bytes of each storage form
SIZES = {"f64_strict": 8, "f64_fast": 8, "f64_q60": 8, "f32_ref": 4, "f32": 4, "f16s": 2, "bf16s": 2, "f16c": 2}
WORK_GROUP = 1024
LARGEST = 8192 * 8192 * 40     # node updates of the largest listed pass

# (Cin, Cout) of the warm-start operator's 3x3 convolutions
ENC = [(4, 32), (32, 32), (32, 64), (64, 64), (64, 96), (96, 96), (96, 128), (128, 128), (128, 128), (128, 128)]
DEC = [(128, 128), (128, 128), (128, 96), (96, 96), (96, 64), (64, 64), (64, 32), (32, 32)]
HEAD = (32, 3)


def listed():
    return [
        # the smoke and regression size: launch latency is all there is
        dict(name="smoke_62x30_strict", kind="steps", alg="nptl", lay="stream", prec="f64_strict", w=62, h=30,
             geometry="circle", steps=200),
        # the parity channel (400 x 100, tau 0.6, rho 1.2 / 1.0) of the drop-in form
        dict(name="parity_400x100_strict", kind="steps", alg="nptl", lay="stream", prec="f64_strict", w=400, h=100,
             geometry="open", steps=1000),
        # the bundled settings.json as a whole run: lptl, bundle, circle, a frame every 10 steps
        dict(name="settings_512x128_run", kind="run", alg="lptl", lay="bundle", prec="f64_strict", w=512, h=128,
             geometry="scenario-circle", steps=2000, frame=10),
        # the FP64 sweep's small size, drop-in arithmetic, one lattice in place
        dict(name="sweep_2000x500_strict_npol", kind="steps", alg="npol", lay="collision", prec="f64_strict", w=2000,
             h=500, geometry="circle", steps=100),
        # the same size in the FP64-accuracy form, the swap algorithm
        dict(name="sweep_2000x500_q60_nsol", kind="steps", alg="nsol", lay="bundle", prec="f64_q60", w=2000, h=500,
             geometry="circle", steps=500),
        # the headline channel
        dict(name="headline_8192_q60", kind="steps", alg="nptl", lay="stream", prec="f64_q60", w=8192, h=8192,
             geometry="circle", steps=40),
        # single precision on an ordinary channel, ragged extents
        dict(name="channel_4000x1999_f32", kind="steps", alg="lptl", lay="stream", prec="f32", w=4000, h=1999,
             geometry="circle", steps=200),
        # the precision study's porous channel, FP16 storage
        dict(name="porous_4096_f16s", kind="steps", alg="nptl", lay="stream", prec="f16s", w=4096, h=4096,
             geometry="porous", steps=200),
        # the steady-state loop of the warm-start evaluation: 1000 steps, a residual every 100
        dict(name="steady_1024x256_q60", kind="steady", alg="nptl", lay="stream", prec="f64_q60", w=1024, h=256,
             geometry="porous", steps=1000, k=100),
        # training data: uneven porous channels in single precision, the tile generate_dataset uses
        dict(name="batch20_f32", kind="batch", prec="f32", domains=20, lo=64, hi=1024, steps=1000, vec=False),
        # one inference of the warm-start operator
        dict(name="nn_forward_1x256", kind="nn_forward", n=1, h=256, w=256),
        # one training step at the batch size and extents the operator is trained with
        dict(name="nn_train_16x256", kind="nn_train", n=16, h=256, w=256),
    ]


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["run", "steady", "batch", "nn_forward", "nn_train"])
    prec = rng.choice(["f64_strict"] * 3 + ["f64_q60"] * 3 + ["f32"] * 2 + ["f16s"] * 2 + ["f64_fast", "bf16s", "f16c"])

    def log_size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "steps":
        w, h = log_size(48, 6000), log_size(24, 6000)
        steps = max(20, min(1000, int(rng.uniform(1e8, 2e9) / (w * h)), LARGEST // (w * h)))
        return dict(kind=kind, alg=rng.choice(["nptl", "nptl", "lptl", "lptl", "npol", "nsol"]),
                    lay=rng.choice(["stream", "collision", "bundle"]), prec=prec, w=w, h=h,
                    geometry=rng.choice(["open", "circle", "porous"]), steps=steps)
    if kind == "run":
        return dict(kind=kind, alg=rng.choice(["nptl", "lptl", "npol", "nsol"]),
                    lay=rng.choice(["stream", "collision", "bundle"]), prec=rng.choice(["f64_strict", "f64_q60"]),
                    w=log_size(100, 1200), h=log_size(50, 400), geometry="scenario-circle", steps=rng.randint(500, 2000),
                    frame=rng.choice([5, 10, 25, 100]))
    if kind == "steady":
        return dict(kind=kind, alg=rng.choice(["nptl", "lptl"]), lay=rng.choice(["stream", "bundle"]),
                    prec=rng.choice(["f64_q60", "f64_q60", "f32", "f64_strict"]), w=log_size(128, 1500),
                    h=log_size(64, 600), geometry="porous", steps=1000, k=rng.choice([50, 100]))
    if kind == "batch":
        p = rng.choice(["f32", "f16s", "bf16s", "f64_q60"])
        return dict(kind=kind, prec=p, domains=rng.randint(2, 20), lo=rng.randint(64, 128), hi=rng.randint(256, 1024),
                    steps=rng.randint(200, 1000), vec=p in ("f16s", "bf16s") and rng.random() < 0.7)
    if kind == "nn_forward":
        return dict(kind=kind, n=rng.choice([1, 1, 2, 5]), h=16 * rng.randint(4, 16), w=rng.choice([128, 256, 384, 1024]))
    return dict(kind="nn_train", n=rng.randint(2, 16), h=16 * rng.randint(4, 16), w=rng.choice([64, 128, 256]))


# ---- inputs ----------------------------------------------------------------------------------


def _physics(case, seed):
    """Relaxation time and inlet density of a seed: the stable range the repository's studies use."""
    r = np.random.default_rng(seed * 7919 + 1)
    tau = 0.6 + 0.02 * float(r.random())
    if case.get("prec") in ("f16s", "bf16s", "f16c", "f32"):
        return tau, 1.01 + 0.01 * float(r.random())
    return tau, (1.01 + 0.02 * float(r.random())) if case.get("geometry") == "porous" else 1.18 + 0.02 * float(r.random())


def _porous(w, h, seed):
    """Walls on the first and last row and one disk (radius 3 to 11) in most cells of a 24-node grid."""
    r = np.random.default_rng(seed * 6151 + 17)
    c = 24
    gy, gx = h // c + 1, w // c + 1
    rad = r.uniform(3.0, 11.0, (gy, gx)) * (r.random((gy, gx)) < 0.9)
    cy = np.arange(gy)[:, None] * c + 0.5 * c + (0.5 * c - rad) * r.uniform(-1, 1, (gy, gx))
    cx = np.arange(gx)[None, :] * c + 0.5 * c + (0.5 * c - rad) * r.uniform(-1, 1, (gy, gx))
    f = dict(dtype=torch.float32, device="cuda")
    rad, cy, cx = (torch.tensor(a, **f) for a in (rad, cy, cx))
    ys, xs = torch.arange(h, device="cuda"), torch.arange(w, device="cuda")
    iy, ix = (ys // c)[:, None], (xs // c)[None, :]
    d2 = (ys[:, None] + 0.5 - cy[iy, ix]) ** 2 + (xs[None, :] + 0.5 - cx[iy, ix]) ** 2
    m = (d2 <= rad[iy, ix] ** 2) & (rad[iy, ix] > 0)
    m[0, :] = True
    m[h - 1, :] = True
    return m.to(torch.int8).cpu().numpy()


def _mask(case, seed):
    """(H, W) int8 solid mask, or None where the handler builds the scenario's own geometry."""
    w, h, g = case["w"], case["h"], case["geometry"]
    if g == "scenario-circle":
        return None
    if g == "porous":
        return _porous(w, h, seed)
    m = np.zeros((h, w), dtype=np.int8)
    m[0, :] = 1
    m[h - 1, :] = 1
    if g == "circle":
        r, cx, cy = h // 8, w // 4, h // 2
        ys, xs = np.arange(h)[:, None], np.arange(w)[None, :]
        x0, x1 = max(0, cx - r), min(w, cx + r + 1)
        m[:, x0:x1] |= ((xs[:, x0:x1] - cx) ** 2 + (ys - cy) ** 2 <= r * r).astype(np.int8)
    return m


def _batch_domains(case, seed):
    r = np.random.default_rng(seed * 31 + 5)
    size = np.random.default_rng(case["domains"] * 65537 + case["lo"] * 257 + case["hi"])   # the case's own
    doms = []
    for i in range(case["domains"]):
        w, h = (int(size.integers(case["lo"], case["hi"] + 1)) for _ in range(2))
        doms.append({"mask": _porous(w, h, seed * 1000 + i), "relaxation_time": float(r.uniform(0.6, 1.0)),
                     "inlet_density": float(r.uniform(1.001, 1.03)), "outlet_density": 1.0})
    return doms


def _nn_inputs(case, seed):
    """Solid masks, the three per-sample scalars, and targets of a batch of channels."""
    n, h, w = case["n"], case["h"], case["w"]
    r = np.random.default_rng(seed * 13 + 3)
    masks = np.stack([_porous(w, h, seed * 100 + i) for i in range(n)])
    feats = np.empty((n, 3), dtype=np.float32)
    for i in range(n):
        tau, rin = float(r.uniform(0.55, 1.0)), float(r.uniform(1.001, 1.05))
        g, nu = (rin - 1.0) / (w + 1), (tau - 0.5) / 3.0
        feats[i] = [1.0, (tau - 0.775) * 4.0, math.log10(max(abs(g) / 3.0 * 64.0 / nu, 1e-12)) + 2.25]
    targets = r.standard_normal((n, h, w, 3)).astype(np.float32)
    return masks, feats, targets


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "steady", "run"):
        tau, rin = _physics(case, seed)
        mask = _mask(case, seed)
        total = case["steps"] if kind == "run" else 10 ** 9
        props = plbm.Properties(case["alg"], case["lay"], False, WORK_GROUP, total, case.get("frame", 10 ** 9),
                                "circle" if mask is None else "Hagen-Poiseuille", case["h"], case["w"], 0.0, 0.0, rin,
                                0.0, 0.0, 1.0, tau)
        return {"case": case, "handler": plbm.create_handler(props, precision=case["prec"], mask=mask)}
    if kind == "batch":
        b = plbm.Batch(_batch_domains(case, seed), precision=case["prec"])
        if case["vec"]:
            b.set_tile(32, 4 + 256 * 2 + plbm.BATCH_TILE_VEC, 4)
        else:
            b.set_tile(32, 4 + 256 * 8, 16)
        return {"case": case, "batch": b}
    from portlbm_gb300 import warmstart
    masks, feats, targets = _nn_inputs(case, seed)
    return {"case": case, "model": warmstart.NeuralOperator(seed), "masks": torch.from_numpy(masks).cuda(),
            "feats": feats, "targets": torch.from_numpy(targets).cuda(),
            "count": float((masks == 0).sum() * 3), "loss": torch.zeros(1, dtype=torch.float32, device="cuda"),
            "grad": torch.empty((case["n"], case["h"], case["w"], 3), dtype=torch.bfloat16, device="cuda")}


class _Field(np.ndarray):
    """A result array of a handler that keeps the handler, whose memory it is, alive."""


def _fields(h):
    out = {}
    for name, get in (("rho", h.get_densities), ("jx", h.get_x_velocities), ("jy", h.get_y_velocities),
                      ("jabs", h.get_absolute_velocities)):
        out[name] = get(copy=False).view(_Field)
        out[name].handler = h
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        h = state["handler"]
        h.run_steps(case["steps"])
        h.sync_results()
        return _fields(h)
    if kind == "run":
        h = state["handler"]
        h.initialize()
        h.start()
        h.block_until_finished()
        return _fields(h)
    if kind == "steady":
        h = state["handler"]
        # a target that is never met: every pass is the same number of steps
        steps, residual = h.run_to_residual(0.0, case["k"], case["steps"])
        return {"steps": steps, "residual": residual, **_fields(h)}
    if kind == "batch":
        b = state["batch"]
        b.run(case["steps"], mode="persistent_graph")
        return [[b.result(i, f) for f in range(3)] for i in range(case["domains"])]
    model, n, hh, ww = state["model"], case["n"], case["h"], case["w"]
    x = model.assemble(state["masks"], state["feats"])
    pred = model.forward(x, n, hh, ww)
    if kind == "nn_forward":
        return pred
    state["loss"].zero_()
    rc = model.lib.plbm_nn_mse(pred.data_ptr(), state["targets"].data_ptr(), state["masks"].data_ptr(),
                               state["grad"].data_ptr(), state["loss"].data_ptr(), n * hh * ww, 3,
                               1.0 / state["count"], model._stream())
    if rc != 0:
        raise RuntimeError(f"plbm_nn_mse failed ({rc})")
    model.zero_grad()
    model.backward(state["grad"])
    model.adam(lr=1e-3)
    return {"pred": pred, "loss": state["loss"], "gradients": model.params.g, "weights": model.params.w}


# ---- what a pass cannot do without ------------------------------------------------------------


def _nn_flops(n, h, w):
    f = 0.0
    for lvl in range(5):
        for ci, co in ENC[2 * lvl:2 * lvl + 2]:
            f += 2.0 * n * (h >> lvl) * (w >> lvl) * 9 * ci * co
    for k, lvl in enumerate((3, 2, 1, 0)):
        for ci, co in DEC[2 * k:2 * k + 2]:
            f += 2.0 * n * (h >> lvl) * (w >> lvl) * 9 * ci * co
    return f + 2.0 * n * h * w * 9 * HEAD[0] * HEAD[1]


def work(case):
    """The state read once and written once, the results (and frames) written once; 97 operations a
    node update (the reference's BGK update); the operator's convolutions, three times for a
    training step."""
    kind = case["kind"]
    if kind in ("nn_forward", "nn_train"):
        weights = sum(9 * ci * co for ci, co in ENC + DEC + [HEAD])
        px = case["n"] * case["h"] * case["w"]
        flops = _nn_flops(case["n"], case["h"], case["w"])
        if kind == "nn_forward":
            return {"bytes": px * (1 + 2 * 3) + 2 * weights, "flops": flops}
        return {"bytes": px * (1 + 2 * 3 + 4 * 3) + 4 * weights * 6, "flops": 3 * flops}
    if kind == "batch":
        nodes = case["domains"] * (0.5 * (case["lo"] + case["hi"])) ** 2
    else:
        nodes = case["w"] * case["h"]
    frames = case["steps"] // case["frame"] if kind == "run" else 1
    return {"bytes": nodes * (18 * SIZES[case["prec"]] + frames * 8 * (3 if kind == "batch" else 4)),
            "flops": 97.0 * nodes * case["steps"]}


# ---- the same results in 64 bits, plain torch ------------------------------------------------------

_W = [1 / 36, 1 / 9, 1 / 36, 1 / 9, 4 / 9, 1 / 9, 1 / 36, 1 / 9, 1 / 36]


def _scenario_circle(w, h):
    xx, vv = w + 2, h + 2
    mx, my, r = 2 * xx // 10, vv // 2, vv // 5
    y, x = np.arange(1, h + 1)[:, None], np.arange(1, w + 1)[None, :]
    m = ((x - mx) ** 2 + (y - my) ** 2 <= r * r) & (abs(x - mx) <= r) & (abs(y - my) <= r)
    m = m.astype(np.int8)
    m[0, :] = 1
    m[h - 1, :] = 1
    return m


def _lbm_exact(mask, tau, rin, rout, steps, outlet_constant=False, before=0):
    """D2Q9 BGK from rest in float64: pull streaming, half-way bounce-back, the density outlet.
    Returns rho, jx, jy, |j| after `steps`, and jx, jy after `before` steps."""
    solid = torch.from_numpy(mask.astype(bool)).cuda()
    h, w = mask.shape
    cx, cy = [d % 3 - 1 for d in range(9)], [d // 3 - 1 for d in range(9)]
    pad = torch.ones((h + 2, w + 2), dtype=torch.bool, device="cuda") & False
    pad[1:h + 1, 1:w + 1] = solid
    bounce = [pad[1 - cy[d]:1 - cy[d] + h, 1 - cx[d]:1 - cx[d] + w].clone() for d in range(9)]
    f = torch.empty((9, h + 2, w + 2), dtype=torch.float64, device="cuda")   # with the ghost layer
    for d in range(9):
        f[d] = _W[d]
        f[d, 1:h + 1, 0] = _W[d] * rin
        f[d, 1:h + 1, w + 1] = _W[d] * rout
    fluid = ~solid
    border = fluid[1:h - 1, w - 1]
    jyo = torch.zeros(h, dtype=torch.float64, device="cuda")
    om = 1.0 / tau
    early = None
    for step in range(steps):
        p = []
        for d in range(9):
            v = f[d, 1 - cy[d]:1 - cy[d] + h, 1 - cx[d]:1 - cx[d] + w]
            p.append(v.clone() if d == 4 else torch.where(bounce[d], f[8 - d, 1:h + 1, 1:w + 1], v))
        if not outlet_constant:
            b = [v[1:h - 1, w - 1] for v in p]
            xv = b[1] + b[4] + b[7] + 2.0 * (b[8] + b[5] + b[2]) - rout
            hd, hy = 0.5 * (b[1] - b[7]), 0.5 * jyo[1:h - 1]
            new = {0: b[8] - hd - xv / 6 - hy, 3: b[5] - xv * 2 / 3, 6: b[2] + hd - xv / 6 + hy}
            for d, v in new.items():
                p[d][1:h - 1, w - 1] = torch.where(border, v, p[d][1:h - 1, w - 1])
        right, left = p[2] + p[5] + p[8], p[0] + p[3] + p[6]
        rho = left + right + p[1] + p[4] + p[7]
        jx, jy = right - left, p[6] + p[7] + p[8] - p[0] - p[1] - p[2]
        usq = jx * jx + jy * jy
        rest = rho - 1.5 * usq
        for d in range(9):
            cu = cx[d] * jx + cy[d] * jy
            feq = _W[d] * (rest + 3.0 * cu + 4.5 * cu * cu) if d != 4 else _W[4] * rest
            inner = f[d, 1:h + 1, 1:w + 1]
            inner.copy_(torch.where(fluid, p[d] - om * (p[d] - feq), inner))
        if w >= 2:
            jyo = torch.where(fluid[:, w - 2], jy[:, w - 2], jyo)
        if step + 1 == before:
            early = (torch.where(fluid, jx, 0.0), torch.where(fluid, jy, 0.0))
    out = [torch.where(fluid, rho, -1.0)] + [torch.where(fluid, v, 0.0) for v in (jx, jy, usq.sqrt())]
    return [v.reshape(-1) for v in out], early


def _conv(x, wt, bias):
    """3x3 convolution, NHWC, zero padding, weights [co][(ky * 3 + kx) * ci + c]."""
    n, h, w, ci = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    y = bias.expand(n * h * w, -1)
    for t in range(9):
        ky, kx = divmod(t, 3)
        y = y + xp[:, ky:ky + h, kx:kx + w].reshape(-1, ci) @ wt[:, t * ci:(t + 1) * ci].T
    return y.reshape(n, h, w, -1)


def _nn_exact(case, seed):
    masks, feats, targets = _nn_inputs(case, seed)
    r = np.random.default_rng(seed)
    n, h, w = case["n"], case["h"], case["w"]
    params = []
    for ci, co in ENC + DEC + [HEAD]:
        wt = (r.standard_normal((co, 9 * ci)) * np.sqrt(2.0 / (9 * ci))).astype(np.float32)
        wt = torch.from_numpy(wt).cuda().to(torch.bfloat16).double().requires_grad_(case["kind"] == "nn_train")
        params.append((wt, torch.zeros(co, dtype=torch.float64, device="cuda", requires_grad=case["kind"] == "nn_train")))
    x = torch.zeros((n, h, w, 4), dtype=torch.float64, device="cuda")
    m = torch.from_numpy(masks).cuda()
    x[..., 0] = m.double()
    x[..., 1:] = torch.from_numpy(feats).cuda().to(torch.bfloat16).double()[:, None, None, :]
    it = iter(params)

    def layer(v, relu=True):
        v = _conv(v, *next(it))
        return v.relu() if relu else v

    skips, cur = [], x
    for lvl in range(5):
        cur = layer(layer(cur))
        skips.append(cur)
        if lvl < 4:
            k = cur.shape
            cur = cur.reshape(k[0], k[1] // 2, 2, k[2] // 2, 2, k[3]).mean(dim=(2, 4))
    for lvl in (3, 2, 1, 0):
        cur = layer(cur.repeat_interleave(2, dim=1).repeat_interleave(2, dim=2))
        cur = layer(cur + skips[lvl])
    pred = layer(cur, relu=False)
    if case["kind"] == "nn_forward":
        return pred.detach()
    fl = (m == 0)[..., None]
    loss = (torch.where(fl, pred - torch.from_numpy(targets).cuda().double(), 0.0) ** 2).sum() / (float((masks == 0).sum()) * 3)
    loss.backward()
    grads = []
    for wt, b in params:      # each segment starts on a multiple of 128 values
        for g in (wt.grad, b.grad):
            g = g.reshape(-1)
            grads.append(torch.nn.functional.pad(g, (0, -g.numel() % 128)))
    return {"pred": pred.detach(), "loss": loss.detach().reshape(1), "gradients": torch.cat(grads), "weights": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("nn_forward", "nn_train"):
        return _nn_exact(case, seed)
    if kind == "batch":
        out = []
        for d in _batch_domains(case, seed):
            fields, _ = _lbm_exact(d["mask"], d["relaxation_time"], d["inlet_density"], 1.0, case["steps"])
            out.append(fields[:3])
        return out
    w, h = case["w"], case["h"]
    tau, rin = _physics(case, seed)
    mask = _mask(case, seed)
    if mask is None:
        mask = _scenario_circle(w, h)
    # the buffered algorithms keep the outlet ghost constant where the last column starts a subdomain
    side = {"npol": 32, "nsol": 30}.get(case["alg"])
    constant = side is not None and (w - 1) % side == 0
    fields, early = _lbm_exact(mask, tau, rin, 1.0, case["steps"], constant,
                               case["steps"] - case["k"] if kind == "steady" else 0)
    out = dict(zip(("rho", "jx", "jy", "jabs"), fields))
    if kind == "steady":
        jx, jy = fields[1].reshape(h, w), fields[2].reshape(h, w)
        num = ((jx - early[0]) ** 2).sum() + ((jy - early[1]) ** 2).sum()
        out |= {"steps": None, "residual": float((num / ((jx ** 2).sum() + (jy ** 2).sum())).sqrt() / case["k"])}
    return out
