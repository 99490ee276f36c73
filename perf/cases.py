"""Timed cases of the absorption-correction framework.

Every case is a call that a user of the library makes, through its public
entry points, on seeded synthetic inputs: segmented volumes painted with the
label recipe of ``anacor_public_gb300.synth`` (crystal ellipsoid, liquor
shell, torus loop, two bubbles; here with torch on the GPU, so that a fresh
volume costs milliseconds), some of them with the loop's stem running to the
volume's wall, as a mounted sample's does.

kind        the call
----        --------
dropin      ``worker.ray_tracing_overall``: host arrays in, host A_h out, as
            AnACor's worker process calls the library
rescan      a resident ``tracer.Plan`` that gets another set of reflections
            (``set_reflections`` + ``run`` + ``result``)
resident    a resident plan with its reflections in place (``run`` + ``result``)
batch       ``tracer.Batch``: several samples in one captured launch, replayed
bisection   ``tracer.bisection``: the iterative-bisection mode
gridbuild   ``gridding.GriddingMap.build`` and nearest lookups on the new map
gridlookup  ``gridding.GriddingMap.interpolate`` on a map that is kept
predict     ``surrogate.Surrogate.predict_device`` on device rows
train       ``surrogate.Surrogate.train``: Adam steps on a training set
"""
import math
import os

import numpy as np
import torch

from anacor_public_gb300 import gridding, surrogate, tracer, worker

VACUUM, LIQUOR, LOOP, CRYSTAL, BUBBLE = 0, 1, 2, 3, 4
MU = (0.010, 0.007, 0.012, 0.0)   # liquor, loop, crystal, bubble, per um
XRAY = (-1.0, 0.0, 0.0)
AXIS = (0.0, 1.0, 0.0)
WIDTH, FEATURES, DEPTH = 256, 64, 4


def listed():
    return [
        # the smallest call: one worker's last few reflections of a coarse volume; launches and host set-up
        dict(name="dropin_tiny", kind="dropin", z=64, y=56, x=61, stride=2, refl=4, stem=False),
        # a small sample with every crystal voxel, as the quick-look run of a new data set
        dict(name="dropin_small", kind="dropin", z=96, y=96, x=96, stride=1, refl=300, stem=False),
        # the standard beamline sample and its whole data set, from host arrays
        dict(name="dropin_beamline", kind="dropin", z=512, y=512, x=400, stride=4, refl=20000, stem=False),
        # another sweep of a mounted sample that is kept on the GPU; odd sizes, stem to the wall
        dict(name="rescan_mounted", kind="rescan", z=301, y=347, x=263, stride=5, refl=3001, stem=True),
        # a high-resolution volume with strong absorbers, every crystal voxel, a few reflections
        dict(name="resident_highabs", kind="resident", z=1024, y=1024, x=800, stride=1, refl=32, stem=False),
        # several samples of a session corrected together
        dict(name="batch_session", kind="batch", samples=6, dim_lo=128, dim_hi=420, refl_lo=500, refl_hi=6000),
        # the bisection mode on a mid-size sample
        dict(name="bisection_mid", kind="bisection", z=288, y=240, x=257, stride=3, refl=701, cls=4),
        # the absorption map at its default grid, then the lookups of a first sweep
        dict(name="gridbuild_default", kind="gridbuild", z=512, y=512, x=400, stride=8, theta=360, phi=180, refl=2000),
        # bilinear lookups of a whole data set on a map that is kept
        dict(name="gridlookup_linear", kind="gridlookup", z=256, y=256, x=250, stride=6, theta=360, phi=180,
             refl=20000, linear=True),
        # the surrogate on a million reflections, and on a handful
        dict(name="predict_million", kind="predict", rows=1000000, members=4),
        dict(name="predict_few", kind="predict", rows=1000, members=4),
        # training at the default batch and schedule
        dict(name="train_default", kind="train", steps=24, batch=4096, members=4, data=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    a = _log(rng, lo, hi)
    return [max(lo, min(hi, int(a * rng.uniform(0.75, 1.3)))) for _ in range(3)]


def _stride_for(dims, voxels):
    """Stride that leaves about `voxels` crystal voxels of the recipe's ellipsoid."""
    n = 4.0 / 3.0 * math.pi * 20 * 14 * 10 * (min(dims) / 96.0) ** 3
    return max(1, int(round((n / voxels) ** (1.0 / 3.0))))


def draw(rng):
    kind = rng.choice(["dropin", "dropin", "rescan", "resident", "batch", "bisection", "gridbuild", "gridlookup",
                       "predict", "predict", "train"])
    if kind in ("dropin", "rescan", "resident"):
        z, y, x = _dims(rng, 60, 640)
        refl = _log(rng, 3, 20000)
        stride = _stride_for((z, y, x), max(300, min(40000, int(rng.uniform(2e7, 2e8) / refl))))
        return dict(kind=kind, z=z, y=y, x=x, stride=stride, refl=refl, stem=rng.random() < 0.5)
    if kind == "batch":
        lo = _log(rng, 96, 200)
        return dict(kind=kind, samples=rng.randint(2, 8), dim_lo=lo, dim_hi=2 * lo, refl_lo=rng.randint(100, 900),
                    refl_hi=rng.randint(1000, 5000))
    if kind == "bisection":
        z, y, x = _dims(rng, 64, 400)
        refl = _log(rng, 16, 1500)
        return dict(kind=kind, z=z, y=y, x=x, stride=_stride_for((z, y, x), max(300, int(rng.uniform(1e6, 1e7) / refl))),
                    refl=refl, cls=rng.choice([3, 4]))
    if kind in ("gridbuild", "gridlookup"):
        z, y, x = _dims(rng, 96, 400)
        theta, phi = rng.choice([(360, 180), (180, 90), (121, 67), (240, 122)])
        d = dict(kind=kind, z=z, y=y, x=x, stride=_stride_for((z, y, x), rng.randint(300, 3000)), theta=theta, phi=phi,
                 refl=_log(rng, 100, 20000))
        if kind == "gridlookup":
            d["linear"] = rng.random() < 0.5
        return d
    if kind == "predict":
        return dict(kind=kind, rows=_log(rng, 100, 1000000), members=rng.choice([1, 2, 3, 4, 4, 4, 5, 8]))
    return dict(kind=kind, steps=rng.randint(4, 24), batch=1024 * rng.randint(1, 8), members=rng.randint(2, 5),
                data=_log(rng, 5000, 100000))


# ------------------------------------------------------------------ inputs

def _euler(a, b, c):
    rz = lambda t: np.array([[math.cos(t), -math.sin(t), 0], [math.sin(t), math.cos(t), 0], [0, 0, 1]])  # noqa: E731
    ry = np.array([[math.cos(b), 0, math.sin(b)], [0, 1, 0], [-math.sin(b), 0, math.cos(b)]])
    return rz(a) @ ry @ rz(c)


def _paint(dims, rng, stem):
    """int8 [Z][Y][X] label volume on the GPU; lengths scale with the smallest axis."""
    Z, Y, X = dims
    sc = min(dims) / 96.0
    semi = np.array([20.0, 14.0, 10.0]) * sc
    rot = _euler(*rng.uniform(0.0, 2.0 * math.pi, 3))
    normal = rng.normal(size=3)
    normal /= np.linalg.norm(normal)
    centre = [(n - 1) / 2.0 for n in dims]
    balls = []
    for _ in range(2):   # bubbles in the middle of the liquor shell
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        balls.append(rot @ (u * (semi + 3.0 * sc)))
    vol = torch.zeros((Z, Y, X), dtype=torch.int8, device="cuda")
    yy = (torch.arange(Y, device="cuda", dtype=torch.float32) - centre[1])[None, :, None]
    xx = (torch.arange(X, device="cuda", dtype=torch.float32) - centre[2])[None, None, :]
    slab = max(1, int(6e7) // (Y * X))
    for z0 in range(0, Z, slab):
        zz = (torch.arange(z0, min(Z, z0 + slab), device="cuda", dtype=torch.float32) - centre[0])[:, None, None]
        q = [float(rot[0, k]) * zz + float(rot[1, k]) * yy + float(rot[2, k]) * xx for k in range(3)]
        cry = sum((q[k] / float(semi[k])) ** 2 for k in range(3)) <= 1.0
        liq = sum((q[k] / float(semi[k] + 6.0 * sc)) ** 2 for k in range(3)) <= 1.0
        h = float(normal[0]) * zz + float(normal[1]) * yy + float(normal[2]) * xx
        rho = torch.sqrt(torch.clamp(zz * zz + yy * yy + xx * xx - h * h, min=0.0))
        loop = (rho - 30.0 * sc) ** 2 + h * h <= (3.0 * sc) ** 2
        if stem:
            loop = loop | ((zz * zz + xx * xx <= (4.0 * sc) ** 2) & (yy < -28.0 * sc))
        b = vol[z0:z0 + slab]
        b[loop & ~liq] = LOOP
        b[liq] = LIQUOR
        for p in balls:
            b[((zz - p[0]) ** 2 + (yy - p[1]) ** 2 + (xx - p[2]) ** 2 <= (3.0 * sc) ** 2) & liq & ~cry] = BUBBLE
        b[cry] = CRYSTAL
    return vol


def _crystal(vol, stride):
    """(z, y, x) of the crystal voxels whose indices are multiples of the stride, int64 on the host."""
    c = torch.nonzero(vol[::stride, ::stride, ::stride] == CRYSTAL) * stride
    return np.ascontiguousarray(c.cpu().numpy().astype(np.int64))


def _reflections(n, rng):
    """omega over the turn; s1 at 2theta in [5, 120] degrees from the beam, any azimuth."""
    omega = rng.uniform(0.0, 2.0 * math.pi, n)
    tth, az = np.deg2rad(rng.uniform(5.0, 120.0, n)), rng.uniform(0.0, 2.0 * math.pi, n)
    s1 = np.stack([-np.cos(tth), np.sin(tth) * np.cos(az), np.sin(tth) * np.sin(az)], 1)
    return np.ascontiguousarray(s1), omega


def _sample(dims, stride, refl, stem, rng, mu_factor=1.0):
    vol = _paint(dims, rng, stem)
    s1, omega = _reflections(refl, rng)
    return dict(label=vol.cpu().numpy(), coords=_crystal(vol, stride), s1=s1, omega=omega, xray=np.array(XRAY),
                axis=np.array(AXIS), F=np.ascontiguousarray(_euler(*rng.uniform(0.0, 2.0 * math.pi, 3)).reshape(-1)),
                voxel=np.array([0.3, 0.3, 0.3]), mu=np.array(MU) * mu_factor * rng.uniform(0.8, 1.2))


def _mu_factor(case):
    return 5.0 if case["kind"] == "resident" else 1.0   # strong absorbers in the high-resolution case


def _samples(case, seed):
    rng = np.random.default_rng([seed, 11])
    if case["kind"] != "batch":
        return [_sample((case["z"], case["y"], case["x"]), case["stride"], case["refl"], case.get("stem", False), rng,
                        _mu_factor(case))]
    out = []
    sizes = np.random.default_rng([case["samples"], case["dim_lo"], case["refl_lo"]])   # of the case, not of the seed
    for k in range(case["samples"]):
        dims = tuple(int(d) for d in np.exp(sizes.uniform(math.log(case["dim_lo"]), math.log(case["dim_hi"]), 3)))
        n = int(math.exp(sizes.uniform(math.log(case["refl_lo"]), math.log(case["refl_hi"]))))
        out.append(_sample(dims, _stride_for(dims, 6000), n, k % 2 == 1, rng))
    return out


def _x7(n, rng):
    """Network inputs: omega / 2pi and two unit vectors, as ``surrogate.inputs`` gives them."""
    a, b = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    return np.concatenate([rng.uniform(0.0, 1.0, (n, 1)), a, b], 1).astype(np.float32)


def _weights(members, rng):
    """Parameters [members][214280] of the layout W1 b1 .. W4 b4 w5 b5 (padded): He weights, small biases."""
    p = np.zeros((members, 214280), dtype=np.float32)
    for m in range(members):
        o = 0
        for layer in range(DEPTH):
            k = FEATURES if layer == 0 else WIDTH
            p[m, o:o + WIDTH * k] = rng.normal(size=WIDTH * k) * math.sqrt(2.0 / k)
            p[m, o + WIDTH * k:o + WIDTH * k + WIDTH] = rng.normal(size=WIDTH) * 0.05
            o += WIDTH * k + WIDTH
        p[m, o:o + WIDTH] = rng.normal(size=WIDTH) / 16.0
        p[m, o + WIDTH] = 0.1 * rng.normal()
    return p


def _fourier(rng):
    b = rng.normal(size=(32, 7)) * 0.35
    b[:, 0] = np.rint(b[:, 0])
    return b.astype(np.float32)


def _network(case, seed):
    rng = np.random.default_rng([seed, 23])
    return _weights(case["members"], rng), _fourier(rng), _x7(case["rows"], rng)


SCALE = (-1.2, 0.25)   # mean and standard deviation of log A_h


class _Grid:
    """A plan and its map, released together."""

    def __init__(self, s, case):
        self.plan = tracer.Plan(s["label"], s["coords"], s["voxel"], s["mu"])
        self.map = gridding.GriddingMap(self.plan, case["theta"], case["phi"], method=2)

    def __del__(self):
        self.map.close()
        self.plan.close()


class _Batch:
    """The plans of a session, their captured launch and its stream."""

    def __init__(self, samples):
        self.plans = []
        for s in samples:
            p = tracer.Plan(s["label"], s["coords"], s["voxel"], s["mu"])
            p.set_reflections(s["s1"], s["omega"], s["xray"], s["axis"], s["F"])
            p.configure(12, 512, 1)
            self.plans.append(p)
        self.torch_stream = torch.cuda.Stream()
        self.stream = self.torch_stream.cuda_stream
        self.batch = tracer.Batch(self.plans)
        self.batch.configure(12)
        self.batch.capture(self.stream)

    def __del__(self):
        self.batch.close()
        for p in self.plans:
            p.close()


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind == "predict":
        params, fourier, x7 = _network(case, seed)
        m = surrogate.Surrogate(members=case["members"], seed=1)
        m.set_params(params)
        m.set_fourier(fourier)
        m.scale = SCALE
        n = case["rows"]
        st.update(model=m, x7=torch.from_numpy(x7).cuda(), mean=torch.empty(n, device="cuda"),
                  spread=torch.empty(n, device="cuda"))
        return st
    if kind == "train":
        rng = np.random.default_rng([seed, 31])
        m = surrogate.Surrogate(members=case["members"], seed=int(rng.integers(1 << 30)), fourier_scale=0.35)
        x7 = _x7(case["data"], rng)
        w = rng.normal(size=(7, 4)) * 0.8
        log_ah = -1.2 + 0.25 * np.sin(x7.astype(np.float64) @ w).sum(1)   # smooth in the directions, as log A_h is
        m.set_data(x7, log_ah)
        st.update(model=m)
        return st
    samples = _samples(case, seed)
    s = samples[0]
    if kind == "batch":
        st.update(batch=_Batch(samples))
        return st
    if kind in ("dropin", "bisection"):
        st.update(s=s)
        return st
    if kind in ("rescan", "resident"):
        p = tracer.Plan(s["label"], s["coords"], s["voxel"], s["mu"])
        p.configure(12, 1024, 1)
        st.update(plan=p)
        if kind == "rescan":
            st.update(s={k: s[k] for k in ("s1", "omega", "xray", "axis", "F")})
        else:
            p.set_reflections(s["s1"], s["omega"], s["xray"], s["axis"], s["F"])
        return st
    g = _Grid(s, case)
    if kind == "gridlookup":
        g.map.build()
    st.update(grid=g, s={k: s[k] for k in ("s1", "omega", "xray", "axis", "F")})
    return st


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "dropin":
        s = state["s"]
        return {"ah": worker.ray_tracing_overall(s["label"], s["coords"], s["s1"], s["omega"], s["xray"], s["axis"],
                                                 s["F"], s["voxel"], s["mu"], num_workers=os.cpu_count() or 1)}
    if kind == "rescan":
        s, p = state["s"], state["plan"]
        p.set_reflections(s["s1"], s["omega"], s["xray"], s["axis"], s["F"])
        p.run()
        return {"ah": p.result()}
    if kind == "resident":
        state["plan"].run()
        return {"ah": state["plan"].result()}
    if kind == "batch":
        b = state["batch"]
        b.batch.replay(b.stream)
        b.batch.wait(b.stream)
        return {"ah": b.batch.results(b.stream)}
    if kind == "bisection":
        s = state["s"]
        return {"ah": tracer.bisection(s["label"], s["coords"], s["s1"], s["omega"], s["xray"], s["axis"], s["F"],
                                       s["voxel"], s["mu"], num_cls=case["cls"])}
    if kind == "gridbuild":
        s, g = state["s"], state["grid"].map
        g.build()
        return {"ah": g.interpolate(s["s1"], s["omega"], s["xray"], s["axis"], s["F"], method="nearest")}
    if kind == "gridlookup":
        s, g = state["s"], state["grid"].map
        return {"ah": g.interpolate(s["s1"], s["omega"], s["xray"], s["axis"], s["F"],
                                    method="linear" if case["linear"] else "nearest")}
    if kind == "predict":
        state["model"].predict_device(state["x7"].data_ptr(), case["rows"], state["mean"].data_ptr(),
                                      state["spread"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"mean": state["mean"], "spread": state["spread"]}
    loss = state["model"].train(case["steps"], batch=case["batch"], total_steps=20000)
    return {"loss": loss, "params": state["model"].get_params()}


# -------------------------------------------------------------------- work

def _voxel_count(case):
    """Crystal voxels on the lattice, from the ellipsoid's volume."""
    n = 4.0 / 3.0 * math.pi * 20 * 14 * 10 * (min(case["z"], case["y"], case["x"]) / 96.0) ** 3
    return n / case["stride"] ** 3


#: Arithmetic a leg cannot do without: three exit distances, one point of each of about three material
#: boundaries (a multiply-add per axis), the total length (three products, a root), a term per segment and the
#: exponent's share.
LEG_FLOPS = 60.0


def work(case):
    kind = case["kind"]
    if kind == "predict":
        n = case["rows"]
        return {"bytes": n * (28.0 + 8.0) + case["members"] * 214280 * 4.0,
                "flops": 2.0 * n * case["members"] * (FEATURES * WIDTH + 3 * WIDTH * WIDTH + WIDTH)}
    if kind == "train":
        # a step reads its batch, reads and writes the parameters and both Adam moments
        per = case["members"] * (214280 * 24.0 + case["batch"] * (FEATURES * 2.0 + 4.0))
        return {"bytes": case["steps"] * per,
                "flops": case["steps"] * 6.0 * case["batch"] * case["members"] * (FEATURES * WIDTH + 3 * WIDTH * WIDTH + WIDTH)}
    if kind == "batch":
        b = f = 0.0
        sizes = np.random.default_rng([case["samples"], case["dim_lo"], case["refl_lo"]])
        for _ in range(case["samples"]):
            dims = tuple(int(d) for d in np.exp(sizes.uniform(math.log(case["dim_lo"]), math.log(case["dim_hi"]), 3)))
            n = int(math.exp(sizes.uniform(math.log(case["refl_lo"]), math.log(case["refl_hi"]))))
            nv = _voxel_count(dict(z=dims[0], y=dims[1], x=dims[2], stride=_stride_for(dims, 6000)))
            b += dims[0] * dims[1] * dims[2] + 24.0 * nv + 40.0 * n
            f += 2.0 * LEG_FLOPS * nv * n
        return {"bytes": b, "flops": f}
    nv, vol, n = _voxel_count(case), float(case["z"] * case["y"] * case["x"]), case["refl"]
    if kind == "gridlookup":
        rows = 8.0 if case["linear"] else 2.0   # map rows of a reflection
        return {"bytes": rows * 4.0 * nv * n + 40.0 * n, "flops": 10.0 * nv * n}
    if kind == "gridbuild":
        dirs = case["theta"] * case["phi"]
        return {"bytes": vol + 24.0 * nv + 4.0 * nv * dirs + 8.0 * nv * n, "flops": LEG_FLOPS * nv * dirs + 4.0 * nv * n}
    return {"bytes": vol + 24.0 * nv + 40.0 * n, "flops": 2.0 * LEG_FLOPS * nv * n}


# ------------------------------------------------------------------- exact
#
# The same quantities in 64 bits with plain torch: the march visits every increment of every leg.

FACE_ORDER = ((2, 0, 6), (1, 0, 4), (0, 0, 2), (2, 1, 1), (1, 1, 5), (0, 1, 3))   # axis, far side?, face code


def _rotated(s, i):
    x, y, z = s["axis"]
    c, sn = math.cos(s["omega"][i]), math.sin(s["omega"][i])
    k = 1 - c
    R = np.array([[c + x * x * k, x * y * k - z * sn, y * sn + x * z * k],
                  [z * sn + x * y * k, c + y * y * k, -x * sn + y * z * k],
                  [-y * sn + x * z * k, x * sn + y * z * k, c + z * z * k]])
    T = (R @ np.asarray(s["F"]).reshape(3, 3)).T
    return T @ s["xray"], T @ s["s1"][i]


def _angles(v, incident):
    a, b, c = (-v if incident else v)
    r = math.sqrt(a * a + b * b)
    if b == 0:
        return math.atan(-c / (-r + 0.001)), math.atan(-a / (b + 0.001))
    if b < 0:
        return math.atan(-c / r), math.atan(-a / b)
    t = math.atan(-c / r)
    return (math.pi - t if c < 0 else -math.pi - t), -math.atan(a / b)


def _face_rules(th, ph):
    """(steps per increment (z, y, x), C rounding, count kind) of each exit face 1..6; a face that the angles
    exclude keeps zeros."""
    with np.errstate(divide="ignore", invalid="ignore"):   # a face that such a ray never leaves through may divide by 0
        return _face_rules_of(np.float64(th), np.float64(ph))


def _face_rules_of(th, ph):
    q = np.zeros((7, 3))
    rnd = np.zeros(7, dtype=bool)
    at, ap, up = abs(th), abs(ph), th > 0
    near = at < np.pi / 2
    if at <= np.pi / 2:
        q[6] = (np.tan(ph), -np.tan(th) / np.cos(ph), -1)
    if at >= np.pi / 2:
        q[1] = (-np.tan(ph), -np.tan(np.pi - th) / np.cos(ap), 1)
    if near:
        zx, zy = -1 / np.tan(ap), -np.tan(th) / np.sin(ap)
        if ph < 0:
            q[2] = (-1, zy, zx)
        else:
            q[3] = (1, zy, zx)
    else:
        zx, zy = 1 / np.tan(ap), -np.tan(np.pi - th) / np.sin(ap)
        if ph > 0:
            q[2] = (-1, zy, zx)
        else:
            q[3] = (1, zy, zx)
    if near:
        yz, yx = np.sin(ph) / np.tan(at), -np.cos(ap) / np.tan(at)
    else:
        yz, yx = -np.sin(ph) / np.tan(np.pi - at), np.cos(ap) / np.tan(np.pi - at)
    if up:
        q[4] = (yz, -1, yx)
    else:
        q[5] = (yz, 1, yx)
    rnd[[6, 2, 3, 1]] = not up
    rnd[5] = True
    return q, rnd, near


def _exit_faces(v, incident, c, dims):
    d = np.array([v[0], v[2], v[1]])   # z, y, x components
    t = []
    for axis, far, _ in FACE_ORDER:
        u = (float(dims[axis] if far else 0) - c[:, axis].double()) / (float(d[axis]) + 0.0)
        t.append(-u if incident else u)
    t = torch.stack(t, 1)
    t = torch.where(t >= 0, t, torch.full_like(t, math.inf))
    best = torch.argmin(t, 1)
    return torch.tensor([f for _, _, f in FACE_ORDER], device=c.device)[best]


def _points(c, i, q, rnd):
    """Rounded, unclamped positions c + i q; i broadcasts over the last axis."""
    v = c.double()[:, None, :] + i[..., None].double() * q[:, None, :]
    return torch.where(rnd[:, None, None], torch.trunc(v + torch.copysign(torch.full_like(v, 0.5), v)), torch.floor(v))


def _leg(vol, dims, c, v, incident, voxel):
    """Lengths [n][4] (liquor, loop, crystal, bubble) of one leg of every voxel."""
    th, ph = _angles(v, incident)
    qt, rt, near = _face_rules(th, ph)
    dev = c.device
    face = _exit_faces(v, incident, c, dims)
    q, rnd = torch.tensor(qt, device=dev)[face], torch.tensor(rt, device=dev)[face]
    z, y, x = c[:, 0], c[:, 1], c[:, 2]
    more = 0 if near else 1
    steps = torch.stack([z, dims[2] - x, z + 1, dims[0] - z + more, y + 1, dims[1] - y + more, x + 1], 1).gather(
        1, face[:, None])[:, 0]
    top = torch.tensor(dims, device=dev, dtype=torch.float64) - 1
    flat = vol.reshape(-1)
    count = torch.zeros((len(c), 5), dtype=torch.int64, device=dev)
    length = torch.zeros(len(c), dtype=torch.int64, device=dev)
    idx = torch.arange(len(c), device=dev)   # legs that still run
    i0, chunk = 0, 32
    while len(idx):
        i = torch.arange(i0, i0 + chunk, device=dev)[None, :]
        p = torch.minimum(_points(c[idx], i, q[idx], rnd[idx]).clamp_(min=0.0), top).long()
        lab = flat[(p[..., 0] * dims[1] + p[..., 1]) * dims[2] + p[..., 2]].long()
        alive = torch.cumprod(((lab != VACUUM) & (i < steps[idx][:, None])).to(torch.int8), 1).bool()
        length[idx] += alive.sum(1)
        count[idx] += torch.stack([(alive & (lab == k)).sum(1) for k in range(5)], 1)
        idx = idx[alive[:, -1]]
        i0 += chunk
    last = torch.clamp(length - 1, min=0)
    p = torch.minimum(_points(c, last[:, None], q, rnd).clamp_(min=0.0), top)[:, 0]
    total = ((p - c.double()) * torch.tensor(voxel, device=dev)).square().sum(1).sqrt()
    scale = torch.where(last > 0, total / torch.clamp(last, min=1).double(), torch.zeros_like(total))
    return count[:, 1:].double() * scale[:, None]


def _bisect(longest, shortest, c, q, vol, dims, inward, code):
    """The boundary search of every ray: (point, parameter)."""
    longest, shortest = longest.clone(), shortest.clone()
    mid = (longest + shortest) / 2
    flat = vol.reshape(-1)
    while True:
        on = longest - shortest > 1.0
        if not bool(on.any()):
            break
        m = (longest + shortest) / 2
        p = torch.floor(c.double() + m[:, None] * q).long()
        for a in range(3):
            p[:, a].clamp_(0, dims[a] - 1)
        hit = flat[(p[:, 0] * dims[1] + p[:, 1]) * dims[2] + p[:, 2]] == code
        far = hit if inward else ~hit
        mid = torch.where(on, m, mid)
        longest = torch.where(on & far, m, longest)
        shortest = torch.where(on & ~far, m, shortest)
    return torch.floor(c.double() + torch.floor(mid)[:, None] * q), mid


def _bisection_leg(vol, dims, c, v, incident, voxel, cls):
    th, ph = _angles(v, incident)
    face = _exit_faces(v, incident, c, dims)
    q = torch.tensor(_face_rules(th, ph)[0], device=c.device)[face]
    z, y, x = c[:, 0], c[:, 1], c[:, 2]
    reach = torch.stack([z, dims[2] - 1 - x, z, dims[0] - 1 - z, y, dims[1] - 1 - y, x], 1).gather(
        1, face[:, None])[:, 0].double()
    zero = torch.zeros_like(reach)
    vox = torch.tensor(voxel, device=c.device)
    dist = lambda a, b: ((a - b) * vox).square().sum(1).sqrt()  # noqa: E731
    l1 = lambda a, b: (a - b).abs().sum(1)                      # noqa: E731
    start = c.double()
    air, m_air = _bisect(reach, zero, c, q, vol, dims, True, VACUUM)
    cr, m_cr = _bisect(m_air, zero, c, q, vol, dims, False, CRYSTAL)
    li, m_li = _bisect(m_air, m_cr, c, q, vol, dims, True, LOOP)
    seen = l1(li, air) / 3 > 1
    lo, _ = _bisect(m_air, m_li, c, q, vol, dims, False, LOOP)
    end = seen & (l1(li, lo) / 3 <= 2)
    loop = seen & ~end
    bub = torch.zeros_like(loop)
    bi = bo = air
    if cls > 3:
        bi, m_bi = _bisect(m_air, m_cr, c, q, vol, dims, True, BUBBLE)
        bo, _ = _bisect(m_air, m_bi, c, q, vol, dims, False, BUBBLE)
        bub = ~end & (l1(bi, air) > 1) & (l1(bi, bo) / 3 > 2)
    # the lengths are read by the number of points: five count a pair as loop, seven the second pair as bubble
    lo_l = torch.where(loop & ~bub, dist(li, lo), torch.where(bub & ~loop, dist(bi, bo), zero))
    bu_l = torch.where(loop & bub, dist(bi, bo), zero)
    total, cr_l = dist(start, air), dist(start, cr)
    return torch.stack([total - lo_l - bu_l - cr_l, lo_l, cr_l, bu_l], 1)


def _traced(s, cls=0):
    dims = s["label"].shape
    vol = torch.from_numpy(s["label"]).cuda()
    c = torch.from_numpy(s["coords"]).cuda()
    mu = torch.from_numpy(s["mu"]).cuda()
    out = []
    for i in range(len(s["omega"])):
        xr, sr = _rotated(s, i)
        legs = [(_bisection_leg(vol, dims, c, v, inc, s["voxel"], cls) if cls else _leg(vol, dims, c, v, inc, s["voxel"]))
                for v, inc in ((xr, True), (sr, False))]
        out.append(torch.exp(-((legs[0] + legs[1]) @ mu)).mean())
    return torch.stack(out).cpu().numpy()


def _axis(n, half):
    pad = int(np.round((n // 6) / 2))
    edge = np.round(half * 7 / 6)
    return pad, np.linspace(-edge, edge, n + 2 * pad, endpoint=False) / 180 * np.pi


def _grid_exact(s, case):
    """Nearest lookups: every reflection's two map rows are marched anew."""
    dims = s["label"].shape
    vol, c = torch.from_numpy(s["label"]).cuda(), torch.from_numpy(s["coords"]).cuda()
    mu = torch.from_numpy(s["mu"]).cuda()
    (tp, ta), (pp, pa) = _axis(case["theta"], 180), _axis(case["phi"], 90)
    tg = np.linspace(-180, 180, case["theta"], endpoint=False) / 180 * np.pi
    pg = np.linspace(-90, 90, case["phi"], endpoint=False) / 180 * np.pi

    def value(v, incident):
        th, ph = _angles(v, incident)
        k = []
        for a, ax, pad, n in ((th, ta, tp, case["theta"]), (ph, pa, pp, case["phi"])):
            i = int((a - ax[0]) / ((ax[-1] - ax[0]) / (len(ax) - 1)))
            k.append((min(max(i, 0), len(ax) - 1) - pad) % n)
        t, p = tg[k[0]], pg[k[1]]
        d = np.array([math.cos(t) * math.sin(p), -math.cos(t) * math.cos(p), -math.sin(t)])
        return _leg(vol, dims, c, d, False, s["voxel"]) @ mu

    out = []
    for i in range(len(s["omega"])):
        xr, sr = _rotated(s, i)
        out.append(torch.exp(-(value(xr, True) + value(sr, False))).mean())
    return torch.stack(out).cpu().numpy()


def _leg_seconds(voxels, dims):
    """Rough time of one `_leg` on this card."""
    return (max(dims) / 96.0 + 1.0) * (40 * 1.2e-5 + voxels * 32 * 400.0 / 3e12)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train" or kind == "gridlookup":
        return None   # the steps amplify rounding; the lookups would need every map row marched
    if kind == "predict":
        params, fourier, x7 = _network(case, seed)
        p = torch.from_numpy(params).cuda().double()
        b = torch.from_numpy(fourier).cuda().double()
        means, spreads = [], []
        for r in range(0, case["rows"], 1 << 17):
            x = torch.from_numpy(x7[r:r + (1 << 17)]).cuda().double()
            f = 2 * math.pi * (x @ b.T)
            f = torch.cat([torch.sin(f), torch.cos(f)], 1)
            ys = []
            for m in range(case["members"]):
                h, o = f, 0
                for layer in range(DEPTH):
                    k = FEATURES if layer == 0 else WIDTH
                    h = h @ p[m, o:o + WIDTH * k].reshape(WIDTH, k).T + p[m, o + WIDTH * k:o + WIDTH * k + WIDTH]
                    h = 0.5 * h * torch.erfc(-h / math.sqrt(2.0))
                    o += WIDTH * k + WIDTH
                ys.append(torch.exp(SCALE[0] + SCALE[1] * (h @ p[m, o:o + WIDTH] + p[m, o + WIDTH])))
            a = torch.stack(ys)
            means.append(a.mean(0))
            spreads.append(a.std(0, unbiased=False) / a.mean(0))
        return {"mean": torch.cat(means), "spread": torch.cat(spreads)}
    if kind == "batch":
        cost = 0.0
    else:
        n, dims = _voxel_count(case), (case["z"], case["y"], case["x"])
        cost = 2 * case["refl"] * (8e-3 if kind == "bisection" else _leg_seconds(n, dims))
    if cost > 16.0:
        return None
    samples = _samples(case, seed)
    if kind == "batch":
        cost = sum(2 * len(s["omega"]) * _leg_seconds(len(s["coords"]), s["label"].shape) for s in samples)
        return {"ah": [_traced(s) for s in samples]} if cost <= 16.0 else None
    if kind == "gridbuild":
        return {"ah": _grid_exact(samples[0], case)}
    return {"ah": _traced(samples[0], case["cls"] if kind == "bisection" else 0)}
