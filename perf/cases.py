"""What a user of this framework has it do, as cases that can be timed and checked.

A case is a survey (mesh, stations, data kind, transform) and one of the ways
an inversion drives it:

  matrix_free  data of one model and the gradient of a misfit, box terms
               recomputed on every call (device buffers)
  subsets      the same over a batch of uneven station subsets in one call
  calculator   the same through the jif3D-shaped host classes and numpy arrays
  setup        a new geometry: first data in FP64, the sensitivity matrix
               built on the device, one batched step with it
  stored       a step of an inversion on a built sensitivity matrix: data of a
               batch of models, weighted misfit, gradients
  refine       a batch of models from the inversion grid to a finer forward
               grid and a batch of gradients back

`listed()` holds one or two sizes of each, from a tutorial-sized call to the
largest survey of jif3d_gb300/workloads.py; `draw()` gives others of the same
ranges.
"""
import math

import numpy as np
import torch

from jif3d_gb300 import capi, gravmag

KINDS = {"scalar": capi.SCALAR, "tensor": capi.TENSOR, "magnetic": capi.MAGNETIC,
         "joint": capi.JOINT, "mag_gradient": capi.MAG_GRADIENT,
         "magnetization": capi.MAGNETIZATION}
RAW = {"scalar": 1, "tensor": 9, "magnetic": 3, "joint": 10, "mag_gradient": 1,
       "magnetization": 3}
# stored rows per station of the device-resident sensitivity
STORED = {"scalar": 1, "tensor": 6, "magnetic": 3, "joint": 7, "mag_gradient": 1,
          "magnetization": 3}
TRANSFORMS = {"none": capi.T_NONE, "ftg_invariant": capi.T_FTG_INVARIANT,
              "total_field": capi.T_TOTAL_FIELD, "tfa": capi.T_TFA}
STORAGES = {"fp32": capi.STORE_FP32, "f16x2": capi.STORE_F16X2}
INC, DEC, FS = math.radians(60.0), math.radians(10.0), 50000.0  # inducing field
GRAV = 6.67428e-11
# typical data and data errors: g_z (m/s^2), FTG (1/s^2), magnetics (nT)
SCALE = {"scalar": 2e-5, "tensor": 2e-8, "joint": 2e-8, "magnetic": 50.0, "mag_gradient": 1e-14,
         "magnetization": 50.0}
SIGMA = {"scalar": 1e-7, "tensor": 1e-9, "joint": 1e-9, "magnetic": 1.0, "mag_gradient": 1e-15,
         "magnetization": 1.0}
# floating-point work of one corner evaluation of a kind's terms and their use
TERM_FLOPS = {"scalar": 110, "tensor": 210, "magnetic": 210, "joint": 225, "mag_gradient": 240,
              "magnetization": 216}


def listed():
    return [
        # a tutorial-sized survey: launches and latency count
        dict(name="gz_tiny", family="matrix_free", kind="scalar", transform="none", nx=12, ny=10,
             nz=6, nst=16, layout="grid", height=1.0, nbg=0, corners="sums"),
        # the plain g_z survey with three background layers, as a program with host arrays calls it
        dict(name="gz_calculator", family="calculator", kind="scalar", transform="none", nx=30,
             ny=30, nz=15, nst=400, layout="grid", height=1.0, nbg=3, corners="sums"),
        # one model of the joint g_z + FTG survey, nothing stored
        dict(name="joint_one_model", family="matrix_free", kind="joint", transform="none", nx=64,
             ny=64, nz=32, nst=1024, layout="grid", height=50.0, nbg=0, corners="sums"),
        # the largest matrix-free survey of the configurations
        dict(name="joint_large", family="matrix_free", kind="joint", transform="none", nx=96,
             ny=96, nz=48, nst=2500, layout="grid", height=1.0, nbg=3, corners="sums"),
        # remanent magnetisation (three cell blocks), odd sizes, scattered stations
        dict(name="magnetization_ragged", family="matrix_free", kind="magnetization",
             transform="none", nx=31, ny=27, nz=15, nst=211, layout="scatter", height=30.0, nbg=0,
             corners="sums"),
        # a mesh whose corners and sizes come as decimals, so that corners are not running sums
        dict(name="ftg_given_corners", family="matrix_free", kind="tensor", transform="none",
             nx=24, ny=21, nz=12, nst=120, layout="scatter", height=25.0, nbg=0, corners="given"),
        # total-field-anomaly magnetics over uneven station subsets
        dict(name="tfa_subsets", family="subsets", kind="magnetic", transform="tfa", nx=48, ny=48,
             nz=24, nst=1024, layout="grid", height=30.0, nbg=0, corners="sums", nsub=8,
             smallest=64, largest=512),
        # a new geometry: first data, the fp16 pair sensitivity and a line search of models with it
        dict(name="survey_setup", family="setup", kind="joint", transform="none", nx=64, ny=64,
             nz=32, nst=1024, layout="grid", height=50.0, nbg=0, corners="sums", storage="f16x2",
             nmodels=24),
        # the batched inversion step: 256 models on the joint survey
        dict(name="batched_step", family="stored", kind="joint", transform="none", nx=64, ny=64,
             nz=32, nst=1024, layout="grid", height=50.0, nbg=0, corners="sums", storage="f16x2",
             nmodels=256),
        # a few line-search trials with the default storage
        dict(name="line_search", family="stored", kind="joint", transform="none", nx=64, ny=64,
             nz=32, nst=1024, layout="grid", height=50.0, nbg=0, corners="sums", storage="fp32",
             nmodels=4),
        # one model's step with the default storage, FTG data through their invariant
        dict(name="ftg_stored", family="stored", kind="tensor", transform="ftg_invariant", nx=64,
             ny=64, nz=32, nst=1600, layout="grid", height=50.0, nbg=0, corners="sums",
             storage="fp32", nmodels=1),
        # models to a grid refined twice along each axis, gradients back
        dict(name="refine_batch", family="refine", nx=64, ny=64, nz=32, fx=2, fy=2, fz=2,
             nmodels=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["matrix_free", "matrix_free", "matrix_free", "subsets", "calculator",
                         "setup", "stored", "stored", "stored", "refine"])
    if family == "refine":
        fx, fy, fz = (rng.choice([1, 2, 4]) for _ in range(3))
        c = dict(family=family, nx=_log_int(rng, 6, 64), ny=_log_int(rng, 6, 64),
                 nz=_log_int(rng, 4, 32), fx=fx, fy=fy, fz=fz)
        fine = c["nx"] * c["ny"] * c["nz"] * fx * fy * fz
        c["nmodels"] = max(1, min(_log_int(rng, 1, 256), (1 << 27) // fine))
        return c
    kind = rng.choice({"subsets": ["magnetic", "scalar", "tensor"],
                       "calculator": ["scalar", "tensor"],
                       "stored": ["scalar", "tensor", "joint", "magnetic"],
                       "setup": ["scalar", "tensor", "joint", "magnetic"]}.get(
                           family, ["scalar", "tensor", "joint", "magnetic", "mag_gradient",
                                    "magnetization"]))
    transform = rng.choice({"tensor": ["none", "ftg_invariant"],
                            "magnetic": ["none", "tfa", "total_field"],
                            "magnetization": ["none", "tfa", "total_field"]}.get(kind, ["none"]))
    if family == "calculator":
        transform = "none"
    nbg = rng.choice([0, 0, 3]) if kind in ("scalar", "tensor", "joint") else 0
    c = dict(family=family, kind=kind, transform=transform, nbg=nbg,
             layout=rng.choice(["grid", "scatter"]), height=rng.choice([1.0, 10.0, 30.0, 50.0]),
             corners="sums")
    top = {"matrix_free": (44, 28, 2500), "subsets": (48, 24, 1024), "calculator": (30, 15, 400),
           "setup": (64, 32, 1024), "stored": (64, 32, 1024)}[family]
    if family in ("setup", "stored") and kind in ("scalar", "joint"):
        top = (32, 20, 1024)
    c.update(nx=_log_int(rng, 6, top[0]), ny=_log_int(rng, 6, top[0]), nz=_log_int(rng, 4, top[1]),
             nst=_log_int(rng, 16 if family in ("setup", "stored") else 4, top[2]))
    if c["layout"] == "grid":
        c["nst"] = max(2, int(round(math.sqrt(c["nst"])))) ** 2
    shape = rng.random() if family == "matrix_free" else 1.0
    if shape < 0.2:  # corners given: eight corners a cell
        c.update(corners="given", nx=_log_int(rng, 6, 32), ny=_log_int(rng, 6, 32),
                 nz=_log_int(rng, 4, 16))
    elif shape < 0.35:  # the largest meshes: gravity over layers, ground stations on a grid
        c.update(kind=rng.choice(["scalar", "joint"]), transform="none", nbg=3, layout="grid",
                 nx=_log_int(rng, 44, 96), ny=_log_int(rng, 44, 96), nz=_log_int(rng, 24, 48),
                 nst=rng.randint(4, 24) ** 2, height=1.0)
    if family == "subsets":
        small = rng.randint(1, max(1, c["nst"] // 8))
        c.update(nsub=rng.randint(1, 12), smallest=small,
                 largest=max(small, min(c["nst"], _log_int(rng, 8, 512))))
    if family in ("setup", "stored"):
        c["storage"] = rng.choice(["fp32", "f16x2"])
        c["nmodels"] = _log_int(rng, 1, 8 if c["storage"] == "fp32" else 256)
    return c


# ---------------------------------------------------------------------------
# Inputs, from the seed alone
def _mesh(case):
    """Corner coordinates (n + 1) and cell sizes (n) of the three axes, as a
    program has them: running sums of the sizes, or decimals of both."""
    axes = []
    for n, cell, growth in ((case["nx"], 50.0, 1.0), (case["ny"], 50.0, 1.0),
                            (case["nz"], 25.0, 1.05)):
        sizes = cell * growth ** np.arange(n)
        if case.get("corners") == "given":
            # uneven sizes with two decimals, corners with two decimals around a local origin
            sizes = np.round(sizes * (1.0 + 0.1 * np.sin(1.7 * np.arange(n))), 2)
            start = -round(0.37 * sizes.sum(), 2) if growth == 1.0 else 0.0
            c = np.round(start + np.concatenate([[0.0], np.cumsum(sizes)]), 2)
        else:
            c = np.zeros(n + 1)
            for i in range(n):
                c[i + 1] = c[i] + sizes[i]
        axes.append((c, sizes))
    return axes


def _stations(case, axes, rng):
    x, y = axes[0][0], axes[1][0]
    if case["layout"] == "grid":
        n = int(round(math.sqrt(case["nst"])))
        gx = x[0] + (x[-1] - x[0]) * (np.arange(n) + 0.5) / n
        gy = y[0] + (y[-1] - y[0]) * (np.arange(n) + 0.5) / n
        X, Y = np.meshgrid(gx, gy, indexing="ij")
        return np.stack([X.ravel(), Y.ravel(), np.full(X.size, -case["height"])], axis=1)
    n = case["nst"]
    return np.stack([rng.uniform(x[0], x[-1], n), rng.uniform(y[0], y[-1], n),
                     -case["height"] - rng.uniform(0.0, 20.0, n)], axis=1)


def _cell_values(case, n, gen):
    """n models [n][parameters]: density anomalies (kg/m^3: smooth bodies and
    noise), susceptibilities or magnetisations."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kind = case.get("kind", "scalar")
    dev = gen.device
    if kind in ("magnetic", "mag_gradient"):
        v = torch.exp(math.log(0.005) + torch.randn(n, nx * ny * nz, generator=gen, device=dev,
                                                    dtype=torch.float64)).clamp(max=0.1)
    elif kind == "magnetization":
        v = 0.5 * torch.randn(n, 3 * nx * ny * nz, generator=gen, device=dev, dtype=torch.float64)
    else:
        u = torch.rand(4, 5, generator=gen, device=dev, dtype=torch.float64)
        X, Y, Z = torch.meshgrid(*[(torch.arange(m, device=dev, dtype=torch.float64) + 0.5) / m
                                   for m in (nx, ny, nz)], indexing="ij")
        base = torch.zeros_like(X)
        for b in u:
            amp = 300.0 if float(b[4]) < 0.5 else -300.0
            base += amp * torch.exp(-((X - b[0]) ** 2 + (Y - b[1]) ** 2 + (Z - b[2]) ** 2) /
                                    (2 * (0.05 + 0.15 * b[3]) ** 2))
        v = base.reshape(1, -1) + 50.0 * torch.randn(n, nx * ny * nz, generator=gen, device=dev,
                                                     dtype=torch.float64)
    nbg = case.get("nbg", 0)
    if nbg:
        layers = 2400.0 + 200.0 * torch.arange(nbg, device=dev, dtype=torch.float64)
        v = torch.cat([v, layers.expand(n, nbg)], dim=1)
    return v.contiguous()


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 17])
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    axes = _mesh(case)
    i = dict(axes=axes, models=_cell_values(case, case.get("nmodels", 1), gen))
    if case["family"] == "refine":
        fine = i["models"].shape[1] * case["fx"] * case["fy"] * case["fz"]
        i["gradients"] = torch.randn(case["nmodels"], fine, generator=gen, device="cuda",
                                     dtype=torch.float64)
        return i
    i["stations"] = _stations(case, axes, rng)
    i["thick"] = np.array([200.0, 500.0, 10000.0])[:case["nbg"]]
    dpm = RAW[case["kind"]] if case["transform"] == "none" else 1
    nd = case["nst"]
    if case["family"] == "subsets":
        # uneven sizes that belong to the survey, other stations with another seed
        sizes = np.random.default_rng(105).integers(case["smallest"], case["largest"] + 1,
                                                    case["nsub"])
        i["subsets"] = [np.sort(rng.choice(case["nst"], int(n), replace=False)) for n in sizes]
        nd = int(sizes.sum())
    unit = torch.full((dpm,), SCALE[case["kind"]], device="cuda", dtype=torch.float64)
    sigma = torch.full((dpm,), SIGMA[case["kind"]], device="cuda", dtype=torch.float64)
    if case["kind"] == "joint":
        unit[0], sigma[0] = SCALE["scalar"], SIGMA["scalar"]
    if case["transform"] == "ftg_invariant":
        unit, sigma = unit * unit, sigma * sigma
    noise = torch.randn(case.get("nmodels", 1), nd, dpm, generator=gen, device="cuda",
                        dtype=torch.float64)
    i["observed"] = (noise[0] * unit).reshape(-1)
    i["inv_var"] = (1.0 / (sigma * sigma)).repeat(nd)
    i["misfit"] = (noise[0] / sigma).reshape(-1)
    return i


# ---------------------------------------------------------------------------
# What a program has in hand, and one pass
def _context(case, i, stream):
    ctx = capi.Context(0)
    ctx.set_stream(stream.cuda_stream)
    (x, xs), (y, ys), (z, zs) = i["axes"]
    ctx.set_mesh(x, y, z, xs, ys, zs)
    if case["family"] != "refine":
        st = i["stations"]
        ctx.set_background(i["thick"])
        ctx.set_stations(st[:, 0], st[:, 1], st[:, 2])
        ctx.set_kind(KINDS[case["kind"]], INC, DEC, FS)
        ctx.set_transform(TRANSFORMS[case["transform"]], INC, DEC)
    return ctx


def _prepare_calculator(case, i):
    Model = gravmag.ThreeDGravityModel()
    Model.SetMeshSize(case["nx"], case["ny"], case["nz"])
    Model.SetXCellSizes(i["axes"][0][1])
    Model.SetYCellSizes(i["axes"][1][1])
    Model.SetZCellSizes(i["axes"][2][1])
    values = i["models"][0].cpu().numpy()
    ngrid = Model.GetNModelElements()
    Model.SetDensities()[...] = values[:ngrid].reshape(Model.GetDensities().shape)
    Model.SetBackgroundThicknesses(i["thick"])
    Model.SetBackgroundDensities(values[ngrid:])
    tensor = case["kind"] == "tensor"
    Data = gravmag.TensorGravityData() if tensor else gravmag.ScalarGravityData()
    for p in i["stations"]:
        Data.AddMeasurementPoint(*p)
    Calc = gravmag.MinMemGravMagCalculator(
        gravmag.TensorGB300GravityImp() if tensor else gravmag.ScalarGB300GravityImp())
    return dict(family="calculator", calc=Calc, model=Model, data=Data,
                misfit=i["misfit"].cpu().numpy())


def prepare(case, seed):
    i = _inputs(case, seed)
    if case["family"] == "calculator":
        return _prepare_calculator(case, i)
    stream = torch.cuda.Stream()
    s = dict(family=case["family"], stream=stream, models=i["models"],
             nmodels=i["models"].shape[0])
    if case["family"] == "refine":
        (x, xs), (y, ys), (z, zs) = i["axes"]
        fine = [np.repeat(v / f, f) for v, f in ((xs, case["fx"]), (ys, case["fy"]),
                                                 (zs, case["fz"]))]
        corners = [np.concatenate([[0.0], np.cumsum(v)]) for v in fine]
        ctx = s["ctx"] = capi.Context(0)
        ctx.set_stream(stream.cuda_stream)
        ctx.set_mesh(*corners, *fine)
        ctx.set_refinement(xs, ys, zs)
        s["gradients"] = i["gradients"]
        s["fine"] = torch.zeros_like(i["gradients"])
        s["coarse"] = torch.zeros_like(i["models"])
        return s
    ctx = s["ctx"] = _context(case, i, stream)
    nparm = i["models"].shape[1]
    nd = i["observed"].numel()
    like = dict(device="cuda", dtype=torch.float64)
    if case["family"] == "subsets":
        s.update(subsets=i["subsets"], misfit=i["misfit"], data=torch.zeros(nd, **like),
                 grad=torch.zeros(case["nsub"], nparm, **like))
        return s
    s.update(data=torch.zeros(s["nmodels"], nd, **like),
             grad=torch.zeros(s["nmodels"], nparm, **like))
    if case["family"] == "matrix_free":
        s["misfit"] = i["misfit"]
        return s
    s.update(storage=STORAGES[case["storage"]], observed=i["observed"], inv_var=i["inv_var"],
             first=torch.zeros(nd, **like))
    if case["family"] == "stored":
        ctx.build_sensitivity(s["storage"])
    torch.cuda.synchronize()
    return s


def _step(s):
    ctx, n = s["ctx"], s["nmodels"]
    ctx.batched_forward_device(n, s["models"].data_ptr(), s["data"].data_ptr())
    with torch.cuda.stream(s["stream"]):
        misfit = (s["data"] - s["observed"]) * s["inv_var"]
    ctx.batched_lqderivative_device(n, s["models"].data_ptr(), misfit.data_ptr(),
                                    s["grad"].data_ptr())
    return {"data": s["data"], "grad": s["grad"]}


def run(s):
    family = s["family"]
    if family == "calculator":
        data = s["calc"].Calculate(s["model"], s["data"])
        return {"data": data, "grad": s["calc"].LQDerivative(s["model"], s["data"], s["misfit"])}
    ctx = s["ctx"]
    if family == "matrix_free":
        ctx.forward_device(s["models"].data_ptr(), s["data"].data_ptr())
        ctx.lqderivative_device(s["models"].data_ptr(), s["misfit"].data_ptr(),
                                s["grad"].data_ptr())
        return {"data": s["data"], "grad": s["grad"]}
    if family == "subsets":
        ctx.subsets_forward_device(s["subsets"], s["models"].data_ptr(), s["data"].data_ptr())
        ctx.subsets_lqderivative_device(s["subsets"], s["models"].data_ptr(),
                                        s["misfit"].data_ptr(), s["grad"].data_ptr())
        return {"data": s["data"], "grad": s["grad"]}
    if family == "refine":
        ctx.refine_project_device(s["nmodels"], s["models"].data_ptr(), s["fine"].data_ptr())
        ctx.refine_combine_device(s["nmodels"], s["gradients"].data_ptr(),
                                  s["coarse"].data_ptr())
        return {"fine": s["fine"], "coarse": s["coarse"]}
    if family == "setup":
        ctx.forward_device(s["models"].data_ptr(), s["first"].data_ptr())
        ctx.build_sensitivity(s["storage"])
        return {"first": s["first"], **_step(s)}
    return _step(s)


# ---------------------------------------------------------------------------
# The work that cannot be left out
def work(case):
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["family"] == "refine":
        fine = cells * case["fx"] * case["fy"] * case["fz"]
        return {"bytes": 2.0 * 8 * case["nmodels"] * (cells + fine),
                "flops": float(case["nmodels"] * fine)}
    kind, nmod = case["kind"], case.get("nmodels", 1)
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if case["corners"] == "given":
        nodes = 8 * cells
    nst, grads = case["nst"], 1
    if case["family"] == "subsets":
        nst = case["nsub"] * 0.5 * (case["smallest"] + case["largest"])
        grads = case["nsub"]
    nparm = (3 if kind == "magnetization" else 1) * cells + case["nbg"]
    dpm = RAW[kind] if case["transform"] == "none" else 1
    vectors = 8.0 * ((nmod + 1) * nparm + nmod * grads * nparm + 2 * nmod * nst * dpm)
    terms = float(nodes * nst * TERM_FLOPS[kind])
    if case["family"] in ("matrix_free", "subsets", "calculator"):
        passes = 3 if case["transform"] in ("ftg_invariant", "total_field") else 2
        return {"bytes": vectors, "flops": passes * terms}
    passes = 3 if case["transform"] in ("ftg_invariant", "total_field") else 2
    elements = float(nst * STORED[kind] * cells * (3 if kind == "magnetization" else 1))
    step = {"bytes": passes * 4 * elements + vectors, "flops": passes * 2 * elements * nmod}
    if case["family"] == "setup":
        copies = 2 if case["storage"] == "f16x2" else 1  # the fp16 pair keeps its transpose too
        step["bytes"] += copies * 4 * elements
        step["flops"] += 2 * terms
    return step


# ---------------------------------------------------------------------------
# The same in 64 bits, with torch alone
def _terms(kind, d):
    """Corner terms of the seven components a kind uses, for offsets d
    (station - corner) [stations][x][y][z]."""
    dx, dy, dz = d
    xx, yy, zz = dx * dx, dy * dy, dz * dz
    r = torch.sqrt(xx + yy + zz)

    def ln(u, rest):  # ln(max(u + r, eps)), without the cancellation where u is negative
        return torch.log(torch.where(u < 0, rest / (r - u), u + r).clamp(min=2.0 ** -52))
    out = {}
    if kind in ("scalar", "joint"):
        out["gz"] = (dx * ln(dy, xx + zz) + dy * ln(dx, yy + zz) +
                     dz * torch.atan2(dz * r, dx * dy))
    if kind != "scalar":
        out["xx"] = torch.atan2(dy * dz, dx * r)
        out["yy"] = torch.atan2(dx * dz, dy * r)
        out["zz"] = torch.atan2(dx * dy, dz * r)
        out["xy"] = ln(dz, xx + yy)
        out["xz"] = ln(dy, xx + zz)
        out["yz"] = ln(dx, yy + zz)
    return out


def _prisms(kind, st, corners, shared):
    """Prism values [component][stations][cells] from the corner terms;
    shared: the corners of neighbouring cells are the same, n + 1 an axis, else
    lower and upper corners alternate, 2 n an axis."""
    d = [st[:, a].reshape(-1, 1, 1, 1) - corners[a].reshape([1] + [-1 if b == a else 1
                                                                   for b in range(3)])
         for a in range(3)]
    out = {}
    for name, f in _terms(kind, d).items():
        for a in (1, 2, 3):
            if shared:
                f = torch.diff(f, dim=a)
            else:
                n = f.shape[a]
                lo, hi = (f.index_select(a, torch.arange(k, n, 2, device=f.device))
                          for k in (0, 1))
                f = hi - lo
        scale = GRAV if name in ("xx", "yy", "zz") else -GRAV
        out[name] = (scale * f).reshape(f.shape[0], -1)
    return out


def _rows(kind, p):
    """Raw sensitivity rows [raw][stations][parameters] from prism values."""
    if kind == "scalar":
        return [p["gz"]]
    tensor = [p[n] for n in ("xx", "xy", "xz", "xy", "yy", "yz", "xz", "yz", "zz")]
    if kind == "tensor":
        return tensor
    if kind == "joint":
        return [p["gz"]] + tensor
    b = (math.cos(INC) * math.cos(DEC), math.cos(INC) * math.sin(DEC), math.sin(INC))
    if kind == "magnetization":
        f = 1e9 * 4e-7 * math.pi / (4 * math.pi * GRAV)
        return [f * torch.cat([tensor[3 * k + j] for j in range(3)], dim=1) for k in range(3)]
    if kind == "mag_gradient":
        f = FS * 1e-7 / GRAV
        return [f * (b[0] * p["xz"] + b[1] * p["yz"] + b[2] * p["zz"])]
    f = FS / (4 * math.pi * GRAV)
    return [f * sum(b[j] * tensor[3 * k + j] for j in range(3)) for k in range(3)]


def _layers(kind, st, axes, thick):
    """Background rows [raw][stations][layers]: infinite sheets less the part
    that the mesh takes (stations above the mesh)."""
    x, y, z = (a[0] for a in axes)
    top, cols = 0.0, []
    for t in thick:
        bottom = top + t
        rows = [torch.zeros(st.shape[0], 1, device=st.device, dtype=st.dtype)
                for _ in range(RAW[kind])]
        if kind in ("scalar", "joint"):
            rows[0] = rows[0] + 2 * math.pi * GRAV * t
        if top < z[-1]:
            box = [torch.tensor(v, device=st.device, dtype=st.dtype)
                   for v in ((x[0], x[-1]), (y[0], y[-1]), (top, min(bottom, z[-1])))]
            rows = [a - b for a, b in zip(rows, _rows(kind, _prisms(kind, st, box, True)))]
        cols.append(rows)
        top = bottom
    return [torch.cat([c[r] for c in cols], dim=1) for r in range(RAW[kind])]


def _jacobian(case, i, st):
    """Raw rows [stations][raw][parameters] of a few stations."""
    kind = case["kind"]
    shared = case["corners"] == "sums"
    corners = []
    for c, size in i["axes"]:
        c = torch.tensor(c, device=st.device, dtype=st.dtype)
        size = torch.tensor(size, device=st.device, dtype=st.dtype)
        corners.append(c if shared else torch.stack([c[:-1], c[:-1] + size], 1).reshape(-1))
    rows = _rows(kind, _prisms(kind, st, corners, shared))
    if kind == "mag_gradient":
        below = st + torch.tensor([0.0, 0.0, 1.0], device=st.device, dtype=st.dtype)
        rows = [rows[0] - _rows(kind, _prisms(kind, below, corners, shared))[0]]
    if case["nbg"]:
        rows = [torch.cat(v, dim=1) for v in zip(rows, _layers(kind, st, i["axes"], i["thick"]))]
    return torch.stack(rows, dim=1)


def _transformed(case, raw):
    """Data [..., stations, data] of raw data [..., stations, raw] and the
    derivative [..., stations, data, raw]."""
    t = case["transform"]
    if t == "none":
        return raw, None
    d = raw.unbind(-1)
    if t == "ftg_invariant":
        v = (d[0] * d[4] + d[4] * d[8] + d[0] * d[8] - d[3] * d[1] - d[7] * d[5] - d[2] * d[6])
        g = torch.stack([d[4] + d[8], -d[3], -d[6], -d[1], d[0] + d[8], -d[7], -d[2], -d[5],
                         d[0] + d[4]], dim=-1)
    elif t == "total_field":
        v = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        g = raw / v.unsqueeze(-1)
    else:
        b = torch.tensor([math.cos(INC) * math.cos(DEC), math.cos(INC) * math.sin(DEC),
                          math.sin(INC)], device=raw.device, dtype=raw.dtype)
        v, g = raw @ b, b.expand_as(raw)
    return v.unsqueeze(-1), g.unsqueeze(-2)


def exact(case, seed):
    i = _inputs(case, seed)
    models = i["models"]
    if case["family"] == "refine":
        f = (case["fx"], case["fy"], case["fz"])
        n = (case["nx"], case["ny"], case["nz"])
        m = models.reshape(-1, *n)
        g = i["gradients"].reshape(-1, n[0], f[0], n[1], f[1], n[2], f[2])
        for a in range(3):
            m = m.repeat_interleave(f[a], dim=a + 1)
        return {"fine": m.reshape(models.shape[0], -1),
                "coarse": g.sum(dim=(2, 4, 6)).reshape(models.shape[0], -1)}
    st = torch.tensor(i["stations"], device="cuda")
    groups = i.get("subsets") or [np.arange(st.shape[0])]
    nodes = np.prod([c.size * (1 if case["corners"] == "sums" else 2) for c, _ in i["axes"]])
    chunk = int(max(1, min(64, 1.5e7 // nodes)))
    nmod = models.shape[0]
    grad = torch.zeros(nmod * len(groups), models.shape[1], device="cuda", dtype=torch.float64)
    data, at = [], 0
    dpm = RAW[case["kind"]] if case["transform"] == "none" else 1
    for k, group in enumerate(groups):
        for s0 in range(0, len(group), chunk):
            idx = torch.as_tensor(group[s0:s0 + chunk], device="cuda")
            J = _jacobian(case, i, st[idx])
            ns, raw, npar = J.shape
            J = J.reshape(ns * raw, npar)
            d, dT = _transformed(case, (models @ J.T).reshape(nmod, ns, raw))
            here = slice(at * dpm, (at + ns) * dpm)
            if case["family"] in ("stored", "setup"):
                mis = ((d.reshape(nmod, -1) - i["observed"][here]) * i["inv_var"][here])
            else:
                mis = i["misfit"][here].expand(nmod, -1)
            w = mis.reshape(nmod, ns, dpm, 1)
            w = (w if dT is None else (w * dT).sum(dim=2)).reshape(nmod, ns * raw)
            grad[k * nmod:(k + 1) * nmod] += 2.0 * (w @ J)
            data.append(d.reshape(nmod, -1))
            at += ns
    out = {"data": torch.cat(data, dim=1), "grad": grad}
    if case["family"] == "calculator":
        return {"data": out["data"][0], "grad": out["grad"][0]}
    if case["family"] == "subsets":
        return {"data": out["data"][0], "grad": grad}
    if case["family"] == "setup":
        return {"first": out["data"][0], **out}
    return out
