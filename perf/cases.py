"""The measured workloads of the NUFFT engine: what its users run, through the public plans.

A case is a dict of plain values:

  kind    "t1", "t2"   one type-1 / type-2 transform
          "t12"        a type-2 and a type-1 transform on the same points
          "normal"     type 2, then type 1 of its samples (one step of an iterative solver)
          "many"       `vecs` type-1 transforms of different strengths on the same points
          "t3"         a type-3 transform, `vecs` strength vectors at once
          "batch"      `vecs` type-1 transforms of uneven sizes in one Batch, half 2D, half 3D
  dim, dtype, tol, sign, order, M; n0, n1, n2: modes per dimension; K, X, S: targets and box
  half-widths of type 3; dist: "uniform", "blob" (one Gaussian cluster, sigma 0.1, wrapped) or
  "radial" (points along spokes through the origin); rebin: whether a pass also hands the plan
  new points (set_points), as a program does whose points change from call to call.
  upsampfac, width, tile: plan options, 0 for the plan's own choice.
"""
import math
import random

import torch

import neonufft_b200 as nnb

DTYPES = {"f32": (torch.float32, torch.complex64, 4), "f64": (torch.float64, torch.complex128, 8)}


def _case(name, kind, dim, dtype, tol, M, modes=(), dist="uniform", rebin=True, sign=-1, order=1,
          vecs=1, K=0, X=0.0, S=0.0, upsampfac=2.0, width=0, tile=0):
    n = list(modes) + [1] * (3 - len(modes))
    c = dict(kind=kind, dim=dim, dtype=dtype, tol=tol, M=M, n0=n[0], n1=n[1], n2=n[2], dist=dist,
             rebin=rebin, sign=sign, order=order, vecs=vecs, K=K, X=X, S=S, upsampfac=upsampfac,
             width=width, tile=tile)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # A short signal at the default tolerance: launches and latency, hardly any arithmetic.
        _case("1d-small", "t12", 1, "f32", 1e-3, 2000, (1000,)),
        # A long irregularly sampled series in double precision; odd number of modes.
        _case("1d-large", "t12", 1, "f64", 1e-9, 5_000_000, (200_001,), sign=1),
        # One small image's worth of samples whose points change from call to call.
        _case("2d-image", "t1", 2, "f32", 1e-6, 100_000, (256, 256), width=8),
        # One step of an iterative 2D reconstruction on radial samples: fixed points, ragged box.
        _case("2d-solver-step", "normal", 2, "f32", 1e-5, 3_000_001, (777, 640), dist="radial",
              rebin=False),
        # Type-2 and type-1 pair on a volume, new points: the ordinary 3D job.
        _case("3d-pair", "t12", 3, "f32", 1e-6, 10_000_000, (128, 128, 128), width=8),
        # The largest single transform, with the options tuned for its size.
        _case("3d-large", "t1", 3, "f32", 1e-6, 100_000_000, (256, 256, 256), width=8,
              upsampfac=1.875, tile=4),
        # Several strength vectors on the same points (an odd count, ragged box).
        _case("3d-vectors", "many", 3, "f32", 1e-5, 2_000_003, (100, 96, 81), vecs=5,
              rebin=False, order=0),
        # Double precision on clustered points.
        _case("3d-double", "t12", 3, "f64", 1e-6, 3_000_000, (96, 96, 96), dist="blob"),
        # Double precision at a tight tolerance: wide kernels.
        _case("3d-double-tight", "t12", 3, "f64", 1e-9, 500_000, (64, 60, 64), rebin=False),
        # Type 3 at a large space-bandwidth product: new points on both sides every call.
        _case("type3-2d", "t3", 2, "f32", 1e-5, 5_000_000, K=5_000_000, X=50.0, S=200.0),
        # Type 3 in a volume, several vectors at once on fixed points.
        _case("type3-3d-vectors", "t3", 3, "f32", 1e-5, 300_000, K=200_001, X=5.0, S=20.0,
              vecs=4, rebin=False),
        # Uneven 2D and 3D transforms run as one captured batch; `M` bounds the largest.
        _case("batch", "batch", 0, "f32", 1e-6, 3_000_000, vecs=24, rebin=False, width=8),
    ]


def _width(case):
    if case["width"]:
        return case["width"]
    return min(16, max(2, math.ceil(-math.log10(case["tol"] / 10.0))))


def _seconds(case):
    """A rough time of one pass, to keep drawn cases below the largest listed one."""
    t = 0.0
    for dim, M, modes in _shapes(case):
        w = _width(case)
        cell = (1 if case["dtype"] == "f32" else 3) * (5e-13 if dim == 3 and w <= 8 else 4e-12)
        cells = math.prod(max(2 * w, 2 * n) for n in modes)
        both = 2 if case["kind"] in ("t12", "normal", "t3") else 1
        t += case["vecs"] * both * (M * (w ** dim * cell + 1e-10) + cells * 3e-11) / max(
            1, case["vecs"] if case["kind"] == "batch" else 1)
    return t


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        kind = rng.choice(["t1", "t2", "t12", "normal", "many", "t3", "t3", "batch"])
        dtype = rng.choice(["f32", "f32", "f64"])
        tol = rng.choice([1e-3, 1e-4, 1e-5, 1e-6] if dtype == "f32" else [1e-6, 1e-9, 1e-12])
        dim = rng.choice([1, 2, 2, 3, 3])
        M = log_int(1000, 20_000_000)
        common = dict(dist=rng.choice(["uniform", "uniform", "blob", "radial"]),
                      rebin=rng.random() < 0.6, sign=rng.choice([-1, 1]),
                      order=rng.choice([0, 1, 1]))
        if kind == "batch":
            c = _case(None, kind, 0, "f32", tol, log_int(30_000, 3_000_000),
                      vecs=rng.randint(4, 24), rebin=False, sign=common["sign"])
        elif kind == "t3":
            # box half-widths around a product that gives fine grids of an affordable size
            top = {1: 1e5, 2: 1e4, 3: 150.0}[dim]
            product = math.exp(rng.uniform(math.log(20.0), math.log(top)))
            ratio = rng.uniform(1.0, 4.0)
            X = round(math.sqrt(product / ratio), 3)
            c = _case(None, kind, dim, dtype, tol, min(M, 5_000_000),
                      K=log_int(1000, 5_000_000), X=X, S=round(X * ratio, 3),
                      vecs=rng.choice([1, 1, 2, 3, 4]), rebin=common["rebin"],
                      sign=common["sign"])
        else:
            top = {1: 400_000, 2: 1500, 3: 200}[dim]
            low = {1: 100, 2: 32, 3: 16}[dim]
            modes = [log_int(low, top) for _ in range(dim)]
            c = _case(None, kind, dim, dtype, tol, M, modes,
                      vecs=rng.randint(2, 8) if kind == "many" else 1, **common)
        if _seconds(c) < 0.012:
            return c


def _shapes(case):
    """(dim, points, modes) of each transform of a case."""
    if case["kind"] == "batch":
        r = random.Random(case["M"] * 64 + case["vecs"])
        shapes = []
        for i in range(case["vecs"]):
            dim = 2 + i % 2
            M = int(math.exp(r.uniform(math.log(10_000), math.log(case["M"]))))
            n = [r.randint(40, 512 if dim == 2 else 128) for _ in range(dim)]
            shapes.append((dim, M, n))
        return shapes
    if case["kind"] == "t3":
        nf1 = int(4 * case["X"] * case["S"] / math.pi) + _width(case) + 2
        return [(case["dim"], max(case["M"], case["K"]), [nf1] * case["dim"])]
    return [(case["dim"], case["M"], [case["n0"], case["n1"], case["n2"]][: case["dim"]])]


def _points(gen, dim, M, dist, dtype):
    def uniform():
        return torch.rand(M, generator=gen, device="cuda", dtype=torch.float64)

    def wrap(x):
        return torch.remainder(x + math.pi, 2 * math.pi) - math.pi

    if dist == "blob":
        centre = [2 * math.pi * torch.rand(1, generator=gen, device="cuda", dtype=torch.float64)
                  for _ in range(dim)]
        pts = [wrap(centre[d] + 0.1 * torch.randn(M, generator=gen, device="cuda",
                                                  dtype=torch.float64)) for d in range(dim)]
    elif dist == "radial" and dim > 1:
        per = max(1, int(math.sqrt(M)))
        j = torch.arange(M, device="cuda", dtype=torch.float64)
        spoke = torch.floor(j / per)
        r = 2 * math.pi * (torch.remainder(j, per) + uniform()) / per - math.pi
        a = spoke * 2.399963229728653
        pts = [r * torch.cos(a), r * torch.sin(a)]
        if dim == 3:
            z = torch.remainder(spoke * 0.618033988749895, 1.0) * 2 - 1
            s = torch.sqrt(1 - z * z)
            pts = [pts[0] * s, pts[1] * s, r * z]
    else:
        pts = [uniform() * (2 * math.pi) - math.pi for _ in range(dim)]
    return [p.to(dtype).contiguous() for p in pts]


def _normal(gen, n, cdt):
    rdt = torch.float32 if cdt == torch.complex64 else torch.float64
    return torch.view_as_complex(torch.randn(n, 2, generator=gen, device="cuda", dtype=rdt))


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    rdt, cdt, _ = DTYPES[case["dtype"]]
    kind, M, vecs = case["kind"], case["M"], case["vecs"]
    s = {}
    if kind == "batch":
        s["parts"] = [(dim, M, n, _points(gen, dim, M, "blob" if i % 4 >= 2 else "uniform", rdt),
                       _normal(gen, M, cdt))
                      for i, (dim, M, n) in enumerate(_shapes(case))]
        return s
    if kind == "t3":
        def box(n, half):
            return [((torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1)
                     * half).to(rdt) for _ in range(case["dim"])]

        s["loc"], s["targets"] = box(M, case["X"]), box(case["K"], case["S"])
        s["c"] = _normal(gen, M * vecs, cdt)
        return s
    s["loc"] = _points(gen, case["dim"], M, case["dist"], rdt)
    (_, _, modes), = _shapes(case)
    if kind in ("t1", "t12", "many"):
        s["c"] = _normal(gen, M * vecs, cdt)
    if kind in ("t2", "t12", "normal"):
        s["f"] = _normal(gen, math.prod(modes), cdt)
    return s


def _strides(modes):
    out = [1]
    for n in modes[:-1]:
        out.append(out[-1] * n)
    return out


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    rdt, cdt, _ = DTYPES[case["dtype"]]
    tile = (4, 4, 1) if case["tile"] == 4 else (0, 0, 0)
    opt = nnb.Options(tol=case["tol"], upsampfac=case["upsampfac"], order=case["order"],
                      n_spread=case["width"], tile=tile)
    kind, M, vecs = case["kind"], case["M"], case["vecs"]

    def empty(n):
        return torch.empty(n, dtype=cdt, device="cuda")

    if kind == "batch":
        s["plan"] = nnb.Batch(opt, rdt, num_streams=16)
        s["out"] = []
        for dim, M, n, loc, c in s["parts"]:
            s["out"].append(empty(math.prod(n)))
            s["plan"].add(1, case["sign"], loc, n, c, s["out"][-1], _strides(n))
        return s
    if kind == "t3":
        s["plan"] = nnb.PlanT3(opt, case["sign"], M, s["loc"], case["K"], s["targets"],
                               batch_size=vecs)
        s["out"] = empty(case["K"] * vecs)
        return s
    (_, _, modes), = _shapes(case)
    s["strides"] = _strides(modes)
    s["plan"] = nnb.Plan(opt, case["sign"], M, s["loc"], modes)
    if kind in ("t1", "t12", "many", "normal"):
        s["modes_out"] = empty(math.prod(modes) * vecs)
    if kind in ("t2", "t12", "normal"):
        s["samples_out"] = empty(M)
    return s


def run(s):
    case, plan = s["case"], s["plan"]
    kind, M = case["kind"], case["M"]
    if kind == "batch":
        plan.execute(nnb.Batch.GRAPH)
        return s["out"]
    if kind == "t3":
        if case["rebin"]:
            plan.set_input_points(M, s["loc"])
            plan.set_output_points(case["K"], s["targets"])
        plan.reset()
        plan.add_input(s["c"], M)
        plan.transform(s["out"], case["K"])
        return s["out"]
    if case["rebin"]:
        plan.set_points(M, s["loc"])
    out = {}
    if kind in ("t2", "t12", "normal"):
        plan.transform_type_2(s["f"], s["strides"], s["samples_out"])
        out["samples"] = s["samples_out"]
    if kind == "many":
        plan.transform_type_1_many(s["c"], s["modes_out"], case["vecs"], s["strides"])
    elif kind in ("t1", "t12", "normal"):
        plan.transform_type_1(s["samples_out"] if kind == "normal" else s["c"], s["modes_out"],
                              s["strides"])
    if kind != "t2":
        out["modes"] = s["modes_out"]
    return out


def work(case):
    """Inputs read once and outputs written once; per point and vector 4 flops (a complex value
    by a real weight, accumulated) for each of the kernel's w^dim cells, and the FFTs."""
    _, _, size = DTYPES[case["dtype"]]
    w, vecs, kind = _width(case), case["vecs"], case["kind"]
    nbytes = flops = 0.0

    def fft(cells):
        return 5.0 * cells * math.log2(max(2, cells))

    for dim, M, modes in _shapes(case):
        cells = math.prod(max(2 * w, int(n * case["upsampfac"])) for n in modes)
        n = math.prod(modes)
        if kind == "t3":
            nbytes += size * dim * (M + case["K"]) * case["rebin"]
            nbytes += 2.0 * size * vecs * (M + case["K"])
            flops += vecs * (4.0 * w ** dim * (M + case["K"]) + fft(cells))
            continue
        passes = 1 if kind == "batch" else 2 if kind in ("t12", "normal") else vecs
        nbytes += size * dim * M * case["rebin"] + 2.0 * size * (M + n) * passes
        flops += passes * (4.0 * w ** dim * M + fft(cells))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # The same plan (width, shape and grid of the kernel) with its sums in another order: the
    # engine's other spreading methods against the default one differ by up to 1.1e-6 (clustered
    # points) and 2.3e-7 (others) in single, 1.8e-15 in double precision; about four times that.
    return {"rel": 4.4e-6} if case["dtype"] == "f32" else {"rel": 8e-15}


# ---- 64-bit sums, without the engine ------------------------------------------------------------
def _mode_numbers(n, order):
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    if order == 1:
        return k - n // 2
    return torch.where(k < n - n // 2, k, k - n)


def _waves(sign, x, k):
    """exp(i sign x_j k_m), points by modes."""
    ph = sign * x[:, None] * k[None, :]
    return torch.polar(torch.ones_like(ph), ph)


def _factors(sign, loc, modes, order):
    """The exponentials of one set of points as two factors: modes of the last dimension, and of
    the others together (1D: coarse and fine steps of the mode number)."""
    dim = len(modes)
    if dim == 1:
        n = modes[0]
        fine = max(1, int(math.sqrt(n)))
        coarse = -(-n // fine)
        start = -(n // 2)
        a = _waves(sign, loc[0], start + fine * torch.arange(coarse, device="cuda",
                                                             dtype=torch.float64))
        return a, _waves(sign, loc[0], torch.arange(fine, device="cuda", dtype=torch.float64))
    e = [_waves(sign, loc[d], _mode_numbers(modes[d], order)) for d in range(dim)]
    if dim == 2:
        return e[1], e[0]
    return e[2], (e[1][:, :, None] * e[0][:, None, :]).reshape(len(loc[0]), -1)


def _from_blocks(F, modes, order):
    """The modes, x fastest, from the product of the two factors."""
    F = F.reshape(-1)
    if len(modes) == 1:
        F = F[: modes[0]]
        if order == 0:
            F = torch.roll(F, -(modes[0] // 2))
    return F.clone()


def _to_blocks(f, modes, rows, cols, order):
    if len(modes) == 1:
        if order == 0:
            f = torch.roll(f, modes[0] // 2)
        f = torch.cat([f, torch.zeros(rows * cols - modes[0], dtype=f.dtype, device="cuda")])
    return f.reshape(rows, cols)


def _chunks(loc, modes):
    width = math.prod(modes[:-1]) + modes[-1] if len(modes) > 1 else 2 * int(math.sqrt(modes[0]))
    step = max(1, int(6e7 // max(1, width)))
    for a in range(0, len(loc[0]), step):
        yield a, [x[a:a + step].double() for x in loc]


def _exact_type1(sign, loc, c, modes, order):
    total = None
    for a, x in _chunks(loc, modes):
        A, B = _factors(sign, x, modes, order)
        part = (A * c[a:a + len(x[0])].to(torch.complex128)[:, None]).T @ B
        total = part if total is None else total + part
    return _from_blocks(total, modes, order)


def _exact_type2(sign, loc, f, modes, order):
    out = []
    for _, x in _chunks(loc, modes):
        A, B = _factors(sign, x, modes, order)
        F = _to_blocks(f.to(torch.complex128), modes, A.shape[1], B.shape[1], order)
        out.append(((A @ F) * B).sum(1))
    return torch.cat(out)


def _exact_type3(sign, loc, targets, c, vecs):
    M, K = len(loc[0]), len(targets[0])
    loc, targets = [x.double() for x in loc], [x.double() for x in targets]
    c = c.to(torch.complex128).reshape(vecs, M)
    out = torch.empty(vecs, K, dtype=torch.complex128, device="cuda")
    step = max(1, int(1e8 // M))
    for a in range(0, K, step):
        ph = torch.zeros((), device="cuda", dtype=torch.float64)
        for x, t in zip(loc, targets):
            ph = ph + (sign * t[a:a + step])[None, :] * x[:, None]
        out[:, a:a + step] = c @ torch.polar(torch.ones_like(ph), ph)
    return out.reshape(-1)


def exact(case, seed):
    kind, vecs = case["kind"], case["vecs"]
    if kind == "t3":
        if float(case["M"]) * case["K"] > 1.2e11:
            return None
        s = _inputs(case, seed)
        return _exact_type3(case["sign"], s["loc"], s["targets"], s["c"], vecs)
    passes = 2 if kind in ("t12", "normal") else 1 if kind == "batch" else vecs
    if passes * sum(float(M) * math.prod(n) for _, M, n in _shapes(case)) > 2.0e13:
        return None
    s = _inputs(case, seed)
    sign, order = case["sign"], case["order"]
    if kind == "batch":
        return [_exact_type1(sign, loc, c, n, order) for _, _, n, loc, c in s["parts"]]
    (_, M, modes), = _shapes(case)
    out = {}
    if kind in ("t2", "t12", "normal"):
        out["samples"] = _exact_type2(sign, s["loc"], s["f"], modes, order)
    if kind == "many":
        out["modes"] = torch.cat([_exact_type1(sign, s["loc"], s["c"][v * M:(v + 1) * M], modes,
                                               order) for v in range(vecs)])
    elif kind in ("t1", "t12", "normal"):
        c = out["samples"] if kind == "normal" else s["c"]
        out["modes"] = _exact_type1(sign, s["loc"], c, modes, order)
    return out
