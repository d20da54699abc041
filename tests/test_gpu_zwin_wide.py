"""3D transforms with kernel widths 9 to 16 on the z-window kernels (the automatic method,
csrc/zwin_wide.cu) against the shared-memory slabs and the FP64 direct sums."""
import numpy as np
import pytest

from test_gpu_methods import direct, run_t12, width_bound

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("w", list(range(9, 17)))
@pytest.mark.parametrize("type_", [1, 2])
@pytest.mark.parametrize("points", ["uniform", "tiny", "cluster"])
def test_wide_matches_slabs_and_direct(dtype, w, type_, points, cuda, engine, oracle):
    """Partial tiles; grids of 2 w cells, where the region wraps around; several batches on one
    plane beside planes further apart than a window."""
    rng = np.random.default_rng(10 * w + type_)
    modes = [3, 2, 4] if points == "tiny" else [21, 18, 25]
    pts = [rng.uniform(-4, 4, 700) for _ in range(3)]
    if points == "cluster":
        pts = [np.concatenate([0.3 + rng.uniform(0, 0.01, 500), rng.uniform(-np.pi, np.pi, 30)])
               for _ in range(3)]
    n_in = len(pts[0]) if type_ == 1 else int(np.prod(modes))
    inp = rng.standard_normal(n_in) + 1j * rng.standard_normal(n_in)
    out, info = run_t12(engine, cuda, dtype, -1, pts, inp, modes, type_, n_spread=w)
    assert info["spread_method"] == 3 and info["n_spread"] == w
    slab, info1 = run_t12(engine, cuda, dtype, -1, pts, inp, modes, type_, n_spread=w,
                          spread_method=1)
    assert info1["spread_method"] == 1
    # the same kernel and grid in another order of the sums. Cluster: about n = 500 random
    # strengths on the same cells; the partial sums of an order grow like sqrt(i), each rounded
    # with u = 6e-8, so that the sum of size sqrt(n) carries u n / sqrt(2): relative errors of
    # u sqrt(n / 2) = 1e-6 per order, 2e-6 between two, doubled for the chance of small sums.
    # The slabs take the kernel values from the formula, whose rounded square root (6e-8) is
    # multiplied by beta = 2.3 w: 3 beta 6e-8 over three dimensions on points that share their
    # cells, 6.6e-6 at w = 16; it averages out over uniform ones.
    same = 4e-6 + 3 * 2.3 * w * 6e-8 if points == "cluster" else 2e-6
    assert oracle.rel_l2(out, slab) < (same if dtype == "float32" else 1e-13)
    ref = direct(oracle, type_, -1, pts, inp, modes, dtype)
    assert oracle.rel_l2(out, ref) < width_bound(dtype, w)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_wide_type3_batch(dtype, cuda, engine, oracle):
    """Type 3 with three vectors, and a named tile, which keeps the slabs."""
    torch = cuda
    rng = np.random.default_rng(4)
    M, K, B = 500, 400, 3
    x = [rng.uniform(-2, 2, M).astype(dtype) for _ in range(3)]
    s = [rng.uniform(-3, 3, K).astype(dtype) for _ in range(3)]
    cd = np.complex64 if dtype == "float32" else np.complex128
    c = (rng.standard_normal(M * B) + 1j * rng.standard_normal(M * B)).astype(cd)
    outs = []
    for tile, method in [((0, 0, 0), 3), ((8, 8, 4), 1)]:
        plan = engine.PlanT3(engine.Options(tol=1e-9, tile=tile), 1, M,
                             [torch.from_numpy(a).cuda() for a in x], K,
                             [torch.from_numpy(a).cuda() for a in s], batch_size=B)
        assert plan.info()["spread_method"] == method
        out = torch.zeros(K * B, dtype=getattr(torch, "complex64" if dtype == "float32"
                                               else "complex128"), device="cuda")
        plan.add_input(torch.from_numpy(c).cuda(), M)
        plan.transform(out, K)
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy())
        plan.close()
    assert oracle.rel_l2(outs[0], outs[1]) < (2e-6 if dtype == "float32" else 1e-13)
    ph = sum(a.astype(np.float64)[:, None] * t.astype(np.float64)[None, :] for a, t in zip(x, s))
    ref = np.concatenate([c[b * M:(b + 1) * M].astype(np.complex128) @ np.exp(1j * ph)
                          for b in range(B)])
    assert oracle.rel_l2(outs[0], ref) < (2e-5 if dtype == "float32" else 1e-7)


@pytest.mark.parametrize("dtype,w", [("float64", 10), ("float64", 16), ("float32", 9)])
def test_wide_not_slower_than_slabs_on_small_grids(dtype, w, cuda, engine):
    """On grids of a few columns the z-window kernels take chunks of a few planes, so that they still
    fill the GPU: a pair of transforms of 3e4 points on 32^3 cells in a third (double precision) to a
    fifth of what the shared-memory slabs take, where chunks of 4 w planes took half as long again
    (w = 10)."""
    torch = cuda
    rng = np.random.default_rng(w)
    modes, M = [16, 16, 16], 30_000
    rdt = getattr(torch, dtype)
    cdt = torch.complex64 if dtype == "float32" else torch.complex128
    x = [torch.from_numpy(rng.uniform(-np.pi, np.pi, M)).to(rdt).cuda() for _ in modes]
    c = torch.ones(M, dtype=cdt, device="cuda")
    f = torch.empty(16 ** 3, dtype=cdt, device="cuda")
    ms = {}
    for method in (0, 1):
        plan = engine.Plan(engine.Options(tol=1e-6, n_spread=w, spread_method=method), -1, M, x,
                           modes)
        plan.enable_timing()
        for reps in (3, 20):  # warm-up, then timed
            plan.stage_times()
            for _ in range(reps):
                plan.transform_type_1(c, f, [1, 16, 256])
                plan.transform_type_2(f, [1, 16, 256], c)
        t = plan.stage_times()
        ms[method] = t["spread"][0] + t["interp"][0]
        plan.close()
        c.fill_(1)
    assert ms[0] < 0.7 * ms[1], ms
