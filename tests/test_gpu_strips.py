"""1D and 2D transforms on strip-sorted points (method 1 with the automatic tile, csrc/strip.cu)
against the FP64 direct sums and the thread-per-point method, at the sizes where its runs, batches,
strips and windows end."""
import numpy as np
import pytest

from test_gpu_methods import direct, run_t12, width_bound

pytestmark = pytest.mark.gpu


def _check(engine, cuda, oracle, dtype, w, type_, pts, modes, **opt):
    rng = np.random.default_rng(w)
    M = len(pts[0])
    n_in = M if type_ == 1 else int(np.prod(modes))
    inp = rng.standard_normal(n_in) + 1j * rng.standard_normal(n_in)
    out, info = run_t12(engine, cuda, dtype, 1, pts, inp, modes, type_, n_spread=w, **opt)
    assert info["spread_method"] == 1
    tpp, _ = run_t12(engine, cuda, dtype, 1, pts, inp, modes, type_, n_spread=w, spread_method=2,
                     **opt)
    ref = direct(oracle, type_, 1, pts, inp, modes, dtype)
    # the same kernel and grid: another order of the sums. Single precision: the values are sums
    # of up to M w^d terms of relative error 6e-8 (measured 2e-7); double: 1e-16 (measured 1e-15)
    assert oracle.rel_l2(out, tpp) < (2e-6 if dtype == "float32" else 1e-13)
    if opt.get("upsampfac", 2.0) == 2.0:
        assert oracle.rel_l2(out, ref) < width_bound(dtype, w)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("w", list(range(2, 17)))
@pytest.mark.parametrize("type_", [1, 2])
@pytest.mark.parametrize("modes,M", [([41], 777), ([20, 17], 777), ([20, 17], 80)])
def test_widths(dtype, w, type_, modes, M, cuda, engine, oracle):
    """Every width; grids of a few windows (strips and rows wrap around); 80 points on 40 x 34
    cells are spread one by one, 777 through windows."""
    rng = np.random.default_rng(w + type_)
    pts = [rng.uniform(-4, 4, M) for _ in modes]
    _check(engine, cuda, oracle, dtype, w, type_, pts, modes)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("M", [1, 7, 8, 9, 15, 16, 17, 255, 256, 257, 2049])
@pytest.mark.parametrize("type_", [1, 2])
@pytest.mark.parametrize("modes", [[3], [500], [2, 3], [61, 45]])
def test_run_lengths(dtype, M, type_, modes, cuda, engine, oracle):
    """Point counts around the batch, run and CTA sizes, on sparse and on tiny grids (narrower
    than a strip's region)."""
    rng = np.random.default_rng(M)
    pts = [rng.uniform(-np.pi, np.pi, M) for _ in modes]
    _check(engine, cuda, oracle, dtype, 6, type_, pts, modes)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("type_", [1, 2])
@pytest.mark.parametrize("M", [60, 3000])
def test_odd_grid(dtype, type_, M, cuda, engine, oracle):
    """An odd fine grid (37 x 31): rows start 8-byte aligned only in single precision."""
    rng = np.random.default_rng(3)
    pts = [rng.uniform(-np.pi, np.pi, M) for _ in range(2)]
    _check(engine, cuda, oracle, dtype, 7, type_, pts, [25, 21], upsampfac=1.5)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("type_", [1, 2])
@pytest.mark.parametrize("modes", [[64], [40, 30]])
def test_clusters(dtype, type_, modes, cuda, engine, oracle):
    """Runs that lie in one cell, and runs that jump over rows, strips and the periodic edge."""
    rng = np.random.default_rng(5)
    pts = [np.concatenate([np.full(4000, 0.3), np.full(50, np.pi - 1e-4), np.full(50, -np.pi),
                           rng.uniform(-np.pi, np.pi, 100)]) for _ in modes]
    _check(engine, cuda, oracle, dtype, 6, type_, pts, modes)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("w", [2, 5, 7, 8, 11])
@pytest.mark.parametrize("share", [1.0, 0.6, 0.05])
def test_clusters_on_sparse_grids(dtype, w, share, cuda, engine, oracle):
    """Points that are sparse on average (17 cells a point) of which a share lies in a few cells:
    the crowded places go through windows, the rest is added directly, and all through windows
    where nearly all is crowded. Against the thread-per-point method in double precision."""
    rng = np.random.default_rng(w)
    M, modes = 400_003, [1300, 1301]
    n = int(share * M)
    pts = [np.concatenate([0.7 + 0.005 * rng.standard_normal(n),
                           rng.uniform(-np.pi, np.pi, M - n)]).astype(dtype) for _ in modes]
    c = rng.uniform(0.5, 1.5, M).astype(dtype).astype(complex)
    out, info = run_t12(engine, cuda, dtype, 1, pts, c, modes, 1, n_spread=w)
    assert info["spread_method"] == 1
    ref, _ = run_t12(engine, cuda, "float64", 1, pts, c, modes, 1, n_spread=w, spread_method=2)
    # Strengths of one sign, so that sums grow. Single precision: a cell's sum is made of runs of
    # 64 or 128 values in registers, up to M / 64 = 6250 of them added to the grid: rounding errors
    # of u = 6e-8 at random in growing sums, u (sqrt(128) + sqrt(6250)) / sqrt(3) = 3.1e-6, and the
    # kernel values' 3e-7. Added one by one, the 4e5 values leave 6e-6 (a share of 0.05) to 3e-4.
    # Double precision: 1e-16 in place of u, the values one by one in the reference.
    assert oracle.rel_l2(out, ref) < (4e-6 if dtype == "float32" else 1e-13)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("w,type_", [(2, 1), (7, 1), (7, 2), (16, 1)])
@pytest.mark.parametrize("points", ["uniform", "band", "cell"])
@pytest.mark.parametrize("modes", [[2_500_003], [3000, 2900]])
def test_few_points_on_large_grids(dtype, w, points, modes, type_, cuda, engine, oracle):
    """Few points on a large grid: the strips' bins are widened, so that their number follows that
    of the points. "band": some of them lie closely, in any order within the wide bins (2 points a
    cell in 1D); "cell": most of them in one cell, for which the bins are narrowed again."""
    rng = np.random.default_rng(w)
    M = 9000
    near = {"uniform": 0, "band": 4000, "cell": 6000}[points]
    span = {"uniform": 0, "band": 8e-4 * np.pi if len(modes) == 1 else 0.1, "cell": 1e-6}[points]
    pts = [np.concatenate([rng.uniform(0.5, 0.5 + span, near), rng.uniform(-4, 4, M - near)])
           for _ in modes]
    pts[0][-1], pts[0][-2] = np.pi - 1e-6, -np.pi  # the periodic edge
    n_in = M if type_ == 1 else int(np.prod(modes))
    inp = rng.standard_normal(n_in) + 1j * rng.standard_normal(n_in)
    out, _ = run_t12(engine, cuda, dtype, 1, pts, inp, modes, type_, n_spread=w)
    pts = [p.astype(dtype) for p in pts]
    ref, _ = run_t12(engine, cuda, "float64", 1, pts, inp, modes, type_, n_spread=w,
                     spread_method=2)
    # Single precision: sums of up to 6000 values, u sqrt(6000 / 2) = 3.3e-6 at random signs if added
    # one by one (u = 6e-8), and 16 of them at once at least here: 8e-7; the kernel values' 1e-7 and
    # the rounding of beta, which both sides deconvolve by their own value
    assert oracle.rel_l2(out, ref) < (2e-6 if dtype == "float32" else 1e-13)


@pytest.mark.parametrize("modes,tile", [([4_000_003], (512, 0, 0)), ([4000, 3800], (64, 16, 0))])
def test_bins_follow_the_points(modes, tile, cuda, engine):
    """A plan of few points holds no more than 64 bytes a point, or the 16 MB of 2^21 bins, above
    what it holds with the tiles of the shared-memory kernels."""
    M = 9000
    x = [cuda.rand(M, device="cuda") * 6 - 3 for _ in modes]
    held = []
    for t in [(0, 0, 0), tile]:
        plan = engine.Plan(engine.Options(tol=1e-6, tile=t), -1, M, x, modes)
        held.append(plan.info()["device_bytes"])
        plan.close()
    # one byte of flags per 128 points, the scan's block sums and roundings up besides
    assert held[0] <= held[1] + max(64 * M, 8 * 2 ** 21) + 65536


@pytest.mark.parametrize("w", [2, 4, 7, 10, 16])
@pytest.mark.parametrize("modes", [[100], [40, 31]])
def test_many_points_in_a_few_cells(w, modes, cuda, engine, oracle):
    """Millions of strengths of one sign in a few cells, single precision: runs are longer and
    the runs of a warp summed before they go to the grid."""
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(w)
    M = 12_000_000
    pts = [(0.7 + 0.02 * torch.randn(M, generator=gen, device="cuda")) for _ in modes]
    c = torch.rand(M, generator=gen, device="cuda").to(torch.complex64)
    out = []
    for dtype, opt in [(torch.float32, {}), (torch.float64, {"spread_method": 2})]:
        cd = torch.complex64 if dtype == torch.float32 else torch.complex128
        plan = engine.Plan(engine.Options(tol=1e-6, n_spread=w, **opt), 1, M,
                           [x.to(dtype) for x in pts], modes)
        f = torch.empty(int(np.prod(modes)), dtype=cd, device="cuda")
        plan.transform_type_1(c.to(cd), f, [1] + modes[:1][:len(modes) - 1])
        torch.cuda.synchronize()
        out.append(f.cpu().numpy())
        plan.close()
    # A run sums M / (148 24 (32 // w)) values one by one, 211 at w = 2 to 1690 at w = 16, and the
    # sums of 148 24 = 3552 warps are added to a cell at most: rounding errors of u = 6e-8 at random
    # in growing sums, u (sqrt(1690) + sqrt(3552)) / sqrt(3) = 3.5e-6; the kernel values' 3e-7
    assert oracle.rel_l2(out[0], out[1]) < 4e-6


def spectrum_ratio(beta, w, upsampfac):
    x = np.linspace(-w / 2, w / 2, 20001)
    phi = np.exp(beta * (np.sqrt(np.maximum(0, 1 - 4 * x * x / w ** 2)) - 1))
    return phi.sum() / (phi * np.cos(np.pi / upsampfac * x)).sum()


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("w", [2, 3, 7, 8, 11])
@pytest.mark.parametrize("upsampfac", [1.25, 2.0, 8.0])
@pytest.mark.parametrize("type_", [1, 2])
@pytest.mark.parametrize("modes", [[41], [12, 10, 9]])
def test_kernel_polynomials(dtype, w, upsampfac, type_, modes, cuda, engine, oracle):
    """Kernel values by polynomials (the default kernels) against the formula (method 2), over the
    shapes of the kernel: the smallest upsampling leaves the largest edge value, the largest the
    steepest pieces (w = 3 then stays with the formula in single precision)."""
    rng = np.random.default_rng(w)
    pts = [rng.uniform(-np.pi, np.pi, 500) for _ in modes]
    n_in = 500 if type_ == 1 else int(np.prod(modes))
    inp = rng.standard_normal(n_in) + 1j * rng.standard_normal(n_in)
    a, _ = run_t12(engine, cuda, dtype, 1, pts, inp, modes, type_, n_spread=w, upsampfac=upsampfac)
    b, info = run_t12(engine, cuda, dtype, 1, pts, inp, modes, type_, n_spread=w,
                      upsampfac=upsampfac, spread_method=2)
    assert info["spread_method"] == 2
    # Single precision: a weight is off by up to 3e-7 of its value (the formula's square root is
    # rounded before it is multiplied by beta), and the deconvolution scales the outermost modes up
    # by phi_hat(0) / phi_hat(pi / upsampfac), 153 at w = 11 and upsampling 1.25. Double: 1e-15.
    up = spectrum_ratio(info["es_beta"], w, upsampfac)
    assert oracle.rel_l2(a, b) < (3e-7 * max(10, up) if dtype == "float32" else 1e-15 * max(100, up))
