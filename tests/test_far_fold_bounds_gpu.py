"""What a sweep leaves out by passing over far folds stays below 2^-36 (FP32c) or 2^-58 (FP64) of the sum of the
absolute terms of every output of every target: column by column, component by component, whatever the near records
add (nothing, where they coincide with the target, weigh in another column only, or are orthogonal to its vector).

Tolerances.  Against the oracle: 1e-4 (FP32c) and 1e-12 (FP64) of the output's own sum of absolute terms: packed
coordinates below 16 are off by 2^-21, exponents of terms at 11 widths by 0.69 (2 11 sqrt(3) 1.2 2^-20 + 2^-16) <
4.2e-5, and in FP64 the same with 2^-53 in place of 2^-24.  Against sums over slices that are too small to pass over
anything, in the same frame and the same folds: FP32 partial sums agree bit by bit, what remains is the bound and the
2^-46 of the compensated additions, 2^-35; FP64 roundings of 9,000 additions at random signs on either side, 2^-53 (95 + 95) < 3e-14.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA = 0.05
ORACLE_TOL = {"fp32c": 1e-4, "fp64": 1e-12}
SLICE_TOL = {"fp32c": 2.0 ** -35, "fp64": 3e-14}


def _kernel(name, precision, sigma=SIGMA):
    from registration_b200 import kernelFunctions as kf
    return kf.Kernel(name=name, sigma=sigma, order=10 if name == "gauss" else 3, precision=precision)


def _factors(name, x, y, sigma=SIGMA):
    """K and K' 2 / (x - y) of every pair (the Laplacian of order 3)."""
    u = np.linalg.norm(x[:, None] - y[None], axis=2) / sigma
    if name == "gauss":
        k = np.exp(-0.5 * u * u)
        return k, -k / sigma ** 2
    e = np.exp(-u)
    return (1 + u * (1 + u * (0.4 + u / 15))) * e, -(0.2 + u * (0.2 + u / 15)) * e / sigma ** 2


def _dev(*a):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in a]


def _near_and_far(n, m, dist, rng):
    """Targets within 0.3 widths, half of the sources as near, the others `dist` widths away."""
    x = SIGMA * rng.uniform(-0.3, 0.3, (n, 3))
    y = SIGMA * rng.uniform(-0.3, 0.3, (m, 3))
    y[m // 2:, 0] += dist * SIGMA
    return x, y


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("name", ["gauss", "laplacian"])
@pytest.mark.parametrize("n,dist", [(1, 8.5), (65, 11.0)])
def test_columns_have_their_own_bounds(precision, name, n, dist):
    """Near sources weigh in column 0 only, far ones in column 1 only."""
    rng = np.random.default_rng(n)
    x, y = _near_and_far(n, 8192, dist, rng)
    b = np.zeros((8192, 3))
    b[:4096, 0] = rng.standard_normal(4096)
    b[4096:, 1] = rng.standard_normal(4096)
    xd, yd, bd = _dev(x, y, b)
    f = _kernel(name, precision).applyK(yd, bd, firstVar=xd).cpu().numpy()
    k, _ = _factors(name, x, y)
    tol = max(ORACLE_TOL[precision], 0 if name == "gauss" else 1e-6)   # (FP32 literals in the Laplacian's tables)
    assert (np.abs(f - k @ b) <= tol * (k @ np.abs(b))).all()


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("name", ["gauss", "laplacian"])
@pytest.mark.parametrize("near", ["coincide", "orthogonal"])
@pytest.mark.parametrize("n,dist", [(1, 8.5), (65, 11.0)])
def test_gradients_whose_near_terms_vanish(precision, name, near, n, dist):
    """Near sources at the very place of the targets, or with <u, v> = 0."""
    rng = np.random.default_rng(n)
    x, y = _near_and_far(n, 8192, dist, rng)
    u, v = np.zeros((n, 3)), rng.standard_normal((8192, 3))
    u[:, 0] = rng.uniform(0.5, 2, n)
    if near == "coincide":
        x[:] = x[0]
        y[:4096] = x[0]
    else:
        v[:4096, 0] = 0.0
    xd, yd, ud, vd = _dev(x, y, u, v)
    g = _kernel(name, precision).applyDiffKT(yd, [ud], [vd], firstVar=xd).cpu().numpy()
    _, k1 = _factors(name, x, y)
    t = (k1 * (u @ v.T))[:, :, None] * (x[:, None] - y[None])
    tol = max(ORACLE_TOL[precision], 0 if name == "gauss" else 1e-6)
    assert (np.abs(g - t.sum(axis=1)) <= tol * np.abs(t).sum(axis=1)).all()


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("n", [6200, 7001])
def test_adjoint_of_orthogonal_clusters(precision, n):
    """Two clusters whose momenta and covectors are orthogonal within each: all there is comes from the other one."""
    import torch
    from registration_b200 import pointEvolution as evol
    rng = np.random.default_rng(n)
    x, _ = _near_and_far(n, 2, 0, rng)
    h = n // 2
    x[h:, 0] += 11 * SIGMA
    a, p = np.zeros((n, 3)), np.zeros((n, 3))
    a[:h, 1], p[h:, 1] = rng.uniform(0.5, 2, h), rng.uniform(0.5, 2, n - h)
    p[:h, 2], a[h:, 2] = rng.uniform(0.5, 2, h), rng.uniform(0.5, 2, n - h)
    xd, ad, pd = _dev(x, a, p)
    pxt, _ = evol.covector(torch.stack([xd, xd]), ad[None], pd, _kernel("gauss", precision), 0.0)
    got = pxt[0].cpu().numpy()[:, 0]   # the component along the line of the clusters, where p has none
    _, k1 = _factors("gauss", x, x)
    t = k1 * (p @ a.T + a @ p.T) * (x[:, None, 0] - x[None, :, 0])
    assert (np.abs(got - t.sum(axis=1)) <= ORACLE_TOL[precision] * np.abs(t).sum(axis=1)).all()


def _cloud(layout, n, m, rng):
    t = np.linspace(0, 1, max(n, m))
    line = np.stack([t, 0.2 * np.sin(9 * t), 0.1 * np.cos(7 * t)], axis=1)
    if layout == "line":
        return line[:n].copy(), line[:m].copy()
    if layout == "flat":           # one coordinate is the same for all
        return line[:n] * [1, 1, 0], line[:m] * [1, 1, 0]
    if layout == "plane":          # two dimensions
        return line[:n, :2].copy(), line[:m, :2].copy()
    if layout == "clusters":       # targets twelve widths away from either cluster of sources
        y = line[:m] * 0.1
        y[m // 2:, 0] += 1.5
        return line[:n] * 0.2 + np.array([0.7, 0.0, 0.0]), y
    return rng.uniform(0, 1, (n, 3)), rng.uniform(0, 1, (m, 3))


def _weights(kind, m, d, rng):
    b = rng.standard_normal((m, d))
    if kind == "steep":
        b *= np.exp(np.linspace(-40, 10, m))[:, None]
    elif kind == "zero":
        b[: m // 2] = 0.0
    elif kind == "tiny":
        b *= 1e-20
    elif kind == "scaled":         # columns of very different size
        b *= np.array([1.0, 1e-12, 1e8])[:d]
    elif kind == "sparse":         # a few records of each column
        b *= rng.uniform(size=b.shape) < 0.02
    return b


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("layout", ["line", "flat", "plane", "clusters", "random"])
@pytest.mark.parametrize("n,m,kind", [(1, 6145, "plain"), (65, 6600, "steep"), (129, 7999, "zero"), (640, 9001, "tiny"),
                                      (129, 9001, "scaled"), (640, 7999, "sparse"), (65, 9001, "plain")])
def test_sums_equal_those_of_small_slices(precision, layout, n, m, kind):
    """Slices of 6,112 sources and one fold of records without weight, which keeps the frame: 192 folds, all counted."""
    import torch
    rng = np.random.default_rng(n + m)
    for name in ("gauss", "laplacian"):
        K = _kernel(name, precision)
        x, y = _cloud(layout, n, m, rng)
        d = x.shape[1]
        b, u = _weights(kind, m, d, rng), rng.standard_normal((n, d))
        corner = np.repeat(np.stack([np.minimum(x.min(0), y.min(0)), np.maximum(x.max(0), y.max(0))]), 16, axis=0)
        zero = np.zeros((32, d))
        pad = -m % 32
        yp, bp = np.concatenate([y, np.repeat(y[-1:], pad, axis=0)]), np.concatenate([b, np.zeros((pad, d))])
        xd, yd, bd, ud = _dev(x, np.concatenate([yp, corner]), np.concatenate([bp, zero]), u)
        f, g = K.applyK(yd, bd, firstVar=xd), K.applyDiffKT(yd, [ud], [bd], firstVar=xd)
        fs, gs = torch.zeros_like(f), torch.zeros_like(g)
        for i in range(0, len(yp), 6112):
            ys, bs = _dev(np.concatenate([yp[i:i + 6112], corner]), np.concatenate([bp[i:i + 6112], zero]))
            fs += K.applyK(ys, bs, firstVar=xd)
            gs += K.applyDiffKT(ys, [ud], [bs], firstVar=xd)
        k, k1 = _factors(name, x, y)
        fabs = k @ np.abs(b)
        gabs = ((np.abs(k1 * (u @ b.T)))[:, :, None] * np.abs(x[:, None] - y[None])).sum(axis=1)
        tol = SLICE_TOL[precision]
        # FP32 terms below the smallest normal number are flushed one by one: they count as nothing on either side
        floor = 1e-38 if precision == "fp32c" else 0.0
        assert (np.abs((f - fs).cpu().numpy()) <= tol * 1.01 * fabs + floor).all(), name
        assert (np.abs((g - gs).cpu().numpy()) <= tol * 1.01 * gabs + floor / SIGMA).all(), name


@pytest.mark.parametrize("precision,tol", [("fp32c", 2e-5), ("fp64", 1e-11)])
@pytest.mark.parametrize("n", [6200, 7001])
def test_shots_of_narrow_kernels(oracle_lib, precision, tol, n):
    """Three steps of a line of points twenty widths long and their adjoint."""
    import torch
    from oracle import lddmm_ref as ref
    from registration_b200 import pointEvolution as evol
    rng = np.random.default_rng(n)
    x, _ = _cloud("line", n, n, rng)
    at = rng.standard_normal((3, n, 3)) * 0.3 / n
    px = rng.standard_normal((n, 3))
    K, RK = _kernel("gauss", precision), ref.Kernel(name="gauss", sigma=SIGMA)
    xd, ad, pd = _dev(x, at, px)
    xt, _ = evol.shoot(xd, ad, K)
    want = ref.landmarkDirectEvolutionEuler(x, at, RK)
    assert np.abs(xt.cpu().numpy() - want).max() <= tol * np.abs(want - x).max()
    pxt, _ = evol.covector(_dev(want)[0], ad, pd, K, 1.0)
    pw = ref.landmarkHamiltonianCovector(x, at, px, RK, 1.0)[0]
    assert np.abs(pxt.cpu().numpy() - pw).max() <= tol * max(np.abs(pw - px).max(), 1e-300)


@pytest.mark.parametrize("precision,tol", [("fp32c", 2e-5), ("fp64", 1e-11)])
@pytest.mark.parametrize("norm", ["current", "measure"])
def test_curve_terms_of_narrow_kernels(oracle_lib, precision, tol, norm):
    """3,301 edges (6,602 sources), forty widths: values and gradients against the oracle, within `tol` of the sums of absolute terms."""
    from oracle import lddmm_ref as ref
    from registration_b200 import curves as cv
    from registration_b200 import geometry as geo
    v, e = geo.ellipse_curve(3301, 1.0, 0.6)
    vt = v * 1.02 + 0.01
    K, RK = _kernel("gauss", precision), ref.Kernel(name="gauss", sigma=SIGMA)
    C, T = cv.Curve(FV=[e, v]), cv.Curve(FV=[e, vt])
    RC, RT = ref.Curve(FV=[e, v]), ref.Curve(FV=[e, vt])
    length = np.linalg.norm(C.lenel, axis=1)
    y, w = np.concatenate([C.centers, T.centers]), np.concatenate([length, 2 * np.linalg.norm(T.lenel, axis=1)])
    k, k1 = _factors("gauss", C.centers, y)
    want = getattr(ref, "curve_" + norm + "NormDef")(RC, RT, RK)
    assert abs(getattr(cv, norm + "NormDef")(C, T, K) - want) <= tol * (length @ (k @ w))
    got, gw = getattr(cv, norm + "NormGradient")(C, T, K), getattr(ref, "curve_" + norm + "NormGradient")(RC, RT, RK)
    d = np.linalg.norm(C.centers[:, None] - y[None], axis=2)
    gmag = (np.abs(k1) * d * w).sum(axis=1) * length + 2 * (k @ w)
    assert np.abs(got - gw).max() <= tol * 4 * gmag.max()


# FP32 shots and adjoints look for far folds from 12,289 points on
@pytest.mark.parametrize("n", [12288, 12289])
def test_large_fp32_shots_of_narrow_kernels(oracle_lib, n):
    test_shots_of_narrow_kernels(oracle_lib, "fp32c", 2e-5, n)


def test_adjoint_of_large_orthogonal_clusters():
    """As test_adjoint_of_orthogonal_clusters; every 37th row is compared."""
    import torch
    from registration_b200 import pointEvolution as evol
    n = 12801
    rng = np.random.default_rng(n)
    x, _ = _near_and_far(n, 2, 0, rng)
    h = n // 2
    x[h:, 0] += 11 * SIGMA
    a, p = np.zeros((n, 3)), np.zeros((n, 3))
    a[:h, 1], p[h:, 1] = rng.uniform(0.5, 2, h), rng.uniform(0.5, 2, n - h)
    p[:h, 2], a[h:, 2] = rng.uniform(0.5, 2, h), rng.uniform(0.5, 2, n - h)
    xd, ad, pd = _dev(x, a, p)
    pxt, _ = evol.covector(torch.stack([xd, xd]), ad[None], pd, _kernel("gauss", "fp32c"), 0.0)
    got = pxt[0].cpu().numpy()[::37, 0]
    y, u, v = x[::37], p[::37], a[::37]
    _, k1 = _factors("gauss", y, x)
    t = k1 * (u @ a.T + v @ p.T) * (y[:, None, 0] - x[None, :, 0])
    assert (np.abs(got - t.sum(axis=1)) <= ORACLE_TOL["fp32c"] * np.abs(t).sum(axis=1)).all()
