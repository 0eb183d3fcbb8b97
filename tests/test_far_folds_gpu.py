"""Sweeps pass over folds of 32 sources that are too far from a target group to count.

Every target's sum must stay what the sum over all pairs gives: the far part
that is left out is bounded by 2^-36 (FP32c) or 2^-58 (FP64) of the sum of the
absolute terms, so a row's error is compared with that sum.

Tolerances.  FP32c: packed coordinates below 16 (the cloud spans at most 1.6 =
27 units of the Gaussian's frame, 46 of the Laplacian's) carry 2^-21 each, so a
difference is off by 2^-20 and the exponent of a term at distance r by
2 sqrt(3) r 2^-20 + 4 r^2 2^-24; rows count while their largest terms have r^2 <=
110, which gives 0.69 (3.5e-5 + 2.6e-5) = 4.2e-5, and half of that for the
Laplacian: 1e-4.  FP64: the same with 2^-53 in place of 2^-24 and r^2 / 2 up to
700, on both sides: 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA = 0.05


def _points(layout, n, m, rng):
    """Targets and sources whose memory order follows the shape (so that folds are compact) or not."""
    t = np.linspace(0, 1, max(n, m))
    line = np.stack([t, 0.2 * np.sin(9 * t), 0.1 * np.cos(7 * t)], axis=1)
    if layout == "line":           # a curve of 20 kernel widths
        return line[:n].copy(), line[:m].copy()
    if layout == "clusters":       # targets twelve widths away from either cluster of sources
        y = line[:m] * 0.1
        y[m // 2:, 0] += 1.5
        return line[:n] * 0.2 + np.array([0.7, 0.0, 0.0]), y
    return rng.uniform(0, 1, (n, 3)), rng.uniform(0, 1, (m, 3))   # no order at all


def _weights(kind, m, rng):
    b = rng.standard_normal((m, 3))
    if kind == "steep":            # the first sources weigh next to nothing, the last a lot
        b *= np.exp(np.linspace(-40, 10, m))[:, None]
    if kind == "zero":
        b[: m // 2] = 0.0
    if kind == "tiny":
        b *= 1e-30
    return b


@pytest.mark.parametrize("precision,tol", [("fp32c", 1e-4), ("fp64", 1e-12)])
@pytest.mark.parametrize("name,order", [("gauss", 10), ("laplacian", 3)])
@pytest.mark.parametrize("layout", ["line", "clusters", "random"])
@pytest.mark.parametrize("n,m,kind", [(129, 1023, "plain"), (1, 1057, "steep"), (640, 31, "plain"),
                                      (300, 1600, "zero"), (65, 992, "tiny")])
def test_rows_keep_their_sums(oracle_lib, precision, tol, name, order, layout, n, m, kind):
    import torch
    from oracle import lddmm_ref as ref
    from registration_b200 import kernelFunctions as kf
    rng = np.random.default_rng(n + m)
    x, y = _points(layout, n, m, rng)
    b, p = _weights(kind, m, rng), rng.standard_normal((n, 3))
    K = kf.Kernel(name=name, sigma=SIGMA, order=order, precision=precision)
    xd, yd, bd, pd = (torch.from_numpy(t).cuda() for t in (x, y, b, p))
    dense = ref.kernel_matrix(ref.Kernel(name=name, sigma=SIGMA, order=order), x, y)
    dist = np.linalg.norm(x[:, None] - y[None], axis=2)
    bmax, pmax = np.abs(b).max(axis=1), np.abs(p).max(axis=1)
    cond = dense @ bmax
    # FP32 holds no digits of rows whose terms all lie below 2^-100 of the weights or near the smallest float
    rows = cond > (max(1e-30 * bmax.max(), 1e-36) if precision == "fp32c" else 0.0)
    f = K.applyK(yd, bd, firstVar=xd).cpu().numpy()
    err = np.abs(f - oracle_lib.applyk(x, y, b, SIGMA, K.order)).max(axis=1)
    assert (err[rows] <= tol * cond[rows]).all()
    g = K.applyDiffKT(yd, [pd], [bd], firstVar=xd).cpu().numpy()
    err = np.abs(g - oracle_lib.applykdifft(x, y, p[None], b[None], SIGMA, K.order)).max(axis=1)
    gcond = 3 * pmax * (((dense * dist) @ bmax) / SIGMA ** 2 + cond / SIGMA)
    assert (err[rows] <= tol * gcond[rows]).all()


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_weights_are_never_passed_over(precision, bad):
    """As in the sum over all pairs a bad weight reaches every row of its column, and no other column."""
    import torch
    from registration_b200 import kernelFunctions as kf
    n, m = 300, 2000
    x, y = _points("line", n, m, None)
    b = np.ones((m, 3))
    b[m - 7, 1] = bad
    K = kf.Kernel(name="gauss", sigma=SIGMA, precision=precision)
    f = K.applyK(torch.from_numpy(y).cuda(), torch.from_numpy(b).cuda(), firstVar=torch.from_numpy(x).cuda())
    f = f.cpu().numpy()
    assert not np.isfinite(f[:, 1]).any() and np.isfinite(f[:, [0, 2]]).all()


@pytest.mark.parametrize("precision,tol", [("fp32c", 2e-5), ("fp64", 1e-11)])
@pytest.mark.parametrize("norm", ["varifold", "current", "measure"])
@pytest.mark.parametrize("level", [3, 4])
def test_data_terms_of_narrow_kernels(oracle_lib, precision, tol, norm, level):
    """Values and gradients where most of the sphere is far (1280 and 5120 cells, sigma 0.06), within `tol` of the
    sums of the absolute terms."""
    from oracle import lddmm_ref as ref
    from registration_b200 import geometry as geo
    from registration_b200 import kernelFunctions as kf
    from registration_b200 import surfaces as sf
    rng = np.random.default_rng(level)
    sigma = 0.06
    v, f = geo.icosphere(level)
    vt = geo.bumped_sphere(v, f, 5, 0.3, 0.1, rng)
    K, RK = kf.Kernel(name="gauss", sigma=sigma, precision=precision), ref.Kernel(name="gauss", sigma=sigma)
    S, T = sf.Surface(FV=[f, v]), sf.Surface(FV=[f, vt])
    RS, RT = ref.Surface(FV=[f, v]), ref.Surface(FV=[f, vt])
    sfx = "_pairs" if norm == "varifold" else ""
    area = np.linalg.norm(S.surfel, axis=1)
    y = np.concatenate([S.centers, T.centers])
    w = np.concatenate([area, np.linalg.norm(T.surfel, axis=1)])
    vmag, gmag = 0.0, np.zeros(len(area))
    for k in range(len(area)):
        d = np.linalg.norm(S.centers[k] - y, axis=1)
        kw = 2 * np.exp(-d ** 2 / (2 * sigma ** 2)) * w
        vmag += area[k] * kw.sum()
        gmag[k] = (kw * (area[k] * d / sigma ** 2 + 2 * np.sqrt(area[k]))).sum()
    want = getattr(ref, norm + "NormDef" + sfx)(RS, RT, RK)
    assert abs(getattr(sf, norm + "NormDef")(S, T, K) - want) <= tol * vmag
    g, gw = getattr(sf, norm + "NormGradient")(S, T, K), getattr(ref, norm + "NormGradient" + sfx)(RS, RT, RK)
    assert np.linalg.norm(g - gw) <= tol * 6 * np.linalg.norm(gmag)


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("d,cloud", [(3, "sphere"), (2, "square"), (3, "crowd")])
def test_ordered_target_rows_change_nothing(precision, d, cloud):
    """From 32,768 points on a sum over its own points groups its targets by cells of a grid (or, where over 2,048
    rows share a cell, as they lie).  Same terms and same FP32 partial sums: against the sum with separate targets
    only the far folds left out (2^-36 of the absolute terms) may differ, 1e-9 of the largest row."""
    import torch
    from registration_b200 import kernelFunctions as kf
    from registration_b200 import pointEvolution as evol
    n = 33001
    rng = np.random.default_rng(5)
    x = rng.standard_normal((n, d))
    if cloud == "sphere":
        x /= np.linalg.norm(x, axis=1, keepdims=True)
    elif cloud == "square":
        x = np.stack([np.arange(n) % 182, np.arange(n) // 182], axis=1) / 182.0
    else:
        x *= 0.01
        x[7] = 30.0
    a = rng.standard_normal((n, d))
    K = kf.Kernel(name="gauss", sigma=0.04, precision=precision)
    xd, ad = torch.from_numpy(x).cuda(), torch.from_numpy(a).cuda()
    for got, want in ((K.applyK(xd, ad), K.applyK(xd, ad, firstVar=xd.clone())),
                      (K.applyDiffKT(xd, [ad], [ad]), K.applyDiffKT(xd, [ad], [ad], firstVar=xd.clone()))):
        assert float((got - want).abs().max()) <= 1e-9 * float(want.abs().max())
    # steps of a shot and of its adjoint against the separate sums.  FP32c: one step (later ones are packed in the
    # first step's frame, the separate sums in their own), and two steps against FP64 within the 1e-5 of its shots
    # (not for the crowd, whose outlier at 750 widths costs FP32 coordinates ten bits)
    T = 2 if precision == "fp64" else 1
    at = torch.stack([ad, 0.5 * ad])[:T] * 1e-3
    xt, _ = evol.shoot(xd, at, K, dt=0.5)
    want = xd
    for t in range(T):
        step = 0.5 * K.applyK(want, at[t], firstVar=want.clone())
        want = want + step
        assert float((xt[t + 1] - want).abs().max()) <= 1e-8 * float(step.abs().max())
    # (the adjoint's six-term inner products are added in another order than applyDiffKT's: FP64 only)
    pxt, _ = evol.covector(xt, at, ad, K, 1.0, dt=0.5)
    p = ad
    for t in reversed(range(T if precision == "fp64" else 0)):
        step = 0.5 * K.applyDiffKT(xt[t], [p - 2 * at[t], at[t]], [at[t], p], firstVar=xt[t].clone())
        p = p + step
        assert float((pxt[t] - p).abs().max()) <= 1e-8 * float(step.abs().max())
    if precision == "fp32c" and cloud != "crowd":
        K64 = kf.Kernel(name="gauss", sigma=0.04, precision="fp64")
        at = torch.stack([ad, 0.5 * ad]) * 1e-3
        got, want = evol.shoot(xd, at, K)[0], evol.shoot(xd, at, K64)[0]
        assert float((got - want).norm()) <= 1e-5 * float((want - xd).norm())
        got, ref64 = (evol.covector(want, at, ad, k, 1.0)[0] for k in (K, K64))
        assert float((got - ref64).norm()) <= 1e-5 * float((ref64 - ad).norm())


@pytest.mark.parametrize("name,order", [("gauss", 10), ("laplacian", 3)])
@pytest.mark.parametrize("cloud", ["uniform", "crowd"])
def test_ordered_fp64_sums_equal_unordered_ones(name, order, cloud):
    """FP64 sums of 2^30 pairs and more order both point sets; two halves of the targets stay below that.  The same
    terms in another order: 40,000 roundings of 2^-53 at random signs, 1e-12 of the largest row."""
    import torch
    from registration_b200 import kernelFunctions as kf
    n, m = 33001, 40007
    g = torch.Generator(device="cuda").manual_seed(3)
    opt = dict(dtype=torch.float64, device="cuda", generator=g)
    x, y = torch.rand((n, 3), **opt), torch.rand((m, 3), **opt)
    if cloud == "crowd":
        x, y = 0.01 * x, 0.01 * y
        x[5], y[11] = 2.0, -2.0
    a, p = torch.randn((m, 3), **opt), torch.randn((n, 3), **opt)
    K = kf.Kernel(name=name, sigma=0.05, order=order, precision="fp64")
    h = n // 2
    f = K.applyK(y, a, firstVar=x)
    want = torch.cat([K.applyK(y, a, firstVar=x[:h]), K.applyK(y, a, firstVar=x[h:])])
    assert float((f - want).abs().max()) <= 1e-12 * float(want.abs().max())
    f = K.applyDiffKT(y, [p], [a], firstVar=x)
    want = torch.cat([K.applyDiffKT(y, [p[:h]], [a], firstVar=x[:h]), K.applyDiffKT(y, [p[h:]], [a], firstVar=x[h:])])
    assert float((f - want).abs().max()) <= 1e-12 * float(want.abs().max())
