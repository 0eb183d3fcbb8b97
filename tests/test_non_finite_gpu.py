"""FP64 sums with one non-finite coordinate.

The coordinates are packed around the centre of their bounding box, so an infinite or NaN one may make more rows NaN
than the plain formula does (the centre is not finite either); a row that stays finite has to be the plain formula's,
and a row that is NaN there has to be non-finite here.  Rows compare within 1e-12 of the largest finite row (1e-6 for
the Laplacian, whose reference polynomials are FP32 literals).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA = 0.3
BAD = {"inf": np.inf, "-inf": -np.inf, "nan": np.array([0x7FF8000000000000], dtype=np.uint64).view(np.float64)[0],
       "-nan": np.array([0xFFF8000000000000], dtype=np.uint64).view(np.float64)[0]}


def _plain(name, x, y):
    """K of plain FP64 numpy (the Laplacian of order 3)."""
    d = (x[:, None] - y[None]) / SIGMA
    r2 = (d ** 2).sum(axis=2)
    if name == "gauss":
        return np.exp(-0.5 * r2)
    u = np.sqrt(r2)
    return (1 + u * (1 + u * (0.4 + u / 15.0))) * np.exp(-u)


@pytest.mark.parametrize("where", ["target", "source"])
@pytest.mark.parametrize("bad", list(BAD))
@pytest.mark.parametrize("name,order", [("gauss", 10), ("laplacian", 3)])
def test_sums_keep_non_finite_coordinates(name, order, bad, where):
    import torch
    from registration_b200 import kernelFunctions as kf
    rng = np.random.default_rng(3)
    x, y = rng.uniform(0, 1, (257, 3)), rng.uniform(0, 1, (700, 3))
    a, p = rng.standard_normal((700, 3)), rng.standard_normal((257, 3))
    (x if where == "target" else y)[5, 1] = BAD[bad]
    K = kf.Kernel(name=name, sigma=SIGMA, order=order, precision="fp64")
    with np.errstate(all="ignore"):
        k = _plain(name, x, y)
        want = (k[:, :, None] * a[None]).sum(axis=1)
    xd, yd, ad, pd = (torch.from_numpy(t).cuda() for t in (x, y, a, p))
    got = K.applyK(yd, ad, firstVar=xd).cpu().numpy()
    fin = np.isfinite(got).all(axis=1)
    wfin = np.isfinite(want).all(axis=1)
    assert not (fin & ~wfin).any()
    if fin.any():
        assert np.abs(got[fin] - want[fin]).max() <= (1e-12 if name == "gauss" else 1e-6) * np.abs(want[wfin]).max()
    # every term of a gradient sum carries x - y
    bad_rows = ~np.isfinite(x).all(axis=1) | ~np.isfinite(y).all()
    g = K.applyDiffKT(yd, [pd], [ad], firstVar=xd).cpu().numpy()
    assert not np.isfinite(g[bad_rows]).all(axis=1).any()
    # sums over the points themselves: the same coordinate is a target's and a source's
    z = rng.uniform(0, 1, (600, 3))
    z[7, 2] = BAD[bad]
    zd, u, v, w = (torch.from_numpy(t).cuda() for t in (z, *rng.standard_normal((3, 600, 3))))
    for f in (K.applyDiffK(zd, u, v), K.applyDDiffK11and12(zd, u, v, w), K.applyDDiffK11(zd, u, v, w)):
        assert not torch.isfinite(f).all(dim=1).any()   # K' (x - y) of an infinite difference is 0 inf


@pytest.mark.parametrize("bad", list(BAD))
@pytest.mark.parametrize("name,order", [("gauss", 10), ("laplacian", 3)])
def test_shots_keep_non_finite_points(name, order, bad):
    """One point off the scale (600 points: the general path): no other point moves by its momentum."""
    import torch
    from registration_b200 import kernelFunctions as kf
    from registration_b200 import pointEvolution as evol
    rng = np.random.default_rng(4)
    n = 600
    x, a = rng.uniform(0, 1, (n, 3)), 0.01 * rng.standard_normal((1, n, 3))
    x[9, 0] = BAD[bad]
    K = kf.Kernel(name=name, sigma=SIGMA, order=order, precision="fp64")
    xt, energy = evol.shoot(torch.from_numpy(x).cuda(), torch.from_numpy(a).cuda(), K, with_energy=True)
    xt = xt.cpu().numpy()
    with np.errstate(all="ignore"):
        k = _plain(name, x, x)
        want = x + (k[:, :, None] * a[0][None]).sum(axis=1)
    tol = 1e-12 if name == "gauss" else 1e-6
    fin, wfin = np.isfinite(xt[1]).all(axis=1), np.isfinite(want).all(axis=1)
    assert not (fin & ~wfin).any()
    if fin.any():
        assert np.abs(xt[1][fin] - want[fin]).max() <= tol
    assert not np.isfinite(float(energy))   # <a, K a> has the bad row's term
    pxt, _ = evol.covector(torch.from_numpy(np.stack([x, x])).cuda(), torch.from_numpy(a).cuda(),
                           torch.from_numpy(a[0]).cuda(), K, 1.0)
    assert not torch.isfinite(pxt[0]).all(dim=1).any()


@pytest.mark.parametrize("bad", list(BAD))
@pytest.mark.parametrize("norm", ["varifold", "current", "measure"])
def test_data_terms_keep_non_finite_vertices(norm, bad):
    """1,280 cells, one vertex off the scale: neither the value nor the gradient of its cells is a number."""
    import torch
    from registration_b200 import geometry as geo
    from registration_b200 import kernelFunctions as kf
    from registration_b200 import surfaces as sf
    v, f = geo.icosphere(3)
    w = v.copy()
    w[3, 1] = BAD[bad]
    K = kf.Kernel(name="gauss", sigma=SIGMA, precision="fp64")
    S, T = sf.Surface(FV=[f, torch.from_numpy(w).cuda()]), sf.Surface(FV=[f, torch.from_numpy(1.05 * v).cuda()])
    assert not np.isfinite(float(getattr(sf, norm + "NormDef")(S, T, K)))
    g = getattr(sf, norm + "NormGradient")(S, T, K)
    g = g.cpu().numpy() if hasattr(g, "cpu") else np.asarray(g)
    near = np.unique(f[(f == 3).any(axis=1)])
    assert not np.isfinite(g[near]).all(axis=1).any()


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_varifold_normals_of_cells_without_area(precision):
    """Without a floor under the areas the unit normal of a cell without area is 0 / 0 and reaches every cell's sum,
    also those of cells so far away that other folds of that size are passed over (5,120 cells, sigma 0.05)."""
    import torch
    from registration_b200 import _dataterm as dt
    from registration_b200 import geometry as geo
    from registration_b200 import kernelFunctions as kf
    from registration_b200 import surfaces as sf
    v, whole = geo.icosphere(4)
    f = whole.copy()
    f[3000] = f[3000, 0]
    K = kf.Kernel(name="gauss", sigma=0.05, precision=precision)
    S, T = sf.Surface(FV=[f, torch.from_numpy(v).cuda()]), sf.Surface(FV=[whole, 1.01 * v])
    val, g = dt.dataterm("varifold", S.vertices, S.device_shape(), T.centers, T.surfel, K, grad=True, eps1=0.0, eps2=0.0)
    assert not np.isfinite(float(val))
    assert not torch.isfinite(g).all(dim=1).any()
