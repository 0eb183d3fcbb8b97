"""FP64 sums over a few hundred sources, on both sides of the 384 up to which one thread adds a target's sources in
the reference's order: every output within 5e-13 of its sum of absolute terms (480 roundings of 2^-53 on either side,
1.1e-13, and a few more per term; the oracle's exponential and ours differ by 2^-52 and the exponents, below 60, by
60 2^-52 = 1.3e-14)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA, TOL = 0.2, 5e-13


@pytest.mark.parametrize("m", [383, 384, 385, 416, 417, 480, 481])
@pytest.mark.parametrize("name,order", [("gauss", 10), ("laplacian", 3)])
def test_few_sources(oracle_lib, name, order, m):
    from registration_b200 import kernelFunctions as kf
    rng = np.random.default_rng(m)
    K = kf.Kernel(name=name, sigma=SIGMA, order=order, precision="fp64")
    y, b = rng.uniform(0, 1, (m, 3)), rng.standard_normal((m, 3))
    for n in (1, 65, 300):
        x, a = rng.uniform(0, 1, (n, 3)), rng.standard_normal((n, 3))
        mag = oracle_lib.applyk(x, y, np.abs(b), SIGMA, K.order)
        assert (np.abs(K.applyK(y, b, firstVar=x) - oracle_lib.applyk(x, y, b, SIGMA, K.order)) <= TOL * mag).all()
        # |K' 2 (x - y) <u, v>| <= |u| |v| K |x - y| / sigma^2
        gmag = np.abs(a).max() * 3 * 2 / SIGMA ** 2 * mag.sum(axis=1, keepdims=True)
        want = oracle_lib.applykdifft(x, y, a[None], b[None], SIGMA, K.order)
        assert (np.abs(K.applyDiffKT(y, [a], [b], firstVar=x) - want) <= TOL * gmag).all()
    u, p = rng.standard_normal((2, m, 3))
    size = np.abs(u).max() * np.abs(b).max() * np.abs(p).max() * m / SIGMA ** 4
    for got, want in ((K.applyDiffK(y, u, b), oracle_lib.applykdiff1(y, u, b, SIGMA, K.order)),
                      (K.applyDiffK1and2(y, u, b), oracle_lib.applykdiff1and2(y, u, b, SIGMA, K.order)),
                      (K.applyDDiffK11and12(y, u, b, p), oracle_lib.applykdiff11and12(y, u, b, p, SIGMA, K.order))):
        assert np.abs(got - want).max() <= TOL * size


@pytest.mark.parametrize("n", [384, 385, 480])
def test_epdiff_of_few_points(oracle_lib, n):
    from oracle import lddmm_ref as ref
    from registration_b200 import kernelFunctions as kf
    from registration_b200 import pointEvolution as evol
    rng = np.random.default_rng(n)
    x, a = rng.uniform(0, 1, (n, 3)), 0.01 * rng.standard_normal((n, 3))
    xt, at = evol.landmarkEPDiff(5, x, a, kf.Kernel(name="gauss", sigma=SIGMA, precision="fp64"))[:2]
    xw, aw = ref.landmarkEPDiff(5, x, a, ref.Kernel(name="gauss", sigma=SIGMA))[:2]
    assert np.abs(xt - xw).max() <= 1e-11 and np.abs(at - aw).max() <= 1e-11 * np.abs(aw).max()
