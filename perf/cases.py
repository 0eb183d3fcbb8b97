"""The work that users of the point-LDDMM framework have it do, as measured cases.

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges,
``prepare(case, seed)`` what a program holds before the call, ``run(state)`` one
pass through the public entry points, ``work(case)`` the bytes and operations
the pass cannot do without, and ``exact(case, seed)`` its outputs in 64 bits by
plain dense torch.

Kinds of work:

* ``sum``       one kernel sum, ``Kernel.applyK`` or ``Kernel.applyDiffKT``, on
                points uniform in the unit cube (the kernel-sum sweep, 1k to 1M);
* ``gradient``  ``landmarkHamiltonianGradient``: shot and adjoint of a surface's
                vertices, what a matching iteration asks for;
* ``norm``      one data-attachment value or gradient of a deformed surface
                against its target;
* ``objective`` the differentiable objective, forward and backward;
* ``match``     a whole curve match of a few iterations, host loop included;
* ``template``  a trial value and a gradient of template estimation, whose
                subjects share ragged launches (the serving engine's kernels).

Surfaces are icospheres (or the patch of the V vertices nearest to an axis, for
sizes between the subdivisions) with seeded Gaussian bumps as targets and smooth
momenta that move the surface by about a tenth of its radius.
"""
import logging
import math

import numpy as np
import torch

from registration_b200 import autograd as ag
from registration_b200 import curveMatching as CM
from registration_b200 import curves as cv
from registration_b200 import geometry as geo
from registration_b200 import kernelFunctions as kf
from registration_b200 import pointEvolution as evol
from registration_b200 import surfaceMatching as SM
from registration_b200 import surfaceTemplate as ST
from registration_b200 import surfaces as sf

AXIS = np.array([0.36, 0.48, 0.8])
_MESHES = {}


def listed():
    return [
        # a small interactive match: 256-vertex curve, ten conjugate-gradient iterations, host loop included
        dict(name="match_curve_256", kind="match", n=256, sigma=0.5, sigma_dist=0.5, iters=10),
        # the smallest kernel sum of the sweep: launches and latency
        dict(name="applyk_1k", kind="sum", op="applyK", n=1024, m=1024, kernel="gauss", sigma=0.05, precision="fp32c"),
        # the headline kernel sum
        dict(name="applyk_1m", kind="sum", op="applyK", n=1 << 20, m=1 << 20, kernel="gauss", sigma=0.05,
             precision="fp32c"),
        # gradient sum of the Laplacian kernel between two sets of ragged sizes
        dict(name="diffkt_laplacian_100k", kind="sum", op="applyDiffKT", n=100003, m=131072, kernel="laplacian",
             sigma=0.05, precision="fp32c"),
        # the plain FP64 path of the same sums
        dict(name="applyk_fp64_64k", kind="sum", op="applyK", n=65536, m=65536, kernel="gauss", sigma=0.05,
             precision="fp64"),
        # shot and adjoint of a small served surface
        dict(name="gradient_3k", kind="gradient", n=3166, sigma=0.12, steps=10, precision="fp32c"),
        # shot and adjoint of the surface-matching configuration
        dict(name="gradient_10k", kind="gradient", n=10242, sigma=0.2, steps=10, precision="fp32c"),
        # the FP64 data-term value that the line search compares, same configuration
        dict(name="varifold_value_fp64_10k", kind="norm", norm="varifold", grad=False, n=10242, sigma=0.1,
             precision="fp64"),
        # its FP32c gradient, once per iteration
        dict(name="varifold_gradient_10k", kind="norm", norm="varifold", grad=True, n=10242, sigma=0.1,
             precision="fp32c"),
        # the data-term value of the largest served surfaces
        dict(name="varifold_value_50k", kind="norm", norm="varifold", grad=False, n=50000, sigma=0.05,
             precision="fp32c"),
        # the differentiable objective on a large surface: checkpointed trajectory, current data term
        dict(name="objective_40k", kind="objective", norm="current", n=40962, sigma=0.05, sigma_dist=0.02, steps=20,
             checkpoint=5, precision="fp32c"),
        # one trial and one gradient of template estimation, eight subjects
        dict(name="template_8x2562", kind="template", n=2562, subjects=8, sigma=0.2, sigma_dist=0.1, steps=10),
    ]


def _size(rng, lo, hi):
    """An odd or ragged size, spread over the logarithm of the range."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("match", "sum", "sum", "sum", "gradient", "gradient", "norm", "norm", "norm", "objective",
                       "template"))
    sd = round(rng.uniform(0.05, 0.3), 3)   # deformation widths of the served stream; data-term width half of it
    prec = "fp64" if rng.random() < 0.3 else "fp32c"
    if kind == "match":
        return dict(kind=kind, n=_size(rng, 48, 500), sigma=0.5, sigma_dist=round(rng.uniform(0.2, 0.6), 3),
                    iters=rng.randint(3, 10))
    if kind == "sum":
        kern = rng.choice(("gauss", "laplacian"))
        op = rng.choice(("applyK", "applyDiffKT"))
        top = 1 << 17 if prec == "fp64" else 1 << 19
        return dict(kind=kind, op=op, n=_size(rng, 200, top), m=_size(rng, 200, top), kernel=kern,
                    sigma=round(rng.uniform(0.03, 0.2), 3), precision=prec)
    if kind == "gradient":
        return dict(kind=kind, n=_size(rng, 300, 15000 if prec == "fp64" else 50000), sigma=sd, steps=10,
                    precision=prec)
    if kind == "norm":
        return dict(kind=kind, norm=rng.choice(("varifold", "varifold", "current", "measure")),
                    grad=rng.random() < 0.4, n=_size(rng, 300, 50000), sigma=round(sd / 2, 4), precision=prec)
    if kind == "objective":
        return dict(kind=kind, norm=rng.choice(("varifold", "current")), n=_size(rng, 600, 40000), sigma=sd,
                    sigma_dist=round(sd / 2, 4), steps=10, checkpoint=rng.choice((2, 5)), precision=prec)
    return dict(kind=kind, n=_size(rng, 400, 6000), subjects=rng.randint(2, 8), sigma=sd, sigma_dist=round(sd / 2, 4),
                steps=10)


# ---- inputs ---------------------------------------------------------------------------------
def _mesh(n):
    """The icosphere of n vertices, or the patch of the n vertices of the next finer one nearest to AXIS."""
    if n not in _MESHES:
        level = next(k for k in range(12) if 10 * 4 ** k + 2 >= n)
        key = ("sphere", level)
        if key not in _MESHES:
            _MESHES[key] = geo.icosphere(level)
        v, f = _MESHES[key]
        if n < len(v):
            keep = np.zeros(len(v), dtype=bool)
            keep[np.argsort(-(v @ AXIS), kind="stable")[:n]] = True
            new = np.cumsum(keep) - 1
            v, f = v[keep], new[f[keep[f].all(axis=1)]]
        _MESHES[n] = (v, f)
    return _MESHES[n]


def _bumps(v, rng, count, width, amp):
    """A smooth scalar field on the sphere: a sum of seeded Gaussian bumps."""
    c = rng.standard_normal((count, 3))
    c /= np.linalg.norm(c, axis=1, keepdims=True)
    a = rng.uniform(-amp, amp, count)
    out = np.zeros(len(v))
    for i in range(count):
        out += a[i] * np.exp(-((v - c[i]) ** 2).sum(axis=1) / (2 * width ** 2))
    return out


def _surface(case, seed):
    """(template vertices, faces, target vertices): the target moved along the normals by 8 bumps."""
    rng = np.random.default_rng([seed, 1])
    v, f = _mesh(case["n"])
    return v, f, v * (1 + _bumps(v, rng, 8, 0.25, 0.15))[:, None]


def _momenta(case, v, seed, steps, scale=1.0):
    """Momenta (steps, n, 3) whose flow moves the points by about a tenth of the radius."""
    rng = np.random.default_rng([seed, 2])
    rows = 1.0 + 0.5 * len(v) * case["sigma"] ** 2   # about the row sum of the kernel matrix
    field = _bumps(v, rng, 12, 0.4, 1.0)
    at = np.empty((steps,) + v.shape)
    for t in range(steps):
        at[t] = (0.1 * scale / rows) * (field[:, None] * v + 0.3 * rng.standard_normal(v.shape))
    return at


def _kernel(sigma, precision, name="gauss"):
    return kf.Kernel(name=name, sigma=sigma, order=3 if name == "laplacian" else 10, precision=precision)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _sum_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    opt = dict(dtype=torch.float64, device="cuda", generator=g)
    x = torch.rand((case["n"], 3), **opt)
    y = torch.rand((case["m"], 3), **opt)
    a = torch.randn((case["m"], 3), **opt)
    p = torch.randn((case["n"], 3), **opt)
    return x, y, a, p


def _curves(case, seed):
    rng = np.random.default_rng([seed, 3])
    v, _ = geo.ellipse_curve(case["n"], 1.0, 0.6)
    vt, _ = geo.bumped_curve(v, 4, 0.3, 0.1, rng, n_out=case["n"])
    return v, vt


def _template_inputs(case, seed):
    rng = np.random.default_rng([seed, 4])
    v, f = _mesh(case["n"])
    targets = [v * (1 + _bumps(v, rng, 8, 0.25, 0.15))[:, None] for _ in range(case["subjects"])]
    T, K = case["steps"], case["subjects"]
    prior = _momenta(case, v, seed, T, 0.3)
    stack = np.stack([_momenta(case, v, 1000 * seed + k, T, 0.5) for k in range(K)])
    dprior = _momenta(case, v, 1000 * seed + 101, T, 0.3)
    dstack = np.stack([_momenta(case, v, 1000 * seed + 201 + k, T, 0.5) for k in range(K)])
    return v, f, targets, prior, stack, dprior, dstack


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sum":
        x, y, a, p = _sum_inputs(case, seed)
        return dict(case=case, K=_kernel(case["sigma"], case["precision"], case["kernel"]), x=x, y=y, a=a, p=p)
    if kind == "match":
        logging.disable(logging.INFO)
        v, vt = _curves(case, seed)
        param = CM.CurveMatchingParam(timeStep=0.1, KparDiff=_kernel(case["sigma"], "fp32c"),
                                      KparDist=_kernel(case["sigma_dist"], "fp32c"), sigmaError=0.02,
                                      errorType="current")
        return dict(case=case, param=param, template=cv.Curve(pointSet=v), target=cv.Curve(pointSet=vt))
    if kind == "template":
        v, f, targets, prior, stack, dprior, dstack = _template_inputs(case, seed)
        param = SM.SurfaceMatchingParam(timeStep=1.0 / case["steps"], KparDiff=_kernel(case["sigma"], "fp32c"),
                                        KparDist=_kernel(case["sigma_dist"], "fp32c"), sigmaError=0.1,
                                        errorType="varifold")
        st = ST.SurfaceTemplate(HyperTmpl=sf.Surface(FV=[f, v]), Targets=[sf.Surface(FV=[f, t]) for t in targets],
                                param=param, verb=False)
        st.at, st.atAll = _dev(prior), _dev(stack)
        st.objectiveFun()
        return dict(case=case, st=st, dir=ST.Direction(_dev(dprior), _dev(dstack)))
    v, f, vt = _surface(case, seed)
    if kind == "gradient":
        rng = np.random.default_rng([seed, 5])
        px = (_bumps(v, rng, 8, 0.25, 1.0)[:, None] * v + 0.1 * rng.standard_normal(v.shape)) / len(v)
        return dict(case=case, K=_kernel(case["sigma"], case["precision"]), x0=_dev(v),
                    at=_dev(_momenta(case, v, seed, case["steps"])), px1=_dev(px))
    if kind == "norm":
        rng = np.random.default_rng([seed, 6])
        xdef = v * (1 + _bumps(v, rng, 8, 0.3, 0.08))[:, None]
        fv = sf.Surface(FV=[f, _dev(xdef)])
        tgt = sf.Surface(FV=[f, _dev(vt)])
        fv.device_shape()
        name = case["norm"] + ("NormGradient" if case["grad"] else "NormDef")
        return dict(case=case, K=_kernel(case["sigma"], case["precision"]), fv=fv, tgt=tgt, call=getattr(sf, name))
    geom = ag.Geometry(sf.Surface(FV=[f, v]), sf.Surface(FV=[f, vt]), _kernel(case["sigma"], case["precision"]),
                       _kernel(case["sigma_dist"], case["precision"]), case["norm"])
    return dict(case=case, geom=geom, x0=_dev(v).requires_grad_(True),
                at=_dev(_momenta(case, v, seed, case["steps"])).requires_grad_(True))


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sum":
        if case["op"] == "applyK":
            return state["K"].applyK(state["y"], state["a"], firstVar=state["x"])
        return state["K"].applyDiffKT(state["y"], [state["p"]], [state["a"]], firstVar=state["x"])
    if kind == "gradient":
        return evol.landmarkHamiltonianGradient(state["x0"], state["at"], state["px1"], state["K"], 1.0,
                                                getCovector=True)
    if kind == "norm":
        return state["call"](state["fv"], state["tgt"], state["K"])
    if kind == "objective":
        at, x0 = state["at"], state["x0"]
        E = ag.lddmm_objective(at, x0, state["geom"], checkpoint_every=case["checkpoint"])
        gat, gx0 = torch.autograd.grad(E, (at, x0))
        return E, gat, gx0
    if kind == "match":
        cm = CM.CurveMatching(Template=state["template"], Target=state["target"], param=state["param"],
                              maxIter=case["iters"], verb=False)
        cm.optimizeMatching()
        return cm.obj, cm.at, cm.xt
    st = state["st"]
    value = st.updateTry(state["dir"], 0.5)
    grd = st.getGradient(st.gradCoeff)
    return float(value), grd.prior, grd.stack


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    """Operations per pair: 8 for the squared distance (3 dimensions), 1 exponential, 2 per accumulated value and
    per term of an inner product; bytes: each input read once, each output written once."""
    kind, n = case["kind"], case["n"]
    lap = 6 if case.get("kernel") == "laplacian" else 0
    if kind == "sum":
        per = 15 + lap + (6 if case["op"] == "applyDiffKT" else 0)
        m = case["m"]
        return {"bytes": 8 * 3 * (2 * n + 2 * m) + (24 * n if case["op"] == "applyDiffKT" else 0),
                "flops": float(n) * m * per}
    if kind == "match":
        T, it = 10, case["iters"]
        # an iteration: some eleven trial steps (shot and value), one gradient, two products
        return {"bytes": 8 * 2 * n * (4 + T), "flops": float(n) * n * it * (11 * (T * 11 + 24) + T * 19 + 30 + T * 22)}
    f = len(_mesh(n)[1])
    pairs_norm = 1.5 * float(f) * f
    shot = lambda T: float(n) * n * 15 * T          # noqa: E731
    adjoint = lambda T: float(n) * n * 28 * T       # noqa: E731
    if kind == "gradient":
        T = case["steps"]
        return {"bytes": 8 * 3 * n * (1 + T + 1 + 2 * (T + 1) + T), "flops": shot(T) + adjoint(T)}
    if kind == "norm":
        per = {"varifold": 19, "current": 15, "measure": 11}[case["norm"]] + (18 if case["grad"] else 0)
        return {"bytes": 24 * n + 24 * f + 48 * f + (24 * n if case["grad"] else 8),
                "flops": (2.0 * f * f if case["grad"] else pairs_norm) * per}
    if kind == "objective":
        T = case["steps"]
        per = 19 if case["norm"] == "varifold" else 15
        return {"bytes": 24 * n * (2 * T + 2) + 72 * f,
                "flops": 2 * shot(T) + adjoint(T) + pairs_norm * per + 2.0 * f * f * (per + 18)}
    T, K = case["steps"], case["subjects"]
    return {"bytes": 24 * n * T * (K + 1) * 4,
            "flops": (K + 1) * (shot(T) + adjoint(T)) + K * (pairs_norm * 19 + 2.0 * f * f * 37)}


# ---- the same outputs in 64 bits, by plain torch -----------------------------------------------
# The Laplacian polynomials carry the coefficients of the single-precision literals that the sums are defined by.
_P3 = [1.0, 1.0, float(np.float32(0.4)), float(np.float32(1.0) / np.float32(15.0))]
_Q3 = [float(np.float32(1.0) / np.float32(5.0))] * 2 + [float(np.float32(1.0) / np.float32(15.0))]


def _blocks(n, m):
    step = max(1, int(1.5e8 // max(1, m)))
    return range(0, n, step), step


def _dist2(x, y):
    r2 = (x[:, None, 0] - y[None, :, 0]) ** 2
    for j in range(1, x.shape[1]):
        r2 += (x[:, None, j] - y[None, :, j]) ** 2
    return r2


def _kval(r2, sigma, lap):
    if not lap:
        return torch.exp(r2 / (-2 * sigma ** 2))
    u = torch.sqrt(r2) / sigma
    return (_P3[0] + u * (_P3[1] + u * (_P3[2] + u * _P3[3]))) * torch.exp(-u)


def _kdif(r2, sigma, lap):
    """K' in K = K(r^2): the gradient of K is 2 K' (x - y)."""
    if not lap:
        return torch.exp(r2 / (-2 * sigma ** 2)) / (-2 * sigma ** 2)
    u = torch.sqrt(r2) / sigma
    return (_Q3[0] + u * (_Q3[1] + u * _Q3[2])) * torch.exp(-u) / (-2 * sigma ** 2)


def _apply(x, y, b, sigma, lap=False):
    out = torch.empty((x.shape[0], b.shape[1]), dtype=torch.float64, device=x.device)
    rows, step = _blocks(x.shape[0], y.shape[0])
    for i in rows:
        out[i:i + step] = _kval(_dist2(x[i:i + step], y), sigma, lap) @ b
    return out


def _apply_diff(x, y, u, w, sigma, lap=False):
    """sum_l K' 2 (x_k - y_l) <u_k, w_l>"""
    out = torch.empty_like(x)
    rows, step = _blocks(x.shape[0], y.shape[0])
    for i in rows:
        g = _kdif(_dist2(x[i:i + step], y), sigma, lap) * (u[i:i + step] @ w.T)
        out[i:i + step] = 2 * (x[i:i + step] * g.sum(dim=1, keepdim=True) - g @ y)
    return out


def _shoot(x0, at, sigma, dt):
    xt, e = [x0], 0.0
    for a in at:
        v = _apply(xt[-1], xt[-1], a, sigma)
        e = e + dt * (a * v).sum()
        xt.append(xt[-1] + dt * v)
    return torch.stack(xt), e


def _adjoint(xt, at, px1, sigma, dt):
    T = len(at)
    pxt, dat = [px1], []
    for t in reversed(range(T)):
        p, a = pxt[0], at[t]
        dat.insert(0, 2 * a - p)
        f = _apply_diff(xt[t], xt[t], torch.cat([p - 2 * a, a], 1), torch.cat([a, p], 1), sigma)
        pxt.insert(0, p + dt * f)
    return torch.stack(pxt), torch.stack(dat)


def _cells(v, f):
    x = [v[f[:, j]] for j in range(3)]
    return (x[0] + x[1] + x[2]) / 3, torch.linalg.cross(x[1] - x[0], x[2] - x[0])


def _weights(norm, s1, s2):
    a1 = torch.sqrt((s1 ** 2).sum(1, keepdim=True) + 1e-10)
    a2 = torch.sqrt((s2 ** 2).sum(1, keepdim=True) + 1e-10)
    if norm == "current":
        return s1 @ s2.T
    if norm == "measure":
        return a1 @ a2.T
    return (1 + ((s1 / a1) @ (s2 / a2).T) ** 2) * (a1 @ a2.T)


def _norm(norm, v, f, c2, s2, sigma):
    """<S1,S1> - 2 <S1,S2>; its gradient (that of |S1 - S2|^2) by automatic differentiation, block by block."""
    c1, s1 = _cells(v, f)
    total, rows = 0.0, _blocks(len(c1), len(c1) + len(c2))
    for i in rows[0]:
        k = slice(i, i + rows[1])
        total = total + (_kval(_dist2(c1[k], c1), sigma, False) * _weights(norm, s1[k], s1)).sum()
        total = total - 2 * (_kval(_dist2(c1[k], c2), sigma, False) * _weights(norm, s1[k], s2)).sum()
    return total


def _norm_gradient(norm, v, f, c2, s2, sigma):
    """By the symmetry of the first term its gradient is twice that of <S1, S1'> with S1' held: one set of rows at a
    time, each with its own small graph."""
    v = v.detach().requires_grad_(True)
    c1, s1 = _cells(v, f)
    ch, sh = c1.detach(), s1.detach()
    gc, gs = torch.zeros_like(ch), torch.zeros_like(sh)
    rows, step = _blocks(len(ch), 4 * (len(ch) + len(c2)))
    for i in rows:
        ck = ch[i:i + step].clone().requires_grad_(True)
        sk = sh[i:i + step].clone().requires_grad_(True)
        e = 2 * (_kval(_dist2(ck, ch), sigma, False) * _weights(norm, sk, sh)).sum() \
            - 2 * (_kval(_dist2(ck, c2), sigma, False) * _weights(norm, sk, s2)).sum()
        gc[i:i + step], gs[i:i + step] = torch.autograd.grad(e, (ck, sk))
    return torch.autograd.grad((c1, s1), v, (gc, gs))[0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "match":
        return None
    if kind == "sum":
        if float(case["n"]) * case["m"] > 6e10:
            return None
        x, y, a, p = _sum_inputs(case, seed)
        lap = case["kernel"] == "laplacian"
        if case["op"] == "applyK":
            return _apply(x, y, a, case["sigma"], lap)
        return _apply_diff(x, y, p, a, case["sigma"], lap)
    if kind == "template":
        return _exact_template(case, seed)
    state_rng = np.random.default_rng
    v, f, vt = _surface(case, seed)
    fd = _dev(f)
    if kind == "gradient":
        rng = state_rng([seed, 5])
        px = (_bumps(v, rng, 8, 0.25, 1.0)[:, None] * v + 0.1 * rng.standard_normal(v.shape)) / len(v)
        at, dt = _dev(_momenta(case, v, seed, case["steps"])), 1.0 / case["steps"]
        xt, _ = _shoot(_dev(v), at, case["sigma"], dt)
        pxt, dat = _adjoint(xt, at, _dev(px), case["sigma"], dt)
        return dat, xt, pxt
    c2, s2 = _cells(_dev(vt), fd)
    if kind == "norm":
        rng = state_rng([seed, 6])
        x = _dev(v * (1 + _bumps(v, rng, 8, 0.3, 0.08))[:, None])
        call = _norm_gradient if case["grad"] else _norm
        out = call(case["norm"], x, fd, c2, s2, case["sigma"])
        return out if case["grad"] else float(out)
    at, dt, K = _dev(_momenta(case, v, seed, case["steps"])), 1.0 / case["steps"], case["sigma"]
    xt, e = _shoot(_dev(v), at, K, dt)
    e = e + _norm(case["norm"], xt[-1], fd, c2, s2, case["sigma_dist"])
    px1 = -_norm_gradient(case["norm"], xt[-1], fd, c2, s2, case["sigma_dist"])
    pxt, dat = _adjoint(xt, at, px1, K, dt)
    return e, torch.stack([dt * _apply(xt[t], xt[t], dat[t], K) for t in range(len(at))]), -pxt[0]


def _exact_template(case, seed):
    v, f, targets, prior, stack, dprior, dstack = _template_inputs(case, seed)
    T, K, sg, sd = case["steps"], case["subjects"], case["sigma"], case["sigma_dist"]
    dt, s2, fd, x0 = 1.0 / T, 0.1 ** 2, _dev(f), _dev(v)
    cells = [_cells(_dev(t), fd) for t in targets]
    prior, stack, dprior, dstack = (_dev(t) for t in (prior, stack, dprior, dstack))
    value = 0.0
    for c, s in cells:   # |S_k|^2 of the targets
        value += float((_kval(_dist2(c, c), sd, False) * _weights("varifold", s, s)).sum()) / s2
    xt, e = _shoot(x0, prior - 0.5 * dprior, sg, dt)
    value += float(e)
    for k in range(K):
        xk, ek = _shoot(xt[-1], stack[k] - 0.5 * dstack[k], sg, dt)
        value += float(ek) + float(_norm("varifold", xk[-1], fd, *cells[k], sd)) / s2
    xt, _ = _shoot(x0, prior, sg, dt)
    pt, dats = torch.zeros_like(x0), []
    for k in range(K):
        xk, _ = _shoot(xt[-1], stack[k], sg, dt)
        px1 = -_norm_gradient("varifold", xk[-1], fd, *cells[k], sd) / s2
        pxt, dat = _adjoint(xk, stack[k], px1, sg, dt)
        pt = pt + pxt[0]
        dats.append(dat)
    _, dat0 = _adjoint(xt, prior, pt, sg, dt)
    coeff = case["n"] * T
    return value, dat0 / coeff, torch.stack(dats) / coeff
