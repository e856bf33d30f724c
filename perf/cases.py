"""Performance cases of the particle FMM: what users have it evaluate.

Every case goes through the public entry points (``FMMParticleContext.evaluate``
on host arrays, ``.evaluate_device`` on device pointers, ``LaplaceFMM`` under
autograd).  The keys of a case:

  kernel   an FMMKernel name (``autograd``: LaplaceFMM, forward and backward)
  form     "plain" (FP64) or "mixed"
  n        source points;  n_trg: separate targets (0: the sources themselves)
  dist     "uniform" in the unit cube, "gauss" (8 clusters, sigma 0.02) or
           "surface" (area-uniform on a triaxial ellipsoid)
  m, leaf  multipole order, max points per leaf
  layers   "sl" single layer, "sldl" single and double layer
  setup    True: points are new at each call (particles that move);
           False: the tree is built once in prepare and each pass evaluates
           densities on it (the matrix-vector product of an iterative solver)
  box      "free" or "lattice" (period 1, sum over all images)
  io       "device" (FP64 CUDA tensors) or "host32" (float32 numpy arrays)
"""
import math

import numpy as np
import torch

import pvfmm_b200 as P
from pvfmm_b200.autograd import LaplaceFMM

_DEFAULTS = dict(form="plain", n_trg=0, dist="uniform", m=6, leaf=200, layers="sl", setup=True, box="free",
                 io="device")

# flops of one source-target pair (reference include/kernel.txx:1277, 1352,
# 1367, 1406, 1493; potential and gradient together 18)
_PAIR_FLOPS = dict(LaplacePotential=9, LaplaceGradient=16, LaplacePotGrad=18, StokesPressure=16, StokesVelocity=29,
                   StokesVelocityGrad=94, BiotSavartPotential=24, autograd=18)
# components of the equivalent densities and check potentials
_EXPANSION = dict(LaplacePotential=(1, 1), LaplaceGradient=(1, 1), LaplacePotGrad=(1, 1), StokesPressure=(3, 1),
                  StokesVelocity=(3, 3), StokesVelocityGrad=(3, 9), BiotSavartPotential=(3, 3), autograd=(1, 1))
_VECTOR = ("StokesPressure", "StokesVelocity", "StokesVelocityGrad", "BiotSavartPotential")


def _case(name, kernel, n, **kw):
    c = dict(_DEFAULTS, kernel=kernel, n=n, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a few thousand particles, as in a test, a notebook or a small
        # dynamics step: launches and host round trips count
        _case("laplace-2k", "LaplacePotential", 2_000, leaf=60),
        # the ordinary FP64 potential evaluation at the reference's example size
        _case("laplace-100k", "LaplacePotential", 100_000, leaf=300),
        # potential and field of strongly clustered particles (N-body step), large
        _case("potgrad-gauss-4m-mixed", "LaplacePotGrad", 4_000_000, form="mixed", dist="gauss", m=8, leaf=256),
        # the same step in full FP64, an odd count
        _case("potgrad-gauss-1m-plain", "LaplacePotGrad", 1_000_003, dist="gauss", m=8, leaf=256),
        # Stokes flow of point forces (suspension step), FP32 near field
        _case("stokes-1m-mixed", "StokesVelocity", 1_000_000, form="mixed", leaf=300),
        # the same in FP64 at a moderate count
        _case("stokes-60k-plain", "StokesVelocity", 60_001),
        # matrix-vector product of a boundary-integral solver: surface points,
        # tree kept, new densities
        _case("surface-2m-matvec-mixed", "LaplacePotential", 2_000_000, form="mixed", dist="surface", m=8, leaf=128,
              setup=False),
        # differentiable potential: loss, density and position gradients
        _case("autograd-1m", "autograd", 1_000_000, form="mixed", m=8, leaf=256),
        # periodic cell of charges (molecular dynamics, cosmology)
        _case("periodic-1m-mixed", "LaplacePotential", 1_000_000, form="mixed", m=8, leaf=256, box="lattice"),
        # velocity gradient for vortex stretching and stresses: nine outputs
        _case("stokesgrad-200k-mixed", "StokesVelocityGrad", 200_000, form="mixed"),
        # layer potentials of a surface at points off it: single and double
        # layer, separate ragged targets, FP64
        _case("layers-150k-plain", "LaplacePotential", 150_001, n_trg=70_003, dist="surface", layers="sldl", leaf=150),
        # the reference's float interface on host arrays: gradient at separate
        # targets, copies inside
        _case("host-grad-31k-f32", "LaplaceGradient", 31_013, n_trg=12_345, form="mixed", leaf=100, io="host32"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kernel = rng.choice(("LaplacePotential", "LaplacePotential", "LaplaceGradient", "LaplacePotGrad", "StokesVelocity",
                         "StokesVelocity", "StokesPressure", "StokesVelocityGrad", "BiotSavartPotential", "autograd"))
    vector = kernel in _VECTOR
    m = rng.choice((4, 6) if vector else (4, 6, 8, 10))
    c = _case(None, kernel, _log_uniform(rng, 1_000, 300_000 if vector else 1_000_000),
              form=rng.choice(("plain", "mixed")), dist=rng.choice(("uniform", "gauss", "surface")), m=m,
              leaf=_log_uniform(rng, 12 * m, 50 * m))
    if rng.random() < 0.5:
        c["n"] |= 1
    option = rng.random()
    if kernel != "autograd":
        if rng.random() < 0.35:
            c["n_trg"] = max(1, int(c["n"] * rng.uniform(0.1, 1.5)))
        if rng.random() < 0.25:
            c["setup"] = False
        if option < 0.2 and kernel in ("LaplacePotential", "StokesVelocity"):
            c["layers"] = "sldl"
        elif option < 0.35 and kernel == "LaplacePotential":
            c.update(box="lattice", n_trg=0, dist="uniform", m=min(c["m"], 6))
        elif option < 0.5:
            c.update(io="host32", form="mixed", n=min(c["n"], 200_000))
            c["n_trg"] = min(c["n_trg"], 200_000)
    # no drawn case asks for more than the largest listed one
    limit = _cost(listed()[2])
    while _cost(c) > 0.5 * limit:
        c["n"] = c["n"] * 2 // 3
        c["n_trg"] = c["n_trg"] * 2 // 3
    return c


def _shape(case):
    """(targets, mean sources of a leaf, leaves, neighbour leaves) of the tree
    the case leads to: leaves split above `leaf` points (sources and targets
    counted) and are on average 0.45 full."""
    n, nt = case["n"], case["n_trg"] or case["n"]
    full = max(1.0, 0.45 * case["leaf"])
    leaves = max(1.0, (n + nt) / full)
    near = min(leaves, {"uniform": 27.0, "gauss": 27.0, "surface": 11.0}[case["dist"]])
    return nt, n / leaves, leaves, near


def _flops(case):
    """Flops of the FMM's stages (pairs, surface products, V-list products)."""
    nt, per_leaf, leaves, near = _shape(case)
    ki, ko = _EXPANSION[case["kernel"]]
    m = case["m"]
    ns = 6 * (m - 1) ** 2 + 2
    pf = _PAIR_FLOPS[case["kernel"]]
    pairs = nt * per_leaf * near * pf * (2 if case["layers"] == "sldl" else 1)
    surfaces = (case["n"] + nt) * ns * pf
    products = leaves * 4 * 2.0 * (ns * ki) * (ns * ko)
    vlist = 0.0
    if leaves > 8:
        offsets = {"uniform": 26.0, "gauss": 20.0, "surface": 10.0}[case["dist"]]
        vlist = leaves / 8 * offsets * 4 * m * m * (m + 1) * 512.0 * ki * ko
    return pairs, surfaces + products, vlist


def _cost(case):
    pairs, chain, vlist = _flops(case)
    form = 1.0 if case["form"] == "mixed" else 2.0
    return (pairs * form + chain * 2 + vlist * form) * (2 if case["kernel"] == "autograd" else 1)


def work(case):
    nt = case["n_trg"] or case["n"]
    k0, k1 = (1, 1) if case["kernel"] == "autograd" else P.KERNEL_DIMS[P.FMMKernel[case["kernel"]]]
    per_src = k0 + (k0 + 3 if case["layers"] == "sldl" else 0)
    if case["setup"]:
        per_src += 3
    words = case["n"] * per_src + nt * (k1 + (3 if case["setup"] and case["n_trg"] else 0))
    flops = sum(_flops(case))
    if case["kernel"] == "autograd":  # weights in, gradients of densities and positions out, two evaluations
        words += case["n"] * 5
        flops *= 2
    return {"bytes": float(words * (4 if case["io"] == "host32" else 8)), "flops": float(flops)}


def tolerance(case):
    """About four times what two correct builds differ by, measured over 42
    cases of these ranges with another reciprocal square root in every pair
    kernel and with the V-list summed in another order.  FP64: 2.6e-13 at most
    (8e-14 for Laplace), where the pseudo-inverse amplifies the rounding of the
    check potentials; the Stokes double layer, with its larger check
    potentials, 2.2e-10.  Mixed: 1e-6, and 2.3e-6 (single values 1.9e-4)
    between the mixed and the plain form for position gradients."""
    if case["form"] == "plain":
        return {"rel": 1e-9 if case["layers"] == "sldl" and case["kernel"] == "StokesVelocity" else 1.2e-12}
    return {"rel": 5e-6, "max": 6e-4}


def _points(case, n, gen, dist):
    kw = dict(device="cuda", dtype=torch.float64, generator=gen)
    if dist == "uniform":
        return torch.rand(n, 3, **kw)
    if dist == "gauss":
        centres = 0.1 + 0.8 * torch.rand(8, 3, **kw)
        comp = torch.randint(0, 8, (n,), device="cuda", generator=gen)
        return (centres[comp] + 0.02 * torch.randn(n, 3, **kw)).clamp(0.0, 1.0)
    # area-uniform on the ellipsoid: directions accepted in proportion to the area element
    axes = torch.tensor([0.45, 0.3, 0.15], device="cuda", dtype=torch.float64)
    u = torch.nn.functional.normalize(torch.randn(int(2.4 * n) + 2000, 3, **kw), dim=1)
    keep = torch.rand(u.shape[0], **kw) < (u / axes).norm(dim=1) * axes.min()
    return (0.5 + u[keep] * axes)[:n].contiguous()


def _inputs(case, seed):
    """Positions, densities and targets (CUDA, FP64) made from the seed."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kw = dict(device="cuda", dtype=torch.float64, generator=gen)
    n, kernel = case["n"], case["kernel"]
    k0 = 1 if kernel == "autograd" else P.KERNEL_DIMS[P.FMMKernel[kernel]][0]
    x = _points(case, n, gen, case["dist"])
    q = torch.randn(n, k0, **kw) if k0 == 3 else 2 * torch.rand(n, k0, **kw) - 1
    if case["box"] == "lattice":
        q -= q.mean(dim=0)  # a periodic cell without net charge
    dl = None
    if case["layers"] == "sldl":  # the surface normal and the layer density, in the order the kernels read them
        nrm = torch.nn.functional.normalize(torch.randn(n, 3, **kw), dim=1)
        mu = torch.randn(n, k0, **kw)
        dl = torch.cat([nrm, mu], dim=1) if k0 == 1 else torch.cat([mu, nrm], dim=1)
    t = None
    if case["n_trg"]:
        t = _points(case, case["n_trg"], gen, "uniform" if case["dist"] == "surface" else case["dist"])
    w = torch.rand(n, **kw) if kernel == "autograd" else None
    return x, q, dl, t, w


# One context serves all evaluations of new points, as a program keeps it
# from step to step; the last one made is kept here.
_kept = {}


def _new_context(case):
    if case["kernel"] == "autograd":
        return LaplaceFMM(max_points=case["leaf"], multipole_order=case["m"], precision=case["form"])
    box = 1.0 if case["box"] == "lattice" else -1.0
    kernel = P.FMMKernel[case["kernel"]]
    if case["io"] == "host32":
        ctx = P.FMMParticleContext(box, case["leaf"], case["m"], kernel, dtype=np.float32)
    else:
        ctx = P.FMMParticleContext(box, case["leaf"], case["m"], kernel, dtype=np.float64,
                                   precision=P.PRECISION_MIXED if case["form"] == "mixed" else P.PRECISION_PLAIN)
    if case["box"] == "lattice":
        ctx.set_periodic_bc(lattice=True)
    return ctx


def _context(case):
    if not case["setup"]:  # the tree lives in the context: one context per set of points
        return _new_context(case)
    key = tuple(case[k] for k in ("kernel", "form", "m", "leaf", "box", "io"))
    if key not in _kept:
        _kept.clear()
        _kept[key] = _new_context(case)
    return _kept[key]


def prepare(case, seed):
    x, q, dl, t, w = _inputs(case, seed)
    s = {"case": case, "ctx": _context(case)}
    if case["kernel"] == "autograd":
        return dict(s, x=x, q=q.reshape(-1), w=w)
    if case["io"] == "host32":
        s.update(x=x.float().cpu().numpy().reshape(-1), q=q.float().cpu().numpy().reshape(-1),
                 dl=None if dl is None else dl.float().cpu().numpy().reshape(-1))
        s["t"] = s["x"] if t is None else t.float().cpu().numpy().reshape(-1)
    else:
        t = x if t is None else t
        k1 = P.KERNEL_DIMS[P.FMMKernel[case["kernel"]]][1]
        s.update(x=x, q=q.contiguous(), dl=dl, t=t, out=torch.empty(t.shape[0], k1, device="cuda", dtype=torch.float64))
    if not case["setup"]:
        torch.cuda.synchronize()
        _evaluate(s, True)
    return s


def _evaluate(s, setup):
    ctx = s["ctx"]
    if s["case"]["io"] == "host32":
        return ctx.evaluate(s["x"], s["q"], s["dl"], s["t"], setup)
    x, t, out = s["x"], s["t"], s["out"]
    ctx.evaluate_device(x.data_ptr(), s["q"].data_ptr(), x.shape[0], t.data_ptr(), out.data_ptr(), t.shape[0], setup,
                        torch.cuda.current_stream().cuda_stream, None if s["dl"] is None else s["dl"].data_ptr())
    return out


def run(s):
    if s["case"]["kernel"] == "autograd":
        x = s["x"].detach().requires_grad_()
        q = s["q"].detach().requires_grad_()
        phi = s["ctx"](x, q)
        (s["w"] * phi * phi).sum().backward()
        return {"phi": phi.detach(), "grad_q": q.grad, "grad_x": x.grad}
    return _evaluate(s, s["case"]["setup"])


def _direct(kernel, x, q, t):
    """FP64 sum over all pairs, r = target - source, r == 0 left out."""
    pi4 = 4 * math.pi
    outs = []
    tc = 1024
    for a in range(0, t.shape[0], tc):
        tt = t[a:a + tc]
        acc = 0.0
        for b in range(0, x.shape[0], 8192):
            d = [tt[:, None, i] - x[None, b:b + 8192, i] for i in range(3)]
            f = q[b:b + 8192].T
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            y = torch.where(r2 > 0, r2.rsqrt(), torch.zeros_like(r2))
            if kernel == "LaplacePotential":
                v = [y @ f[0]]
            elif kernel in ("LaplaceGradient", "LaplacePotGrad"):
                y3 = y * y * y
                v = ([y @ f[0]] if kernel == "LaplacePotGrad" else []) + [(d[i] * y3) @ f[0] for i in range(3)]
            else:
                rf = d[0] * f[0] + d[1] * f[1] + d[2] * f[2]
                y3 = y * y * y
                if kernel == "StokesVelocity":
                    g = rf * y3
                    v = [y @ f[i] + (d[i] * g).sum(1) for i in range(3)]
                elif kernel == "StokesPressure":
                    v = [(rf * y3).sum(1)]
                elif kernel == "BiotSavartPotential":
                    v = [(y3 * d[k]) @ f[j] - (y3 * d[j]) @ f[k] for j, k in ((1, 2), (2, 0), (0, 1))]
                else:
                    c = 3 * rf * y * y
                    v = [((d[j] * f[i] - d[i] * f[j] - c * d[i] * d[j] + (rf if i == j else 0.0)) * y3).sum(1)
                         for i in range(3) for j in range(3)]
            acc = acc + torch.stack(v, dim=1)
        outs.append(acc)
    return torch.cat(outs) / (2 * pi4 if kernel in ("StokesVelocity", "StokesVelocityGrad") else pi4)


def exact(case, seed):
    kernel = case["kernel"]
    nt = case["n_trg"] or case["n"]
    ops = {"LaplacePotential": 1, "StokesVelocityGrad": 10}.get(kernel, 3)
    # the all-pairs sum of large cases takes too long; a periodic sum is not
    # one; double-layer values are scaled to the unit box as the reference
    # scales them, which is no direct sum in the caller's frame
    if case["box"] != "free" or case["layers"] == "sldl" or float(case["n"]) * nt * ops > 1.5e11:
        return None
    x, q, _, t, w = _inputs(case, seed)
    t = x if t is None else t
    if case["io"] == "host32":
        x, q, t = x.float().double(), q.float().double(), t.float().double()
    if kernel == "autograd":
        phi = _direct("LaplacePotential", x, q, x)[:, 0]
        g = 2 * w * phi
        back = _direct("LaplacePotGrad", x, torch.stack([g], dim=1), x)
        fwd = _direct("LaplaceGradient", x, q, x)
        return {"phi": phi, "grad_q": back[:, 0], "grad_x": -q * back[:, 1:] - g[:, None] * fwd}
    v = _direct(kernel, x, q, t)
    return v.reshape(-1).cpu().numpy() if case["io"] == "host32" else v
