"""Cases to time: N-body evaluations through the package's public calls.

Three paths are covered, over the sizes and options they are used with:

* "fmm":    one FMM evaluation (partition, upward, traverse, downward, results),
            in the FP64 and the mixed form, one-sided by `Context.evaluate` or
            mutual by the staged calls, on device or pinned host buffers, results
            in the caller's or in Morton order;
* "bh":     one Barnes-Hut step by `Context.bh_evaluate`, FP64 or FP32 walk;
* "direct": the FP64 direct sum at sampled targets, the check behind every
            verified parameter choice (`Context.direct`).

The mixed form and the FP32 walk carry FP32 accuracy, so a program that asks for
them keeps their potentials and accelerations as FP32; the FP64 forms' results
stay FP64.  (The chooser's network is left out: it is asked once per system, and
its time is small beside the evaluations it chooses for.)
"""
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parent.parent


def _package():
    """The package directory has a hyphen in its name: import it as tapas_reduce_b200."""
    if "tapas_reduce_b200" not in sys.modules:
        d = ROOT / "tapas-reduce_b200"
        spec = importlib.util.spec_from_file_location(
            "tapas_reduce_b200", d / "__init__.py", submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["tapas_reduce_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["tapas_reduce_b200"]


def _fmm(name, form, dist, n, P, theta, ncrit, mem="device", mutual=0, order="original"):
    c = {"path": "fmm", "form": form, "dist": dist, "n": n, "P": P, "theta": theta,
         "ncrit": ncrit, "mem": mem, "mutual": mutual, "order": order}
    return dict(c, name=name) if name else c


def _bh(name, form, dist, n, theta, ncrit, order="original"):
    c = {"path": "bh", "form": form, "dist": dist, "n": n, "theta": theta, "ncrit": ncrit,
         "eps2": 1e-6, "order": order}
    return dict(c, name=name) if name else c


def _direct(name, dist, n, targets):
    c = {"path": "direct", "dist": dist, "n": n, "targets": targets}
    return dict(c, name=name) if name else c


def listed():
    return [
        # A first try or a unit test of a user's own program: a few thousand bodies,
        # where the number of launches and host round trips is the time.
        _fmm("fmm_fp64_sphere_2500", "fp64", "sphere_surface", 2500, 6, 0.35, 16),
        _fmm("fmm_mixed_gauss_1500", "mixed", "two_gaussians", 1500, 4, 0.5, 64),
        # The -m 1 option by the staged calls, an odd body count, small leaves, results in
        # Morton order (a program that keeps its bodies in that order).
        _fmm("fmm_fp64_mutual_gauss_30011", "fp64", "two_gaussians", 30011, 8, 0.5, 32,
             mutual=1, order="sorted"),
        # The reference example's default setting (P=10, theta=0.4, ncrit=64), both forms.
        _fmm("fmm_fp64_cube_100k", "fp64", "uniform_cube", 100000, 10, 0.4, 64),
        _fmm("fmm_mixed_cube_100k", "mixed", "uniform_cube", 100000, 10, 0.4, 64),
        # A galaxy-like system of strongly varying density.
        _fmm("fmm_mixed_plummer_1m", "mixed", "plummer", 1000000, 10, 0.4, 64),
        # Boundary-element-like surface charges at high order: mixed on the device, and the
        # plain FP64 form for a program that holds its bodies in (pinned) host memory.
        _fmm("fmm_mixed_sphere_1m_p15", "mixed", "sphere_surface", 1000000, 15, 0.4, 128),
        _fmm("fmm_fp64_host_sphere_1m_p15", "fp64", "sphere_surface", 1000000, 15, 0.4, 128,
             mem="host"),
        # The benchmark's headline workload and the largest case, at the setting its
        # parameter chooser picks for a tolerance of 1e-6.
        _fmm("fmm_mixed_sphere_16m", "mixed", "sphere_surface", 16000000, 12, 0.35, 128),
        # The Barnes-Hut sample as it is (one body per leaf, FP64), and the benchmark's walk.
        _bh("bh_fp64_plummer_20k_ncrit1", "fp64", "plummer", 20000, 0.5, 1),
        _bh("bh_fp32_plummer_4m", "mixed", "plummer", 4000000, 0.5, 32),
        # The accuracy check of a 1M-body run on 4000 sampled targets.
        _direct("direct_sphere_1m_4000", "sphere_surface", 1000000, 4000),
    ]


def _log_int(rng, a, b):
    n = int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    return max(a, min(b, n | 1 if rng.random() < 0.5 else n))


DISTS = ("uniform_cube", "plummer", "sphere_surface", "two_gaussians")


def draw(rng):
    """One more case: sizes over their logarithm, every distribution, form and option.  The upper
    sizes depend on the form and the distribution so that none costs more than the largest
    listed case (volume-filling bodies have far more close pairs than a surface)."""
    u = rng.random()
    if u < 0.70:
        form = rng.choice(("fp64", "mixed", "mixed"))
        dist = rng.choice(DISTS)
        mutual = 1 if rng.random() < 0.2 else 0
        most = 300000 if form == "fp64" else 8000000 if dist == "sphere_surface" else 1500000
        n = _log_int(rng, 1000, most)
        mem = "host" if n <= 1000000 and rng.random() < 0.25 else "device"
        return _fmm(None, form, dist, n, rng.randint(4, 12 if n > 500000 else 16),
                    round(rng.uniform(0.35, 0.6), 2), rng.choice((32, 64, 128)), mem, mutual,
                    rng.choice(("original", "original", "sorted")))
    if u < 0.88:
        form = rng.choice(("fp64", "mixed"))
        n = _log_int(rng, 1000, 300000 if form == "fp64" else 2000000)
        return _bh(None, form, rng.choice(("uniform_cube", "plummer", "two_gaussians")), n,
                   round(rng.uniform(0.45, 0.8), 2), rng.choice((1, 8, 32)),
                   rng.choice(("original", "sorted")))
    n = _log_int(rng, 20000, 3000000)
    return _direct(None, rng.choice(DISTS), n,
                   _log_int(rng, 100, min(4096, int(6e9 // n))))


def _bodies(dist, n, seed):
    """x, y, z, q on the GPU: the distributions of the package's `datasets`, from torch's
    generator (a 16M-body set in milliseconds)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))

    def uni():
        return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)

    def gauss():
        return torch.randn(n, generator=g, device="cuda", dtype=torch.float64)

    if dist == "uniform_cube":
        x, y, z, q = 2 * uni() - 1, 2 * uni() - 1, 2 * uni() - 1, uni()
        return x, y, z, q / q.sum()
    if dist == "plummer":  # scale radius 1, r < 100: the radius from the truncated distribution
        u = (uni() + 2.0 ** -54) * (1 + 1e-4) ** -1.5
        r = 1 / torch.sqrt(u ** (-2.0 / 3.0) - 1)
        c, ph = 2 * uni() - 1, 2 * math.pi * uni()
        s = torch.sqrt(torch.clamp(1 - c * c, min=0))
        return (r * s * torch.cos(ph), r * s * torch.sin(ph), r * c,
                torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64))
    if dist == "sphere_surface":
        x, y, z = gauss(), gauss(), gauss()
        r = torch.sqrt(x * x + y * y + z * z)
        q = 2 * uni() - 1
        return x / r, y / r, z / r, q - q.mean()
    side = torch.where(uni() < 0.5, -0.5, 0.5).to(torch.float64)
    return (side + 0.1 * gauss(), 0.1 * gauss(), 0.1 * gauss(),
            torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64))


def _targets(n, k, seed):
    return np.sort(np.random.default_rng(seed).choice(n, size=min(k, n), replace=False))


def prepare(case, seed):
    tb = _package()
    n = case["n"]
    host = case.get("mem") == "host"
    b = [v.contiguous() for v in _bodies(case["dist"], n, seed)]
    out = None
    if case["path"] != "direct":
        out = torch.zeros((n, 4), dtype=torch.float64, device="cuda")
    if host:
        b = [v.cpu().pin_memory() for v in b]
        out = out.cpu().pin_memory()
    torch.cuda.synchronize()
    ctx = tb.Context(torch.cuda.current_device())
    state = {"tb": tb, "case": case, "ctx": ctx, "bodies": b, "out": out,
             "prec": tb.FP64 if case.get("form") == "fp64" else tb.MIXED,
             "order": tb.ORDER_SORTED if case.get("order") == "sorted" else tb.ORDER_ORIGINAL}
    if case["path"] == "direct":
        # the bodies of the evaluation that is to be checked are in the context already
        ctx.partition(*b, ncrit=64)
        state["targets"] = _targets(n, case["targets"], seed)
    return state


def _kept(case, out, pot, acc):
    if case["form"] == "mixed":
        out = out.to(torch.float32)
    return {"pot": out[:, pot], "acc": out[:, acc]}


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["path"] == "direct":
        d = ctx.direct(state["targets"])
        return {"pot": d[:, 0], "acc": d[:, 1:]}
    x, y, z, q = state["bodies"]
    out, prec = state["out"], state["prec"]
    if case["path"] == "bh":
        ctx.bh_evaluate(x, y, z, q, ncrit=case["ncrit"], theta=case["theta"], eps2=case["eps2"],
                        precision=prec, order=state["order"], out=out)
        return _kept(case, out, 3, slice(0, 3))
    if case["mutual"]:
        ctx.partition(x, y, z, q, ncrit=case["ncrit"])
        ctx.upward(case["P"], prec)
        ctx.traverse(case["theta"], 1, prec)
        ctx.downward(prec)
        ctx.results(state["order"], out=out)
    else:
        ctx.evaluate(x, y, z, q, P=case["P"], ncrit=case["ncrit"], theta=case["theta"],
                     precision=prec, order=state["order"], out=out)
    return _kept(case, out, 0, slice(1, 4))


def _near_cells(case):
    """Cells of a body's own size within the acceptance radius (width / theta) of its cell."""
    t = case["theta"]
    return math.pi / t ** 2 if case["dist"] == "sphere_surface" else 4.19 / t ** 3


def work(case):
    """Bodies in, results out; 20 flop per body pair, and per translation the triangular
    double sum of an M2L.  The numbers of pairs are estimates from the acceptance radius
    and a half-full leaf."""
    n = case["n"]
    if case["path"] == "direct":
        return {"bytes": 32.0 * n + 40.0 * case["targets"], "flops": 20.0 * n * case["targets"]}
    near = _near_cells(case)
    fill = max(1.0, 0.5 * case["ncrit"])
    if case["path"] == "bh":
        levels = max(1.0, math.log(n / fill, 8))
        return {"bytes": 64.0 * n, "flops": 20.0 * n * min(n, near * (7 * levels + fill))}
    P = case["P"]
    m2l = 8.0 * sum((j + 1) * (P - j) ** 2 for j in range(P))
    leaves = max(1.0, n / fill)
    return {"bytes": 64.0 * n,
            "flops": 20.0 * n * min(n, near * fill) + m2l * leaves * min(leaves, 1.5 * near)}


def _direct_sum(x, y, z, q, ti, eps2, sign):
    """sum_j q_j / r and sign * sum_j q_j (x_i - x_j) / r^3 at the targets ti, FP64;
    pairs at zero (softened) distance left out."""
    n, k = x.numel(), ti.numel()
    pot = torch.empty(k, dtype=torch.float64, device=x.device)
    acc = torch.empty((k, 3), dtype=torch.float64, device=x.device)
    step = max(1, int(3.0e6 // n))  # a block of a few tens of MB stays in the L2
    for a in range(0, k, step):
        t = ti[a:a + step]
        dx, dy, dz = (v[t][:, None] - v[None, :] for v in (x, y, z))
        r2 = (dx * dx).addcmul_(dy, dy).addcmul_(dz, dz)
        if eps2:
            w = r2.add_(eps2).rsqrt_()
        else:
            w = torch.where(r2 > 0, r2.rsqrt(), 0.0)
        s = w * q[None, :]
        pot[a:a + step] = s.sum(1)
        s.mul_(w).mul_(w)
        for d, v in enumerate((dx, dy, dz)):
            acc[a:a + step, d] = sign * (s * v).sum(1)
    return pot, acc


def exact(case, seed):
    """The direct sum in FP64, where it takes seconds; None for the larger body counts."""
    n = case["n"]
    pairs = float(n) * (case["targets"] if case["path"] == "direct" else n)
    if pairs > 4.2e10:
        return None
    x, y, z, q = _bodies(case["dist"], n, seed)
    if case["path"] == "direct":
        ti = torch.from_numpy(_targets(n, case["targets"], seed)).cuda()
        pot, acc = _direct_sum(x, y, z, q, ti, 0.0, -1.0)
        return {"pot": pot.cpu().numpy(), "acc": acc.cpu().numpy()}
    ti = torch.arange(n, device="cuda")
    if case.get("order") == "sorted":
        ti = _morton_order(x, y, z)
    if case["path"] == "bh":  # softened, the body itself included
        pot, acc = _direct_sum(x, y, z, q, ti, case["eps2"], -1.0)
    else:
        pot, acc = _direct_sum(x, y, z, q, ti, 0.0, -1.0)
    if case.get("mem") == "host":
        pot, acc = pot.cpu(), acc.cpu()
    return {"pot": pot, "acc": acc}


def _morton_order(x, y, z):
    """The bodies' order by Morton key: 19 levels in the cube over every coordinate of bodies
    1..n-1 and the z of body 0, which is the cube the tree is built in."""
    c = torch.cat([x[1:], y[1:], z]) if x.numel() > 1 else z
    lo, hi = c.min(), c.max()
    pitch = (hi - lo) / 2.0 ** 19
    key = torch.zeros_like(x, dtype=torch.int64)
    a = [((v - lo) / pitch).to(torch.int64) for v in (x, y, z)]
    a = [torch.where(v == 1 << 19, v - 1, v) & 0x7FFFF for v in a]  # the upper face
    for bit in range(19):
        for d in range(3):
            key |= ((a[d] >> bit) & 1) << (3 * bit + d)
    return torch.sort(key, stable=True).indices
