"""Workloads of the point fast Gauss transform, one dict of plain values each.

Every case goes through a public entry point of `fgt_b200`: `pfgt_device`
(device arrays), `pfgt` (host arrays), `Plan.execute` (fixed points, new
strengths) or `pfgt_batch` (many instances).  Inputs come from the seed alone.

Keys of a case: call (device, host, plan, batch), dim, nd, n (sources),
targets (none, same, uniform), m (targets), points (uniform, sphere,
clusters, wiggly), delta, eps, period, charge, dipole, pgh, pghtarg (0 none,
1 potential, 2 + gradient, 3 + hessian), prec (auto, fp64, mixed); a batch
has count, nmin, nmax instead of the sizes and of delta and eps.
"""
import ctypes
import math

import numpy as np
import torch

import fgt_b200 as F

PREC = {"auto": F.PREC_AUTO, "fp64": F.PREC_FP64, "mixed": F.PREC_MIXED}


def _case(name, **kw):
    c = dict(name=name, call="device", dim=3, nd=1, n=0, targets="none", m=0, points="uniform",
             delta=1e-4, eps=1e-6, period=0, charge=True, dipole=False, pgh=1, pghtarg=0,
             prec="auto")
    c.update(kw)
    return c


def listed():
    return [
        # one small transform from host arrays: all latency (a particle code's step)
        _case("host_3e3_pot", call="host", n=3001, delta=1e-3, eps=1e-6),
        # 3D uniform sources = targets, potential: an ordinary call
        _case("uniform_1e5_pot", n=100000, delta=1e-4, eps=1e-6),
        # many small and middling transforms, uneven sizes and parameters
        dict(name="batch_60", call="batch", count=60, nmin=1000, nmax=100000),
        # the test driver's curve: charges and dipoles, hessians at separate targets
        _case("wiggly_dipole_hess", n=60007, targets="uniform", m=50003, points="wiggly",
              delta=1e-3, eps=1e-6, dipole=True, pgh=1, pghtarg=3),
        # 2D, two densities, gradients, high accuracy (boundary and volume data)
        _case("wiggly2d_nd2_grad", dim=2, nd=2, n=400009, targets="uniform", m=300007,
              points="wiggly", delta=1e-5, eps=1e-9, pgh=2, pghtarg=2),
        # repeated transforms of fixed points with new strengths (an iterative solver)
        _case("plan_1e6_pot", call="plan", n=1000003, points="sphere", delta=1e-4, eps=1e-6),
        # 2D periodic, four densities, gradients, 1e7 points
        _case("periodic2d_nd4_1e7", dim=2, nd=4, n=10000000, delta=1e-6, eps=1e-6, period=1,
              pgh=2),
        # 64 Gaussian clusters, deep tree, uniform targets, nine digits
        _case("clusters_2e6_1e-9", n=2000000, targets="uniform", m=2000000, points="clusters",
              delta=1e-5, eps=1e-9, pgh=2, pghtarg=2),
        # the whole pipeline in FP64 at six digits
        _case("sphere_2e6_fp64", n=2000000, targets="same", points="sphere", delta=1e-4,
              eps=1e-6, pgh=2, pghtarg=2, prec="fp64"),
        # nine digits with dense boxes: plane waves do the work
        _case("sphere_4e6_1e-9", n=4000000, targets="same", points="sphere", delta=1e-4,
              eps=1e-9, pgh=2, pghtarg=2),
        # twelve digits, few large boxes
        _case("sphere_15e5_1e-12", n=1500000, targets="same", points="sphere", delta=1e-2,
              eps=1e-12, pgh=2, pghtarg=2),
        # the headline call: 1e7 sources and targets on a sphere + 1% background
        _case("sphere_1e7_mixed", n=10000000, targets="same", points="sphere", delta=1e-4,
              eps=1e-6, pgh=2, pghtarg=2),
    ]


def draw(rng):
    def logu(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["device3", "device3", "device3", "fp64", "fp64", "two_d", "periodic",
                       "options", "host", "plan", "batch"])
    if kind == "batch":
        nmax = int(logu(1e4, 1e5))
        return dict(call="batch", count=rng.randint(16, 60), nmin=1000, nmax=nmax)
    delta = float("%.3g" % logu(1e-6, 1e-1))
    if kind == "device3":
        c = _case("", n=int(logu(1e4, 1e7)), delta=delta, eps=rng.choice([1e-3, 1e-4, 1e-6]),
                  points=rng.choice(["uniform", "sphere", "clusters"]),
                  targets=rng.choice(["none", "same", "uniform"]), pgh=rng.choice([1, 2]))
        if c["points"] == "uniform" or c["targets"] == "uniform":
            # a volume of boxes; the near field of a large delta sums most pairs directly
            c["delta"] = float("%.3g" % logu(1e-5, 1e-2))
            c["n"] = min(c["n"], 2000003)
    elif kind == "fp64":
        c = _case("", n=int(logu(1e4, 1.5e6)), delta=float("%.3g" % logu(1e-5, 1e-2)),
                  eps=rng.choice([1e-8, 1e-9, 1e-10, 1e-12]),
                  points=rng.choice(["sphere", "clusters"]), targets=rng.choice(["none", "same"]),
                  pgh=rng.choice([1, 2]))
    elif kind == "two_d":
        c = _case("", dim=2, nd=rng.choice([1, 2, 3]), n=int(logu(1e4, 2e6)), delta=delta,
                  eps=rng.choice([1e-3, 1e-6, 1e-9, 1e-12]),
                  points=rng.choice(["uniform", "wiggly", "clusters"]),
                  targets=rng.choice(["none", "uniform"]), pgh=rng.choice([1, 2, 3]))
    elif kind == "periodic":
        c = _case("", dim=rng.choice([2, 3]), nd=rng.choice([1, 4]), n=int(logu(2e4, 1e6)),
                  delta=float("%.3g" % logu(1e-6, 1e-3)), eps=rng.choice([1e-3, 1e-6, 1e-9]),
                  period=1, pgh=rng.choice([1, 2]))
        if c["dim"] == 3:
            c["delta"] = max(c["delta"], 1e-5)
            c["nd"] = 1
    elif kind == "options":
        c = _case("", dim=rng.choice([1, 2, 3]), nd=rng.choice([1, 2]), n=int(logu(1e3, 1e5)),
                  delta=float("%.3g" % logu(1e-4, 1e-2)), eps=rng.choice([1e-3, 1e-6, 1e-9]),
                  points="wiggly", charge=rng.random() < 0.5, dipole=True, pgh=rng.choice([1, 2, 3]),
                  targets=rng.choice(["none", "uniform"]))
    elif kind == "plan":
        c = _case("", call="plan", n=int(logu(1e4, 1e6)), delta=float("%.3g" % logu(1e-5, 1e-2)),
                  eps=rng.choice([1e-3, 1e-6, 1e-9]), points=rng.choice(["sphere", "clusters"]),
                  pgh=rng.choice([1, 2]))
    else:
        c = _case("", call="host", n=int(logu(1e3, 1e5)), delta=float("%.3g" % logu(1e-4, 1e-2)),
                  eps=rng.choice([1e-3, 1e-6, 1e-9]), points=rng.choice(["uniform", "sphere"]),
                  pgh=rng.choice([1, 2]))
    c["n"] |= 1
    if c["targets"] == "uniform":
        c["m"] = int(c["n"] * rng.uniform(0.3, 1.0)) + 1
    if c["targets"] != "none":
        c["pghtarg"] = c["pgh"]
    del c["name"]
    return c


def _points(g, kind, n, dim, lo=-0.5):
    """n points of the box of side 1 whose lower corner is at `lo`."""
    def u(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    def z(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    if kind == "uniform":
        return u(n, dim) + lo
    if kind == "sphere":  # surface of radius 0.4 with 1% uniform background
        v = z(n, dim)
        v *= 0.4 / v.norm(dim=1, keepdim=True)
        bg = u(n, 1) < 0.01
        return torch.where(bg, u(n, dim) - 0.5, v) + (lo + 0.5)
    if kind == "clusters":  # 64 isotropic Gaussians of sizes 1e-3 .. 5e-2, clipped to the box
        cen = u(64, dim) - 0.5
        sig = torch.exp(u(64) * math.log(50.0) + math.log(1e-3))
        lab = torch.randint(64, (n,), generator=g, device="cuda")
        return (cen[lab] + z(n, dim) * sig[lab, None]).clamp(-0.5, 0.5) + (lo + 0.5)
    # r = 0.3 + 0.12 cos(6 theta) curve / surface and three special points
    th, ph = u(n) * math.pi, u(n) * 2 * math.pi
    rr = 0.3 + 0.12 * torch.cos(6 * th)
    if dim == 3:
        p = torch.stack([rr * th.sin() * ph.cos(), rr * th.sin() * ph.sin(), rr * th.cos()], 1)
    elif dim == 2:
        p = torch.stack([rr * ph.cos(), rr * ph.sin()], 1)
    else:
        p = (torch.cos(th) / 2)[:, None]
    p = p + (lo + 0.5)
    p[0], p[1], p[2] = lo, lo + 1.0, lo + 0.05
    return p


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, dim, nd = case["n"], case["dim"], case["nd"]
    src = _points(g, case["points"], n, dim)
    if case["targets"] == "same":
        trg = src.clone()
    elif case["targets"] == "uniform":
        trg = _points(g, "uniform", case["m"], dim)
    else:
        trg = None

    def z(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    q = z(n, nd) if case["charge"] else None
    ds = rn = None
    if case["dipole"]:
        ds, rn = z(n, nd), z(n, dim)
        rn /= rn.norm(dim=1, keepdim=True)
    return src, q, rn, ds, trg


def _batch_inputs(case, seed):
    """Instances of uneven sizes and parameters, half uniform, half on a sphere."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for i in range(case["count"]):
        # sizes even over their logarithm; the rest of an instance comes from the seed
        n = int(case["nmin"] * (case["nmax"] / case["nmin"]) ** ((i + 0.5) / case["count"]))
        if i % 2:
            src = rng.uniform(-0.5, 0.5, (n, 3))
        else:
            src = rng.standard_normal((n, 3))
            src *= rng.uniform(0.3, 0.45) / np.linalg.norm(src, axis=1, keepdims=True)
        out.append(dict(nd=1, dim=3, delta=float(np.exp(rng.uniform(np.log(1e-5), np.log(1e-2)))),
                        eps=float(rng.choice([1e-3, 1e-6])), iperiod=0, sources=src,
                        charge=rng.uniform(-1, 1, (n, 1)), ifpgh=1))
    return out


def _outputs(n, nd, dim, pgh):
    nh = dim * (dim + 1) // 2
    shapes = [(n, nd), (n, dim, nd), (n, nh, nd)][:pgh]
    return [torch.zeros(*s, device="cuda", dtype=torch.float64) for s in shapes]


def prepare(case, seed):
    if case["call"] == "batch":
        return dict(case=case, instances=_batch_inputs(case, seed))
    src, q, rn, ds, trg = _inputs(case, seed)
    st = dict(case=case)
    if case["call"] == "device":
        st["in"] = (src, q, rn, ds, trg)
        st["out"] = _outputs(case["n"], case["nd"], case["dim"], case["pgh"])
        m = 0 if trg is None else trg.shape[0]
        st["outt"] = _outputs(m, case["nd"], case["dim"], case["pghtarg"]) if m else []
        st["stream"] = torch.cuda.Stream()
        o = F.FgtOpts()
        F.lib().fgt_opts_default(ctypes.byref(o))
        o.device_ptrs, o.precision = 1, PREC[case["prec"]]
        o.stream = st["stream"].cuda_stream
        st["opts"] = o
        return st

    def host(t):
        return None if t is None else t.cpu().numpy()

    st["in"] = src, q, rn, ds, trg = [host(t) for t in (src, q, rn, ds, trg)]
    if case["call"] == "plan":
        st["plan"] = F.Plan(case["nd"], case["dim"], case["delta"], case["eps"], case["period"],
                            src, targets=trg, precision=PREC[case["prec"]])
    return st


def run(state):
    c = state["case"]
    if c["call"] == "batch":
        return [r["pot"] for r in F.pfgt_batch(state["instances"])]
    src, q, rn, ds, trg = state["in"]
    if c["call"] == "device":
        def p(t):
            return 0 if t is None else t.data_ptr()

        out, outt = state["out"], state["outt"]
        po, pt = [p(t) for t in out] + [0] * 3, [p(t) for t in outt] + [0] * 3
        state["stream"].wait_stream(torch.cuda.current_stream())
        F.pfgt_device(state["opts"], c["nd"], c["dim"], c["delta"], c["eps"], c["period"], 1.0,
                      [0.0] * c["dim"], c["n"], p(src), int(c["charge"]), p(q), int(c["dipole"]),
                      p(rn), p(ds), c["pgh"], po[0], po[1], po[2],
                      0 if trg is None else trg.shape[0], p(trg), c["pghtarg"], pt[0], pt[1],
                      pt[2])
        return out + outt
    if c["call"] == "plan":
        r = state["plan"].execute(charge=q, dipstr=ds, rnormal=rn, ifpgh=c["pgh"],
                                  ifpghtarg=c["pghtarg"])
    else:
        r = F.pfgt(c["nd"], c["dim"], c["delta"], c["eps"], c["period"], src, charge=q, dipstr=ds,
                   rnormal=rn, ifpgh=c["pgh"], targets=trg, ifpghtarg=c["pghtarg"],
                   precision=PREC[c["prec"]])
    return [r[k] for k in ("pot", "grad", "hess", "pottarg", "gradtarg", "hesstarg") if k in r]


def work(case):
    """Inputs read once, outputs written once; flops of the spreading and the
    interpolation stencils (w = digits + 2 cells a side) that the accuracy
    asks for, one per strength component and one per output component."""
    if case["call"] == "batch":
        mean = (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        pts = case["count"] * mean
        return {"bytes": pts * 8 * 5, "flops": pts * 4 * 6.5 ** 3}
    n, dim, nd = case["n"], case["dim"], case["nd"]
    m = {"none": 0, "same": n, "uniform": case["m"]}[case["targets"]]
    nc = [0, 1, 1 + dim, 1 + dim + dim * (dim + 1) // 2]
    ins = dim + nd * case["charge"] + (nd + dim) * case["dipole"]
    words = n * (ins + nd * nc[case["pgh"]]) + m * (dim + nd * nc[case["pghtarg"]])
    w = math.ceil(-math.log10(case["eps"])) + 2
    comps = case["charge"] + dim * case["dipole"]
    # value and one derivative share a stencil sweep; second derivatives take another
    sweeps = [0, 1, 2, 3]
    flops = 2.0 * w ** dim * nd * (n * (comps + sweeps[case["pgh"]]) + m * sweeps[case["pghtarg"]])
    return {"bytes": 8.0 * words, "flops": flops}


def _direct(src, q, rn, ds, trg, delta, pgh, period):
    """Gaussian sums in 64 bits: sources sorted along x, targets in runs along
    x, each with the sources within reach (terms below 1e-20 left out)."""
    n, dim = src.shape
    reach = math.sqrt(46.0 * delta)
    nh = dim * (dim + 1) // 2
    pairs = [(k, k) for k in range(dim)] + [(a, b) for a in range(dim) for b in range(a + 1, dim)]
    if dim == 2:
        pairs = [(0, 0), (0, 1), (1, 1)]
    if period:  # images that reach the box
        for k in range(dim):
            parts = []
            for s in (-1.0, 0.0, 1.0):
                keep = (src[:, k] + s).abs() <= 0.5 + reach
                sh = src[keep].clone()
                sh[:, k] += s
                parts.append((sh, *[None if t is None else t[keep] for t in (q, rn, ds)]))
            src = torch.cat([p[0] for p in parts])
            q, rn, ds = [None if t is None else torch.cat([p[i + 1] for p in parts])
                         for i, t in enumerate((q, rn, ds))]
    o = torch.argsort(src[:, 0])
    src = src[o]
    q, rn, ds = [None if t is None else t[o] for t in (q, rn, ds)]
    to = torch.argsort(trg[:, 0])
    ts, m, nd = trg[to], trg.shape[0], (q if q is not None else ds).shape[1]
    out = [torch.zeros(m, *s, device=src.device, dtype=src.dtype)
           for s in ((nd,), (dim, nd), (nh, nd))[:pgh]]
    i0, step = 0, 2048
    while i0 < m:
        t = ts[i0:i0 + step]
        ends = torch.stack([t[0, 0] - reach, t[-1, 0] + reach])
        a, b = torch.searchsorted(src[:, 0].contiguous(), ends).tolist()
        for j0 in range(a, b, 32768):
            j1 = min(b, j0 + 32768)
            r = [t[:, k:k + 1] - src[None, j0:j1, k] for k in range(dim)]
            e = torch.exp(-sum(x * x for x in r) / delta)
            f = 2.0 / delta
            for strengths, dip in ((q, False), (ds, True)):
                if strengths is None:
                    continue
                s = strengths[j0:j1]
                if dip:  # (n . d/ds) exp(-r^2/delta) = f (r . n) e
                    nv = [rn[None, j0:j1, k] for k in range(dim)]
                    rdn = sum(x * y for x, y in zip(r, nv))
                    out[0][i0:i0 + step] += (f * rdn * e) @ s
                    if pgh >= 2:
                        for k in range(dim):
                            out[1][i0:i0 + step, k] += (f * e * (nv[k] - f * rdn * r[k])) @ s
                    if pgh >= 3:
                        for h, (k, l) in enumerate(pairs):
                            w = -f * (nv[k] * r[l] + nv[l] * r[k]) + f * f * rdn * r[k] * r[l]
                            if k == l:
                                w = w - f * rdn
                            out[2][i0:i0 + step, h] += (f * e * w) @ s
                else:
                    out[0][i0:i0 + step] += e @ s
                    if pgh >= 2:
                        for k in range(dim):
                            out[1][i0:i0 + step, k] += (-f * r[k] * e) @ s
                    if pgh >= 3:
                        for h, (k, l) in enumerate(pairs):
                            w = f * f * r[k] * r[l] - (f if k == l else 0.0)
                            out[2][i0:i0 + step, h] += (w * e) @ s
        i0 += step
    res = []
    for x in out:
        y = torch.empty_like(x)
        y[to] = x
        res.append(y)
    return res


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["call"] == "batch":
        got = []
        for c in _batch_inputs(case, seed):
            src, q = (torch.from_numpy(c[k]).to(dev) for k in ("sources", "charge"))
            got.append(_direct(src, q, None, None, src, c["delta"], 1, 0)[0])
        return got
    n = case["n"]
    m = {"none": 0, "same": n, "uniform": case["m"]}[case["targets"]]
    sweeps = [0, 1, 3, 7]
    cost = n * (n * sweeps[case["pgh"]] + m * sweeps[case["pghtarg"]])
    cost *= min(1.0, 2 * math.sqrt(46 * case["delta"]) + 0.02) * (2 if case["dipole"] else 1)
    if cost > 2e11:  # more pairs than 20 seconds hold
        return None
    src, q, rn, ds, trg = _inputs(case, seed)
    r = _direct(src, q, rn, ds, src, case["delta"], case["pgh"], case["period"])
    if m:
        r += _direct(src, q, rn, ds, trg, case["delta"], case["pghtarg"], case["period"])
    return r
