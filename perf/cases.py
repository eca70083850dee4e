"""Performance cases: the work that users of the engine have it do.

A case names a kind of curve collection, its size and a method; ``prepare``
makes the curves from a seed and takes them to the point where the timed call
starts, ``run`` makes one call through the public Python interface, and
``exact`` gives the linking numbers in 64 bits without the engine.

  rings    a chain of small rings, each linked with the next
  mail     a sheet of linked rings on a square grid
  walks    a few closed random walks that interpenetrate, summed directly
  pair     a closed curve against four others, in host arrays, one call each
  polymer  many closed random walks at a fixed density, Barnes-Hut
  mixed    torus knots and walks of 16 to 2^18 segments, Barnes-Hut
  knit     yarn courses of a knitted tube (closed splines), from the control
           points to the certificate
  cert     closed walks, from the curves in host memory to the certificate
"""
import math

import numpy as np
import torch

from fastlinkingnumbers_b200 import _native
from fastlinkingnumbers_b200.api import ComputeLinkingNumberDirectFast, Engine, LinkingNumberCertificate, Model

BSPLINE, CATMULL, POLYLINE = 0, 1, 3

_engine = None


def engine():
    """The program's engine: created once and kept, as a program that makes many calls does."""
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


def listed():
    return [
        # Hand-sized curves in host memory, one against four others: the per-pair
        # function of the reference's compute_link.h, where the call itself costs
        # more than the sum.
        {"name": "pair", "kind": "pair", "n1": 300, "n2": 211},
        # The smallest batched call, with both methods: 64 rings of 32 segments.
        {"name": "rings_fp64", "kind": "rings", "loops": 64, "ngon": 32, "method": "fp64"},
        {"name": "rings_bh", "kind": "rings", "loops": 64, "ngon": 32, "method": "bh"},
        # Many tiny loops, ~40,000 linked or nearly linked pairs: the mixed
        # direct sum (the default precision) and the default method.
        {"name": "mail_mixed", "kind": "mail", "rows": 100, "cols": 100, "ngon": 48, "method": "mixed"},
        {"name": "mail_bh", "kind": "mail", "rows": 100, "cols": 100, "ngon": 48, "method": "bh"},
        # Direct sums of loops of a few thousand segments, odd sizes: the
        # reference's other method, in both precisions.
        {"name": "walks_fp64", "kind": "walks", "loops": 12, "steps": 4001, "method": "fp64"},
        {"name": "walks_mixed", "kind": "walks", "loops": 16, "steps": 5003, "method": "mixed"},
        # Barnes-Hut on a small, an ordinary and the benchmark's polymer system.
        {"name": "polymer_small", "kind": "polymer", "loops": 60, "steps": 1999},
        {"name": "polymer", "kind": "polymer", "loops": 200, "steps": 50000},
        # Loops of very different sizes in one call (half knots, half walks).
        {"name": "mixed", "kind": "mixed", "loops": 1000},
        # Whole calls of verifycurves from curves in memory: yarn of a knitted
        # tube (the size of the bundled garment inputs), and long closed walks.
        {"name": "knit_cert", "kind": "knit", "loops": 39, "stitches": 60, "spline": BSPLINE, "method": "bh"},
        {"name": "walk_cert", "kind": "cert", "loops": 100, "steps": 20011},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "rings", "mail", "walks", "polymer", "polymer", "mixed", "knit", "cert"])
    if kind == "pair":
        return {"kind": kind, "n1": _log(rng, 16, 3000), "n2": _log(rng, 16, 3000)}
    if kind == "rings":
        return {"kind": kind, "loops": _log(rng, 16, 512), "ngon": _log(rng, 16, 64),
                "method": rng.choice(["fp64", "mixed", "bh"])}
    if kind == "mail":
        return {"kind": kind, "rows": _log(rng, 12, 100), "cols": _log(rng, 12, 100), "ngon": _log(rng, 16, 64),
                "method": rng.choice(["fp64", "mixed", "bh"])}
    if kind == "walks":
        return {"kind": kind, "loops": rng.randint(4, 16), "steps": _log(rng, 500, 5000),
                "method": rng.choice(["fp64", "mixed"])}
    if kind == "polymer":
        steps = _log(rng, 1000, 50000)
        return {"kind": kind, "loops": _log(rng, 20, min(300, 6e6 / steps)), "steps": steps}
    if kind == "mixed":
        return {"kind": kind, "loops": _log(rng, 50, 1000)}
    if kind == "knit":
        return {"kind": kind, "loops": rng.randint(10, 70), "stitches": _log(rng, 20, 100),
                "spline": rng.choice([BSPLINE, CATMULL]), "method": rng.choice(["bh", "mixed"])}
    steps = _log(rng, 1000, 20000)
    return {"kind": kind, "loops": _log(rng, 20, min(100, 2e6 / steps)), "steps": steps}


# ---------------------------------------------------------------- curves


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _walk(g, loops, steps, sigma=1.0):
    """(loops, steps, 3) closed Gaussian walks about their centroids."""
    s = torch.randn(loops * 3, steps, generator=g, device="cuda", dtype=torch.float64) * sigma
    s -= s.mean(dim=1, keepdim=True)
    p = torch.cumsum(s, dim=1)
    p -= p.mean(dim=1, keepdim=True)
    return p.reshape(loops, 3, steps).transpose(1, 2)


def _cube(loops, steps):
    """Cube side at the benchmark's density: 400 for 200 loops of 50,000 steps."""
    return 400.0 * (loops * steps / 1e7) ** (1 / 3)


def _rings(g, case):
    n, m = case["loops"], case["ngon"]
    t = 2 * math.pi * torch.arange(m, device="cuda", dtype=torch.float64) / m
    flat = torch.stack([torch.cos(t), torch.sin(t), torch.zeros_like(t)], dim=1)
    up = flat[:, [0, 2, 1]]
    p = torch.stack([flat if i % 2 == 0 else up for i in range(n)])
    p += 0.04 * (_rand(g, n, m, 3) - 0.5)
    p[:, :, 0] += 1.6 * torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
    return p


def _mail(g, case):
    rows, cols, m = case["rows"], case["cols"], case["ngon"]
    t = 2 * math.pi * torch.arange(m, device="cuda", dtype=torch.float64) / m
    a = torch.arange(rows, device="cuda", dtype=torch.float64)
    b = torch.arange(cols, device="cuda", dtype=torch.float64)
    phi = torch.where(torch.arange(rows, device="cuda") % 2 == 0, math.radians(25.0), -math.radians(25.0)).double()
    p = torch.empty(rows, cols, m, 3, device="cuda", dtype=torch.float64)
    p[..., 0] = torch.cos(t) + 1.3 * a[:, None, None]
    p[..., 1] = torch.sin(t) * torch.cos(phi)[:, None, None] + 1.3 * b[None, :, None]
    p[..., 2] = (torch.sin(t) * torch.sin(phi)[:, None, None]).expand(rows, cols, m)
    p = p.reshape(rows * cols, m, 3)
    return p + 0.02 * (_rand(g, rows * cols, m, 3) - 0.5)


def _walks(g, case):
    n, m = case["loops"], case["steps"]
    return _walk(g, n, m) + _cube(n, m) * _rand(g, n, 1, 3)


def _mixed(g, case):
    """Half torus knots, half walks; sizes log-uniform in [16, 2^18], the centres in a cube of
    side 600 for 5,000 loops and as dense for fewer."""
    n = case["loops"]
    size = torch.exp(math.log(16) + _rand(g, n) * (math.log(2 ** 18) - math.log(16))).long().tolist()
    knot = (_rand(g, n) < 0.5).tolist()
    pq = [(p, q) for p in range(2, 10) for q in range(2, 10) if math.gcd(p, q) == 1 and p != q]
    which = torch.randint(len(pq), (n,), generator=g, device="cuda").tolist()
    centre = 600.0 * (n / 5000.0) ** (1 / 3) * _rand(g, n, 3)
    out = []
    for k in range(n):
        m = max(size[k], 16)
        if knot[k]:
            p, q = pq[which[k]]
            t = 2 * math.pi * torch.arange(m, device="cuda", dtype=torch.float64) / m
            r = 1.0 + 0.4 * torch.cos(q * t)
            v = torch.stack([r * torch.cos(p * t), r * torch.sin(p * t), 0.4 * torch.sin(q * t)], dim=1)
            v = v * (0.5 * m ** 0.25 + 1.0)
        else:
            v = _walk(g, 1, m, 0.3)[0]
        out.append(v + centre[k])
    return out


def _knit(g, case):
    """Courses of a plain-knitted tube: `stitches` stitches of 16 control points around each
    course, neighbouring courses interlocked, the points jittered."""
    n, m = case["loops"], case["stitches"]
    k = torch.arange(16 * m, device="cuda", dtype=torch.float64)
    t = 2 * math.pi * k / 16
    width = 5.5
    x = k / 16 * width + 1.2 * torch.sin(2 * t)
    radius = width * m / (2 * math.pi) + 0.9 * torch.cos(2 * t)
    ang = 2 * math.pi * x / (width * m)
    z = 4.0 * torch.cos(t)
    p = torch.stack([radius * torch.cos(ang), radius * torch.sin(ang), z], dim=1).repeat(n, 1, 1)
    p[:, :, 2] += 4.6 * torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
    return p + 0.04 * (_rand(g, n, 16 * m, 3) - 0.5)


_MAKE = {"rings": _rings, "mail": _mail, "walks": _walks, "polymer": _walks, "mixed": _mixed, "knit": _knit,
         "cert": _walks}


def _curves(case, seed):
    """The curves' control points as a BCC file stores them (float32 values): a list of (n, 3)
    tensors, or one (loops, n, 3) tensor."""
    c = _MAKE[case["kind"]](_gen(seed), case)
    if torch.is_tensor(c):
        return c.float().double().contiguous()
    return [v.float().double() for v in c]


def _pair_curves(case, seed):
    """A closed curve and four that coil around it a random number of times each (their linking
    numbers), in host arrays."""
    r = np.random.default_rng(int(seed) + 99)
    out = []
    for k in range(5):
        n = case["n1"] if k == 0 else case["n2"]
        t = 2 * np.pi * np.arange(n) / n + r.uniform(0, 6)
        if k == 0:
            c = np.stack([np.cos(t), np.sin(t), np.zeros(n)], axis=1)
        else:
            w = int(r.integers(-n // 16, n // 16 + 1))
            tube = 0.2 + 0.1 * k / 4
            c = np.stack([(1 + tube * np.cos(w * t)) * np.cos(t), (1 + tube * np.cos(w * t)) * np.sin(t),
                          tube * np.sin(w * t)], axis=1)
        out.append(np.ascontiguousarray(c + r.uniform(-0.002, 0.002, size=c.shape)))
    return out


def _host(curves):
    """(counts of closed curves, xyz) in host memory, as Model.SetCurves takes them."""
    if torch.is_tensor(curves):
        return np.full(curves.shape[0], -curves.shape[1], dtype=np.int32), curves.reshape(-1, 3).cpu().numpy()
    return np.array([-len(c) for c in curves], dtype=np.int32), torch.cat(curves).cpu().numpy()


# ---------------------------------------------------------------- the calls


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pair":
        engine()
        return {"case": case, "curves": _pair_curves(case, seed)}
    counts, xyz = _host(_curves(case, seed))
    if kind in ("knit", "cert"):
        return {"case": case, "engine": engine(), "counts": counts, "xyz": xyz,
                "spline": case.get("spline", POLYLINE), "direct": case.get("method", "bh") != "bh"}
    # The linking-number stage: polylines after Discretize and their potential
    # pairs, resident in device memory, with the caller's output arrays.
    off, poly, pairs, _ = Model().SetCurves(POLYLINE, counts, xyz).Prepare(engine=engine())
    dev = torch.device("cuda")
    n = len(off) - 1
    n = n * (n - 1) // 2  # the output arrays have room for every pair of loops
    method = case.get("method", "bh")
    st = {"case": case, "engine": engine(), "npairs": len(pairs), "nloops": len(off) - 1, "bh": method == "bh",
          "xyz": torch.from_numpy(poly).to(dev), "off": torch.from_numpy(off).to(dev),
          "pairs": torch.from_numpy(pairs).to(dev), "lk": torch.zeros(n, dtype=torch.float64, device=dev),
          "err": torch.zeros(n, dtype=torch.float64, device=dev),
          "flags": torch.zeros(n, dtype=torch.int32, device=dev)}
    precision = _native.PREC_FP64 if method == "fp64" else _native.PREC_MIXED
    st["params"] = _native.default_params(precision=precision)
    return st


def _table(a, n):
    """The rows of `a` in a table with a row for each of the n pairs of loops."""
    t = np.zeros((n,) + a.shape[1:], dtype=a.dtype)
    t[:len(a)] = a
    return t


def run(st):
    kind = st["case"]["kind"]
    if kind == "pair":
        first, *others = st["curves"]
        return [ComputeLinkingNumberDirectFast(first, c) for c in others]
    if kind in ("knit", "cert"):
        model = Model().SetCurves(st["spline"], st["counts"], st["xyz"])
        cert = LinkingNumberCertificate().ComputeFromModel(model, force_direct_sum=st["direct"], engine=st["engine"])
        pairs, lk, err, flags = cert.pairs()
        n = len(st["counts"]) * (len(st["counts"]) - 1) // 2
        return {"entries": _table(cert.entries(), n), "pairs": _table(pairs, n), "lk": _table(lk, n),
                "err": _table(err, n), "flags": _table(flags, n)}
    st["engine"].linking_numbers_device(
        st["xyz"].data_ptr(), st["off"].data_ptr(), st["nloops"], st["pairs"].data_ptr(), st["npairs"],
        st["lk"].data_ptr(), st["err"].data_ptr(), st["flags"].data_ptr(),
        method="barneshut" if st["bh"] else "directsum", params=st["params"])
    return {"lk": st["lk"], "err": st["err"], "flags": st["flags"]}


# ---------------------------------------------------------------- work

TERM = 60      # operations of a segment-pair term (vectors, norms, dots, determinant, angle)
NEAR = 400     # Barnes-Hut operations per segment and interpenetrating loop at the polymer density


def _overlap(loops, extent, cube):
    """Loops whose boxes meet a given one's: boxes of side `extent`, centres uniform in a cube."""
    x = min(1.0, extent / cube)
    return (loops - 1) * (1 - (1 - x) ** 2) ** 3


def work(case):
    kind = case["kind"]
    if kind == "pair":
        return {"bytes": 96 * (case["n1"] + case["n2"]) + 32, "flops": 4 * TERM * case["n1"] * case["n2"]}
    if kind == "rings":
        seg, pairs, pair_segs = case["loops"] * case["ngon"], case["loops"] - 1, case["ngon"] ** 2
    elif kind == "mail":
        seg, pairs = case["rows"] * case["cols"] * case["ngon"], 4 * case["rows"] * case["cols"]
        pair_segs = case["ngon"] ** 2
    elif kind == "walks":
        seg, pairs = case["loops"] * case["steps"], case["loops"] * (case["loops"] - 1) // 2
        pair_segs = case["steps"] ** 2
    elif kind in ("polymer", "cert"):
        n, m = case["loops"], case["steps"]
        near = _overlap(n, 1.15 * math.sqrt(m), _cube(n, m))
        seg, pairs, pair_segs = 1.4 * n * m, n * near / 2, None
        flops = NEAR * seg * near / 2
    elif kind == "mixed":
        n = case["loops"]
        seg, pairs = n * (2 ** 18 - 16) / math.log(2 ** 14), 8 * n
        flops, pair_segs = NEAR * seg * 8, None
    else:
        n = case["loops"]
        seg, pairs = 16.0 * n * case["stitches"], 3 * n
        pair_segs = (16.0 * case["stitches"]) ** 2
    if pair_segs is not None:
        flops = TERM * pairs * pair_segs if case["method"] != "bh" else NEAR * 2 * seg
    return {"bytes": 24 * seg + 28 * pairs, "flops": flops}


# ---------------------------------------------------------------- 64 bits


def _gauss(p0, p1, b):
    """Gauss integral of the segments p0 -> p1 (..., n, 3) with the closed polylines b (..., m, 3)
    in FP64: per segment pair the signed areas of the two spherical triangles of its
    quadrilateral, over 4 pi."""
    b1 = torch.roll(b, -1, -2)

    def vec(q, p):
        return [q[..., None, :, k] - p[..., :, None, k] for k in range(3)]

    def dot(u, v):
        return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]

    va, vb, vc, vd = vec(b, p0), vec(b, p1), vec(b1, p1), vec(b1, p0)
    la, lb, lc, ld = (torch.sqrt(dot(v, v)) for v in (va, vb, vc, vd))
    det = (va[0] * (vb[1] * vc[2] - vb[2] * vc[1]) + va[1] * (vb[2] * vc[0] - vb[0] * vc[2])
           + va[2] * (vb[0] * vc[1] - vb[1] * vc[0]))
    ca = dot(vc, va)
    d1 = la * lb * lc + dot(va, vb) * lc + ca * lb + dot(vc, vb) * la
    d2 = la * ld * lc + dot(va, vd) * lc + ca * ld + dot(vc, vd) * la
    return (torch.atan2(det, d1) + torch.atan2(det, d2)).sum(dim=(-1, -2)) / (2 * math.pi)


def _links(curves, pairs):
    """FP64 linking numbers of equal-sized closed polylines (loops, n, 3) for each pair. The
    integral is a whole number for closed polylines that do not touch; the sum is rounded to it."""
    n = curves.shape[1]
    nxt = torch.roll(curves, -1, 1)
    out = torch.zeros(len(pairs), dtype=torch.float64, device="cuda")
    block = 25_000_000  # segment pairs at a time
    step = max(1, block // (n * n))
    for k in range(0, len(pairs), step):
        i, j = pairs[k:k + step, 0], pairs[k:k + step, 1]
        for r in range(0, n, max(1, block // n)):
            h = min(n, r + max(1, block // n))
            out[k:k + step] += _gauss(curves[i, r:h], nxt[i, r:h], curves[j])
    return torch.round(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pair":
        a, *others = (torch.from_numpy(c).cuda() for c in _pair_curves(case, seed))
        return [float(torch.round(_gauss(a, torch.roll(a, -1, 0), b))) for b in others]
    if kind in ("mixed", "knit", "cert") or (kind == "polymer" and case["loops"] * case["steps"] > 300_000):
        return None
    c = _curves(case, seed)
    lo, hi = c.amin(dim=1), c.amax(dim=1)
    meet = ((lo[:, None] <= hi[None]) & (lo[None] <= hi[:, None])).all(dim=-1)
    pairs = torch.nonzero(torch.triu(meet, diagonal=1))
    lk = torch.zeros(len(c) * (len(c) - 1) // 2, dtype=torch.float64, device="cuda")
    lk[:len(pairs)] = _links(c, pairs)
    return {"lk": lk, "err": torch.zeros_like(lk) if case.get("method") in ("fp64", "mixed") else None, "flags": None}
