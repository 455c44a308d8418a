"""What this library is used for, as timed cases.

Every case goes through the public entry points of ``qbgpu``: assembly of the
boundary operators, the Beyn contour step in both precision forms, the
sigma_min sweep and the EBIM eigen step. ``exact`` restates each of them in
plain torch / numpy at 64 bits (Bessel functions of a real argument by
recurrences and asymptotics, complex wavenumbers by the multiplication theorem).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quantumbilliards.jl_gb300"))
import qbgpu as qb  # noqa: E402

TWO_PI = 2.0 * math.pi
SVD_TOL = 1e-10
HOLE = (0.3, 0.1, 0.2)
# outer boundary length, diameter and area of the shapes
SHAPES = {
    "circle": (TWO_PI, 2.0, math.pi),
    "circle_hole": (TWO_PI, 2.0, math.pi * 0.96),
    "star": (8.28, 2.4, math.pi * 1.02),
    "stadium": (4.0 + TWO_PI, 4.0, 4.0 + math.pi),
}


def listed():
    return [
        # one matrix of a small discretisation on the host: the smallest call, all latency
        dict(name="matrix dlp 128", kind="matrix", form="dlp", shape="circle", n=128, k=20.0),
        # the matrices of a wavenumber window, written to the caller's device buffers
        dict(name="matrices dlp 602 x24", kind="matrices", form="dlp", shape="star", n=602, k=60.0, nk=24, deriv=False),
        # A, A', A'' of a domain with a hole, as an EBIM window wants them
        dict(name="matrices cfie 1030 d2", kind="matrices", form="cfie", shape="circle_hole", n=858, k=80.0, nk=1, deriv=True),
        # a Beyn disk low in the spectrum: small operators, launches and latencies
        dict(name="beyn mixed 256", kind="beyn", form="cfie", shape="stadium", n=256, k=20.0, nq=16, cols=32, disks=1, mixed=True, chunk=0, tuned=False),
        # the benchmark's disk: star, 48 nodes, 64 probes and their 64 of the regrowth
        dict(name="beyn mixed 2048", kind="beyn", form="cfie", shape="star", n=2048, k=200.0, nq=48, cols=128, disks=1, mixed=True, chunk=0, tuned=True),
        # several disks of the desymmetrised stadium in one batch (m = n / 4)
        dict(name="beyn mixed 1024 x8 disks", kind="beyn", form="dlp", shape="stadium", n=4096, k=300.5, nq=48, cols=96, disks=8, mixed=True, chunk=0, tuned=True),
        # high in the spectrum: large operators streamed through the handle in two groups
        dict(name="beyn mixed 5002 streamed", kind="beyn", form="cfie", shape="stadium", n=5002, k=400.0, nq=16, cols=96, disks=1, mixed=True, chunk=8, tuned=True),
        # the drop-in form, FP64 throughout
        dict(name="beyn fp64 1502", kind="beyn", form="cfie", shape="star", n=1502, k=140.0, nq=24, cols=64, disks=1, mixed=False, chunk=0, tuned=True),
        # the whole call of a spectrum driver: eigenvalues of one disk
        dict(name="solve mixed 1030", kind="solve", form="cfie", shape="circle_hole", n=858, k=90.0, nq=40, r=40, mixed=True),
        # the sweep of sigma_min over a fine grid of wavenumbers, and over larger operators
        dict(name="sweep dlp 512 x200", kind="sweep", form="dlp", shape="circle", n=512, k=40.0, nk=200, width=2.0),
        dict(name="sweep cfie 1130 x16", kind="sweep", form="cfie", shape="stadium", n=1130, k=75.0, nk=16, width=0.2),
        # one EBIM window
        dict(name="ebim 2048", kind="ebim", form="cfie", shape="stadium", n=2048, k=150.0, nev=5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _even(x, to=2):
    return int(round(x / to)) * to


def draw(rng):
    kind = rng.choice(["matrix", "matrices", "beyn", "beyn", "beyn", "beyn64", "solve", "sweep", "ebim"])
    form, shape = rng.choice([("dlp", "circle"), ("dlp", "star"), ("cfie", "star"), ("cfie", "circle_hole"), ("cfie", "stadium")])
    c = dict(kind=kind, form=form, shape=shape)

    def size(lo, hi):
        n = _even(_log(rng, lo, hi))
        c.update(n=n, k=round(max(3.0, n * TWO_PI / (SHAPES[shape][0] * rng.uniform(8.0, 11.0))), 3))
        return n

    if kind == "matrix":
        size(64, 1200)
    elif kind == "matrices":
        n = size(100, 1600)
        c.update(deriv=rng.random() < 0.5)
        c.update(nk=max(1, int(_log(rng, 1, min(48, 24 * (700.0 / n) ** 2 + 1)))))
    elif kind in ("beyn", "beyn64"):
        mixed = kind == "beyn"
        c.update(kind="beyn", mixed=mixed, tuned=rng.random() < 0.7, disks=1, chunk=0)
        if mixed and rng.random() < 0.25:  # disks of a reduced operator
            c.update(form="dlp", shape="stadium")
            shape = "stadium"
            n = 4 * int(_log(rng, 100, 1024))
            c.update(n=n, k=round(n * TWO_PI / (SHAPES[shape][0] * rng.uniform(8.0, 11.0)), 3), disks=rng.randint(2, 8), nq=_even(rng.uniform(24, 48)))
        else:
            n = size(128, 4000 if mixed else 1500)
            most = (16 * 5000.0 ** 3 if mixed else 24 * 1500.0 ** 3) / float(n) ** 3
            c.update(nq=max(6, min(rng.randint(16, 64), int(most))))
            if mixed and rng.random() < 0.2:
                c.update(chunk=max(2, c["nq"] // 3))
        c.update(cols=rng.randint(16, min(128, c["n"] // 8)) if c["n"] >= 136 else 16)
    elif kind == "solve":
        form, shape = c["form"], c["shape"] = "cfie", rng.choice(["circle_hole", "stadium"])
        size(200, 1500)
        length, _, area = SHAPES[shape]
        count = area * c["k"] / TWO_PI
        c.update(nq=rng.randint(32, 48), r=int(count + 12), mixed=rng.random() < 0.7)
    elif kind == "sweep":
        n = size(100, 1200)
        c.update(nk=max(2, min(rng.randint(16, 200), int(200 * (512.0 / n) ** 3))), width=round(rng.uniform(0.1, 2.0), 3))
    else:
        c.update(form="cfie", shape=rng.choice(["circle_hole", "stadium"]))
        shape = c["shape"]
        size(160, 2048)
        c.update(nev=rng.randint(3, 8))
    return c


def _reduced(case):
    return case["kind"] == "beyn" and case["form"] == "dlp" and case["shape"] == "stadium"


def _dim(case):
    n = case["n"]
    if _reduced(case):
        return n // 4
    if case["shape"] != "circle_hole":
        return n
    hole = max(20, int(round(n * HOLE[2])))
    return n + hole + hole % 2


def _k0(case, seed):
    return case["k"] + float(np.random.default_rng([seed, 1]).uniform(0.0, 0.4))


def _ks(case, seed):
    k0 = _k0(case, seed)
    if case["kind"] == "sweep":
        return np.linspace(k0, k0 + case["width"], case["nk"])
    return k0 + 0.01 * np.arange(case.get("nk", 1))


def _disks(case, seed):
    return _k0(case, seed) + np.arange(case.get("disks", 1)), 0.5


def _cols(case):
    return 2 * case["r"] if case["kind"] == "solve" else case["cols"]


def _probes(case, seed):
    rng = np.random.default_rng([seed, 2])
    shape = (_dim(case), _cols(case))
    return np.asfortranarray(math.sqrt(0.5) * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)))


def _panels(case):
    """Panel counts at degree 9 that the library's tuner comes to at 1e-13 (7695 and 863 for the benchmark's disk)."""
    if not case.get("tuned", True):
        return None
    return int(3.8 * case["n"]) + 50, 9, int(1.8 * (case["k"] + case.get("disks", 1)) * SHAPES[case["shape"]][1]) + 50, 9


def _ebim_dk(case):
    return 8.0 / _count(case)


def _count(case):
    """Eigenvalues per unit of k (Weyl)."""
    length, _, area = SHAPES[case["shape"]]
    return max(1.0, area * case["k"] / TWO_PI - length / (2.0 * TWO_PI))


def _nearest(case, lam, k0):
    """The eigenvalues well inside the disk, as many as are expected there."""
    lam = lam[np.argsort(np.abs(lam - k0))][:max(1, int(0.7 * _count(case)) - 2)]
    return lam[np.argsort(lam.real)]


def prepare(case, seed):
    shape = case["shape"]
    b = {"circle": qb.make_circle, "star": qb.make_star, "stadium": qb.make_full_stadium, "circle_hole": lambda: qb.make_circle_with_hole(1.0, HOLE)}[shape]()
    if case["form"] == "dlp":
        sol = qb.DLP_kress(1.0, b) if shape != "stadium" else qb.DLP_kress_global_corners(1.0, b, symmetry=qb.XYReflection(-1, -1))
    else:
        sol = qb.CFIE_kress(1.0, b) if shape != "stadium" else qb.CFIE_kress_global_corners(1.0, b)
    pts, sol = qb.points_with_n(sol, b, case["n"], case["k"])
    ws = qb.Workspace(sol, pts)
    if ws.dim != _dim(case):
        raise ValueError("the discretisation has %d nodes, not %d" % (ws.dim, _dim(case)))
    s = dict(case=case, sol=sol, pts=pts, ws=ws, k0=_k0(case, seed), ks=_ks(case, seed), seed=seed)
    if case["kind"] == "matrices":
        m = case["nk"] * (3 if case["deriv"] else 1)
        s["out"] = torch.empty((m, ws.dim, ws.dim), dtype=torch.complex128, device="cuda")
        s["ptrs"] = [s["out"][i].data_ptr() for i in range(m)]
    elif case["kind"] == "beyn":
        s["V"] = _probes(case, seed)
    return s


def run(s):
    case, ws = s["case"], s["ws"]
    kind = case["kind"]
    if kind == "matrix":
        return qb.construct_matrices(s["sol"], s["pts"], ws, s["k0"])
    if kind == "matrices":
        qb.assemble_noalloc(ws, s["ks"], s["ptrs"], deriv=case["deriv"])
        return s["out"]  # column-major matrices
    if kind == "beyn":
        k0s, R = _disks(case, s["seed"])
        bh = qb.BeynHandle(ws, k0s if case["disks"] > 1 else k0s[0], R, case["nq"], mixed=case["mixed"], cheb=_panels(case), node_chunk=case["chunk"])
        try:
            return bh.moments(s["V"])
        finally:
            bh.close()
    if kind == "solve":
        k0, R = s["k0"], 0.5
        lam = qb.solve(s["sol"], s["pts"], k0, R, nq=case["nq"], r=case["r"], svd_tol=SVD_TOL, rng=np.random.default_rng([s["seed"], 2]), mixed=case["mixed"], ws=ws, cheb=_panels(case))
        return _nearest(case, lam, k0)
    if kind == "sweep":
        return qb.sigma_min(ws, s["ks"])
    return qb.ebim.solve(ws, s["k0"], _ebim_dk(case), nev=case["nev"])


def work(case):
    d = float(_dim(case))
    entry = 150.0  # operations of one kernel entry: two Bessel orders and the fold
    kind = case["kind"]
    if kind in ("matrix", "matrices"):
        m = case.get("nk", 1)
        return dict(bytes=16.0 * d * d * m * (3 if case.get("deriv") else 1) + 64.0 * d, flops=entry * d * d * m)
    if kind in ("beyn", "solve"):
        nodes, cols = float(case["nq"] * case.get("disks", 1)), float(_cols(case))
        entries = nodes * d * d * (4.0 if _reduced(case) else 1.0)
        out = 32.0 * d * cols * case.get("disks", 1) if kind == "beyn" else 16.0 * cols
        return dict(bytes=16.0 * d * cols + out + 64.0 * d, flops=entry * entries + nodes * (8.0 / 3.0 * d ** 3 + 8.0 * d * d * cols))
    if kind == "sweep":
        return dict(bytes=64.0 * d + 16.0 * case["nk"], flops=case["nk"] * (entry * d * d + 8.0 / 3.0 * d ** 3))
    return dict(bytes=64.0 * d + 32.0 * case["nev"], flops=3.0 * entry * d * d + 8.0 / 3.0 * d ** 3 + 16.0 * d ** 2 * 20.0)


# --------------------------------------------------------------------------
# the same in plain torch and numpy at 64 bits
# --------------------------------------------------------------------------
def _arc(radius, angle, shift, cx, cy):
    def at(u):
        t = angle * u + shift
        c, s = np.cos(t), np.sin(t)
        return (cx + radius * c, cy + radius * s), (-radius * angle * s, radius * angle * c), (-radius * angle ** 2 * c, -radius * angle ** 2 * s)
    return at, radius * angle


def _line(p, q):
    def at(u):
        z = 0.0 * u
        return (p[0] + u * (q[0] - p[0]), p[1] + u * (q[1] - p[1])), (z + q[0] - p[0], z + q[1] - p[1]), (z, z)
    return at, math.hypot(q[0] - p[0], q[1] - p[1])


def _star(u):
    t = TWO_PI * u
    r, r1, r2 = 1.0 + 0.2 * np.cos(5 * t), -1.0 * np.sin(5 * t), -5.0 * np.cos(5 * t)
    c, s = np.cos(t), np.sin(t)
    w = TWO_PI
    return (r * c, r * s), (w * (r1 * c - r * s), w * (r1 * s + r * c)), (w * w * (r2 * c - 2 * r1 * s - r * c), w * w * (r2 * s + 2 * r1 * c - r * s))


def _nodes(case):
    """Components as dicts of float64 CUDA vectors; the parameter runs over 2 pi, a hole backwards."""
    def sample(pieces, n):
        sig = TWO_PI * (np.arange(n) + 0.5) / n
        lens = np.array([l for _, l in pieces])
        cum = np.concatenate([[0.0], np.cumsum(lens)])
        at = sig / TWO_PI * cum[-1]
        out = np.zeros((7, n))
        out[6] = sig
        which = np.clip(np.searchsorted(cum, at, side="right") - 1, 0, len(lens) - 1)
        for j, (f, l) in enumerate(pieces):
            m = which == j
            p, t, a = f((at[m] - cum[j]) / l)
            f1 = cum[-1] / (TWO_PI * l)
            out[0, m], out[1, m] = p
            out[2, m], out[3, m] = t[0] * f1, t[1] * f1
            out[4, m], out[5, m] = a[0] * f1 * f1, a[1] * f1 * f1
        return out

    shape, n = case["shape"], case["n"]
    if shape == "star":
        comps = [sample([(_star, 1.0)], n)]
    elif shape == "stadium":
        comps = [sample([_arc(1.0, math.pi / 2, 0.0, 1.0, 0.0), _line((1.0, 1.0), (-1.0, 1.0)), _arc(1.0, math.pi, math.pi / 2, -1.0, 0.0), _line((-1.0, -1.0), (1.0, -1.0)), _arc(1.0, math.pi / 2, 1.5 * math.pi, 1.0, 0.0)], n)]
    else:
        comps = [sample([_arc(1.0, TWO_PI, 0.0, 0.0, 0.0)], n)]
        if shape == "circle_hole":
            h = sample([_arc(HOLE[2], TWO_PI, 0.0, HOLE[0], HOLE[1])], _dim(case) - n)[:, ::-1].copy()
            h[2:4] *= -1.0
            comps.append(h)
    names = ("x", "y", "dx", "dy", "ddx", "ddy", "ts")
    return [{k: torch.tensor(v, device="cuda") for k, v in zip(names, c)} for c in comps]


def _miller(x, top):
    """J0, J1, Y0, Y1 by backward recurrence from order `top` and the Neumann series of Y."""
    hi, lo = torch.zeros_like(x), torch.full_like(x, 1e-250)
    norm, sy0, sy1, j1 = (torch.zeros_like(x) for _ in range(4))
    for m in range(top, 0, -1):  # lo = J_m, hi = J_{m+1}, up to one factor
        q = m // 2
        if m % 2 == 0:
            norm += 2.0 * lo
            sy0 += ((-1.0) ** q / q) * lo
        elif m == 1:
            j1 = lo
        else:
            sy1 += ((-1.0) ** q * (2.0 * q + 1.0) / (q * (q + 1.0))) * lo
        hi, lo = lo, (2.0 * m / x) * lo - hi
    s = 1.0 / (norm + lo)
    j0, j1 = lo * s, j1 * s
    lg = torch.log(0.5 * x) + np.euler_gamma
    y0 = (2.0 / math.pi) * lg * j0 - (4.0 / math.pi) * s * sy0
    y1 = (2.0 / math.pi) * ((lg - 1.0) * j1 - j0 / x - s * sy1)
    return j0, j1, y0, y1


def _hankel(x):
    """J0, J1, Y0, Y1 by the asymptotic expansion for large x."""
    got = []
    c, s = torch.cos(x), torch.sin(x)
    amp = torch.sqrt(1.0 / (math.pi * x))
    for nu in (0, 1):
        P, Q, t = torch.zeros_like(x), torch.zeros_like(x), torch.ones_like(x)
        for m in range(26):
            if m % 2 == 0:
                P += (-1.0) ** (m // 2) * t
            else:
                Q += (-1.0) ** (m // 2) * t
            t = t * ((4.0 * nu * nu - (2.0 * m + 1.0) ** 2) / (8.0 * (m + 1.0))) / x
        if nu == 0:  # phase x - pi/4
            C, S = c + s, s - c
        else:  # phase x - 3 pi/4
            C, S = s - c, -(c + s)
        got.append((amp * (P * C - Q * S), amp * (P * S + Q * C)))
    return got[0][0], got[1][0], got[0][1], got[1][1]


def _real_bessel(x):
    out = [torch.empty_like(x) for _ in range(4)]
    for at, f in ((x < 2.0, lambda t: _miller(t, 24)), ((x >= 2.0) & (x < 25.0), lambda t: _miller(t, 76)), (x >= 25.0, _hankel)):
        if bool(at.any()):
            for o, v in zip(out, f(x[at])):
                o[at] = v
    return out


def _bessel(k, r):
    """H0, H1, J0, J1 of k r; complex k by C_v(l x) = l^v sum_m (1 - l^2)^m (x/2)^m / m! C_{v+m}(x), l = k / Re k."""
    kr = k.real if isinstance(k, complex) else k
    x = kr * r
    j0, j1, y0, y1 = _real_bessel(x)
    if not isinstance(k, complex) or k.imag == 0.0:
        return torch.complex(j0, y0), torch.complex(j1, y1), j0.to(torch.complex128), j1.to(torch.complex128)
    lam = k / kr
    q = 1.0 - lam * lam
    got = []
    for a, b in ((j0, j1), (y0, y1)):
        s0, s1 = a.to(torch.complex128), b.to(torch.complex128)
        t = torch.ones_like(x)  # (x/2)^m / m!
        lo, hi, qm = a, b, 1.0 + 0j
        for m in range(1, 40):
            t = t * (0.5 * x / m)
            qm *= q
            lo, hi = hi, (2.0 * m / x) * hi - lo
            d0, d1 = t * lo, t * hi
            s0 += qm * d0
            s1 += qm * d1
            if m >= 12 and m % 4 == 0 and abs(qm) * float(torch.maximum(d0.abs().max(), d1.abs().max())) < 1e-17:
                break
        got.append((s0, lam * s1))
    (J0, J1), (Y0, Y1) = got
    return J0 + 1j * Y0, J1 + 1j * Y1, J0, J1


def _kress(n):
    m = torch.zeros(n, dtype=torch.float64, device="cuda")
    m[1:n // 2] = 1.0 / torch.arange(1, n // 2, dtype=torch.float64, device="cuda")
    m[n // 2 + 1:] = m[1:n // 2].flip(0)
    i = torch.arange(n, device="cuda")
    c = -TWO_PI * torch.fft.ifft(m).real - (2.0 * TWO_PI / n ** 2) * (1.0 - 2.0 * (i % 2))
    return c[(i[:, None] - i[None, :]) % n]


def _pair(p, q):
    dx, dy = p["x"][:, None] - q["x"][None, :], p["y"][:, None] - q["y"][None, :]
    r = torch.hypot(dx, dy)
    return r, q["dy"][None, :] * dx - q["dx"][None, :] * dy


def _operator(case, comps, k, deriv=False):
    """A(k) (and A', A'') of the unreduced operator; I - D, or I - (D + i k S)."""
    cfie = case["form"] == "cfie"
    off = np.concatenate([[0], np.cumsum([len(c["x"]) for c in comps])])
    out = [torch.zeros((off[-1], off[-1]), dtype=torch.complex128, device="cuda") for _ in range(3 if deriv else 1)]
    ik, pi = 1j * k, math.pi
    for a, p in enumerate(comps):
        for b, q in enumerate(comps):
            r, inner = _pair(p, q)
            w = TWO_PI / len(q["x"])
            speed = torch.hypot(q["dx"], q["dy"])[None, :]
            if a == b:
                eye = torch.eye(len(r), dtype=torch.bool, device="cuda")
                r = torch.where(eye, torch.ones_like(r), r)
                h0, h1, j0, j1 = _bessel(k, r)
                R = _kress(len(r))
                lt = torch.log(4.0 * torch.sin(0.5 * (p["ts"][:, None] - p["ts"][None, :])) ** 2 + eye)
                l1 = -k / TWO_PI * inner * j1 / r
                D = R * l1 + w * (0.5j * k * inner * h1 / r - l1 * lt)
                kap = -(p["dx"] * p["ddy"] - p["dy"] * p["ddx"]) / (p["dx"] ** 2 + p["dy"] ** 2) / TWO_PI
                D[eye] = (w * kap).to(torch.complex128)
                blk = [eye.to(torch.complex128) - D]
                if deriv:
                    kr = k * r
                    D1 = R * (-(inner * k * j0) / TWO_PI) + w * (inner * k * (lt * j0 + 1j * pi * h0) / TWO_PI)
                    D2 = R * (inner * (kr * j1 - j0) / TWO_PI) + w * (inner * (lt * (j0 - kr * j1) + 1j * pi * (h0 - kr * h1)) / TWO_PI)
                    D1[eye] = D2[eye] = 0.0
                    blk += [-D1, -D2]
                if cfie:
                    s = speed[0]
                    m1 = -j0 * speed / TWO_PI
                    S = R * m1 + w * (0.5j * h0 * speed - m1 * lt)
                    half = np.euler_gamma / pi
                    S[eye] = torch.diagonal(R) * (-s / TWO_PI) + w * ((0.5j - half) - torch.log((k * k / 4.0) * s * s + 0j) / TWO_PI) * s
                    blk[0] = blk[0] - ik * S
                    if deriv:
                        S1 = R * (r * speed * j1 / TWO_PI) - w * (r * speed * (lt * j1 + 1j * pi * h1) / TWO_PI)
                        S2 = R * (r * speed * (kr * j0 - j1) / (TWO_PI * k)) + w * (r * speed * (lt * (j1 - kr * j0) - 1j * pi * kr * h0 + 1j * pi * h1) / (TWO_PI * k))
                        S1[eye] = (-w * s / (pi * k)).to(torch.complex128)
                        S2[eye] = (w * s / (pi * k * k)).to(torch.complex128)
                        blk[1] = blk[1] - 1j * S - ik * S1
                        blk[2] = blk[2] - 2j * S1 - ik * S2
            else:
                h0, h1, _, _ = _bessel(k, r)
                S = w * 0.5j * h0 * speed
                blk = [-(w * 0.5j * k * inner * h1 / r + ik * S)]
                if deriv:  # the sign of the double layer's derivatives between components is the operator's definition
                    kr = k * r
                    S1, S2 = w * (-0.5j) * r * h1 * speed, w * 0.5j * r * (h1 - kr * h0) * speed / k
                    blk += [-(w * (-0.5j) * inner * k * h0 + 1j * S + ik * S1), -(w * (-0.5j) * inner * (h0 - kr * h1) + 2j * S1 + ik * S2)]
            for o, x in zip(out, blk):
                o[off[a]:off[a + 1], off[b]:off[b + 1]] = x
    return out if deriv else out[0]


def _reduced_operator(p, k, R, lt):
    """I - D on a quarter of the stadium's nodes, odd in x and y: the Kress entry and three image kernels."""
    n = len(p["x"])
    m = n // 4
    f = torch.arange(m, device="cuda")
    out = torch.eye(m, dtype=torch.complex128, device="cuda")
    for idx, sign in ((f, 1.0), (n // 2 - 1 - f, -1.0), (n - 1 - f, -1.0), ((f + n // 2) % n, 1.0)):
        r, inner = _pair({g: v[f] for g, v in p.items()}, {g: v[idx] for g, v in p.items()})
        w = TWO_PI / n
        if sign > 0 and int(idx[0]) == 0:
            eye = torch.eye(m, dtype=torch.bool, device="cuda")
            r = torch.where(eye, torch.ones_like(r), r)
            _, h1, _, j1 = _bessel(k, r)
            l1 = -k / TWO_PI * inner * j1 / r
            D = R * l1 + w * (0.5j * k * inner * h1 / r - l1 * lt)
            kap = -(p["dx"] * p["ddy"] - p["dy"] * p["ddx"]) / (p["dx"] ** 2 + p["dy"] ** 2) / TWO_PI
            D[eye] = (w * kap[f]).to(torch.complex128)
        else:
            D = sign * w * 0.5j * k * inner * _bessel(k, r)[1] / r
        out -= D
    return out


def _moments(case, seed, V):
    comps = _nodes(case)
    if _reduced(case):
        m = case["n"] // 4
        R = _kress(case["n"])[:m, :m]
        ts = comps[0]["ts"][:m]
        lt = torch.log(4.0 * torch.sin(0.5 * (ts[:, None] - ts[None, :])) ** 2 + torch.eye(m, dtype=torch.float64, device="cuda"))
    k0s, rad = _disks(case, seed)
    V = torch.tensor(V, device="cuda")
    A0 = torch.zeros((len(k0s),) + tuple(V.shape), dtype=torch.complex128, device="cuda")
    A1 = torch.zeros_like(A0)
    nq = case["nq"]
    for d, k0 in enumerate(k0s):
        for j in range(nq):
            e = complex(math.cos(TWO_PI * j / nq), math.sin(TWO_PI * j / nq))
            z = complex(k0) + rad * e
            T = _reduced_operator(comps[0], z, R, lt) if _reduced(case) else _operator(case, comps, z)
            X = torch.linalg.solve(T, V)
            A0[d] += (rad / nq) * e * X
            A1[d] += (rad / nq) * e * z * X
    return A0, A1


def _largest(C, nev):
    """The nev eigenpairs of largest modulus of C, by subspace iteration."""
    n = C.shape[0]
    p = min(n, 12 * nev + 24)
    g = torch.Generator(device="cuda").manual_seed(7)
    Q = torch.randn(n, p, dtype=torch.complex128, device="cuda", generator=g)
    for _ in range(40):
        Q, _ = torch.linalg.qr(C @ Q)
    mu, Y = np.linalg.eig((Q.conj().T @ (C @ Q)).cpu().numpy())
    o = np.argsort(-np.abs(mu), kind="stable")[:nev]
    return mu[o], Q @ torch.tensor(Y[:, o], device="cuda")


def exact(case, seed):
    kind = case["kind"]
    if kind == "matrix":
        return _operator(case, _nodes(case), _k0(case, seed)).cpu().numpy()
    if kind == "matrices":
        comps = _nodes(case)
        every = [_operator(case, comps, float(k), case["deriv"]) for k in _ks(case, seed)]
        every = [m[i] for i in range(3) for m in every] if case["deriv"] else every
        return torch.stack([m.T for m in every])
    if kind == "beyn":
        A0, A1 = (a.cpu().numpy() for a in _moments(case, seed, _probes(case, seed)))
        return (A0, A1) if case["disks"] > 1 else (A0[0], A1[0])
    if kind == "solve":
        A0, A1 = (a[0] for a in _moments(case, seed, _probes(case, seed)))
        U, S, W = torch.linalg.svd(A0, full_matrices=False)
        rk = int((S >= SVD_TOL).sum())
        B = U[:, :rk].conj().T @ (A1 @ W[:rk].conj().T) / S[:rk]
        lam = np.linalg.eigvals(B.cpu().numpy())
        return _nearest(case, lam, _k0(case, seed))
    comps = _nodes(case)
    if kind == "sweep":
        sig = []
        for k in _ks(case, seed):
            C = torch.linalg.inv(_operator(case, comps, float(k)))
            X = torch.randn(C.shape[0], 12, dtype=torch.complex128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
            for _ in range(25):
                X, _ = torch.linalg.qr(C.conj().T @ (C @ X))
            sig.append(1.0 / np.linalg.svd((C @ X).cpu().numpy(), compute_uv=False)[0])
        return np.array(sig)
    k, dk, nev = _k0(case, seed), _ebim_dk(case), case["nev"]
    A, dA, ddA = _operator(case, comps, k, deriv=True)
    C = torch.linalg.solve(A, dA)
    mu, V = _largest(C, nev)
    mul, U = _largest(C.conj().T.contiguous(), nev)
    kc, tens = [], []
    for j in range(nev):
        lam = 1.0 / mu[j]
        if not (abs(lam.real) < dk and abs(lam.imag) < dk):
            continue
        u, v = U[:, int(np.argmin(np.abs(mul - np.conj(mu[j]))))], V[:, j]
        num, den = complex(torch.vdot(u, ddA @ v)), complex(torch.vdot(u, dA @ v))
        t = -lam - (0.5 * lam * lam * num / den if abs(den) > 1e-15 else 0.0)
        if abs(t.real) < dk:
            kc.append(k + t.real)
            tens.append(abs(t))
    return np.array(kc), np.array(tens)
