"""What is measured: the calls a user of this framework makes, through `electricbubbles_gb300.api`.

A case is one call, or the few calls that belong together, on drops like those of the
repository's configurations: radii in [0.5, 1] (0.2 to 1 from 256 drops on), a 2- or
3-fold perturbation of a few per cent, nodes at equal arclength, some 5 radii apart. The kinds:

  apply    one operator apply on an installed geometry: what a caller's own GMRES (the
           gfortran `matvec_` callback) asks for
  solve    a new geometry and the GMRES solve on it: half an RK stage
  rk2      a whole RK2 step from positions in device memory: the time loop
  batch    an RK2 step of many independent single-drop simulations held by one context
  vjp      the transpose of an RK2 step: the backward pass of a gradient, step by step
  cauchy   the Cauchy sum on scattered points (its own tree on each call)

`exact` restates all of them in plain torch float64 with direct sums over all pairs.
"""
import functools
import math

import numpy as np
import torch

from electricbubbles_gb300.api import Context

PI = math.pi


def listed():
    return [
        # the smallest call: one drop, the operator in a caller's own GMRES loop; latency counts
        dict(name="apply_1x256", kind="apply", op="stokes", drops=1, nodes=256, prec="fp64"),
        # the reference's loop on one drop (256 nodes): a time step of a dozen small kernels a stage
        dict(name="rk2_1x256", kind="rk2", drops=1, nodes=256, mode="fp64"),
        # the Laplace operator in a caller's own loop, drops of uneven, odd sizes (117 to 890 nodes)
        dict(name="apply_laplace_ragged", kind="apply", op="laplace", drops=37, nodes=351, ragged=True, prec="fp64"),
        # SOLVEI as the reference runs it, FP64 throughout, on the workload of the benchmark
        dict(name="solve_64x512_fp64", kind="solve", op="stokes", drops=64, nodes=512, mode="fp64"),
        # the benchmark's headline: the same solve with the FP32 inner operator
        dict(name="solve_64x512_refined", kind="solve", op="stokes", drops=64, nodes=512, mode="fp32_refined"),
        # SOLVE_LAPL with the deflation that production runs use with many drops
        dict(name="solve_laplace_64x512", kind="solve", op="laplace", drops=64, nodes=512, mode="fp32_refined", deflate=True),
        # the production time step of the same workload
        dict(name="rk2_64x512_refined", kind="rk2", drops=64, nodes=512, mode="fp32_refined", deflate=True),
        # wall-bounded flow, FP64 as the reference runs it
        dict(name="solve_wall_16x256", kind="solve", op="stokes", drops=16, nodes=256, mode="fp64", wall=True),
        # the large configuration: a million nodes
        dict(name="solve_1024x1024", kind="solve", op="stokes", drops=1024, nodes=1024, mode="fp32_refined"),
        # 256 uneven simulations in lockstep (128 to 4,096 nodes each)
        dict(name="batch_256", kind="batch", sims=256, nmin=128, nmax=4096, mode="fp32_refined"),
        # one step of a gradient's backward pass: two stages rerun and transposed
        dict(name="vjp_32x64", kind="vjp", drops=32, nodes=64, mode="fp64"),
        # DAPIF2 on scattered points, an odd number of them
        dict(name="cauchy_60001", kind="cauchy", points=60001, prec="fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """The same kinds over their ranges: from one drop of 64 nodes to a quarter of a million
    nodes for an apply, 16,000 (plain FP64) or 130,000 (refined) for a solve."""
    kind = rng.choice(["apply", "apply", "solve", "solve", "rk2", "batch", "vjp", "cauchy"])
    if kind == "cauchy":
        return dict(kind=kind, points=_log(rng, 700, 200000) | 1, prec=rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "batch":
        lo = 2 ** rng.randint(6, 8)
        return dict(kind=kind, sims=_log(rng, 3, 120), nmin=lo, nmax=lo * 2 ** rng.randint(1, 4),
                    mode=rng.choice(["fp64", "fp32_refined", "fp32_refined"]))
    if kind == "vjp":
        return dict(kind=kind, drops=rng.randint(1, 48), nodes=2 ** rng.randint(5, 6), mode="fp64")
    if kind == "rk2":
        n = 2 ** rng.randint(6, 10)
        return dict(kind=kind, drops=_log(rng, 1, 30000 // n), nodes=n, mode=rng.choice(["fp64", "fp32_refined"]),
                    deflate=True)
    op = rng.choice(["stokes", "laplace"])
    ragged = rng.random() < 0.5
    n = _log(rng, 64, 1500)
    if kind == "apply":
        return dict(kind=kind, op=op, drops=_log(rng, 1, 250000 // n), nodes=n, ragged=ragged,
                    prec=rng.choice(["fp64", "fp64", "fp32"]), wall=op == "stokes" and rng.random() < 0.2)
    mode = rng.choice(["fp64", "fp32_refined"])
    return dict(kind=kind, op=op, drops=_log(rng, 1, (16000 if mode == "fp64" else 130000) // n), nodes=n,
                ragged=ragged, mode=mode, deflate=op == "laplace", wall=op == "stokes" and rng.random() < 0.2)


# ---- inputs --------------------------------------------------------------------------
@functools.lru_cache(maxsize=4096)
def _shape(n, amp, mode):
    """n nodes at equal arclength on r = 1 + amp cos(mode theta), by Newton's method on the
    arclength's Fourier series."""
    m = 512
    th = 2 * PI * np.arange(m) / m
    c = np.fft.rfft(np.hypot(1 + amp * np.cos(mode * th), amp * mode * np.sin(mode * th)))[:m // 2:mode].real / m
    k = mode * np.arange(1, min(c.size, 40))
    b = goal = 2 * PI * np.arange(n) / n
    for _ in range(12):
        s = b + (2 * c[1:k.size + 1] / (k * c[0])) @ np.sin(np.outer(k, b))
        b = b - (s - goal) / (1 + (2 * c[1:k.size + 1] / c[0]) @ np.cos(np.outer(k, b)))
    return (1 + amp * np.cos(mode * b)) * np.exp(1j * b)


def _sizes(*case):
    """Random numbers for the sizes of a case's drops, the same for every seed."""
    return np.random.default_rng(case)


def _drops(case, rng):
    """nd and the nodes z of the case's drops, one to a cell of a jittered square grid."""
    k, n = case["drops"], case["nodes"]
    nd = np.full(k, n)
    if case.get("ragged"):
        nd = np.maximum(48, np.rint(n * np.exp(_sizes(k, n).uniform(-1.1, 0.93, k)))).astype(int) | 1
    rad = np.exp(rng.uniform(np.log(0.2 if k >= 256 else 0.5), 0.0, k))
    side = int(math.ceil(math.sqrt(k)))
    cell, wall = (3.0 if case.get("wall") else 5.0), bool(case.get("wall"))
    room = 0.5 * cell - 1.1 * rad - 0.1
    spot = cell * (np.arange(k) % side + 1j * (np.arange(k) // side)) + room * (rng.uniform(-1, 1, k) + 1j * rng.uniform(-1, 1, k))
    amp, mode, turn = rng.integers(3, 8, k) / 100.0, rng.integers(2, 4, k), rng.uniform(0, 2 * PI, k)
    z = np.concatenate([c + r * np.exp(1j * t) * _shape(int(m), float(a), int(w))
                        for c, r, t, m, a, w in zip(spot, rad, turn, nd, amp, mode)])
    if wall:  # the wall is y = 0
        z = z + 1j * (0.3 - z.imag.min())
    return nd.astype(np.int32), z


def _waves(nd, rng, real=False):
    """A smooth density: a few random Fourier modes on each drop."""
    out = []
    for n in nd:
        th = np.exp(2j * PI * np.arange(n) / n)
        v = sum((rng.standard_normal() + 1j * rng.standard_normal()) * th ** p / (1 + abs(p)) for p in range(-4, 5))
        out.append(v.real if real else v)
    return np.concatenate(out)


def _ends(nd):
    e = np.concatenate([[0], np.cumsum(nd)]).astype(int)
    return list(zip(e[:-1], e[1:]))


def _geometry(nd, z):
    """What EXTRACTDAT leaves in COMMON: dz (clockwise), ds/da, the curvature and the centres."""
    dz, ds, ka, zk = [], [], [], []
    for a, b in _ends(nd):
        n = b - a
        w = np.fft.fftfreq(n, 1.0 / n)
        w[n // 2] = 0.0 if n % 2 == 0 else w[n // 2]
        f = np.fft.fft(z[a:b])
        z1, z2 = np.fft.ifft(1j * w * f), np.fft.ifft(-w * w * f)
        s = np.abs(z1)
        dz.append(-z1)
        ds.append(s)
        ka.append(-(z1.conj() * z2).imag / s ** 3)
        zk.append(z[a:b].mean())
    return np.concatenate(dz), np.concatenate(ds), np.concatenate(ka), np.array(zk)


def _flat(z):
    return np.ascontiguousarray(z).view(np.float64).copy()


def _inputs(case, seed):
    """The case's host arrays, from the seed alone (the sizes from the case)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "cauchy":
        p = case["points"]
        return dict(z=rng.uniform(-1, 1, p) + 1j * rng.uniform(-1, 1, p),
                    q=(rng.standard_normal(p) + 1j * rng.standard_normal(p)) / p)
    if kind == "batch":
        s = case["sims"]
        lo, hi = math.log2(case["nmin"]), math.log2(case["nmax"])
        nd = 2 ** np.rint(_sizes(s, case["nmin"], case["nmax"]).uniform(lo, hi, s)).astype(int)
        z = np.concatenate([_shape(int(n), float(a) / 100.0, 2) for n, a in zip(nd, rng.integers(1, 10, s))])
        return dict(nd=nd.astype(np.int32), y=_flat(z), e0=rng.uniform(0.1, 1.0, s), cap=0.0)
    nd, z = _drops(case, rng)
    if kind in ("rk2", "vjp"):
        d = dict(nd=nd, y=_flat(z), e0=float(rng.uniform(0.3, 0.7)), cap=0.1)
        return dict(d, v=_flat(_waves(nd, rng))) if kind == "vjp" else d
    dz, ds, ka, zk = _geometry(nd, z)
    d = dict(nd=nd, z=z, dz=dz, dsda=ds, kappa=ka, zk=zk)
    if kind == "apply":
        d["x"] = _waves(nd, rng, True) if case["op"] == "laplace" else _flat(_waves(nd, rng))
    elif case["op"] == "laplace":  # GETBCs with a random part of the other field component
        d["x"] = -2.0 * z.real + rng.uniform(-0.2, 0.2) * z.imag
    else:  # SETVELF's surface tension, and a far field
        d["x"] = _flat(-0.5 * dz / ds + 0.5j * rng.uniform(0.0, 0.2) * z.conj())
    return d


DT = 1e-3  # the time step of the repository's configurations
_stream = None


def prepare(case, seed):
    global _stream
    if _stream is None:  # one stream for a program's contexts and its own torch work
        _stream = torch.cuda.Stream()
    d = _inputs(case, seed)
    st = {k: torch.from_numpy(v).cuda() if isinstance(v, np.ndarray) and k not in ("nd", "e0") else v for k, v in d.items()}
    # a gradient's solves run tighter than a time step's: the transposed second derivatives
    # amplify their residual by the square of the wavenumber
    ctx = Context(lap_deflate=1 if case.get("deflate") else 0, gmres_tol=1e-13 if case["kind"] == "vjp" else 0.0)
    ctx.set_stream(_stream.cuda_stream)
    st.update(case=dict(case), ctx=ctx)
    if case.get("wall"):
        ctx.set_wall(1)
    if case["kind"] == "batch":
        ctx.batch_define(np.ones(case["sims"], np.int32), d["e0"])
    if case["kind"] == "apply":
        ctx.set_geometry(d["nd"], *(st[k] for k in ("z", "dz", "dsda", "kappa", "zk")))
    if "x" in st:
        st["out"] = torch.empty_like(st["x"])
    if case["kind"] in ("rk2", "batch", "vjp"):
        st["out"] = torch.empty_like(st["y"])
    return st


def run(state):
    st, c, ctx = state, state["case"], state["ctx"]
    kind = c["kind"]
    with torch.cuda.stream(_stream):
        if kind == "cauchy":
            return ctx.dapif2(st["z"], st["q"], c["prec"])
        if kind == "apply":
            return (ctx.fasmvp if c["op"] == "stokes" else ctx.fasmvp_lap)(st["x"], c["prec"], out=st["out"])
        if kind == "solve":
            ctx.set_geometry(st["nd"], st["z"], st["dz"], st["dsda"], st["kappa"], st["zk"])
            return (ctx.solvei if c["op"] == "stokes" else ctx.solve_lapl)(st["x"], c["mode"], out=st["out"])[0]
        if kind == "vjp":
            st["out"].copy_(st["v"])  # the cotangent is updated in place
            par, _ = ctx.rk2_vjp(st["nd"], DT, st["y"], st["out"], cap=st["cap"], e0=st["e0"], mode=c["mode"])
            return {"y": st["out"], "e0": par["e0"], "cap": par["cap"]}
        st["out"].copy_(st["y"])  # the step updates the positions in place
        e0 = 0.0 if kind == "batch" else st["e0"]
        ctx.rk2(st["nd"], DT, st["out"], cap=st["cap"], e0=e0, mode=c["mode"])
        return st["out"]


def _size(case):
    if case["kind"] == "cauchy":
        return case["points"]
    if case["kind"] == "batch":  # the mean of a log-uniform size
        return int(case["sims"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"]))
    return case["drops"] * case["nodes"]


def work(case):
    """Bytes: the inputs and outputs once. Operations: per node and layer sum the pairs with
    some 50 near neighbours and four expansions of the order the precision needs (or all
    pairs, where that is less), times the sums that the call cannot do without: one for an
    apply, about 10 for a solve, 22 for a stage
    (two solves, two sums); a transposed step reruns three stages and transposes two."""
    n, kind = _size(case), case["kind"]
    two = kind in ("rk2", "batch", "vjp") or case.get("op") == "stokes"
    order = 20 if "fp32" in case.get("prec", "") + case.get("mode", "") else 44
    per = min(n, 50) * (30 if two else 12) + min(4 * 8 * order * (2 if two else 1), n * 30)
    sums = {"apply": 1, "cauchy": 1, "solve": 10, "rk2": 44, "batch": 44, "vjp": 110}[kind]
    return {"bytes": n * {"apply": 88, "cauchy": 48, "solve": 88, "rk2": 32, "batch": 32, "vjp": 48}[kind],
            "flops": float(n * per * sums)}


# ---- the same in plain torch, 64 bits, direct sums over all pairs ----------------------
def _pairs(nt, ns):
    """Slices of the targets that keep a block of pairs within a gigabyte."""
    step = max(1, (1 << 26) // max(1, ns))
    return [slice(i, min(nt, i + step)) for i in range(0, nt, step)]


def _inv(d):
    """1 / d, with 0 for the pair of a point and itself."""
    same = d == 0
    return torch.where(same, 0.0, 1.0 / torch.where(same, 1.0, d))


def _cauchy(zt, zs, q):
    """sum_j q_j / (zt - zs_j), a point itself left out."""
    return torch.cat([_inv(zt[s, None] - zs[None, :]) @ q for s in _pairs(len(zt), len(zs))])


def _stokes(z, dz, h, u, sign, wall=False):
    """The layer sum of CADAPDR (sign -1) and CADAPMOD (sign +1); the images across y = 0."""
    qa, qb = u * dz * h / (2j * PI), (u * dz.conj() - u.conj() * dz) * h / (2j * PI)
    out = []
    for s in _pairs(len(z), len(z)):
        r = -_inv(z[s, None] - z[None, :])  # 1 / (z_j - z_t)
        d = z[None, :] - z[s, None]
        g = r @ qa + sign * ((r @ qb).conj() - (d * (r * r).conj()) @ qa.conj())
        if wall:
            g1, g2, d1 = qa.conj() - qb.conj(), 2j * z.imag * qa.conj(), -qb.conj()
            t = 1.0 / (z.conj()[None, :] - z[s, None])
            t2 = t * t
            far = (d * (g1 * t2 + 2.0 * g2 * t2 * t).conj()).sum(1)
            g = g + t @ g1 + t2 @ g2 + sign * (2.0 * (t2 @ g2).conj() + (t @ d1).conj() - far)
        out.append(g)
    return torch.cat(out)


class _Geo:
    """The arrays of one geometry on the GPU, and the two operators on it."""

    def __init__(self, nd, z, dz, ds, ka, zk, wall=False):
        dev = z.device
        self.nd, self.z, self.dz, self.ds, self.ka, self.zk, self.wall = [int(n) for n in nd], z, dz, ds, ka, zk, wall
        n = torch.tensor(self.nd, device=dev)
        self.of = torch.repeat_interleave(torch.arange(len(self.nd), device=dev), n)
        self.h = (2 * PI / n.double())[self.of]

    def _per_drop(self, v):
        return torch.zeros(len(self.nd), dtype=v.dtype, device=v.device).index_add(0, self.of, v)

    def laplace(self, u):
        cf = _cauchy(self.z, self.z, u * self.dz * self.h)
        return u + self.h * self.ka * self.ds * u / (2 * PI) - cf.imag / PI - 2 * self.h * self.ds * u

    def stokes(self, u):
        z, dz, h = self.z, self.dz, self.h
        za = self._per_drop(h * u)[self.of]
        pk = self._per_drop(2 * h / PI * (u * dz / (z - self.zk[self.of]) ** 2).real)[self.of]
        own = h * self.ka / (2 * PI) * (self.ds * u + u.conj() * dz ** 2 / self.ds)
        return u + za + 0.5j * pk * z + own + _stokes(z, dz, h, u, -1.0, self.wall)


def _solve(op, b, cplx):
    """op(x) = b by GMRES with full reorthogonalisation, to rounding."""
    pack = (lambda v: torch.view_as_real(v).reshape(-1)) if cplx else (lambda v: v)
    unpack = (lambda v: torch.view_as_complex(v.reshape(-1, 2))) if cplx else (lambda v: v)
    x, scale = torch.zeros_like(pack(b)), pack(b).norm()
    for _ in range(2):
        r = pack(b - op(unpack(x)))
        beta = r.norm()
        if not beta > 1e-15 * scale:
            break
        V, H = [r / beta], np.zeros((161, 160))
        for j in range(min(160, len(r))):
            w = pack(op(unpack(V[j])))
            Q = torch.stack(V)
            c = Q @ w
            w = w - c @ Q
            c2 = Q @ w
            w = w - c2 @ Q
            H[:j + 1, j], H[j + 1, j] = (c + c2).cpu().numpy(), float(w.norm())
            e = np.zeros(j + 2)
            e[0] = float(beta)
            y, *_ = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) < 1e-14 * float(scale) or H[j + 1, j] < 1e-15:
                break
            V.append(w / H[j + 1, j])
        x = x + torch.as_tensor(y, device=x.device) @ torch.stack(V)[:len(y)]
    return unpack(x)


def _wave(n, dev):
    w = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev)
    w[n // 2] = 0.0
    return w


def _by_size(nd):
    """The drops of each size: the size and the (drops, size) table of their nodes."""
    e = _ends(nd)
    return [(n, np.stack([np.arange(*e[i]) for i in range(len(nd)) if nd[i] == n])) for n in sorted(set(int(m) for m in nd))]


def _each(nd, f, *vs):
    """f on the drops of each size at once, rows of samples in, rows of samples out."""
    got, order = [], []
    for n, at in _by_size(nd):
        i = torch.as_tensor(at, device=vs[0].device)
        r = f(n, *(v[i] for v in vs))
        got.append(r.reshape(-1))
        order.append(i.reshape(-1))
    return torch.cat(got)[torch.argsort(torch.cat(order))]


def _diff(n, f):
    return torch.fft.ifft(torch.fft.fft(f) * 1j * _wave(n, f.device))


def _anti(n, f):
    w = _wave(n, f.device)
    return torch.fft.ifft(torch.where(w == 0, 0, torch.fft.fft(f) / torch.where(w == 0, 1, 1j * w)))


def _fine(n, f, real):
    """Samples at twice the nodes: FINTERC, or FINTER for a real sample (which drops the
    imaginary part of mode n/2 - 1 and the real part of mode n/2)."""
    c = torch.fft.fft(f.to(torch.complex128))
    h = n // 2
    if real:
        c = torch.cat([c[:, :h - 1], c[:, h - 1:h].real.to(c.dtype), 1j * c[:, h:h + 1].imag, c[:, h + 1:]], 1)
    else:
        c = torch.cat([c[:, :h], 0 * c[:, h:h + 1], c[:, h + 1:]], 1)
    w = torch.cat([c[:, :h + 1], torch.zeros_like(c), c[:, h + 1:]], 1)
    r = torch.fft.ifft(w) * 2
    return r.real if real else r


def _filter(n, f):
    i = np.minimum(np.arange(n), n - np.arange(n))
    sig = torch.as_tensor(np.exp(-10.0 * (i.astype(np.float32) / np.float32(n // 2)).astype(np.float64) ** 25), device=f.device)
    c = torch.fft.fft(f) / n * sig
    c = torch.cat([c[:, :n // 2], 0 * c[:, n // 2:n // 2 + 1], c[:, n // 2 + 1:]], 1)
    re, im = (p + (torch.where(p.abs() < 1e-13, torch.zeros_like(p), p) - p).detach() for p in (c.real, c.imag))
    return torch.fft.ifft(torch.complex(re, im)) * n


def _f(nd, z, e0, cap, solve):
    """F: the velocity of the nodes z (complex), with e0 per drop (its own, or one for all)."""
    z1 = _each(nd, _diff, z)
    z2 = _each(nd, _diff, z1)
    ds = z1.abs()
    m = (z1.conj() * z2).imag
    geo = _Geo(nd, z, -z1, ds, -m / ds ** 3, torch.stack([z[a:b].mean() for a, b in _ends(nd)]))
    dz, h = geo.dz, geo.h
    ul = solve(geo, "laplace", -2.0 * z.real)
    uc = ul * dz
    odd, even = (lambda f, r: lambda n, v: _fine(n, v, r)[:, 1::2]), (lambda n, v: _fine(n, v, True)[:, 0::2])
    src = torch.complex(_each(nd, odd(_fine, True), z.real), _each(nd, odd(_fine, True), z.imag))
    tgt = torch.complex(_each(nd, even, z.real), _each(nd, even, z.imag))
    q = _each(nd, odd(_fine, False), uc) * h
    psi = -_cauchy(tgt, src, q).real / (2 * PI) - z.imag
    dphi = -_each(nd, _diff, psi.to(torch.complex128)).real / ds
    g = dz * dphi ** 2
    late = 2 * PI * (nd[-1] - 1) / nd[-1]  # SETVELF's alpha, left over from the last drop
    rhs = -0.5 * dz / ds + 0.5j * cap * z.conj()
    rhs = rhs + 0.25j * e0 * _each(nd, lambda n, v: late * v.mean(1, keepdim=True) + _anti(n, v) - _anti(n, v)[:, :1], g)
    u = solve(geo, "stokes", rhs)
    gw = _stokes(z, dz, h, u, 1.0) - u.conj() * h * geo.ka * dz ** 2 / (2 * PI * ds)
    gw = gw + (h * (-z2 / z1).real * u - 2 * h * _each(nd, _diff, u)) / (2j * PI) + 0.5j * cap * z.conj()
    un = (gw * dz.conj()).real / ds
    tt = -_each(nd, _anti, (-m / ds ** 2 * un).to(torch.complex128)).real
    return _each(nd, _filter, -(un * 1j * dz + tt * dz) / ds)


def _by_gmres(geo, op, b):
    return _solve(getattr(geo, op), b, op == "stokes")


def _matrices(geo, op):
    """The operators as dense real matrices (for autograd)."""
    z, dz, h, n = geo.z, geo.dz, geo.h, len(geo.z)
    eye = torch.eye(n, dtype=torch.bool, device=z.device)
    d = torch.where(eye, 1.0, z[None, :] - z[:, None])  # z_j - z_t
    r = torch.where(eye, 0.0, 1.0 / d)
    if op == "laplace":
        return (r * (dz * h)[None, :]).imag / PI + torch.diag(1 + h * geo.ka * geo.ds / (2 * PI) - 2 * h * geo.ds)
    c = (h / (2j * PI))[None, :] * dz[None, :]
    same = geo.of[:, None] == geo.of[None, :]
    e = 0.5j * z[:, None] * h[None, :] / PI * (dz / (z - geo.zk[geo.of]) ** 2)[None, :]
    f = 0.5j * z[:, None] * h[None, :] / PI * (dz / (z - geo.zk[geo.of]) ** 2).conj()[None, :]
    own = h * geo.ka / (2 * PI)
    P = c * r + c.conj() * r.conj() + torch.where(same, h[None, :] + e, 0.0) + torch.diag(1 + own * geo.ds + 0j)
    k = (h / (2j * PI)).conj()[None, :]
    Q = -k * dz[None, :] * r.conj() + k * dz.conj()[None, :] * torch.where(eye, 0.0, d) * r.conj() ** 2
    Q = Q + torch.where(same, f, 0.0) + torch.diag(own * dz ** 2 / geo.ds)
    A, B = P + Q, P - Q
    return torch.stack([torch.stack([A.real, -B.imag], -1), torch.stack([A.imag, B.real], -1)], 1).reshape(2 * n, 2 * n)


def _by_dense(geo, op, b):
    if op == "laplace":
        return torch.linalg.solve(_matrices(geo, op), b)
    return torch.view_as_complex(torch.linalg.solve(_matrices(geo, op), torch.view_as_real(b).reshape(-1)).reshape(-1, 2))


def _heun(nd, y, e0, cap, solve=_by_gmres):
    z = torch.view_as_complex(y.reshape(-1, 2))
    k1 = _f(nd, z, e0, cap, solve)
    k2 = _f(nd, z + DT * k1, e0, cap, solve)
    return torch.view_as_real(z + 0.5 * DT * (k1 + k2)).reshape(-1)


def exact(case, seed):
    n, kind = _size(case), case["kind"]
    if n > {"apply": 200000, "cauchy": 250000, "solve": 34000, "rk2": 34000, "batch": 100000, "vjp": 4200}[kind]:
        return None  # minutes of direct sums
    d = _inputs(case, seed)
    t = {k: torch.from_numpy(v).cuda() for k, v in d.items() if isinstance(v, np.ndarray) and k != "nd"}
    if kind == "cauchy":
        return _cauchy(t["z"], t["z"], t["q"])
    if kind == "rk2":
        return _heun(d["nd"], t["y"], d["e0"], d["cap"])
    if kind == "batch":
        return torch.cat([_heun(d["nd"][i:i + 1], t["y"][2 * a:2 * b], float(d["e0"][i]), d["cap"])
                          for i, (a, b) in enumerate(_ends(d["nd"]))])
    if kind == "vjp":
        y = t["y"].requires_grad_()
        p = torch.tensor([d["e0"], d["cap"]], dtype=torch.float64, device="cuda", requires_grad=True)
        gy, gp = torch.autograd.grad(_heun(d["nd"], y, p[0], p[1], _by_dense), (y, p), t["v"])
        return {"y": gy, "e0": float(gp[0]), "cap": float(gp[1])}
    geo = _Geo(d["nd"], t["z"], t["dz"], t["dsda"], t["kappa"], t["zk"], bool(case.get("wall")))
    if case["op"] == "laplace":
        return geo.laplace(t["x"]) if kind == "apply" else _solve(geo.laplace, t["x"], False)
    x = torch.view_as_complex(t["x"].reshape(-1, 2))
    r = geo.stokes(x) if kind == "apply" else _solve(geo.stokes, x, True)
    return torch.view_as_real(r).reshape(-1)
