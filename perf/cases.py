"""The work a user of the library has it do, as cases that can be timed and checked.

Each case is one pass through the package's public entry points: heatbath chains of one lattice
(GaugeField), many chains at once (Batch), Wilson flows with and without measurements (GradientFlow),
the observables of a configuration, and flow measurements from the server (Server).  The sizes are
those of the repository's own configurations (8^4 to 48^4, the mixed batch, the serving mix) with
ragged lattices beside them; FP64 links carry the chains, FP64 and FP32 links the flows.

Configurations are rough SU(3) fields made from the seed: links scattered about the identity so
that the plaquette is near the 0.6 of beta = 6, in a random gauge.

exact() restates the arithmetic in plain torch, in complex128: staples, the Cabibbo-Marinari
heatbath with Kennedy-Pendleton steps on the Philox link streams, the RK3 flow and the clover
observables.
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package; its folder's name is not a Python identifier, so it is loaded by path."""
    if "ecmc_qcb_b200" not in sys.modules:
        d = os.path.join(_ROOT, "ecmc-qcb_b200")
        spec = importlib.util.spec_from_file_location("ecmc_qcb_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["ecmc_qcb_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["ecmc_qcb_b200"]


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # plaquette, Q and E of a small configuration: the smallest calls, launches and latency
        _observables("obs-8", (8, 8, 8, 8), 18),
        # plaquette, Q and E of a full-size configuration, as a run measures each saved one
        _observables("obs-32", (32, 32, 32, 32), 18),
        # the small run: a short stretch of an 8^4 chain, then its plaquette
        _heatbath("hb-8", (8, 8, 8, 8), 18, sweeps=10, n_hits=2, shift=False, clover=False),
        # a run's schedule on a ragged lattice in the compressed storage: a random global shift,
        # sweeps, plaquette and topology
        _heatbath("hb-ragged-12real", (20, 14, 18, 26), 12, sweeps=5, n_hits=2, shift=True, clover=True),
        # the flagship chain: 32^4, N_hits = 2
        _heatbath("hb-32", (32, 32, 32, 32), 18, sweeps=4, n_hits=2, shift=False, clover=False),
        # many chains at once (an eighth of the 256-chain mix), N_hits = 1, compressed storage
        {"name": "batch", "kind": "batch", "n8": 12, "n12": 12, "n16": 6, "n24": 2, "reals": 12, "sweeps": 5,
         "n_hits": 1},
        # a measured FP64 flow of a mid-size configuration
        _flow("flow-16-f64", (16, 16, 16, 16), 64, 18, n_steps=11, n_rk=1, measured=True),
        # the measured FP64 flow of a full-size configuration
        _flow("flow-32-f64", (32, 32, 32, 32), 64, 18, n_steps=5, n_rk=1, measured=True),
        # the same in FP32 links
        _flow("flow-32-f32", (32, 32, 32, 32), 32, 18, n_steps=9, n_rk=1, measured=True),
        # smoothing only, on a ragged lattice in compressed FP32 links, then one measurement
        _flow("flow-ragged-f32-12real", (24, 20, 28, 22), 32, 12, n_steps=1, n_rk=20, measured=False),
        # the largest: a 48^4 configuration's measured flow in compressed FP32 links
        _flow("flow-48-f32-12real", (48, 48, 48, 48), 32, 12, n_steps=4, n_rk=1, measured=True),
        # the server: requests of several sizes at once, the largest on its own kernels
        {"name": "serve", "kind": "serve", "n8": 3, "n12": 2, "n16": 2, "n24": 1, "reals": 18, "flow_time": 1.0},
    ]


def _observables(name, L, reals):
    return {"name": name, "kind": "observables", **_ext(L), "reals": reals}


def _heatbath(name, L, reals, sweeps, n_hits, shift, clover):
    return {"name": name, "kind": "heatbath", **_ext(L), "reals": reals, "sweeps": sweeps, "n_hits": n_hits,
            "beta": 6.0, "shift": shift, "clover": clover}


def _flow(name, L, prec, reals, n_steps, n_rk, measured):
    return {"name": name, "kind": "flow", **_ext(L), "prec": prec, "reals": reals, "n_steps": n_steps, "n_rk": n_rk,
            "measured": measured}


def _ext(L):
    return {"Lx": L[0], "Ly": L[1], "Lz": L[2], "Lt": L[3]}


def _draw_lattice(rng, most):
    """Even extents, each spread over 4..48 on a log scale, at most `most` sites."""
    while True:
        L = [2 * round(math.exp(rng.uniform(math.log(2), math.log(24)))) for _ in range(4)]
        if 256 <= L[0] * L[1] * L[2] * L[3] <= most:
            return L


def draw(rng: random.Random):
    kind = rng.choice(["observables", "heatbath", "heatbath", "batch", "flow", "flow", "flow", "serve"])
    if kind == "observables":
        c = _observables("", _draw_lattice(rng, 32**4), rng.choice([18, 18, 12]))
    elif kind == "heatbath":
        L = _draw_lattice(rng, 32**4)
        most = max(1, min(12, 4 * 32**4 // math.prod(L)))
        c = _heatbath("", L, rng.choice([18, 18, 12]), sweeps=rng.randint(1, most), n_hits=rng.choice([1, 2, 2, 3]),
                      shift=rng.random() < 0.5, clover=rng.random() < 0.5)
        c["beta"] = round(rng.uniform(5.7, 6.3), 3)
    elif kind == "batch":
        c = {"kind": "batch", "n8": rng.randint(0, 16), "n12": rng.randint(0, 12), "n16": rng.randint(0, 6),
             "n24": rng.randint(0, 2), "reals": rng.choice([18, 12]), "sweeps": rng.randint(2, 5),
             "n_hits": rng.choice([1, 1, 2])}
        c["n8"] += c["n12"] + c["n16"] + c["n24"] == 0
    elif kind == "flow":
        L = _draw_lattice(rng, 32**4)
        prec = rng.choice([64, 32, 32])
        steps = rng.randint(2, max(2, min(24, (5 if prec == 64 else 9) * 32**4 // math.prod(L))))
        n_rk = rng.choice([1, 1, 2, 5])
        measured = rng.random() < 0.7
        c = _flow("", L, prec, rng.choice([18, 12]), n_steps=max(2, 1 + (steps - 1) // n_rk) if measured else 1,
                  n_rk=n_rk if measured else steps, measured=measured)
    else:
        c = {"kind": "serve", "n8": rng.randint(0, 5), "n12": rng.randint(1, 4), "n16": rng.randint(0, 2),
             "n24": rng.randint(0, 1), "reals": rng.choice([18, 12]), "flow_time": round(rng.uniform(0.2, 1.0), 2)}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- configurations
EPS = 0.02      # flow step
SPREAD = 0.21   # scatter of the links about the identity: plaquette near 0.6
SEED_HB = 1234567


def _lattice(case):
    return case["Lx"], case["Ly"], case["Lz"], case["Lt"]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _unitary(m):
    """SU(3) matrices from the first two columns of m: Gram-Schmidt, third column by cross product."""
    a = m[..., 0] / m[..., 0].abs().square().sum(-1, keepdim=True).sqrt()
    b = m[..., 1] - a * (a.conj() * m[..., 1]).sum(-1, keepdim=True)
    b = b / b.abs().square().sum(-1, keepdim=True).sqrt()
    c = torch.stack([a[..., (i + 1) % 3] * b[..., (i + 2) % 3] - a[..., (i + 2) % 3] * b[..., (i + 1) % 3]
                     for i in range(3)], -1).conj()
    return torch.stack([a, b, c], -1)


def _configuration(L, seed):
    """Links (Lt, Lz, Ly, Lx, 4, 3, 3): V x 4 x 3 x 3 with x fastest, the library's order."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    shape = (L[3], L[2], L[1], L[0])

    def gauss(*s):
        return torch.complex(torch.randn(*s, dtype=torch.float64, device=dev, generator=gen),
                             torch.randn(*s, dtype=torch.float64, device=dev, generator=gen))

    g = _unitary(gauss(*shape, 3, 3))
    U = torch.empty(*shape, 4, 3, 3, dtype=torch.complex128, device=dev)
    one = torch.eye(3, dtype=torch.complex128, device=dev)
    for mu in range(4):
        U[..., mu, :, :] = _mul(_mul(g, _unitary(one + SPREAD * gauss(*shape, 3, 3))), _dag(_at(g, mu, 1)))
    return U


def _store(case):
    q = _package()
    return q.STORE_12 if case["reals"] == 12 else q.STORE_18


def _field(L, prec, store, U):
    f = _package().GaugeField(L, prec, store)
    torch.cuda.synchronize()
    f.upload_device_ptr(U.data_ptr())
    f.sync()
    return f


def _mix(case):
    """Lattice sizes of a batch or of a set of requests."""
    return [n for n in (8, 12, 16, 24) for _ in range(case["n%d" % n])]


def _requests(case):
    """(size, measurements) of each request: t = L^2/32, at most flow_time."""
    return [(n, int(round(min(n * n / 32, case["flow_time"]) / EPS)) + 1) for n in _mix(case)]


def _betas(n):
    return [round(5.7 + 0.6 * ((i * 7) % 13) / 13, 4) for i in range(n)]


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    q = _package()
    kind = case["kind"]
    s = {"case": case, "sweep": 0}
    if kind in ("observables", "heatbath", "flow"):
        L = _lattice(case)
        U = _configuration(L, seed)
        s["field"] = _field(L, q.PREC_F64, _store(case) if kind != "flow" else q.STORE_18, U)
        if kind != "observables":
            s["links"] = torch.empty_like(U).view(-1, 4, 3, 3)
        if kind == "flow":
            s["flow"] = q.GradientFlow(s["field"], EPS, prec=case["prec"], store=_store(case))
    elif kind == "batch":
        Ls = _mix(case)
        # launch shape 0: what the tuner picks for such mixes
        s["batch"] = b = q.Batch([(n,) * 4 for n in Ls], _betas(len(Ls)), [seed * 1000 + i for i in range(len(Ls))],
                                 q.PREC_F64, _store(case))
        b.set_variant(0)
        for i, n in enumerate(Ls):
            b.upload(i, _configuration((n,) * 4, seed * 1000 + i).cpu().numpy())
    else:
        s["inputs"] = [_configuration((n,) * 4, seed * 1000 + i).cpu().numpy()
                       for i, (n, _) in enumerate(_requests(case))]
        s["server"] = q.Server(40 << 30, prec=q.PREC_F32, store=_store(case))
    return s


def _export(s, field):
    """The links in the library's exchange order, in the program's own buffer."""
    field.download_device_ptr(s["links"].data_ptr())
    field.sync()
    return s["links"]


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "observables":
        return {"plaquette": s["field"].plaquette(), "QE": np.array(s["field"].clover_qe())}
    if kind == "heatbath":
        f = s["field"]
        if case["shift"]:
            f.random_shift(SEED_HB, s["sweep"])
        for _ in range(case["sweeps"]):
            f.hb_sweep(case["beta"], case["n_hits"], SEED_HB, s["sweep"])
            s["sweep"] += 1
        out = {"plaquette": f.plaquette()}
        if case["clover"]:
            out["QE"] = np.array(f.clover_qe())
        out["links"] = _export(s, f)
        return out
    if kind == "batch":
        b = s["batch"]
        b.sweep(case["n_hits"], case["sweeps"])
        return {"plaquettes": b.plaquette(), "links": b.download(0)}
    if kind == "flow":
        fl = s["flow"]
        if case["measured"]:
            tqe, p = fl.measure(s["field"], case["n_steps"], case["n_rk"], plaquette=True)
            out = {"tQE": tqe, "plaquettes": p}
        else:
            fl.copy(s["field"])
            fl.rk3_step(case["n_rk"])
            out = {"QE": np.array(fl.field.clover_qe()), "plaquettes": np.array([fl.field.plaquette()])}
        out["links"] = _export(s, fl.field)
        return _kept(out, case["prec"])
    for i, (n, steps) in enumerate(_requests(case)):
        s["server"].submit(i, (n,) * 4, s["inputs"][i], EPS, steps)
    s["server"].wait(60.0)
    out = {}
    while (r := s["server"].poll()) is not None:
        out["request %d" % r[0]] = r[1]
    return _kept(out, 32)


def _kept(out, prec):
    """What a program keeps of a flow in FP32 links: numbers of that precision."""
    if prec == 64:
        return out
    return {k: v.astype(np.float32) if isinstance(v, np.ndarray) else v.to(torch.complex64) for k, v in out.items()}


# ---------------------------------------------------------------- work
def _flow_flops(sites, stages):
    # per link and stage: 6 staples of 42 complex multiply-adds, the force's 23, the exponential's
    # square and sums (18 + 18), its coefficients and the update (27)
    return sites * stages * 4 * (8 * (6 * 42 + 23 + 36 + 27) + 200)


_CLOVER_FLOPS = 6 * (4 * 60 * 8 + 100)  # a site: six planes, four leaves of 60 complex multiply-adds


def work(case):
    kind = case["kind"]
    link = {18: 144, 12: 96}[case["reals"]] // (2 if case.get("prec", 64) == 32 or kind == "serve" else 1)
    if kind == "observables":
        V = math.prod(_lattice(case))
        return {"bytes": 4 * V * link, "flops": V * (_CLOVER_FLOPS + 6 * 27 * 16)}
    if kind in ("heatbath", "batch"):
        V = math.prod(_lattice(case)) if kind == "heatbath" else sum(n**4 for n in _mix(case))
        # a link update: the staple, then 3 subgroups a hit of 24 complex multiply-adds, three
        # Philox calls and the Kennedy-Pendleton step
        per = 8 * 6 * 42 + case["n_hits"] * 3 * (8 * 24 + 100)
        obs = V * 6 * 27 * 16 + (V * _CLOVER_FLOPS if case.get("clover") else 0)
        out = 4 * V * 144 if kind == "heatbath" else 4 * _mix(case)[0] ** 4 * 144
        return {"bytes": 2 * 4 * V * link * case["sweeps"] + 4 * V * link + out,
                "flops": 4 * V * case["sweeps"] * per + obs}
    if kind == "flow":
        V = math.prod(_lattice(case))
        steps = case["n_rk"] * (case["n_steps"] - 1 if case["measured"] else 1)
        alg = 32 if case["prec"] == 32 else 64
        moved = 4 * V * 144 + steps * 4 * V * (6 * link + 4 * alg) + 4 * V * 144 + case["n_steps"] * 4 * V * link
        return {"bytes": moved, "flops": _flow_flops(V, 3 * steps) + case["n_steps"] * V * _CLOVER_FLOPS}
    sites = sum(n**4 * (steps - 1) for n, steps in _requests(case))
    meas = sum(n**4 * steps for n, steps in _requests(case))
    first = sum(n**4 for n, _ in _requests(case))
    return {"bytes": 4 * first * 144 + sites * 4 * (6 * link + 4 * 32) + meas * 4 * link,
            "flops": _flow_flops(sites, 3) + meas * _CLOVER_FLOPS}


# ---------------------------------------------------------------- the same in plain torch
def _mul(a, b):
    return a[..., :, 0:1] * b[..., 0:1, :] + a[..., :, 1:2] * b[..., 1:2, :] + a[..., :, 2:3] * b[..., 2:3, :]


def _dag(a):
    return a.conj().transpose(-1, -2)


def _at(a, mu, step):
    """The field a at x + step * mu (site dimensions t, z, y, x come first)."""
    return torch.roll(a, -step, 3 - mu)


def _staple(u, mu):
    """compute_staple: sum over nu of U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+ and its mirror."""
    total = torch.zeros_like(u[0])
    for nu in range(4):
        if nu != mu:
            total += _mul(_mul(_at(u[nu], mu, 1), _dag(_at(u[mu], nu, 1))), _dag(u[nu]))
            total += _at(_mul(_dag(_mul(u[mu], _at(u[nu], mu, 1))), u[nu]), nu, -1)
    return total


def _trace(a):
    return a[..., 0, 0] + a[..., 1, 1] + a[..., 2, 2]


def _observe(u):
    """Plaquette, Q and E of the configuration."""
    V = u[0][..., 0, 0].numel()
    plaq, F = 0.0, {}
    for mu in range(4):
        for nu in range(mu + 1, 4):
            corner, other = _mul(u[mu], _at(u[nu], mu, 1)), _mul(u[nu], _at(u[mu], nu, 1))
            leaf = _mul(corner, _dag(other))
            plaq += _trace(leaf).real.sum().item() / 3
            c = leaf + _at(_mul(_dag(u[mu]), _mul(leaf, u[mu])), mu, -1)  # leaf 2: the plaquette of x - mu
            down = _mul(_mul(_dag(u[nu]), leaf), u[nu])                  # leaf 4: that of x - nu
            c += _at(down, nu, -1)
            um = _at(u[mu], nu, 1)                                       # leaf 3: that of x - mu - nu
            c += _at(_at(_mul(_mul(_dag(um), down), um), nu, -1), mu, -1)
            F[mu, nu] = (c - _dag(c)) / 8
    q = (_trace(_mul(F[0, 1], F[2, 3])) - _trace(_mul(F[0, 2], F[1, 3])) + _trace(_mul(F[0, 3], F[1, 2]))).real
    e = sum(0.5 * f.abs().square().sum().item() for f in F.values())
    return plaq / (6 * V), q.sum().item() / (4 * math.pi**2), e / V


def _force(u, mu):
    """proj_lie(-U A)"""
    m = -_mul(u[mu], _staple(u, mu))
    m = (m - _dag(m)) / 2
    return m - (_trace(m) / 3)[..., None, None] * torch.eye(3, dtype=m.dtype, device=m.device)


def _exp(x):
    """exp of small matrices: the Taylor sum on x / 4 to 18 terms, squared twice."""
    one = torch.eye(3, dtype=x.dtype, device=x.device)
    x = x / 4
    e = one + x / 18
    for n in range(17, 0, -1):
        e = one + _mul(x, e) / n
    e = _mul(e, e)
    return _mul(e, e)


def _rk3(u, eps):
    z = [_force(u, mu) for mu in range(4)]
    u = [_mul(_exp(eps / 4 * z[mu]), u[mu]) for mu in range(4)]
    z = [8 / 9 * _force(u, mu) - 17 / 36 * z[mu] for mu in range(4)]
    u = [_mul(_exp(eps * z[mu]), u[mu]) for mu in range(4)]
    z = [3 / 4 * _force(u, mu) - z[mu] for mu in range(4)]
    return [_mul(_exp(eps * z[mu]), u[mu]) for mu in range(4)]


def _measure(u, n_steps, n_rk):
    """(t, Q, E) rows and plaquettes of a measured flow, and its last configuration."""
    rows, plaq, t = [], [], 0.0
    for k in range(n_steps):
        p, q, e = _observe(u)
        rows.append((t, q, e))
        plaq.append(p)
        if k + 1 < n_steps:
            for _ in range(n_rk):
                u = _rk3(u, EPS)
                t += EPS
    return np.array(rows), np.array(plaq), u


_M32 = 0xFFFFFFFF


def _philox(c, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors or integers holding 32-bit words."""
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & _M32) ^ c[1] ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c[3] ^ k1, p0 & _M32]
    return c


class _Draws:
    """The uniforms of each link's stream for one sweep: call n gives draws 2n and 2n + 1."""

    def __init__(self, link, seed, sweep):
        self.link, self.seed, self.sweep = link, seed, sweep

    def call(self, n, sel=slice(None)):
        link = self.link[sel]
        c = _philox([n, link, torch.full_like(link, self.sweep), torch.full_like(link, 0x48420001)],
                    self.seed & _M32, (self.seed >> 32) & _M32)
        return [((hi << 21) | (lo >> 11)).double() * 2.0**-53 for hi, lo in ((c[0], c[1]), (c[2], c[3]))]


def _su2_step(w, beta, draws, n):
    """Kennedy-Pendleton quaternions for w, and the next call of each stream."""
    k = w.square().sum(-1).sqrt()
    v = w / k[:, None]
    scale = -0.75 / (beta * k)
    a0 = torch.zeros_like(k)
    left = torch.arange(k.numel(), device=k.device)
    n = n.clone()
    while left.numel():
        d, r1 = draws.call(n[left], left)
        r2, r3 = draws.call(n[left] + 1, left)
        c = torch.cos(2 * math.pi * r2)
        x = scale[left] * (torch.log(r1) + c * c * torch.log(r3))
        ok = d * d <= 1 - x
        a0[left[ok]] = 1 - 2 * x[ok]
        n[left] += 2
        left = left[~ok]
    phi, ct = draws.call(n)
    rs = (1 - a0 * a0).sqrt()
    ct = 2 * ct - 1
    st = (1 - ct * ct).sqrt()
    x = [a0, rs * st * torch.cos(2 * math.pi * phi), rs * st * torch.sin(2 * math.pi * phi), rs * ct]
    v0, v1, v2, v3 = v.unbind(-1)
    r = (x[0] * v0 + x[1] * v1 + x[2] * v2 + x[3] * v3, -x[0] * v1 + x[1] * v0 - x[2] * v3 + x[3] * v2,
         -x[0] * v2 + x[1] * v3 + x[2] * v0 - x[3] * v1, -x[0] * v3 - x[1] * v2 + x[2] * v1 + x[3] * v0)
    return r, n + 1


def _sweep(u, L, beta, n_hits, seed, sweep):
    """One checkerboard sweep of u, a list of four contiguous (Lt, Lz, Ly, Lx, 3, 3) fields, in place."""
    V = math.prod(L)
    lex = torch.arange(V, device=u[0].device)
    odd = (lex % L[0] + lex // L[0] % L[1] + lex // (L[0] * L[1]) % L[2] + lex // (L[0] * L[1] * L[2])) % 2
    for par in (0, 1):
        at = lex[odd == par]
        for mu in range(4):
            A = _staple(u, mu).view(V, 3, 3)[at]
            m = u[mu].view(V, 3, 3)[at]
            draws = _Draws((at * 4 + mu) & _M32, seed, sweep)
            n = torch.zeros_like(at)
            for hit in range(3 * n_hits):
                i, j = ((0, 1), (1, 2), (0, 2))[hit % 3]
                W = _mul(m, A)
                w = torch.stack([(W[:, i, i].real + W[:, j, j].real) / 2, (W[:, i, j].imag + W[:, j, i].imag) / 2,
                                 (W[:, i, j].real - W[:, j, i].real) / 2, (W[:, i, i].imag - W[:, j, j].imag) / 2], -1)
                (r0, r1, r2, r3), n = _su2_step(w, beta, draws, n)
                mi, mj = m[:, i].clone(), m[:, j].clone()
                m[:, i] = torch.complex(r0, r3)[:, None] * mi + torch.complex(r2, r1)[:, None] * mj
                m[:, j] = torch.complex(-r2, r1)[:, None] * mi + torch.complex(r0, -r3)[:, None] * mj
            u[mu].view(V, 3, 3)[at] = m


def _random_shift(L, seed, idx):
    c = _philox([0, idx & _M32, (idx >> 32) & _M32, 0x53480001], seed & _M32, (seed >> 32) & _M32)
    return [(c[d] * L[d]) >> 32 for d in range(4)]


def _links(u):
    return torch.stack(u, -3).reshape(-1, 4, 3, 3)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("observables", "heatbath", "flow"):
        L = _lattice(case)
        u = [m.contiguous() for m in _configuration(L, seed).unbind(-3)]
    if kind == "observables":
        p, q, e = _observe(u)
        return {"plaquette": p, "QE": np.array([q, e])}
    if kind == "heatbath":
        if case["shift"]:
            sh = _random_shift(L, SEED_HB, 0)
            u = [torch.roll(m, sh[::-1], (0, 1, 2, 3)) for m in u]
        for k in range(case["sweeps"]):
            _sweep(u, L, case["beta"], case["n_hits"], SEED_HB, k)
        p, q, e = _observe(u)
        out = {"plaquette": p, "links": _links(u)}
        if case["clover"]:
            out["QE"] = np.array([q, e])
        return out
    if kind == "flow":
        if case["measured"]:
            rows, plaq, u = _measure(u, case["n_steps"], case["n_rk"])
            return {"tQE": rows, "plaquettes": plaq, "links": _links(u)}
        for _ in range(case["n_rk"]):
            u = _rk3(u, EPS)
        p, q, e = _observe(u)
        return {"QE": np.array([q, e]), "plaquettes": np.array([p]), "links": _links(u)}
    if kind == "batch":
        Ls = _mix(case)
        plaq, first = [], None
        for i, (n, beta) in enumerate(zip(Ls, _betas(len(Ls)))):
            u = [m.contiguous() for m in _configuration((n,) * 4, seed * 1000 + i).unbind(-3)]
            for k in range(case["sweeps"]):
                _sweep(u, (n,) * 4, beta, case["n_hits"], seed * 1000 + i, k)
            plaq.append(_observe(u)[0])
            first = _links(u) if i == 0 else first
        return {"plaquettes": np.array(plaq), "links": first}
    return {"request %d" % i: _measure([m.contiguous() for m in _configuration((n,) * 4, seed * 1000 + i).unbind(-3)],
                                       steps, 1)[0]
            for i, (n, steps) in enumerate(_requests(case))}
