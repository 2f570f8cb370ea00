"""The work that users of this framework have it do, as measurable cases.

Every case is a call through a public entry point on inputs of a size and kind that the
configurations, tests and the benchmark of this repository use (uniform electron gas of 7-57
plane waves, Hubbard rings of 6-16 sites, general blocks with nv != no):

  step      one amplitude iteration of a resident solver (``DeviceSolver.step``): the damped
            update or Anderson mixing, a few digit levels or an FP64-accurate count, Kelvin's
            Simpson grid or Gauss-Legendre points
  update    the drop-in ``ccsd_stanton`` on device arrays
  residual  the drop-in ``stanton_residual`` (the contract of cqcpy's ``_Stanton``), general blocks
  lambda    Lambda iterations of a resident solver (``DeviceSolver.lambda_solve``), the backward pass
  tbar      the tau integral ``int_tbar2``
  energy    ``ft_cc_energy``
  solve     a whole ``ccsd(...).run()`` from host arrays to host amplitudes

Inputs come from the seed alone; ``exact`` evaluates the same equations with torch in FP64.
"""
import math

import numpy as np
import torch

from kelvin_gb300 import _lib, ft_cc_energy, ft_cc_equations, quadrature, systems
from kelvin_gb300.cc_utils import DeviceSolver
from kelvin_gb300.ccsd import ccsd

F_BLOCKS = ("oo", "ov", "vo", "vv")
I_BLOCKS = ("vvvv", "vvvo", "vovv", "vvoo", "vovo", "oovv", "vooo", "ooov", "oooo")
PRECISION = {"fp64": _lib.PREC_FP64, "tc": _lib.PREC_FP64_TC, "mixed": _lib.PREC_MIXED}


def listed():
    return [
        # the smallest request of a served mix: an 8-site ring, a few digit levels, its iteration
        # replayed as a CUDA graph
        {"name": "ring8_step", "kind": "step", "system": "ring", "sites": 8, "U": 2.0, "beta": 1.0,
         "ng": 10, "quad": "lin", "precision": "mixed", "digits": 3, "accel": 0, "graph": True},
        # the intermediate level of the damped ladder on a ring with an odd half (13 sites)
        {"name": "ring13_step", "kind": "step", "system": "ring", "sites": 13, "U": 3.0, "beta": 1.0,
         "ng": 20, "quad": "lin", "precision": "tc", "digits": 5, "accel": 0, "graph": True},
        # the drop-in update at the default precision (FP64 FMAs), 19 plane waves
        {"name": "ueg38_update_fp64", "kind": "update", "system": "ueg", "N": 14, "rs": 4.0, "pw": 19,
         "theta": 0.5, "ng": 10, "quad": "lin", "precision": "fp64", "digits": 7},
        # a user's whole solve of the same system with the benchmarked scheme, host to host
        {"name": "ueg38_solve", "kind": "solve", "system": "ueg", "N": 14, "rs": 4.0, "pw": 19,
         "theta": 0.5, "ng": 10, "quad": "gl", "precision": "mixed", "digits": 3},
        # the backward pass behind E, S, N and the densities
        {"name": "ueg38_lambda", "kind": "lambda", "system": "ueg", "N": 14, "rs": 4.0, "pw": 19,
         "theta": 0.5, "ng": 10, "quad": "lin", "precision": "tc", "digits": 7, "iters": 2},
        # the drop-in update, FP64-accurate on the tensor cores, 27 plane waves
        {"name": "ueg54_update", "kind": "update", "system": "ueg", "N": 14, "rs": 2.0, "pw": 27,
         "theta": 0.5, "ng": 10, "quad": "lin", "precision": "tc", "digits": 7},
        # the benchmarked iteration on the differentiation configuration, 33 plane waves
        {"name": "ueg66_step", "kind": "step", "system": "ueg", "N": 14, "rs": 2.0, "pw": 33,
         "theta": 0.5, "ng": 16, "quad": "gl", "precision": "mixed", "digits": 3, "accel": 3,
         "graph": False},
        # the benchmarked system, 57 plane waves: a few-digit sweep and a refinement sweep
        {"name": "ueg114_step", "kind": "step", "system": "ueg", "N": 38, "rs": 1.0, "pw": 57,
         "theta": 0.25, "ng": 10, "quad": "gl", "precision": "mixed", "digits": 3, "accel": 3,
         "graph": False},
        {"name": "ueg114_refine", "kind": "step", "system": "ueg", "N": 38, "rs": 1.0, "pw": 57,
         "theta": 0.25, "ng": 10, "quad": "gl", "precision": "tc", "digits": 6, "accel": 3,
         "graph": False},
        # general blocks without spin structure, odd extents, one tau point
        {"name": "blocks37x21_residual", "kind": "residual", "nv": 37, "no": 21, "precision": "tc",
         "digits": 7},
        # the two memory passes a caller of the drop-in modules runs by themselves
        {"name": "tbar66", "kind": "tbar", "nv": 66, "no": 66, "ng": 16, "quad": "lin"},
        {"name": "energy66", "kind": "energy", "nv": 66, "no": 66, "ng": 16},
    ]


def draw(rng):
    """One more case of the listed ones' ranges."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "update", "residual", "lambda", "tbar", "energy"])
    if kind == "residual":
        return {"kind": kind, "nv": logint(9, 48), "no": logint(5, 30), "precision": "tc", "digits": 7}
    if kind in ("tbar", "energy"):
        c = {"kind": kind, "nv": logint(10, 66), "no": logint(10, 66), "ng": rng.randint(5, 20)}
        if kind == "tbar":
            c["quad"] = rng.choice(["lin", "lin", "ln", "gl"])
        return c
    c = {"kind": kind}
    if kind == "step" and rng.random() < 0.35:
        c.update(system="ring", sites=rng.randint(6, 16), U=round(rng.uniform(1.0, 4.0), 3),
                 beta=1.0)
    else:
        pw = logint(7, 42 if kind == "step" else 27 if kind == "update" else 21)
        c.update(system="ueg", N=14 if pw >= 19 else 2, rs=round(rng.uniform(1.0, 4.0), 3), pw=pw,
                 theta=round(rng.uniform(0.4, 1.0), 3))
    big = c.get("pw", 0) > 33
    c["ng"] = rng.randint(5, 8 if big else 16)
    c["quad"] = "lin"
    if kind == "step":
        c["precision"], c["digits"] = rng.choice([("mixed", 3), ("mixed", 3), ("tc", 5), ("tc", 6),
                                                  ("tc", 7)])
        c["accel"] = rng.choice([0, 3])
        c["graph"] = c["accel"] == 0 and not big
        c["quad"] = rng.choice(["lin", "gl"])
    elif kind == "update":
        fp64 = c["pw"] <= 19 and rng.random() < 0.4
        c["precision"], c["digits"] = ("fp64" if fp64 else "tc"), 7
    else:
        c["precision"], c["digits"], c["iters"] = "tc", 7, 2
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _rand(shape, seed, scale=1.0):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return torch.randn(shape, generator=g, device=_device(), dtype=torch.float64) * scale


def _antisym(x, p, q):
    return x - x.transpose(p, q)


def _fermi(beta, e, mu):
    x = beta * (e - mu)
    ex = np.exp(-np.abs(x))
    return np.where(x > 0, ex / (1.0 + ex), 1.0 / (1.0 + ex))


def _grid(ng, beta, quad):
    """Nodes, weights and cumulative weights: Simpson's rule with a trapezoid first panel, the
    same on logarithmic points, or Gauss-Legendre (dense)."""
    if quad == "gl":
        x, w = np.polynomial.legendre.leggauss(ng)
        ti, g = 0.5 * beta * (x + 1.0), 0.5 * beta * w
        xq, wq = np.polynomial.legendre.leggauss(ng + 2)
        vinv = np.linalg.inv(np.polynomial.legendre.legvander(x, ng - 1))
        tq = 0.5 * ti[:, None] * (xq[None] + 1.0)
        p = np.polynomial.legendre.legvander(2.0 * tq / beta - 1.0, ng - 1)
        return ti, g, 0.5 * ti[:, None] * np.einsum("q,yqd,dx->yx", wq, p, vinv)
    delta = (math.e - 1.0) / (ng - 1.0) if quad == "ln" else beta / (ng - 1.0)
    s = np.arange(ng) * delta + (1.0 if quad == "ln" else 0.0)
    G = np.zeros((ng, ng))
    for y in range(1, ng):
        if y == 1:
            G[1, :2] = 0.5 * delta
        else:
            G[y] = G[y - 2]
            G[y, y - 2:y + 1] += np.array([1.0, 4.0, 1.0]) * delta / 3.0
    g = np.zeros(ng)
    first = 1 - ng % 2
    if first:
        g[:2] += 0.5 * delta
    for y in range(first, ng - 2, 2):
        g[y:y + 3] += np.array([1.0, 4.0, 1.0]) * delta / 3.0
    if quad == "ln":
        return beta * np.log(s), g * beta / s, G * beta / s[None, :]
    return s, g, G


def _ueg_params(case, seed):
    """(rs, theta) of a seed: the case's, varied by a few percent."""
    r = np.random.RandomState(int(seed) % (1 << 31))
    return case["rs"] * (1.0 + 0.05 * (r.rand() - 0.5)), case["theta"] * (1.0 + 0.05 * (r.rand() - 0.5))


def _system(case, seed):
    """(energies, Fock matrix, <pq||rs> on the device, beta, mu), alpha spin orbitals first."""
    dev = _device()
    if case["system"] == "ring":
        r = np.random.RandomState(int(seed) % (1 << 31))
        L, U, beta = case["sites"], case["U"] * (1.0 + 0.05 * (r.rand() - 0.5)), case["beta"]
        e = -2.0 * np.cos(2.0 * np.pi * np.arange(L) / L) + 0.5 * U
        mu, nb = 0.5 * U, L
        k = torch.arange(L, device=dev)
        keep = (k[:, None, None, None] + k[None, :, None, None] - k[None, None, :, None] - k) % L == 0
        direct = keep.double() * (U / L)
        same = torch.zeros_like(direct)
        kin = e - 0.5 * U
    else:
        rs, theta = _ueg_params(case, seed)
        box = (4.0 * np.pi * case["N"] / 3.0) ** (1.0 / 3.0) * rs
        kf = (9.0 * np.pi / 4.0) ** (1.0 / 3.0) / rs
        beta, nb = 1.0 / (theta * 0.5 * kf * kf), case["pw"]
        m = 4
        r = np.arange(-m, m + 1)
        pts = np.stack(np.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
        pts = pts[np.argsort((pts * pts).sum(1), kind="stable")][:nb]
        kin = 0.5 * (2.0 * np.pi / box) ** 2 * (pts * pts).sum(1)
        d = pts[:, None] - pts[None]
        q2 = (d * d).sum(-1).astype(float)
        v = np.where(q2 > 0, 4.0 * np.pi / box ** 3 * (box / (2.0 * np.pi)) ** 2 / np.maximum(q2, 1.0), 0.0)
        e = kin - v[:, :max(1, case["N"] // 2)].sum(1)
        code = torch.as_tensor(((pts[:, 0] + 20) * 100 + pts[:, 1] + 20) * 100 + pts[:, 2] + 20, device=dev)
        s = code[:, None] + code[None]
        keep = s[:, :, None, None] == s[None, None]
        direct = keep.double() * torch.as_tensor(v, device=dev)[:, None, :, None]
        same = direct
        lo, hi = e.min() - 50.0 / beta - 1.0, e.max() + 50.0 / beta + 1.0
        for _ in range(100):
            mu = 0.5 * (lo + hi)
            lo, hi = (mu, hi) if 2.0 * _fermi(beta, e, mu).sum() < case["N"] else (lo, mu)
    n = 2 * nb
    eri = torch.zeros((n,) * 4, dtype=torch.float64, device=dev)
    A, B = slice(0, nb), slice(nb, n)
    for x, y in ((A, A), (A, B), (B, A), (B, B)):
        eri[x, y, x, y] += same if x is y else direct
    for x, y in ((A, A), (A, B), (B, A), (B, B)):
        eri[x, y, y, x] -= (same if x is y else direct).transpose(2, 3)
    en = np.hstack((e, e))
    fo = torch.as_tensor(_fermi(beta, en, mu), device=dev)
    diag = torch.diagonal(eri, dim1=1, dim2=3)                          # <pr||qr>
    fock = np.diag(np.hstack((kin, kin))) + (diag @ fo).cpu().numpy()
    return en, fock, eri, beta, float(mu)


def _scaled(en, fock, eri, beta, mu):
    """The Fermi-scaled blocks: sqrt(f) on every o index, sqrt(1 - f) on every v index."""
    f = _fermi(beta, en, mu)
    s = {"o": torch.as_tensor(np.sqrt(f), device=eri.device), "v": torch.as_tensor(np.sqrt(1.0 - f), device=eri.device)}
    fm = torch.as_tensor(fock - np.diag(en), device=eri.device)
    F = {b: fm * s[b[0]][:, None] * s[b[1]] for b in F_BLOCKS}
    I = {b: eri * s[b[0]][:, None, None, None] * s[b[1]][:, None, None] * s[b[2]][:, None] * s[b[3]]
         for b in I_BLOCKS}
    return F, I


def _spin_mask(n, dev):
    s = (torch.arange(n, device=dev) >= n // 2).int()
    return s[:, None, None, None] + s[None, :, None, None] == s[None, None, :, None] + s


def _amplitudes(case, seed, en, I, F, beta):
    """Amplitudes as an iteration meets them: the size of the first-order ones, antisymmetric,
    spin-conserving, growing along tau."""
    n, ng = en.shape[0], case["ng"]
    ramp = torch.linspace(0.1, 1.0, ng, dtype=torch.float64, device=_device())
    same = (torch.arange(n, device=_device()) >= n // 2)
    t1 = _rand((ng, n, n), seed + 101, 0.02) * (same[:, None] == same).double() * ramp[:, None, None]
    t2 = _rand((ng, n, n, n, n), seed + 202, 0.1)
    t2 = _antisym(_antisym(t2, 1, 2), 3, 4) * _spin_mask(n, _device()).double()
    t2 = t2 * (I["vvoo"].abs() + 1e-4 * I["vvoo"].abs().max()) * beta * ramp[:, None, None, None, None]
    return t1.contiguous(), t2.contiguous()


def _denominators(en):
    e = torch.as_tensor(en, device=_device())
    d1 = e[:, None] - e
    return d1, e[:, None, None, None] + e[None, :, None, None] - e[None, None, :, None] - e


def _blocks(case, seed):
    """General F and I blocks sliced from one antisymmetric tensor, and amplitudes."""
    nv, no = case["nv"], case["no"]
    n = nv + no
    f, g = _rand((n, n), seed + 1, 0.2), _rand((n,) * 4, seed + 2, 0.1)
    g = _antisym(_antisym(g, 0, 1), 2, 3)
    sl = {"o": slice(0, no), "v": slice(no, n)}
    F = {b: f[sl[b[0]], sl[b[1]]].contiguous() for b in F_BLOCKS}
    I = {b: g[tuple(sl[c] for c in b)].contiguous() for b in I_BLOCKS}
    t1 = _rand((nv, no), seed + 3, 0.05)
    t2 = _antisym(_antisym(_rand((nv, nv, no, no), seed + 4, 0.05), 0, 1), 2, 3).contiguous()
    T1, T2 = -F["vo"], -I["vvoo"]
    return F, I, t1, t2, T1.contiguous(), T2.contiguous()


class _Container(object):
    def __init__(self, **kw):
        self.__dict__.update(kw)


class _View(object):
    """A device buffer as __cuda_array_interface__."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "version": 3,
                                         "data": (int(ptr), False)}


def _tensor(d):
    """A DeviceArray as a torch tensor on the same memory."""
    return torch.as_tensor(_View(d.ptr.value, d.shape, d), device="cuda")


def _dev(ctx, t):
    """A torch tensor as a DeviceArray on the same memory."""
    return _lib.DeviceArray(ctx, t.shape, ptr=t.data_ptr(), owner=t)


def _containers(ctx, F, I):
    return (_Container(**{b: _dev(ctx, F[b].contiguous()) for b in F_BLOCKS}),
            _Container(**{b: _dev(ctx, I[b].contiguous()) for b in I_BLOCKS}))


# ---------------------------------------------------------------------------
# the cases' state and pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    ctx = _lib.context(0)
    kind = case["kind"]
    st = {"case": case, "ctx": ctx}
    if kind == "solve":
        rs, theta = _ueg_params(case, seed)
        s = systems.ueg_recipe(case["N"], rs, case["pw"], theta)
        s.g_aint_tot()
        st["system"] = s
        return st
    prec = (PRECISION[case["precision"]], case["digits"]) if "precision" in case else None
    st["prec"] = prec
    if kind in ("step", "lambda"):
        en, fock, eri, beta, mu = _system(case, seed)
        ti, g, G = _grid(case["ng"], beta, case["quad"])
        torch.cuda.synchronize()
        ctx.set_precision(*prec)
        # several solvers share the device, as in a served stream
        ctx.set_workspace_limit(48 << 30)
        sv = DeviceSolver.from_system(ctx, en, fock, _dev(ctx, eri), beta, mu, ti, g, G)
        sv.full = case["quad"] == "gl"
        if case.get("accel"):
            sv.set_acceleration(case["accel"])
        if case.get("graph"):
            sv.set_graph(True)
        sv.guess(1)
        st["solver"] = sv
        if kind == "step":
            p1, p2 = _lib.vp(), _lib.vp()
            ctx.check(ctx.L.kvft_solver_device_amplitudes(sv.h, _lib.ctypes.byref(p1), _lib.ctypes.byref(p2)),
                      "kvft_solver_device_amplitudes")
            n = en.shape[0]
            st["T"] = (torch.as_tensor(_View(p1.value, (case["ng"], n, n), sv), device="cuda"),
                       torch.as_tensor(_View(p2.value, (case["ng"], n, n, n, n), sv), device="cuda"))
        return st
    if kind == "update":
        en, fock, eri, beta, mu = _system(case, seed)
        F, I = _scaled(en, fock, eri, beta, mu)
        del eri
        t1, t2 = _amplitudes(case, seed, en, I, F, beta)
        st["F"], st["I"] = _containers(ctx, F, I)
        grid = [torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in _grid(case["ng"], beta, case["quad"])]
        st["args"] = [_dev(ctx, x) for x in (t1, t2, *_denominators(en), grid[0], grid[2])]
    elif kind == "residual":
        F, I, t1, t2, T1, T2 = _blocks(case, seed)
        st["F"], st["I"] = _containers(ctx, F, I)
        st["t"], st["T"] = (_dev(ctx, t1), _dev(ctx, t2)), (T1, T2)
        st["dT"] = (_dev(ctx, T1), _dev(ctx, T2))
    else:
        st["args"] = [_dev(ctx, x) for x in _plain_inputs(case, seed)]
    torch.cuda.synchronize()
    return st


def _plain_inputs(case, seed):
    """Inputs of the stand-alone tau integral and energy."""
    nv, no, ng = case["nv"], case["no"], case["ng"]
    t2 = _rand((ng, nv, nv, no, no), seed + 5, 0.05)
    r = np.random.RandomState(int(seed) % (1 << 31))
    if case["kind"] == "energy":
        _, g, _ = _grid(ng, 2.0, "lin")
        return [_rand((ng, nv, no), seed + 6, 0.05), t2, _rand((no, nv), seed + 7, 0.1),
                _rand((no, no, nv, nv), seed + 8, 0.1), torch.as_tensor(g, device=_device())]
    ev, eo = [torch.as_tensor(np.sort(r.rand(k)) * 2.0, device=_device()) for k in (nv, no)]
    d2 = ev[:, None, None, None] + ev[None, :, None, None] - eo[None, None, :, None] - eo
    ti, _, G = _grid(ng, 2.0, case["quad"])
    return [t2, torch.as_tensor(ti, device=_device()), d2.contiguous(),
            torch.as_tensor(np.ascontiguousarray(G), device=_device())]


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "solve":
        s = st["system"]
        cc = ccsd(s, T=s.T, mu=s.mu, max_iter=100, damp=0.5, ngrid=case["ng"], econv=1e-10,
                  quad=case["quad"], precision=case["precision"], digits=case["digits"], accel=3,
                  mix=0.7, low_tconv=3e-4, ctx=ctx)
        omega, omega_cc = cc.run()
        cc.release()
        return {"omega": np.float64(omega), "omega_cc": np.float64(omega_cc), "T1": cc.T1, "T2": cc.T2}
    if st["prec"]:
        ctx.set_precision(*st["prec"])
    if kind == "step":
        energy, res = st["solver"].step(0.5)
        return {"T1": st["T"][0], "T2": st["T"][1], "energy": np.float64(energy), "residual": res}
    if kind == "lambda":
        L1, L2 = st["solver"].lambda_solve({"max_iter": case["iters"], "damp": 0.2, "tconv": 1e-8})
        return {"L1": L1, "L2": L2}
    if kind == "update":
        t1, t2, d1, d2, ti, G = st["args"]
        o1, o2 = ft_cc_equations.ccsd_stanton(st["F"], st["I"], t1, t2, d1, d2, ti, case["ng"], G, ctx=ctx)
        return {"T1": _tensor(o1), "T2": _tensor(o2)}
    if kind == "residual":
        ft_cc_equations.stanton_residual(st["dT"][0], st["dT"][1], st["F"], st["I"], st["t"][0], st["t"][1],
                                         fac=-1.0, ctx=ctx)
        return {"T1": st["T"][0], "T2": st["T"][1]}
    if kind == "tbar":
        t2, ti, d2, G = st["args"]
        return _tensor(quadrature.int_tbar2(case["ng"], t2, ti, d2, G, full=case["quad"] == "gl", ctx=ctx))
    t1, t2, f, eri, g = st["args"]
    return np.float64(ft_cc_energy.ft_cc_energy(t1, t2, f, eri, g, 2.0, ctx=ctx))


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _residual_flops(nv, no, half):
    """Floating-point operations of one residual: the pair ladders, the two ring contractions and
    the n^5 terms, over the spin-conserving products when the blocks conserve spin."""
    if half:
        h = half
        pairs = (h * (h - 1) // 2, h * h, h * (h - 1) // 2)
        return sum(6.0 * p ** 3 for p in pairs) + 40.0 * h ** 6 + 14 * 6 * 2.0 * h ** 5
    pv, po = nv * (nv - 1) / 2.0, no * (no - 1) / 2.0
    ring = (nv * no) ** 3
    n5 = nv * no * (2 * nv * nv * no + 2 * no * no * nv + nv ** 3 + 2 * nv * no * (nv + no) + no ** 3)
    return 2.0 * (2 * pv * po * po + pv * pv * po) + 4.0 * ring + 2.0 * n5


def work(case):
    kind = case["kind"]
    if kind in ("tbar", "energy", "residual"):
        nv, no, ng = case["nv"], case["no"], case.get("ng", 1)
        t2 = 8.0 * ng * (nv * no) ** 2
        if kind == "tbar":
            return {"bytes": 2 * t2 + t2 / ng, "flops": 2.0 * ng * (ng if case["quad"] == "gl" else 3) * (nv * no) ** 2}
        if kind == "energy":
            return {"bytes": t2 + t2 / ng, "flops": 4.0 * ng * (nv * no) ** 2}
        ints = 8.0 * (nv ** 4 + 2 * nv ** 3 * no + 3 * (nv * no) ** 2 + 2 * nv * no ** 3 + no ** 4)
        return {"bytes": ints + 3 * t2, "flops": _residual_flops(nv, no, 0)}
    half = case["sites"] if case["system"] == "ring" else case["pw"]
    ng, t2 = case["ng"], 8.0 * 6 * half ** 4
    one = _residual_flops(2 * half, 2 * half, half) * ng
    if kind == "lambda":
        return {"bytes": 9 * t2 + ng * t2 + case["iters"] * 2 * ng * t2, "flops": case["iters"] * 4.0 * (2 * half) ** 6 * ng}
    sweeps = 14 if kind == "solve" else 1
    return {"bytes": 9 * t2 + sweeps * 2 * ng * t2, "flops": sweeps * one}


# ---------------------------------------------------------------------------
# the same in FP64 with torch
# ---------------------------------------------------------------------------
def _residual(F, I, t1, t2):
    """The spin-orbital CCSD residual (Stanton, Gauss, Watts and Bartlett, J. Chem. Phys. 94, 4334)
    without its driving terms."""
    es = torch.einsum
    tt = es("ai,bj->abij", t1, t1)
    tt = tt - tt.transpose(0, 1)
    tau, ttau = t2 + tt, t2 + 0.5 * tt
    Fae = F["vv"] - 0.5 * es("me,am->ae", F["ov"], t1) - es("fm,amfe->ae", t1, I["vovv"]) \
        - 0.5 * es("afmn,mnef->ae", ttau, I["oovv"])
    Fmi = F["oo"] + 0.5 * es("ei,me->mi", t1, F["ov"]) + es("en,mnie->mi", t1, I["ooov"]) \
        + 0.5 * es("efin,mnef->mi", ttau, I["oovv"])
    Fme = F["ov"] + es("fn,mnef->me", t1, I["oovv"])
    x = es("ej,mnie->mnij", t1, I["ooov"])
    # the tau <mn||ef> tau term of W_abef is carried by W_mnij
    Wmnij = I["oooo"] + x - x.transpose(2, 3) + 0.5 * es("efij,mnef->mnij", tau, I["oovv"])
    x = es("bm,amef->abef", t1, I["vovv"])
    Wabef = I["vvvv"] - x + x.transpose(0, 1)
    W = -I["vovo"].transpose(0, 1) - es("fj,bmef->mbej", t1, I["vovv"]) + es("bn,mnje->mbej", t1, I["ooov"]) \
        - es("fbjn,mnef->mbej", 0.5 * t2 + es("fj,bn->fbjn", t1, t1), I["oovv"])
    R1 = Fae @ t1 - t1 @ Fmi + es("aeim,me->ai", t2, Fme) - es("fn,anfi->ai", t1, I["vovo"]) \
        + 0.5 * es("efim,amef->ai", t2, I["vovv"]) + 0.5 * es("aemn,nmie->ai", t2, I["ooov"])
    x = es("aeij,be->abij", t2, Fae - 0.5 * t1 @ Fme) + es("am,bmij->abij", t1, I["vooo"])
    R2 = x - x.transpose(0, 1)
    x = es("ei,abej->abij", t1, I["vvvo"]) - es("abim,mj->abij", t2, Fmi + 0.5 * Fme @ t1)
    R2 = R2 + x - x.transpose(2, 3)
    x = es("aeim,mbej->abij", t2, W) + es("am,bmij->abij", t1, es("ei,bmej->bmij", t1, I["vovo"]))
    x = x - x.transpose(0, 1)
    R2 = R2 + x - x.transpose(2, 3)
    return R1, R2 + 0.5 * es("abmn,mnij->abij", tau, Wmnij) + 0.5 * es("efij,abef->abij", tau, Wabef)


def _integrate(tb, ti, d, G, full):
    """sum_x G[y,x] w tb[x], w = exp((t_x - t_y) d) for x < y (every x when full), else 1."""
    out = torch.zeros_like(tb)
    for y in range(tb.shape[0]):
        for x in range(tb.shape[0]):
            if G[y, x] != 0.0:
                w = torch.exp((ti[x] - ti[y]) * d) if full or x < y else 1.0
                out[y] += float(G[y, x]) * w * tb[x]
    return out


def _update(F, I, t1, t2, d1, d2, ti, G, full):
    b = [_residual(F, I, a, c) for a, c in zip(t1, t2)]
    return (_integrate(torch.stack([-F["vo"] - r for r, _ in b]), ti, d1, G, full),
            _integrate(torch.stack([-I["vvoo"] - r for _, r in b]), ti, d2, G, full))


def _energy(T1, T2, f, eri, g, beta):
    w = torch.as_tensor(g, device=T1.device)
    q = torch.einsum("y,yabij->abij", w, T2) * 0.25 + 0.5 * torch.einsum("y,yai,ybj->abij", w, T1, T1)
    return float((torch.einsum("y,yai,ia->", w, T1, f) + (q.permute(2, 3, 0, 1) * eri).sum()) / beta)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return None
    if kind == "energy":
        t1, t2, f, eri, g = _plain_inputs(case, seed)
        return np.float64(_energy(t1, t2, f, eri, g, 2.0))
    if kind == "tbar":
        t2, ti, d2, G = _plain_inputs(case, seed)
        return _integrate(t2, ti, d2, G, case["quad"] == "gl")
    if kind == "residual":
        F, I, t1, t2, T1, T2 = _blocks(case, seed)
        R1, R2 = _residual(F, I, t1, t2)
        return {"T1": T1 - R1, "T2": T2 - R2}
    n = 2 * (case["sites"] if case["system"] == "ring" else case["pw"])
    if 30.0 * n ** 6 * case["ng"] * (4 * case["iters"] if kind == "lambda" else 1) > 8e12:
        return None
    en, fock, eri, beta, mu = _system(case, seed)
    F, I = _scaled(en, fock, eri, beta, mu)
    ti, g, G = _grid(case["ng"], beta, case["quad"])
    d1, d2 = _denominators(en)
    full = case["quad"] == "gl"
    if kind == "update":
        t1, t2 = _amplitudes(case, seed, en, I, F, beta)
        o1, o2 = _update(F, I, t1, t2, d1, d2, ti, G, full)
        return {"T1": o1, "T2": o2}
    ng = case["ng"]
    x1 = _integrate((-F["vo"]).expand(ng, n, n).contiguous(), ti, d1, G, full)
    x2 = _integrate((-I["vvoo"]).expand(ng, n, n, n, n).contiguous(), ti, d2, G, full)
    if kind == "step":
        o1, o2 = _update(F, I, x1, x2, d1, d2, ti, G, full)
        T1, T2 = 0.5 * (x1 + o1), 0.5 * (x2 + o2)
        return {"T1": T1, "T2": T2, "energy": np.float64(_energy(T1, T2, F["ov"], I["oovv"], g, beta)),
                "residual": None}
    L1 = ((F["ov"] + torch.einsum("ijab,ybj->yia", I["oovv"], x1)) / beta).contiguous()
    L2 = (I["oovv"] / beta).expand(ng, n, n, n, n).contiguous()
    Gb = g[None, :] * G.T / g[:, None]                 # the integral run backwards
    for _ in range(case["iters"]):
        M1, M2 = torch.zeros_like(L1), torch.zeros_like(L2)
        for s in range(ng):
            for y in range(s, ng):
                if Gb[s, y] != 0.0:
                    M1[s] += float(Gb[s, y]) * torch.exp((ti[s] - ti[y]) * d1.T) * L1[y]
                    M2[s] += float(Gb[s, y]) * torch.exp((ti[s] - ti[y]) * d2.permute(2, 3, 0, 1)) * L2[y]
        for y in range(ng):
            a, b = x1[y].clone().requires_grad_(), x2[y].clone().requires_grad_()
            R1, R2 = _residual(F, I, a, b)
            f = (M1[y].T * R1).sum() + 0.25 * (M2[y].permute(2, 3, 0, 1) * R2).sum()
            ga, gb = torch.autograd.grad(f, (a, b))
            gb = _antisym(_antisym(gb, 0, 1), 2, 3)
            e1 = F["ov"] + torch.einsum("ijab,bj->ia", I["oovv"], x1[y])
            L1[y] = 0.2 * L1[y] + 0.8 * (-e1 - ga.T)
            L2[y] = 0.2 * L2[y] + 0.8 * (-I["oovv"] - gb.permute(2, 3, 0, 1))
    return {"L1": L1, "L2": L2}
