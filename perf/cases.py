"""Timed cases of the GB300 finite-strain FFT crystal-plasticity path.

Each case is work that a user of the library has it do, through the public Python mirror of
the C-ABI, over the range of grids, crystals and options the path serves:

  green   cpfft_green_apply_noalloc on the caller's device buffers (host programs that own
          all device memory; the smallest call of the path)
  mirror  G_K_dF on host arrays (mirror mode: the Fortran driver keeps its own CG)
  pcg     fftPcg, plain FP64 or the mixed form, with an elasto-plastic tangent
  stress  one implicit stress pass of a load step on the device-resident state
  run     whole `compute` sequences (initialisation, homogenised tangent, load steps) of one
          RVE or of several at once
  disp    nodal displacements of an output step
  text    the element result lines of an output step

``exact`` restates the arithmetic in 64 bits with plain torch.
"""
import ctypes
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import cpfft_gb300 as cp
from cpfft_gb300 import rve

CRYSTALS = {"fcc": rve.FCC_VOCE, "bcc": dict(rve.FCC_VOCE, slip_type=2), "bcc48": rve.BCC48_DECK,
            "hcp6": rve.HCP_VOCE, "mrr": rve.MRR_FCC, "ornl": rve.ORNL_FCC}
# time step of each crystal's workload (s): strain rates of 1e-3 / s, the deck's 10 s steps
TSTEP = {"bcc48": 10.0}
# macroscopic strain per load step: the workloads' 1e-3, the deck's 3e-3
STRAIN = {"bcc48": 3.0e-3}
FAST = cp.START_ITERATE | cp.START_TRIAL | cp.TANGENT_F32


def listed():
    return [
        # the smallest call: one operator apply on device buffers, a 16^3 RVE
        {"name": "green-16", "kind": "green", "N": 16, "centered": True, "flgK": True},
        # mirror mode's operator on host fields, a mid-size grid
        {"name": "mirror-64", "kind": "mirror", "N": 64, "centered": True, "flgK": True},
        # a Newton system of the plain form on the reference's odd 63^3 grid
        {"name": "pcg-fp64-63", "kind": "pcg", "N": 63, "fast": False, "grains": 64},
        # a Newton system of the fast form on the headline 128^3 grid
        {"name": "pcg-mixed-128", "kind": "pcg", "N": 128, "fast": True, "grains": 256},
        # stress passes: the plain form, the fast form on the headline grid, the example
        # deck's 48-system crystal, and the dislocation-density law
        {"name": "stress-fcc-64", "kind": "stress", "N": 64, "crystal": "fcc", "fast": False, "grains": 64},
        {"name": "stress-fcc-fast-128", "kind": "stress", "N": 128, "crystal": "fcc", "fast": True, "grains": 256},
        {"name": "stress-bcc48-32", "kind": "stress", "N": 32, "crystal": "bcc48", "fast": False, "grains": 32},
        {"name": "stress-mrr-32", "kind": "stress", "N": 32, "crystal": "mrr", "fast": False, "grains": 32},
        # the 15^3 uniaxial-tension workload in the plain form (first load steps)
        {"name": "run-fp64-15", "kind": "run", "sizes": "15", "steps": 2, "fast": False, "crystal": "fcc", "threads": 1},
        # a batch of RVEs of different sizes in the fast form
        {"name": "run-batch-6", "kind": "run", "sizes": "48,40,33,32,27,24", "steps": 1, "fast": True, "crystal": "fcc", "threads": 6},
        # an output step: nodal displacements, and the stress lines
        {"name": "disp-63", "kind": "disp", "N": 63},
        {"name": "text-48", "kind": "text", "N": 48, "quantity": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["green", "mirror", "pcg", "pcg", "stress", "stress", "stress", "run", "disp", "text"])
    if kind == "green":
        return {"kind": kind, "N": _log(rng, 4, 32), "centered": rng.random() < 0.6, "flgK": rng.random() < 0.8}
    if kind == "mirror":
        return {"kind": kind, "N": _log(rng, 5, 96), "centered": rng.random() < 0.6, "flgK": rng.random() < 0.8}
    if kind == "pcg":
        fast = rng.random() < 0.6
        return {"kind": kind, "N": _log(rng, 9, 112 if fast else 64), "fast": fast, "grains": rng.randint(4, 200)}
    if kind == "stress":
        crystal = rng.choice(["fcc", "fcc", "bcc", "bcc48", "hcp6", "mrr", "ornl"])
        cap = {"mrr": 32, "ornl": 32, "bcc48": 36}.get(crystal, 96)
        return {"kind": kind, "N": _log(rng, 7, cap), "crystal": crystal,
                "fast": rng.random() < 0.5 and crystal not in ("mrr", "ornl"), "grains": rng.randint(2, 200)}
    if kind == "run":
        fast = rng.random() < 0.6
        n = rng.randint(1, 5) if fast else rng.randint(1, 2)
        sizes = [rng.choice([rng.randint(9, 40), 32, 2 * rng.randint(4, 9) + 1]) for _ in range(n)] if fast \
            else [2 * rng.randint(2, 7) + 1 for _ in range(n)]
        return {"kind": kind, "sizes": ",".join(map(str, sizes)), "steps": 1, "fast": fast,
                "crystal": rng.choice(["fcc", "fcc", "bcc", "hcp6"]), "threads": rng.randint(1, 6)}
    if kind == "disp":
        return {"kind": kind, "N": _log(rng, 5, 96)}
    return {"kind": kind, "N": _log(rng, 5, 64), "quantity": rng.choice([1, 2])}


# ---- inputs, from the seed alone ---------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _grains(N, n, g):
    """Grain of every voxel of a periodic Voronoi tessellation with n seeds (voxel
    v = a + N b + N^2 c), and each grain's Haar-random Kocks angles in degrees (n, 3)."""
    seeds = _rand(g, n, 3).float()
    ax = (torch.arange(N, device="cuda", dtype=torch.float32) + 0.5) / N
    pts = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    best = torch.full((len(pts),), 9.0, device="cuda")
    grain = torch.zeros(len(pts), dtype=torch.int64, device="cuda")
    for k in range(n):
        d = pts - seeds[k]
        d = d - d.round()
        r = (d * d).sum(1)
        near = r < best
        best = torch.where(near, r, best)
        grain = torch.where(near, torch.full_like(grain, k), grain)
    u = _rand(g, n, 3)
    ang = torch.stack([360.0 * u[:, 0] - 180.0, torch.rad2deg(torch.acos(2.0 * u[:, 1] - 1.0)),
                       360.0 * u[:, 2] - 180.0], 1)
    return grain, ang


def _rve_input(N, n, crystal, g):
    grain, ang = _grains(N, n, g)
    return {"N": N, "grain": grain, "ang": ang, "kocks": ang[grain].T.contiguous().cpu().numpy(),
            "mat": np.ones(N ** 3, dtype=np.int32), "crystals": [dict(CRYSTALS[crystal])],
            "tstep": TSTEP.get(crystal, 1.0)}


def _deformation(r, n_grains, strain, g):
    """(F at n, F at n+1), each (9, N3): plane-strain compression in two load steps, the first
    twice as large, with grain-scale and voxel-scale fluctuations."""
    N3 = r["N"] ** 3
    eye = torch.eye(3, device="cuda", dtype=torch.float64).reshape(9, 1)
    bar = torch.diag(torch.tensor([1.0, 0.0, -1.0], device="cuda", dtype=torch.float64)).reshape(9, 1)

    def step(size):
        return size * (bar + 0.25 * _randn(g, 9, n_grains)[:, r["grain"]] + 0.05 * _randn(g, 9, N3))

    F1 = eye + step(2.0 * strain)
    F2 = F1 + step(strain)
    return F1, F2


def _tangent(N, n, g):
    """A tangent field dP/dF (81, N3) of an elasto-plastic polycrystal and its two symmetries'
    initial-stress term: per grain a cubic elastic stiffness whose shear moduli plastic flow
    has softened, with the major symmetry the CG needs."""
    grain, _ = _grains(N, n, g)
    soft = torch.exp(math.log(0.06) * _rand(g, n, 1))
    mu, lam = 75.0e3 * soft, 121.0e3 * torch.ones(n, 1, dtype=torch.float64, device="cuda")
    d = torch.eye(3, device="cuda", dtype=torch.float64)
    vol = torch.einsum("ij,kl->ijkl", d, d).reshape(1, 81)
    sym = (torch.einsum("ik,jl->ijkl", d, d) + torch.einsum("il,jk->ijkl", d, d)).reshape(1, 81)
    Q = torch.linalg.qr(_randn(g, n, 3, 3))[0]
    cubic = torch.einsum("gia,gja,gka,gla->gijkl", Q, Q, Q, Q).reshape(n, 81)
    s = 100.0 * _randn(g, n, 3, 3)
    s = 0.5 * (s + s.transpose(1, 2))
    geo = torch.einsum("ik,gjl->gijkl", d, s).reshape(n, 81)
    Kg = lam * vol + mu * sym - 0.4 * mu * cubic + geo
    return Kg.T.contiguous()[:, grain]


def _qmap(N, centered):
    f = torch.arange(N, device="cuda")
    if centered:
        return torch.where(f <= (N - 1) // 2, f, f - N).double()
    half = (N + 1) // 2 if N % 2 else N // 2 + 1
    return (torch.remainder(f - half, N) + 1 - half).double()


def _green(x, N, centered):
    """Re(IDFT(Ghat(q) DFT(x))): (9, N3) -> (9, N3)."""
    X = torch.fft.fftn(x.reshape(3, 3, N, N, N), dim=(2, 3, 4))
    q1 = _qmap(N, centered)
    q = torch.stack(torch.meshgrid(q1, q1, q1, indexing="ij"))
    qq = (q * q).sum(0)
    inv = torch.where(qq > 0, 1.0 / torch.where(qq > 0, qq, torch.ones_like(qq)), torch.zeros_like(qq))
    if centered and N % 2 == 0:
        inv[N // 2], inv[:, N // 2], inv[:, :, N // 2] = 0.0, 0.0, 0.0
    div = (X * q).sum(1) * inv
    Y = div[:, None] * q[None]
    return torch.fft.ifftn(Y, dim=(2, 3, 4)).real.reshape(9, N ** 3)


def _contract(K, x):
    return (K.reshape(9, 9, -1) * x).sum(1)


class _Rve:
    """A Solver on a host thread of its own: a library context belongs to the thread that made
    it, so a program that holds several RVEs drives each from its own thread."""

    def __init__(self, *args, **kw):
        self._pool = ThreadPoolExecutor(1)
        self.solver = self.call(lambda: cp.Solver(*args, **kw))

    def call(self, fn, *args, **kw):
        return self._pool.submit(fn, *args, **kw).result()

    def __del__(self):
        try:
            if getattr(self, "solver", None) is not None:
                self.call(self.solver.close)
            self._pool.shutdown()
        except RuntimeError:  # the interpreter is ending and has stopped the thread
            pass


def _plain_rve(N, centered=True, fast=False):
    """A context for calls that need a grid but no particular microstructure."""
    one = np.ones(N ** 3, dtype=np.int32)
    return _Rve(N, one, np.zeros((3, N ** 3)), [dict(rve.FCC_VOCE)], 1.0,
                cp.G_CENTERED if centered else cp.G_REF_SHIFT,
                cp.PREC_MIXED if fast else cp.PREC_FP64)


def _inputs(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("green", "mirror"):
        N = case["N"]
        x = 1.0e-3 * _randn(g, 9, N ** 3)
        K = _tangent(N, 8, g) if case["flgK"] else None
        return {"x": x, "K": K}
    if kind == "pcg":
        N = case["N"]
        K = _tangent(N, case["grains"], g)
        bar = torch.diag(torch.tensor([1.0e-3, 0.0, -1.0e-3], device="cuda", dtype=torch.float64))
        b = -_green(_contract(K, bar.reshape(9, 1).expand(9, N ** 3)), N, True)
        return {"K": K, "b": b}
    if kind in ("stress", "text"):
        crystal = case.get("crystal", "fcc")
        n = case.get("grains", 16)
        r = _rve_input(case["N"], n, crystal, g)
        r["F1"], r["F2"] = _deformation(r, n, STRAIN.get(crystal, 1.0e-3), g)
        return r
    if kind == "disp":
        N = case["N"]
        return {"F": torch.eye(3, device="cuda", dtype=torch.float64).reshape(9, 1) + 0.01 * _randn(g, 9, N ** 3)}
    return [_rve_input(int(N), max(2, int(N) // 2), case["crystal"], g) for N in case["sizes"].split(",")]


def prepare(case, seed):
    kind = case["kind"]
    inp = _inputs(case, seed)
    state = {"case": dict(case)}
    if kind == "green":
        state.update(inp, y=torch.empty_like(inp["x"]))
    elif kind == "mirror":
        state["rve"] = _plain_rve(case["N"], case["centered"])
        if case["flgK"]:
            state["rve"].call(state["rve"].solver.set_K4, inp["K"].cpu().numpy())
        state["x"] = inp["x"].cpu().numpy()
    elif kind == "pcg":
        fast = case["fast"]
        state["rve"] = _plain_rve(case["N"], True, fast)
        if fast:
            state["rve"].call(state["rve"].solver.set_precond, cp.PRECOND_REFERENCE)
        state["rve"].call(state["rve"].solver.set_K4, inp["K"].cpu().numpy())
        state["b"] = inp["b"].cpu().numpy()
    elif kind in ("stress", "text"):
        fast = bool(case.get("fast"))
        r = _Rve(case["N"], inp["mat"], inp["kocks"], inp["crystals"], inp["tstep"], cp.G_CENTERED)
        if fast:
            r.call(r.solver.set_mode, cp.PREC_MIXED, FAST)
            r.call(r.solver.set_precond, cp.PRECOND_REFERENCE)
            r.call(r.solver.set_schedule, cp.SCHED_QUEUE)
        eye = np.zeros((9, case["N"] ** 3))
        eye[[0, 4, 8]] = 1.0
        # the load step before: its pass, rolled over
        r.call(r.solver.drive_eps_sig, 1, 1, eye, inp["F1"].cpu().numpy(), False)
        r.call(r.solver.commit)
        r.call(r.solver.set_F, None, inp["F2"].cpu().numpy())
        state["rve"] = r
    elif kind == "disp":
        state["rve"] = _plain_rve(case["N"])
        state["rve"].call(state["rve"].solver.set_F, None, inp["F"].cpu().numpy())
    else:
        load = rve.uniaxial_tension(1.0e-3 * case["steps"], case["steps"])
        fast = case["fast"]
        state["rves"] = [dict(N=r["N"], mat_list=r["mat"], kocks=r["kocks"], crystals=r["crystals"],
                              tstep=r["tstep"], nsteps=case["steps"], BC_all=load.BC_all, isNBC=load.isNBC,
                              g_mapping=cp.G_CENTERED if fast else cp.G_REF_SHIFT) for r in inp]
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "green":
        dp = ctypes.POINTER(ctypes.c_double)
        K = state["K"]
        rc = cp.load_library().cpfft_green_apply_noalloc(
            case["N"], cp.G_CENTERED if case["centered"] else cp.G_REF_SHIFT,
            ctypes.cast(state["x"].data_ptr(), dp), None if K is None else ctypes.cast(K.data_ptr(), dp),
            int(case["flgK"]), ctypes.cast(state["y"].data_ptr(), dp), torch.cuda.current_stream().cuda_stream)
        if rc < 0:
            raise cp.CpfftError(rc, "green_apply_noalloc", cp.load_library().cpfft_last_error().decode())
        return state["y"]
    if kind == "run":
        fast = case["fast"]
        out = cp.batch_solve(state["rves"], precision=cp.PREC_MIXED if fast else cp.PREC_FP64,
                             options=FAST if fast else 0, nthreads=case["threads"], want_fields=True)
        return [{"Pbar": o["Pbar"], "F": o["F"], "P": o["P"]} for o in out]
    s = state["rve"].solver
    if kind == "mirror":
        return state["rve"].call(s.G_K_dF, state["x"], case["flgK"])
    if kind == "pcg":
        return state["rve"].call(s.fftPcg, state["b"], 1.0e-10)[0]
    if kind == "stress":
        return state["rve"].call(s.drive_eps_sig, 2, 1)[0]
    if kind == "disp":
        return state["rve"].call(s.f2disp)
    return np.frombuffer(state["rve"].call(s.format_flat, case["quantity"]), dtype=np.uint8)


# ---- the work of a pass ------------------------------------------------------------------
def _green_work(N, flgK, word, transforms=18):
    N3 = N ** 3
    return {"bytes": (18 + (81 if flgK else 0)) * word * N3,
            "flops": (transforms * 2.5 * math.log2(max(N3, 2)) + (162 if flgK else 0)) * N3}


def _stress_work(N, crystal, fast):
    """18 deformation words, the history in and out, P, and the tangent out; the local solve
    of 3 Newton iterations (residual, Jacobian and elimination), set-up and tangent."""
    nh = 55 if crystal in ("mrr", "ornl") else 31
    ns = {"bcc48": 48, "hcp6": 6}.get(crystal, 12)
    flops = 6000.0 + 3 * (240.0 * ns + 400.0) if crystal not in ("mrr", "ornl") else 8000.0 + 3 * 16000.0
    return {"bytes": ((18 + 2 * nh + 9 + 81) * 8 + (324 if fast else 0)) * N ** 3, "flops": flops * N ** 3}


def work(case):
    kind = case["kind"]
    if kind in ("green", "mirror"):
        return _green_work(case["N"], case["flgK"], 8)
    if kind == "pcg":  # nominally 30 iterations: one operator apply and the vector updates each
        word, N = 4 if case["fast"] else 8, case["N"]
        w = _green_work(N, True, word)
        return {"bytes": 30 * (w["bytes"] + 36 * word * N ** 3), "flops": 30 * (w["flops"] + 54 * N ** 3)}
    if kind == "stress":
        return _stress_work(case["N"], case["crystal"], case["fast"])
    if kind == "disp":  # F in, u out; six cosine transforms of three nodal components
        N1 = case["N"] + 1
        return {"bytes": 96.0 * N1 ** 3, "flops": 18 * 2.5 * N1 ** 3 * math.log2(N1)}
    if kind == "text":
        n = 26 if case["quantity"] == 2 else 22
        return {"bytes": (48.0 + 15 * n + 1) * case["N"] ** 3, "flops": 6 * 50.0 * case["N"] ** 3}
    total = {"bytes": 0.0, "flops": 0.0}
    for N in map(int, case["sizes"].split(",")):  # per step 4 stress passes and 13 Krylov solves
        s = _stress_work(N, case["crystal"], case["fast"])
        c = work({"kind": "pcg", "N": N, "fast": case["fast"]})
        for k in total:
            total[k] += case["steps"] * (4 * s[k] + 13 * c[k])
    return total


# ---- 64-bit results ----------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("green", "mirror"):
        i = _inputs(case, seed)
        return _green(_contract(i["K"], i["x"]) if case["flgK"] else i["x"], case["N"], case["centered"])
    if kind == "pcg":
        i = _inputs(case, seed)
        return _pcg(i["K"], i["b"], case["N"])
    if kind == "disp":
        return _displacements(_inputs(case, seed)["F"], case["N"])
    if kind == "stress":
        return _stress(case, _inputs(case, seed))
    return None  # text: bytes; run: a whole solver


def _pcg(K, b, N):
    """G(K : x) = b by CG, far below the tolerance of the timed call."""
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), (r * r).sum()
    end = 1.0e-26 * rr
    for _ in range(400):
        Ap = _green(_contract(K, p), N, True)
        a = rr / (p * Ap).sum()
        x += a * p
        r -= a * Ap
        new = (r * r).sum()
        if new <= end:
            break
        p = r + (new / rr) * p
        rr = new
    return x


def _displacements(F, N, length=100.0):
    """The least-squares nodal positions of the trilinear mesh: (K M M + M K M + M M K) x = B^T F
    on the regular grid, diagonal in the cosine basis, node 1 at the origin."""
    n1, h = N + 1, length / N
    f = F.reshape(3, 3, N, N, N).permute(0, 1, 4, 3, 2)  # [r, j, z, y, x] of voxel a + N b + N^2 c

    def diff(t, axis):  # transpose of the nodal difference along an axis
        z = torch.zeros_like(t.narrow(axis, 0, 1))
        return torch.cat([z, t], axis) - torch.cat([t, z], axis)

    def mean(t, axis):
        z = torch.zeros_like(t.narrow(axis, 0, 1))
        return 0.5 * (torch.cat([z, t], axis) + torch.cat([t, z], axis))

    b = torch.zeros(3, n1, n1, n1, device="cuda", dtype=torch.float64)
    for j, axis in enumerate((3, 2, 1)):  # x fastest in the nodal array [z, y, x]
        t = f[:, j] * (h ** 3 / h)
        for ax in (1, 2, 3):
            t = diff(t, ax) if ax == axis else mean(t, ax)
        b += t
    b[:, 0, 0, 0] = 0.0
    b[:, 0, 0, 0] = -b.sum((1, 2, 3))
    k = torch.arange(n1, device="cuda")
    C = torch.cos(math.pi * ((k[:, None] * k[None]) % (2 * N)).double() / N)
    w = torch.ones(n1, device="cuda", dtype=torch.float64)
    w[0] = w[-1] = 0.5
    c = torch.cos(math.pi * k.double() / N)
    lk, lm = 2.0 / h * (1.0 - c), h / 3.0 * (2.0 + c)

    def outer(u, v, t):
        return torch.einsum("a,b,c->abc", u, v, t)

    lam = outer(lk, lm, lm) + outer(lm, lk, lm) + outer(lm, lm, lk)
    lam[0, 0, 0] = 1.0
    z = _three(b, C) * (2.0 / N) ** 3 * outer(w, w, w) / lam
    z[:, 0, 0, 0] = 0.0
    z = _three(z, C)
    idx = torch.arange(n1, device="cuda", dtype=torch.float64) * h
    X = torch.stack(torch.meshgrid(idx, idx, idx, indexing="ij")[::-1])
    u = z - z[:, :1, :1, :1] - X
    u[:, 0, 0, 0] = 0.0
    return u.reshape(3, -1).T.contiguous()


def _three(b, C):
    for _ in range(3):  # transform the last axis, move it to the front of the three
        b = (b @ C.T).permute(0, 3, 1, 2).contiguous()
    return b


# ---- the stress pass: kinematics, the local equations solved to round-off, P -------------
_VI, _VJ = [0, 1, 2, 0, 1, 0], [0, 1, 2, 1, 2, 2]


def _systems(crystal):
    """(directions, normals) of the crystal's slip systems in its frame, in any order."""
    if crystal == "hcp6":
        a = [[0.5, -math.sqrt(0.75), 0.0], [0.5, math.sqrt(0.75), 0.0], [1.0, 0.0, 0.0]]
        pairs = [(b, [0.0, 0.0, 1.0]) for b in a]
        pairs += [(b, [-b[1], b[0], 0.0]) for b in a]
    else:
        def family(t):
            found = set()
            for i in range(3):
                for j in range(3):
                    for k in range(3):
                        if sorted((i, j, k)) == [0, 1, 2]:
                            for s in range(8):
                                v = tuple((-1 if s >> m & 1 else 1) * t[(i, j, k)[m]] for m in range(3))
                                if v > (0, 0, 0):
                                    found.add(v)
            return sorted(found)

        planes = {"bcc": [(1, 1, 0)], "bcc48": [(1, 1, 0), (1, 1, 2), (1, 2, 3)]}.get(crystal, [(1, 1, 1)])
        along = (1, 1, 1) if crystal in ("bcc", "bcc48") else (1, 1, 0)
        pairs = [(b, n) for p in planes for n in family(p) for b in family(along)
                 if sum(x * y for x, y in zip(b, n)) == 0]
    b = torch.tensor([p[0] for p in pairs], device="cuda", dtype=torch.float64)
    n = torch.tensor([p[1] for p in pairs], device="cuda", dtype=torch.float64)
    return b / b.norm(dim=1, keepdim=True), n / n.norm(dim=1, keepdim=True)


def _stiffness(c):
    C = torch.zeros(6, 6, device="cuda", dtype=torch.float64)
    if c["elastic_type"] == 3:
        c11, c12, c13, c33 = c["C11"], c["C12"], c["C13"], c["C33"]
        C[:3, :3] = torch.tensor([[c11, c12, c13], [c12, c11, c13], [c13, c13, c33]], dtype=torch.float64)
        C[3, 3], C[4, 4], C[5, 5] = c["C44"], c["C55"], c["C55"]
        return C
    lam = c["e"] * c["nu"] / ((1 + c["nu"]) * (1 - 2 * c["nu"]))
    mu = c["e"] / (2 * (1 + c["nu"]))
    C[:3, :3] = lam
    C += torch.diag(torch.tensor([2 * mu] * 3 + [mu] * 3, dtype=torch.float64, device="cuda"))
    return C


def _kocks(ang):
    a = torch.deg2rad(ang)
    ps, th, ph = a[:, 0], a[:, 1], a[:, 2]
    s, c = torch.sin, torch.cos
    r = [-s(ps) * s(ph) - c(ps) * c(ph) * c(th), c(ps) * s(ph) - s(ps) * c(ph) * c(th), c(ph) * s(th),
         s(ps) * c(ph) - c(ps) * s(ph) * c(th), -c(ps) * c(ph) - s(ps) * s(ph) * c(th), s(ph) * s(th),
         c(ps) * s(th), s(ps) * s(th), c(th)]
    return torch.stack(r, 1).reshape(-1, 3, 3)


def _voigt_rotation(R):
    """The 6x6 matrix of R (.) R^T on Voigt vectors of tensor components."""
    out = torch.empty(len(R), 6, 6, device="cuda", dtype=torch.float64)
    for a in range(6):
        i, j = _VI[a], _VJ[a]
        for b in range(6):
            k, l = _VI[b], _VJ[b]
            out[:, a, b] = R[:, i, k] * R[:, j, l] + (R[:, i, l] * R[:, j, k] if b > 2 else 0.0)
    return out


def _minors(t):
    """The rotation of (w23, w13, w12) vectors as the model has it: unsigned minors."""
    pairs = [(1, 2), (0, 2), (0, 1)]
    return torch.stack([t[:, i, k] * t[:, j, l] - t[:, i, l] * t[:, j, k]
                        for i, j in pairs for k, l in pairs], 1).reshape(-1, 3, 3)


def _symsw_tensor():
    B = torch.zeros(6, 6, 3, device="cuda", dtype=torch.float64)
    for a, s, w, v in [(0, 3, 2, 1), (0, 5, 1, -1), (1, 3, 2, 1), (1, 4, 0, -1), (2, 5, 1, 1), (2, 4, 0, 1),
                       (3, 0, 2, .5), (3, 1, 2, -.5), (3, 5, 0, .5), (3, 4, 1, -.5),
                       (4, 1, 0, .5), (4, 2, 0, -.5), (4, 3, 1, .5), (4, 5, 2, .5),
                       (5, 0, 1, .5), (5, 2, 1, -.5), (5, 3, 0, .5), (5, 4, 2, -.5)]:
        B[a, s, w] = v
    return B


def _polar(F):
    R = F.clone()
    for _ in range(12):
        R = 0.5 * (R + torch.linalg.inv(R).transpose(1, 2))
    return R


def _increment(Fn, Fn1):
    """R at n+1 and the unrotated strain increment (engineering shears)."""
    half = 0.5 * (Fn + Fn1)
    L = (Fn1 - Fn) @ torch.linalg.inv(half)
    R = _polar(half)
    D = R.transpose(1, 2) @ (0.5 * (L + L.transpose(1, 2))) @ R
    return _polar(Fn1), torch.stack([D[:, 0, 0], D[:, 1, 1], D[:, 2, 2], 2 * D[:, 0, 1], 2 * D[:, 1, 2],
                                     2 * D[:, 0, 2]], 1)


def _solve(fun, x):
    """Damped Newton on fun(x) -> (residual, Jacobian) for a batch, to round-off."""
    R, J = fun(x)
    n = R.norm(dim=1)
    best, quiet = n.clone(), 0
    for _ in range(80):
        dx = -torch.linalg.solve(J, R)
        step = torch.ones_like(n)
        for _ in range(14):
            y = x + step[:, None] * dx
            Ry = fun(y, False)
            ny = Ry.norm(dim=1)
            bad = ~(ny <= n * (1.0 - 1.0e-4 * step)) & (n > 1.0e-11)
            if not bool(bad.any()):
                break
            step = torch.where(bad, 0.5 * step, step)
        ok = torch.isfinite(ny) & (ny <= torch.maximum(n, torch.full_like(n, 1.0e-11)))
        x = torch.where(ok[:, None], y, x)
        R, J = fun(x)
        n = R.norm(dim=1)
        quiet = quiet + 1 if float(n.max()) < 1.0e-11 or not bool((n < 0.5 * best).any()) else 0
        best = torch.minimum(best, n)
        if quiet >= 2:
            break
    return x


def _stress(case, r):
    if case["N"] > 100 and case["crystal"] != "fcc":
        return None
    c = r["crystals"][0]
    N3 = case["N"] ** 3
    b, n = _systems(case["crystal"])
    tr = _kocks(r["ang"]).transpose(1, 2)
    bs, ns = torch.einsum("gij,sj->gsi", tr, b), torch.einsum("gij,sj->gsi", tr, n)
    A = bs[..., :, None] * ns[..., None, :]
    sym = 0.5 * (A + A.transpose(-1, -2))
    ms0 = torch.stack([sym[..., i, j] * (1.0 if i == j else 2.0) for i, j in zip(_VI, _VJ)], -1)
    qs0 = torch.stack([0.5 * (A[..., 1, 2] - A[..., 2, 1]), 0.5 * (A[..., 0, 2] - A[..., 2, 0]),
                       0.5 * (A[..., 0, 1] - A[..., 1, 0])], -1)
    Rs = _voigt_rotation(tr)
    C = Rs @ _stiffness(c) @ Rs.transpose(1, 2)
    P = torch.empty(9, N3, device="cuda", dtype=torch.float64)
    density = c["h_type"] != 1
    law = _density_law(c, b, n) if density else None
    chunk = 1 << 13 if density else max(1 << 12, (1 << 20) // len(b))
    eye = torch.eye(3, device="cuda", dtype=torch.float64)
    for v0 in range(0, N3, chunk):
        v1 = min(N3, v0 + chunk)
        gr = r["grain"][v0:v1]
        m = v1 - v0
        F1 = r["F1"][:, v0:v1].T.reshape(m, 3, 3)
        F2 = r["F2"][:, v0:v1].T.reshape(m, 3, 3)
        point = {"C": C[gr], "ms0": ms0[gr], "qs0": qs0[gr], "dt": r["tstep"], "c": c, "law": law}
        hard = torch.full((m, 12), c["theta_0"], device="cuda", dtype=torch.float64) if density \
            else torch.full((m, 1), c["tau_y"] + 1.0e-5, device="cuda", dtype=torch.float64)
        sig = torch.zeros(m, 6, device="cuda", dtype=torch.float64)
        Rp = eye.expand(m, 3, 3)
        update = _density_point if density else _voce_point
        sig, hard, Rp, _ = update(point, eye.expand(m, 3, 3), F1, sig, hard, Rp)
        sig, hard, Rp, R = update(point, F1, F2, sig, hard, Rp)
        t = sig[:, [0, 3, 5, 3, 1, 4, 5, 4, 2]].reshape(m, 3, 3)
        P[:, v0:v1] = (torch.linalg.det(F2)[:, None, None] * (R @ t @ R.transpose(1, 2))
                       @ torch.linalg.inv(F2).transpose(1, 2)).reshape(m, 9).T
    return P


def _geometry(p, Fn, Fn1, Rp):
    R, D = _increment(Fn, Fn1)
    T = Rp.transpose(1, 2)
    ms = torch.einsum("mab,msb->msa", _voigt_rotation(T), p["ms0"])
    qc = torch.einsum("mab,msb->msa", _minors(R @ T), p["qs0"])
    return R, D, ms, qc


def _rotated(p, Rp, f):
    """The plastic rotation after the slips f."""
    w = torch.einsum("mab,ms,msb->ma", _minors(Rp.transpose(1, 2)), f, p["qs0"])
    z = torch.zeros_like(w[:, 0])
    W = torch.stack([z, w[:, 2], w[:, 1], -w[:, 2], z, w[:, 0], -w[:, 1], -w[:, 0], z], 1).reshape(-1, 3, 3)
    al = w.norm(dim=1).clamp_min(1.0e-300)[:, None, None]
    half = torch.sin(0.5 * al) / (0.5 * al)
    return (torch.eye(3, device="cuda", dtype=torch.float64) + torch.sin(al) / al * W + 0.5 * half * half * W @ W) @ Rp


def _voce_point(p, Fn, Fn1, nsig, ntt, Rp):
    c, C = p["c"], p["C"]
    R, D, ms, qc = _geometry(p, Fn, Fn1, Rp)
    B = _symsw_tensor()
    nr, th, tv = c["harden_n"], c["theta_0"], c["tau_v"]
    dg = c["gamma_bar"] * p["dt"] if c["alter_mode"] else \
        torch.sqrt(2.0 / 3.0 * ((D[:, :3] ** 2).sum(1) + 0.5 * (D[:, 3:] ** 2).sum(1)))[:, None]
    CD = torch.einsum("mab,mb->ma", C, D)
    Cms = torch.einsum("mab,msb->msa", C, ms)
    # residuals in units of the flow stress
    unit = c["tau_y"]

    def slips(x):
        rs = torch.einsum("msa,ma->ms", ms, x[:, :6])
        pw = (rs.abs() / x[:, 6:]) ** (nr - 1.0)
        return rs, dg * pw * rs / x[:, 6:], dg * pw / x[:, 6:]

    def fun(x, jacobian=True):
        st, tt = x[:, :6], x[:, 6:]
        rs, si, g = slips(x)
        w = torch.einsum("ms,msa->ma", si, qc)
        Bs = torch.einsum("asw,ms->maw", B, st)
        h = 1.0 - (tt - c["tau_y"]) / tv
        hp, dh = h.abs() ** c["voce_m"] * torch.sign(h), -c["voce_m"] / tv * h.abs() ** (c["voce_m"] - 1.0)
        tot = si.abs().sum(1, keepdim=True)
        R1 = st - nsig - CD + torch.einsum("msa,ms->ma", Cms, si) + 2.0 * torch.einsum("maw,mw->ma", Bs, w)
        res = torch.cat([R1, tt - ntt - th * hp * tot], 1) / unit
        if not jacobian:
            return res
        wv = Cms + 2.0 * torch.einsum("maw,msw->msa", Bs, qc)
        J = torch.zeros(len(x), 7, 7, device="cuda", dtype=torch.float64)
        J[:, :6, :6] = torch.eye(6, device="cuda", dtype=torch.float64) + 2.0 * torch.einsum("asw,mw->mas", B, w)
        J[:, :6, :6] += torch.einsum("msa,ms,msb->mab", wv, nr * g, ms)
        J[:, :6, 6] = torch.einsum("msa,ms->ma", wv, -nr * si / tt)
        J[:, 6, :6] = -th * hp * torch.einsum("ms,msa->ma", nr * g * torch.sign(rs), ms)
        J[:, 6, 6] = (1.0 - th * (dh * tot - hp * nr * tot / tt))[:, 0]
        return res, J / unit

    # start: the elastic trial returned along its increment to the rate surface
    r0, dr = torch.einsum("msa,ma->ms", ms, nsig), torch.einsum("msa,ma->ms", ms, CD)
    lim = 0.98 * ntt
    room = torch.where(dr.abs() > 1.0e-300, (torch.sign(dr) * lim - r0) / dr, torch.full_like(dr, 2.0))
    s = room.clamp(min=0.0).min(1, keepdim=True).values.clamp(max=1.0)
    x = _solve(fun, torch.cat([nsig + s * CD, ntt], 1))
    si = slips(x)[1]
    return x[:, :6], x[:, 6:], _rotated(p, Rp, si), R


def _density_law(c, b, n):
    t = torch.linalg.cross(n, b)
    t = t / t.norm(dim=1, keepdim=True)
    Gm = (n @ t.T).abs()
    Hm = torch.linalg.cross(n[:, None].expand(-1, 12, -1), t[None].expand(12, -1, -1)).norm(dim=2)
    kT = c["boltzman"] * 297.0
    G = c["mu_0"] - c["D_0"] / (math.exp(c["T_0"] / 297.0) - 1.0) if c["h_type"] == 4 else c["mu_0"]
    return Gm, Hm, kT, G


def _density_point(p, Fn, Fn1, nsig, nrho, Rp):
    c, C, dt = p["c"], p["C"], p["dt"]
    Gm, Hm, kT, G = p["law"]
    R, D, ms, qc = _geometry(p, Fn, Fn1, Rp)
    B = _symsw_tensor()
    CD = torch.einsum("mab,mb->ma", C, D)
    bb, ornl, Qk = c["burgers"], c["h_type"] == 4, c["G_0_v"] / kT
    cdip = math.sqrt(3.0) * G * bb / (16.0 * math.pi * 0.7)
    cM = 2.0 * kT / (c["u1"] * c["u2"] * c["u3"] * G * bb ** 3)
    E = c["tau_hat_y"] * math.exp(-c["tau_a"] / kT) / kT
    vs = math.exp(-c["G_0_y"]) if c["G_0_y"] < 0.0 else c["G_0_y"]
    unit = 10.0

    def slips(st, rho, m):
        rs = m @ st
        rF, rP = Gm @ rho, Hm @ rho
        if ornl:
            g0, cut = 0.1 * rho * vs * c["u2"] * bb, torch.full_like(rs, c["u3"] * G / c["mu_0"])
        else:
            g0 = c["G_0_y"] * kT / (c["u1"] * c["u3"] * G * bb * bb) * torch.sqrt(rP)
            cut = c["G_0_v"] / (c["u2"] * c["u3"] * bb * bb) * torch.sqrt(rF)
        fr = (rs.abs() - c["u1"] * G * bb * torch.sqrt(rP)) / cut
        sg = torch.where(rs < 0, -1.0, 1.0).double()
        inside = torch.where(fr > 1.0, torch.zeros_like(fr), fr)
        if c["p_v"] == 1.0:
            fp = inside
        else:  # below the passing stress the exponent is 1
            pos = torch.where(inside > 0, inside, torch.ones_like(inside))
            fp = torch.where(inside > 0, pos ** c["p_v"], inside)
        si = torch.where(fr > 1.0, dt * (g0 * c["q_v"] * Qk * c["p_v"] * sg / cut * fr + g0),
                         dt * g0 * sg * torch.exp(-Qk * (1.0 - fp) ** c["q_v"]))
        return rs, rF, rP, si

    def residual(x, C1, m, q, ns, cd, r0):
        st, rho = x[:6] * unit, x[6:] * r0
        rs, rF, rP, si = slips(st, rho, m)
        R1 = st - ns - cd + C1 @ (si @ m) + 2.0 * torch.einsum("asw,s,w->a", B, st, si @ q)
        gd, ars = (si / dt).abs(), rs.abs()
        h = c["u4"] / bb * torch.sqrt(rP) * gd + c["u6"] * cdip / ars / bb * cM * torch.sqrt(rF * rP) * gd \
            - c["u5"] * rho * gd - E * ars * rho * rho * torch.where(gd > 0, torch.where(gd > 0, gd, torch.ones_like(gd)) ** c["tau_hat_v"], torch.zeros_like(gd))
        return torch.cat([R1 / unit, (rho - r0 - dt * h) / r0])

    args = (C, ms, qc, nsig, CD, nrho)
    plain = torch.func.vmap(residual)
    jac = torch.func.vmap(torch.func.jacfwd(residual))

    def fun(x, jacobian=True):
        return (plain(x, *args), jac(x, *args)) if jacobian else plain(x, *args)

    # start inside the passing stresses: the trial pulled back along its increment
    r0, dr = torch.einsum("msa,ma->ms", ms, nsig), torch.einsum("msa,ma->ms", ms, CD)
    lim = c["u1"] * G * bb * torch.sqrt(nrho @ Hm.T)
    room = torch.where(dr.abs() > 1.0e-300, (torch.sign(dr) * lim - r0) / dr, torch.full_like(dr, 2.0))
    s = room.clamp(min=0.02).min(1, keepdim=True).values.clamp(max=1.0)
    x = _solve(fun, torch.cat([(nsig + s * CD) / unit, torch.ones_like(nrho)], 1))
    st, rho = x[:, :6] * unit, x[:, 6:] * nrho
    si = torch.func.vmap(lambda a, b_, m: slips(a, b_, m)[3])(st, rho, ms)
    return st, rho, _rotated(p, Rp, si), R
