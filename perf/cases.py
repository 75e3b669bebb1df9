"""The framework's work, as its users have it done, for timing.

Every case goes through the public Python entry points (deviceclass.Solver,
ensemble.Ensemble, indicator.DeviceMLP) or the C ABI they mirror.  A case is
a dict of plain values: "kind" names the problem family, the rest are its
sizes and switches.  `prepare` builds what a program holds before the call,
`run` is one pass, `exact` the same outputs from plain torch in 64 bits.

Kinds:
  bump      small periodic Cartesian mesh over a smooth bottom (the first
            configuration of the package's problem set), plain path
  lake      curved mesh on the unit square, walls, Gaussian bumps, lake at
            rest plus a ripple (the benchmark problem), any degree and flux
  basin     a curved mesh with a shore that wets and drains, SSP-RK3 and the
            positivity limiter
  island    a lake around a dry island: partial-dry treatment and limiter
  dam       circular dam break with artificial viscosity (modal sensor)
  tsunami   one tsunami scenario, artificial viscosity (modal sensor)
  ensemble  tsunami scenarios batched in one arena, learned indicator: add,
            advance to the horizon, read back, remove
  rhs       one right-hand side on the caller's own device buffers
  train     one snapshot's features and a few training steps of the
            troubled-cell network
"""
from __future__ import annotations

import ctypes
import functools

import numpy as np
import torch

import esdgsem_mpiocca_b200 as esdg
from esdgsem_mpiocca_b200 import host, indicator, problems
from esdgsem_mpiocca_b200.deviceclass import Solver
from esdgsem_mpiocca_b200.ensemble import Ensemble

_ON_CHIP = 32e6  # bytes of state a whole time loop can keep on the chip


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one right-hand side inside another program's step
        dict(name="rhs_24_N4", kind="rhs", N=4, nel=24, flux=0),
        # the smallest solve: 256 elements, 100 steps, launch latency counts
        dict(name="bump_16_N3", kind="bump", N=3, nel=16, flux=2, steps=100),
        # an ordinary research mesh, state handed over and read back on the host
        dict(name="lake_64_N4", kind="lake", N=4, nel=64, flux=0, steps=50, device=False),
        # the headline benchmark mesh, state kept on the device
        dict(name="lake_512_N4", kind="lake", N=4, nel=512, flux=0, steps=10, device=True),
        # the highest degree, rotated elements, rotated ES flux
        dict(name="lake_80_N7", kind="lake", N=7, nel=80, flux=3, steps=10, device=True),
        # a ragged element count (odd elements of 49 nodes)
        dict(name="lake_99_N6", kind="lake", N=6, nel=99, flux=0, steps=10, device=True),
        # wetting and draining: SSP-RK3 with the positivity limiter
        dict(name="basin_192_N2", kind="basin", N=2, nel=192, flux=3, steps=20),
        # a shelf that dries: partial-dry treatment and limiter
        dict(name="island_96_N3", kind="island", N=3, nel=96, flux=0, steps=20),
        # shock capturing at the training configuration's size
        dict(name="dam_256_N4", kind="dam", N=4, nel=256, flux=0, steps=6),
        # one request of the serving stream, solved alone
        dict(name="tsunami_128_N3", kind="tsunami", N=3, nel=128, flux=0, steps=20),
        # an ensemble batch with the learned indicator
        dict(name="ensemble_6_N3", kind="ensemble", N=3, nel=128, members=6, flux=0, steps=30),
        # training the indicator: features of a snapshot, four minibatches
        dict(name="train_N4", kind="train", N=4, nel=128, batch=16384, steps=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["bump", "lake", "lake", "lake", "basin", "island", "dam", "dam", "tsunami", "ensemble", "rhs",
                       "train"])
    flux = rng.choice([0, 2, 3])
    if kind == "bump":
        return dict(kind=kind, N=rng.randint(2, 5), nel=rng.randint(8, 40), flux=flux, steps=rng.randint(20, 120))
    if kind == "lake":
        N = rng.randint(1, 7)
        nel = _log_int(rng, 12, int(1200 / (N + 1)))
        return dict(kind=kind, N=N, nel=nel, flux=flux, steps=rng.randint(4, 20), device=rng.random() < 0.5)
    if kind == "basin":
        N = rng.randint(1, 5)
        return dict(kind=kind, N=N, nel=_log_int(rng, 12, int(700 / (N + 1))), flux=flux, steps=rng.randint(4, 24))
    if kind == "island":
        N = rng.randint(2, 5)
        return dict(kind=kind, N=N, nel=_log_int(rng, 12, int(500 / (N + 1))), flux=0, steps=rng.randint(4, 24))
    if kind == "dam":
        N = rng.randint(2, 6)
        return dict(kind=kind, N=N, nel=_log_int(rng, 12, int(1200 / (N + 1))), flux=flux, steps=rng.randint(3, 12))
    if kind == "tsunami":
        return dict(kind=kind, N=rng.randint(2, 4), nel=_log_int(rng, 24, 192), flux=0, steps=rng.randint(5, 40))
    if kind == "ensemble":
        return dict(kind=kind, N=rng.choice([3, 4]), nel=_log_int(rng, 24, 144), members=rng.randint(2, 8), flux=0,
                    steps=rng.randint(5, 40))
    if kind == "rhs":
        return dict(kind=kind, N=rng.randint(1, 7), nel=_log_int(rng, 8, 96), flux=flux)
    return dict(kind=kind, N=rng.choice([3, 4]), nel=rng.randint(64, 160), batch=rng.choice([4096, 10000, 16384]),
                steps=rng.randint(2, 6))


# ---------------------------------------------------------------------------
# Problems
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _curved_mesh(N, nel, rotate):
    return host.mesh_mapped(N, 0.0, 1.0, 0.0, 1.0, nel, nel, amp=0.03, rotate_seed=rotate)


def _pack(h, hu, hv, K):
    return np.ascontiguousarray(np.stack([a.reshape(K, -1) for a in (h, hu, hv)], axis=1)).reshape(-1)


def _problem(case, seed):
    kind, N, nel, flux = case["kind"], case["N"], case["nel"], case.get("flux", 0)
    rng = np.random.default_rng(seed)
    if kind == "bump":
        pr = problems.periodic_bump(N=N, nel=nel, NumFlux=flux)
        n2 = (N + 1) ** 2
        q = pr.q0.reshape(pr.K, 3, n2)
        cx, cy = rng.uniform(0.6, 1.4, size=2)
        r2 = ((pr.mesh.x - cx) ** 2 + (pr.mesh.y - cy) ** 2).reshape(pr.K, n2)
        q[:, 0] = 1.0 - pr.b.reshape(pr.K, n2) + rng.uniform(0.02, 0.06) * np.exp(-50.0 * r2)
        return pr
    if kind in ("tsunami", "ensemble"):
        pr = problems.tsunami_member(seed % 100000, N=N, sizes=(nel,))
        pr.params.NumFlux = flux
        return pr
    if kind in ("island", "basin"):
        p = host.Params(N=N, CFL=0.3, T=1e9, NumFlux=flux, PositivityPreserving=1, PosPresTOL=1e-3)
        if kind == "island":
            p.PartialDryTreatment = 1
            m = host.mesh_cartesian(N, 0.0, 1.0, 0.0, 1.0, nel, nel)
        else:
            p.rkOrder, p.rkSSP = 3, 1
            m = _curved_mesh(N, nel, 7)
        cx, cy = rng.uniform(0.4, 0.6, size=2)
        b = 1.4 * np.exp(-((m.x - cx) ** 2 + (m.y - cy) ** 2) / 0.18 ** 2)
        wet = np.maximum(0.0, 1.0 - b)
        ripple = 0.02 * np.exp(-((m.x - 0.85) ** 2 + (m.y - 0.2) ** 2) / 0.1 ** 2)
        h = np.where(wet > 0, wet + ripple, 0.0)
        return host.make_problem(p, m, b, _pack(h, 0 * h, 0 * h, m.K))
    m = _curved_mesh(N, nel, 7 if kind == "rhs" or N == 7 else 0)
    if kind == "dam" or kind == "train":
        p = host.Params(N=N, CFL=0.4, DFL=0.1, T=1e9, NumFlux=flux, ArtificialViscosity=1, epsilon_0=0.01,
                        sigma_min=-6.0, sigma_max=-2.0)
        r0 = rng.uniform(0.2, 0.35)
        cx, cy = rng.uniform(0.4, 0.6, size=2)
        h = np.where((m.x - cx) ** 2 + (m.y - cy) ** 2 < r0 * r0, 2.0, 1.0)
        b = np.zeros_like(h)
        return host.make_problem(p, m, b, _pack(h, 0 * h, 0 * h, m.K))
    b = problems.gaussian_bumps(m.x, m.y, seed % 100000)
    cx, cy = rng.uniform(0.25, 0.75, size=2)
    w = rng.uniform(0.03, 0.08)
    h = 1.0 - b + 0.01 * np.exp(-((m.x - cx) ** 2 + (m.y - cy) ** 2) / (w * w))
    p = host.Params(N=N, CFL=0.4, T=1e9, NumFlux=flux)
    return host.make_problem(p, m, b, _pack(h, 0 * h, 0 * h, m.K))


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.copy_(torch.from_numpy(a))
    return t.numpy()


class _DeviceArray:
    """A device buffer of an engine, for torch (__cuda_array_interface__);
    the tensor keeps this object, and this object the engine, alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 2}


def _train_set(case, seed):
    """Feature inputs of one snapshot: a dam break after its first steps, as
    far as its state goes by hand: smooth waves plus a jump."""
    pr = _problem(case, seed)
    rng = np.random.default_rng(seed + 1)
    n2 = (case["N"] + 1) ** 2
    m, q = pr.mesh, pr.q0.reshape(pr.K, 3, n2)
    x, y = m.x.reshape(pr.K, n2), m.y.reshape(pr.K, n2)
    for v, amp in ((0, 0.05), (1, 0.3), (2, 0.3)):
        for _ in range(4):
            k = rng.uniform(4.0, 60.0, size=2)
            q[:, v] += amp * rng.uniform(0.2, 1.0) * np.sin(k[0] * x + k[1] * y + rng.uniform(0, 6.28))
    q += 10.0 ** rng.uniform(-6, -2, size=(pr.K, 1, 1)) * rng.standard_normal(q.shape)
    return pr


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "rhs":
        pr = _problem(case, seed)
        m, bs = pr.mesh, pr.basis
        f64 = [pr.q0, m.Jinv, m.y_xi, m.y_eta, m.x_xi, m.x_eta, pr.Bx, pr.By, pr.b, bs.D, m.nx, m.ny, m.scal]
        i32 = [m.EdgeData, m.ElemToEdge, m.MasterSlave, m.Orientation]
        bufs = [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda() for a in f64]
        bufs += [torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda() for a in i32]
        return dict(case=case, pr=pr, bufs=bufs, out=torch.zeros(pr.q0.size, dtype=torch.float64, device="cuda"))
    if kind == "ensemble":
        sizes = [case["nel"], max(8, case["nel"] * 3 // 4), max(8, case["nel"] // 2)]
        probs = [_problem(dict(case, nel=sizes[k % 3]), seed + 17 * k) for k in range(case["members"])]
        en = Ensemble.for_problems(probs)
        en.set_indicator(2, indicator.IndicatorNet.default(case["N"]))
        return dict(case=case, probs=probs, en=en)
    if kind == "train":
        pr = _train_set(case, seed)
        net = indicator.IndicatorNet.fresh(case["N"] + 1, seed % 1000)
        mlp = indicator.DeviceMLP(net, blocks=64)
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pr.q0, pr.b, pr.basis.VdmInv)]
        X, t, _ = mlp.features(*[a.data_ptr() for a in dev], pr.K)
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        idx = torch.randint(0, pr.K, (case["steps"], case["batch"]), generator=g, device="cuda")
        return dict(case=case, K=pr.K, mlp=mlp, dev=dev, P0=mlp.P.clone(), Pb0=mlp.Pb.clone(),
                    sets=[(X[i].contiguous(), t[i].contiguous()) for i in idx])
    pr = _problem(case, seed)
    s = Solver(pr)
    st = dict(case=case, pr=pr, s=s)
    if case.get("device"):
        st["stream"] = torch.cuda.Stream()
        s.dc.set_stream(st["stream"].cuda_stream)
        st["q"] = torch.as_tensor(_DeviceArray(s.dc, s.dc.state_pointers()[0], pr.q0.size), device="cuda")
        st["q0"] = torch.from_numpy(pr.q0).cuda()
    else:
        st["q0"], st["q"] = _pinned(pr.q0), _pinned(np.zeros_like(pr.q0))
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rhs":
        p, pr, out = state["pr"].params, state["pr"], state["out"]
        rc = esdg.lib().esdg_compute_rhs_noalloc(
            p.N, pr.K, pr.F, p.NumFlux, p.ES, p.g_const, p.PosPresTOL,
            *[ctypes.c_void_p(t.data_ptr()) for t in state["bufs"]], ctypes.c_void_p(out.data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(esdg.lib().esdg_last_error(None).decode())
        return out
    if kind == "ensemble":
        en = state["en"]
        ids = [en.add(pr, T=1e9, max_steps=case["steps"]) for pr in state["probs"]]
        en.advance(case["steps"])
        got = {"q": [en.q(i) for i in ids], "t": [en.status(i)["t"] for i in ids]}
        for i in ids:
            en.remove(i)
        return got
    if kind == "train":
        mlp = state["mlp"]
        X, t, s = mlp.features(*[a.data_ptr() for a in state["dev"]], state["K"])
        # resume from the checkpoint, then one step per minibatch
        mlp.P.copy_(state["P0"])
        mlp.Pb.copy_(state["Pb0"])
        mlp.m.zero_()
        mlp.v.zero_()
        mlp.step_count = 0
        losses = [mlp.train_step(Xb, tb, 1e-3).clone() for Xb, tb in state["sets"]]
        return {"X": X, "t": t, "s": s, "loss": losses, "P": mlp.P, "G": mlp.G}
    s = state["s"]
    if case.get("device"):
        cur = torch.cuda.current_stream()
        state["stream"].wait_stream(cur)
        with torch.cuda.stream(state["stream"]):
            state["q"].copy_(state["q0"])
        t, _ = s.run(T=1e9, max_steps=case["steps"])  # returns when the loop has ended
        return {"q": state["q"], "t": t}
    s.dc.copy_q_from_host(state["q0"])
    t, _ = s.run(T=1e9, max_steps=case["steps"])
    out = {"q": s.dc.copy_q_to_host(state["q"]), "t": t}
    if state["pr"].params.ArtificialViscosity:
        out["visc"] = s.dc.copy_visc_to_host(state["pr"].K)
    return out


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def work(case):
    kind, N, nel = case["kind"], case["N"], case["nel"]
    n = N + 1
    if kind == "train":
        kp = indicator.layout(n)["kp"]
        K, M = nel * nel, case["batch"] * case["steps"]
        return {"bytes": K * (32.0 * n * n + 2 * kp + 8) + M * (2.0 * kp + 4),
                "flops": K * (4.0 * n ** 3 + 30 * n * n) + M * 6.0 * 32 * (kp + 33)}
    if kind == "ensemble":
        sizes = [nel, max(8, nel * 3 // 4), max(8, nel // 2)]
        K = sum(sizes[k % 3] ** 2 for k in range(case["members"]))
    else:
        K = nel * nel
    nodes = float(K * n * n)
    # per node and stage: 2n pair fluxes, the pointwise terms and update, and
    # the interface fluxes (2 faces of n nodes an element)
    flops = nodes * (2 * n * 32.0 + 60 + 2.0 / n * 220)
    av = kind in ("dam", "tsunami", "ensemble")
    if av:  # sensor on every element
        flops += nodes * (4.0 * n + 20)
    if kind == "rhs":
        return {"bytes": nodes * 8 * (3 + 7 + 3) + K * 2 * n * 40.0, "flops": flops}
    stages = 3 if kind == "basin" else 5
    once = nodes * 8 * (3 + 7 + 3) + K * 2 * n * 40.0
    per_stage = nodes * (168.0 + (16 if av else 0))
    total = once if nodes * 152 <= _ON_CHIP else per_stage * stages * case["steps"]
    if kind == "ensemble":
        total += nodes * 8 * 14  # the members' arrays come from the host
    return {"bytes": total, "flops": flops * stages * case["steps"]}


# ---------------------------------------------------------------------------
# exact: the scheme in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Plain:
    """The right-hand side and time steps on arrays [K][eta][xi]."""

    def __init__(self, pr):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        m, p, bs = pr.mesh, pr.params, pr.basis
        self.p, self.n, self.K, self.F = p, p.N + 1, m.K, m.F
        n = self.n
        f = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        nod = lambda a: f(a).reshape(-1, n, n)  # noqa: E731
        self.J, self.b, self.Bx, self.By = nod(m.Jinv), nod(pr.b), nod(pr.Bx), nod(pr.By)
        self.ye, self.yx, self.xe, self.xx = nod(m.y_eta), nod(m.y_xi), nod(m.x_eta), nod(m.x_xi)
        mat = lambda a: f(a).reshape(n, n)  # noqa: E731
        self.D, self.Ds, self.Dh, self.V = mat(bs.D), mat(bs.Dstrong), mat(bs.Dhat), mat(bs.VdmInv)
        self.w = f(bs.wGL)
        self.gf = 1.0 / float(bs.wGL[0])
        self.nx, self.ny, self.sc = (f(a).reshape(-1, n) for a in (m.nx, m.ny, m.scal))
        ed = f(m.EdgeData).long().reshape(-1, 8)
        self.wall = ed[:, 6] == -1
        eL, sL, same = ed[:, 0], ed[:, 2], ed[:, 4] != 0
        eR = torch.where(self.wall, eL, ed[:, 1])
        sR = torch.where(self.wall, sL, ed[:, 3])
        i = torch.arange(n, device=self.dev)
        offs = torch.stack([i, i * n + n - 1, n * n - n + i, i * n])  # trace nodes of sides 0..3
        fwd = i.expand(self.F, n)
        self.ir = torch.where(same[:, None], fwd, n - 1 - fwd)
        own = lambda e, s, k: e[:, None] * n * n + torch.gather(offs[s], 1, k)  # noqa: E731
        self.iL, self.iR, self.iRown = own(eL, sL, fwd), own(eR, sR, self.ir), own(eR, sR, fwd)
        self.eL, self.eR = eL, eR
        e2e = f(m.ElemToEdge).long().reshape(-1, 4) - 1
        orr = f(m.Orientation).long().reshape(-1, 4) != 0
        self.ms = f(m.MasterSlave).double().reshape(-1, 4)[:, :, None]
        j = i.expand(self.K, 4, n)
        self.fidx = e2e[:, :, None] * n + torch.where(orr[:, :, None], j, n - 1 - j)
        self.offs = offs
        self.es, self.minele = f(pr.EleSizes), pr.minEleSize
        self.rk = (pr.rkA, pr.rkB, pr.rkC)
        if p.PartialDryTreatment:
            self.fd = [mat(a) for a in bs.fd()]

    def lift(self, r, face, sign):
        """r += sign ms face J at the element's side nodes; face [F][n]."""
        v = sign * self.ms * face.reshape(-1)[self.fidx]
        out = torch.zeros(self.K, self.n * self.n, dtype=torch.float64, device=self.dev)
        for s in range(4):
            out[:, self.offs[s]] += v[:, s]
        return r + out.reshape(r.shape) * self.J

    def face_states(self, q):
        h, hu, hv = (a.reshape(-1) for a in q)
        L = [a[self.iL] for a in (h, hu, hv)]
        R = [a[self.iR] for a in (h, hu, hv)]
        # wall: the ghost of node ir, normal momentum reflected
        nx, ny = torch.gather(self.nx, 1, self.ir), torch.gather(self.ny, 1, self.ir)
        vn, vt = nx * R[1] + ny * R[2], -ny * R[1] + nx * R[2]
        w = self.wall[:, None]
        R = [R[0], torch.where(w, -nx * vn - ny * vt, R[1]), torch.where(w, -ny * vn + nx * vt, R[2])]
        return L, R

    def riemann(self, q):
        p, g, tol = self.p, self.p.g_const, self.p.PosPresTOL
        (hL, huL, hvL), (hR, huR, hvR) = self.face_states(q)
        bf = self.b.reshape(-1)
        bL, bR = bf[self.iL], bf[self.iR]
        nx, ny = self.nx, self.ny
        zero = torch.zeros_like(hL)

        def vel(h, hu, hv):
            wet = (h >= tol) if p.NumFlux == 0 else (h > tol)
            d = torch.where(wet, h, torch.ones_like(h))
            u, v = torch.where(wet, hu / d, zero), torch.where(wet, hv / d, zero)
            return (torch.where(wet, h, zero) if p.NumFlux == 0 else h), u, v

        hL, uL, vL = vel(hL, huL, hvL)
        hR, uR, vR = vel(hR, huR, hvR)
        n1, n2 = nx, ny
        if p.NumFlux == 3:  # in the face's own frame
            uL, vL, uR, vR = nx * uL + ny * vL, -ny * uL + nx * vL, nx * uR + ny * vR, -ny * uR + nx * vR
            n1, n2 = torch.ones_like(nx), zero
        H, H2 = 0.5 * (hL + hR), 0.5 * (hL * hL + hR * hR)
        U, V = 0.5 * (uL + uR), 0.5 * (vL + vR)
        vn = U * n1 + V * n2
        f = [H * vn, H * U * vn + 0.5 * g * H2 * n1, H * V * vn + 0.5 * g * H2 * n2]
        if p.ES:
            j1 = (g * (hR + bR) - 0.5 * (uR ** 2 + vR ** 2)) - (g * (hL + bL) - 0.5 * (uL ** 2 + vL ** 2))
            j2, j3 = uR - uL, vR - vL
            if p.NumFlux == 2:
                cl = torch.where(hL > tol, torch.sqrt(torch.clamp(g * hL, min=0)), zero)
                cr = torch.where(hR > tol, torch.sqrt(torch.clamp(g * hR, min=0)), zero)
                lam = torch.maximum(cl + torch.maximum(uL.abs(), vL.abs()), cr + torch.maximum(uR.abs(), vR.abs())) / g
                rows = ((1.0, U, V), (U, g * H + U * U, U * V), (V, U * V, g * H + V * V))
                f = [a - 0.5 * lam * (r[0] * j1 + r[1] * j2 + r[2] * j3) for a, r in zip(f, rows)]
            else:
                c = torch.sqrt((0.5 * g * (hL + hR)).abs())
                # eigenvectors as the scheme has them (the shear one unsigned)
                cols = ((1.0, U + n1 * c, V + n2 * c), (0.0, n2, n1), (1.0, U - n1 * c, V - n2 * c))
                lams = (0.5 / g * (vn + c).abs(), (H * vn).abs(), 0.5 / g * (vn - c).abs())
                for col, lm in zip(cols, lams):
                    a = lm * (col[0] * j1 + col[1] * j2 + col[2] * j3)
                    f = [x - 0.5 * cc * a for x, cc in zip(f, col)]
        if p.NumFlux == 3:
            f = [f[0], nx * f[1] - ny * f[2], ny * f[1] + nx * f[2]]
        return [self.sc * self.gf * a for a in f]

    def volume(self, q):
        g = self.p.g_const
        h, hu, hv = q
        inv = torch.where(h > 0, 1.0 / torch.where(h > 0, h, torch.ones_like(h)), torch.zeros_like(h))
        u, v = hu * inv, hv * inv
        d = [0.0, 0.0, 0.0]
        for l in range(self.n):
            for axis in (0, 1):
                at = (lambda a: a[:, :, l:l + 1]) if axis == 0 else (lambda a: a[:, l:l + 1, :])
                Dl = self.D[:, l].reshape(1, 1, -1) if axis == 0 else self.D[:, l].reshape(1, -1, 1)
                A, B = (self.ye, self.xe) if axis == 0 else (-self.yx, -self.xx)
                a, c = 0.5 * (A + at(A)), 0.5 * (B + at(B))
                hA, huA, hvA = 0.5 * (h + at(h)), 0.5 * (hu + at(hu)), 0.5 * (hv + at(hv))
                uA, vA = 0.5 * (u + at(u)), 0.5 * (v + at(v))
                pr = g * hA * hA - 0.25 * g * (h * h + at(h * h))
                d[0] = d[0] + Dl * (a * huA - c * hvA)
                d[1] = d[1] + Dl * (a * (huA * uA + pr) - c * hvA * uA)
                d[2] = d[2] + Dl * (a * huA * vA - c * (hvA * vA + pr))
        return [-self.J * d[0], -self.J * d[1] - g * h * self.Bx, -self.J * d[2] - g * h * self.By]

    def dry_volume(self, q, r):
        """The finite-difference momentum terms of partly dry elements."""
        p, g, tol, n, h = self.p, self.p.g_const, self.p.PosPresTOL, self.n, q[0]
        dry = (torch.clamp(h.reshape(self.K, -1).amin(1), max=1.0) < tol)[:, None, None]
        wet = h > tol
        Dc, Dup, Ddn = self.fd

        def diff(x, axis):
            x = x if axis == 0 else x.transpose(1, 2)
            w = wet if axis == 0 else wet.transpose(1, 2)
            wp = torch.zeros_like(w)
            wm = torch.zeros_like(w)
            wp[:, :, :-1], wm[:, :, 1:] = w[:, :, 1:], w[:, :, :-1]
            central = torch.einsum("il,kjl->kji", Dc, x)
            up, down = torch.einsum("il,kjl->kji", Dup, x), torch.einsum("il,kjl->kji", Ddn, x)
            z = torch.zeros_like(x)
            out = torch.where(wp & wm, central, torch.where(wp, up, torch.where(wm, down, z)))
            out = torch.where(w, out, z)
            return out if axis == 0 else out.transpose(1, 2)

        edge = torch.zeros(n, dtype=torch.float64, device=self.dev)
        edge[0], edge[-1] = self.gf, -self.gf
        bd = 0.5 * g * h * h
        fxb, feb = bd * edge.reshape(1, 1, -1), bd * edge.reshape(1, -1, 1)
        fx, fe, bx, be = diff(g * h, 0), diff(g * h, 1), diff(self.b, 0), diff(self.b, 1)
        ye, yx, xe, xx, J = self.ye, self.yx, self.xe, self.xx, self.J
        d2 = h * (ye * fx - yx * fe) + ye * fxb - yx * feb
        d3 = h * (-xe * fx + xx * fe) - xe * fxb + xx * feb
        r1 = -J * d2 - g * J * h * (ye * bx - yx * be)
        r2 = -J * d3 - g * J * h * (-xe * bx + xx * be)
        return [r[0], torch.where(dry, r1, r[1]), torch.where(dry, r2, r[2])]

    def viscosity(self, q):
        p, N = self.p, self.n - 1
        m = self.b + q[0]
        w = torch.einsum("il,kjl,mj->kim", self.V, m, self.V) ** 2
        n1, n2 = w.sum((1, 2)), w[:, :N, :N].sum((1, 2))
        z1 = n1 - n2 if N < 1 else w[:, N, :].sum(1) + w[:, :N, N].sum(1)
        z2 = w[:, N - 1, :N].sum(1) + w[:, :N - 1, N - 1].sum(1)
        tiny = n1 < 1e-5
        ratio = torch.where(tiny, torch.zeros_like(n1), torch.maximum(z1 / n1, z2 / n2))
        s = torch.log10(ratio)
        lo, hi = p.sigma_min, p.sigma_max
        ramp = p.epsilon_0 * 0.5 * (1.0 + torch.sin(np.pi * (s - 0.5 * (hi + lo)) / (hi - lo)))
        z = torch.zeros_like(s)
        return torch.where(lo >= s, z, torch.where(hi >= s, ramp, z + p.epsilon_0))

    def viscous(self, q, r, eps):
        p, tol, J = self.p, self.p.PosPresTOL, self.J
        h = q[0]
        wet = h > tol
        d = torch.where(wet, h, torch.ones_like(h))
        vel = [torch.where(wet, a / d, torch.zeros_like(a)) for a in q[1:]]
        grads = []
        for w in vel:
            wxi = torch.einsum("il,kjl->kji", self.Dh, w)
            weta = torch.einsum("jl,kli->kji", self.Dh, w)
            flat = w.reshape(-1)
            # walls: the own trace; else the right trace in its own order
            wR = torch.where(self.wall[:, None], flat[self.iL], flat[self.iRown])
            avg = self.sc * self.gf * 0.5 * (flat[self.iL] + wR)
            gx = self.lift(J * (self.ye * wxi - self.yx * weta), self.nx * avg, 1.0)
            gy = self.lift(J * (-self.xe * wxi + self.xx * weta), self.ny * avg, 1.0)
            grads.append((h * gx, h * gy))
        vm = torch.maximum(eps[self.eL], eps[self.eR])[:, None]
        e = eps[:, None, None]
        out = [r[0]]
        for ri, (gx, gy) in zip(r[1:], grads):
            a, c = gx.reshape(-1), gy.reshape(-1)
            fl = 0.5 * vm * (self.nx * (a[self.iL] + a[self.iR]) + self.ny * (c[self.iL] + c[self.iR]))
            fl = torch.where(self.wall[:, None], torch.zeros_like(fl), fl)
            F, G = self.ye * e * gx - self.xe * e * gy, -self.yx * e * gx + self.xx * e * gy
            ri = ri + J * (torch.einsum("il,kjl->kji", self.Ds, F) + torch.einsum("jl,kli->kji", self.Ds, G))
            out.append(self.lift(ri, self.sc * self.gf * fl, 1.0))
        return out

    def rhs(self, q, eps=None):
        r = self.volume(q)
        if self.p.PartialDryTreatment:
            r = self.dry_volume(q, r)
        r = [self.lift(a, f, -1.0) for a, f in zip(r, self.riemann(q))]
        return r if eps is None else self.viscous(q, r, eps)

    def limit(self, q):
        tol = self.p.PosPresTOL
        h, hu, hv = q
        w = self.w[None, :, None] * self.w[None, None, :] / self.J
        mean = [(a * w).sum((1, 2), keepdim=True) / self.es[:, None, None] for a in q]
        ha = torch.where(mean[0].abs() < 1e-5, torch.zeros_like(mean[0]), mean[0])
        hmin = torch.clamp(h.amin((1, 2), keepdim=True), max=0.0)
        th = torch.clamp(ha / torch.where(ha == hmin, torch.ones_like(ha), ha - hmin), max=1.0)
        th = torch.where(ha == hmin, torch.ones_like(th), th)
        z = torch.zeros_like(h)
        hn = torch.where(ha > 0, (th * (h - ha) + ha).abs(), z)
        mom = [torch.where((ha > 0) & (hn > tol), th * (a - b) + b, z) for a, b in zip((hu, hv), mean[1:])]
        bad = hmin < 0
        shallow = h < tol
        return [torch.where(bad, hn, h)] + [torch.where(bad, m, torch.where(shallow, z, a))
                                            for m, a in zip(mom, (hu, hv))]

    def speed(self, q):
        h, hu, hv = q
        wet = h > self.p.PosPresTOL
        d = torch.where(wet, h, torch.ones_like(h))
        z = torch.zeros_like(h)
        return float((torch.sqrt(self.p.g_const * h) + torch.maximum(torch.where(wet, hu / d, z).abs(),
                                                                      torch.where(wet, hv / d, z).abs())).max())

    def loop(self, q0, steps):
        p, n = self.p, self.n
        A, B, C = self.rk
        q = list(torch.as_tensor(q0, device=self.dev).reshape(self.K, 3, n, n).clone().unbind(1))
        t, eps = 0.0, None
        for _ in range(steps):
            dt = self.minele / n * p.CFL / self.speed(q)
            if p.ArtificialViscosity:
                eps = self.viscosity(q)
                vmax = float(eps.max())
                if vmax > 0:
                    dt = min(dt, p.DFL / n ** 2 * self.minele ** 2 / vmax)
            start = q
            k = [torch.zeros_like(a) for a in q]
            for s in range(len(A)):
                if p.ArtificialViscosity and s > 0:
                    eps = self.viscosity(q)
                r = self.rhs(q, eps)
                if p.rkSSP:
                    q = [A[s] * a + B[s] * b + C[s] * dt * c for a, b, c in zip(start, q, r)]
                else:
                    k = [A[s] * a + b for a, b in zip(k, r)]
                    q = [a + C[s] * dt * b for a, b in zip(q, k)]
                if p.PositivityPreserving:
                    q = self.limit(q)
            t += dt
        return torch.stack(q, 1).reshape(-1), t, eps


def _exact_train(case, seed):
    pr = _train_set(case, seed)
    n, N = case["N"] + 1, case["N"]
    n2, L = n * n, indicator.layout(case["N"] + 1)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    q = torch.as_tensor(pr.q0, device=dev).reshape(pr.K, 3, n2)
    b, V = torch.as_tensor(pr.b, device=dev).reshape(pr.K, n2), torch.as_tensor(pr.basis.VdmInv, device=dev)
    V = V.reshape(n, n)
    fields = [q[:, 0] + b, q[:, 1], q[:, 2]]
    X = torch.zeros(pr.K, L["kp"], dtype=torch.float64, device=dev)
    s_eta = None
    for f, v in enumerate(fields):
        mean = v.mean(1, keepdim=True)
        rms = ((v - mean) ** 2).mean(1, keepdim=True).sqrt()
        X[:, f * n2:(f + 1) * n2] = (v - mean) / rms
        sf = torch.clamp(torch.log10(rms ** 2 / (mean ** 2 + rms ** 2)), min=-12.0)[:, 0]
        X[:, 3 * n2 + f] = 0.25 * sf
        s_eta = sf if f == 0 else s_eta
    w = torch.einsum("il,kjl,mj->kim", V, fields[0].reshape(pr.K, n, n), V) ** 2
    t1 = (w[:, N, :].sum(1) + w[:, :N, N].sum(1)) / w.sum((1, 2))
    t2 = (w[:, N - 1, :N].sum(1) + w[:, :N - 1, N - 1].sum(1)) / w[:, :N, :N].sum((1, 2))
    t = torch.clamp(torch.log10(torch.maximum(t1, t2)), -12.0, 0.0) - s_eta
    out = {"X": X, "t": t, "s": s_eta}
    if dev.type != "cuda":  # the minibatches are drawn on the GPU
        return dict(out, loss=[None] * case["steps"], P=None, G=None)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    idx = torch.randint(0, pr.K, (case["steps"], case["batch"]), generator=g, device="cuda")
    P0 = torch.as_tensor(indicator.IndicatorNet.fresh(n, seed % 1000).P, device=dev).double()
    P, m, v = P0.clone(), torch.zeros_like(P0), torch.zeros_like(P0)
    H, losses, G = 32, [], None
    pos = torch.arange(P.numel(), device=dev)
    live = ~(((pos < L["b1"]) & (pos % L["kp"] >= 3 * n2 + 3)) | (pos > L["b3"]))
    for k, i in enumerate(idx):
        W = P.clone().requires_grad_()
        Z = X[i] @ W[:L["b1"]].reshape(H, -1).T + W[L["b1"]:L["w2"]]
        Z = torch.relu(Z) @ W[L["w2"]:L["b2"]].reshape(H, H).T + W[L["b2"]:L["w3"]]
        y = torch.relu(Z) @ W[L["w3"]:L["b3"]] + W[L["b3"]]
        e2 = ((y - t[i]) ** 2).sum()
        G, = torch.autograd.grad(e2 / len(i), W)
        losses.append(e2.detach())
        m, v = 0.9 * m + 0.1 * G, 0.999 * v + 0.001 * G * G
        upd = 1e-3 * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
        P = torch.where(live, P - upd, P)
    G = G.clone()
    G[L["b3"] + 1] = losses[-1]  # the engine keeps the squared error beside the gradient
    return dict(out, loss=losses, P=P, G=G)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":  # the network's decisions have no exact counterpart
        return None
    if kind == "train":
        return _exact_train(case, seed)
    pr = _problem(case, seed)
    plain = _Plain(pr)
    if kind == "rhs":
        q = list(torch.as_tensor(pr.q0, device=plain.dev).reshape(plain.K, 3, plain.n, plain.n).unbind(1))
        return torch.stack(plain.rhs(q), 1).reshape(-1)
    q, t, eps = plain.loop(pr.q0, case["steps"])
    return {"q": q, "t": t} if eps is None or case.get("device") else {"q": q, "t": t, "visc": eps}
