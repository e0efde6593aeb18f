"""The work that users of the solver have it do, as cases that can be timed and compared.

Each case is one call sequence of the public Python API on a synthetic scene of
nelson_b200.problems: whole LevenbergMarquardt solves with the parameters going
in and coming out of host arrays (the call a user makes), one step of a
caller's own loop, a batch of small problems, the gradient of a converged
solution, SE(2) scan alignment, and a system that the caller assembled.

Results of the mixed handles are kept in float32, as a program that chose that
precision keeps them: their Hessian, reduced system and factor are FP32.
`exact` restates the same mathematics in plain torch, in 64 bits.
"""
import math
import random

import numpy as np
import torch

from nelson_b200 import native as N
from nelson_b200 import problems as P

PREC = {"fp64": N.PREC_FP64, "mixed": N.PREC_MIXED}
KIND = {"dense": N.SOLVER_DENSE, "envelope": N.SOLVER_ENVELOPE}


def _ring(name, cams, pts, bc, kmin, kmax, weights, precision, solver, its):
    return dict(name=name, kind="lm", scene="ring", cams=cams, pts=pts, bc=bc, kmin=kmin, kmax=kmax, weights=weights,
                precision=precision, solver=solver, order="", its=its)


def _grid(name, gx, gy, pts, kmin, kmax, precision, solver, order, its, kind="lm"):
    return dict(name=name, kind=kind, scene="grid", gx=gx, gy=gy, cams=gx * gy, pts=pts, bc=9, kmin=kmin, kmax=kmax,
                weights=False, precision=precision, solver=solver, order=order, its=its)


def listed():
    return [
        # a sliding window of a tracker: 20 cameras, 500 points, one tile of the
        # reduced system; latency and launches are all there is
        _ring("window_20", 20, 500, 6, 3, 8, False, "fp64", "dense", 5),
        # a local map with per-observation weights
        _ring("local_64", 64, 5000, 6, 3, 8, True, "mixed", "dense", 6),
        # an object scan, 9-parameter cameras, all cameras connected
        _ring("scan_200_mixed", 200, 50000, 9, 3, 12, False, "mixed", "dense", 10),
        # the same solve where the caller wants FP64 throughout
        _ring("scan_200_fp64", 200, 50000, 9, 3, 12, False, "fp64", "dense", 10),
        # an aerial block with neighbour visibility: envelope solver on the RCM order
        _grid("aerial_432_env", 16, 27, 150000, 2, 12, "mixed", "envelope", "rcm", 6),
        # the large aerial block, dense reduced system of 13,500 rows
        _grid("aerial_1500", 30, 50, 500000, 2, 12, "mixed", "dense", "", 3),
        # one iteration of a caller's own loop over update / computeIncrement /
        # oplus, FP64, ragged sizes (391 cameras: 27.5 tiles of 128 rows)
        _grid("step_391_fp64", 17, 23, 100003, 2, 9, "fp64", "dense", "", 1, kind="step"),
        # many uneven small problems at once, in one persistent launch
        dict(name="batch_128", kind="batch", problems=128, cam_lo=8, cam_hi=64, pt_lo=200, pt_hi=4000, its=6),
        # the backward direction: gradient of a loss on the converged points
        # with respect to observations and weights
        dict(name="adjoint_64", kind="adjoint", cams=64, pts=5000, kmin=3, kmax=8),
        # a long 2D pose graph with loop closures
        dict(name="pose_graph_2000", kind="pose", scene="graph", poses=2000, pts=500, closures=3000, span=30,
             precision="mixed", solver="envelope", order="rcm", its=5),
        # a handful of dense 2D scans, every pair joined
        dict(name="scans_15", kind="pose", scene="full", poses=15, pts=3000, closures=0, span=0, precision="fp64",
             solver="dense", order="amd", its=5),
        # a Hessian that the caller's own code assembled on the host, with
        # camera-camera blocks in U
        dict(name="system_300", kind="system", nu=300, nv=20000, bu=6, kmin=2, kmax=8, band=3, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ring", "ring", "grid", "grid", "step", "batch", "adjoint", "graph", "full", "system"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "ring":
        cams = _log(rng, 12, 300)
        c = _ring("", cams, _log(rng, 15 * cams, 250 * cams), rng.choice([6, 9]), 3, rng.randint(6, min(12, cams)),
                  rng.random() < 0.3, prec, "dense", rng.randint(3, 8))
    elif kind in ("grid", "step"):
        gx, gy = _log(rng, 4, 24), _log(rng, 6, 40)
        step = kind == "step"
        c = _grid("", gx, gy, int(gx * gy * rng.uniform(100, 330)) + rng.randint(0, 9), 2, rng.randint(6, 12), prec,
                  rng.choice(["dense", "envelope"]), rng.choice(["", "rcm", "amd"]), 1 if step else rng.randint(2, 6),
                  "step" if step else "lm")
    elif kind == "batch":
        lo = rng.randint(8, 24)
        c = dict(kind="batch", problems=_log(rng, 8, 128), cam_lo=lo, cam_hi=rng.randint(lo + 1, 64),
                 pt_lo=200, pt_hi=_log(rng, 400, 4000), its=rng.randint(3, 6))
    elif kind == "adjoint":
        cams = _log(rng, 16, 90)
        c = dict(kind="adjoint", cams=cams, pts=_log(rng, 20 * cams, 70 * cams), kmin=3, kmax=rng.randint(6, 9))
    elif kind == "graph":
        n = _log(rng, 100, 2500)
        c = dict(kind="pose", scene="graph", poses=n, pts=_log(rng, 60, 500), closures=int(1.5 * n),
                 span=rng.randint(5, 40), precision=prec, solver=rng.choice(["dense", "envelope"]),
                 order=rng.choice(["", "rcm", "amd"]), its=rng.randint(2, 5))
    elif kind == "full":
        c = dict(kind="pose", scene="full", poses=rng.randint(4, 24), pts=_log(rng, 100, 3000), closures=0, span=0,
                 precision=prec, solver="dense", order=rng.choice(["", "amd"]), its=rng.randint(3, 6))
    else:
        nu = _log(rng, 10, 500)
        c = dict(kind="system", nu=nu, nv=_log(rng, 10 * nu, 80 * nu), bu=rng.choice([3, 6, 9]), kmin=2,
                 kmax=rng.randint(4, 8), band=rng.randint(0, 5), precision=prec)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# Scenes: every array comes from the seed; the numbers of problems, cameras,
# points and (for gradients per edge) edges come from the case alone.
def _scene(case, seed):
    if case["kind"] == "adjoint":
        p = P.ring_scene(case["cams"], case["pts"], case["kmin"], case["kmax"], 6, 1234, weights=True)
        r = np.random.default_rng(seed)
        p.obs = P.project(p.cams_true, p.pts_true, p.cam_idx, p.pt_idx, 6) + r.normal(size=p.obs.shape)
        p.weight = r.uniform(0.5, 2.0, p.ne)
        p.pts = p.pts_true + 0.05 * r.normal(size=p.pts.shape)
        return P.with_fixed_nodes(p, 2)
    if case["scene"] == "ring":
        return P.ring_scene(case["cams"], case["pts"], case["kmin"], case["kmax"], case["bc"], seed,
                            weights=case["weights"])
    return P.grid_scene(case["gx"], case["gy"], case["pts"], case["kmin"], case["kmax"], seed)


def _batch_scenes(case, seed):
    size, r = random.Random(case["problems"]), random.Random(seed)
    return [P.ring_scene(size.randint(case["cam_lo"], case["cam_hi"]), size.randint(case["pt_lo"], case["pt_hi"]), 3, 8,
                         6, r.randrange(1 << 30)) for _ in range(case["problems"])]


def _pose_scene(case, seed):
    if case["scene"] == "graph":
        return P.pose_graph_scene(case["poses"], case["pts"], case["closures"], case["span"], seed=seed)
    return P.scan_align_scene(case["poses"], case["pts"], seed=seed)


def _system(case, seed):
    """Blocks of J'J of random edges: U-V observations, U-U edges within `band` and priors."""
    r = np.random.default_rng(seed)
    nu, nv, bu = case["nu"], case["nv"], case["bu"]
    k = np.minimum(r.integers(case["kmin"], case["kmax"] + 1, nv), nu)
    first = r.integers(0, nu, nv)
    v = np.repeat(np.arange(nv), k)
    u = (first[v] + 3 * (np.arange(v.size) - np.repeat(np.cumsum(k) - k, k))) % nu
    o = np.lexsort((v, u))
    u, v = u[o], v[o]
    keep = np.r_[True, (np.diff(u) != 0) | (np.diff(v) != 0)]
    u, v = u[keep], v[keep]
    a, b = r.normal(size=(u.size, 2, bu)), r.normal(size=(u.size, 2, 3))
    res = r.normal(size=(u.size, 2))
    W = np.einsum("eki,ekj->eij", a, b)
    V = np.zeros((nv, 3, 3))
    np.add.at(V, v, np.einsum("eki,ekj->eij", b, b))
    bV = np.zeros((nv, 3))
    np.add.at(bV, v, np.einsum("eki,ek->ei", b, res))
    D = np.zeros((nu, bu, bu))
    np.add.at(D, u, np.einsum("eki,ekj->eij", a, a))
    bU = np.zeros((nu, bu))
    np.add.at(bU, u, np.einsum("eki,ek->ei", a, res))
    rc, blocks = [], []
    for j in range(nu):  # column by column, rows ascending, the diagonal last
        for i in range(max(0, j - case["band"]), j):
            m = r.normal(size=(bu, bu))
            rc.append((i, j))
            blocks.append(-m)
            D[i] += np.eye(bu)
            D[j] += m.T @ m
        rc.append((j, j))
        blocks.append(None)
    for q, (i, j) in enumerate(rc):
        if i == j:
            blocks[q] = D[j] + np.eye(bu)
    return dict(u_rc=np.array(rc, np.int32), v_rc=np.stack([np.arange(nv)] * 2, 1).astype(np.int32),
                w_rc=np.stack([u, v], 1).astype(np.int32), U=np.array(blocks), V=V + 0.1 * np.eye(3), W=W,
                bU=bU.reshape(-1), bV=bV.reshape(-1))


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("lm", "step"):
        p = _scene(case, seed)
        g = N.BAProblemGPU.from_ba(p, precision=PREC[case["precision"]], perm=case["order"] or None)
        g.set_solver_kind(KIND[case["solver"]])
        return dict(case=case, g=g, cams=p.cams, pts=p.pts, settings=N.LMSettings(maxNumIt=case["its"]))
    if kind == "batch":
        ps = _batch_scenes(case, seed)
        gs = [N.BAProblemGPU.from_ba(p) for p in ps]
        return dict(case=case, gs=gs, b=N.PersistentBatch(gs), start=[(p.cams, p.pts) for p in ps],
                    settings=N.LMSettings(maxNumIt=case["its"]))
    if kind == "adjoint":
        p = _scene(case, seed)
        g = N.BAProblemGPU.from_ba(p)
        g.lm_solve(N.LMSettings(maxNumIt=20))
        g.gn_solve(N.GNSettings(maxNumIt=8, epsIncSquare=1e-26))  # to rounding: LM's acceptance test stops short of it
        return dict(case=case, g=g, dL=g.get_params()[1] - p.pts_true)
    if kind == "pose":
        p = _pose_scene(case, seed)
        g = N.Pose2DGPU.from_scan_align(p, precision=PREC[case["precision"]], order=case["order"] or "natural")
        g.set_solver_kind(KIND[case["solver"]])
        return dict(case=case, g=g, poses=p.poses0, settings=N.LMSettings(maxNumIt=case["its"]))
    s = _system(case, seed)
    g = N.SchurSolverGPU(case["bu"], case["nu"], case["nv"], s["u_rc"], s["v_rc"], s["w_rc"],
                         precision=PREC[case["precision"]])
    return dict(case=case, g=g, s=s)


def _kept(case, *arrays):
    """The results as the caller's program keeps them (see the module's text)."""
    f = np.float32 if case.get("precision") == "mixed" else np.float64
    return [np.asarray(a, f) for a in arrays]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lm":
        g = state["g"]
        g.set_params(state["cams"], state["pts"])
        _, trace, its, _ = g.lm_solve(state["settings"])
        cams, pts = g.get_params()
        return _kept(case, cams, pts, trace[:, 2], trace[:, 3]) + [its]
    if kind == "step":
        g = state["g"]
        g.set_params(state["cams"], state["pts"])
        chi2 = g.update(True)
        mu = 1e-3 * g.max_abs_hdiag()
        ok = g.compute_increment(0.0, mu)
        du, dv = g.increment()
        g.backup()
        g.oplus()
        after = g.update(False)
        return _kept(case, [chi2, mu, after], du, dv) + [int(ok)]
    if kind == "batch":
        for g, (cams, pts) in zip(state["gs"], state["start"]):
            g.set_params(cams, pts)
        _, chi2, its, _, _, _ = state["b"].lm_solve(state["settings"])
        out = [g.get_params() for g in state["gs"]]
        return [np.concatenate([c for c, _ in out]), np.concatenate([p for _, p in out]), chi2, its]
    if kind == "adjoint":
        g_obs, g_w, rep = state["g"].adjoint(dL_dpts=state["dL"], sweeps=3)
        return [g_obs, g_w, int(rep["ok"])]
    if kind == "pose":
        g = state["g"]
        g.set_poses(state["poses"])
        _, trace, its = g.lm_solve(state["settings"])
        return _kept(case, g.get_poses(), trace[:, 2], trace[:, 3]) + [its]
    g, s = state["g"], state["s"]
    g.set_hessian(s["U"], s["V"], s["W"], s["bU"], s["bV"])
    ok, du, dv = g.compute_increment(0.0, 0.05)
    return _kept(case, du, dv) + [int(ok)]


# ---------------------------------------------------------------------------
def _solve_work(n, edges, pairs, bc, np_, prec, solver_rows=None):
    """(bytes, flops) of one computeIncrement with its evaluation: W once out and once in, S and its factor
    once each, observations and points once; S's products, the factorisation and the two solves."""
    t = 4 if prec == "mixed" else 8
    band = n if solver_rows is None else min(n, solver_rows)
    nbytes = edges * (2 * bc * 3 * t + 40) + np_ * (24 + 9 * t) + 2 * n * band * t / (2 if band == n else 1)
    flops = edges * (4 * bc * bc + 60 * bc) + pairs * bc * bc * 6 + (n ** 3 / 3 if band == n else n * band * band) + 4 * n * band
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind in ("lm", "step"):
        lo, hi = case["kmin"], min(case["kmax"], case["cams"])
        ks = range(lo, hi + 1)
        e1, p1 = sum(ks) / len(ks), sum(k * (k + 1) / 2 for k in ks) / len(ks)
        n = case["cams"] * case["bc"]
        rows = None
        if case["solver"] == "envelope" and case["scene"] == "grid":
            rows = (4 * min(case["gx"], case["gy"]) + 5) * case["bc"]
        b, f = _solve_work(n, case["pts"] * e1, case["pts"] * p1, case["bc"], case["pts"], case["precision"], rows)
        return {"bytes": case["its"] * b + 48 * case["pts"], "flops": case["its"] * f}
    if kind == "batch":
        nc, npt = (case["cam_lo"] + case["cam_hi"]) / 2, (case["pt_lo"] + case["pt_hi"]) / 2
        nc3 = (case["cam_lo"] ** 3 + case["cam_hi"] ** 3) / 2
        _, f = _solve_work(6 * nc, npt * 5.5, npt * 18, 6, npt, "fp64")
        f += 6 ** 3 * (nc3 - nc ** 3) / 3
        return {"bytes": case["problems"] * (npt * 5.5 * 40 + npt * 48), "flops": case["problems"] * case["its"] * f}
    if kind == "adjoint":
        n, e = 6 * (case["cams"] - 2), case["pts"] * (case["kmin"] + case["kmax"]) / 2
        _, f = _solve_work(n, e, 3.3 * e, 6, case["pts"], "fp64")
        return {"bytes": e * (40 + 24) + 48 * case["pts"], "flops": f + 4 * e * 800}
    if kind == "pose":
        n = 3 * case["poses"]
        full = case["scene"] == "full"
        edges = case["poses"] * (case["poses"] + 1) / 2 if full else case["poses"] + case["closures"]
        band = n if full else min(n, 3 * 2 * case["span"])
        f = edges * case["pts"] * 60 + n * band * band + 4 * n * band
        return {"bytes": case["its"] * edges * case["pts"] * 48.0, "flops": case["its"] * f}
    e = case["nv"] * (case["kmin"] + case["kmax"]) / 2
    n, bu = case["nu"] * case["bu"], case["bu"]
    b, f = _solve_work(n, e, 3 * e, bu, case["nv"], case["precision"])
    return {"bytes": b + e * bu * 24 + case["nv"] * 120, "flops": f}


# ---------------------------------------------------------------------------
# The same mathematics in 64 bits.
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=_dev())


def _skew(w):
    z = torch.zeros_like(w[..., 0])
    return torch.stack([torch.stack([z, -w[..., 2], w[..., 1]], -1), torch.stack([w[..., 2], z, -w[..., 0]], -1),
                        torch.stack([-w[..., 1], w[..., 0], z], -1)], -2)


class _Ba:
    """Cameras (R, t, f, k1, k2) and points with the residuals, Jacobians and the damped solve."""

    def __init__(self, p):
        self.bc, self.ncv, self.npv = p.bc, p.nc_var, p.np_var
        cams = _t(p.cams)
        self.R = torch.matrix_exp(_skew(cams[:, :3]))
        self.t = cams[:, 3:6].clone()
        n = cams.shape[0]
        self.k = cams[:, 6:9].clone() if p.bc == 9 else _t([[p.f, 0.0, 0.0]]).repeat(n, 1)
        self.X = _t(p.pts).clone()
        self.c0 = _t([p.cx, p.cy])
        cam = np.asarray(p.cam_idx, np.int64)
        if p.cam_fixed is not None:
            cam = np.where(p.cam_fixed == 1, cam + p.nc_var, cam)
        pt = np.asarray(p.pt_idx, np.int64)
        self.order = np.lexsort((cam, pt))
        self.cam = torch.as_tensor(cam[self.order], device=_dev())
        self.pt = torch.as_tensor(pt[self.order], device=_dev())
        self.z = _t(p.obs[self.order])
        self.w = _t(np.ones(p.ne) if p.weight is None else p.weight[self.order])

    def residual(self):
        a = (self.R[self.cam] @ self.X[self.pt][..., None])[..., 0]
        q = a + self.t[self.cam]
        xy = q[:, :2] / q[:, 2:]
        k = self.k[self.cam]
        r2 = (xy * xy).sum(1)
        d = 1 + r2 * (k[:, 1] + k[:, 2] * r2)
        return (k[:, 0] * d)[:, None] * xy + self.c0 - self.z, a, q, xy, k, r2, d

    def chi2(self):
        r = self.residual()[0]
        return float((self.w * (r * r).sum(1)).sum())

    def jacobians(self):
        r, a, q, xy, k, r2, d = self.residual()
        g = 2 * (k[:, 1] + 2 * k[:, 2] * r2)
        e = torch.eye(2, dtype=r.dtype, device=r.device)
        m = k[:, :1, None] * (d[:, None, None] * e + g[:, None, None] * xy[:, :, None] * xy[:, None, :])
        m = torch.cat([m, -(m @ xy[..., None])], 2) / q[:, 2, None, None]
        jp = m @ self.R[self.cam]
        jc = [m @ -_skew(a), m]
        if self.bc == 9:
            f = k[:, 0]
            jc.append(torch.stack([d[:, None] * xy, (f * r2)[:, None] * xy, (f * r2 * r2)[:, None] * xy], 2))
        return r, torch.cat(jc, 2), jp

    def linearise(self):
        r, jc, jp = self.jacobians()
        n, bc, wr = self.R.shape[0], self.bc, self.w[:, None] * r
        wjc, wjp = self.w[:, None, None] * jc, self.w[:, None, None] * jp
        z = lambda *s: torch.zeros(s, dtype=r.dtype, device=r.device)  # noqa: E731
        self.U = z(n, bc, bc).index_add_(0, self.cam, wjc.transpose(1, 2) @ jc)
        self.V = z(self.npv, 3, 3).index_add_(0, self.pt, wjp.transpose(1, 2) @ jp)
        self.W = wjc.transpose(1, 2) @ jp
        self.bU = z(n, bc).index_add_(0, self.cam, (jc.transpose(1, 2) @ wr[..., None])[..., 0])
        self.bV = z(self.npv, 3).index_add_(0, self.pt, (jp.transpose(1, 2) @ wr[..., None])[..., 0])
        return float((wr * r).sum())

    def hdiag(self):
        d = torch.cat([self.U[:self.ncv].diagonal(dim1=1, dim2=2).reshape(-1), self.V.diagonal(dim1=1, dim2=2).reshape(-1)])
        return float(d.abs().max())

    def increment(self, mu):
        n, bc = self.R.shape[0], self.bc
        Vi = torch.linalg.inv(self.V + mu * torch.eye(3, dtype=self.V.dtype, device=self.V.device))
        du, dv = _schur_solve(self.U, None, Vi, self.W, self.cam, self.pt, self.bU, self.bV, n, bc, self.ncv, mu)
        return du, dv

    def apply(self, du, dv):
        n = self.ncv
        d = du.view(n, self.bc)
        self.R = torch.cat([torch.matrix_exp(_skew(d[:, :3])) @ self.R[:n], self.R[n:]])
        self.t = torch.cat([self.t[:n] + d[:, 3:6], self.t[n:]])
        if self.bc == 9:
            self.k = torch.cat([self.k[:n] + d[:, 6:9], self.k[n:]])
        self.X = self.X + dv

    def state(self):
        return self.R, self.t, self.k, self.X

    def restore(self, s):
        self.R, self.t, self.k, self.X = s

    def cams(self):
        tr = self.R.diagonal(dim1=1, dim2=2).sum(1)
        v = torch.stack([self.R[:, 2, 1] - self.R[:, 1, 2], self.R[:, 0, 2] - self.R[:, 2, 0],
                         self.R[:, 1, 0] - self.R[:, 0, 1]], 1)
        th = torch.atan2(0.5 * v.norm(dim=1), 0.5 * (tr - 1))
        w = torch.where(th[:, None] > 1e-6, v * (th / (2 * torch.sin(th).clamp_min(1e-300)))[:, None], 0.5 * v)
        parts = [w, self.t] + ([self.k] if self.bc == 9 else [])
        return torch.cat(parts, 1).cpu().numpy()


def _schur_solve(U, Uoff, Vi, W, cam, pt, bU, bV, n, bc, ncv, mu):
    """-(H + mu I)^-1 b for H = [U W; W' V]; rows sorted by point, `Uoff` = (i, j, blocks) above the diagonal."""
    S = torch.zeros((n * n, bc * bc), dtype=U.dtype, device=U.device)
    Y = W @ Vi[pt]
    at = torch.arange(n, device=U.device)
    eye = torch.eye(bc, dtype=U.dtype, device=U.device)
    S.index_add_(0, at * n + at, (U + mu * eye).reshape(n, -1))
    if Uoff is not None and Uoff[0].numel():
        S.index_add_(0, Uoff[0] * n + Uoff[1], Uoff[2].reshape(-1, bc * bc))
        S.index_add_(0, Uoff[1] * n + Uoff[0], Uoff[2].transpose(1, 2).reshape(-1, bc * bc))
    m = pt.numel()
    for d in range(m):
        e = torch.nonzero(pt[: m - d] == pt[d:])[:, 0] if d else torch.arange(m, device=U.device)
        if not e.numel():
            break
        blk = Y[e] @ W[e + d].transpose(1, 2)
        S.index_add_(0, cam[e] * n + cam[e + d], blk.reshape(-1, bc * bc), alpha=-1)
        if d:
            S.index_add_(0, cam[e + d] * n + cam[e], blk.transpose(1, 2).reshape(-1, bc * bc), alpha=-1)
    S = S.view(n, n, bc, bc).permute(0, 2, 1, 3)[:ncv, :, :ncv].reshape(ncv * bc, ncv * bc)
    bS = -bU.clone()
    bS.index_add_(0, cam, (Y @ bV[pt][..., None])[..., 0])
    du = torch.cholesky_solve(bS[:ncv].reshape(-1, 1), torch.linalg.cholesky(S))[:, 0]
    full = torch.cat([du.view(ncv, bc), torch.zeros((n - ncv, bc), dtype=U.dtype, device=U.device)])
    t = -bV.clone()
    t.index_add_(0, pt, (W.transpose(1, 2) @ full[cam][..., None])[..., 0], alpha=-1)
    return du, (Vi @ t[..., None])[..., 0]


def _lm(prob, its, linearise, hdiag, increment, apply, chi2_of, grad):
    """LevenbergMarquardt with the default settings: costs and dampings as the trace has them."""
    chi2 = linearise()
    costs, mus = [chi2], [0.0]
    mu, v, it = 1e-3 * hdiag(), 2.0, 0
    while it < its:
        sub = 0
        while True:
            du, dv = increment(mu)
            d, b = torch.cat([du.reshape(-1), dv.reshape(-1)]), grad()
            if float(d @ d) <= 1e-30:
                return costs, mus, it
            keep = prob.state()
            apply(du, dv)
            new = chi2_of()
            rho = (chi2 - new) / float(d @ (mu * d - b))
            costs.append(new)
            mus.append(mu)
            if rho > 0:
                if it > 0 and new < 1e-15:
                    return costs, mus, it
                mu *= max(1 / 3, min(2 / 3, 1 - (2 * rho - 1) ** 3))
                v = 2.0
                break
            prob.restore(keep)
            mu *= v
            v *= 2
            sub += 1
            if sub >= 10:
                return costs, mus, it
        chi2 = linearise()
        it += 1
    return costs, mus, it


def _ba_lm(b, its):
    grad = lambda: torch.cat([b.bU[:b.ncv].reshape(-1), b.bV.reshape(-1)])  # noqa: E731
    return _lm(b, its, b.linearise, b.hdiag, b.increment, b.apply, b.chi2, grad)


class _Poses:
    def __init__(self, p):
        self.n = len(p.poses0)
        self.p0 = _t(p.poses_true[:1])
        self.p = _t(p.poses0)
        e = np.array(p.edges)
        self.i, self.j = (torch.as_tensor(e[:, k], device=_dev()) for k in (0, 1))
        self.s, self.nm = _t(np.stack(p.scans)), _t(np.stack(p.normals))

    def state(self):
        return self.p

    def restore(self, s):
        self.p = s

    @staticmethod
    def _turn(th, x):
        c, s = torch.cos(th)[:, None], torch.sin(th)[:, None]
        return torch.stack([c * x[..., 0] - s * x[..., 1], s * x[..., 0] + c * x[..., 1]], -1)

    def edges(self):
        q = torch.cat([self.p0, self.p])
        a, b = q[self.i], q[self.j]
        nn = self._turn(a[:, 2], self.nm[self.i])
        xt = self._turn(b[:, 2], self.s[self.j]) + b[:, None, :2]
        err = ((self._turn(a[:, 2], self.s[self.i]) + a[:, None, :2] - xt) * nn).sum(-1)
        return err, nn, xt

    def chi2(self):
        return float(self.edges()[0].square().sum())

    def linearise(self):
        err, nn, xt = self.edges()
        g = torch.stack([nn[..., 0], nn[..., 1], xt[..., 0] * nn[..., 1] - xt[..., 1] * nn[..., 0]], -1)
        h, b = g.transpose(1, 2) @ g, (g.transpose(1, 2) @ err[..., None])[..., 0]
        m = self.n + 1
        H = torch.zeros((m * m, 9), dtype=h.dtype, device=h.device)
        for x, y, s in ((self.i, self.i, 1), (self.j, self.j, 1), (self.i, self.j, -1), (self.j, self.i, -1)):
            H.index_add_(0, x * m + y, h.reshape(-1, 9), alpha=s)
        self.H = H.view(m, m, 3, 3).permute(0, 2, 1, 3).reshape(3 * m, 3 * m)[3:, 3:].contiguous()
        v = torch.zeros((m, 3), dtype=h.dtype, device=h.device)
        self.b = (v.index_add_(0, self.i, b).index_add_(0, self.j, b, alpha=-1))[1:].reshape(-1)
        return float(err.square().sum())

    def increment(self, mu):
        A = self.H + mu * torch.eye(self.H.shape[0], dtype=self.H.dtype, device=self.H.device)
        return torch.cholesky_solve(-self.b[:, None], torch.linalg.cholesky(A))[:, 0], self.b[:0]

    def apply(self, d, _):
        d = d.view(-1, 3)
        w = d[:, 2]
        small = w.abs() < 1e-9
        ws = torch.where(small, torch.ones_like(w), w)
        a = torch.where(small, 1 - w * w / 6, torch.sin(ws) / ws)
        b = torch.where(small, w / 2, (1 - torch.cos(ws)) / ws)
        t = self._turn(w, self.p[:, None, :2])[:, 0]
        self.p = torch.stack([t[:, 0] + a * d[:, 0] - b * d[:, 1], t[:, 1] + b * d[:, 0] + a * d[:, 1],
                              self.p[:, 2] + w], 1)


def _edge_cost(d, x, R, t, f, c0, z, w):
    """w |r|^2 / 2 of one edge at camera tangent d (left update) and point x + d[6:]."""
    K = _skew(d[:3])
    q = (torch.eye(3, dtype=d.dtype, device=d.device) + K + 0.5 * K @ K) @ (R @ (x + d[6:9])) + t + d[3:6]
    r = f * q[:2] / q[2] + c0 - z
    return 0.5 * w * (r * r).sum()


def _adjoint(p):
    b = _Ba(p)
    _ba_lm(b, 40)
    n, ncv = b.R.shape[0], b.ncv
    d0 = torch.zeros(9, dtype=torch.float64, device=_dev())
    f = lambda d, x, R, t, ff, z, w: _edge_cost(d, x, R, t, ff, b.c0, z, w)  # noqa: E731
    grad = torch.func.grad(f)
    idx = torch.cat([b.cam[:, None] * 6 + torch.arange(6, device=_dev()),
                     n * 6 + b.pt[:, None] * 3 + torch.arange(3, device=_dev())], 1)
    keep = torch.cat([torch.arange(6 * ncv, device=_dev()), torch.arange(6 * n, 6 * n + 3 * b.npv, device=_dev())])
    m = 6 * n + 3 * b.npv
    for last in (False, False, True):  # two Newton steps to the exact stationary point, then its Hessian
        args = (b.X[b.pt], b.R[b.cam], b.t[b.cam], b.k[b.cam][:, 0], b.z, b.w)
        h = torch.func.vmap(torch.func.jacfwd(grad), in_dims=(None,) + (0,) * 6)(d0, *args)
        H = torch.zeros(m * m, dtype=torch.float64, device=_dev())
        H.index_add_(0, (idx[:, :, None] * m + idx[:, None, :]).reshape(-1), h.reshape(-1))
        H = H.view(m, m)[keep][:, keep]
        if last:
            break
        g = torch.func.vmap(grad, in_dims=(None,) + (0,) * 6)(d0, *args)
        v = torch.zeros(m, dtype=torch.float64, device=_dev()).index_add_(0, idx.reshape(-1), g.reshape(-1))[keep]
        s = torch.linalg.solve(H, -v)
        b.apply(s[:6 * ncv], s[6 * ncv:].view(-1, 3))
    dL = torch.cat([torch.zeros(6 * ncv, dtype=torch.float64, device=_dev()), (b.X - _t(p.pts_true)).reshape(-1)])
    mu = torch.zeros(m, dtype=torch.float64, device=_dev())
    mu[keep] = torch.linalg.solve(H, dL)
    r, jc, jp = b.jacobians()
    s = (jc @ mu[idx[:, :6]][..., None] + jp @ mu[idx[:, 6:]][..., None])[..., 0]
    back = np.argsort(b.order)
    return [(b.w[:, None] * s).cpu().numpy()[back], -(s * r).sum(1).cpu().numpy()[back], None]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lm", "step"):
        b = _Ba(_scene(case, seed))
        if kind == "lm":
            costs, mus, _ = _ba_lm(b, case["its"])
            return [b.cams(), b.X.cpu().numpy(), np.array(costs), np.array(mus), None]
        chi2 = b.linearise()
        mu = 1e-3 * b.hdiag()
        du, dv = b.increment(mu)
        if case["order"]:  # the increment comes in the solver's camera order
            g = N.rcm_order if case["order"] == "rcm" else N.amd_order_camera_graph
            p = _scene(case, seed)
            perm = g(case["cams"], case["pts"], p.cam_idx, p.pt_idx)
            du_out = torch.empty_like(du).view(-1, 9)
            du_out[torch.as_tensor(perm.astype(np.int64), device=du.device)] = du.view(-1, 9)
        else:
            du_out = du
        b.apply(du, dv)
        return [np.array([chi2, mu, b.chi2()]), du_out.cpu().numpy().reshape(-1), dv.cpu().numpy().reshape(-1), None]
    if kind == "batch":
        cams, pts, chi2 = [], [], []
        for p in _batch_scenes(case, seed):
            b = _Ba(p)
            costs, _, _ = _ba_lm(b, case["its"])
            cams.append(b.cams())
            pts.append(b.X.cpu().numpy())
            chi2.append(b.chi2())
        return [np.concatenate(cams), np.concatenate(pts), np.array(chi2), None]
    if kind == "adjoint":
        return _adjoint(_scene(case, seed))
    if kind == "pose":
        q = _Poses(_pose_scene(case, seed))
        costs, mus, _ = _lm(q, case["its"], q.linearise, lambda: float(q.H.diagonal().abs().max()), q.increment,
                            q.apply, q.chi2, lambda: q.b)
        return [q.p.cpu().numpy(), np.array(costs), np.array(mus), None]
    s = _system(case, seed)
    o = np.lexsort((s["w_rc"][:, 0], s["w_rc"][:, 1]))
    cam, pt = (torch.as_tensor(s["w_rc"][o, k].astype(np.int64), device=_dev()) for k in (0, 1))
    rc, mu = s["u_rc"], 0.05
    dg = rc[:, 0] == rc[:, 1]
    i, j = (torch.as_tensor(rc[~dg, k].astype(np.int64), device=_dev()) for k in (0, 1))
    U, nu, bu = _t(s["U"]), case["nu"], case["bu"]
    dgt = torch.as_tensor(dg, device=_dev())
    Vi = torch.linalg.inv(_t(s["V"]) + mu * torch.eye(3, dtype=torch.float64, device=_dev()))
    du, dv = _schur_solve(U[dgt], (i, j, U[~dgt]), Vi, _t(s["W"][o]), cam, pt, _t(s["bU"]).view(nu, bu),
                          _t(s["bV"]).view(-1, 3), nu, bu, nu, mu)
    return [du.cpu().numpy(), dv.cpu().numpy().reshape(-1), None]
