"""The work that a user of this framework has it do, as cases to be measured.

A case is one pass through the public API (the binding of the C ABI, host
arrays in and out): an LM run on a problem that the program keeps, a whole call
that creates the problem, optimises, reads back and releases it, a batch of
local windows, or the covariance of a solution.  The scenes and their sizes are
those of the benchmark workloads and of the tests (circle, sphere, loop,
windows, the EUCM ring); the seed of `prepare` is the scene's seed.

`exact` restates the same optimisation in 64 bits with plain torch (dense
reduced system, no code of this repository beyond the scene generator)."""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "sophus_rs_gb300" not in sys.modules:
        d = os.path.join(ROOT, "sophus-rs_gb300")
        spec = importlib.util.spec_from_file_location("sophus_rs_gb300", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        m = importlib.util.module_from_spec(spec)
        sys.modules["sophus_rs_gb300"] = m
        spec.loader.exec_module(m)
    return sys.modules["sophus_rs_gb300"]


# ------------------------------------------------------------------ cases ----
def listed():
    return [
        # a tracker's local map: the smallest call there is, 10 cameras, all latency
        dict(name="circle10", kind="circle", cams=10, points=500, iters=10),
        # the reference's own benchmark problem: EUCM camera, its params free,
        # the whole call (create, 20 iterations, read back, release)
        dict(name="ring10_call", kind="ring", cams=10, points=500, iters=20, free=True),
        # a mapping server's batch of local windows of uneven size, kept and re-optimised
        dict(name="windows128", kind="windows", count=128, sizes=1, iters=10, call=False),
        # the same from a front end that makes new windows for each call
        dict(name="windows24_call", kind="windows", count=24, sizes=2, iters=10, call=True),
        # photo collection around an object: dense reduced system, FP32 linearisation
        dict(name="sphere100", kind="sphere", cams=100, points=20000, iters=8),
        # the same with the iterative solver of the reduced system (block-Jacobi PCG)
        dict(name="sphere121_pcg", kind="pcg", cams=121, points=12007, iters=6),
        # a video sequence that closes a loop: small, the headline size, and twice that
        dict(name="loop300", kind="loop", cams=300, points=60000, iters=8),
        dict(name="loop1500", kind="loop", cams=1500, points=300000, iters=5),
        dict(name="loop3000", kind="loop", cams=3000, points=600000, iters=2),
        # the sequence with odometry: pose-graph edges along it, priors on two poses
        dict(name="graph151", kind="graph", cams=151, points=15013, iters=6),
        # uncertainty of a solution: covariance blocks of every pose and of some points
        dict(name="cov_loop300", kind="cov", scene="loop", cams=300, points=60000),
        dict(name="cov_sphere40", kind="cov", scene="sphere", cams=40, points=5001),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circle", "ring", "windows", "sphere", "pcg", "loop", "loop", "graph", "cov"])
    if kind == "circle":
        return dict(kind=kind, cams=rng.randint(5, 40), points=_log_int(rng, 200, 4000), iters=rng.randint(4, 10))
    if kind == "ring":
        return dict(kind=kind, cams=rng.randint(4, 18), points=_log_int(rng, 100, 1500), iters=rng.randint(5, 20),
                    free=rng.random() < 0.7)
    if kind == "windows":
        call = rng.random() < 0.4
        return dict(kind=kind, count=_log_int(rng, 6, 40 if call else 110), sizes=rng.randint(3, 9999),
                    iters=rng.randint(4, 10), call=call)
    if kind == "sphere":
        return dict(kind=kind, cams=rng.randint(25, 140), points=_log_int(rng, 1500, 20000), iters=rng.randint(3, 8))
    if kind == "pcg":
        return dict(kind=kind, cams=rng.randint(50, 140), points=_log_int(rng, 3000, 20000), iters=rng.randint(3, 6))
    if kind == "loop":
        cams = _log_int(rng, 60, 2600)
        return dict(kind=kind, cams=cams, points=cams * rng.randint(80, 200) + rng.randint(0, 99),
                    iters=rng.randint(2, 5) if cams < 1500 else 2)
    if kind == "graph":
        cams = _log_int(rng, 70, 400)
        return dict(kind=kind, cams=cams, points=cams * rng.randint(60, 150) + rng.randint(0, 99),
                    iters=rng.randint(3, 6))
    scene = rng.choice(["loop", "sphere"])
    cams = _log_int(rng, 60, 300) if scene == "loop" else rng.randint(20, 90)
    return dict(kind=kind, scene=scene, cams=cams, points=cams * rng.randint(80, 200) + rng.randint(0, 99))


# ----------------------------------------------------------------- inputs ----
def _rel_pose(tm, tn, noise):
    """exp(noise) composed with the pose of n in m's frame (first order is enough: it is a measurement)."""
    qm, qn = tm[:4], tn[:4]
    S = _package().synth
    inv = qm * np.array([1.0, -1.0, -1.0, -1.0])
    rel = np.concatenate([S._quat_mul(inv, qn), S._quat_rot(inv) @ (tn[4:] - tm[4:])])
    return S._se3_exp_left(noise, rel)


def _scene(case, seed):
    """Host arrays of one problem, from the seed alone."""
    S = _package().synth
    kind = case.get("scene", case["kind"])
    if kind == "circle":
        return S.generate(S.CIRCLE, case["cams"], case["points"], seed=seed)
    if kind == "ring":
        return S.ring_box_eucm(case["cams"], case["points"], seed=seed, intrinsics_free=case["free"])
    if kind in ("sphere", "pcg"):
        prob = S.generate(S.SPHERE, case["cams"], case["points"], seed=seed)
    else:
        prob = S.generate(S.LOOP, case["cams"], case["points"], seed=seed)
    if case["kind"] == "cov":  # at a solution, the scale held by a second fixed pose
        prob.poses, prob.points = prob.poses_true.copy(), prob.points_true.copy()
        prob.pose_const[:2] = 1
    if case["kind"] == "graph":
        rng = np.random.default_rng(seed)
        n, T = prob.n_cam, prob.poses_true
        prob.edge_pose = np.array([(j, (j + 1) % n) for j in range(n)], np.int32)
        prob.edge_mn = np.array([_rel_pose(T[m], T[k], 0.002 * rng.standard_normal(6)) for m, k in prob.edge_pose])
        prob.prior_pose = np.array([0, n // 2], np.int32)
        prob.prior_mean = T[prob.prior_pose].copy()
        prob.prior_precision = np.array([1e4 * np.eye(6)] * 2)
        prob.pose_const = np.zeros(n, np.uint8)
    return prob


def _window_scenes(case, seed):
    """Windows of 5 to 40 cameras and 200 to 4000 points: the sizes are the case's, the scenes the seed's."""
    S = _package().synth
    sizes = np.random.default_rng(case["sizes"])
    shapes = [(int(sizes.integers(5, 41)), int(sizes.integers(200, 4001))) for _ in range(case["count"])]
    return [S.generate(S.WINDOW, n, m, seed=1000003 * int(seed) + i) for i, (n, m) in enumerate(shapes)]


def _params(case, damping):
    pkg = _package()
    return pkg.OptParams(num_iterations=case["iters"], initial_lm_damping=damping, function_tolerance=0.0,
                         gradient_tolerance=0.0, parameter_tolerance=0.0, max_consecutive_rejects=1 << 40)


def _queries(prob):
    """Every free pose with itself and with the next one, and points spread over the scene."""
    free = [j for j in range(prob.n_cam) if not prob.pose_const[j]]
    pts = sorted({int(k) for k in np.linspace(0, prob.n_pt - 1, 128)})
    pose, point = 1, 2
    return ([((pose, j), (pose, j)) for j in free], [((pose, a), (pose, b)) for a, b in zip(free, free[1:])],
            [((point, k), (point, k)) for k in pts], [((pose, free[len(free) // 2]), (point, k)) for k in pts])


def prepare(case, seed):
    native = _package().native
    if case["kind"] == "windows":
        scenes = _window_scenes(case, seed)
        state = dict(case=case, scenes=scenes, params=_params(case, scenes[0].initial_lm_damping))
        if not case["call"]:
            state["problems"] = native.create_problems(scenes)
        return state
    prob = _scene(case, seed)
    if case["kind"] == "cov":
        return dict(case=case, problem=native.Problem(prob, device=0), queries=_queries(prob))
    state = dict(case=case, scene=prob, params=_params(case, prob.initial_lm_damping))
    if case["kind"] != "ring":
        p = native.Problem(prob, device=0)
        if case["kind"] == "graph":
            p.set_pose_priors(prob.prior_pose, prob.prior_mean, prob.prior_precision)
        if case["kind"] == "pcg":
            p.set_linear_solver(native.LINSOLVE_PCG_BLOCK_JACOBI)
        state["problem"] = p
    return state


# -------------------------------------------------------------------- run ----
def run(state):
    native = _package().native
    case = state["case"]
    if case["kind"] == "cov":
        p = state["problem"]
        p.covariance_prepare()
        return [np.stack(p.covariance_blocks(q)) for q in state["queries"]]
    if case["kind"] == "windows":
        scenes = state["scenes"]
        problems = native.create_problems(scenes) if case["call"] else state["problems"]
        if not case["call"]:
            for p, s in zip(problems, scenes):
                p.set_variables(s.poses, s.points)
        results = native.batch_optimize(problems, state["params"])
        variables = [p.variables() for p in problems]
        if case["call"]:
            for p in problems:
                p.close()
        return dict(poses=np.concatenate([v[0] for v in variables]), points=np.concatenate([v[1] for v in variables]),
                    costs=np.array([[r.merit for r in recs] for recs, *_ in results]))
    scene = state["scene"]
    if case["kind"] == "ring":
        with native.Problem(scene, device=0) as p:
            recs, _ = p.optimize(state["params"])
            poses, points = p.variables()
            out = dict(poses=poses, points=points, costs=np.array([r.merit for r in recs]))
            if case["free"]:
                out["camera"] = p.intrinsics()
        return out
    p = state["problem"]
    p.set_variables(scene.poses, scene.points)
    recs, _ = p.optimize(state["params"])
    poses, points = p.variables()
    return dict(poses=poses, points=points, costs=np.array([r.merit for r in recs]))


# ------------------------------------------------------------------- work ----
def _track():
    """Mean of L and of L (L + 1) / 2 over the loop's tracks: L geometric(0.12) clipped to [3, 25]."""
    p, m1, m2 = 0.12, 0.0, 0.0
    for k in range(1, 400):
        w, length = p * (1 - p) ** (k - 1), min(25, max(3, k))
        m1 += w * length
        m2 += w * length * (length + 1) / 2
    return m1, m2


def _one(kind, cams, points, iters):
    """Bytes and flops of an LM run: each iteration reads the observations (pixel
    pair, two indices) and the variables and writes the variables; its
    operations are the Jacobians and their products (about 350 per
    observation), the Schur products (216 per pair of a point's observations
    in S, 36 more per observation for Z) and the factorisation and the
    solution of the reduced system (dense, or the band of the longest track)."""
    if kind in ("loop", "graph"):
        length, pairs = _track()
        band = 150
        factor = 6 * cams * float(band) ** 2 + 8 * 6 * cams * band
    else:
        length = min(25.0, 0.9 * cams) if kind in ("sphere", "pcg") else float(cams)
        pairs = length * (length + 1) / 2
        factor = (6.0 * cams) ** 3 / 3 + 4 * (6.0 * cams) ** 2
    obs = length * points
    return {"bytes": iters * (24.0 * obs + 48.0 * points + 112.0 * cams),
            "flops": iters * (386.0 * obs + 216.0 * pairs * points + factor)}


def work(case):
    if case["kind"] == "windows":  # cameras uniform in [5, 40], points uniform in [200, 4000]
        mean = {"bytes": 0.0, "flops": 0.0}
        for cams in range(5, 41):
            for k, v in _one("circle", cams, 2100, case["iters"]).items():
                mean[k] += case["count"] * v / 36
        return mean
    if case["kind"] == "cov":  # H and S once, then the factor and the inverse of S
        w = _one(case["scene"], case["cams"], case["points"], 1)
        n = 6.0 * case["cams"]
        return {"bytes": w["bytes"] + 16 * n * n, "flops": w["flops"] + n ** 3}
    return _one(case["kind"], case["cams"], case["points"], case["iters"])


# --------------------------------------------------- 64-bit plain solution ----
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_device())


def _hat(w):
    z = torch.zeros_like(w[..., 0])
    return torch.stack([torch.stack([z, -w[..., 2], w[..., 1]], -1), torch.stack([w[..., 2], z, -w[..., 0]], -1),
                        torch.stack([-w[..., 1], w[..., 0], z], -1)], -2)


def _rot(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)], -1),
        torch.stack([2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)], -1),
        torch.stack([2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1)], -2)


def _qmul(a, b):
    aw, av, bw, bv = a[..., :1], a[..., 1:], b[..., :1], b[..., 1:]
    return torch.cat([aw * bw - (av * bv).sum(-1, keepdim=True), aw * bv + bw * av + torch.linalg.cross(av, bv)], -1)


def _mul(a, b):
    return torch.cat([_qmul(a[..., :4], b[..., :4]), (_rot(a[..., :4]) @ b[..., 4:, None])[..., 0] + a[..., 4:]], -1)


def _inv(a):
    q = torch.cat([a[..., :1], -a[..., 1:4]], -1)
    return torch.cat([q, -(_rot(q) @ a[..., 4:, None])[..., 0]], -1)


def _exp(xi):
    """SE(3) exponential of [omega; nu]; series below 1e-4 rad (error below 1e-17)."""
    w, v = xi[..., :3], xi[..., 3:]
    t2 = (w * w).sum(-1, keepdim=True)
    small = t2 < 1e-8
    s2 = torch.where(small, torch.ones_like(t2), t2)
    t = s2.sqrt()
    half = torch.where(small, 0.5 - t2 / 48 + t2 * t2 / 3840, torch.sin(0.5 * t) / t)
    cosh = torch.where(small, 1 - t2 / 8 + t2 * t2 / 384, torch.cos(0.5 * t))
    a = torch.where(small, 0.5 - t2 / 24 + t2 * t2 / 720, (1 - torch.cos(t)) / s2)[..., None]
    b = torch.where(small, 1 / 6 - t2 / 120 + t2 * t2 / 5040, (t - torch.sin(t)) / (s2 * t))[..., None]
    h = _hat(w)
    V = torch.eye(3, dtype=xi.dtype, device=xi.device) + a * h + b * (h @ h)
    return torch.cat([cosh, half * w, (V @ v[..., None])[..., 0]], -1)


def _log(a):
    """SE(3) logarithm."""
    q = torch.where(a[..., :1] < 0, -a[..., :4], a[..., :4])
    v = q[..., 1:]
    n2 = (v * v).sum(-1, keepdim=True)
    small = n2 < 1e-8
    n = torch.where(small, torch.ones_like(n2), n2).sqrt()
    r = n2 / (q[..., :1] ** 2)
    f = torch.where(small, 2 / q[..., :1] * (1 - r / 3 + r * r / 5), 2 * torch.atan2(n, q[..., :1]) / n)
    w = f * v
    t2 = (w * w).sum(-1, keepdim=True)
    tiny = t2 < 1e-4
    t = torch.where(tiny, torch.ones_like(t2), t2).sqrt()
    c = torch.where(tiny, 1 / 12 + t2 / 720 + t2 * t2 / 30240,
                    (1 - 0.5 * t * torch.cos(0.5 * t) / torch.sin(0.5 * t)) / torch.where(tiny, torch.ones_like(t2), t2))
    h = _hat(w)
    Vi = torch.eye(3, dtype=a.dtype, device=a.device) - 0.5 * h + c[..., None] * (h @ h)
    return torch.cat([w, (Vi @ a[..., 4:, None])[..., 0]], -1)


class _Exact:
    """The Schur-complement LM loop in 64 bits on dense torch matrices."""

    def __init__(self, prob):
        self.poses, self.points = _t(prob.poses), _t(prob.points)
        self.oc, self.op, self.uv = _t(prob.obs_cam, torch.long), _t(prob.obs_pt, torch.long), _t(prob.obs_uv)
        self.cam = _t(prob.intrinsics)
        self.eucm = prob.camera_model == 1
        if self.eucm:
            self.cam = torch.cat([self.cam, _t(prob.eucm_alpha_beta)])
        self.nk = len(self.cam) if prob.intrinsics_free else 0
        self.delta = prob.huber_delta
        const = _t(prob.pose_const, torch.bool)
        self.free = torch.nonzero(~const)[:, 0]
        self.nf = len(self.free)
        self.block = torch.full((prob.n_cam,), -1, dtype=torch.long, device=_device())
        self.block[self.free] = torch.arange(self.nf, device=_device())
        # one observation per (point, pose) in these scenes: a reduced term each
        self.cnt_f = torch.bincount(self.oc, minlength=prob.n_cam).double()[self.free]
        self.cnt_m = torch.bincount(self.op, minlength=prob.n_pt).double()
        self.edges = getattr(prob, "edge_pose", None)
        self.gauge = None
        if self.edges is not None:
            self.em, self.en = _t(prob.edge_pose[:, 0], torch.long), _t(prob.edge_pose[:, 1], torch.long)
            self.emn = _t(prob.edge_mn)
            self.pp, self.pE, self.pW = _t(prob.prior_pose, torch.long), _t(prob.prior_mean), _t(prob.prior_precision)
            self.cnt_f += torch.bincount(torch.cat([self.em, self.en]), minlength=prob.n_cam).double()
            self.cnt_f[self.pp] += 1
        elif int(const.sum()) == 1:
            self.gauge = int(torch.nonzero(const)[0])
        # points in the order of the first camera that sees them, in chunks: few cameras each
        order = torch.argsort(self.op, stable=True)
        self.oc, self.op, self.uv = self.oc[order], self.op[order], self.uv[order]
        start = torch.cumsum(torch.cat([torch.zeros(1, device=_device()), self.cnt_m[:-1]]), 0).long()
        rank = torch.argsort(torch.argsort(self.oc[start.clamp(max=len(self.oc) - 1)], stable=True))
        order = torch.argsort(rank[self.op], stable=True)
        self.oc, self.op, self.uv = self.oc[order], self.op[order], self.uv[order]
        step, key = 4000, rank[self.op]
        cuts = torch.searchsorted(key, torch.arange(0, prob.n_pt + step, step, device=_device()))
        self.chunks = [(int(a), int(b)) for a, b in zip(cuts[:-1], cuts[1:]) if b > a]
        self.rank = rank

    # residuals (and what the Jacobians need) of the observations a..b
    def _project(self, poses, points, cam, a, b):
        cw = _inv(poses)
        R = _rot(cw[:, :4])[self.oc[a:b]]
        x = (R @ points[self.op[a:b], :, None])[..., 0] + cw[self.oc[a:b], 4:]
        u, v = x[:, 0] / x[:, 2], x[:, 1] / x[:, 2]
        if self.eucm:
            rho = (cam[5] * (u * u + v * v) + 1).sqrt()
            norm = cam[4] * rho + (1 - cam[4])
        else:
            rho = norm = torch.ones_like(u)
        pix = torch.stack([u / norm * cam[0] + cam[2], v / norm * cam[1] + cam[3]], -1)
        return self.uv[a:b] - pix, R, x, u, v, rho, norm

    def _weight(self, r):
        if not self.delta > 0:
            return torch.ones_like(r[:, 0])
        n = r.norm(dim=1)
        c = torch.where(n <= self.delta, n * n, 2 * self.delta * n - self.delta ** 2)
        return torch.where(n > 0, c.sqrt() / torch.where(n > 0, n, torch.ones_like(n)), torch.zeros_like(n))

    def _edge_res(self, poses):
        return _log(_mul(_mul(_inv(poses[self.em]), poses[self.en]), _inv(self.emn)))

    def _prior_res(self, poses):
        return _log(_mul(poses[self.pp], _inv(self.pE)))

    def cost(self, poses, points, cam):
        total = torch.zeros((), dtype=torch.float64, device=_device())
        for a, b in self.chunks:
            r = self._project(poses, points, cam, a, b)[0]
            total = total + (self._weight(r)[:, None] * r).square().sum()
        if self.edges is not None:
            g = self._prior_res(poses)
            total = total + self._edge_res(poses).square().sum() + torch.einsum("ki,kij,kj->", g, self.pW, g)
        return float(total)

    def _jacobians(self, a, b):
        r, R, x, u, v, rho, norm = self._project(self.poses, self.points, self.cam, a, b)
        k, z = self.cam, x[:, 2]
        o = torch.zeros_like(u)
        if self.eucm:
            dx, dy = k[4] * k[5] * u / rho, k[4] * k[5] * v / rho
            n2 = norm * norm
            M = torch.stack([torch.stack([(norm - u * dx) / n2, -u * dy / n2], -1),
                             torch.stack([-v * dx / n2, (norm - v * dy) / n2], -1)], -2)
        else:
            M = torch.eye(2, dtype=u.dtype, device=u.device).expand(len(u), 2, 2)
        P = torch.stack([torch.stack([1 / z, o, -u / z], -1), torch.stack([o, 1 / z, -v / z], -1)], -2)
        D = torch.diag(k[:2]) @ M @ P @ R
        p = self.points[self.op[a:b]]
        Jf, Jm = torch.cat([D @ _hat(-p), D], -1), -D
        Jc = None
        if self.nk:
            one = torch.ones_like(u)
            cols = [torch.stack([-u / norm, o], -1), torch.stack([o, -v / norm], -1), torch.stack([-one, o], -1),
                    torch.stack([o, -one], -1)]
            if self.eucm:
                n2, da, db = norm * norm, rho - 1, k[4] * (u * u + v * v) / (2 * rho)
                cols += [torch.stack([k[0] * u * d / n2, k[1] * v * d / n2], -1) for d in (da, db)]
            Jc = torch.stack(cols, -1)
        return self._weight(r)[:, None] * r, Jf, Jm, Jc

    def system(self, nu, keep):
        """S (free poses, then the camera params), its right-hand side, and per chunk what the points need."""
        n, nk = 6 * self.nf + self.nk, self.nk
        S = torch.zeros((n, n), dtype=torch.float64, device=_device())
        grad_f = torch.zeros(n, dtype=torch.float64, device=_device())
        rhs = torch.zeros(n, dtype=torch.float64, device=_device())
        diag = torch.cat([self.cnt_f.repeat_interleave(6), torch.full((nk,), float(len(self.oc)), device=_device())])
        S.diagonal().add_(nu * diag)
        kept = []
        for i, (a, b) in enumerate(self.chunks):
            r, Jf, Jm, Jc = self._jacobians(a, b)
            pts, local = torch.unique(self.op[a:b], return_inverse=True)
            m = len(pts)
            fb = self.block[self.oc[a:b]]
            on = fb >= 0
            fbs, row = torch.unique(fb[on], return_inverse=True)
            nl = 6 * len(fbs) + nk
            V = torch.zeros((m, 3, 3), dtype=torch.float64, device=_device()).index_add_(0, local, Jm.mT @ Jm)
            V.diagonal(dim1=1, dim2=2).add_(nu * self.cnt_m[pts, None])
            gm = torch.zeros((m, 3), dtype=torch.float64, device=_device())
            gm.index_add_(0, local, -(Jm.mT @ r[..., None])[..., 0])
            W = torch.zeros((m, nl, 3), dtype=torch.float64, device=_device())
            six = torch.arange(6, device=_device())
            rows = 6 * row[:, None] + six
            W[local[on, None], rows] = Jf[on].mT @ Jm[on]
            U = torch.zeros((nl, nl), dtype=torch.float64, device=_device())
            blocks = torch.zeros((len(fbs), 6, 6), dtype=torch.float64, device=_device())
            blocks.index_add_(0, row, Jf[on].mT @ Jf[on])
            at = 6 * torch.arange(len(fbs), device=_device())[:, None] + six
            U[at[:, :, None], at[:, None, :]] = blocks
            g = torch.zeros(nl, dtype=torch.float64, device=_device())
            g.index_add_(0, rows.reshape(-1), -(Jf[on].mT @ r[on, :, None]).reshape(-1))
            if nk:
                W[:, nl - nk:] = torch.zeros((m, nk, 3), dtype=torch.float64, device=_device()).index_add_(0, local, Jc.mT @ Jm)
                fc = torch.zeros((len(fbs), 6, nk), dtype=torch.float64, device=_device())
                fc.index_add_(0, row, Jf[on].mT @ Jc[on])
                U[:nl - nk, nl - nk:] = fc.reshape(-1, nk)
                U[nl - nk:, :nl - nk] = fc.reshape(-1, nk).T
                U[nl - nk:, nl - nk:] = (Jc.mT @ Jc).sum(0)
                g[nl - nk:] = -(Jc.mT @ r[..., None]).sum(0)[:, 0]
            Vi = torch.linalg.inv(V)
            flat = lambda X: X.transpose(0, 1).reshape(nl, 3 * m)  # noqa: E731
            Y = W @ Vi
            to = torch.cat([(6 * fbs[:, None] + six).reshape(-1), 6 * self.nf + torch.arange(nk, device=_device())])
            S[to[:, None], to[None, :]] += U - flat(Y) @ flat(W).T
            grad_f[to] += g
            rhs[to] += g - torch.einsum("mij,mj->i", Y, gm)
            if keep:
                kept.append((pts, to, W if keep == "all" else None, Vi, gm, (a, b), local, on, rows))
        if self.edges is not None:
            self._pose_costs(S, grad_f, rhs)
        return S, grad_f, rhs, kept, diag

    def _pose_costs(self, S, grad, rhs):
        x0 = torch.zeros(6, dtype=torch.float64, device=_device())
        jac = torch.func.vmap(torch.func.jacfwd(lambda x, l, r: _log(_mul(_mul(l, _exp(x)), r))), in_dims=(None, 0, 0))
        six = torch.arange(6, device=_device())
        Dn = jac(x0, _inv(self.poses[self.em]), _mul(self.poses[self.en], _inv(self.emn)))
        g = self._edge_res(self.poses)
        for A, sa, pa in ((-Dn, -1, self.em), (Dn, 1, self.en)):
            ra = 6 * self.block[pa][:, None] + six
            v = -(A.mT @ g[..., None]).reshape(-1)
            grad.index_add_(0, ra.reshape(-1), v)
            rhs.index_add_(0, ra.reshape(-1), v)
            for B, pb in ((-Dn, self.em), (Dn, self.en)):
                rb = 6 * self.block[pb][:, None] + six
                S.index_put_((ra[:, :, None].expand(-1, 6, 6), rb[:, None, :].expand(-1, 6, 6)), A.mT @ B, accumulate=True)
        one = torch.zeros((len(self.pp), 7), dtype=torch.float64, device=_device())
        one[:, 0] = 1
        Jp = jac(x0, one, _mul(self.poses[self.pp], _inv(self.pE)))
        g = self._prior_res(self.poses)
        ra = 6 * self.block[self.pp][:, None] + six
        v = -(Jp.mT @ self.pW @ g[..., None]).reshape(-1)
        grad.index_add_(0, ra.reshape(-1), v)
        rhs.index_add_(0, ra.reshape(-1), v)
        S.index_put_((ra[:, :, None].expand(-1, 6, 6), ra[:, None, :].expand(-1, 6, 6)), Jp.mT @ self.pW @ Jp, accumulate=True)

    def _solve(self, S, rhs):
        """Cholesky of the Jacobi-scaled system and two steps of refinement; None where S is not positive."""
        d = S.diagonal().rsqrt()
        C = d[:, None] * S * d[None, :]
        L, info = torch.linalg.cholesky_ex(C)
        if int(info):
            return None
        b = (d * rhs)[:, None]
        y = torch.cholesky_solve(b, L)
        for _ in range(2):
            y = y + torch.cholesky_solve(b - C @ y, L)
        return d * y[:, 0]

    def step(self, nu, merit):
        S, grad_f, rhs, kept, diag = self.system(nu, "some")
        xf = self._solve(S, rhs)
        del S
        if xf is None:
            return merit, 2 * nu, False
        dm = torch.zeros_like(self.points)
        grad_m = torch.zeros_like(self.points)
        for pts, to, _, Vi, gm, (a, b), local, on, rows in kept:
            _, Jf, Jm, Jc = self._jacobians(a, b)
            dx = torch.zeros((b - a, 2), dtype=torch.float64, device=_device())
            dx[on] = (Jf[on] @ xf[to[rows]][..., None])[..., 0]
            if self.nk:
                dx = dx + (Jc @ xf[-self.nk:])
            t = torch.zeros((len(pts), 3), dtype=torch.float64, device=_device())
            t.index_add_(0, local, (Jm.mT @ dx[..., None])[..., 0])
            dm[pts] = (Vi @ (gm - t)[..., None])[..., 0]
            grad_m[pts] = gm
        if self.gauge is not None:
            # the scale about the one fixed camera leaves every residual as it
            # is: the exact step has no component along it in the damping's metric
            c = self.poses[self.gauge, 4:]
            vf = torch.zeros((self.nf, 6), dtype=torch.float64, device=_device())
            vf[:, 3:] = self.poses[self.free, 4:] - c
            vf = torch.cat([vf.reshape(-1), torch.zeros(self.nk, dtype=torch.float64, device=_device())])
            vm = self.points - c
            num = (vf * diag * xf).sum() + (vm * self.cnt_m[:, None] * dm).sum()
            den = (vf * diag * vf).sum() + (vm * self.cnt_m[:, None] * vm).sum()
            xf, dm = xf - num / den * vf, dm - num / den * vm
        poses = self.poses.clone()
        new = _mul(_exp(xf[:6 * self.nf].reshape(-1, 6)), self.poses[self.free])
        new = torch.cat([new[:, :4] / new[:, :4].norm(dim=1, keepdim=True), new[:, 4:]], -1)
        poses[self.free] = torch.cat([torch.where(new[:, :1] < 0, -new[:, :4], new[:, :4]), new[:, 4:]], -1)
        points = self.points + dm
        cam = self.cam + xf[6 * self.nf:] if self.nk else self.cam
        trial = self.cost(poses, points, cam)
        predicted = float(nu * ((xf * xf).sum() + (dm * dm).sum()) + (xf * grad_f).sum() + (dm * grad_m).sum())
        rho = (merit - trial) / predicted if predicted else 0.0
        if rho > 0 and trial < merit:
            self.poses, self.points, self.cam = poses, points, cam
            return trial, nu * max(1 - (2 * rho - 1) ** 3, 1 / 3), True
        return merit, 2 * nu, False

    def optimise(self, iters, nu):
        merit, costs = self.cost(self.poses, self.points, self.cam), []
        for _ in range(iters):
            merit, nu, _ = self.step(nu, merit)
            costs.append(merit)
        return dict(poses=self.poses.cpu().numpy(), points=self.points.cpu().numpy(), costs=np.array(costs),
                    camera=self.cam.cpu().numpy())

    def covariance(self, queries):
        S, _, _, kept, _ = self.system(0.0, "all")
        d = S.diagonal().rsqrt()
        Z = torch.cholesky_inverse(torch.linalg.cholesky(d[:, None] * S * d[None, :]))
        Z = d[:, None] * Z * d[None, :]
        where = {}
        for c, k in enumerate(kept):
            for i, q in enumerate(k[0].tolist()):
                where[q] = (c, i)

        def rows(pose):
            b = int(self.block[pose])
            return slice(6 * b, 6 * b + 6)

        def of(row, col):
            if row[0] == 1 and col[0] == 1:
                return Z[rows(row[1]), rows(col[1])]
            c, i = where[col[1]]
            to, W, Vi = kept[c][1], kept[c][2][i], kept[c][3][i]
            Y = W @ Vi
            if row[0] == 1:
                return -(Z[rows(row[1])][:, to] @ Y)
            return Vi + Y.T @ Z[to][:, to] @ Y

        return [torch.stack([of(r, c) for r, c in q]).cpu().numpy() for q in queries]


def exact(case, seed):
    if case["kind"] == "windows":
        got = []
        for s in _window_scenes(case, seed):
            got.append(_Exact(s).optimise(case["iters"], s.initial_lm_damping))
        return dict(poses=np.concatenate([g["poses"] for g in got]), points=np.concatenate([g["points"] for g in got]),
                    costs=np.stack([g["costs"] for g in got]))
    prob = _scene(case, seed)
    e = _Exact(prob)
    if case["kind"] == "cov":
        return e.covariance(_queries(prob))
    out = e.optimise(case["iters"], prob.initial_lm_damping)
    if not (case["kind"] == "ring" and case["free"]):
        out.pop("camera")
    return out
