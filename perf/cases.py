"""The work that a SLAM program has this library do, as cases that can be timed.

Each case is a dict of plain values; ``kind`` says which public call it makes:

* ``match``    ``find_matches`` of two frames' descriptors;
* ``track``    ``map_optimise(1, True, 50)``: the newest frame against the fixed map;
* ``window``   ``map_optimise(window, False, rounds)``: a local window of a map, from map arrays;
* ``cull``     ``map_cull`` of a map given as arrays;
* ``solve``    a bundle adjustment of an uploaded problem from its initial state, and its result;
* ``step``     ``linear_step``: one linearisation and one damped solve (gradient, right-hand side, step);
* ``batch``    ``solve_batch`` of independent local windows;
* ``adjoint``  gradients of a loss of the solved state with respect to pixels and intrinsics.

Scenes are the three of the repository's generator (cameras on an arc, on a
random walk, on a closed loop; the sizes of its named workloads), drawn here
with torch so that a million observations take a fraction of a second. Every
map has zeroslam's gauge (frames 0 and 1 fixed) and every landmark is seen at
least twice.
"""

import functools
import math

import numpy as np
import torch

from zeroslam_gb300 import ba, scenes

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
FX, FY, CX, CY = scenes.INTRINSICS
HUBER = math.sqrt(5.991)  # map::optimise's loss
PRECISION = {"fp64": ba.FP64, "mixed": ba.MIXED}


def listed():
    return [
        # Matching the descriptors of a frame against the previous one's, each
        # frame of a sequence (an odd count: a detector gives what it finds).
        dict(name="match_frames", kind="match", lhs=2000, rhs=1987, k=2),
        # The pose of each new frame against the fixed map: the smallest solve.
        dict(name="track_frame", kind="track", scene="arc", K=5, L=1500),
        # Local bundle adjustment after a keyframe: the newest 20 frames of a
        # walk's map, through the whole call from map arrays to map arrays.
        dict(name="window_map", kind="window", scene="walk", K=60, L=12000, window=20, rounds=10, precision="fp64"),
        # Culling the map after that.
        dict(name="cull_map", kind="cull", scene="walk", K=200, L=50000),
        # The small scene: ten keyframes, latency and launches.
        dict(name="solve_small", kind="solve", scene="arc", K=10, L=500, iterations=10, precision="fp64"),
        # Global bundle adjustment of a million observations, the headline
        # workload, in both arithmetic forms. Eight iterations: the damping is
        # then near 1, and later steps move along directions that the mixed
        # form leaves open (its result says less than its cost there).
        dict(name="solve_walk_mixed", kind="solve", scene="walk", K=200, L=50000, iterations=8, precision="mixed"),
        dict(name="solve_walk_fp64", kind="solve", scene="walk", K=200, L=50000, iterations=8, precision="fp64"),
        # Closing a 1,000-keyframe loop: the largest reduced system.
        dict(name="solve_loop_mixed", kind="solve", scene="loop", K=1000, L=200000, iterations=6, precision="mixed"),
        dict(name="step_loop_fp64", kind="step", scene="loop", K=1000, L=200000, precision="fp64"),
        # Many independent local windows at once (several maps, or sub-maps):
        # in FP64 to their end; in the mixed form, whose windows are solved in
        # FP32, for as many iterations as say more than its rounding does.
        dict(name="batch_fp64", kind="batch", windows=64, kmax=30, lmax=3000, iterations=10, precision="fp64"),
        dict(name="batch_mixed", kind="batch", windows=256, kmax=30, lmax=3000, iterations=3, precision="mixed"),
        # Gradients through the solve (a learned front end).
        dict(name="adjoint", kind="adjoint", scene="arc", K=50, L=10000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["match", "track", "window", "cull", "solve", "solve", "solve", "step", "step", "batch", "batch",
                       "adjoint"])
    if kind == "match":
        return dict(kind=kind, lhs=_log(rng, 300, 6000), rhs=_log(rng, 300, 20000), k=rng.choice([1, 2, 2, 4]))
    if kind == "track":
        return dict(kind=kind, scene="arc", K=rng.randint(4, 12), L=_log(rng, 150, 4000))
    if kind == "window":
        return dict(kind=kind, scene="walk", K=rng.randint(20, 120), L=_log(rng, 2000, 20000),
                    window=rng.randint(5, 20), rounds=10, precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "cull":
        return dict(kind=kind, scene="walk", K=rng.randint(20, 200), L=_log(rng, 1000, 50000))
    if kind == "batch":
        precision = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, windows=_log(rng, 8, 64 if precision == "fp64" else 256), kmax=rng.randint(8, 30),
                    lmax=_log(rng, 400, 3000), iterations=10 if precision == "fp64" else 3, precision=precision)
    if kind == "adjoint":
        return dict(kind=kind, scene="arc", K=rng.randint(8, 50), L=_log(rng, 300, 10000))
    scene = rng.choice(["arc", "walk", "walk", "loop"])
    if scene == "arc":
        K, L = rng.randint(6, 50), _log(rng, 300, 8000)
    elif scene == "walk":
        K, L = rng.randint(40, 200), _log(rng, 4000, 50000)
    else:
        K, L = rng.randint(300, 1000), _log(rng, 40000, 200000)
    precision = rng.choice(["fp64", "mixed"])
    if kind == "step":
        return dict(kind=kind, scene=scene, K=K, L=L, precision="fp64")
    if scene == "loop":
        precision = "mixed"
    return dict(kind=kind, scene=scene, K=K, L=L, precision=precision,
                iterations=10 if scene == "arc" else 6 if scene == "loop" else 8)


# ------------------------------------------------------------------- scenes

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 17)
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=F64)


def _qmul(a, b):  # quaternions x, y, z, w
    av, aw, bv, bw = a[..., :3], a[..., 3:], b[..., :3], b[..., 3:]
    return torch.cat([aw * bv + bw * av + torch.linalg.cross(av, bv), aw * bw - (av * bv).sum(-1, keepdim=True)], -1)


def _qmat(q):
    x, y, z, w = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).unflatten(-1, (3, 3))


def _plus(q, t, d):
    """exp(d) (q, t) of SE(3); d = (omega, upsilon)."""
    om, up = d[..., :3], d[..., 3:]
    th2 = (om * om).sum(-1, keepdim=True)
    th = th2.sqrt()
    small = th2 < 1e-12
    ts, t2 = torch.where(small, 1.0, th), torch.where(small, 1.0, th2)
    dq = torch.cat([om * torch.where(small, 0.5 - th2 / 48, torch.sin(0.5 * ts) / ts),
                    torch.where(small, 1 - th2 / 8, torch.cos(0.5 * ts))], -1)
    c1 = torch.linalg.cross(om, up)
    dt = up + torch.where(small, 0.5, (1 - torch.cos(ts)) / t2) * c1 \
        + torch.where(small, 1 / 6, (ts - torch.sin(ts)) / (t2 * ts)) * torch.linalg.cross(om, c1)
    return _qmul(dq, q), torch.einsum("kij,kj->ki", _qmat(dq), t) + dt


def _cameras(kind, K, g):
    """Centres [K, 3] and headings [K] of the cameras (yaw about y)."""
    if kind == "arc":  # 36 degrees of a 1 m circle, every axis through the origin
        th = torch.deg2rad(-18.0 + 36.0 * torch.arange(K, device=DEV, dtype=F64) / max(1, K - 1))
        return torch.stack([torch.sin(th), 0 * th, -torch.cos(th)], 1), -th
    if kind == "walk":  # 0.1 m steps, 3 degrees of yaw jitter
        yaw = torch.cumsum(torch.cat([torch.zeros(1, device=DEV, dtype=F64), math.radians(3.0) * _normal(g, K - 1)]), 0)
        step = 0.1 * torch.stack([torch.sin(yaw), 0 * yaw, torch.cos(yaw)], 1)
        c = torch.cat([torch.zeros(1, 3, device=DEV, dtype=F64), torch.cumsum(step[:-1], 0)])
        return c + torch.tensor([0.0, 0.0, -10.0], device=DEV, dtype=F64), yaw
    a = 2 * math.pi * torch.arange(K, device=DEV, dtype=F64) / K  # a 100 m loop, looking along it
    r = 100.0 / (2 * math.pi)
    return torch.stack([r * torch.cos(a), 0 * a, r * torch.sin(a)], 1), -a


def _candidates(kind, n, g):
    if kind == "arc":
        return torch.stack([_uniform(g, n, -2, 2), _uniform(g, n, -2, 2), _uniform(g, n, 1, 7)], 1)
    if kind == "walk":
        return torch.stack([_uniform(g, n, -15, 15), _uniform(g, n, -5, 5), _uniform(g, n, -15, 15)], 1)
    r = 100.0 / (2 * math.pi)
    rad, ang = _uniform(g, n, (r - 4) ** 2, (r + 4) ** 2).sqrt(), _uniform(g, n, 0, 2 * math.pi)
    return torch.stack([rad * torch.cos(ang), _uniform(g, n, -3, 3), rad * torch.sin(ang)], 1)


# Pixel noise, initial pose noise (rad, m), landmark noise (relative to the
# distance from the nearest camera that sees it), depth range.
SHAPE = {"arc": (1.0, 0.02, 0.05, 0.03, 1e-12, math.inf), "walk": (1.0, 0.01, 0.03, 0.02, 0.5, 7.0),
         "loop": (0.5, 0.001, 0.003, 0.02, 1.0, 5.7)}
# A tracked estimate that is refined, with sub-pixel keypoints (track, batch).
TRACKED = (0.5, 0.002, 0.005, 0.005, 1e-12, math.inf)
# The true state, with keypoints fine enough that it is (near) a minimum.
CONVERGED = (0.1, 0.002, 0.005, 0.005, 1e-12, math.inf)
# A map that was optimised when its last keyframe came. No keypoint lies
# beyond Huber's threshold: whether an outlier's weight gets its second-order
# term is decided by the last bit of its residual, so that a solve with
# outliers ends elsewhere after any change of rounding.
MAPPED = (0.3, 0.0003, 0.0005, 0.0003, 0.5, 7.0)


def _scene(kind, K, L, seed, shape=None, geometry=None):
    """A scene drawn from ``seed``; ``geometry`` (another seed) keeps what is seen from where."""
    sigma, rot, trans, rel, zmin, zmax = shape or SHAPE[kind]
    g = _gen(seed if geometry is None else geometry)
    centre, yaw = _cameras(kind, K, g)
    q = torch.stack([0 * yaw, torch.sin(-0.5 * yaw), 0 * yaw, torch.cos(0.5 * yaw)], 1)
    R = _qmat(q)
    t = -torch.einsum("kij,kj->ki", R, centre)
    Xs, poses, lms, uvs, kept = [], [], [], [], 0
    chunk = max(256, int(2e7 // K))
    for _ in range(1000):  # candidates until L landmarks are seen twice
        X = _candidates(kind, min(chunk, 8 * L + 64), g)
        Xc = torch.einsum("kij,lj->lki", R, X) + t
        z = Xc[..., 2]
        u, v = FX * Xc[..., 0] / z + CX, FY * Xc[..., 1] / z + CY
        vis = (z >= zmin) & (z <= zmax) & (u >= 0) & (u < scenes.WIDTH) & (v >= 0) & (v < scenes.HEIGHT)
        good = torch.nonzero(vis.sum(1) >= 2)[: L - kept, 0]
        li, ki = torch.nonzero(vis[good], as_tuple=True)
        Xs.append(X[good])
        poses.append(ki)
        lms.append(li + kept)
        uvs.append(torch.stack([u[good][li, ki], v[good][li, ki]], 1))
        kept += good.numel()
        if kept >= L:
            break
    X, pose, lm, uv = torch.cat(Xs), torch.cat(poses), torch.cat(lms), torch.cat(uvs)
    g = _gen(seed) if geometry is not None else g
    uv = uv + sigma * _normal(g, *uv.shape)
    d = torch.cat([rot * _normal(g, K, 3), trans * _normal(g, K, 3)], 1)
    if kind == "loop":  # drift to 0.5 m and 2 degrees at the end
        axis = torch.nn.functional.normalize(_normal(g, 2, 3), dim=1)
        s = torch.arange(K, device=DEV, dtype=F64)[:, None] / max(1, K - 1)
        d = d + s * torch.cat([math.radians(2.0) * axis[0], 0.5 * axis[1]])
    d[0] = 0
    q0, t0 = _plus(q, t, d)
    near = torch.zeros(L, dtype=F64, device=DEV).scatter_reduce(0, lm, (X[lm] - centre[pose]).norm(dim=1), "amin",
                                                                include_self=False)
    X0 = X + rel * near[:, None] * _normal(g, L, 3)
    fixed = np.zeros(K, np.uint8)
    fixed[:2 if K > 2 else 1] = 1
    n = lambda a: np.ascontiguousarray(a.cpu().numpy())  # noqa: E731
    return scenes.Scene(name=kind, poses=n(torch.cat([t0, q0], 1)), pose_fixed=fixed, landmarks=n(X0),
                        landmark_fixed=np.zeros(L, np.uint8), obs_pose=n(pose.int()), obs_landmark=n(lm.int()),
                        obs_uv=n(uv), gt_poses=n(torch.cat([t, q], 1)), gt_landmarks=n(X))


def _case_scene(case, seed):
    shape = {"track": TRACKED, "adjoint": CONVERGED, "window": MAPPED}.get(case["kind"])
    # the adjoint's result has a row an observation
    return _scene(case["scene"], case["K"], case["L"], seed, shape, 0 if case["kind"] == "adjoint" else None)


def _windows(case, seed):
    r = np.random.default_rng(5)  # the sizes are the case's, the scenes the seed's
    out = []
    for i in range(case["windows"]):
        K, L = int(r.integers(5, case["kmax"] + 1)), int(r.integers(200, case["lmax"] + 1))
        out.append(_scene("arc", K, L, seed * 4099 + i, TRACKED))
    return out


def _descriptors(case, seed):
    """Near copies (0-40 of 256 bits flipped) of the right set's descriptors, and others."""
    r = np.random.default_rng([int(seed), 7])
    nl, nr = case["lhs"], case["rhs"]
    rhs = r.integers(0, 256, (nr, 32), dtype=np.uint8)
    dup = np.flatnonzero(r.random(nr) < 0.05)
    rhs[dup] = rhs[r.integers(0, nr, dup.size)]
    lhs = r.integers(0, 256, (nl, 32), dtype=np.uint8)
    near = np.flatnonzero(r.random(nl) < 0.6)
    flip = np.argsort(r.random((near.size, 256)), axis=1) < r.integers(0, 41, near.size)[:, None]
    lhs[near] = rhs[r.integers(0, nr, near.size)] ^ np.packbits(flip, axis=1)
    return lhs, rhs


# --------------------------------------------------------------- the passes

def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "match":
        s["lhs"], s["rhs"] = _descriptors(case, seed)
        s["ba"] = ba.BundleAdjuster()
        return s
    if kind == "batch":
        s["ba"] = ba.BundleAdjuster(precision=PRECISION[case["precision"]])
        s["ba"].set_batch(_windows(case, seed))
        return s
    sc = _case_scene(case, seed)
    s["ba"] = h = ba.BundleAdjuster(precision=PRECISION[case.get("precision", "fp64")])
    if kind in ("track", "window"):
        s["map"] = scenes.slam_map(sc)
    elif kind == "cull":
        s["map"] = scenes.cull_map(sc, seed=seed, truth=True)
    elif kind == "adjoint":
        h.set_problem(sc)
        h.set_state(sc.gt_poses, sc.gt_landmarks)  # an estimate that has converged elsewhere
        s["dp"], s["dl"] = _loss_gradient(case, seed)
    else:
        h.set_problem(sc)
    return s


# The damping a few iterations into a solve (it starts at a few thousand and falls by 3 each iteration).
STEP_LAMBDA = 50.0


def _loss_gradient(case, seed):
    r = np.random.default_rng([int(seed), 11])
    return r.standard_normal((case["K"], 6)), r.standard_normal((case["L"], 3))


def _rows(found, case):
    """The matches in the room there is for them, -1 after the last."""
    out = np.full(case["k"] * case["lhs"], -1, found.dtype)
    out[:found.size] = found
    return out


def run(s):
    case, h = s["case"], s["ba"]
    kind = case["kind"]
    if kind == "match":
        m = h.find_matches(s["lhs"], s["rhs"], 32.0, case["k"], case["k"] * case["lhs"])
        return [_rows(m["lhs_index"].view(np.int64), case), _rows(m["rhs_index"].view(np.int64), case),
                _rows(m["score"], case)]
    if kind == "track":
        frames, _, rep = h.map_optimise(s["map"], 1, True, 50)
        return [frames, rep.solve.chi2_final]
    if kind == "window":
        frames, landmarks, rep = h.map_optimise(s["map"], case["window"], False, case["rounds"])
        return [frames, landmarks, rep.solve.chi2_final]
    if kind == "cull":
        erase, mean, _ = h.map_cull(s["map"])
        return [erase, mean]
    if kind == "step":
        d = h.linear_step(STEP_LAMBDA, want_S=False)
        return [d["bs"], d["delta"], d["b"]]
    if kind == "adjoint":
        duv, dintr, _ = h.adjoint(s["dp"], s["dl"])
        return [duv, dintr]
    h.reset_state()
    if kind == "batch":
        _, reports, _ = h.solve_batch(case["iterations"])
        poses, landmarks = h.get_state()
        return [poses, landmarks, np.array([r.chi2_final for r in reports])]
    rep = h.solve(case["iterations"])
    poses, landmarks = h.get_state()
    return [poses, landmarks, rep.chi2_final]


# -------------------------------------------------------- what cannot be less

@functools.lru_cache(maxsize=64)
def _counts(key):
    """Observations and pose pairs (a >= b) over the landmarks of a case's scenes."""
    case = dict(key)
    M = pairs = 0
    for sc in _windows(case, 0) if case["kind"] == "batch" else [_case_scene(case, 0)]:
        c = np.bincount(sc.obs_landmark).astype(np.int64)
        M += int(c.sum())
        pairs += int((c * (c + 1) // 2).sum())
    return M, pairs


def work(case):
    kind = case["kind"]
    if kind == "match":  # 8 words of exclusive or, popcount and sum a pair
        return dict(bytes=32 * (case["lhs"] + case["rhs"]) + 24 * case["k"] * case["lhs"], flops=24 * case["lhs"] * case["rhs"])
    M, pairs = _counts(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    if kind == "batch":
        n3 = sum(216 * k**3 for k in range(5, case["kmax"] + 1)) / (case["kmax"] - 4) * case["windows"]
        K, L = case["windows"] * (5 + case["kmax"]) // 2, case["windows"] * (200 + case["lmax"]) // 2
    else:
        K, L = case["K"], case["L"]
        n3 = (6 * K) ** 3
    if kind == "cull":
        return dict(bytes=12 * M + 41 * L + 128 * K, flops=35 * M // 2)
    if kind == "track":  # one pose: its observations, 27 sums each, a few iterations
        return dict(bytes=24 * L + 12 * M + 192 * K, flops=4 * 300 * L)
    if kind == "window":  # the newest frames' share of the map
        f = min(1.0, 2 * case["window"] / K)
        M, pairs, L, n3 = int(M * f), int(pairs * f), int(L * f), n3 * f**3
    passes = case.get("iterations", case.get("rounds", 1))
    # a linearisation (about 250 operations an observation), W (36 multiply-adds),
    # the products of the pairs (108 multiply-adds), a Cholesky factor, a cost
    flops = passes * (400 * M + 216 * pairs + n3 / 3)
    nbytes = 24 * M + 2 * (56 * K + 24 * L)
    if kind == "adjoint":  # the exact Hessian once and its solve; a gradient a pixel
        nbytes += 16 * M
    return dict(bytes=nbytes, flops=flops)


# ------------------------------------------------------ the same in 64 bits

class _Problem:
    def __init__(self, sc, huber=False):
        T = lambda a, d: torch.as_tensor(np.ascontiguousarray(a), device=DEV).to(d)  # noqa: E731
        p = T(sc.poses, F64)
        self.t, self.q, self.X = p[:, :3], p[:, 3:], T(sc.landmarks, F64)
        self.pose, self.lm, self.uv = T(sc.obs_pose, torch.long), T(sc.obs_landmark, torch.long), T(sc.obs_uv, F64)
        self.pfree, self.lfree = T(sc.pose_fixed, F64) == 0, T(sc.landmark_fixed, F64) == 0
        self.K, self.L, self.huber = self.q.shape[0], self.X.shape[0], huber
        order = torch.argsort(self.lm, stable=True)
        self.pose, self.lm, self.uv, self.order = self.pose[order], self.lm[order], self.uv[order], order
        # every ordered pair of observations of one landmark
        c = torch.bincount(self.lm, minlength=self.L)
        start = torch.cumsum(c, 0) - c
        self.pair_count, self.pair_start = c[self.lm], start[self.lm]

    def point(self, q, t, X):
        return torch.einsum("mij,mj->mi", _qmat(q)[self.pose], X[self.lm]) + t[self.pose]

    def residual(self, Xc):
        z = Xc[:, 2]
        front = (z >= 1e-12)[:, None]
        r = self.uv - torch.stack([FX * Xc[:, 0] / z + CX, FY * Xc[:, 1] / z + CY], 1)
        return torch.where(front, r, (-0.3 * z)[:, None].expand(-1, 2)), front

    def chi2(self, q, t, X):
        e2 = self.residual(self.point(q, t, X))[0].square().sum(1)
        if self.huber:
            e2 = torch.where(e2 <= HUBER**2, e2, 2 * e2.sqrt() * HUBER - HUBER**2)
        return e2.sum().item()

    def linearise(self):
        Xc = self.point(self.q, self.t, self.X)
        r, front = self.residual(Xc)
        x, y, z = Xc.unbind(1)
        o = torch.zeros_like(z)
        Jc = torch.stack([FX / z, o, -FX * x / z**2, o, FY / z, -FY * y / z**2], 1).unflatten(1, (2, 3))
        behind = torch.tensor([[0, 0, 0.3], [0, 0, 0.3]], device=DEV, dtype=F64)
        Jc = torch.where(front[:, :, None], Jc, behind)
        P = torch.stack([o, z, -y, -z, o, x, y, -x, o], 1).unflatten(1, (3, 3))
        Jp = -torch.cat([Jc @ P, Jc], 2) * self.pfree[self.pose, None, None]
        Jl = -(Jc @ _qmat(self.q)[self.pose]) * self.lfree[self.lm, None, None]
        e2 = r.square().sum(1)
        w1 = torch.ones_like(e2)
        W = torch.eye(2, device=DEV, dtype=F64).expand(e2.numel(), 2, 2)
        if self.huber:
            out = e2 > HUBER**2
            w1 = torch.where(out, HUBER / e2.clamp(min=1e-300).sqrt(), w1)
            w2 = torch.where(out, -0.5 * w1 / e2.clamp(min=1e-300), 0.0)
            take = (w1 + 2 * w2 * e2) > 0
            W = w1[:, None, None] * W + torch.where(take, 2 * w2, 0.0)[:, None, None] * r[:, :, None] * r[:, None, :]
        JpW, JlW = Jp.transpose(1, 2) @ W, Jl.transpose(1, 2) @ W
        g = w1[:, None] * r
        return self.blocks(JpW @ Jp, JpW @ Jl, JlW @ Jl, -(Jp * g[:, :, None]).sum(1), -(Jl * g[:, :, None]).sum(1))

    def blocks(self, pp, pl, ll, bp, bl):
        add = lambda n, i, v: torch.zeros(n, *v.shape[1:], device=DEV, dtype=F64).index_add_(0, i, v)  # noqa: E731
        return add(self.K, self.pose, pp), pl, add(self.L, self.lm, ll), add(self.K, self.pose, bp), add(self.L, self.lm, bl)

    def solve(self, lin, lam):
        """The damped system by its Schur complement: b_s, and the step of poses and landmarks (None: not positive)."""
        Hpp, Hpl, Hll, bp, bl = lin
        K, n = self.K, 6 * self.K
        inv = torch.zeros_like(Hll)
        A = Hll + lam * torch.eye(3, device=DEV, dtype=F64)
        inv[self.lfree] = torch.linalg.inv(A[self.lfree])
        W = Hpl @ inv[self.lm]
        S = torch.zeros(K * K, 36, device=DEV, dtype=F64)
        at = torch.cumsum(self.pair_count, 0)
        lo = 0
        while lo < at.numel():  # a few million pairs at a time
            base = at[lo] - self.pair_count[lo]
            hi = max(lo + 1, int(torch.searchsorted(at, base + 3_000_000)))
            i = torch.repeat_interleave(torch.arange(lo, hi, device=DEV), self.pair_count[lo:hi])
            j = self.pair_start[i] + torch.arange(i.numel(), device=DEV) - (at[i] - self.pair_count[i] - base)
            C = sum(W[i][:, :, k, None] * Hpl[j][:, None, :, k] for k in range(3))
            S.index_add_(0, self.pose[i] * K + self.pose[j], C.flatten(1), alpha=-1.0)
            lo = hi
        S = S.view(K, K, 6, 6)
        ks = torch.arange(K, device=DEV)
        S[ks, ks] += Hpp + lam * torch.eye(6, device=DEV, dtype=F64)
        S = S.permute(0, 2, 1, 3).reshape(n, n)
        bs = bp.index_add(0, self.pose, (W @ bl[self.lm][:, :, None])[:, :, 0], alpha=-1.0).reshape(n)
        F, info = torch.linalg.cholesky_ex(S)
        if int(info) != 0:
            return bs, None, None
        dp = torch.cholesky_solve(bs[:, None], F).view(K, 6)
        v = bl.index_add(0, self.lm, (Hpl.transpose(1, 2) @ dp[self.pose][:, :, None])[:, :, 0], alpha=-1.0)
        return bs, dp, (inv @ v[:, :, None])[:, :, 0]

    def lm_solve(self, iterations):
        """Levenberg-Marquardt as factor_graph::solve runs it; chi2 of the result."""
        lin = self.linearise()
        diag = max(torch.diagonal(lin[0], dim1=1, dim2=2).max().item(), torch.diagonal(lin[2], dim1=1, dim2=2).max().item())
        lam, nu, chi2 = 1e-5 * min(5e10, diag), 2.0, self.chi2(self.q, self.t, self.X)
        stop = 1e-10 * chi2
        for _ in range(iterations):
            last, failures = chi2, 0
            while failures < 10:
                _, dp, dl = self.solve(lin, lam)
                rho = -1.0
                if dp is not None:
                    q, t = _plus(self.q, self.t, dp)
                    q, t = torch.where(self.pfree[:, None], q, self.q), torch.where(self.pfree[:, None], t, self.t)
                    X = torch.where(self.lfree[:, None], self.X + dl, self.X)
                    new = self.chi2(q, t, X)
                    scale = (dp * (lam * dp + lin[3])).sum().item() + (dl * (lam * dl + lin[4])).sum().item() + 1e-3
                    rho = (chi2 - new) / scale
                if rho > 0 and math.isfinite(new):
                    lam *= max(1 / 3, min(1 - (2 * rho - 1) ** 3, 2 / 3))
                    nu, chi2 = 2.0, new
                    self.q, self.t, self.X = q, t, X
                    lin = self.linearise()
                    break
                lam, nu, failures = lam * nu, 2 * nu, failures + 1
            if failures >= 10 or last - chi2 < stop or not math.isfinite(lam):
                break
        return chi2

    def state(self):
        return torch.cat([self.t, self.q], 1), self.X


def _window(cm, window, fix_landmarks):
    """map::optimise's choice of frames, landmarks and edges of a map, as a problem."""
    F, L = cm.F, cm.L
    lm = np.repeat(np.arange(L), np.diff(cm.landmark_obs))
    fixed = (cm.frame_id == 0) | ((cm.frame_id == 1) & (F > 2)) | (cm.frame_id < cm.frame_id_generator - window)
    seen = np.bincount(lm[~fixed[cm.obs_frame]], minlength=L) > 0
    frame = (cm.frame_id >= cm.frame_id_generator - 1 - 2 * window) & (np.bincount(cm.obs_frame[seen[lm]], minlength=F) > 0)
    edge = seen[lm] & frame[cm.obs_frame]
    if fix_landmarks:
        edge &= ~fixed[cm.obs_frame]
    return lm, fixed, seen, edge


def exact(case, seed):
    kind = case["kind"]
    if kind == "match":
        lhs, rhs = _descriptors(case, seed)
        bits = [torch.as_tensor(2 * np.unpackbits(d, axis=1).astype(np.float32) - 1, device=DEV) for d in (lhs, rhs)]
        dist = ((256 - bits[0] @ bits[1].T) / 2).double()
        near = torch.topk(dist, case["k"], dim=1, largest=False).values
        return [None, None, _rows(near[near < 32.0].cpu().numpy(), case)]
    if kind == "batch":
        if case["windows"] * case["iterations"] > 800:
            return None  # window by window: over 20 seconds
        got = []
        for sc in _windows(case, seed):
            p = _Problem(sc)
            chi2 = p.lm_solve(case["iterations"])
            got.append((*p.state(), chi2))
        return [torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got]),
                torch.tensor([g[2] for g in got], dtype=F64)]
    sc = _case_scene(case, seed)
    if kind == "cull":
        return [None, _exact_cull(scenes.cull_map(sc, seed=seed, truth=True))]
    if kind in ("track", "window"):
        cm = scenes.slam_map(sc)
        track = kind == "track"
        lm, fixed, seen, edge = _window(cm, 1 if track else case["window"], track)
        sc.obs_pose, sc.obs_landmark, sc.obs_uv = cm.obs_frame[edge], lm[edge], cm.obs_keypoint[edge]
        sc.pose_fixed = (fixed | (np.bincount(cm.obs_frame[edge], minlength=cm.F) == 0)).astype(np.uint8)
        sc.landmark_fixed = np.ones(cm.L, np.uint8) if track else (~seen).astype(np.uint8)
        p = _Problem(sc, huber=True)
        chi2 = p.lm_solve(50 if track else case["rounds"])
        frames = torch.cat([_qmat(p.q).flatten(1), p.t], 1)
        return [frames, chi2] if track else [frames, p.X, chi2]
    if kind == "adjoint":
        sc.poses, sc.landmarks = sc.gt_poses, sc.gt_landmarks
    p = _Problem(sc)
    if kind == "step":
        lin = p.linearise()
        bs, dp, dl = p.solve(lin, STEP_LAMBDA)
        flat = lambda a, b: torch.cat([a.flatten(), b.flatten()])  # noqa: E731
        return [bs, flat(dp, dl), flat(lin[3], lin[4])]
    if kind == "adjoint":
        return _exact_adjoint(p, *_loss_gradient(case, seed))
    chi2 = p.lm_solve(case["iterations"])
    return [*p.state(), chi2]


def _exact_cull(cm):
    """The mean pixel error of each landmark that map::cull computes one for, -1 elsewhere."""
    lm = np.repeat(np.arange(cm.L), np.diff(cm.landmark_obs))
    has = cm.obs_frame >= 0
    lm, f, kp = lm[has], cm.obs_frame[has], cm.obs_keypoint[has].astype(np.float64)
    Rt, intr = cm.frame_pose[f], cm.frame_intrinsics[f]
    Xc = np.einsum("mij,mj->mi", Rt[:, :9].reshape(-1, 3, 3), cm.landmarks[lm]) + Rt[:, 9:]
    with np.errstate(divide="ignore", invalid="ignore"):
        px = intr[:, :2] * Xc[:, :2] / Xc[:, 2:] + intr[:, 2:]
    err = np.where(Xc[:, 2] < 1e-12, 5.991, np.linalg.norm(kp - px, axis=1))
    count = np.bincount(lm, minlength=cm.L)
    mean = np.bincount(lm, err, minlength=cm.L) / np.maximum(count, 1)
    n = np.diff(cm.landmark_obs)
    last = np.where(n > 0, cm.obs_frame_id[np.maximum(cm.landmark_obs[1:] - 1, 0)], 0)
    early = (cm.landmark_id + 500 < cm.landmark_id_generator) | (n == 0) | (count == 0) \
        | ((n <= 4) & (last + 7 < cm.frame_id_generator))
    return np.where(early, -1.0, mean)


def _exact_adjoint(p, dp, dl):
    """Implicit-function gradients with the exact Hessian of half the squared residuals."""
    def cost(x, Xc0, R, uv, th):  # x: pose perturbation (6) and landmark's (3), second order in x
        om, up = x[:3], x[3:6]
        Y = Xc0 + R @ x[6:]
        Y = Y + torch.linalg.cross(om, Y) + 0.5 * torch.linalg.cross(om, torch.linalg.cross(om, Y)) + up \
            + 0.5 * torch.linalg.cross(om, up)
        r = uv - (th[:2] * Y[:2] / Y[2] + th[2:])
        return 0.5 * (r * r).sum()

    th = torch.tensor([FX, FY, CX, CY], device=DEV, dtype=F64)
    zero = torch.zeros(9, device=DEV, dtype=F64)
    each = lambda f: torch.func.vmap(f, in_dims=(None, 0, 0, 0, None), chunk_size=100_000)  # noqa: E731
    grad = torch.func.grad(cost)

    args = (zero, p.point(p.q, p.t, p.X), _qmat(p.q)[p.pose], p.uv, th)
    m = torch.cat([p.pfree[p.pose, None].expand(-1, 6), p.lfree[p.lm, None].expand(-1, 3)], 1).double()
    H = each(torch.func.hessian(cost))(*args) * m[:, :, None] * m[:, None, :]
    lin = p.blocks(H[:, :6, :6], H[:, :6, 6:], H[:, 6:, 6:], m[:, :6], m[:, 6:])
    a = [torch.as_tensor(dp, device=DEV) * p.pfree[:, None], torch.as_tensor(dl, device=DEV) * p.lfree[:, None]]
    hold = (~p.pfree).double()[:, None, None] * torch.eye(6, device=DEV, dtype=F64)  # fixed poses stay
    _, vp, vl = p.solve((lin[0] + hold, lin[1], lin[2], *a), 0.0)
    if vp is None:
        return None
    v = torch.cat([vp[p.pose], vl[p.lm]], 1) * m
    along = lambda f: torch.func.vmap(f, in_dims=(0, None, 0, 0, 0, None), chunk_size=100_000)  # noqa: E731
    duv = along(lambda w, x, *rest: torch.func.grad(lambda uv: grad(x, rest[0], rest[1], uv, rest[3]) @ w)(rest[2]))(v, *args)
    dth = along(lambda w, x, *rest: torch.func.grad(lambda i: grad(x, rest[0], rest[1], rest[2], i) @ w)(rest[3]))(v, *args)
    out = torch.empty_like(duv)
    out[p.order] = -duv
    return [out, -dth.sum(0)]
