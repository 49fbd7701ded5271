"""Performance cases: what users of this package have it do, through its public entry points.

A case is one call (or one reset + call on a handle that the program keeps) of the bundle
adjuster, the batched triplet adjustment, the triplet stage, rotation averaging or the
BundlePointStructure producer, on seeded synthetic data of the shapes that the package's own
scene generators, tests and benchmark use.  The library takes and returns host arrays, so a pass
goes from host inputs to host results.  ``exact`` restates each path in plain FP64 torch.

The number of LM iterations of a case is bounded to the part of the run in which rounding does not
yet decide the path: long runs converge along nearly free directions, FP32 blocks amplify their
own rounding from about the eighth iteration on, and at the fifth step of the triplet setting a
few of thousands of triplets have converged so far that the last bits accept or reject it.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from v3dsfmtoolkit_b200 import capi, scenes

PRECOND_WEIGHTS = "v3dsfmtoolkit_b200/precond_weights.npy"
STD, COMMON, VARYING, STEREO = scenes.MODEL_STD, scenes.MODEL_COMMON, scenes.MODEL_VARYING, scenes.MODEL_STEREO


def listed():
    return [
        # a small plain adjustment, as run after every few images: one call from arrays to arrays,
        # where launches, synchronisations and set-up decide
        dict(name="circle20_fp64", kind="ba", scene="circle", cams=20, points=2000, mode=0, precision="fp64",
             iterations=10, keep=False),
        # a submodel of an uncalibrated collection: per-camera intrinsics (13 unknowns per camera)
        dict(name="varying25", kind="ba", scene="varying", cams=25, points=3001, mode=4, precision="mixed",
             iterations=6, keep=False),
        # the 200-camera distortion adjustment with the default options on a kept handle (the loop
        # of adjusting, filtering and adjusting again)
        dict(name="sequence200", kind="ba", scene="sequence", cams=200, points=50000, mode=4, precision="mixed",
             iterations=6, keep=True),
        # the same scene type in FP64 as one call: construction, minimisation, results
        dict(name="sequence200_fp64_call", kind="ba", scene="sequence", cams=200, points=50000, mode=4,
             precision="fp64", iterations=24, keep=False),
        # the rig adjuster over a long stereo sequence, FP64, as one call
        dict(name="stereo300_fp64_call", kind="ba", scene="stereo", cams=300, points=40000, mode=0, precision="fp64",
             iterations=12, keep=False),
        # the largest adjustment: 2,000 cameras, ~1M points, PCG (the solver picked by size)
        dict(name="cluster2000_pcg", kind="ba", scene="cluster", cams=2000, points=1000000, mode=0, precision="mixed",
             iterations=6, keep=True, precond="jacobi"),
        # a mid-sized clustered scene with the trained preconditioner, FP64 blocks
        dict(name="cluster800_learned", kind="ba", scene="cluster", cams=800, points=150000, mode=0,
             precision="fp64", iterations=6, keep=True, precond="learned"),
        # all triplets of a collection adjusted in one launch on a kept batch
        dict(name="triplets4096", kind="triplets", count=4096, lo=50, hi=800, iterations=4, keep=True),
        # the triplets of one new image: a small batch as one call
        dict(name="triplets61_call", kind="triplets", count=61, lo=50, hi=800, iterations=4, keep=False),
        # triangulation, filtering and adjustment of all triplets, from flat host arrays
        dict(name="tripletstage4096", kind="stage", count=4096, lo=30, hi=800, iterations=3),
        # rotation averaging of a large view graph, one call
        dict(name="rotations10000", kind="rotations", views=10000, pairs=200000, keep=False),
        # flat bundle inputs of a reconstruction with half a million tracks
        dict(name="point_structure500k", kind="structure", tracks=500000, required=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circle", "varying", "sequence", "sequence", "stereo", "cluster", "triplets", "triplets", "stage",
                       "rotations", "rotations", "structure"])
    precision, keep = rng.choice(["mixed", "fp64"]), rng.random() < 0.5
    longest = 6 if precision == "mixed" else 20
    ba = dict(kind="ba", scene=kind, precision=precision, keep=keep)
    if kind == "circle":
        return dict(ba, cams=rng.randint(5, 60), points=_log(rng, 150, 8000), mode=0, iterations=rng.randint(4, min(longest, 10)))
    if kind == "varying":
        return dict(ba, cams=rng.randint(8, 40), points=_log(rng, 400, 6000), mode=rng.randint(0, 4),
                    iterations=rng.randint(3, 6))
    if kind == "sequence":
        cams = rng.randint(12, 200)
        return dict(ba, cams=cams, points=_log(rng, 40 * cams, 250 * cams), mode=rng.randint(0, 4),
                    iterations=rng.randint(4, longest), fixed=rng.choice([0, 0, 2]))
    if kind == "stereo":
        cams = rng.randint(12, 300)
        return dict(ba, cams=cams, points=_log(rng, 40 * cams, 130 * cams), mode=0, iterations=rng.randint(3, min(longest, 10)))
    if kind == "cluster":
        return dict(ba, cams=100 * rng.randint(7, 18), points=_log(rng, 50000, 700000), mode=0, iterations=rng.randint(2, 4),
                    precond=rng.choice(["jacobi", "jacobi", "learned"]))
    if kind == "triplets":
        return dict(kind=kind, count=_log(rng, 8, 4000), lo=rng.randint(20, 80), hi=rng.randint(90, 800),
                    iterations=rng.randint(2, 4), keep=keep)
    if kind == "stage":
        return dict(kind=kind, count=_log(rng, 8, 4000), lo=rng.randint(20, 80), hi=rng.randint(90, 800), iterations=rng.randint(2, 3))
    if kind == "rotations":
        views = _log(rng, 60, 9000)
        return dict(kind=kind, views=views, pairs=rng.randint(6, 20) * views, keep=keep)
    return dict(kind=kind, tracks=_log(rng, 2000, 450000), required=rng.randint(2, 4))


# ---- inputs --------------------------------------------------------------------------------------


def _expm(w):
    return scenes.rodrigues(w)


def _noisy_cameras(rng, R, T, rot, trans):
    axis = rng.normal(size=(len(R), 3))
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    return _expm(axis * rot) @ R, T + rng.normal(scale=1.0, size=T.shape) * trans


def _scene_arrays(sc):
    return dict(model=sc.model, mode=sc.mode, thr=sc.inlier_threshold, K=sc.K, R=sc.R, T=sc.T, dist=sc.dist, X=sc.X,
                meas=sc.meas, view=sc.view, point=sc.point)


def _stereo(cams, points, seed):
    """A toed-in binocular rig on a curving path; every point seen from up to six poses ahead of it."""
    rng = np.random.default_rng(seed)
    k = lambda f, cx, cy: np.array([[f, 0, cx], [0, f, cy], [0, 0, 1.0]])  # noqa: E731
    rig_K = np.stack([k(700.0, 320.0, 240.0), k(705.0, 318.0, 242.0)])
    rig_R = _expm(np.array([[0.0, 0.0, 0.0], [0.0, math.radians(-2.0), 0.0]]))
    rig_T = np.stack([np.zeros(3), -rig_R[1] @ np.array([0.3, 0.0, 0.0])])
    t = np.arange(cams, dtype=np.float64)
    centers = np.stack([0.5 * np.sin(0.15 * t), 0.1 * np.cos(0.2 * t), 0.8 * t], axis=1)
    R = _expm(np.stack([0 * t, 0.05 * np.sin(0.1 * t), 0 * t], axis=1))
    T = -np.einsum("nij,nj->ni", R, centers)
    more = 2 * points + 200          # candidates; the first `points` that are seen often enough are taken
    X = np.stack([rng.uniform(-4, 4, more), rng.uniform(-3, 3, more), rng.uniform(6, 0.8 * cams + 9, more)], axis=1)
    pose = np.clip(np.floor((X[:, 2] - 12.0) / 0.8), 0, cams - 1).astype(int)[:, None] + np.arange(6)
    at = np.minimum(pose, cams - 1)
    Y = np.einsum("mwij,mj->mwi", R[at], X) + T[at]
    Z = np.einsum("lij,mwj->mwli", rig_R, Y) + rig_T
    h = np.einsum("lij,mwlj->mwli", rig_K, Z)
    q = h[..., :2] / h[..., 2:]
    ok = (pose < cams)[..., None] & (Z[..., 2] > 0.5) & (q >= 0).all(-1) & (q < np.array([640.0, 480.0])).all(-1)
    kept = ok.sum((1, 2)) >= 3
    kept &= np.cumsum(kept) <= points
    ok &= kept[:, None, None]
    p, w, sub = np.nonzero(ok)
    meas = q[ok] + rng.normal(scale=0.5, size=(len(p), 2))
    bad = rng.random(len(p)) < 0.01
    meas[bad] += rng.normal(scale=30.0, size=(int(bad.sum()), 2))
    R0, T0 = _noisy_cameras(rng, R, T, 0.01, 0.02)
    X = X[kept]
    return dict(model=STEREO, mode=0, thr=2.0, K=np.zeros((1, 3, 3)), R=R0, T=T0, dist=None,
                X=X + rng.normal(scale=0.05, size=X.shape), meas=meas, view=pose[p, w].astype(np.int32),
                point=(np.cumsum(kept) - 1)[p].astype(np.int32), rig_K=rig_K, rig_R=rig_R, rig_T=rig_T,
                sub=sub.astype(np.int32))


def _cluster(cams, points, seed):
    """Groups of 100 cameras around neighbouring centres, tracks of a mean length of six inside a
    group, 5% of the points between two groups and seen from both; made on the GPU."""
    per, groups = 100, cams // 100
    rng = np.random.default_rng(seed)
    gc = np.stack([12.0 * np.arange(groups), np.zeros(groups), np.zeros(groups)], axis=1)
    grp = np.repeat(np.arange(groups), per)
    ang, elev = 2 * np.pi * rng.uniform(size=cams), rng.uniform(-0.3, 0.3, size=cams)
    centers = gc[grp] + 8.0 * np.stack([np.cos(ang) * np.cos(elev), np.sin(ang) * np.cos(elev), np.sin(elev)], axis=1)
    R, T = scenes.look_at(centers, gc[grp] + rng.normal(scale=0.5, size=(cams, 3)), np.array([0.0, 0.0, 1.0]))
    dev, gen = torch.device("cuda"), torch.Generator("cuda").manual_seed(seed)
    Rd, Td = torch.tensor(R, device=dev), torch.tensor(T, device=dev)
    f64 = dict(device=dev, dtype=torch.float64, generator=gen)
    X, view, point, meas, have = [], [], [], [], 0
    while have < points:
        m = min(100000, 1000 + 2 * (points - have))
        length = torch.empty(m, device=dev).geometric_(0.2, generator=gen).long() + 1
        cross = torch.rand(m, **f64) < 0.05
        g = torch.randint(0, max(groups - 1, 1), (m,), device=dev, generator=gen)
        base = torch.tensor(gc, device=dev)[g]
        base[:, 0] += 6.0 * cross
        x = base + 5.0 * torch.rand(m, 3, **f64) - 2.5
        cand = torch.rand(m, per, device=dev, generator=gen).topk(24, dim=1).indices
        cand = cand + per * (g[:, None] + (cross[:, None] & (torch.rand(m, 24, **f64) < 0.5)))
        y = torch.einsum("mcij,mj->mci", Rd[cand], x) + Td[cand]
        q = 1000.0 * y[..., :2] / y[..., 2:] + torch.tensor([320.0, 240.0], device=dev, dtype=torch.float64)
        vis = (y[..., 2] > 0.5) & (q >= 0).all(-1) & (q[..., 0] < 640) & (q[..., 1] < 480)
        kept = vis.sum(1) >= 2
        kept &= have + kept.cumsum(0) <= points
        take = vis & (vis.cumsum(1) <= length[:, None]) & kept[:, None]
        key = torch.where(take, cand, cams)
        key, o = key.sort(1)
        sel = key < cams
        noise = torch.randn(m, 24, 2, **f64)
        meas.append((q.gather(1, o[..., None].expand(-1, -1, 2)) + noise)[sel].cpu().numpy())
        view.append(key[sel].int().cpu().numpy())
        ids = have + kept.long().cumsum(0) - 1
        point.append(ids[:, None].expand(-1, 24)[sel].int().cpu().numpy())
        X.append((x + 0.02 * torch.randn(m, 3, **f64))[kept].cpu().numpy())
        have += int(kept.sum())
    R0, T0 = _noisy_cameras(rng, R, T, 0.005, 0.02)
    K = np.broadcast_to(np.array([[1000.0, 0, 320], [0, 1000, 240], [0, 0, 1]]), (cams, 3, 3)).copy()
    return dict(model=STD, mode=0, thr=1e6, K=K, R=R0, T=T0, dist=None, X=np.concatenate(X), meas=np.concatenate(meas),
                view=np.concatenate(view), point=np.concatenate(point))


def _ba_scene(case, seed):
    name, cams, points = case["scene"], case["cams"], case["points"]
    if name == "circle":
        return _scene_arrays(scenes.circle_scene(n_cams=cams, n_points=points, seed=seed))
    if name == "sequence":
        return _scene_arrays(scenes.sequence_scene(n_cams=cams, n_points=points, mode=case["mode"], seed=seed))
    if name == "varying":
        return _scene_arrays(scenes.varying_scene(n_cams=cams, n_points=points, mode=case["mode"], seed=seed))
    return (_stereo if name == "stereo" else _cluster)(cams, points, seed)


def _triplet_geometry(rng, n):
    """Three cameras per triplet around a common target: baselines U[0.5, 2], angles U[5, 30] degrees."""
    b, alpha = rng.uniform(0.5, 2.0, n), np.deg2rad(rng.uniform(5.0, 30.0, n))
    D = b / (2 * np.sin(alpha / 2))
    ang = alpha[:, None] * np.array([-1.0, 0.0, 1.0])
    c = np.stack([D[:, None] * np.sin(ang), 0 * ang, D[:, None] * (1 - np.cos(ang))], axis=2).reshape(-1, 3)
    target = np.repeat(np.stack([0 * D, 0 * D, D], axis=1), 3, axis=0)
    R, T = scenes.look_at(c, target, np.array([0.0, -1.0, 0.0]))
    return b, D, R, T


def _points_of(rng, case, D):
    counts = rng.permutation(np.linspace(case["lo"], case["hi"], len(D)).round().astype(int))
    owner = np.repeat(np.arange(len(D)), counts)
    X = D[owner, None] * (rng.uniform(-0.18, 0.18, size=(len(owner), 3)) + np.array([0.0, 0.0, 1.0]))
    return counts, owner, X


def _triplets(case, seed):
    rng, n = np.random.default_rng(seed), case["count"]
    b, D, R, T = _triplet_geometry(rng, n)
    counts, owner, X = _points_of(rng, case, D)
    cam = 3 * owner[:, None] + np.arange(3)
    Y = np.einsum("mvij,mj->mvi", R[cam], X) + T[cam]
    meas = 1000.0 * Y[..., :2] / Y[..., 2:] + np.array([320.0, 240.0])
    meas += rng.normal(scale=0.5, size=meas.shape)
    R0, T0 = _noisy_cameras(rng, R, T, 0.01, 0.02 * np.repeat(b, 3)[:, None])
    X0 = X + rng.normal(size=X.shape) * (0.01 * D[owner, None])
    first = np.cumsum(counts) - counts
    i32 = lambda a: np.ascontiguousarray(a, dtype=np.int32)  # noqa: E731
    K = np.broadcast_to(np.array([[1000.0, 0, 320], [0, 1000, 240], [0, 0, 1]]), (3 * n, 3, 3)).copy()
    return dict(n_cams=i32(np.full(n, 3)), n_points=i32(counts), n_obs=i32(3 * counts), thr=np.ones(n), K=K, R=R0, T=T0,
                X=X0, meas=np.ascontiguousarray(meas.reshape(-1, 2)), view=i32(np.tile(np.arange(3), len(owner))),
                point=i32(np.repeat(np.arange(len(owner)) - first[owner], 3)))


def _stage(case, seed):
    rng, n = np.random.default_rng(seed), case["count"]
    b, D, R, T = _triplet_geometry(rng, n)
    counts, owner, X = _points_of(rng, case, D)
    focal = rng.uniform(700.0, 1200.0, size=(n, 3))
    cam = 3 * owner[:, None] + np.arange(3)
    Y = np.einsum("mvij,mj->mvi", R[cam], X) + T[cam]
    f = focal[owner][..., None]
    q = Y[..., :2] / Y[..., 2:] + 0.3 * rng.normal(size=(len(owner), 3, 2)) / f
    wrong = np.where(rng.random(n) < 0.05, 0.7, 0.1)[owner, None]       # a few triplets are to be dropped
    bad = rng.random((len(owner), 3)) < wrong
    far, phi = rng.uniform(5.0, 40.0, size=bad.shape), rng.uniform(0, 2 * np.pi, size=bad.shape)
    q += np.where(bad[..., None], far[..., None] * np.stack([np.cos(phi), np.sin(phi)], axis=2) / f, 0.0)
    seen = np.ones(bad.shape, dtype=bool)
    two = rng.permutation(len(owner))[: len(owner) // 20]
    seen[two, rng.integers(0, 3, size=len(two))] = False
    R0, T0 = _noisy_cameras(rng, R, T, np.deg2rad(0.01), 0.0005 * np.repeat(b, 3)[:, None])
    i32 = lambda a: np.ascontiguousarray(a, dtype=np.int32)  # noqa: E731
    return dict(count=n, R=np.ascontiguousarray(R0.reshape(n, 3, 3, 3)), T=np.ascontiguousarray(T0.reshape(n, 3, 3)),
                focal=focal, tracks_of=i32(np.concatenate([[0], np.cumsum(counts)])),
                track_ptr=i32(np.concatenate([[0], np.cumsum(seen.sum(1))])), view=i32(np.nonzero(seen)[1]),
                pos=np.ascontiguousarray(q[seen], dtype=np.float32))


def _rotations(case, seed):
    """A view graph: neighbours along the capture order and random loop closures, in random order."""
    rng, n = np.random.default_rng(seed), case["views"]
    R = _expm(rng.normal(size=(n, 3)))
    near = np.concatenate([np.stack([np.arange(n - d), np.arange(d, n)], axis=1) for d in range(1, 6)])
    a, b = rng.integers(0, n, size=(2, 2 * case["pairs"]))
    far = np.unique((np.minimum(a, b) * n + np.maximum(a, b))[a != b])
    far = rng.permutation(far)[: max(0, case["pairs"] - len(near))]
    pairs = np.concatenate([near, np.stack([far // n, far % n], axis=1)])
    pairs = pairs[rng.permutation(len(pairs))]
    flip = rng.random(len(pairs)) < 0.5
    pairs[flip] = pairs[flip, ::-1]
    rel = _expm(rng.normal(scale=math.radians(1.0), size=(len(pairs), 3))) @ R[pairs[:, 1]] @ R[pairs[:, 0]].transpose(0, 2, 1)
    R0 = R @ _expm(rng.normal(scale=math.radians(5.0), size=(n, 3)))
    return np.ascontiguousarray(rel), np.ascontiguousarray(pairs, dtype=np.int32), np.ascontiguousarray(R0)


def _tracks(case, seed):
    rng, n = np.random.default_rng(seed), case["tracks"]
    # the same track lengths for every seed, in another order
    length = rng.permutation(np.where(np.arange(n) % 50 == 0, 0, 1 + np.random.default_rng(n).geometric(0.25, size=n)))
    ptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    K = int(ptr[-1])
    return dict(track_ptr=ptr, pos=rng.normal(size=(n, 3)), view=rng.integers(0, 500, size=K, dtype=np.int32),
                id=rng.integers(0, 1 << 20, size=K, dtype=np.int32),
                mpos=rng.uniform(0, 640, size=(K, 2)).astype(np.float32))


def _handle(case, s):
    h = capi.Handle(s["model"], s["mode"], s["thr"], s["K"], s["R"], s["T"], s["dist"], s["X"], s["meas"], s["view"],
                    s["point"], s.get("rig_K"), s.get("rig_R"), s.get("rig_T"), s.get("sub"))
    if case.get("fixed"):
        h.set_nonvarying(case["fixed"], 0, 0)
    return h


def _ba_options(case):
    o = dict(max_iterations=case["iterations"],
             precision=capi.PRECISION_FP64 if case["precision"] == "fp64" else capi.PRECISION_MIXED)
    if case.get("precond"):
        # tight enough that the adjusted parameters do not depend on where the solver stops
        o.update(solver=capi.SOLVER_PCG, pcg_tolerance=1e-10, pcg_max_iterations=2000,
                 preconditioner=capi.PRECOND_LEARNED if case["precond"] == "learned" else capi.PRECOND_BLOCK_JACOBI)
    return o


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ba":
        st = dict(case=case, scene=_ba_scene(case, seed), options=_ba_options(case))
        if case.get("precond") == "learned":
            st["precond"] = capi.PrecondModel.load(PRECOND_WEIGHTS)
        if case["keep"]:
            st["handle"] = _handle(case, st["scene"])
            if "precond" in st:
                st["handle"].set_precond_model(st["precond"])
        return st
    if kind == "triplets":
        st = dict(case=case, flat=_triplets(case, seed))
        if case["keep"]:
            st["batch"] = capi.Batch.from_flat(st["flat"])
        return st
    if kind == "stage":
        return dict(case=case, flat=_stage(case, seed))
    if kind == "rotations":
        st = dict(case=case, graph=_rotations(case, seed))
        if case["keep"]:
            st["graph_handle"] = capi.Rotations(*st["graph"])
        return st
    return dict(case=case, tracks=_tracks(case, seed))


# ---- one pass ------------------------------------------------------------------------------------


def _ba_out(s, params, r):
    K, R, T, dist, X = params
    out = dict(R=R, T=T, X=X, cost=float(r.cost), initial_cost=float(r.initial_cost), status=int(r.status),
               iterations=int(r.iterations))
    if s["model"] in (COMMON, VARYING):
        out.update(K=K, dist=dist)
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ba":
        h = state.get("handle")
        if h is not None:
            h.reset_params()
            r = h.minimize(**state["options"])
            return _ba_out(state["scene"], h.get_params(), r)
        h = _handle(case, state["scene"])
        if "precond" in state:
            h.set_precond_model(state["precond"])
        r = h.minimize(**state["options"])
        out = _ba_out(state["scene"], h.get_params(), r)
        h.close()
        return out
    if kind == "triplets":
        b = state.get("batch")
        if b is not None:
            b.reset()
        else:
            b = capi.Batch.from_flat(state["flat"])
        res, _ = b.minimize(max_iterations=case["iterations"])
        R, T, X = b.get_all_params()
        if state.get("batch") is None:
            b.close()
        return dict(R=R, T=T, X=X, cost=np.array([r.cost for r in res]),
                    iterations=np.array([r.iterations for r in res], dtype=np.int32))
    if kind == "stage":
        return capi.triplet_stage_flat(state["flat"], max_iterations=case["iterations"])
    if kind == "rotations":
        h = state.get("graph_handle")
        if h is not None:
            h.reset()
            r = h.minimize(max_iterations=8)
            return dict(R=h.get(), cost=float(r.cost), iterations=int(r.iterations))
        R, r = capi.refine_consistent_rotations(*state["graph"], max_iterations=8)
        return dict(R=R, cost=float(r.cost), iterations=int(r.iterations))
    return capi.bundle_point_structure(state["tracks"], case["required"])


# ---- what a pass cannot do without ----------------------------------------------------------------


def work(case):
    """Inputs read once and results written once; the arithmetic of the LM iterations (per
    observation the projection and its derivatives, per pair of a track's observations one block
    product, and the factorisation of the band or block-sparse camera system)."""
    kind = case["kind"]
    if kind == "ba":
        n, m = case["cams"], case["points"]
        track = {"circle": 4.0, "varying": 5.5, "sequence": 7.5, "stereo": 11.0, "cluster": 5.6}[case["scene"]]
        pairs = {"circle": 10.0, "varying": 18.0, "sequence": 33.0, "stereo": 66.0, "cluster": 26.0}[case["scene"]]
        da = 6 + (2 * case["mode"] - 1 if case["scene"] == "varying" and case["mode"] > 0 else 0)
        params = 8.0 * (24 * n + 6 * m)
        observations = (0.0 if case["keep"] else 24.0) * track * m
        system = n * da * (6.0 * 12) ** 2 if case["scene"] != "cluster" else 100.0 * 2 * 36 * 60 * n
        flops = case["iterations"] * (400.0 * track * m + pairs * m * (6.0 * da + 2.0 * da * da) + system)
        return dict(bytes=params + observations, flops=flops)
    if kind in ("triplets", "stage"):
        m = case["count"] * (case["lo"] + case["hi"]) / 2.0
        flops = case["iterations"] * m * (3 * 548.0 + 6 * 216.0 + 66.0)
        if kind == "stage":
            return dict(bytes=m * (36.0 + 4 + 24 + 3) + case["count"] * 480.0, flops=flops)
        return dict(bytes=m * (48.0 if case["keep"] else 24 + 72 + 24.0) + case["count"] * 600.0, flops=flops)
    if kind == "rotations":
        rel = (0.0 if case["keep"] else 80.0) * case["pairs"]
        return dict(bytes=rel + 144.0 * case["views"], flops=8 * 2 * 200.0 * case["pairs"])
    obs = 5.0 * case["tracks"]
    return dict(bytes=case["tracks"] * (28.0 + 28) + obs * (16.0 + 28), flops=0.0)


# ---- the same in plain FP64 torch -----------------------------------------------------------------


def _dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(dtype)


def _sum_to(n, index, values):
    return torch.zeros((n,) + values.shape[1:], dtype=values.dtype, device=values.device).index_add_(0, index, values)


def _cross(v):
    z = torch.zeros_like(v[:, 0])
    return torch.stack([z, -v[:, 2], v[:, 1], v[:, 2], z, -v[:, 0], -v[:, 1], v[:, 0], z], dim=1).view(-1, 3, 3)


def _rodrigues(w):
    th = w.norm(dim=1)[:, None, None]
    small = th <= 1e-6
    th = torch.where(small, torch.ones_like(th), th)
    J = _cross(w)
    eye = torch.eye(3, dtype=w.dtype, device=w.device)
    return torch.where(small, eye, eye + torch.sin(th) / th * J + (1 - torch.cos(th)) / th**2 * (J @ J))


class _Adjust:
    """Levenberg-Marquardt of many independent bundle problems side by side (a single adjustment
    is one problem): Huber weights frozen across a trial step, points eliminated, dense Cholesky of
    every problem's camera system, Nielsen's damping schedule."""

    def __init__(self, s, prob_cam, prob_pt, fixed=0):
        self.s, self.fixed = s, fixed
        self.model, self.mode = s["model"], s["mode"]
        self.ni = scenes.intrinsic_dim(self.mode) if self.model in (COMMON, VARYING) else 0
        self.dA = 6 + (self.ni if self.model == VARYING else 0)
        self.dC = self.ni if self.model == COMMON else 0
        self.pc, self.pp = prob_cam, prob_pt
        self.B = int(prob_cam.max()) + 1
        first = torch.full((self.B,), len(prob_cam), device="cuda").scatter_reduce_(
            0, prob_cam, torch.arange(len(prob_cam), device="cuda"), "amin")
        self.local = torch.arange(len(prob_cam), device="cuda") - first[prob_cam]
        self.n = int(self.local.max()) + 1
        self.cam, self.pt, self.meas = s["cam"], s["pt"], s["m"]
        order = torch.sort(self.pt, stable=True).indices
        self.cam, self.pt, self.meas = self.cam[order], self.pt[order], self.meas[order]
        self.sub = s["sub"][order] if self.model == STEREO else None
        self.po = self.pp[self.pt]
        self.M, self.N = len(self.pp), len(self.pc)
        count = torch.bincount(self.pt, minlength=self.M)
        self.start = count.cumsum(0) - count
        self.count = count
        self.ar = s["K"][..., 1, 1] / s["K"][..., 0, 0] if self.model == COMMON else None
        self.length = (_sum_to(self.B, self.pc, s["T"].square().sum(1) + 3.0)
                       + _sum_to(self.B, self.pp, s["X"].square().sum(1))).sqrt()

    def project(self, p, derivatives):
        R, T, X = p["R"][self.cam], p["T"][self.cam], p["X"][self.pt]
        v = (R @ X[:, :, None])[..., 0]
        Y = Z = v + T
        if self.model == STEREO:
            Rl, K = self.s["rig_R"][self.sub], self.s["rig_K"][self.sub]
            Z = (Rl @ Y[:, :, None])[..., 0] + self.s["rig_T"][self.sub]
        else:
            K = p["K"] if self.model == COMMON else p["K"][self.cam]
        P = torch.zeros(len(X), 2, 3, dtype=X.dtype, device=X.device)
        z = Z[:, 2]
        G = None
        if self.model in (STD, STEREO):
            h = (K @ Z[:, :, None])[..., 0]
            e = h[:, :2] / h[:, 2:] - self.meas
            if derivatives:
                fx = K[:, 0, 0]
                fy = K[:, 1, 1] / K[:, 0, 0] * fx
                P[:, 0, 0], P[:, 0, 2] = fx / z, -fx * Z[:, 0] / z**2
                P[:, 1, 1], P[:, 1, 2] = fy / z, -fy * Z[:, 1] / z**2
                if self.model == STEREO:
                    P = P @ Rl
        else:
            d = p["dist"] if self.model == COMMON else p["dist"][self.cam]
            k1, k2, p1, p2 = d.unbind(-1)
            x, y = Z[:, 0] / z, Z[:, 1] / z
            r2 = x * x + y * y
            kr = 1 + k1 * r2 + k2 * r2 * r2
            xd = kr * x + 2 * p1 * x * y + p2 * (r2 + 2 * x * x)
            yd = kr * y + 2 * p2 * x * y + p1 * (r2 + 2 * y * y)
            e = torch.stack([K[..., 0, 0] * xd + K[..., 0, 1] * yd + K[..., 0, 2], K[..., 1, 1] * yd + K[..., 1, 2]], dim=1)
            e = e - self.meas
            if derivatives:
                fx = K[..., 0, 0].expand(len(X))
                fy = (self.ar if self.model == COMMON else K[:, 1, 1] / K[:, 0, 0]) * fx
                dk = 2 * k1 + 4 * k2 * r2
                j00 = kr + x * x * dk + 2 * p1 * y + 6 * p2 * x
                j01 = x * y * dk + 2 * p1 * x + 2 * p2 * y
                j11 = kr + y * y * dk + 6 * p1 * y + 2 * p2 * x
                for r, (a, b, f) in enumerate(((j00, j01, fx), (j01, j11, fy))):
                    P[:, r, 0], P[:, r, 1], P[:, r, 2] = f * a / z, f * b / z, -f * (a * x + b * y) / z
                o, l = torch.zeros_like(x), torch.ones_like(x)
                G = torch.stack([
                    torch.stack([xd, l, o, fx * x * r2, fx * x * r2 * r2, 2 * fx * x * y, fx * (r2 + 2 * x * x)], dim=1),
                    torch.stack([yd, o, l, fy * y * r2, fy * y * r2 * r2, fy * (r2 + 2 * y * y), 2 * fy * x * y], dim=1)],
                    dim=1)[:, :, : self.ni]
        if not derivatives:
            return e
        A = torch.cat([P if not (self.model in (COMMON, VARYING) and self.mode == -1) else 0 * P, -P @ _cross(v)], dim=2)
        if self.model == VARYING:
            A = torch.cat([A, G], dim=2)
        C = G if self.model == COMMON and self.dC else torch.zeros(len(X), 2, 0, dtype=X.dtype, device=X.device)
        return e, A, P @ R, C

    def linearize(self, p):
        e, A, B, C = self.project(p, True)
        norm = e.norm(dim=1)
        thr = self.s["thr"][self.po]
        w = torch.where(norm < thr, torch.ones_like(norm), (thr / norm).sqrt())
        A, B, C = A * w[:, None, None], B * w[:, None, None], C * w[:, None, None]
        A[self.local[self.cam] < self.fixed] = 0.0
        r = (-w[:, None] * e)[:, :, None]
        At, Bt, Ct = A.mT, B.mT, C.mT
        L = dict(A=A, B=B, C=C, w=w, err=_sum_to(self.B, self.po, r.square().sum((1, 2))),
                 U=_sum_to(self.N, self.cam, At @ A), X=_sum_to(self.N, self.cam, At @ C),
                 ga=_sum_to(self.N, self.cam, (At @ r)[..., 0]), V=_sum_to(self.M, self.pt, Bt @ B),
                 Y=_sum_to(self.M, self.pt, Bt @ C), gb=_sum_to(self.M, self.pt, (Bt @ r)[..., 0]),
                 Z=_sum_to(self.B, self.po, Ct @ C), gc=_sum_to(self.B, self.po, (Ct @ r)[..., 0]))
        return L

    def step(self, L, lam):
        B, n, dA, dC = self.B, self.n, self.dA, self.dC
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        Vi = torch.linalg.inv(L["V"] + lam[self.pp][:, None, None] * eye)
        q = (Vi @ L["gb"][:, :, None])[..., 0]
        W = L["A"].mT @ L["B"]
        Wv = W @ Vi[self.pt]
        blocks = torch.zeros(B * n * n, dA * dA, dtype=torch.float64, device="cuda")
        bound = (self.count * self.count).cumsum(0)
        a, size = 0, 6_000_000
        while a < self.M:                       # all ordered pairs of a track's observations, in pieces
            base = int(bound[a - 1]) if a else 0
            b = max(a + 1, int(torch.searchsorted(bound, base + size, right=True)))
            c = self.count[a:b]
            of = torch.repeat_interleave(torch.arange(a, b, device="cuda"), c * c)
            at = torch.arange(len(of), device="cuda") - (bound[a:b] - c * c - base)[of - a]
            k, m = self.start[of] + at // self.count[of], self.start[of] + at % self.count[of]
            i, l = self.cam[k], self.cam[m]
            blocks.index_add_(0, (self.pc[i] * n + self.local[i]) * n + self.local[l], -(Wv[k] @ W[m].mT).reshape(len(of), -1))
            a = b
        own = (self.pc * n + self.local) * n + self.local
        blocks.index_add_(0, own, (L["U"] + lam[self.pc][:, None, None] * torch.eye(dA, dtype=torch.float64, device="cuda")).reshape(self.N, -1))
        S = torch.zeros(B, n * dA + dC, n * dA + dC, dtype=torch.float64, device="cuda")
        S[:, : n * dA, : n * dA] = blocks.view(B, n, n, dA, dA).transpose(2, 3).reshape(B, n * dA, n * dA)
        rhs = torch.zeros(B, n * dA + dC, dtype=torch.float64, device="cuda")
        slot = self.pc * n + self.local
        ga = L["ga"] - _sum_to(self.N, self.cam, (W @ q[self.pt][:, :, None])[..., 0])
        rhs[:, : n * dA] = _sum_to(B * n, slot, ga).view(B, -1)
        if dC:
            ViY = Vi @ L["Y"]
            edge = _sum_to(B * n, slot, L["X"] - _sum_to(self.N, self.cam, W @ ViY[self.pt])).view(B, n * dA, dC)
            S[:, : n * dA, n * dA:], S[:, n * dA:, : n * dA] = edge, edge.mT
            S[:, n * dA:, n * dA:] = (L["Z"] + lam[:, None, None] * torch.eye(dC, dtype=torch.float64, device="cuda")
                                      - _sum_to(B, self.pp, L["Y"].mT @ ViY))
            rhs[:, n * dA:] = L["gc"] - _sum_to(B, self.pp, (L["Y"].mT @ q[:, :, None])[..., 0])
        if self.fixed:
            k = self.fixed * dA
            S[:, :k], S[:, :, :k], rhs[:, :k] = 0.0, 0.0, 0.0
            S[:, range(k), range(k)] = 1.0
        x = torch.cholesky_solve(rhs[:, :, None], torch.linalg.cholesky(S))[..., 0]
        da = x[:, : n * dA].reshape(B * n, dA)[slot]
        dc = x[:, n * dA:]
        back = _sum_to(self.M, self.pt, (W.mT @ da[self.cam][:, :, None])[..., 0])
        if dC:
            back = back + (L["Y"] @ dc[self.pp][:, :, None])[..., 0]
        return da, q - (Vi @ back[:, :, None])[..., 0], dc

    def moved(self, p, da, db, dc):
        t = dict(p, R=_rodrigues(da[:, 3:6].contiguous()) @ p["R"], T=p["T"] + da[:, :3], X=p["X"] + db)
        if self.model in (COMMON, VARYING) and self.ni:
            K, dist = p["K"].clone(), p["dist"].clone()
            d = dc[0] if self.model == COMMON else da[:, 6:]
            ar = self.ar if self.model == COMMON else K[:, 1, 1] / K[:, 0, 0]
            if self.ni >= 7:
                dist[..., 2] += d[..., 5]
                dist[..., 3] += d[..., 6]
            if self.ni >= 5:
                dist[..., 0] += d[..., 3]
                dist[..., 1] += d[..., 4]
            if self.ni >= 3:
                K[..., 0, 2] += d[..., 1]
                K[..., 1, 2] += d[..., 2]
            K[..., 0, 0] += d[..., 0]
            K[..., 1, 1] = ar * K[..., 0, 0]
            t.update(K=K, dist=dist)
        return t

    def minimize(self, iterations, tau=1e-3):
        p = {k: self.s[k] for k in ("K", "R", "T", "dist", "X")}
        B = self.B
        live = torch.ones(B, dtype=torch.bool, device="cuda")
        lam = nu = cost = first = None
        done = torch.zeros(B, dtype=torch.int32, device="cuda")
        status = torch.zeros(B, dtype=torch.int32, device="cuda")
        for it in range(iterations):
            L = self.linearize(p)
            cost = L["err"] if cost is None else torch.where(live, L["err"], cost)
            gmax = torch.zeros(B, dtype=torch.float64, device="cuda")
            dmax = torch.zeros_like(gmax)
            vary = self.local >= self.fixed
            for owner, g, D in ((self.pc[vary], L["ga"][vary], L["U"][vary]), (self.pp, L["gb"], L["V"]),
                                (torch.arange(B, device="cuda"), L["gc"], L["Z"])):
                if g.shape[1]:
                    gmax.scatter_reduce_(0, owner, g.abs().amax(1), "amax")
                    dmax.scatter_reduce_(0, owner, D.diagonal(dim1=1, dim2=2).amax(1), "amax")
            if it == 0:
                first, lam, nu = L["err"], tau * dmax, torch.full_like(dmax, 2.0)
            stop = live & (gmax < 1e-10)
            status[stop] = 2
            live = live & ~stop
            da, db, dc = self.step(L, lam)
            d2 = _sum_to(B, self.pc, da.square().sum(1)) + _sum_to(B, self.pp, db.square().sum(1)) + dc.square().sum(1)
            dg = (_sum_to(B, self.pc, (da * L["ga"]).sum(1)) + _sum_to(B, self.pp, (db * L["gb"]).sum(1))
                  + (dc * L["gc"]).sum(1))
            stop = live & (d2.sqrt() < 1e-10 * (self.length + 1e-10))
            status[stop] = 1
            live = live & ~stop
            t = self.moved(p, da, db, dc)
            new = _sum_to(B, self.po, (L["w"][:, None] * self.project(t, False)).square().sum(1))
            rho = (L["err"] - new) / (lam * d2 + dg)
            ok = live & (rho > 0)
            if B == 1:
                p = t if bool(ok) else p
            else:
                for key, owner in (("R", self.pc), ("T", self.pc), ("X", self.pp)):
                    m = ok[owner].view((-1,) + (1,) * (p[key].dim() - 1))
                    p[key] = torch.where(m, t[key], p[key])
            lam = torch.where(ok, (lam * torch.clamp(1 - (2 * rho - 1) ** 3, min=1 / 3)).clamp(min=1e-10), lam * nu)
            nu = torch.where(ok, torch.full_like(nu, 2.0), nu * 2)
            done += live.int()
            if not bool(live.any()):
                break
        return p, cost, first, status, done


def _host(t):
    return t.cpu().numpy()


def _exact_ba(case, s):
    s = dict(s)
    n, m = len(s["R"]), len(s["X"])
    s.update(cam=_dev(s["view"], torch.int64), pt=_dev(s["point"], torch.int64), m=_dev(s["meas"]),
             thr=_dev([s["thr"]]), dist=_dev(s["dist"] if s["dist"] is not None else np.zeros(4)))
    for k in ("K", "R", "T", "X", "rig_K", "rig_R", "rig_T"):
        if s.get(k) is not None:
            s[k] = _dev(s[k])
    if s.get("sub") is not None:
        s["sub"] = _dev(s["sub"], torch.int64)
    zero = lambda k: torch.zeros(k, dtype=torch.int64, device="cuda")  # noqa: E731
    p, cost, first, _, _ = _Adjust(s, zero(n), zero(m), case.get("fixed", 0)).minimize(case["iterations"])
    out = dict(R=_host(p["R"]), T=_host(p["T"]), X=_host(p["X"]), cost=float(cost[0]), initial_cost=float(first[0]),
               status=None, iterations=None)
    if s["model"] in (COMMON, VARYING):
        out.update(K=_host(p["K"]), dist=_host(p["dist"]))
    return out


def _exact_triplets(case, f):
    n = len(f["n_cams"])
    prob_pt = torch.repeat_interleave(torch.arange(n, device="cuda"), _dev(f["n_points"], torch.int64))
    prob_cam = torch.arange(n, device="cuda").repeat_interleave(3)
    owner = prob_pt.repeat_interleave(3)
    first = _dev(np.cumsum(f["n_points"]) - f["n_points"], torch.int64)
    s = dict(model=STD, mode=0, K=_dev(f["K"]), R=_dev(f["R"]), T=_dev(f["T"]), X=_dev(f["X"]), dist=None,
             thr=_dev(f["thr"]), m=_dev(f["meas"]), cam=_dev(f["view"], torch.int64) + 3 * owner,
             pt=_dev(f["point"], torch.int64) + first[owner])
    p, cost, _, _, _ = _Adjust(s, prob_cam, prob_pt).minimize(case["iterations"])
    return dict(R=_host(p["R"]), T=_host(p["T"]), X=_host(p["X"]), cost=_host(cost), iterations=None)


def _exact_stage(case, f):
    """Linear triangulation, the float filter of the measurements, the survival tests, and the
    adjustment of the survivors with K = I."""
    n = f["count"]
    R, T, pos = _dev(f["R"]).view(-1, 3, 3), _dev(f["T"]).view(-1, 3), _dev(f["pos"])
    ptr, of = _dev(f["track_ptr"], torch.int64), _dev(f["tracks_of"], torch.int64)
    tracks = ptr[1:] - ptr[:-1]
    owner = torch.repeat_interleave(torch.arange(n, device="cuda"), of[1:] - of[:-1])
    track = torch.repeat_interleave(torch.arange(len(tracks), device="cuda"), tracks)
    view = _dev(f["view"], torch.int64)
    cam = 3 * owner[track] + view
    P = torch.cat([R, T[:, :, None]], dim=2)[cam]
    rows = pos[:, :, None] * P[:, 2:3] - P[:, :2]                   # (measurements, 2, 4)
    A = torch.zeros(len(tracks), 3, 2, 4, dtype=torch.float64, device="cuda")
    A[track, torch.arange(len(track), device="cuda") - ptr[track]] = rows
    A = A.view(-1, 6, 4)
    A[..., 3] *= -1.0
    cols = list(A.unbind(2))                                        # modified Gram-Schmidt of [A | b]
    r = {}
    for i in range(3):
        r[i, i] = cols[i].norm(dim=1)
        cols[i] = cols[i] / r[i, i][:, None]
        for j in range(i + 1, 4):
            r[i, j] = (cols[i] * cols[j]).sum(1)
            cols[j] = cols[j] - r[i, j][:, None] * cols[i]
    x2 = r[2, 3] / r[2, 2]
    x1 = (r[1, 3] - r[1, 2] * x2) / r[1, 1]
    x0 = (r[0, 3] - r[0, 2] * x2 - r[0, 1] * x1) / r[0, 0]
    X = torch.stack([x0, x1, x2], dim=1)
    y = (R[cam] @ X[track][:, :, None])[..., 0] + T[cam]
    d = (y[:, :2] / y[:, 2:]).float() - pos.float()
    dist = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).double().sqrt().float().double()
    kept = _dev(f["focal"])[owner[track], view] * dist < 1.0
    good = _sum_to(len(tracks), track, kept.int()) >= 3
    survivors, before = _sum_to(n, owner, good.int()), _sum_to(n, owner, torch.ones_like(owner))
    accepted = (survivors >= 50) & (survivors.double() >= 0.5 * before.double())
    cost = torch.zeros(n, dtype=torch.float64, device="cuda")
    R, T, X = R.clone(), T.clone(), X.clone()
    if bool(accepted.any()):
        ids = torch.cumsum(accepted.int(), 0) - 1
        pts = good & accepted[owner]
        new = torch.cumsum(pts.int(), 0) - 1
        use = kept & pts[track]
        mine = accepted.repeat_interleave(3)
        count = int(accepted.sum())
        s = dict(model=STD, mode=0, K=torch.eye(3, dtype=torch.float64, device="cuda").expand(3 * count, 3, 3),
                 R=R[mine], T=T[mine], X=X[pts], dist=None, thr=torch.ones(count, dtype=torch.float64, device="cuda"),
                 m=pos[use], cam=(3 * ids[owner[track]] + view)[use].long(), pt=new[track][use].long())
        p, c, _, _, _ = _Adjust(s, torch.arange(count, device="cuda").repeat_interleave(3),
                                ids[owner][pts].long()).minimize(case["iterations"])
        R[mine], T[mine], X[pts], cost[accepted] = p["R"], p["T"], p["X"], c
    return dict(R=_host(R.view(n, 3, 3, 3)), T=_host(T.view(n, 3, 3)), X=_host(X), cost=_host(cost))


def _exact_rotations(rel, pairs, R0):
    """Each view's 3x3 damped block solved on its own, as the residual attaches one measurement of
    every pair to either view."""
    rel, R = _dev(rel), _dev(R0)
    i, j = _dev(pairs, torch.int64).unbind(1)
    n = len(R)
    unit = _cross(torch.eye(3, dtype=torch.float64, device="cuda"))

    def residual(R):
        return R[j] - rel @ R[i]

    lam, nu, cost = None, 2.0, 0.0
    for it in range(8):
        e = residual(R)
        err = float(2 * e.square().sum())
        cost = err
        U, g = torch.zeros(n, 3, 3, dtype=torch.float64, device="cuda"), torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        for at, M in ((i, -rel @ R[i]), (j, R[j])):
            J = (M[:, None] @ unit).reshape(len(M), 3, 9)
            U.index_add_(0, at, J @ J.mT)
            g.index_add_(0, at, -(J @ e.reshape(-1, 9, 1))[..., 0])
        if lam is None:
            lam = 1e-3 * float(U.diagonal(dim1=1, dim2=2).max())
        d = torch.linalg.solve(U + lam * torch.eye(3, dtype=torch.float64, device="cuda"), g[:, :, None])[..., 0]
        if float(d.norm()) < 1e-10 * (math.sqrt(3.0 * n) + 1e-10):
            break
        new = R @ _rodrigues(d)
        rho = (err - float(2 * residual(new).square().sum())) / (lam * float(d.square().sum()) + float((d * g).sum()))
        if rho > 0:
            R, lam, nu = new, max(lam * max(1 / 3, 1 - (2 * rho - 1) ** 3), 1e-10), 2.0
        else:
            lam, nu = lam * nu, 2 * nu
    return dict(R=_host(R), cost=cost, iterations=None)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ba":
        return _exact_ba(case, _ba_scene(case, seed))
    if kind == "triplets":
        return _exact_triplets(case, _triplets(case, seed))
    if kind == "stage":
        return _exact_stage(case, _stage(case, seed))
    if kind == "rotations":
        return _exact_rotations(*_rotations(case, seed))
    t = _tracks(case, seed)
    length = np.diff(t["track_ptr"])
    keep = length >= case["required"]
    return dict(points3d=t["pos"][keep], measurements=t["mpos"][np.repeat(keep, length)].astype(np.float64))
