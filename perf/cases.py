"""The performance cases: what users of this framework have it do, through its public entry points.

* ``run``     — a whole program: constructors, ``run_simulation``, the converged node state.
* ``trial``   — one HHT step of a kept engine that ends back at the committed state, as the time
  loop does it with a step that it rejects (run_simulations: loads, step, result, rollback).
* ``retry``   — the time loop's Δt halving: a step at Δt is rejected and taken again at Δt/2, so
  the preconditioner of the changed tangent has to be factorised anew in each of the two steps.
* ``contact`` — the contact element with caller-owned device buffers (eb_contact_eval_noalloc).
* ``meshsdf`` — a vessel mesh to the signed distance grid that the contact uses (from_mesh).
* ``mlptrain``, ``mlpgrad``, ``mlpforward`` — training, gradient and inference of the learned warm start.

Scenes are those of the package's ``scenes`` module with sizes, velocities and radii varied by the
seed.  All times are of the steady state of a user's loop: engines, plans and models are kept.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "endobeams.jl_gb300")


def _eb():
    if "endobeams_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("endobeams_gb300", os.path.join(PKG, "__init__.py"),
                                                      submodule_search_locations=[PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["endobeams_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["endobeams_gb300"]


def _scenes():
    _eb()
    from endobeams_gb300 import scenes
    return scenes


def listed():
    return [
        # the smallest whole program: the clamped beam of the package's smoke test, 20 steps
        dict(name="run_cantilever", kind="run", scene="cantilever", n=20, steps=20),
        # smallest contact scene, one simulation, FP64 throughout: a ring on the ground plane
        dict(name="trial_ring64", kind="trial", scene="ring", n=64, sims=1, surface="plane"),
        # one mid-sized net on a sphere SDF, FP64 throughout
        dict(name="trial_net33", kind="trial", scene="net", n=33, sims=1),
        # a batch of nets of mixed sizes (20 to 40 nodes a side) that share one SDF
        dict(name="trial_nets16", kind="trial", scene="net", n=40, sims=16),
        # one stent of few wires with long wire segments between the crossings
        dict(name="trial_stent16x250", kind="trial", scene="stent", wires=16, n=250, sims=1, solver="scene"),
        # one stent of an odd size, the settings of the population runs
        dict(name="trial_stent24x150", kind="trial", scene="stent", wires=24, n=150, sims=1, solver="batch"),
        # the single full-size stent (48 wires, 200 elements a wire)
        dict(name="trial_stent48x200", kind="trial", scene="stent", wires=48, n=200, sims=1, solver="scene"),
        # Δt halving: two factorisations and two steps
        dict(name="retry_stent32x121", kind="retry", scene="stent", wires=32, n=121, sims=1, solver="batch"),
        # a small stent population with the settings of the population runs and the learned initial guess
        dict(name="trial_stents8", kind="trial", scene="stent", wires=0, n=220, sims=8, solver="batch"),
        # contact elements of a caller with its own device memory, quadratic SDF of 61 points an axis
        dict(name="contact_20011", kind="contact", n=20011, grid=61),
        # a closed vessel-like mesh onto a 64³ grid
        dict(name="meshsdf_5120x64", kind="meshsdf", sub=4, grid=64),
        # one epoch of training of the warm-start network
        dict(name="mlptrain_65536", kind="mlptrain", n=65536, batch=8192),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "trial", "trial", "trial", "trial", "retry", "contact", "meshsdf", "mlpgrad", "mlpforward"])
    if kind == "run":
        return dict(kind="run", scene="cantilever", n=_logint(rng, 7, 90), steps=rng.randint(5, 20))
    if kind == "trial":
        scene = rng.choice(["ring", "net", "stent", "stent"])
        if scene == "ring":
            return dict(kind="trial", scene="ring", n=_logint(rng, 24, 400), sims=1, surface=rng.choice(["plane", "sdf"]))
        if scene == "net":
            sims = _logint(rng, 1, 12)
            return dict(kind="trial", scene="net", n=rng.randint(20, 40), sims=sims)
        sims = _logint(rng, 1, 4)
        return dict(kind="trial", scene="stent", wires=rng.choice([16, 24, 32]) if sims == 1 else 0,
                    n=rng.randint(100, 210), sims=sims, solver=rng.choice(["scene", "batch"]))
    if kind == "retry":
        return dict(kind="retry", scene="stent", wires=rng.choice([16, 24, 32]), n=rng.randint(100, 170), sims=1,
                    solver=rng.choice(["scene", "batch"]))
    if kind == "contact":
        return dict(kind="contact", n=_logint(rng, 300, 20000), grid=rng.randint(21, 64))
    if kind == "meshsdf":
        sub = rng.randint(1, 4)
        return dict(kind="meshsdf", sub=sub, grid=rng.randint(15, 63))
    return dict(kind=kind, n=_logint(rng, 500, 60000))


# ------------------------------------------------------------------ scenes


def _build(case, seed):
    """(confs, params, inters) of a case: public constructors, sizes of the case, values of the seed."""
    S = _scenes()
    rng = np.random.default_rng([seed, case["n"], 7])
    confs, inters = [], []
    if case["scene"] == "cantilever":
        conf, params, inter = S.cantilever(n_elem=case["n"], steps=case["steps"])
        conf.nodes.ud[1:] = 0.2 * rng.standard_normal((len(conf.nodes) - 1, 3)) * np.array([1e-3, 1.0, 1.0])
        conf.nodes.udn = conf.nodes.ud.copy()
        conf.beams.E *= rng.uniform(0.8, 1.2)
        params.tolerance_residual = 1e-5
        return [conf], params, [inter]
    if case["scene"] == "ring":
        conf, params, inter = S.ring_drop(n_elem=case["n"], surface=case["surface"], height=rng.uniform(1.0e-4, 1.5e-4))
        conf.nodes.ud[:] = rng.uniform(0.8, 1.2) * np.array([0.05, 0.0, -0.1])
        conf.nodes.udn = conf.nodes.ud.copy()
        params.tolerance_residual = 1e-5
        return [conf], params, [inter]
    if case["scene"] == "net":
        sdf = S.sphere_sdf()
        for s in range(case["sims"]):
            # sides from 20 to the case's largest, the same ones for every seed
            side = case["n"] if s == 0 else 20 + (7 * s) % max(1, case["n"] - 19)
            conf, params, inter = S.net_on_sphere(side, seed=1000 * (seed % 1000003) + s, sdf=sdf, drop=rng.uniform(-5e-5, -2e-5))
            conf.nodes.ud[:] = np.array([0.0, 0.0, -0.05]) * rng.uniform(0.8, 1.2)
            conf.nodes.udn = conf.nodes.ud.copy()
            confs.append(conf)
            inters.append(inter)
        params.tolerance_residual = 1e-5
        return confs, params, inters
    tols = []
    for s in range(case["sims"]):
        wires = case["wires"] or (16, 24, 32, 48)[s % 4]
        # one simulation: the case's size; a population: sizes from 100 elements a wire up to it
        n = case["n"] if case["sims"] == 1 else 100 + (37 * s) % (case["n"] - 99)
        R = rng.uniform(3.97e-3, 4.03e-3)
        # every q-th node of a wire is a crossing: the q of a 4 mm, 45 degree stent of 20 mm, so that the
        # node count does not depend on the seed
        q = max(1, round(n * math.pi * 4e-3 / (wires // 2 * 0.02)))
        conf, params, inter = S.braided_stent(wires=wires, R=R, pitch_deg=rng.uniform(44.8, 45.2), elems_per_wire=n,
                                              crossing_every=q, grid=None, cyl_radius=R * rng.uniform(0.87, 0.9))
        conf.nodes.ud[:] = 1e-2 * rng.standard_normal(3)
        conf.nodes.udn = conf.nodes.ud.copy()
        X, c = conf.nodes.X0, conf.beams.conn
        le = np.linalg.norm(X[c[:, 1]] - X[c[:, 0]], axis=1).mean()
        tols.append(1e-8 if le >= 1.2e-4 else 1e-7)
        confs.append(conf)
        inters.append(inter)
    if case["solver"] == "batch":  # the settings that the population benchmark steps its stents with
        params.krylov_restart = 32
        params.refactor_its = 200
        params.refactor_policy = "cost"
        params.refactor_cost = 0.12
        params.band_lu = "tensor"
        params.linear_tol = 1e-4
        if case["sims"] > 1:
            params.warm_start = "learned_x0"
    params.tolerance_residual = max(tols)
    return confs, params, inters


def _icosphere(sub, rng):
    """A closed triangle mesh (20·4^sub triangles) of a bumpy, stretched sphere; 1-based triangles."""
    g = (1 + math.sqrt(5)) / 2
    V = [(-1, g, 0), (1, g, 0), (-1, -g, 0), (1, -g, 0), (0, -1, g), (0, 1, g), (0, -1, -g), (0, 1, -g),
         (g, 0, -1), (g, 0, 1), (-g, 0, -1), (-g, 0, 1)]
    T = np.array([(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2),
                  (10, 7, 6), (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11),
                  (6, 2, 10), (8, 6, 7), (9, 8, 1)])
    V = np.array(V, float)
    V /= np.linalg.norm(V, axis=1)[:, None]
    for _ in range(sub):
        E = np.sort(np.concatenate([T[:, [0, 1]], T[:, [1, 2]], T[:, [2, 0]]]), axis=1)
        U, inv = np.unique(E, axis=0, return_inverse=True)
        M = V[U[:, 0]] + V[U[:, 1]]
        M /= np.linalg.norm(M, axis=1)[:, None]
        m = inv.reshape(3, -1) + len(V)
        a, b, c = T.T
        T = np.concatenate([np.stack(t, 1) for t in ((a, m[0], m[2]), (b, m[1], m[0]), (c, m[2], m[1]), (m[0], m[1], m[2]))])
        V = np.concatenate([V, M])
    k = rng.uniform(1.0, 2.0, (6, 3))
    ph = rng.uniform(0, 2 * np.pi, 6)
    r = 4e-3 * (1 + 0.03 * np.sin(V @ k.T + ph).sum(1))
    return V * r[:, None] * np.array([1.0, 0.8, 1.3]), T + 1


def _contact_records(n, rng):
    """n packed element records (96 doubles: positions, displacements, rotations, increments, velocities,
    l0, Rₑ⁰, stiffness, inertia, radius) of 0.3 mm wire elements around a 10 mm sphere, about half touching."""
    r = np.zeros((n, 96))
    c = rng.standard_normal((n, 3))
    c *= ((0.010 + rng.uniform(-0.5e-4, 1.2e-4, n)) / np.linalg.norm(c, axis=1))[:, None]
    t = np.cross(c, rng.standard_normal((n, 3)))
    t /= np.linalg.norm(t, axis=1)[:, None]
    l0 = rng.uniform(2e-4, 4e-4, n)
    X1, X2 = c - 0.5 * l0[:, None] * t, c + 0.5 * l0[:, None] * t

    def rot(th):  # n rotation vectors -> column-major rotation matrices
        a = np.linalg.norm(th, axis=1)[:, None, None]
        K = np.zeros((n, 3, 3))
        K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -th[:, 2], th[:, 1], -th[:, 0]
        K -= K.transpose(0, 2, 1)
        M = np.eye(3) + np.sin(a) / a * K + (1 - np.cos(a)) / a ** 2 * (K @ K)
        return M

    e3 = np.cross(t, c)
    e3 /= np.linalg.norm(e3, axis=1)[:, None]
    Re0 = np.stack([t, np.cross(e3, t), e3], axis=2)
    f = lambda M: M.transpose(0, 2, 1).reshape(n, 9)
    r[:, 0:3], r[:, 3:6] = X1, X2
    r[:, 6:12] = 1e-6 * rng.standard_normal((n, 6))
    r[:, 12:21], r[:, 21:30] = f(rot(0.02 * rng.standard_normal((n, 3)))), f(rot(0.02 * rng.standard_normal((n, 3))))
    r[:, 30:39], r[:, 39:48] = f(rot(0.005 * rng.standard_normal((n, 3)))), f(rot(0.005 * rng.standard_normal((n, 3))))
    r[:, 48:60] = 0.05 * rng.standard_normal((n, 12))
    r[:, 60:72] = 10.0 * rng.standard_normal((n, 12))
    r[:, 72] = l0
    r[:, 73:82] = f(Re0)
    E, rho, rad = 5e10, 6500.0, 5e-5
    A, I = math.pi * rad ** 2, math.pi * rad ** 4 / 4
    G = E / 2.66
    for k, v in enumerate((E * A, 2 * G * I, 4 * E * I, 4 * E * I, -2 * G * I, 2 * E * I, 2 * E * I)):
        r[:, 82 + k] = v / l0
    r[:, 89:92] = rho * 2 * I, rho * I, rho * I
    r[:, 92], r[:, 94] = rho * A, rad
    return r


# ------------------------------------------------------------------ the cases


def prepare(case, seed):
    kind = case["kind"]
    eb = _eb()
    if kind == "run":
        (conf,), params, (inter,) = _build(case, seed)
        nd = conf.nodes
        return dict(case=case, X=nd.X0, ud=nd.ud.copy(), conn=conf.beams.conn + 1, E=conf.beams.E.copy(), conf=conf,
                    params=params)
    if kind in ("trial", "retry"):
        confs, params, inters = _build(case, seed)
        eng = eb.GpuSimulations(confs, params, inters)
        if params.warm_start != "off":
            from endobeams_gb300 import warm_start as W
            eng.set_warm_start(W.WarmStartModel.load(os.path.join(PKG, "models", "warm_start_stents.npz")))
        dt = params.initial_timestep
        if case["scene"] == "stent":
            eng.set_tolerances(residual=params.tolerance_residual)
        loads = eng.loads_all(dt)
        return dict(case=case, eng=eng, dt=np.full(eng.n, dt), loads=loads)
    rng = np.random.default_rng([seed, case.get("n", 0), 11])
    if kind == "contact":
        n, g = case["n"], case["grid"]
        h = 0.0225 / (g - 1)
        xs = -h * (g - 1) / 2 + h * np.arange(g)
        Z, Y, Xg = np.meshgrid(xs, xs, xs, indexing="ij")
        sdf = np.sqrt(Xg ** 2 + Y ** 2 + Z ** 2) - 0.010 * (1 + 0.01 * rng.standard_normal())
        dev = torch.device("cuda")
        return dict(case=case, inp=torch.from_numpy(_contact_records(n, rng)).to(dev), sdf=torch.from_numpy(sdf).to(dev),
                    out=torch.zeros((n, 301), dtype=torch.float64, device=dev),
                    flags=torch.zeros(n, dtype=torch.int32, device=dev), gauss=np.ascontiguousarray(eb.GAUSS),
                    props=np.array([1e4, 0.1, 1e-3, 1e-3]),
                    surf=np.array([1, 0, 0, 0, 0, g, g, g, xs[0], xs[0], xs[0], h, h, h], float))
    if kind == "meshsdf":
        V, T = _icosphere(case["sub"], rng)
        g = case["grid"]
        lo, hi = V.min(0), V.max(0)
        h = float((hi - lo).max()) / (g - 7)
        o = (lo + hi) / 2 - h * (g - 1) / 2
        return dict(case=case, V=V, T=T, origin=o, h=h, dims=(g, g, g))
    n = case["n"]
    X = np.zeros((n, 48), np.float32)
    X[:, :39] = rng.standard_normal((n, 39))
    Tg = rng.standard_normal((n, 6)).astype(np.float32)
    from endobeams_gb300 import warm_start as W
    p = W.init_params(seed % 100003, out_gain=1.0)
    p[48 * 128:48 * 128 + 128] = 0.1 * rng.standard_normal(128)
    return dict(case=case, X=X, T=Tg, p=p)


def run(state):
    case = state["case"]
    kind = case["kind"]
    eb = _eb()
    if kind == "run":
        c0 = state["conf"]
        nodes = eb.NodesBeams(state["X"], None, state["ud"])
        beams = eb.Beams(nodes, state["conn"], state["E"], 0.33, 7850.0, 5e-4, 0.0)
        conf = eb.BeamsConfiguration(nodes, beams, c0.loads, c0.bcs)
        res = eb.run_simulation(conf, state["params"])
        return dict(u=nodes.un, ud=nodes.udn, udd=nodes.uddn, wd=nodes.wdn, R=nodes.Rn, k=np.asarray(res.ks[0]))
    if kind in ("trial", "retry"):
        eng = state["eng"]
        eng.set_loads_all(state["loads"])
        k, st = eng.step(state["dt"])
        if kind == "retry":
            eng.rollback()
            eng.set_loads_all(state["loads"])
            k, st = eng.step(0.5 * state["dt"])
        if eng.n == 1:
            out = eng.state(0)
        else:
            out = dict(u=eng.displacements())
        eng.rollback()
        # w is the predictor's scratch rotation (the corrector does not write it): not a converged result
        out = {f: out[f] for f in ("u", "ud", "udd", "wd", "wdd", "R", "dR") if f in out}
        if case.get("solver") != "batch":  # under inexact Newton (linear_tol 1e-4) the count is solver statistics
            out["k"] = k
        return out
    if kind == "contact":
        from endobeams_gb300 import _lib
        p = lambda a: _lib.ptr(a)
        v = lambda x: ctypes.c_void_p(x.data_ptr())
        _lib.check(_lib.load().eb_contact_eval_noalloc(case["n"], v(state["inp"]), p(state["gauss"]), p(state["props"]),
                                                       p(state["surf"]), v(state["sdf"]), v(state["out"]),
                                                       v(state["flags"]),
                                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return dict(out=state["out"], flags=state["flags"])
    if kind == "meshsdf":
        return eb.DiscreteSignedDistanceField.from_mesh(state["V"], state["T"], state["origin"], state["h"],
                                                        state["dims"]).values
    from endobeams_gb300 import warm_start as W
    if kind == "mlpforward":
        return W.mlp_forward(state["p"], state["X"])
    if kind == "mlpgrad":
        loss, g = W.mlp_loss_grad(state["p"], state["X"], state["T"])
        return dict(loss=loss, grad=g)
    p, losses = W.mlp_train(state["p"], state["X"], state["T"], epochs=1, batch=case["batch"], seed=3)
    return dict(params=p, loss=losses)


def work(case):
    kind = case["kind"]
    if kind == "contact":
        # records and grid read, outputs written; every element's frame and three distance lookups, half of the
        # elements with all three Gauss points in contact
        return dict(bytes=case["n"] * (96 * 8 + 301 * 8 + 4) + 8 * case["grid"] ** 3,
                    flops=case["n"] * (6843 + 0.5 * 3 * 9413))
    if kind == "meshsdf":
        tri, pts = 20 * 4 ** case["sub"], case["grid"] ** 3
        return dict(bytes=72 * tri + 8 * pts, flops=150.0 * tri * pts)
    if kind in ("mlptrain", "mlpgrad", "mlpforward"):
        f = 2.0 * (48 * 128 + 128 * 128 + 128 * 6) * (1 if kind == "mlpforward" else 3)
        return dict(bytes=case["n"] * (4 * 48 + 4 * 6) + 2 * 4 * 23558, flops=case["n"] * f)
    # a step: node state read and written, the element and contact matrices of two Newton iterations evaluated
    if case["scene"] in ("cantilever", "ring"):
        ne = nn = case["n"]
    elif case["scene"] == "net":
        sides = [case["n"] if s == 0 else 20 + (7 * s) % max(1, case["n"] - 19) for s in range(case["sims"])]
        nn, ne = sum(x * x for x in sides), sum(2 * x * (x - 1) for x in sides)
    else:
        ne = 0
        for s in range(case["sims"]):
            n = case["n"] if case["sims"] == 1 else 100 + (37 * s) % (case["n"] - 99)
            ne += n * (case["wires"] or (16, 24, 32, 48)[s % 4])
        nn = ne
    steps = case.get("steps", 2 if kind == "retry" else 1)
    contact = 0 if case["scene"] == "cantilever" else 6843
    return dict(bytes=float(steps) * (2 * 8 * 36 * nn + 8 * 25 * ne), flops=float(steps) * 2 * ne * (26687 + contact))


# ------------------------------------------------------------------ 64-bit values


def _exact_mesh(case, seed):
    if 20 * 4 ** case["sub"] * case["grid"] ** 3 > 60_000_000:
        return None
    rng = np.random.default_rng([seed, case.get("n", 0), 11])
    V, T = _icosphere(case["sub"], rng)
    g = case["grid"]
    lo, hi = V.min(0), V.max(0)
    h = float((hi - lo).max()) / (g - 7)
    o = (lo + hi) / 2 - h * (g - 1) / 2
    xs = [o[a] + h * np.arange(g) for a in range(3)]
    Z, Y, X = np.meshgrid(xs[2], xs[1], xs[0], indexing="ij")
    P = np.stack([X.ravel(), Y.ravel(), Z.ravel()], 1)
    best = np.full(len(P), np.inf)
    omega = np.zeros(len(P))
    dot = lambda a, b: a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1] + a[..., 2] * b[..., 2]
    for t in T - 1:
        A, B, C = V[t]
        # distance: the plane's foot where it lies in the triangle, else the nearest of the three edges
        N = np.cross(B - A, C - A)
        N /= np.linalg.norm(N)
        hgt = (P - A) @ N
        F = P - hgt[:, None] * N
        ins = np.ones(len(P), bool)
        d2 = np.full(len(P), np.inf)
        for a, b in ((A, B), (B, C), (C, A)):
            e = b - a
            ins &= (np.cross(e, F - a) @ N) >= 0
            s = np.clip((P - a) @ e / (e @ e), 0, 1)
            q = P - (a + s[:, None] * e)
            d2 = np.minimum(d2, dot(q, q))
        best = np.minimum(best, np.where(ins, hgt ** 2, d2))
        a, b, c = A - P, B - P, C - P
        la, lb, lc = np.sqrt(dot(a, a)), np.sqrt(dot(b, b)), np.sqrt(dot(c, c))
        omega += 2 * np.arctan2(dot(a, np.cross(b, c)), la * lb * lc + dot(a, b) * lc + dot(a, c) * lb + dot(b, c) * la)
    d = np.sqrt(best)
    return np.where(np.abs(omega) > 2 * np.pi, d, -d).reshape(g, g, g)


def exact(case, seed):
    kind = case["kind"]
    if kind == "meshsdf":
        return _exact_mesh(case, seed)
    if kind not in ("mlpforward", "mlpgrad"):
        return None
    st = prepare(case, seed)
    p = torch.from_numpy(st["p"])
    o1, o2, o3 = 48 * 128, 48 * 128 + 128, 48 * 128 + 128 + 128 * 128
    o4, o5 = o3 + 128, o3 + 128 + 128 * 6
    bf = lambda a: a.bfloat16().double()  # the network's weights are BF16 values
    W = [bf(p[:o1]).reshape(48, 128), p[o1:o2].double(), bf(p[o2:o3]).reshape(128, 128), p[o3:o4].double(),
         bf(p[o4:o5]).reshape(128, 6), p[o5:].double()]
    W = [w.clone().requires_grad_(True) for w in W]
    X, T = torch.from_numpy(st["X"]).double(), torch.from_numpy(st["T"]).double()
    silu = torch.nn.functional.silu
    Y = silu(silu(X @ W[0] + W[1]) @ W[2] + W[3]) @ W[4] + W[5]
    if kind == "mlpforward":
        return Y.detach().numpy()
    loss = ((Y - T) ** 2).mean()
    loss.backward()
    return dict(loss=float(loss.detach()), grad=torch.cat([w.grad.reshape(-1) for w in W]).numpy())
