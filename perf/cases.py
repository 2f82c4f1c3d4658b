"""The calls whose speed matters to a user of the integrator, as plain cases.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges,
``prepare`` builds what a program holds before the call (models, ensembles,
plans, servers, environments, with seeded inputs of the parameter studies),
``run`` is one call through the public entry points, ``work`` what the call
cannot do without and ``exact`` the solution of the same equations by an
independent integration where that is affordable.

Kinds of a case:
  study     ``Model.solve`` of one (NS, K) parameter study in the reference
            layout, with dense output (the drop-in interface)
  ensemble  ``Ensemble.plan().launch()``: a ragged batch, one CUDA graph
  solve     ``Ensemble.solve()``: the same without a captured plan
  env       ``CKM1DVecEnv.step``: one environment step of a PPO rollout
  served    ``SolveServer``: a burst of requests, admitted, solved in time
            slices and read back
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "coupled-bubble-control_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from cbc_b200 import scenes  # noqa: E402
from cbc_b200.ensemble import Ensemble  # noqa: E402
from cbc_b200.envs.pos_control import CKM1DVecEnv  # noqa: E402
from cbc_b200.models import SolverSpec  # noqa: E402
from cbc_b200.serving import Request, SolveServer  # noqa: E402

MAX_STEPS = 1_000_000
# bubble counts of the ragged batches and their weights
MIXES = {
    "study": ((2, 3, 4, 6, 8), (0.4, 0.2, 0.2, 0.1, 0.1)),     # the mixed-K ensemble
    "served": ((2, 4, 8, 16), (0.25, 0.25, 0.25, 0.25)),       # the request stream
    "odd": ((1, 3, 5, 7, 11, 20), (0.2, 0.2, 0.2, 0.2, 0.1, 0.1)),
}


def _case(name, kind, **kw):
    c = {"name": name, "kind": kind, "K": 2, "mix": "", "ns": 1, "span_lo": 1.0, "span_hi": 1.0, "samples": 0,
         "field": "SW_A", "nk": 2, "solver": "richardson", "grid": False}
    c.update(kw)
    return c


def listed():
    return [
        # one bubble pair looked at by hand: the smallest call, all latency
        _case("single_k2", "study", K=2, ns=1, span_lo=0.05, span_hi=0.05, samples=64, grid=True),
        # one cluster of eight through part of a period, dense output on the exact grid
        _case("single_k8", "study", K=8, ns=1, span_lo=0.2, span_hi=0.2, samples=32, grid=True),
        # the plain parameter study (1,024 pairs) over a shorter span
        _case("study_k2", "study", K=2, ns=1024, span_lo=2.0, span_hi=2.0, samples=32),
        # a study that fills the GPU with one K, reference layout
        _case("study_k6", "study", K=6, ns=4099, span_lo=0.5, span_hi=0.5, samples=16),
        # the mixed-K ensemble at its full number of systems, spans shortened
        _case("mixed_65536", "ensemble", mix="study", ns=65536, span_lo=0.2, span_hi=2.0),
        # the same kind of batch at an odd, smaller number of systems
        _case("mixed_5001", "ensemble", mix="study", ns=5001, span_lo=0.1, span_hi=1.0),
        # the direct coupling solver on the mixed batch
        _case("mixed_lu", "ensemble", mix="study", ns=16384, span_lo=0.1, span_hi=0.5, solver="lu"),
        # bubble counts without a kernel of their own, uniform field, three harmonics
        _case("odd_const", "solve", mix="odd", ns=1500, span_lo=0.05, span_hi=0.15, field="CONST", nk=3),
        # one step of 1,024 position-control environments
        _case("env_1024", "env", K=4, ns=1024, span_lo=5.0, span_hi=5.0, field="SW_N"),
        # a burst of requests of the served stream
        _case("served_256", "served", mix="served", ns=256, span_lo=0.1, span_hi=0.5),
        # large clusters with dense output, a few systems per SM
        _case("large_k32", "solve", K=32, ns=1024, span_lo=0.1, span_hi=0.1, samples=64),
        # medium clusters, one of them per warp or fewer
        _case("large_k16", "solve", K=16, ns=2050, span_lo=0.2, span_hi=0.2, samples=32),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("study", "study", "ensemble", "ensemble", "solve", "env", "served"))
    c = _case("", kind)
    del c["name"]
    c["field"] = rng.choice(("SW_A", "SW_A", "SW_A", "SW_N", "CONST"))
    c["nk"] = rng.choice((2, 2, 2, 1, 3))
    c["solver"] = rng.choice(("richardson", "richardson", "richardson", "lu"))
    if kind == "study":
        c["K"] = rng.choice((1, 2, 2, 3, 4, 5, 6, 8, 8, 12, 16, 24, 32))
        c["ns"] = int(_log(rng, 1, 24000 / c["K"] ** 1.5))
        c["span_lo"] = c["span_hi"] = round(_log(rng, 0.05, 0.6), 3)
        c["samples"] = rng.choice((0, 16, 32, 64))
        c["grid"] = rng.random() < 0.3
    elif kind in ("ensemble", "solve"):
        c["mix"] = rng.choice(("study", "study", "served", "odd", ""))
        c["K"] = rng.choice((2, 3, 4, 6, 8, 16, 32)) if not c["mix"] else 2
        top = {"study": 65536, "served": 6000, "odd": 6000, "": 48000 / c["K"] ** 1.5}[c["mix"]]
        c["ns"] = int(_log(rng, 32, top))
        c["span_lo"] = 0.05
        c["span_hi"] = round(_log(rng, 0.1, 1.0 if c["mix"] == "study" else 0.4), 3)
        if c["solver"] == "lu":
            c["span_hi"] = round(0.05 + 0.3 * (c["span_hi"] - 0.05), 3)
        c["samples"] = rng.choice((0, 0, 16))
    elif kind == "env":
        c.update(K=rng.choice((1, 2, 3, 4, 5, 6)), ns=int(_log(rng, 16, 2048)), field=rng.choice(("SW_N", "SW_A")),
                 nk=2, solver="richardson")
        c["span_lo"] = c["span_hi"] = round(_log(rng, 0.5, 5.0), 3)
    else:
        c.update(mix="served", ns=int(_log(rng, 8, 400)), span_lo=0.05, span_hi=round(rng.uniform(0.1, 0.5), 3),
                 solver="richardson")
    return c


def _spec(case):
    return SolverSpec(lin_solver=case["solver"], dense_mode="grid" if case["grid"] else "reference")


def _ndo(case):
    return int(round(case["span_hi"] * case["samples"])) + 1 if case["samples"] else 0


def _scene(case, seed):
    """Seeded systems of the parameter studies: water, R0 ~ U[2,8] um,
    PA ~ U[0,1.5] bar (1.2 for the large clusters), neighbours at least
    20 max(R0) apart within half a wavelength (one for the large clusters)."""
    rng = np.random.default_rng(seed)
    ns, nk = case["ns"], case["nk"]
    if case["mix"]:
        ks, w = MIXES[case["mix"]]
        # as many of each K as the weights say, in a random order
        cut = np.round(np.cumsum(w) / np.sum(w) * ns).astype(int)
        Ks = rng.permutation(np.repeat(np.asarray(ks, np.int32), np.diff(np.concatenate([[0], cut]))))
    else:
        Ks = np.full(ns, case["K"], np.int32)
    large = int(Ks.max()) > 16
    half = 0.5 if large else 0.25
    R0 = [rng.uniform(2.0, 8.0, int(k)) for k in Ks]
    PA = rng.uniform(0.0, 1.2 if large else 1.5, (nk, ns))
    PS = rng.uniform(0.0, 2.0, (nk, ns))
    X0 = []
    for k, r in zip(Ks, R0):
        gap = 20.0 * float(r.max()) * 1e-6 / scenes.LAMBDA1
        X0.append(np.sort(rng.uniform(-half, half - (k - 1) * gap, int(k))) + np.arange(k) * gap)
    FR = np.tile(25.0 * np.arange(1, nk + 1)[:, None], (1, ns))
    return scenes.Scene(K=Ks, R0=R0, PA=PA, FR=FR, PS=PS, X0=X0,
                        t_end=rng.uniform(case["span_lo"], case["span_hi"], ns), ac=case["field"], ndo=_ndo(case))


def _saved(tensors):
    return [(t, t.clone()) for t in tensors]


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "study":
        m = scenes.build_model(_scene(case, seed), solver_spec=_spec(case))
        m._ensure_buffers()
        d = m.runtime.device_buffers
        st["model"] = m
        st["start"] = _saved([d.state.actual_time, d.state.time_step, d.state.actual_state, d.dense.dense_index,
                              d.status.actual_event, d.status.status_flags, d.status.total_steps,
                              d.status.rejected_steps, d.status.convergece_success,
                              d.status.convergence_failures])
    elif kind in ("ensemble", "solve"):
        e = Ensemble.from_scene(_scene(case, seed), solver_spec=_spec(case))
        e.to_device()
        st["ens"] = e
        st["start"] = _saved([e.dev[k] for k in ("state", "t", "h", "event", "status", "dense_index", "steps",
                                                 "rejected", "conv_ok", "conv_fail", "lin_iters")])
        if kind == "ensemble":
            st["plan"] = e.plan(MAX_STEPS)
    elif kind == "env":
        # after one step, so that the timed step starts from moving bubbles
        env = CKM1DVecEnv(num_envs=case["ns"], num_bubbles=case["K"], acoustic_field=case["field"],
                          time_step_length=case["span_hi"], seed=int(seed) % 100000)
        rng = np.random.default_rng(seed)
        act = [torch.from_numpy(rng.uniform(0.0, 1.5, (case["ns"], 2)).astype(np.float32)).cuda() for _ in range(2)]
        env.reset()
        env.step(act[0])
        st.update(env=env, actions=act[1])
        st["start"] = _saved([env.ens.dev["state"], env.ens.dev["steps"], env.targets, env.algo_steps,
                              env.total_rewards, env.reset_count])
    else:
        st["scene"] = _scene(case, seed)
        st["server"] = SolveServer(max_systems=512, nk=case["nk"], ac=case["field"],
                                   freqs_khz=tuple(25.0 * (i + 1) for i in range(case["nk"])), keep_results=True)
    return st


def run(state):
    for t, t0 in state.get("start", ()):     # the same initial state again
        t.copy_(t0)
    kind = state["kind"]
    if kind == "study":
        m = state["model"]
        m.solve(max_steps=MAX_STEPS, kernel_steps=2048)
        d = m.runtime.device_buffers
        out = {"state": d.state.actual_state, "t": d.state.actual_time, "h": d.state.time_step,
               "status": d.status.status_flags, "steps": d.status.total_steps, "rejected": d.status.rejected_steps,
               "conv_ok": d.status.convergece_success}
        if m._execution_spec.ndo:
            out.update(dense_index=d.dense.dense_index, dense_time=d.dense.dense_time,
                       dense_state=d.dense.dense_state)
        return out
    if kind in ("ensemble", "solve"):
        e = state["ens"]
        if kind == "ensemble":
            state["plan"].launch()
        else:
            e.solve(MAX_STEPS)
        keys = ["state", "t", "h", "event", "status", "steps", "rejected", "conv_ok", "lin_iters"]
        return {k: e.dev[k] for k in keys + (["dense_index", "dense_time", "dense_state"] if e.ndo else [])}
    if kind == "env":
        env = state["env"]
        obs, rewards, terminated, time_outs, info = env.step(state["actions"])
        return {"obs": obs, "rewards": rewards, "terminated": terminated, "time_outs": time_outs,
                "final_obs": info["final_observation"], "targets": env.targets, "state": env.ens.dev["state"]}
    srv, sc = state["server"], state["scene"]
    srv.completed.clear()
    for i in range(sc.ns):
        srv.submit(Request(rid=i, K=int(sc.K[i]), R0=sc.R0[i], PA=sc.PA[:, i], PS=sc.PS[:, i], X0=sc.X0[i],
                           span=float(sc.t_end[i])))
    while not srv.idle():
        srv.step()
    got = sorted(srv.completed, key=lambda r: r.rid)
    return {"state": np.concatenate([r.result["state"] for r in got]), "t": np.array([r.result["t"] for r in got]),
            "h": np.array([r.result["h"] for r in got]), "status": np.array([r.status for r in got]),
            "steps": np.array([r.result["steps"] for r in got])}


STEPS_PER_PERIOD = 3000.0    # step attempts a period takes at rtol = atol = 1e-9, about
SWEEPS = 16.0                # Richardson sweeps of one right-hand side, about


def work(case):
    if case["mix"]:
        ks, w = (np.asarray(v, dtype=np.float64) for v in MIXES[case["mix"]])
    else:
        ks, w = np.array([float(case["K"])]), np.array([1.0])
    periods = 0.5 * (case["span_lo"] + case["span_hi"])
    n2 = 2.0 * ks
    solve = SWEEPS * (20.0 * ks ** 2 + 12.0 * ks) if case["solver"] == "richardson" else n2 * n2 * (n2 + 2.0)
    step = 6.0 * (130.0 * ks + 35.0 * ks ** 2 + solve) + 240.0 * ks + 10.0
    flops = case["ns"] * periods * STEPS_PER_PERIOD * float(np.sum(w * step))
    # per bubble: state in and out, 13 constants; per system: K x K x 3 couplings, rows, scalars
    per = 8.0 * (4 * 2 + 13) * ks + 24.0 * ks ** 2 + 8.0 * (5 + 4 * case["nk"] + 8)
    dense = _ndo(case) * 8.0 * (4.0 * ks + 1.0)
    return {"bytes": case["ns"] * float(np.sum(w * (per + dense))), "flops": flops}


# ---- the same equations, integrated independently ---------------------------

def _rhs(hb, s, K, nk, field):
    """dy/dt of system s of a model's host buffers, y = (R, X, U, V)[K]; the
    implicit coupling system is solved by numpy's dense solver."""
    up, sp, cp = hb.params.unit_params[:, s, :K], hb.params.system_params[:, s], hb.params.control_params[:, s]
    M = hb.params.coupling_matrices[:, :K, s, :K]
    m0, m1, m2 = M[0].T, M[1].T, M[2].T
    PA, om, ph, wv = (cp[i * nk:(i + 1) * nk][:, None] for i in range(4))
    w0, l0 = 2 * np.pi * sp[1], 2 * np.pi * sp[2]
    eye = np.eye(K)
    off = 1.0 - eye

    def f(t, y):
        R, X, U, V = y.reshape(4, K)
        s_t, c_t = np.sin(w0 * om * t + ph), np.cos(w0 * om * t + ph)
        arg = l0 * wv * X[None, :] + ph
        sx, cx = np.sin(arg), np.cos(arg)
        if field == "CONST":
            pa, pt = np.sum(PA * s_t) + 0 * X, np.sum(PA * om * c_t) + 0 * X
            px = ux = 0 * X
        else:
            a, b = (cx, -sx) if field == "SW_A" else (sx, cx)
            pa, pt = np.sum(PA * a * s_t, 0), np.sum(PA * om * a * c_t, 0)
            px, ux = np.sum(PA * wv * b * s_t, 0), np.sum(PA * sp[4] * b * c_t, 0)
        delta = X[:, None] - X[None, :]
        sg = np.sign(delta)
        rd = off / np.maximum(np.abs(delta), 1e-30)
        h0, h1 = R * U * U, R * R * U
        h2, h3 = h1 * V, R ** 3 * V
        t0 = 2.5 * sg * rd ** 2 * h2 + rd ** 3 * (h3 * V) + 2.0 * rd * h0
        t1 = sg * rd ** 2 * h1 + rd ** 3 * h3
        t2 = 2.0 * sg * rd ** 2 * h0 + 5.0 * rd ** 3 * h2
        g0, g1 = -np.sum(m0 * t0, 1), -0.5 * np.sum(m0 * t1, 1)
        tn, tg2, tg3 = np.sum(m1 * t2, 1), np.sum(m1 * t1, 1), np.sum(m2 * t1, 1)
        q = 1.0 + up[7] * U
        N = ((up[0] + up[1] * U) * R ** -sp[0] - up[2] * q - up[3] / R - up[4] * U / R
             - 1.5 * (1.0 - up[7] * U / 3.0) * U * U - q * up[5] * pa - up[6] * pt * R + up[8] * V * V)
        D = R - up[7] * R * U + up[4] * up[7]
        force = -up[10] * R ** 3 * px - up[11] * R * (V * sp[3] - ux)
        b0 = (N + g0 + g1 * V) / D
        b1 = 3.0 * force * up[9] / R ** 3 - 3.0 * U * V / R + tn + tg2 * U / R + tg3 / R ** 2
        A = np.block([[eye + m0 * rd * R ** 2 / D[:, None], 0.5 * m0 * sg * rd ** 2 * R ** 3 / D[:, None]],
                      [-m1 * sg * rd ** 2 * R ** 2, eye - m1 * rd ** 3 * R ** 3]])
        return np.concatenate([U, V, np.linalg.solve(A, np.concatenate([b0, b1]))])

    return f


_SEQ = [2 * (i + 1) for i in range(8)]


def _extrapolated(f, t, y, H):
    """One step of length H by the extrapolated modified midpoint rule
    (Gragg, Bulirsch, Stoer): the result and the last correction."""
    rows, f0 = [], f(t, y)
    for j, n in enumerate(_SEQ):
        h = H / n
        a, b = y, y + h * f0
        for i in range(1, n):
            a, b = b, a + 2.0 * h * f(t + i * h, b)
        row = [0.5 * (a + b + h * f(t + H, b))]
        for k in range(j):
            row.append(row[k] + (row[k] - rows[j - 1][k]) / ((n / _SEQ[j - k - 1]) ** 2 - 1.0))
        rows.append(row)
    return rows[-1][-1], rows[-1][-1] - rows[-1][-2]


def _integrate(f, y, times):
    """y at each of the increasing times, from y at t = 0; None where the
    step size collapses."""
    t, H, out = 0.0, 1e-3, []
    for te in times:
        while t < te:
            step = min(H, te - t)
            if step < 1e-12:
                return None
            with np.errstate(all="ignore"):
                yn, e = _extrapolated(f, t, y, step)
                err = float(np.max(np.abs(e) / (1e-14 + 1e-13 * np.abs(yn))))
            if err <= 1.0:
                y, t = yn, (te if step == te - t else t + step)
                H = max(H, step * min(4.0, 0.8 * max(err, 1e-9) ** (-1.0 / 15.0)))
            else:
                H = step * max(0.1, 0.8 * err ** (-1.0 / 15.0)) if math.isfinite(err) else 0.1 * step
        out.append(y)
    return out


def exact(case, seed):
    """End states (and samples on the exact grid) of a few systems over a
    short span; everything else takes too long in plain numpy."""
    K, ns = case["K"], case["ns"]
    if case["kind"] != "study" or ns * case["span_hi"] * K ** 1.5 > 6.0:
        return None
    m = scenes.build_model(_scene(case, seed), solver_spec=_spec(case))
    hb = m.runtime.host_buffers
    ndo = m._execution_spec.ndo
    state = np.array(hb.state.actual_state)
    dense = np.zeros((ndo,) + state.shape)
    for s in range(ns):
        te = float(hb.state.time_end[s])
        times = [te * (i / (ndo - 1)) for i in range(1, ndo)] if case["grid"] and ndo > 1 else [te]
        y0 = state[:, s, :K].reshape(-1)
        ys = _integrate(_rhs(hb, s, K, case["nk"], case["field"]), y0, times)
        if ys is None:
            return None
        if len(times) == ndo - 1:
            for i, y in enumerate([y0] + ys):
                dense[i, :, s, :K] = y.reshape(4, K)
        state[:, s, :K] = ys[-1].reshape(4, K)
    out = {"state": state, "t": np.array(hb.state.time_end), "h": None, "status": None, "steps": None,
           "rejected": None, "conv_ok": None}
    if ndo:
        out.update(dense_index=None, dense_time=None, dense_state=dense if case["grid"] and ndo > 1 else None)
    return out
