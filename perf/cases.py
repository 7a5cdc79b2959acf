"""Workloads of the Cauchy estimator and its consumers, each through the public Python API.

A case is a dict of plain values: its kind (which entry points a pass calls),
the model family (``cauchyfriendly_gb300.workloads``; the system matrices are
those of the family's seed 0, the measurement history is drawn from the seed)
and its sizes.  The families are the repository's own benchmark and test
problems:

  two_state    2-state LTI, one measurement a step
  four_state   4-state LTI (the sliding-window and gradient configuration)
  three_state  3-state LTI of the plain configuration
  five_state   5-state, two process-noise columns, two measurements a step
  five_ltv     the 5-state time-varying sliding-window configuration
"""
import math

import numpy as np

from cauchyfriendly_gb300 import BatchedCauchyEstimator, CauchyEstimator, RelativeSystem2D
from cauchyfriendly_gb300 import workloads as W
from cauchyfriendly_gb300.adjoint import AdjointBatch, loglik_weights
from cauchyfriendly_gb300.windows import SlidingWindowManager


def listed():
    return [
        # one small estimator stepped measurement by measurement, its estimate read after each: an
        # embedded filter's loop, where launches and round trips are the cost
        {"name": "plain_2state", "kind": "plain", "family": "two_state", "steps": 6},
        # one estimator run to the end of its window, 1e5 terms in its last updates: a 4-state
        # tracking problem, and a 5-state one with two measurements a step and odd shapes
        {"name": "plain_4state", "kind": "plain", "family": "four_state", "steps": 8},
        {"name": "plain_5state", "kind": "plain", "family": "five_state", "steps": 4},
        # Monte-Carlo batches of 3-state estimators of unequal length (the benchmark's
        # distribution), a small ragged one and the benchmark's whole batch
        {"name": "batch_small", "kind": "batch", "n": 331, "steps_lo": 4, "steps_hi": 9},
        {"name": "batch_full", "kind": "batch", "n": 4096, "steps_lo": 4, "steps_hi": 9},
        # sliding-window estimation, the online mode: many small windows, and the heavy 5-state
        # time-varying one whose full windows carry most of the terms
        {"name": "windows_4state", "kind": "windows", "family": "four_state", "window": 7, "steps": 16, "n": 1},
        {"name": "windows_5state", "kind": "windows", "family": "five_ltv", "window": 5, "steps": 7, "n": 1},
        # maximum-likelihood tuning: log-likelihoods of a batch of window lives and their gradients
        {"name": "gradient_4state", "kind": "gradient", "family": "four_state", "steps": 7, "n": 24},
        # the relative 2-D pdf of two 5-state estimators (conjunction analysis): pairs, moments and grid
        {"name": "relative_5state", "kind": "relative", "family": "five_state", "updates": 6, "nx": 13, "ny": 13},
        # pdf plots of the current estimate: a marginal curve and a full 2-D surface
        {"name": "marginal_1d", "kind": "grid1d", "family": "three_state", "updates": 9, "nx": 801},
        {"name": "surface_2d", "kind": "grid2d", "family": "two_state", "updates": 6, "nx": 101, "ny": 83},
        # the joint pdf at scattered points (particles, a likelihood's argument)
        {"name": "points_4state", "kind": "points", "family": "four_state", "updates": 6, "points": 256, "keep": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "batch", "windows", "gradient", "relative", "grid1d", "grid2d", "points"])
    if kind == "plain":
        fam = rng.choice(["two_state", "three_state", "four_state", "five_state"])
        lo, hi = {"two_state": (3, 10), "three_state": (3, 11), "four_state": (3, 8), "five_state": (2, 4)}[fam]
        return {"kind": kind, "family": fam, "steps": rng.randint(lo, hi)}
    if kind == "batch":
        lo = rng.randint(2, 6)
        return {"kind": kind, "n": _log_int(rng, 3, 4096), "steps_lo": lo, "steps_hi": rng.randint(lo, 9)}
    if kind == "windows":
        fam = rng.choice(["two_state", "four_state", "five_ltv"])
        w = rng.randint(3, {"two_state": 9, "four_state": 7, "five_ltv": 4}[fam])
        return {"kind": kind, "family": fam, "window": w, "steps": w + rng.randint(1, 8),
                "n": _log_int(rng, 1, 2 if fam == "five_ltv" else 8)}
    if kind == "gradient":
        fam = rng.choice(["two_state", "three_state", "four_state"])
        return {"kind": kind, "family": fam, "steps": rng.randint(3, 7), "n": _log_int(rng, 1, 64)}
    if kind == "relative":
        fam = rng.choice(["two_state", "three_state", "five_state"])
        hi = {"two_state": 6, "three_state": 7, "five_state": 5}[fam]
        return {"kind": kind, "family": fam, "updates": rng.randint(3, hi), "nx": _log_int(rng, 5, 24),
                "ny": _log_int(rng, 5, 24)}
    if kind == "grid1d":
        fam = rng.choice(["two_state", "three_state", "four_state"])
        return {"kind": kind, "family": fam, "updates": rng.randint(3, 6 if fam == "four_state" else 9),
                "nx": _log_int(rng, 11, 4001)}
    if kind == "grid2d":
        fam = rng.choice(["two_state", "three_state", "four_state"])
        return {"kind": kind, "family": fam, "updates": rng.randint(3, 5 if fam == "four_state" else 7),
                "nx": _log_int(rng, 7, 161), "ny": _log_int(rng, 7, 161)}
    fam = rng.choice(["two_state", "four_state"])
    d = {"two_state": 2, "four_state": 4}[fam]
    return {"kind": kind, "family": fam, "updates": rng.randint(3, 5), "points": _log_int(rng, 1, 400),
            "keep": rng.randint(0, d - 1)}


# -- inputs --------------------------------------------------------------------

def _model(family, steps):
    if family == "two_state":
        return W.two_state_lti(0, steps)
    if family == "three_state":
        return W.three_state_lti(0, steps)
    if family == "four_state":
        return W.four_state_lti(0, steps)
    if family == "five_state":
        return W.five_state_two_msmt(0, steps)
    return W.five_state_ltv_windows(0, steps)


def _measure(prob, rng, most=np.inf):
    """A measurement history of the model: Cauchy process and measurement noise from a Cauchy start, no
    draw beyond `most` scales (a pdf is refused where the estimate before it did not exist)."""
    d, p = prob["d"], prob["p"]
    noise = lambda n: np.clip(rng.standard_cauchy(n), -most, most)
    x = prob["b0"] + np.linalg.solve(prob["A0"], noise(d) * prob["p0"])
    z = np.zeros((prob["steps"], p))
    for k in range(prob["steps"]):
        if k > 0:
            Phi = prob["Phi"] if prob["Phi"].ndim == 2 else prob["Phi"][k]
            x = Phi @ x + prob["Gamma"] @ (noise(prob["pncc"]) * prob["beta"])
        z[k] = prob["H"] @ x + noise(p) * prob["gamma"]
    return z


def _problem(case, seed, steps):
    prob = _model(case["family"], steps)
    rng = np.random.Generator(np.random.PCG64([11, seed]))
    prob["msmts"] = _measure(prob, rng, 3.0 if "updates" in case else np.inf)
    return prob, rng


def _max_shape(steps, d, pncc):
    return (steps - 1) * pncc + d


def _constants(rng, n, d, rows):
    """Root points and vertex perturbations, distributed as the constructor's own draws."""
    return 1.0 + rng.uniform(size=(n, d)), rng.uniform(-1.0, 1.0, size=(n, rows))


def _estimator(case, seed, steps):
    prob, rng = _problem(case, seed, steps)
    d, pncc = prob["d"], prob["pncc"]
    rp, bp = _constants(rng, 1, d, _max_shape(steps, d, pncc))
    est = CauchyEstimator(prob["A0"], prob["p0"], prob["b0"], steps, d, 0, pncc, prob["p"], root_point=rp[0],
                          b_pert=bp[0])
    return est, prob, rng


def _step(est, prob, k, j):
    Phi = prob["Phi"] if prob["Phi"].ndim == 2 else prob["Phi"][k]
    return est.step(prob["msmts"][k, j], Phi, prob["Gamma"], prob["beta"], prob["H"][j], prob["gamma"][j])


def _advanced(case, seed):
    """An estimator after case["updates"] updates, more steps to come: its g-tables are in place."""
    est, prob, rng = _estimator(case, seed, case["updates"] // _DIMS[case["family"]][2] + 1)
    for u in range(case["updates"]):
        _step(est, prob, u // prob["p"], u % prob["p"])
    return est, prob, rng


def _centre(est):
    return np.round(np.nan_to_num(est.moments()["raw_mean"].real, nan=0.0, posinf=0.0, neginf=0.0), 2)


def _span(c, half, n):
    """n grid points about c: the step leaves the last one half a step early, then clamped to the end."""
    return c - half, c + half, 2.0 * half / (n - 1.5)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plain":
        est, prob, _ = _estimator(case, seed, case["steps"])
        return {"kind": kind, "est": est, "prob": prob}
    if kind == "batch":
        probs = W.batched_three_state(case["n"], seed=0, steps_lo=case["steps_lo"], steps_hi=case["steps_hi"])
        rng = np.random.Generator(np.random.PCG64([12, seed]))
        n, mx = case["n"], case["steps_hi"]
        msm = np.zeros((n, mx, 1))
        for i, p in enumerate(probs):
            msm[i, :p["steps"]] = W.simulate(p, rng, 0.05, 100.0)
        stack = lambda k: np.stack([p[k] for p in probs])
        steps = np.array([p["steps"] for p in probs], np.int32)
        rp, bp = _constants(rng, n, 3, _max_shape(int(steps.max()), 3, 1))
        est = BatchedCauchyEstimator(stack("A0"), stack("p0"), stack("b0"), steps, 3, 0, 1, 1, rp, bp)
        return {"kind": kind, "est": est, "msmts": msm,
                "model": [stack(k) for k in ("Phi", "Gamma", "beta", "H", "gamma")]}
    if kind == "windows":
        n, w, steps = case["n"], case["window"], case["steps"]
        prob, rng = _problem(case, seed, steps)
        msm = np.stack([prob["msmts"]] + [_measure(prob, rng) for _ in range(n - 1)], axis=1)  # (steps, n, p)
        d, pncc = prob["d"], prob["pncc"]
        cs = [_constants(rng, n, d, _max_shape(w, d, pncc)) for _ in range(w)]
        tile = lambda a: np.ascontiguousarray(np.broadcast_to(a, (n,) + a.shape))
        Phi = prob["Phi"] if prob["Phi"].ndim == 3 else np.broadcast_to(prob["Phi"], (steps, d, d))
        return {"kind": kind, "window": w, "start": [tile(prob[k]) for k in ("A0", "p0", "b0")],
                "dims": (d, pncc, prob["p"]), "msmts": msm, "Phi": [tile(P) for P in Phi],
                "model": [tile(prob[k]) for k in ("Gamma", "beta", "H", "gamma")],
                "root_point": np.stack([c[0] for c in cs]), "b_pert": np.stack([c[1] for c in cs])}
    if kind == "gradient":
        n, steps = case["n"], case["steps"]
        prob, rng = _problem(case, seed, steps)
        d, pncc = prob["d"], prob["pncc"]
        rp, bp = _constants(rng, n, d, _max_shape(steps, d, pncc))
        lens = [max(2, steps - (i % 3 if i else 0)) for i in range(n)]  # the last lives of a run are shorter
        msm = [_measure(prob, rng)[:k].reshape(-1) for k in lens]
        runs = AdjointBatch(d, pncc, 1, lens, np.stack([prob["A0"]] * n), np.stack([prob["p0"]] * n),
                            np.stack([prob["b0"]] * n), rp, bp)
        return {"kind": kind, "runs": runs, "msmts": msm,
                "model": [prob[k] for k in ("Phi", "Gamma", "beta", "H", "gamma")]}
    if kind == "relative":
        a, prob, rng = _advanced(case, 2 * seed)
        b, _, _ = _advanced(case, 2 * seed + 1)
        d = prob["d"]
        T = np.zeros((2, d))
        T[0, 0] = T[1, min(2, d - 1)] = 1.0
        c = T @ (_centre(b) - _centre(a))
        grid = [*_span(c[0], 1.0, case["nx"]), *_span(c[1], 1.0, case["ny"])]
        return {"kind": kind, "ests": (a, b), "T": T, "nu": rng.uniform(-1.0, 1.0, d), "grid": grid}
    est, prob, rng = _advanced(case, seed)
    d = prob["d"]
    nu = 2.0 * rng.uniform(size=d)
    c = _centre(est)
    if kind == "grid1d":
        return {"kind": kind, "est": est, "grid": _span(c[0], 2.0, case["nx"]), "nu": nu}
    if kind == "grid2d":
        return {"kind": kind, "est": est, "gx": _span(c[0], 1.0, case["nx"]), "gy": _span(c[1], 1.0, case["ny"]),
                "nu": nu}
    keep = case["keep"]
    x = c + 0.3 * np.clip(rng.standard_cauchy((case["points"], d)), -10.0, 10.0)
    return {"kind": kind, "est": est, "keep": keep, "x": x if keep == 0 else np.ascontiguousarray(x[:, :keep]),
            "nu": nu[:d - keep]}


# -- one pass --------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "plain":
        est, prob = state["est"], state["prob"]
        est.reset()
        out = []
        for k in range(prob["steps"]):
            for j in range(prob["p"]):
                err = _step(est, prob, k, j)
                m = est.moments()
                out.append((m, err, est.num_terms()))
        return {"raw_fz": np.array([o[0]["raw_fz"] for o in out]), "raw_mean": np.stack([o[0]["raw_mean"] for o in out]),
                "raw_cov": np.stack([o[0]["raw_cov"] for o in out]), "gscale": np.array([o[0]["gscale"] for o in out]),
                "mean": np.stack([o[0]["mean"] for o in out]), "cov": np.stack([o[0]["cov"] for o in out]),
                "err": np.array([o[1] for o in out]), "terms": np.array([o[2] for o in out])}
    if kind == "batch":
        state["est"].reset()
        return state["est"].run(state["msmts"], *state["model"], shared_model=False)
    if kind == "windows":
        d, pncc, p = state["dims"]
        mgr = SlidingWindowManager(state["window"], *state["start"], d, pncc, p, root_point=state["root_point"],
                                   b_pert=state["b_pert"], no_window="fullest")
        Gamma, beta, H, gamma = state["model"]
        out, fz = [], []
        for k, z in enumerate(state["msmts"]):
            out.append(mgr.step(z, state["Phi"][k], Gamma, beta, H, gamma))
            fz.append([m["fz"] for m in mgr.last])
        mgr.close()
        return {"xhat": np.array([[m[0] for m in s] for s in out]), "Phat": np.array([[m[1] for m in s] for s in out]),
                "window": np.array([[m[2] for m in s] for s in out]), "err": np.array([[m[3] for m in s] for s in out]),
                "fz": np.array(fz)}
    if kind == "gradient":
        runs = state["runs"]
        fz = runs.forward(state["msmts"], *state["model"])
        grads = runs.backward([loglik_weights(f) for f in fz])
        return {"fz": np.concatenate(fz), **{k: np.stack([g[k] for g in grads]) for k in grads[0]}}
    if kind == "relative":
        rel = RelativeSystem2D(*state["ests"], state["T"], with_term_approx=True, term_approx_eps=1e-8,
                               bar_nu_full=state["nu"])
        X, Y, Z, nx, ny = rel.grid(*state["grid"])
        out = {"mean": rel.moments["mean"], "cov": rel.moments["cov"], "x": X, "y": Y, "z": Z,
               "counts": np.array([rel.pairs, rel.approxed_out, nx, ny])}
        rel.close()
        return out
    est = state["est"]
    if kind == "grid1d":
        x, y = est.cpdf_1d_grid(0, 0, *state["grid"], state["nu"])
        return {"x": x, "y": y}
    if kind == "grid2d":
        x, y, z = est.cpdf_2d_grid(0, 0, 1, state["gx"], state["gy"], state["nu"])
        return {"x": x, "y": y, "z": z}
    if state["keep"] == 0:
        f = est.cpdf_nd(state["x"])
    else:
        f = est.cpdf_marginal(state["x"], list(range(state["keep"])), state["nu"])
    return {"f": f.real}  # the imaginary part is rounding


# -- the work of a pass ----------------------------------------------------------

# terms present after each update's measurement of the families' systems, and the share that
# stays after the reduction (counted on the CPU; other measurement histories differ by a few percent)
_TERMS = {
    "two_state": [3, 12, 39, 112, 305, 812, 2141, 5618, 14695, 38159],
    "three_state": [2, 6, 20, 66, 197, 556, 1503, 3592, 8163, 20171, 47537],
    "four_state": [5, 30, 140, 600, 2460, 9763, 37758, 142167],
    "five_state": [6, 36, 168, 784, 2960, 10760, 36758, 157038, 502771, 1868307],
    "five_ltv": [6, 36, 168, 784, 2960, 10760, 36758, 157038, 502771, 1868307],
    "batch": [4, 20, 80, 270, 870, 2600, 7200, 19000, 50000],
}
_KEPT = 0.45
_DIMS = {"two_state": (2, 1, 1), "three_state": (3, 1, 1), "four_state": (4, 1, 1), "five_state": (5, 2, 2),
         "five_ltv": (5, 2, 2), "batch": (3, 1, 1)}


def _rows(family, u):
    d, pncc, p = _DIMS[family]
    return d + pncc * (u // p) * (0.5 if d > 2 else 0.8)


def _terms(family, u):
    t = _TERMS[family]
    return t[min(u, len(t) - 1)]


def _update_flops(family, u):
    """One update: rows, g values and moments of every post-measurement term; vertex solves and
    table cells of every kept one."""
    d, _, _ = _DIMS[family]
    m, n = _rows(family, u), _terms(family, u)
    cells = sum(math.comb(int(m), k) for k in range(d))
    term = 7 * m * d + m + 8 * (1 + d + d * d) + 22
    kept = cells * (m + 22) + math.comb(int(m), d) * (2 * d ** 3 / 3 + 2 * d * d + 2 * max(m - d, 0) * d)
    return n * term + _KEPT * n * kept


def _run_flops(family, updates):
    return sum(_update_flops(family, u) for u in range(updates))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        mean = [0.5 * (case["steps_lo"] + case["steps_hi"])]
        lo, hi = case["steps_lo"], case["steps_hi"]
        fl = sum(_run_flops("batch", s) for s in range(lo, hi + 1)) / (hi - lo + 1) * case["n"]
        return {"bytes": 8.0 * case["n"] * mean[0] * (1 + 2 * 13 + 2), "flops": fl}
    fam = case["family"]
    d, pncc, p = _DIMS[fam]
    moments = 16.0 * (1 + d + d * d)
    if kind == "plain":
        return {"bytes": case["steps"] * p * (moments + 8.0 * d * (d + 2)), "flops": _run_flops(fam, case["steps"] * p)}
    if kind == "windows":
        w, s, n = case["window"], case["steps"], case["n"]
        fl = sum(_run_flops(fam, min(w, s - k) * p) for k in range(s)) * n
        return {"bytes": n * s * p * (moments + 8.0 * d * (d + 2)), "flops": fl}
    if kind == "gradient":
        # a forward run, its recorded values again, and a reverse of about twice the forward's arithmetic
        fl = 4.0 * case["n"] * _run_flops(fam, case["steps"])
        return {"bytes": case["n"] * 8.0 * (case["steps"] + d * d + 2 * d + 3), "flops": fl}
    u = case["updates"]
    kept, m = max(1.0, _KEPT * _terms(fam, u - 1)), _rows(fam, u - 1)
    table = 16.0 * sum(math.comb(int(m), k) for k in range(d)) + 8.0 * m * (d + 1)
    if kind == "relative":
        pts = case["nx"] * case["ny"]
        return {"bytes": 2 * kept * table + 24.0 * pts,
                "flops": kept * kept * (4 * 2 * m * d + 2 * m * (4 * m + 30) + 0.06 * pts * 2 * m * 56)}
    if kind == "grid1d":
        return {"bytes": kept * table + 16.0 * case["nx"], "flops": kept * (case["nx"] * 8.0 + m * (2 + d) + 22)}
    if kind == "grid2d":
        pts = case["nx"] * case["ny"]
        return {"bytes": kept * table + 24.0 * pts, "flops": kept * m * (56.0 * pts + 4 * m + 60)}
    # points: every (point, term) lowered d - 2 times into its children, the last level's cells summed
    fl = case["points"] * kept * (m ** max(1, d - 2)) * 60.0
    return {"bytes": kept * table + 8.0 * case["points"] * (d + 1), "flops": fl}


# -- 64-bit values in plain numpy ------------------------------------------------

class _Series:
    """The estimator's characteristic function without merging any terms: every term of an update
    spawns one child per row the measurement integrates, plus itself.  G(s), the coefficient of a term
    at the sign vector s of its rows, comes from the parent's two coefficients at the sign vectors with the
    integrated row positive and negative.  Rows of one direction within a term count as one: the later ones
    stay in the arrays, not live, and take their sign from the first."""

    MOST = 60_000  # terms

    def __init__(self, prob, updates, root):
        d = prob["d"]
        self.levels, self.raw = [], []
        A, p, b = prob["A0"][None], prob["p0"][None], prob["b0"][None]
        live = np.ones(p.shape, bool)
        for u in range(updates):
            k, j = divmod(u, prob["p"])
            old = A.shape[1]
            if u > 0 and j == 0:
                Phi = prob["Phi"] if prob["Phi"].ndim == 2 else prob["Phi"][k]
                n, pncc = A.shape[0], prob["pncc"]
                A, b = A @ Phi.T, b @ Phi.T
                A = np.concatenate([A, np.broadcast_to(prob["Gamma"].T, (n, pncc, d))], axis=1)
                p = np.concatenate([p, np.broadcast_to(prob["beta"], (n, pncc))], axis=1)
                live = np.concatenate([live, np.ones((n, pncc), bool)], axis=1)
                A, p, live, _, _ = self._merge(A, p, live)
            H, gam = prob["H"][j], prob["gamma"][j]
            n, m, _ = A.shape
            h = A @ H
            orth = (np.abs(h) < 1e-10) | ~live
            hs = np.where(orth, 1.0, h)
            mu = np.concatenate([A / hs[:, :, None], np.zeros((n, 1, d))], axis=1)
            rho = np.concatenate([p * np.where(orth, 1.0, np.abs(h)), np.full((n, 1), gam)], axis=1)
            alive = np.concatenate([live, np.ones((n, 1), bool)], axis=1)
            free = np.concatenate([orth, np.zeros((n, 1), bool)], axis=1)  # rows kept as they are
            zeta = prob["msmts"][k, j] - b @ H
            par, piv = np.nonzero(~free)  # parent, integrated row (m: the measurement's own)
            if len(par) > self.MOST:
                raise OverflowError
            others = np.array([[l for l in range(m + 1) if l != t] for t in range(m + 1)])[piv]
            pick = (par[:, None], others)
            fr = free[pick]
            A = mu[pick] - np.where(fr[..., None], 0.0, 1.0) * mu[par, piv][:, None, :]
            p, live = rho[pick], alive[pick]
            b = b[par] + zeta[par][:, None] * mu[par, piv]
            L = {"par": par, "piv": piv, "others": others, "flip": np.sign(hs), "q": np.where(fr, 0.0, p), "m": m,
                 "rho": rho[par, piv], "zeta": zeta[par], "old": old, "scale": 1.0}
            self.levels.append(L)
            s = np.where(A @ root > 0, 1.0, -1.0)
            y = -np.einsum("nm,nmd->nd", p * s, A) + 1j * b
            A, p, live, L["rep"], L["sgn"] = self._merge(A, p, live)
            g = self.g(np.arange(len(par)), s) / (2 * np.pi)
            fz = g.sum()
            mean = (g[:, None] * y).sum(0) / (1j * fz.real)
            cov = -np.einsum("n,ni,nj->ij", g, y, y) / fz - np.outer(mean, mean)
            L["scale"] = 1.0 / (2 * np.pi * fz.real)
            self.raw.append((fz, mean, cov, L["scale"]))
        self.A, self.p, self.b = A, p, b

    @staticmethod
    def _merge(A, p, live):
        norm = np.where(live, np.abs(A).sum(2), 1.0)
        A, p, live = A / norm[:, :, None], p * norm, live.copy()
        n, m, _ = A.shape
        rep, sgn = np.broadcast_to(np.arange(m), (n, m)).copy(), np.ones((n, m))
        for i in range(m):
            for k in range(i + 1, m):
                for sg in (1.0, -1.0):
                    same = live[:, i] & live[:, k] & (np.abs(A[:, i] - sg * A[:, k]) < 1e-8).all(1)
                    rep[same, k], sgn[same, k] = i, sg
                    p[same, i] += p[same, k]
                    p[same, k] = 0.0
                    live[same, k] = False
        A = np.where(live[:, :, None], A, 0.0)
        return A, np.where(live, p, 0.0), live, rep, sgn

    def g(self, ids, s, level=None):
        level = len(self.levels) - 1 if level is None else level
        L = self.levels[level]
        par, piv, m, all_ = L["par"][ids], L["piv"][ids], L["m"], np.arange(len(ids))
        s = np.take_along_axis(s, L["rep"][ids], axis=1) * L["sgn"][ids]
        ysum = (L["q"][ids] * s).sum(1)
        full = np.ones((len(ids), m + 1))
        np.put_along_axis(full, L["others"][ids], s, axis=1)
        vals = []
        for sg in (1.0, -1.0):
            full[all_, piv] = sg
            sp = (full[:, :m] * L["flip"][par])[:, :L["old"]]
            vals.append(np.ones(len(ids), complex) if level == 0 else self.g(par, sp, level - 1))
        z = 1j * L["zeta"][ids]
        return (vals[0] / (ysum + L["rho"][ids] + z) - vals[1] / (ysum - L["rho"][ids] + z)) * L["scale"]


def _series_of(case, seed, updates):
    """The unmerged sum, or None where it would hold too many terms."""
    p = _DIMS[case["family"]][2]
    steps = case["steps"] if case["kind"] == "plain" else updates // p + 1
    if updates > 7 or _TERMS[case["family"]][updates - 1] > 1000:
        return None
    prob, rng = _problem(case, seed, steps)
    rp, _ = _constants(rng, 1, prob["d"], _max_shape(steps, prob["d"], prob["pncc"]))
    nu = 2.0 * rng.uniform(size=prob["d"])
    try:
        return _Series(prob, updates, rp[0]), rng, nu
    except OverflowError:
        return None


def _axis(lo, hi, res):
    n = int(math.ceil((hi - lo) / res + 1))
    x = lo + res * np.arange(n)
    x[-1] = hi
    return x


def _surface(S, x1, x2):
    """The pdf at points (x1, x2) of a two-state sum: each term's half-plane cells in polar angle."""
    A, p, b = S.A, S.p, S.b
    n, m, _ = A.shape
    th = np.arctan2(-A[:, :, 0], A[:, :, 1])
    th = np.where(th < 0, th + np.pi, th)
    th = np.where(th >= np.pi, th - np.pi, th)
    th = np.sort(th, axis=1)
    th = np.concatenate([th, th[:, :1] + np.pi], axis=1)
    f = np.zeros(len(x1))
    ids = np.arange(n)
    for c in range(m):
        tm = 0.5 * (th[:, c] + th[:, c + 1])
        s = np.where(A[:, :, 0] * np.cos(tm)[:, None] + A[:, :, 1] * np.sin(tm)[:, None] > 0, 1.0, -1.0)
        wide = th[:, c + 1] - th[:, c] > 1e-9
        g = np.where(wide, S.g(ids, s), 0.0)
        gam = -np.einsum("nm,nmd->nd", p * s, A)
        c1, s1, c2, s2 = np.cos(th[:, c]), np.sin(th[:, c]), np.cos(th[:, c + 1]), np.sin(th[:, c + 1])
        for t in np.nonzero(wide)[0]:
            g1, g2 = gam[t, 0] + 1j * (b[t, 0] - x1), gam[t, 1] + 1j * (b[t, 1] - x2)
            f += (g[t] * (s2[t] / (g1 * (g1 * c2[t] + g2 * s2[t])) - s1[t] / (g1 * (g1 * c1[t] + g2 * s1[t])))).real
    return 2.0 * f / (2 * np.pi) ** 2


def exact(case, seed):
    kind = case["kind"]
    if kind == "plain":
        got = _series_of(case, seed, case["steps"] * _DIMS[case["family"]][2])
        if got is None:
            return None
        raw = got[0].raw
        return {"raw_fz": np.array([r[0] for r in raw]), "raw_mean": np.stack([r[1] for r in raw]),
                "raw_cov": np.stack([r[2] for r in raw]), "gscale": np.array([r[3] for r in raw]),
                "mean": None, "cov": None, "err": None, "terms": None}  # after the numeric checks' replacements
    if kind not in ("grid1d", "grid2d", "points"):
        return None
    if kind != "grid1d" and case["family"] != "two_state":
        return None
    got = _series_of(case, seed, case["updates"])
    if got is None:
        return None
    S, rng, nu = got
    c = np.round(S.raw[-1][1].real, 2)
    if kind == "grid2d":
        gx, gy = _axis(*_span(c[0], 1.0, case["nx"])), _axis(*_span(c[1], 1.0, case["ny"]))
        X, Y = np.meshgrid(gx, gy)
        X, Y = X.reshape(-1), Y.reshape(-1)
        return {"x": X, "y": Y, "z": _surface(S, X, Y)}
    if kind == "points" and case["keep"] == 0:
        x = c + 0.3 * np.clip(rng.standard_cauchy((case["points"], 2)), -10.0, 10.0)
        return {"f": _surface(S, x[:, 0], x[:, 1])}
    if kind == "points":
        x = (c + 0.3 * np.clip(rng.standard_cauchy((case["points"], 2)), -10.0, 10.0))[:, 0]
    else:
        x = _axis(*_span(c[0], 2.0, case["nx"]))
    a = S.A[:, :, 0]
    s = np.where(np.abs(a) > 1e-15, np.sign(a), np.sign(S.A @ nu))
    w, ids = (S.p * np.abs(a)).sum(1), np.arange(len(a))
    gl, gr = S.g(ids, -s), S.g(ids, s)
    f = np.zeros(len(x))
    for i0 in range(0, len(ids), 512):
        t = slice(i0, i0 + 512)
        off = 1j * (S.b[t, 0][None] - x[:, None])
        f += (gl[t] / (w[t] + off) - gr[t] / (-w[t] + off)).real.sum(1)
    f /= 2 * np.pi
    return {"x": x, "y": f} if kind == "grid1d" else {"f": f}
