"""Device memory the library keeps between uses, looked at from a process of
its own, in which nothing else holds any."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = """
import numpy as np, torch
from cauchyfriendly_gb300 import BatchedCauchyEstimator, CauchyEstimator, RelativeSystem2D, workloads as W
from cauchyfriendly_gb300.adjoint import AdjointBatch, loglik_weights

MB = 1 << 20
torch.cuda.init()
torch.zeros(1, device="cuda")
free = lambda: torch.cuda.mem_get_info()[0] // MB
rng = np.random.Generator(np.random.PCG64(1))

def estimator(family, updates, seed=0):
    steps = updates + 1
    q = family(seed=seed, steps=steps)
    d = q["d"]
    e = CauchyEstimator(q["A0"], q["p0"], q["b0"], steps, d, 0, 1, 1, root_point=1.0 + rng.uniform(size=d),
                        b_pert=rng.uniform(-1.0, 1.0, steps - 1 + d))
    for k in range(updates):
        e.step(q["msmts"][k, 0], q["Phi"], q["Gamma"], q["beta"], q["H"][0], q["gamma"][0])
    return e

def batch(n):
    probs = W.batched_three_state(n, seed=0)
    s = lambda k: np.stack([q[k] for q in probs])
    z = np.zeros((n, 9, 1))
    for i, q in enumerate(probs):
        z[i, :q["steps"]] = q["msmts"]
    b = BatchedCauchyEstimator(s("A0"), s("p0"), s("b0"), np.array([q["steps"] for q in probs], np.int32), 3, 0, 1, 1,
                               1.0 + rng.uniform(size=(n, 3)), rng.uniform(-1.0, 1.0, (n, 11)))
    b.run(z, *[s(k) for k in ("Phi", "Gamma", "beta", "H", "gamma")], shared_model=False, outputs=False)
    return b
"""


def _run(script):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", SETUP + script], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "checked" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]


def test_memory_of_a_relative_system_closed_last_goes_back():
    """With no handle and no relative system alive the library keeps 256 MiB
    at most, whichever went last."""
    _run("""
a, b = (estimator(W.three_state_lti, 8, seed) for seed in (0, 1))
make = lambda: RelativeSystem2D(a, b, np.eye(3)[:2], bar_nu_full=np.array([0.3, 0.5, -0.2]))
make().close()
a.close(), b.close()
start = free()  # the kernels are loaded, and the library keeps what it may
a, b = (estimator(W.three_state_lti, 8, seed) for seed in (0, 1))
rel = make()
assert start - free() > 1024, (start, free())
a.close(), b.close()
rel.close()
assert start - free() <= 256, (start, free())
print("checked")
""")


def test_trimmed_memory_goes_back_to_the_device():
    """trim_memory() without a threshold is for those who need the memory
    elsewhere: the device has it while the handle lives."""
    _run("""
b = batch(256)
b.reset()
before = free()
released = b.trim_memory() // MB
assert released > 512, released
assert free() - before > 0.9 * released, (before, free(), released)
b.close()
print("checked")
""")


def test_a_grid_in_one_chunk_takes_no_partial_sums():
    """A pdf surface of so many points that each sums its terms in one go
    needs the points and the values, 24 bytes a point, and no more; the values
    are those of the same points in a small grid."""
    _run("""
e = estimator(W.two_state_lti, 1)
nu = np.array([0.7, 1.3])
e.cpdf_2d_grid(0, 0, 1, (-1.0, 1.0, 0.25), (-1.0, 1.0, 0.25), nu)
start = free()
X, Y, Z = e.cpdf_2d_grid(0, 0, 1, (-1.0, 1.0, 2.0 ** -12), (-1.0, 1.0, 2.0 ** -10), nu)
took = (start - free()) * MB
assert len(X) == 8193 * 2049
assert took <= 26 * len(X) + 64 * MB, took / len(X)
x, y, z = e.cpdf_2d_grid(0, 0, 1, (-1.0, 1.0, 0.25), (-1.0, 1.0, 0.25), nu)
at = np.searchsorted(Y.reshape(2049, 8193)[:, 0], y) * 8193 + np.searchsorted(X[:8193], x)
assert np.array_equal(X[at], x) and np.array_equal(Y[at], y)
assert np.allclose(Z[at], z, rtol=1e-12, atol=0.0)
xs, ys = e.cpdf_1d_grid(0, 0, -1.0, 1.0, 2.0 ** -20, nu)
xt, yt = e.cpdf_1d_grid(0, 0, -1.0, 1.0, 0.125, nu)
at = np.searchsorted(xs, xt)
assert np.array_equal(xs[at], xt) and np.allclose(ys[at], yt, rtol=1e-9, atol=0.0)
print("checked")
""")
