"""Device memory the library keeps between uses: what it hands back, what is
there for its own other buffers when the device is full, and handles that
grow and go on several threads at once.  Memory is looked at from a process of
its own, in which nothing else holds any."""
import os
import subprocess
import sys
import threading

import numpy as np
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


@pytest.mark.parametrize("what", ["points", "gradient"])
def test_buffers_outside_the_pool_on_a_full_device(what):
    """The pool holds gigabytes that no handle uses and the rest of the device
    is taken: the pdf at points and the gradient, whose buffers are not the
    pool's, find their memory there."""
    _run("""
what = %r
x = rng.standard_normal((16, 4))
q = W.four_state_lti(seed=0, steps=7)
n = 24

def call():
    if what == "points":
        return small.cpdf_nd(x)
    c = np.random.Generator(np.random.PCG64(2))
    runs = AdjointBatch(4, 1, 1, [7] * n, np.stack([q["A0"]] * n), np.stack([q["p0"]] * n), np.stack([q["b0"]] * n),
                        1.0 + c.uniform(size=(n, 4)), c.uniform(-1.0, 1.0, (n, 10)))
    fz = runs.forward([q["msmts"].reshape(-1)] * n, *[q[k] for k in ("Phi", "Gamma", "beta", "H", "gamma")])
    g = runs.backward([loglik_weights(f) for f in fz])
    out = np.concatenate([np.concatenate(fz)] + [r[k].reshape(-1) for r in g for k in sorted(r)])
    runs.close()
    return out

small = estimator(W.four_state_lti, 5)
other = estimator(W.four_state_lti, 5)
want = call()
small.close()
small = estimator(W.four_state_lti, 5)
want = call()
small.close()
rng = np.random.Generator(np.random.PCG64(1))
small = estimator(W.four_state_lti, 5)
before = free()
want = call()
small.close()
rng = np.random.Generator(np.random.PCG64(1))
small = estimator(W.four_state_lti, 5)
held = free()
big = batch(1024)
big.close()
assert held - free() > 3500, (held, free())  # more than the call takes
filler = torch.empty((free() - 256) * MB, dtype=torch.uint8, device="cuda")
got = call()
assert np.allclose(got, want, rtol=1e-9, atol=1e-12 * np.abs(want).max())
print("checked")
""" % what)


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


def test_handles_growing_and_going_on_several_threads():
    """Four threads make, step, trim and destroy batches of their own sizes,
    whose buffers pass from one to another through the pool: the results are
    those of one thread."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cauchyfriendly_gb300 import BatchedCauchyEstimator
    from cauchyfriendly_gb300 import workloads as W

    def run(n, seed):
        probs = W.batched_three_state(n, seed=seed, steps_lo=4, steps_hi=7)
        rng = np.random.Generator(np.random.PCG64(seed))
        s = lambda k: np.stack([q[k] for q in probs])
        z = np.zeros((n, 7, 1))
        for i, q in enumerate(probs):
            z[i, :q["steps"]] = q["msmts"]
        b = BatchedCauchyEstimator(s("A0"), s("p0"), s("b0"), np.array([q["steps"] for q in probs], np.int32), 3, 0, 1,
                                   1, 1.0 + rng.uniform(size=(n, 3)), rng.uniform(-1.0, 1.0, (n, 9)))
        out = []
        for _ in range(2):
            out.append(b.run(z, *[s(k) for k in ("Phi", "Gamma", "beta", "H", "gamma")], shared_model=False))
            b.reset()
            b.trim_memory(1 << 20)
        b.close()
        return out

    jobs = [(n, 10 * t + r) for t in range(4) for r, n in enumerate((17, 160, 41, 300))]
    want = {j: run(*j) for j in jobs}
    got, failed = {}, []

    def work(t):
        try:
            for j in jobs[4 * t: 4 * t + 4]:
                got[j] = run(*j)
        except Exception as e:  # pragma: no cover
            failed.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for j in jobs:
        for a, b in zip(got[j], want[j]):
            for k in a:
                assert np.array_equal(a[k], b[k], equal_nan=True), (j, k)
