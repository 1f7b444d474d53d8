"""The workspace of the context-free calls: shared by threads, given back (B200)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(seed):
    rng = np.random.default_rng(seed)
    rows, cols = 3 + seed, 5 + 2 * seed
    x, y = np.meshgrid(0.2 * np.arange(rows + 1), 0.1 * np.arange(cols + 1), indexing="ij")
    pos = np.stack([x, y, 0.02 * rng.standard_normal(x.shape)], -1)[None]
    return pos, rng.standard_normal((1, rows, cols)), rng.uniform(-1, 2, (200 + 900 * seed, 3))


def test_threads_share_the_workspace_and_it_is_given_back():
    """Calls of several threads at once, of different sizes and kinds, give what each gives alone; so do calls after
    the workspace was released, between and during them."""
    import uvlm_b200 as U

    def work(seed):
        pos, gamma, t = _case(seed)
        A = np.eye(40 + 30 * seed) * 3 + np.random.default_rng(seed).standard_normal((40 + 30 * seed,) * 2) * 0.1
        b = np.arange(len(A), dtype=float)
        return [U.InducedVelocity(t, pos, gamma), U.InducedVelocity(t, pos, gamma, "mixed"), U.dense_solve(A, b)[0],
                U.dense_solve(A, b, "tf32")[0]]

    alone = [work(s) for s in range(4)]
    got, errors = [[] for _ in range(4)], []

    def run(s):
        try:
            for _ in range(6):
                got[s].append(work(s))
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=run, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    U.release_workspace()
    for t in threads:
        t.join()
    assert not errors
    for s in range(4):
        for rep in got[s]:
            for a, b in zip(rep, alone[s]):
                np.testing.assert_array_equal(a, b)
    U.release_workspace()
    for a, b in zip(work(2), alone[2]):
        np.testing.assert_array_equal(a, b)
    with pytest.raises(U.UVLMError):
        U.release_workspace(63)


def _free_bytes():
    import torch

    return torch.cuda.mem_get_info(0)[0]


def test_memory_kept_after_a_large_call_is_bounded_and_given_back():
    """A call that takes over 1 GB keeps at most 256 MiB when it returns, also after several such calls at once, and
    nothing after release_workspace (each to 32 MiB, the driver's own granularity)."""
    import uvlm_b200 as U

    pos, gamma, _ = _case(0)
    t = np.random.default_rng(1).uniform(5, 9, (3_000_000, 3))
    U.InducedVelocity(t[:1000], pos, gamma)  # the kernels are loaded
    U.release_workspace()
    before, slack = _free_bytes(), 32 << 20
    U.InducedVelocity(t, pos, gamma)
    assert before - _free_bytes() <= (256 << 20) + slack
    threads = [threading.Thread(target=lambda: U.InducedVelocity(t[:1_000_000], pos, gamma)) for _ in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert before - _free_bytes() <= (256 << 20) + slack
    U.InducedVelocity(t[:100_000], pos, gamma)
    U.release_workspace()
    assert before - _free_bytes() <= slack


_DRIVER_CONTEXT = """
import ctypes as C, sys
import numpy as np
cuda = C.CDLL("libcuda.so.1")
ctx, now, dev, flags, active = C.c_void_p(), C.c_void_p(), C.c_int(), C.c_uint(), C.c_int()
assert cuda.cuInit(0) == 0 and cuda.cuDeviceGet(C.byref(dev), 0) == 0
assert cuda.cuCtxCreate_v2(C.byref(ctx), 0, dev) == 0
sys.path[:0] = sys.argv[2:]
import test_gpu_workspace as T
import uvlm_b200 as U
out = []
for call in T.CALLS:
    out.append(np.asarray(call()))
    assert cuda.cuCtxGetCurrent(C.byref(now)) == 0 and now.value == ctx.value, "another context is current"
U.release_workspace()
assert cuda.cuCtxGetCurrent(C.byref(now)) == 0 and now.value == ctx.value, "another context is current"
assert cuda.cuDevicePrimaryCtxGetState(dev, C.byref(flags), C.byref(active)) == 0 and not active.value
np.savez(sys.argv[1], *out)
"""


def _gradients():
    from uvlm_b200.warmstart import MLP

    rng = np.random.default_rng(3)
    net = MLP(seed=1)
    return net.gradients(rng.standard_normal((100, 8)).astype(np.float32), rng.standard_normal(100).astype(np.float32))[0]


def _call(f):
    def run():
        import uvlm_b200 as U

        return f(U)

    return run


CALLS = [_call(lambda U: U.InducedVelocity(_case(2)[2], *_case(2)[:2])),
         _call(lambda U: U.InducedVelocity(_case(2)[2], *_case(2)[:2], precision="mixed")),
         _call(lambda U: U.dense_solve(np.eye(70) * 3 + np.ones((70, 70)) * 0.1, np.arange(70.0))[0]),
         _gradients]


def test_calls_stay_in_the_callers_context(tmp_path):
    """A program that works in a driver context of its own: the calls give the same results there, leave it current, and
    bring up no other context (arrays of one context cannot be read from another)."""
    import os
    import subprocess
    import sys

    here = os.path.dirname(os.path.abspath(__file__))
    path = str(tmp_path / "out.npz")
    p = subprocess.run([sys.executable, "-c", _DRIVER_CONTEXT, path, os.path.dirname(here), here], capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    with np.load(path) as got:
        for name, call in zip(got.files, CALLS):
            np.testing.assert_array_equal(got[name], call())
