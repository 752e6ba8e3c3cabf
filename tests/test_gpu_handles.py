"""GPU: several handles, streams and host threads at a time -- what one of them
sets, keeps or gives back does not reach the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def functional(mdf, k):
    return mdf.optibasis.HermiteLossFunc(2.0, 4, 0.95, [k] * 3, 20736.0, 20736, [30.0] * 3)


def test_functionals_of_two_meshes_in_turn(mdf):
    import torch
    c = torch.from_numpy(mdf.optibasis.bspline_initial_basis(2.0, 4, 4)[None]).cuda()
    big = functional(mdf, 256)
    want = mdf.optibasis.ik_error_loss(c, big)
    small = functional(mdf, 224)
    other = mdf.optibasis.ik_error_loss(c, small)
    for _ in range(2):
        assert torch.equal(mdf.optibasis.ik_error_loss(c, big), want)
        assert torch.equal(mdf.optibasis.ik_error_loss(c, small), other)
    assert want.item() != other.item()


@pytest.mark.parametrize("k", [32, 200, 256])
def test_functional_in_order_with_torch(mdf, k):
    """a value read at once on torch's default stream is this call's, with coefficients made just before"""
    import torch
    f = functional(mdf, k)
    base = mdf.optibasis.bspline_initial_basis(2.0, 4, 4)
    for _ in range(20):
        s = 1.0 + 0.01 * _
        c = torch.from_numpy(base[None]).cuda() * s
        assert mdf.optibasis.ik_error_loss(c, f).item() == f.evaluate(base * s, grads=False)[0][0]


@pytest.mark.parametrize("n", [1, 21845, 21846, 87382, 174763, 262145, 3000000])
def test_frames_come_back_whole(mdf, n):
    """sizes around one piece of the read-back (512 KB), all of them, and above 64 MB; a few bytes
    past a multiple of 2 MB, which an upload from pageable memory delivers last"""
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 50, (n, 3))
    for _ in range(10 if n < 1000000 else 1):
        sys = mdf.MDSystem(pos, (50.0,) * 3, precision=1)
        assert np.array_equal(sys.positions(), pos)
    v = rng.normal(size=(n, 3))
    sys.set_velocities(v)
    assert np.array_equal(sys.velocities(), v)


def test_two_threads_read_frames(mdf):
    """each thread's system comes back unmixed while both read through the device's shared memory"""
    import threading
    rng = np.random.default_rng(5)
    pos = [rng.uniform(0, 50, (n, 3)) for n in (150000, 70001)]
    sys = [mdf.MDSystem(p, (50.0,) * 3, precision=1) for p in pos]
    wrong = []

    def read(s, p):
        for _ in range(40):
            if not np.array_equal(s.positions(), p):
                wrong.append(len(p))
                return

    th = [threading.Thread(target=read, args=a) for a in zip(sys, pos)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not wrong


LAST_SYSTEM = """
import numpy as np, torch, mdforce as mdf
def free_after_a_frame(n):
    sys = mdf.MDSystem(np.zeros((n, 3)), (50.0,) * 3, precision=1)
    sys.positions()
    del sys
    return torch.cuda.mem_get_info()[0]
before = free_after_a_frame(10)
print(before - free_after_a_frame(2000000))
"""


def test_last_system_gives_its_staging_back(mdf):
    """the device's pool is empty when the last system that used it is gone (a process of its own: no other system)"""
    import os
    import subprocess
    import sys
    env = dict(os.environ, PYTHONPATH=os.path.dirname(os.path.dirname(mdf.__file__)))
    out = subprocess.run([sys.executable, "-c", LAST_SYSTEM], env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert int(out.stdout) < 24 << 20  # of the 48 MB that a frame took


def test_map_after_one_that_memory_does_not_hold(mdf):
    with pytest.raises(mdf.core.MDExcptCuda):
        mdf.ErrorEstimate_SPME_Ik((1024, 1024, 1024), (30.0,) * 3, 0.95, 6)
    em = mdf.ErrorEstimate_SPME_Ik((16, 16, 16), (30.0,) * 3, 0.95, 6)
    assert np.isfinite(em.rms()).all()
