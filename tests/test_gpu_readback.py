"""Positions and counters read back into page-locked and ordinary buffers: every remainder of a warp's
share, odd offsets, sizes on both sides of the direct form's limit, more handles than one page of flags
holds, and reads behind queued work that outlasts the watch of a flag. Integers: exact."""
import numpy as np
import pytest
import torch

import pscbfm_b200 as P
from oracle import oracle as O
from pscbfm_b200 import systems as S

pytestmark = pytest.mark.gpu


def _free(n, side):
    k = np.arange(n)
    h = side // 2
    xyz = 2 * np.stack([k % h, (k // h) % h, k // (h * h)], axis=1)
    return S.from_bonds((side,) * 3, xyz, np.zeros((0, 2)), seed=29)


def _pinned(n):
    return torch.empty(3 * n + 8, dtype=torch.int32, pin_memory=True).numpy()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 1000])
def test_read_back_of_any_size_and_offset(n):
    s = _free(n, 32)
    u = P.UpdaterGPUScBFM_AB_Type(0).load_system(s)
    u.runSimulationOnGPU(7)
    want = O.run(s, 7)[0]
    assert np.array_equal(u.get_coords(), want)
    for off in range(5):
        flat = _pinned(n)
        flat[:] = -77
        u.get_coords(flat[off:off + 3 * n].reshape(n, 3))
        assert np.array_equal(flat[off:off + 3 * n].reshape(n, 3), want)
        assert (flat[:off] == -77).all() and (flat[off + 3 * n:] == -77).all()
    u.close()


@pytest.mark.parametrize("make", [lambda: S.serpentine_chains(128, 32, 0.65, seed=3),     # below 2 MB
                                  lambda: S.serpentine_chains(128, 32, 0.7, seed=3)])     # above
def test_read_back_around_the_direct_limit(make):
    s = make()
    u = P.UpdaterGPUScBFM_AB_Type(0).load_system(s)
    u.runSimulationOnGPU(3)
    want = u.get_coords()
    assert np.array_equal(want, O.run(s, 3)[0])
    assert np.array_equal(u.get_coords(_pinned(s.n)[:3 * s.n].reshape(s.n, 3)), want)
    u.close()


def test_many_handles_and_queued_work():
    s = S.serpentine_chains(32, 16, 0.3, seed=8)
    want, ost = O.run(s, 5)
    for _ in range(2):   # the second time on flags given back
        us = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s) for _ in range(70)]
        bufs = [_pinned(s.n)[:3 * s.n].reshape(s.n, 3) for _ in us]
        for u in us:
            u.run_async(5)
        for u, b in zip(us, bufs):
            u.get_coords(b)
        for k in (69, 0, 33):
            us[k].close()
        for u, b in zip(us, bufs):
            assert np.array_equal(b, want)
        for k in range(1, 33):
            st = us[k].stats()
            assert (st["attempted"], st["tentative"], st["accepted"]) == ost
        for u in us:
            u.close()
    u = P.UpdaterGPUScBFM_AB_Type(0).load_system(s)
    buf = _pinned(s.n)[:3 * s.n].reshape(s.n, 3)
    u.run_async(2000)   # several milliseconds
    u.get_coords(buf)
    assert np.array_equal(buf, O.run(s, 2000)[0])
    u.run_async(2000)
    assert u.stats()["mcs"] == 4000
    assert np.array_equal(u.get_coords(), O.run(s, 4000)[0])
    u.close()
