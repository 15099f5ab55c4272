"""Long and short runs of a Batch, its reports of failed sweeps, and the shares of the SMs it plans with."""
import numpy as np
import pytest

import pscbfm_b200 as P
from oracle import oracle as O
from pscbfm_b200 import systems as S

pytestmark = pytest.mark.gpu


def load(s, seed=None, **kw):
    return P.UpdaterGPUScBFM_AB_Type(0).load_system(s, seed=seed, **kw)


def four_colours():
    """Four monomers bonded to each other: every one has a colour of its own."""
    xyz = np.array([[8, 8, 8], [10, 8, 8], [9, 10, 8], [9, 9, 10]])
    return S.from_bonds((32, 32, 32), xyz, [(a, b) for a in range(4) for b in range(a + 1, 4)], seed=4)


def test_batch_refuses_runs_past_32_bits_of_sub_steps():
    """2^30 MCS of four colours are 2^32 sub-steps: refused like the same call on the system alone, for the
    whole batch, and nothing has moved; the next run is the trajectory's first."""
    systems = [four_colours(), S.serpentine_chains(32, 16, 0.3, seed=40)]
    members = [load(s) for s in systems]
    assert members[0].n_colors()[0] == 4
    b = P.Batch(members)
    for call in (lambda: b.run(1 << 30), lambda: b.run_async(1 << 30), lambda: b.run_timed(1 << 30),
                 lambda: b.run_each([1 << 30, 1]), lambda: members[0].runSimulationOnGPU(1 << 30)):
        with pytest.raises(ValueError, match="too many sub-steps"):
            call()
    for s, m in zip(systems, members):
        assert m.stats()["mcs"] == 0 and m.substep() == 0
        assert np.array_equal(m.get_coords(), s.xyz)
    b.run(5)
    for s, m in zip(systems, members):
        assert np.array_equal(m.get_coords(), O.run(s, 5)[0])
    b.close()
