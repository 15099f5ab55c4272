"""The persistent sweep (one cooperative launch, each CTA holding its share of the slots) against the
oracle where its plan can go wrong: fewer slots than one chunk, ragged and uneven colour groups, both
ways of clearing the marks, code words shared between CTAs, more candidates per thread than are
prepared ahead, neighbour references that do not fit in shared memory, walls. Integers: every
comparison is exact."""
import numpy as np
import pytest

import pscbfm_b200 as P
from oracle import oracle as O
from pscbfm_b200 import systems as S

pytestmark = pytest.mark.gpu


def _linked_melt(side, phi, every):
    """Serpentine chains with bonds along y and z between some monomers two cells apart in adjacent rows:
    four bonds on some monomers (64-bit codes), neighbours far apart in the numbering."""
    s = S.serpentine_chains(side, 64, phi, seed=19)
    rows, cols = s.bonds()
    bonds = [np.stack([rows, cols], axis=1)[rows < cols]]
    for axis, step in ((1, (0, 2, 0)), (2, (0, 0, 2))):
        order = np.lexsort((s.xyz[:, axis], s.xyz[:, 3 - axis], s.xyz[:, 0]))
        a, b = order[:-1], order[1:]
        pair = np.all(s.xyz[b] - s.xyz[a] == step, axis=1) & ((s.xyz[a, axis] // 2) % 2 == 0) & (np.abs(b - a) > 1)
        bonds.append(np.stack([a[pair], b[pair]], axis=1)[::every])
    return S.from_bonds(s.box, s.xyz, np.concatenate(bonds), seed=23)


CASES = {
    "one_chunk": (lambda: S.serpentine_chains(64, 20, 0.0001, seed=3), [1, 60]),
    "ragged_33": (lambda: S.from_bonds((128, 128, 128), [[2 * j, 0, 0] for j in range(33)],
                                       [(j, j + 1) for j in range(32)], seed=5), [40, 1, 60]),
    "dilute_listed_marks": (lambda: S.serpentine_chains(128, 37, 0.02, seed=7), [3, 40]),
    "dense_cleared_marks": (lambda: S.serpentine_chains((64, 128, 64), 13, 0.45, seed=9), [1, 25]),
    "three_colours": (lambda: S.rings_and_free(64), [30, 7]),
    "walls_ragged_box": (lambda: S.walled(S.serpentine_chains((100, 64, 90), 41, 0.3, seed=11), walls=5), [20, 20]),
    "linked_64bit": (lambda: _linked_melt(64, 0.9, 1), [25]),
    "melt_1_9M_refs_in_global": (lambda: S.serpentine_chains(256, 64, 0.9, seed=13), [2]),
    "linked_1_9M_64bit": (lambda: _linked_melt(256, 0.9, 5), [2]),
}


@pytest.mark.parametrize("name", list(CASES))
def test_persistent_sweep_vs_oracle(name):
    build, chunks = CASES[name]
    s = build()
    u = P.UpdaterGPUScBFM_AB_Type(0)
    u.load_system(s, mode=P.MODE_PERSISTENT)
    assert u.path() == P.MODE_PERSISTENT
    assert u.representation() == (1 if int(s.nbr_count.max()) <= 3 else 2)
    for c in chunks:
        u.runSimulationOnGPU(c)
    want, ost = O.run(s, sum(chunks))
    st = u.stats()
    assert np.array_equal(u.get_coords(), want), name
    assert (st["attempted"], st["tentative"], st["accepted"]) == ost
    u.validate()
    # the launch leaves no marks behind: another path goes on from its state
    u.set_mode(P.MODE_GRAPH)
    u.runSimulationOnGPU(2)
    assert np.array_equal(u.get_coords(), O.run(s, sum(chunks) + 2)[0]), name
    u.close()


def test_auto_takes_one_launch_for_long_runs_of_the_melt():
    """AUTO on the 1M-monomer melt: a run of 5 MCS replays the graph (two launches per sub-step), one
    of 6 MCS is a single persistent launch; mixed, the positions stay the oracle's."""
    s = S.dense_melt()
    u = P.UpdaterGPUScBFM_AB_Type(0).load_system(s)
    counts = []
    for n in (5, 6, 1, 7):
        before = u.launch_count()
        u.runSimulationOnGPU(n)
        counts.append(u.launch_count() - before)
    assert counts[0] == 2 * 2 * 5 and counts[2] == 2 * 2 * 1
    assert counts[1] <= 2 and counts[3] <= 2   # the sweep, and the scrub of the graph's last marks
    assert np.array_equal(u.get_coords(), O.run(s, 19)[0])
    u.close()


@pytest.mark.parametrize("make", [lambda: S.serpentine_chains(64, 8, 0.5, seed=3), lambda: S.serpentine_chains(64, 64, 0.6, seed=3),
                                  lambda: S.serpentine_chains((32, 128, 128), 8, 0.3, seed=3),
                                  lambda: S.walled(S.serpentine_chains((64, 64, 50), 37, 0.7, seed=3), 4)])
def test_auto_between_cluster_and_persistent(make):
    """AUTO's choice between the cluster and the persistent sweep depends on the run's length: runs of one
    MCS and longer ones in turn, on both sides of the line, give the oracle's positions and counters."""
    s = make()
    u = P.UpdaterGPUScBFM_AB_Type(0).load_system(s)
    for n in (1, 3, 1, 2):
        u.runSimulationOnGPU(n)
    want, ost = O.run(s, 7)
    st = u.stats()
    assert np.array_equal(u.get_coords(), want)
    assert (st["attempted"], st["tentative"], st["accepted"]) == ost
    u.validate()
    u.close()
