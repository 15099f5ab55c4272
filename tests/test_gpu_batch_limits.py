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


@pytest.mark.parametrize("name", ["resident", "gather", "cluster", "slab"])
def test_long_batch_runs_are_several_launches(name):
    """The kernels that hold a system for many sub-steps count a CTA's moves in 32 bits: a launch has at most
    65536 sub-steps (times 16384 slots of a colour: 2^30 moves), and a longer run is several launches of the
    same trajectory and counters, for members that end within the first or the second of them."""
    mcs = 32768 + 700   # of two colours: 65536 sub-steps and 1400
    s = {"cluster": S.small_chains(), "slab": S.serpentine_chains(64, 64, 0.8, seed=13)}.get(
        name, S.serpentine_chains(32, 16, 0.05, seed=40))
    repr_ = P.REPR_GATHER if name == "gather" else P.REPR_AUTO
    members = [load(s, seed=q, representation=repr_) for q in (5, 6, 7)]
    b = P.Batch(members, cluster=name in ("cluster", "slab"))
    b.run(1)
    n0 = b.launch_count()
    b.run_each([mcs, 900, mcs - 600])
    assert b.launch_count() - n0 == 2
    for q, m, k in zip((5, 6, 7), members, (mcs, 900, mcs - 600)):
        u = load(s, seed=q, representation=repr_)
        u.runSimulationOnGPU(1)
        u.runSimulationOnGPU(k)
        assert m.stats() == u.stats() and m.substep() == u.substep()
        assert np.array_equal(m.get_coords(), u.get_coords())
        m.validate()
        u.close()
    b.close()


def test_failed_sweep_is_reported_by_every_later_sweep():
    """A system whose sweep timed out (injected on the host) is not advanced again, and no later sweep of it
    returns as if it were: in the batch after its plan was made anew, in another batch, alone; a run that was
    never waited for is reported too. The other members go on, and a system set up again is a new one."""
    s = S.serpentine_chains(128, 32, 0.1, seed=3)
    a, c = load(s, seed=1), load(s, seed=2)
    b = P.Batch([a, c])
    a.inject_barrier_stall()
    with pytest.raises(P.BfmCudaError, match="timed out"):
        b.run(2)
    for on in (False, True):   # (the plan is made again, with reports of its own)
        b.set_cluster(on)
    with pytest.raises(P.BfmCudaError, match="timed out"):
        b.run(1)
    other = P.Batch([a])
    with pytest.raises(P.BfmCudaError, match="timed out"):
        other.run(1)
    other.run_async(1)         # two runs of two batches, neither waited for
    b.run_async(1)
    with pytest.raises(P.BfmCudaError, match="timed out"):
        a.synchronize()
    other.close()
    a.set_mode(P.MODE_PERSISTENT)
    with pytest.raises(P.BfmCudaError, match="timed out"):
        a.runSimulationOnGPU(1)
    b.close()
    assert np.array_equal(c.get_coords(), O.run(s, 4, seed=2)[0])
    a.cleanup()
    load_again = a.load_system(s, seed=1, mode=P.MODE_PERSISTENT)
    load_again.runSimulationOnGPU(3)
    assert np.array_equal(a.get_coords(), O.run(s, 3, seed=1)[0])


def test_stalled_sweep_ends_at_its_limit_of_two_seconds():
    """A wait that cannot end (injected on the host) ends after 2 s, alone and in a batch: the GPU is not held
    longer. (The CTAs of a cooperative launch start together, so no wait depends on other streams' work.)"""
    import time
    s = S.serpentine_chains(128, 32, 0.1, seed=3)
    u = load(s, mode=P.MODE_PERSISTENT)
    u.runSimulationOnGPU(1)
    m = load(s)
    b = P.Batch([m])
    b.run(1)
    for stalled, run in ((u, lambda: u.runSimulationOnGPU(2)), (m, lambda: b.run(2))):
        stalled.inject_barrier_stall()
        t = time.perf_counter()
        with pytest.raises(P.BfmCudaError, match="timed out"):
            run()
        assert 1.0 < time.perf_counter() - t < 8.0
    b.close()


def test_clusters_of_both_code_widths_run_side_by_side():
    """Chains (32-bit codes) and chains linked across (64-bit) on clusters are two launches; neither waits
    for the other: together they take less than one after the other."""
    chains = S.serpentine_chains((64, 64, 32), 32, 0.6, seed=64)
    rows, cols = chains.bonds()
    at = {tuple(r): i for i, r in enumerate(chains.xyz)}
    across = [(i, at[q]) for r, i in at.items() for q in ((r[0], r[1] + 2, r[2]), (r[0], r[1], r[2] + 2))
              if q in at and abs(at[q] - i) > 1][::3]
    bonds = {(int(min(p)), int(max(p))) for p in [*zip(rows, cols), *across]}
    linked = S.from_bonds(chains.box, chains.xyz, sorted(bonds), seed=65)
    assert linked.nbr_count.max() > 3
    kinds = [chains, linked]

    def timed(systems):
        members = [load(s) for s in systems]
        b = P.Batch(members)
        n0 = b.launch_count()
        b.run(20)
        assert b.launch_count() - n0 == len(systems)   # a cluster launch each, and no resident one
        ms = min(b.run_timed(300) for _ in range(3))
        for s, m in zip(systems, members):
            assert np.array_equal(m.get_coords(), O.run(s, 20 + 3 * 300)[0])
            m.validate()
        b.close()
        return ms

    one, other, both = timed(kinds[:1]), timed(kinds[1:]), timed(kinds)
    assert both < 0.85 * (one + other), (one, other, both)


def test_short_runs_of_many_large_members_take_the_grid_phase():
    """64 systems of 29K monomers are two launches of slab sweeps, which load and write back every slot: a run of
    one MCS takes the grid-phase kernels instead (two launches per sub-step). The trajectories go on across both,
    and across changes of the members and of the kernels' settings."""
    s = S.serpentine_chains(64, 64, 0.9, seed=5)
    members = [load(s, seed=200 + i) for i in range(64)]
    b = P.Batch(members)

    def launches(run, *a):
        n0 = b.launch_count()
        run(*a)
        return b.launch_count() - n0

    assert launches(b.run, 1) == 4
    assert launches(b.run, 3) == 2
    assert launches(b.run, 1) == 4
    b.set_block(128)
    assert launches(b.run, 1) == 4
    assert launches(b.run_each, [2] * 3 + [1] * 61) == 2
    b.set_cluster(False)
    assert launches(b.run, 2) == 8
    b.set_cluster(True)
    b.run_timed(1)
    b.run_async(1)
    b.run_async(2)
    for i in (0, 2, 3, 40, 63):
        k = 1 + 3 + 1 + 1 + (2 if i < 3 else 1) + 2 + 1 + 1 + 2
        want, ost = O.run(s, k, seed=200 + i)
        st = members[i].stats()
        assert np.array_equal(members[i].get_coords(), want), i
        assert (st["attempted"], st["tentative"], st["accepted"]) == ost and st["mcs"] == k
        members[i].validate()
    b.close()


def test_autotuner_with_short_trials_picks_the_path_of_long_runs():
    """Trials of two MCS are no measure of what a launch costs however long it runs: 96 systems of 60K monomers,
    whose slab sweeps take longer than the grid phase for two MCS and less for a hundred, are tuned for the sweeps."""
    s = S.serpentine_chains(128, 64, 0.23, seed=5)
    members = [load(s, seed=300 + i) for i in range(96)]
    b = P.Batch(members)
    b.run(3)
    rep = b.autotune(2)
    spent = 3 + rep["mcs_spent"]
    assert rep["cluster"], rep["trials"]
    tuned = min(b.run_timed(40) for _ in range(2))
    b.set_cluster(False)
    other = min(b.run_timed(40) for _ in range(2))
    assert tuned < other
    want, ost = O.run(s, spent + 160, seed=395)
    st = members[95].stats()
    assert np.array_equal(members[95].get_coords(), want)
    assert (st["attempted"], st["tentative"], st["accepted"]) == ost
    b.close()


def timed_in_threads(runs, times=3):
    """The least wall time of `times` rounds in which every function of runs is called 8 times on a thread of its own."""
    import threading
    import time

    def again(run):
        for _ in range(8):
            run()

    best = 1e9
    for _ in range(times):
        threads = [threading.Thread(target=again, args=(r,)) for r in runs]
        t = time.perf_counter()
        for x in threads:
            x.start()
        for x in threads:
            x.join()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("name,most", [("60K", 2.5), ("131K", 2.8), ("8K", 2.5)])
def test_threads_share_the_sms(name, most):
    """Eight threads that each run a system of their own again and again: sweeps that take most of the SMs alone run
    side by side on fewer, with the trajectories of each alone, in much less time than one after the other."""
    s = {"60K": lambda: S.serpentine_chains(128, 64, 0.23, seed=5), "131K": lambda: S.serpentine_chains(128, 256, 0.5),
         "8K": S.small_chains}[name]()
    us = [load(s, seed=400 + i) for i in range(8)]
    alone = load(s, seed=1)
    one = timed_in_threads([lambda: alone.runSimulationOnGPU(100)])
    all8 = timed_in_threads([lambda u=u: u.runSimulationOnGPU(100) for u in us])
    for k in (7, 1):
        for u in us:
            u.run_async(k)
    for i in (0, 3, 7):
        v = load(s, seed=400 + i, mode=P.MODE_GRAPH)
        v.runSimulationOnGPU(3 * 800 + 8)
        assert us[i].stats() == v.stats() and np.array_equal(us[i].get_coords(), v.get_coords())
        us[i].validate()
        v.close()
    assert all8 < most * one, (one, all8)


@pytest.mark.parametrize("name,most", [("2x60K", 4.0), ("4x8K", 3.0)])
def test_batches_in_threads_share_the_sms(name, most):
    """The same for batches in eight threads, whose plans change with the number of others beside them, and change
    back when a batch runs alone again."""
    s, each = (S.serpentine_chains(128, 64, 0.23, seed=5), 2) if name == "2x60K" else (S.small_chains(), 4)
    members = [[load(s, seed=500 + each * i + k) for k in range(each)] for i in range(8)]
    batches = [P.Batch(m) for m in members]
    one = timed_in_threads([lambda: batches[0].run(100)])
    all8 = timed_in_threads([lambda b=b: b.run(100) for b in batches])
    again = timed_in_threads([lambda: batches[0].run(100)], times=4)
    for b in batches:
        b.run_async(3)
    for i, total in ((0, 10 * 800 + 3), (3, 3 * 800 + 3), (7, 3 * 800 + 3)):
        m = members[i][-1]
        v = load(s, seed=500 + each * i + each - 1, mode=P.MODE_GRAPH)
        v.runSimulationOnGPU(total)
        assert m.stats() == v.stats() and np.array_equal(m.get_coords(), v.get_coords())
        m.validate()
        v.close()
    assert all8 < most * one and again < 1.5 * one, (one, all8, again)
    for b in batches:
        b.close()
