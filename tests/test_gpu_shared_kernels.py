"""The kernels that hold a system in shared memory (one CTA, or a cluster of CTAs) against the oracle
where their layouts can go wrong: lattices of one and two words, every remainder of the slots per
warp, both forms of the resident check and the group size between them, groups too large for 16-bit
list entries, neighbour references that do not fit, walls, three colours, 64-bit codes, and calls that
end inside and on the edges of a block of step entries. Integers: every comparison is exact."""
import numpy as np
import pytest

import pscbfm_b200 as P
from oracle import oracle as O
from pscbfm_b200 import systems as S

pytestmark = pytest.mark.gpu


def _free(n, side):
    """n unbonded monomers on a 2-spaced grid: one colour group of n."""
    k = np.arange(n)
    h = side // 2
    xyz = 2 * np.stack([k % h, (k // h) % h, k // (h * h)], axis=1)
    return S.from_bonds((side,) * 3, xyz, np.zeros((0, 2)), seed=29)


SYSTEMS = {
    "one_word_lattice": lambda: S.from_bonds((4, 4, 4), [[0, 0, 0], [2, 2, 2]], [], seed=2),
    "two_word_lattice": lambda: S.from_bonds((8, 4, 4), [[0, 0, 0], [2, 0, 0], [4, 0, 0]], [(0, 1), (1, 2)], seed=3),
    "group_1024": lambda: S.serpentine_chains(32, 32, 0.5, seed=5),
    "group_1056": lambda: S.serpentine_chains(32, 33, 0.52, seed=6),
    "ragged_3_per_thread": lambda: S.serpentine_chains((64, 32, 32), 31, 0.63, seed=7),
    "free_8200_direct": lambda: _free(8200, 64),
    "refs_do_not_fit": lambda: S.serpentine_chains(64, 64, 0.3, seed=8),
    "walls": lambda: S.walled(S.serpentine_chains((30, 64, 50), 17, 0.4, seed=9), walls=7),
    "three_colours": lambda: S.rings_and_free(32),
    "codes_64bit": lambda: S.square_network(64),
}


@pytest.mark.parametrize("mode", ["resident", "cluster"])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_shared_memory_kernels_vs_oracle(name, mode):
    s = SYSTEMS[name]()
    m = {"resident": P.MODE_RESIDENT, "cluster": P.MODE_CLUSTER}[mode]
    u = P.UpdaterGPUScBFM_AB_Type(0)
    u.load_system(s, mode=m)
    if mode == "resident" or name not in ("one_word_lattice",):
        assert u.path() == m
    nc = u.n_colors()[0]
    done = 0
    # sub-steps per call: below, on and across the blocks of 8 step entries
    for mcs in (1, 16 // nc, 16 // nc + 1, 33):
        u.runSimulationOnGPU(mcs)
        done += mcs
    want, ost = O.run(s, done)
    st = u.stats()
    assert np.array_equal(u.get_coords(), want)
    assert (st["attempted"], st["tentative"], st["accepted"]) == ost
    u.validate()
    u.close()


@pytest.mark.parametrize("n, side", [(8192, 64), (8193, 64), (16384, 64), (16385, 64), (32768, 128), (32769, 128)])
def test_cluster_forms_vs_oracle(n, side):
    """16, 17, 32, 33, 64 and 65 chunks of 32 slots per CTA of a cluster of 16: both sides of the edges
    between the cluster kernel's forms."""
    s = _free(n, side)
    u = P.UpdaterGPUScBFM_AB_Type(0).load_system(s, mode=P.MODE_CLUSTER)
    assert u.path() == P.MODE_CLUSTER
    for mcs in (1, 9):
        u.runSimulationOnGPU(mcs)
    want, ost = O.run(s, 10)
    st = u.stats()
    assert np.array_equal(u.get_coords(), want)
    assert (st["attempted"], st["tentative"], st["accepted"]) == ost
    u.validate()
    u.close()


@pytest.mark.parametrize("mode", ["resident", "cluster", "persistent"])
def test_entries_made_on_the_device_vs_the_callbacks(mode):
    """Kernels that run many sub-steps make the counter stream's entries themselves; a callback's come
    from the host. Both forms of the same stream, and runs that change between them, give the same system,
    also past 2^32 sub-steps."""
    s = S.serpentine_chains(32, 16, 0.4, seed=12)
    m = {"resident": P.MODE_RESIDENT, "cluster": P.MODE_CLUSTER, "persistent": P.MODE_PERSISTENT}[mode]
    for first in (0, 2**32 - 5):
        at = [0]

        def draw():
            v = P.updater.counter_draw(s.seed, at[0])
            at[0] += 1
            return v

        a, b, c = (P.UpdaterGPUScBFM_AB_Type(0) for _ in range(3))
        for u in (a, b, c):
            u.load_system(s, mode=m)
            u.set_substep(first)
        c.set_mode(P.MODE_GRAPH)
        nc = a.n_colors()[0]
        done = first
        for k, mcs in enumerate((1, 4, 7, 20)):
            a.runSimulationOnGPU(mcs)
            c.runSimulationOnGPU(mcs)
            if k % 2 == 0:
                b.runSimulationOnGPU(mcs)
            else:
                at[0] = 2 * done
                b.set_draw_callback(draw)
                b.runSimulationOnGPU(mcs)
                b.set_seed(s.seed)
                b.set_substep(done + mcs * nc)
            done += mcs * nc
            assert a.path() == m
            assert np.array_equal(a.get_coords(), b.get_coords()), (mode, first, k)
            assert np.array_equal(a.get_coords(), c.get_coords()), (mode, first, k)
        for u in (a, b, c):
            u.validate()
            u.close()


@pytest.mark.parametrize("cluster", [True, False])
def test_batch_members_with_callbacks_beside_streams(cluster):
    """Members on the counter stream, whose kernels make their entries, beside two that share one host
    generator: its draws go to them sub-step by sub-step, in the members' order."""
    systems = [S.serpentine_chains(32, 16, 0.3, seed=50), S.serpentine_chains(32, 16, 0.4, seed=51),
               S.serpentine_chains(128, 32, 0.2, seed=52), S.serpentine_chains(64, 64, 0.3, seed=53)]
    plan = [[5, 9, 3, 12], [4, 0, 6, 1]]
    called = (1, 2)
    draws = {m: [] for m in called}
    at = 0
    for mcs in plan:   # both have two colours: two draws per sub-step
        for t in range(2 * max(mcs)):
            for m in called:
                if t < 2 * mcs[m]:
                    draws[m] += [P.updater.counter_draw(77, at), P.updater.counter_draw(77, at + 1)]
                    at += 2
    k = iter(range(at))
    members = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s) for s in systems]
    for m in called:
        members[m].set_draw_callback(lambda: P.updater.counter_draw(77, next(k)))
    b = P.Batch(members)
    b.set_cluster(cluster)
    for mcs in plan:
        b.run_each(mcs)
    for m, (s, u) in enumerate(zip(systems, members)):
        mcs = sum(p[m] for p in plan)
        want = O.run(s, mcs, draws=np.array(draws[m], dtype=np.uint32)) if m in called else O.run(s, mcs)
        assert np.array_equal(u.get_coords(), want[0]), m
    b.close()


@pytest.mark.parametrize("count", [1, 7, 8, 16, 40])
def test_batch_members_on_clusters_vs_oracle(count):
    """Members that fit one CTA on the SMs a batch leaves over: clusters of 16, 8 and 4 CTAs and none at
    all, members of different sizes, 64-bit codes, a callback's member and idle ones in one launch."""
    big = [S.serpentine_chains(64, 32, 0.25, seed=60), S.serpentine_chains(64, 31, 0.22, seed=61),
           S.square_network(64), S.walled(S.serpentine_chains((64, 64, 50), 37, 0.2, seed=62), 4)]
    systems = [big[k % 4] if k < 16 else S.serpentine_chains(32, 16, 0.3, seed=63) for k in range(count)]
    members = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s) for s in systems]
    mcs = [9 - k % 5 for k in range(count)]
    k = iter(range(10**6))
    members[0].set_draw_callback(lambda: P.updater.counter_draw(systems[0].seed, next(k)))
    b = P.Batch(members)
    b.run_each(mcs)
    b.set_cluster(False)
    b.run_each(mcs)
    b.set_cluster(True)
    b.run_each(mcs)
    want = {}
    for s, m, t in zip(systems, members, mcs):
        if (id(s), t) not in want:
            want[id(s), t] = O.run(s, 3 * t)
        assert np.array_equal(m.get_coords(), want[id(s), t][0])
        st = m.stats()
        assert (st["attempted"], st["tentative"], st["accepted"]) == want[id(s), t][1]
        m.validate()
    b.close()


def test_idle_cluster_members_across_blocks_of_entries():
    """Members on clusters that idle for several blocks of step entries while another runs, one that is
    idle from the start, and runs that end on the first and the last entry of a block."""
    systems = [S.serpentine_chains(64, 32, 0.25, seed=64), S.serpentine_chains(64, 31, 0.22, seed=65),
               S.square_network(64)]
    members = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s) for s in systems]
    b = P.Batch(members)
    plan = [[40, 1, 13], [4, 25, 0], [8, 8, 8], [0, 12, 31]]
    for mcs in plan:
        b.run_each(mcs)
    for s, m, t in zip(systems, members, np.sum(plan, axis=0)):
        assert np.array_equal(m.get_coords(), O.run(s, int(t))[0]), s.name
        m.validate()
    b.close()


def test_idle_members_beside_longer_ones():
    """A batch whose members stop at different sub-steps: the shared-memory kernels skip the idle entries
    that follow a member's last sub-step, inside and across blocks of step entries."""
    systems = [S.serpentine_chains(32, 16, 0.3, seed=40), S.small_chains(), S.crosslinked_network(),
               S.rings_and_free(32), S.serpentine_chains(64, 64, 0.6, seed=41)]
    members = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s) for s in systems]
    b = P.Batch(members)
    plan = [[1, 9, 40, 5, 17], [8, 0, 3, 33, 0], [16, 16, 1, 0, 7]]
    for mcs in plan:
        b.run_each(mcs)
    for s, m, t in zip(systems, members, np.sum(plan, axis=0)):
        assert np.array_equal(m.get_coords(), O.run(s, int(t))[0]), s.name
        m.validate()
    b.close()


def test_batch_slab_sweeps_in_waves_vs_oracle():
    """More members than one cooperative launch holds (each of at least eight CTAs), beside resident members
    and a 64-bit network: the launches run one after the other, and every trajectory is its own."""
    big = S.serpentine_chains(128, 64, 0.45)
    systems = [big] * 20 + [S.crosslinked_network(), S.serpentine_chains(128, 37, 0.1), S.serpentine_chains(32, 16, 0.3)]
    members = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s, seed=60 + i) for i, s in enumerate(systems)]
    b = P.Batch(members)
    n0 = b.launch_count()
    b.run(2)
    assert b.launch_count() - n0 <= 5   # two or three waves, the 64-bit wave, the resident launch
    for i in (0, 7, 19, 20, 21, 22):
        want, ost = O.run(systems[i], 2, seed=60 + i)
        st = members[i].stats()
        assert np.array_equal(members[i].get_coords(), want), i
        assert (st["attempted"], st["tentative"], st["accepted"]) == ost
        members[i].validate()
    # alone, then in a batch again, then as two launches per sub-step
    u = members[21]
    u.set_mode(P.MODE_PERSISTENT)
    u.runSimulationOnGPU(3)
    b.run(1)
    u.set_mode(P.MODE_GRAPH)
    u.runSimulationOnGPU(2)
    assert np.array_equal(u.get_coords(), O.run(systems[21], 8, seed=81)[0])
    b.close()


def test_batch_barrier_timeout_is_reported():
    """A member whose barrier cannot complete (injected on the host) ends at the wait's time limit and the
    batch's run reports it; the device stays usable for other members."""
    s = S.serpentine_chains(128, 32, 0.1, seed=3)
    members = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s, seed=q) for q in (1, 2)]
    b = P.Batch(members)
    members[0].inject_barrier_stall()
    with pytest.raises(P.BfmCudaError, match="timed out"):
        b.run(2)
    assert np.array_equal(members[1].get_coords(), O.run(s, 2, seed=2)[0])
    b.close()
