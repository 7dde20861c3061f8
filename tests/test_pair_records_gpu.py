"""The packed pair loops at the edges of their layouts, against the FP64 oracle with the
bound of the other energy tests (1e-5 relative).

* k_mc's mover records (two residues to a record, g lanes a residue j, charged span
  first): molecules from 1 residue up, odd counts, none or all residues charged, rigid
  and flexible movers, cluster and thread shapes that change g, resident or not;
* proposals prepared a step ahead: movers with more residues than the threads that prepare
  them, one molecule (never ahead), two (often not), a flexible one among rigid ones;
* k_init_pairs' groups (128 and 256 residues of whole molecules): molecules at and past
  the limits, many small ones, crowders with and without the repulsive term.
"""
import numpy as np
import pytest

import oracle
from cgppd_gb300 import workloads
from test_engine_gpu import REL, engine_for, oracle_for, oracle_matrix

pytestmark = pytest.mark.gpu


def system(lengths, box, crowders=0, seed=5, charge=None, segments=None, nrep=2, repulsive=False):
    rng = np.random.default_rng(seed)
    sigma = rng.uniform(4.5, 7.0, size=21).astype(np.float32)
    sim = workloads.rigid_sim(rng, lengths, box, nrep, sigma, crowders=crowders)
    if charge is not None:
        for m in sim.molecules[:len(lengths)]:
            m.charges[:] = charge
    for k, s in (segments or {}).items():
        sim.molecules[k].segments = [list(s)]
    sim.repulsive_crowding = repulsive
    V, S = rng.uniform(0.0, 1.5, size=(20, 20, 4)), rng.uniform(0.0, 6.28, size=(20, 20, 4))
    return workloads.Workload("pairs", [sim], workloads.contact_table(rng, with_crowder=True), V, S, seed=seed)


def check_state(e, wl, o):
    sim = wl.sims[0]
    pot = e.replicas(0)["potential"]
    for r in range(len(sim.temperatures)):
        xyz, _, _ = e.state(0, r)
        e64 = o.energy_of(xyz, oracle.FP64)
        assert abs(pot[r] - e64) <= REL * abs(e64) + 1e-6, (r, pot[r], e64)
        if not sim.repulsive_crowding:
            ref = oracle_matrix(wl, sim, xyz.astype(np.float32))
            E, _ = e.matrix(0, r)
            assert np.all(np.abs(E - ref) <= REL * np.abs(ref) + 1e-7 * np.abs(ref).max())
    assert e.error_bits() == 0


SMALL = [1, 2, 3, 7, 33, 64, 76]            # full term for every residue
LARGE = [1, 2, 5, 31, 33, 65, 97, 130]      # charged residues first


@pytest.mark.parametrize("cluster,threads", [(1, 128), (1, 512), (3, 256), (8, 512)])
@pytest.mark.parametrize("lengths,charge", [(SMALL, None), (LARGE, None), (LARGE, 0.0), (LARGE, 1.0)])
def test_mover_records(lengths, charge, cluster, threads):
    wl = system(lengths, 170.0, charge=charge)
    o = oracle_for(wl, wl.sims[0])
    for resident in (True, False):
        e = engine_for(wl, wl.sims, cluster=cluster, threads=threads, resident=resident)
        e.run(2, 40)
        e.synchronize()
        check_state(e, wl, o)
        e.close()


@pytest.mark.parametrize("cluster,threads", [(1, 128), (4, 256)])
def test_flexible_mover_among_others(cluster, threads):
    wl = system([33, 40, 7], 120.0, segments={0: range(10, 16), 1: range(20, 31)})
    o = oracle_for(wl, wl.sims[0])
    for resident in (True, False):
        e = engine_for(wl, wl.sims, cluster=cluster, threads=threads, resident=resident)
        e.run(2, 40)
        e.synchronize()
        check_state(e, wl, o)
        e.close()


# Proposals prepared a step ahead (resident launches) against launches that never do
# (global state).  Both take the same draws, so they stay together: each of the 60 steps
# rounds the mover's coordinates (below 256 A, 1.5e-5 A) and no decision is that close.
@pytest.mark.parametrize("lengths,segments", [([40], {}), ([97, 30], {}), ([230, 1, 96, 98], {}), ([12] * 9, {}),
                                              ([33, 40, 120], {1: range(20, 31)})])
@pytest.mark.parametrize("cluster,threads", [(1, 128), (4, 256)])
def test_proposals_a_step_ahead(lengths, segments, cluster, threads):
    same_with_and_without_resident_state(system(lengths, 200.0, segments=segments, seed=11), cluster, threads)


# 4,600 residues over four CTAs: the replica fits shared memory, a second proposal does not
def test_no_room_for_a_second_proposal():
    same_with_and_without_resident_state(system([400] * 11 + [200], 250.0, seed=12), 4, 256)


def same_with_and_without_resident_state(wl, cluster, threads):
    state = {}
    for resident in (True, False):
        e = engine_for(wl, wl.sims, cluster=cluster, threads=threads, resident=resident)
        assert e.launch_shape() == (cluster, threads, resident)
        e.run(2, 30)
        e.synchronize()
        check_state(e, wl, oracle_for(wl, wl.sims[0]))
        state[resident] = [e.state(0, r)[0] for r in range(len(wl.sims[0].temperatures))]
        e.close()
    for a, b in zip(state[True], state[False]):
        assert np.abs(a - b).max() < 2e-3


@pytest.mark.parametrize("repulsive", [False, True])
@pytest.mark.parametrize("lengths,crowders", [([1], 1), ([128, 129, 1], 0), ([256, 257, 40], 30), ([300, 76, 20], 0),
                                              ([17] * 12, 9)])
def test_energies_from_scratch(lengths, crowders, repulsive):
    wl = system(lengths, 260.0, crowders=crowders, repulsive=repulsive and crowders > 0)
    e = engine_for(wl, wl.sims, cluster=1, threads=256)
    o = oracle_for(wl, wl.sims[0], repulsive_crowding=wl.sims[0].repulsive_crowding)
    check_state(e, wl, o)
    assert np.allclose(e.recompute(False), e.replicas(0)["potential"], rtol=1e-12, atol=1e-12)
    e.run(1, 20)
    e.synchronize()
    check_state(e, wl, o)
    e.close()
