"""The engine's calls while the default stream, which its own stream does not wait for, has
work to do."""
import numpy as np
import pytest
import torch

from cgppd_gb300 import engine as eng
from cgppd_gb300 import workloads

pytestmark = pytest.mark.gpu


def busy():
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s on the default stream


LEGACY = 1  # cudaStreamLegacy


def build(config="c4", nrep=4, cluster=2, threads=256):
    wl = workloads.make(config)
    s = wl.sims[0]
    wl.sims = [workloads.Simulation(s.molecules, s.box, s.temperatures[:nrep], s.translate_steps[:nrep],
                                    s.rotate_steps[:nrep], s.move_weights, s.rigid_rotate_prob)]
    return eng.from_workload(wl, cluster=cluster, threads=threads)


def test_first_recompute():
    """The scratch energies are cleared before the first evaluation into them."""
    e = build()
    want = e.recompute(write_state=True)
    busy()
    got = e.recompute(write_state=False)
    torch.cuda.synchronize()
    assert np.array_equal(got, want)
    assert np.array_equal(e.recompute(write_state=False), want)
    e.close()


def positions(e):
    return np.concatenate([e.state(0, r)[0] for r in range(4)])


def test_blocks_on_the_default_stream_and_then_on_the_engines():
    """A block waits for the one before it on a stream that synchronises with the default one."""
    e = build()
    e.run(1, 60)
    e.run(1, 60)
    e.synchronize()
    want, pot = positions(e), e.replicas(0)["potential"]
    e.close()
    e = build()
    busy()
    e.run(1, 60, stream=LEGACY)
    e.run(1, 60)
    e.synchronize()
    assert np.array_equal(positions(e), want) and np.array_equal(e.replicas(0)["potential"], pot)
    e.close()


def test_state_set_and_recomputed(tmp_path):
    """The state that set_state or restore returns from is the one that is evaluated next."""
    a = build()
    a.run(1, 60)
    a.synchronize()
    want, states = a.recompute(write_state=False), [a.state(0, r) for r in range(4)]
    a.checkpoint(tmp_path / "state.ck")
    b = build()
    busy()
    for r in range(4):
        b.set_state(0, r, *states[r])
    assert np.array_equal(b.recompute(write_state=True), want)
    c = build()
    busy()
    c.restore(tmp_path / "state.ck")
    assert np.array_equal(c.recompute(write_state=False), want)
    for e in (a, b, c):
        e.close()


def test_shape_tuned_behind_a_busy_default_stream():
    """Every trial launch runs on a copy of the state that is complete."""
    busy()
    e = build(nrep=7, cluster=0, threads=0)
    assert len(e.tuning()) > 0
    e.run(1, 40)
    e.synchronize()
    assert e.error_bits() == 0
    assert np.allclose(e.replicas(0)["potential"], e.recompute(write_state=False), rtol=1e-5, atol=1e-6)
    e.close()
