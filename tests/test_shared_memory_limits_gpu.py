"""Systems whose per-molecule records fill a CTA's shared memory almost to its end."""
import numpy as np
import pytest

from cgppd_gb300 import CgppdError
from cgppd_gb300 import engine as eng
from cgppd_gb300 import workloads

pytestmark = pytest.mark.gpu


def many_small(count, cluster):
    """One molecule of 32 residues among `count` - 1 of three, on a grid."""
    rng = np.random.default_rng(2)
    e = eng.Engine(workloads.contact_table(rng), seed=3)
    side = int(np.ceil(count ** (1 / 3)))
    box = 24.0 * side
    s = e.add_simulation([300.0, 320.0], [1.0, 1.0], [0.2, 0.2], box)
    for k in range(count):
        n = 32 if k == 0 else 3
        at = 24.0 * np.array([k % side, k // side % side, k // side ** 2]) + 12.0
        step = np.array([3.8, 0.0, 0.0]) if n == 3 else rng.normal(size=(32, 3))
        xyz = at + (np.arange(3)[:, None] - 1) * step if n == 3 else at + 3.0 * step
        e.add_molecule(s, xyz, rng.integers(0, 20, n), rng.choice([-1.0, 0.0, 1.0], n), np.full(n, 5.0))
    e.finalize(cluster, 256)
    return e


@pytest.mark.parametrize("count,cluster", [(860, 8), (1130, 4)])
def test_nearly_full(count, cluster):
    e = many_small(count, cluster)
    e.run(2, 50)
    e.synchronize()
    assert e.error_bits() == 0
    assert np.allclose(e.replicas(0)["potential"], e.recompute(write_state=False), rtol=1e-5, atol=1e-6)
    e.close()


def test_shape_that_is_tried_and_does_not_fit():
    """868 molecules over 8 CTAs pass the size check, but not with the kernel's own part: the
    tuner goes on to another shape, and the failed try leaves no error to a later launch."""
    e = many_small(868, 0)
    assert 8 not in [c for c, _, _ in e.tuning()] and len(e.tuning()) > 0
    e.run(2, 50)
    e.synchronize()
    assert e.error_bits() == 0
    e.close()


def test_past_the_end():
    with pytest.raises(CgppdError):
        many_small(900, 8)
