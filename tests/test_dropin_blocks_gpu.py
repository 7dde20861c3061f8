"""The drop-in energy kernel at the edges of its blocks (32 residues), tiles (128) and CTA
shapes (one, two or four x blocks a CTA), against the FP64 oracle: every exclusion rule,
both crowder forms, periodic and open boxes.  (test_dropin_gpu.py holds the packing, the
golden totals and the entry points.)

The systems here are cut off anywhere and their totals cancel (some to 1/100 of their
largest term), so the bound is on the terms: sigma^2 / r^2 in FP32 is within 4e-7 of
itself (three roundings in r^2, two in sigma^2, 2^-23 of the SFU reciprocal), s^12
within six times that and the contact energy's rounding, 2.6e-6; a Debye-Hueckel term
(rsqrt, ex2 and an argument of a few tens at most) within 4e-6.  So a total lies within
4e-6 of the sum of its terms' magnitudes.
"""
import numpy as np
import pytest

import cgppd_gb300
import oracle
from test_dropin_gpu import ABS, L, eon, synthetic_packed  # noqa: F401  (L: fixture)

pytestmark = pytest.mark.gpu


def cut(pos, meta, n):
    """The first n records (no padding after them: the call's size is n)."""
    return np.ascontiguousarray(pos[:n]), np.ascontiguousarray(meta[:n])


def magnitudes(pos, meta, table20, box, nc, rc):
    """Sum of the magnitudes of the pair terms in kcal/mol (FP64), excluded pairs left out."""
    real = pos[:, 3] != -2.0
    pos, meta = pos[real].astype(np.float64), meta[real].astype(np.float64)
    dom, mol = np.trunc(pos[:, 3]), np.trunc(meta[:, 3])
    bond, chain, crowd = pos[:, 3] - dom, meta[:, 3] - mol, meta[:, 3] == -1.0
    eps = 0.159 * (np.asarray(table20, np.float64).reshape(20, 20) + 2.27)
    total = 0.0
    for a in range(len(pos)):
        b = slice(a + 1, None)
        d = pos[b, :3] - pos[a, :3]
        if box:
            d -= box * np.round(d / box)
        r = np.sqrt((d * d).sum(1)) + 1e-30
        gap = np.arange(a + 1, len(pos)) - a
        if nc:
            keep = ~crowd[b] & ~crowd[a] & (mol[b] != mol[a])
        else:
            keep = ~(((dom[a] != 0) & (dom[b] == dom[a])) | ((bond[a] != 0) & (bond[b] == bond[a])) |
                     ((chain[b] == chain[a]) & (gap < 4)))
        e = eps[int(meta[a, 0]), meta[b, 0].astype(int)]
        s6 = (0.5 * (meta[a, 2] + meta[b, 2]) / r) ** 6
        u = np.abs(4 * e) * s6 * (s6 + 1) + np.abs(2 * e) * (s6 > 0.5) * (e > 0)
        u = 0.5922 * u + 4.151 * np.abs(meta[a, 1] * meta[b, 1]) * np.exp(-r / 10) / r
        if rc:
            u = np.where(crowd[a] | crowd[b], 0.5922 * (6 / r) ** 12 * (r < 15.1), u)
        total += float(u[keep].sum())
    return total


def check(L, refdata, pos, meta, box, rc=False):
    before = L.cgppd_set_repulsive_crowding(int(rc))
    try:
        for nc in (False, True):
            kw = {} if nc or not rc else {"repulsive_crowding": True}
            ref = oracle.E_packed(oracle.FP64, pos, meta, refdata["lj_table"], box, nc=nc, **kw)[2]
            g = eon(L, pos, meta, box, nc=nc)
            terms = magnitudes(pos, meta, refdata["lj_table"], box, nc, rc)
            assert abs(g - ref) <= 4e-6 * terms + ABS, (nc, rc, g, ref, terms)
    finally:
        L.cgppd_set_repulsive_crowding(before)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 160, 257])
@pytest.mark.parametrize("flexible", [0.0, 0.3])
def test_block_edges(L, refdata, n, flexible):  # noqa: F811
    rng = np.random.default_rng(n)
    pos, meta = cut(*synthetic_packed(rng, 9, [30, 61, 17], 90.0, flexible), n)
    for box in (90.0, 0.0):
        check(L, refdata, pos, meta, box)


# tiles on both sides of the shapes' limits (34 and 40 tiles), a partial last tile
@pytest.mark.parametrize("n", [27 * 128, 27 * 128 + 1, 28 * 128 - 31, 33 * 128, 33 * 128 + 1, 39 * 128,
                               39 * 128 + 5, 41 * 128 + 77])
def test_cta_shapes(L, refdata, n):  # noqa: F811
    rng = np.random.default_rng(n)
    pos, meta = cut(*synthetic_packed(rng, 52, [60, 160, 97], 260.0, 0.1, crowders=4), n)
    check(L, refdata, pos, meta, 260.0)


@pytest.mark.parametrize("rc", [False, True])
def test_crowders_among_molecules(L, refdata, rc):  # noqa: F811
    rng = np.random.default_rng(3)
    pos, meta = synthetic_packed(rng, 7, [40, 90, 33], 110.0, 0.2, crowders=9)
    check(L, refdata, pos, meta, 110.0, rc=rc)


def test_no_charges_and_all_charged(L, refdata):  # noqa: F811
    rng = np.random.default_rng(8)
    pos, meta = synthetic_packed(rng, 5, [77], 120.0)
    for q in (0.0, 1.0):
        m = meta.copy()
        m[pos[:, 3] != -2.0, 1] = q
        check(L, refdata, pos, m, 120.0)
