"""The step graph with the lists in a conditional node of their own (large
systems) against the one-node form of a small one: 3 x 3 x 3 copies of a system
side by side in a box and on a grid three times as large move as the system
itself does, through several list builds.

Tolerance: both sides' forces are within 1e-5 (mixed) of the exact ones, of
which the two differ by 2e-5 at most; twelve steps may double that, and 1e-4 of
the change of velocity leaves as much again for the copies' spread.
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _copies(s, m):
    """m x m x m copies of s, its box and PME grid m times as large."""
    shift = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) * s.box
    t = types.SimpleNamespace(
        n=s.n * len(shift), pos=np.concatenate([np.mod(s.pos, s.box) + d for d in shift]), cutoff=s.cutoff,
        ewald_tol=s.ewald_tol, box=s.box * m, grid=tuple(int(g) * m for g in s.grid))
    for k in ("mass", "charge", "sigma", "epsilon", "bond_prm", "angle_prm", "torsion_prm", "torsion_n"):
        setattr(t, k, np.concatenate([np.asarray(getattr(s, k))] * len(shift)))
    for k in ("bonds", "angles", "torsions"):
        a = np.asarray(getattr(s, k))
        setattr(t, k, np.concatenate([a + c * s.n for c in range(len(shift))]).astype(np.int32))
    return t


def test_copies_move_as_the_system_does():
    from nexusmd_gb300 import synthetic as sy
    from nexusmd_gb300.engine import Engine
    s, big = (_copies(sy.config_system(1), m) for m in (1, 3))
    assert big.n > 64000 > s.n
    v0 = np.random.default_rng(2).normal(0.0, 0.4, (s.n, 3))
    out = []
    for t, copies in ((s, 1), (big, 27)):
        eng = Engine(t, precision=1, box="explicit", skin=0.1, rebuild_interval=5)
        eng.set_velocities(np.concatenate([v0] * copies))
        rb = eng.rebuilds()
        eng.step(12, 0.0005)
        assert eng.rebuilds() - rb >= 2
        out.append(eng.state()[1])
        eng.close()
    dv = out[0] - v0
    for c in range(27):
        err = np.linalg.norm(out[1][c * s.n:(c + 1) * s.n] - v0 - dv) / np.linalg.norm(dv)
        assert err <= 1e-4, (c, err)
    print("velocity change, last copy against the system: %.2e" % err)
