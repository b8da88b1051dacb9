"""The switching function where its distance is not below the cutoff: such a
system has plain Lennard-Jones forces, as in the oracle, which asks r > distance
of pairs inside the cutoff.  Distances at the cutoff, one FP64 step below it
(the same FP32 number), just above it and far above; and one batch that holds a
switched system, one whose cutoff is the distance and one whose cutoff is below.

Tolerances as everywhere: forces FP64 1e-9, mixed 1e-5 of the norm; energy terms
1e-9 and 2e-5 of the largest term.
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gas(n, box, seed, cutoff):
    """n charged Lennard-Jones atoms, none closer than 0.14 nm, no bonds."""
    rng = np.random.default_rng(seed)
    per = int(np.ceil(n ** (1 / 3)))
    a = box / per
    sites = (np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    half = min(0.5 * (a - 0.14), 0.2)
    pos = sites[rng.choice(len(sites), n, replace=False)] + rng.uniform(-half / 2, half / 2, (n, 3))
    q = rng.uniform(-0.2, 0.2, n)
    e2, f2 = np.zeros((0, 2), np.int32), np.zeros((0, 2))
    return types.SimpleNamespace(
        n=n, pos=np.mod(pos, box), mass=np.full(n, 12.0), charge=q - q.mean(), sigma=rng.uniform(0.2, 0.3, n),
        epsilon=rng.uniform(0.3, 0.9, n), bonds=e2, bond_prm=f2, angles=np.zeros((0, 3), np.int32), angle_prm=f2,
        torsions=np.zeros((0, 4), np.int32), torsion_prm=f2, torsion_n=np.zeros(0, np.int32), cutoff=cutoff,
        ewald_tol=5e-4, box=np.full(3, float(box)), grid=(24, 24, 24))


def _oracle(oracle, s, switch):
    lb, ub = np.zeros(3), s.box.copy()
    off, lst = oracle.exclusions(s.n, s.bonds)
    d = oracle.describe(s, box_mode=1, lb=lb, ub=ub, use_switch=1, switch_dist=switch, switch_quirk=0)
    return oracle.forces(d, s.pos, oracle.box_explicit(lb, ub), off, lst)


def _compare(F, E, F0, E0, precision):
    err = np.linalg.norm(F - F0) / np.linalg.norm(F0)
    print("force", err, {k: (E[k], E0[k]) for k in ("coulomb", "vdw")})
    assert err <= (1e-5 if precision else 1e-9)
    scale = max(abs(E0[k]) for k in ("coulomb", "vdw", "recip", "self"))
    for k in ("coulomb", "vdw"):
        assert abs(E[k] - E0[k]) <= (2e-5 if precision else 1e-9) * scale + 1e-6, (k, E[k], E0[k])


@pytest.mark.parametrize("switch", [1.0, float(np.nextafter(1.0, 0.0)), float(np.nextafter(1.0, 2.0)), 1.2, 50.0])
@pytest.mark.parametrize("precision", [0, 1])
def test_switch_not_below_the_cutoff(oracle, switch, precision):
    from nexusmd_gb300.engine import Engine
    s = _gas(700, 2.4, 7, 1.0)
    F0, E0 = _oracle(oracle, s, switch)
    eng = Engine(s, precision=precision, box="explicit", use_switch=1, switch_dist=switch)
    F = eng.compute_forces()
    E = eng.energies()
    eng.close()
    _compare(F, E, F0, E0, precision)


@pytest.mark.parametrize("precision", [0, 1])
def test_switch_in_some_systems_of_a_batch(oracle, precision):
    from nexusmd_gb300.engine import Engine
    switch = 0.9
    systems = [_gas(700, 2.4, 11, 1.1), _gas(500, 2.2, 12, 0.9), _gas(611, 2.3, 13, 0.8)]
    eng = Engine(systems, precision=precision, box="explicit", use_switch=1, switch_dist=switch)
    F = eng.compute_forces()
    at = 0
    for k, s in enumerate(systems):
        F0, E0 = _oracle(oracle, s, switch)
        _compare(F[at:at + s.n], eng.energies(k), F0, E0, precision)
        at += s.n
    eng.close()
