"""Phases that take different branches of the return map inside one warp (a
warp holds three hexes, each of its own phase): constant, softening and zero
friction angles, Drucker-Prager beside Mohr-Coulomb; single models against
the CPU oracle, batched ones against single ones.

Where every angle is constant the hooks agree with the oracle to the last
bit; an angle that softens is evaluated by the device's sin and tan, and the
viscosity by its exp and log, so those are compared at the plastic bar
(1e-6 of the field's largest value)."""
import numpy as np
import pytest

from oracle.pyoracle import Checker
from snac_b200 import workloads as W
from snac_b200.batch import SnacBatch
from snac_b200.context import SnacContext
from tests import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("coord", "velocity", "stress", "plastic_strain", "force", "inertial_mass")


def phase(cfg, phi0, phi1, psi1=0.0, c0=2.0e5):
    """cfg's phase with the friction angle softening phi0 -> phi1 over plastic strain 0.001"""
    m = dict(cfg.materials[0])
    m.update(W.mc_phase(c0=c0, c1=0.1 * c0, eps1=0.001, phi=phi1, psi=psi1, flat_tail=1.0e3))
    m["frictionAngle0"] = phi0
    return m


def mixed(base, angles, dp=()):
    """One phase per entry of angles (phi0, phi1, psi1); those numbered in dp Drucker-Prager."""
    cfg = base(5, 3, 5)
    cfg.materials = [phase(cfg, *a, c0=2.0e5 * (1 + i)) for i, a in enumerate(angles)]
    for i in dp:
        cfg.materials[i]["yieldcriterion"] = "druckerprager"
    # neighbours in a triple differ: every order of the phases occurs
    cfg.element_material = np.random.default_rng(29).integers(0, len(angles), cfg.n_elements).astype(np.int32)
    return cfg


CONST, SOFT, ZERO, DIL = (30.0, 30.0), (30.0, 15.0), (0.0, 0.0), (30.0, 30.0, 5.0)
PLASTIC, VISCO = S.plastic_small, S.viscoplastic_small
CASES = {
    "plastic_constant_zero": (PLASTIC, [CONST, ZERO], (), 0.0),
    "plastic_constant_softening": (PLASTIC, [CONST, SOFT], (), 1e-6),
    "plastic_all": (PLASTIC, [CONST, SOFT, ZERO, DIL], (), 1e-6),
    "viscoplastic_all": (VISCO, [CONST, SOFT, ZERO, DIL], (), 1e-6),
    "drucker_prager_beside_mohr_coulomb": (VISCO, [CONST, CONST], (1,), 1e-6),
    "drucker_prager_beside_softening": (VISCO, [SOFT, CONST, CONST], (2,), 1e-6),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_phases_of_one_warp_take_their_own_branches(case):
    base, angles, dp, tol = CASES[case]
    cfg = mixed(base, angles, dp)
    with SnacContext(cfg) as g:
        c = Checker(cfg, "port")
        g.time_step_zero()
        c.time_step_zero()
        g.step(40)
        c.step(40)
        sg, sc = g.state(), c.state()
    eps = sc.plastic_strain.reshape(-1, 10)
    for p in range(len(angles)):  # every phase yields somewhere
        assert np.count_nonzero(eps[cfg.element_material == p]) > 0, p
    for f in FIELDS:
        x, y = getattr(sg, f), getattr(sc, f)
        assert np.all(np.isfinite(y)), f
        assert np.max(np.abs(x - y)) <= tol * np.max(np.abs(y)), f


@pytest.mark.parametrize("split", [0, 1])
def test_batched_models_of_mixed_phases(split):
    cfgs = [mixed(*CASES[c][:2]) for c in ("plastic_all", "viscoplastic_all", "plastic_constant_zero")]
    with SnacBatch(cfgs) as b:
        b.tuning = {"split_classes": split}
        b.time_step_zero()
        b.step(20)
        for cfg, m in zip(cfgs, b.models):
            with SnacContext(cfg) as g:
                g.time_step_zero()
                g.step(20)
                for f in FIELDS:
                    assert np.array_equal(getattr(g.state(), f), getattr(m.state(), f)), f


def test_softening_segment_without_width():
    """A lookup in a segment of width 0 interpolates with 0 / 0: the angles become
    NaN, also where they are the same at both ends, and the tension cutoff is
    the one carried over (0 in an element's first tets), as in the oracle."""
    cfg = VISCO(5, 3, 5)
    cfg.materials = [phase(cfg, 30.0, 30.0)]
    cfg.materials[0].update(nsegments=1, plstrain1=0.0, cohesion1=cfg.materials[0]["cohesion0"])
    with SnacContext(cfg) as g:
        c = Checker(cfg, "port")
        g.time_step_zero()
        c.time_step_zero()
        g.step(20)
        c.step(20)
        sg, sc = g.state(), c.state()
    assert np.count_nonzero(sc.plastic_strain) > 0
    for f in FIELDS:
        x, y = getattr(sg, f), getattr(sc, f)
        assert np.all(np.isfinite(y)), f
        assert np.max(np.abs(x - y)) <= 1e-6 * np.max(np.abs(y)), f
