"""The general geometry of coordinates outside [2^-100, 2^100), in every hook and
every form of the step.

The nodes of the plane z = 0 are put to z = 1e-33, where a roller holds them.
Against coordinates of kilometres that changes no difference of two of them, so
every result has the bits of the run with exact zeros, which takes the short
forms of the geometry."""
import numpy as np
import pytest

from snac_b200 import workloads as W
from snac_b200.abi import State
from snac_b200.adjoint import adjoint, top_surface
from snac_b200.batch import SnacBatch
from snac_b200.context import SnacContext
from tests import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("velocity", "stress", "plastic_strain", "viscosity", "temperature", "force", "inertial_mass",
          "plastic_strain_tensor")


def small(make):
    return lambda: make(7, 3, 5)


MODELS = {
    "elastic": small(S.elastic_small),
    "constant": lambda: S.constant_dt(S.elastic_small(7, 3, 5), 2.0e7),
    "plastic": small(S.plastic_small),
    "phases": small(S.plastic_two_phase),
    "viscoplastic": small(S.viscoplastic_small),
    "drucker_prager": small(S.drucker_prager_small),
    "maxwell": small(S.maxwell_small),
    "thermal_stress": small(S.two_phase_density),
    "adjoint": lambda: W.c5_adjoint(7, 3, 5, cohesion=(2.0e5, 2.0e4)),  # does not yield
    "adjoint_yielding": lambda: W.c5_adjoint(5, 3, 4, dt=1.0e8, v=10.0 * W.CM_PER_YR, extent=(15.0e3, 6.0e3, 12.0e3),
                                             cohesion=(5.0e6, 1.0e6), t_uniform=300.0),
}


def grid(cfg, z0):
    """cfg on a regular grid of its own coordinates, the plane z = 0 at z0"""
    n = (cfg.nx, cfg.ny, cfg.nz)
    a = [lo + (hi - lo) * np.arange(m + 1) / m for lo, hi, m in zip(cfg.min, cfg.max, n)]
    k, j, i = np.meshgrid(*(np.arange(m + 1) for m in reversed(n)), indexing="ij")
    x = np.stack([a[0][i], a[1][j], a[2][k]], -1).reshape(-1, 3)
    assert np.all(x[(k == 0).reshape(-1), 2] == 0.0)
    x[(k == 0).reshape(-1), 2] = z0
    cfg.node_coords = x.reshape(-1)
    return cfg


def both(kind):
    return grid(MODELS[kind](), 0.0), grid(MODELS[kind](), 1.0e-33)


def same(a, b, what=""):
    for f in FIELDS:
        x, y = getattr(a, f), getattr(b, f)
        assert np.all(np.isfinite(x)), (what, f)
        assert np.array_equal(x, y), (what, f)
    moved = a.coord[:, 2] != 0.0
    assert np.array_equal(a.coord[moved], b.coord[moved]) and np.array_equal(a.coord[:, :2], b.coord[:, :2])
    assert np.all(b.coord[~moved, 2] == 1.0e-33)  # still outside the range


def run(cfg, how):
    with SnacContext(cfg) as g:
        g.time_step_zero()
        if how == "steps":
            g.step(30)
        elif how == "hooks":
            for _ in range(12):
                g.solve()
        else:  # the state in host memory, in slabs
            g.step(10)
            s, out = g.state(), State.empty(cfg.n_elements, cfg.n_nodes)
            for _ in range(3):
                g.step_host(s, out, chunks=4)
                s, out = out, s
        return g.state(), g.scalars()


@pytest.mark.parametrize("how", ["steps", "hooks", "host"])
@pytest.mark.parametrize("kind", sorted(k for k in MODELS if not k.startswith("adjoint")))
def test_untame_coordinates_in_every_hook(kind, how):
    (a, sa), (b, sb) = (run(cfg, how) for cfg in both(kind))
    same(a, b)
    assert (sa.dt, sa.min_length_scale, sa.vmax) == (sb.dt, sb.min_length_scale, sb.vmax)


@pytest.mark.parametrize("split", [0, 1])
def test_untame_coordinates_in_a_batch(split):
    kinds = ["elastic", "plastic", "phases", "viscoplastic", "maxwell", "thermal_stress"]
    out = []
    for cfgs in zip(*(both(k) for k in kinds)):
        with SnacBatch(list(cfgs)) as b:
            b.tuning = {"split_classes": split}
            b.time_step_zero()
            b.step(12)
            out.append([m.state() for m in b.models])
    for k, x, y in zip(kinds, *out):
        same(x, y, k)


@pytest.mark.parametrize("kind,steps", [("adjoint", 12), ("adjoint_yielding", 24)])
def test_untame_coordinates_in_the_adjoint(kind, steps):
    out = []
    for cfg in both(kind):
        with SnacContext(cfg) as g:
            g.time_step_zero()
            v, y = top_surface(cfg, g.state())
            r = adjoint(g, steps, 0.9 * v, y + 1.0, w_v=1.0e22, w_h=1.0, state=True)
            out.append((r, g.state()))
    (a, sa), (b, sb) = out
    same(sa, sb)
    assert a.loss == b.loss
    assert (np.count_nonzero(sa.plastic_strain) > 0) == (kind == "adjoint_yielding")
    for k in a.grad:
        if kind == "adjoint_yielding":
            assert np.any(a.grad[k] != 0.0), k
        assert np.array_equal(a.grad[k], b.grad[k]), k
