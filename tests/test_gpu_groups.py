"""The element blocks (groups of 12 hexes, triples per warp) and the node
gather (blocks of 64 nodes, groups fetched pair by pair) at the sizes where
their edges fall, the geometry of coordinates outside the tame range, long runs
of steps and downloads into rows that the device maps, bit
for bit against the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle.pyoracle import Checker
from snac_b200.context import SnacContext
from tests import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("coord", "velocity", "stress", "plastic_strain", "force", "inertial_mass")
MAKE = {"elastic": S.elastic_small, "plastic": S.plastic_small, "phases": S.plastic_two_phase,
        "constant": lambda *s: S.constant_dt(S.elastic_small(*s), 2.0e7)}


def check(cfg, steps=12):
    with SnacContext(cfg) as g:
        c = Checker(cfg, "port")
        g.time_step_zero()
        c.time_step_zero()
        g.step(steps)
        c.step(steps)
        sg, sc = g.state(), c.state()
        for f in FIELDS:
            assert np.all(np.isfinite(getattr(sc, f))), f
            assert np.array_equal(getattr(sg, f), getattr(sc, f)), f
        a, b = g.scalars(), c.scalars()
        assert (a.dt, a.min_length_scale, a.vmax) == (b.dt, b.min_length_scale, b.vmax)


# one hex; one triple; a group and its neighbours; 64 and 65 nodes; one hex wide
# in each direction; blocks of nodes that end inside a row, a plane, a group
@pytest.mark.parametrize("kind", sorted(MAKE))
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 1), (11, 1, 1), (12, 1, 1), (13, 1, 1), (15, 1, 1), (1, 1, 15),
                                   (1, 12, 2), (7, 3, 5), (13, 5, 11), (31, 1, 2)])
def test_edges_of_groups_and_node_blocks(shape, kind):
    check(MAKE[kind](*shape))


# lengths around 1e45 and 1e-35 m: outside [2^-100, 2^100), every triple takes the
# general geometry; 1e-33 m on one node: that node's triples do, the others not
@pytest.mark.parametrize("scale", [1.0e40, 1.0e-40])
def test_untame_coordinates(scale):
    cfg = S.elastic_small(5, 3, 4)
    cfg.min = tuple(scale * x for x in cfg.min)
    cfg.max = tuple(scale * x for x in cfg.max)
    check(cfg)


def test_one_untame_node():
    cfg = S.elastic_small(7, 3, 5)
    k, j, i = np.meshgrid(np.arange(6), np.arange(4), np.arange(8), indexing="ij")
    x = np.stack([i * 12.0e3, j * 8.0e3 - 24.0e3, k * 15.0e3], -1).reshape(-1, 3)
    x[3 + 2 * 8 + 0 * 32, 2] = 1.0e-33
    cfg.node_coords = x.reshape(-1)
    check(cfg)


# long calls run as graphs of 16 steps once 48 single ones have run, from either
# buffer of coordinates: the remainders, and a call that begins at an odd step
@pytest.mark.parametrize("calls", [(100,), (1, 64), (47, 1, 33), (65, 16, 17, 48)])
def test_runs_of_steps(calls):
    cfg = S.plastic_small(5, 4, 3)
    with SnacContext(cfg) as a, SnacContext(cfg) as b:
        a.time_step_zero()
        b.time_step_zero()
        for n in calls:
            a.step(n)
        for _ in range(sum(calls)):
            b.step(1)
        sa, sb = a.state(), b.state()
        for f in FIELDS:
            assert np.array_equal(getattr(sa, f), getattr(sb, f)), f
        assert (a.scalars().dt, a.scalars().time_step) == (b.scalars().dt, b.scalars().time_step)


# page-locked rows at every alignment that a host can give them (16, 8, 4 bytes
# past a boundary of 16), odd and even counts: written whole, nothing beside them
@pytest.mark.parametrize("offset", [0, 8, 4])
@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 4, 3), (8, 5, 7)])
def test_download_into_mapped_rows(shape, offset):
    with SnacContext(S.plastic_small(*shape)) as g:
        g.time_step_zero()
        g.step(5)
        want = g.state()
        got, keep = g.state(), []
        for f in FIELDS:
            w = getattr(want, f)
            t = torch.full((w.nbytes + 48,), 0x5A, dtype=torch.uint8).pin_memory()
            assert t.data_ptr() % 16 == 0
            raw = t.numpy()
            keep.append(raw)
            setattr(got, f, np.frombuffer(raw.data, np.float64, w.size, 16 + offset).reshape(w.shape))
        g.state(got)
        for f, raw in zip(FIELDS, keep):
            w = getattr(want, f)
            assert raw[16 + offset:16 + offset + w.nbytes].tobytes() == w.tobytes(), f
            assert np.all(raw[:16 + offset] == 0x5A) and np.all(raw[16 + offset + w.nbytes:] == 0x5A), f
