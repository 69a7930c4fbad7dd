"""Handles stepped by several host threads at once.  Their node gathers take
different amounts of shared memory (four stages of a small mesh, two of a
middle one); each handle's result is the one it has alone, bit for bit."""
import threading

import numpy as np
import pytest

from snac_b200.context import SnacContext
from tests import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("coord", "velocity", "stress", "plastic_strain", "force", "inertial_mass")
SHAPES = ((9, 9, 9), (27, 25, 27)) * 3
STEPS, NODE_LOOPS = 50, 2000


def run(g):
    g.time_step_zero()
    g.step(STEPS)
    for _ in range(NODE_LOOPS):  # a launch of the node gather each, on its own
        g.loop_nodes_momentum()
    return g.state()


def test_handles_of_two_sizes_on_six_threads():
    alone = {}
    for shape in set(SHAPES):
        with SnacContext(S.elastic_small(*shape)) as g:
            alone[shape] = run(g)
    handles = [SnacContext(S.elastic_small(*shape)) for shape in SHAPES]
    got, gate = [None] * len(SHAPES), threading.Barrier(len(SHAPES))

    def work(i):
        gate.wait()
        try:
            got[i] = run(handles[i])
        except Exception as e:  # raised by the thread that waits
            got[i] = e

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(SHAPES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in handles:
        g.close()
    for shape, b in zip(SHAPES, got):
        if isinstance(b, Exception):
            raise b
        for f in FIELDS:
            assert np.all(np.isfinite(getattr(b, f))), f
            assert np.array_equal(getattr(alone[shape], f), getattr(b, f)), f
