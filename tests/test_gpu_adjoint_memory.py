"""Device memory of the adjoint: what snac_gpu_device_bytes says of its
workspace, and how much stays allocated between calls."""
import ctypes as C

import pytest
import torch

from snac_b200 import workloads as W
from snac_b200.adjoint import adjoint, misfit, top_surface
from snac_b200.context import SnacContext, load_library

pytestmark = pytest.mark.gpu


def device_bytes(ctx) -> int:
    lib = load_library()
    lib.snac_gpu_device_bytes.argtypes = [C.c_void_p, C.POINTER(C.c_longlong)]
    lib.snac_gpu_device_bytes.restype = C.c_int
    b = C.c_longlong(-1)
    ctx._check(lib.snac_gpu_device_bytes(ctx.h, C.byref(b)))
    return b.value


def model():
    g = SnacContext(W.c5_adjoint(32, 16, 32))
    g.time_step_zero()
    return g, top_surface(g.cfg, g.state())


def test_device_bytes_never_decrease():
    """A workspace of some 700 MB (60 states kept) is larger than what stays
    allocated between calls; the count is of bytes allocated since creation."""
    g, target = model()
    with g:
        last = device_bytes(g)
        for call in (lambda: misfit(g, *target), lambda: adjoint(g, 12, *target),
                     lambda: adjoint(g, 60, *target, checkpoint_every=1), lambda: misfit(g, *target),
                     lambda: adjoint(g, 12, *target)):
            call()
            now = device_bytes(g)
            assert now >= last
            last = now


def test_handles_keep_a_bounded_workspace_together():
    """Each handle's workspace is some 420 MB (every second of 60 states kept); ten
    handles keep at most 2 GiB between their calls, and destroying them gives
    all of it back."""
    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    models = [model() for _ in range(10)]
    before = free()
    sizes = []
    for g, target in models:
        last = device_bytes(g)
        adjoint(g, 60, *target, checkpoint_every=2)
        sizes.append(device_bytes(g) - last)
    assert max(sizes) < (512 << 20) and sum(sizes) > (3 << 30)  # each could be kept, all of them not
    # beside the workspaces a call leaves a few hundred KB of staging and graphs
    slack = 16 << 20
    assert before - free() <= (2 << 30) + slack * len(models)
    first = models[0]
    a, b = adjoint(first[0], 6, *first[1]), adjoint(models[-1][0], 6, *models[-1][1])
    assert a.loss == b.loss  # one handle's workspace kept, the other's not
    for g, _ in models:
        g.close()
    assert free() >= before
