"""GPU: a program that takes many shapes in turn finds the plans it made before.

Host time of the workspace query, which plans: 60 shapes take 64-entry caches
round and round without one hit, and then a later pass costs what the first did.
The bar on a later pass is half of the first; from the cache it is a twentieth.
"""
import time

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind", ["qr", "gl"])
def test_many_shapes_in_turn_are_planned_once(cuda, solver_lib, kind):
    import reg_drot
    shapes = [(401 + 3 * k, 350 + 2 * k) for k in range(60)]
    reg_drot.workspace_bytes(kind, 64, 64, 2, cuda)  # the context

    def once():
        t0 = time.perf_counter()
        sizes = [reg_drot.workspace_bytes(kind, m, n, 2, cuda) for m, n in shapes]
        return time.perf_counter() - t0, sizes
    first, sizes = once()
    later = [once() for _ in range(5)]
    assert all(s == sizes for _, s in later)
    assert min(t for t, _ in later) <= 0.5 * first, (first, [t for t, _ in later])
