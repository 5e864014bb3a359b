"""GPU: the mask matvec of the implicit QR adjoint (adj_pcg_kernel) at the edges
of its tiles: the adjoint system's residual, taken in FP64 on the host.

CG stops at a relative residual of 1e-10 of its own recurrence, which rounding
(2^-53 per step, at most a few thousand steps) keeps within 1e-12 or so of the
true one; the bar on the true one is 1e-9.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _solve(shapes, density, scale, seed, cuda):
    from reg_drot.autograd import _Adjoint
    rng = np.random.default_rng(seed)
    descs, cs, gs = [], [], []
    co = vo = ro = qo = 0
    for nr, nc in shapes:
        c = rng.random((nc, nr), dtype=np.float32)
        g = rng.standard_normal((nc, nr)).astype(np.float32)
        g *= (10.0 ** rng.uniform(-scale, scale, (nc, 1))).astype(np.float32)
        descs.append((nr, nc, nr, co, vo, ro, qo, 1.0, 0.5))
        cs.append(c)
        gs.append(g)
        co, vo, ro, qo = co + nr * nc, vo + nr + nc, ro + nr, qo + nc
    # D = phi1 + phi2 - C > 0 on a share `density` of the entries
    phi1 = torch.full((ro,), 0.5 * density, device=cuda)
    phi2 = torch.full((qo,), 0.5 * density, device=cuda)
    cat = [torch.from_numpy(np.concatenate([a.ravel() for a in t])).to(cuda) for t in (cs, gs)]
    adj = _Adjoint(cat[0], phi1, phi2, descs)
    z, iters, rel = adj.solve(cat[1], 1e-10, 5000)
    z = z.cpu().numpy()
    for (nr, nc, _, _, v, *_), c, g, it, r in zip(descs, cs, gs, iters, rel):
        m = (np.float32(density) - c > 0).astype(np.float64)  # [nc, nr]
        a, b = z[v:v + nr], z[v + nr:v + nr + nc]
        gm = g * m
        rhs = np.concatenate([gm.sum(0), gm.sum(1)])
        lhs = np.concatenate([m.sum(0) * a + b @ m, m.sum(1) * b + m @ a])
        assert np.linalg.norm(lhs - rhs) <= 1e-9 * np.linalg.norm(rhs), (nr, nc, it, r)
        assert it < 5000


# one element; one group of lines and part of one; a word and a half; more
# entries than are staged at a time; more lines of a segment than a block holds
SHAPES = [(1, 1), (16, 16), (17, 33), (31, 500), (48, 96), (129, 4097), (5003, 61), (700, 650)]


@pytest.mark.parametrize("density", [0.03, 0.5, 1.0])
def test_masks_at_tile_edges(cuda, density):
    _solve(SHAPES, density, 0, 1, cuda)


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_one_instance(cuda, shape):
    _solve([shape], 0.4, 0, 2, cuda)


def test_more_sides_than_ctas(cuda):
    """Segments of several instances, and of both sides of one, in a CTA."""
    rng = np.random.default_rng(3)
    _solve([tuple(rng.integers(20, 260, 2)) for _ in range(170)], 0.3, 0, 3, cuda)


def test_long_segments(cuda):
    """Segments of more lines than a block of sums holds."""
    _solve([(4200, 4300)] * 20 + [(130, 90)] * 70, 0.1, 0, 4, cuda)


def test_entries_of_very_different_sizes(cuda):
    """Columns scaled by 1e-6 .. 1e6: entries far below the fixed-point scale's
    top digit."""
    _solve([(300, 411), (64, 777)], 0.4, 6, 5, cuda)
