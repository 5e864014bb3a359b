"""GPU: the implicit QR adjoint where the support graph falls apart into components
whose right-hand sides differ by many powers of two.

The components are copies of one another and their upstream gradients equal but
for a power of two, so CG takes the same steps in each and leaves the same
relative residual: 1e-10 where it stops, 1e-9 with the rounding of the recurrence
(the bar of the mask tests).  Matvec sums held on the scale of the largest
component would lose the smaller ones.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nr,nc", [(37, 50), (160, 131)])
def test_every_component_is_solved_to_its_own_scale(cuda, nr, nc):
    from reg_drot.autograd import _Adjoint
    scales = [2.0 ** -k for k in (0, 20, 30, 55, 80)]
    B = len(scales)
    rng = np.random.default_rng(nr)
    cb = rng.random((nc, nr), dtype=np.float32)
    gb = rng.standard_normal((nc, nr)).astype(np.float32)
    c = np.full((B * nc, B * nr), 9.0, np.float32)
    g = rng.standard_normal(c.shape).astype(np.float32)  # off the support: not read
    for k, t in enumerate(scales):
        at = np.s_[k * nc:(k + 1) * nc, k * nr:(k + 1) * nr]
        c[at], g[at] = cb, gb * np.float32(t)
    # D = phi1 + phi2 - C > 0 on 0.3 of a block's entries, on none off the blocks
    phi1 = torch.full((B * nr,), 0.15, device=cuda)
    phi2 = torch.full((B * nc,), 0.15, device=cuda)
    adj = _Adjoint(torch.from_numpy(c).to(cuda).view(-1), phi1, phi2,
                   [(B * nr, B * nc, B * nr, 0, 0, 0, 0, 1.0, 0.5)])
    z, iters, _ = adj.solve(torch.from_numpy(g).to(cuda).view(-1), 1e-10, 5000)
    assert iters[0] < 5000
    z = z.cpu().numpy()
    m = (np.float32(0.15) + np.float32(0.15) - cb > 0).astype(np.float64)
    for k, t in enumerate(scales):
        a, b = z[k * nr:(k + 1) * nr], z[B * nr + k * nc:][:nc]
        gm = gb.astype(np.float64) * m * t
        rhs = np.concatenate([gm.sum(0), gm.sum(1)])
        lhs = np.concatenate([m.sum(0) * a + b @ m, m.sum(1) * b + m @ a])
        assert np.linalg.norm(lhs - rhs) <= 1e-9 * np.linalg.norm(rhs), (t, iters[0])


def test_components_without_a_gradient_stay_zero(cuda):
    from reg_drot.autograd import _Adjoint
    nr, nc, B = 90, 70, 3
    rng = np.random.default_rng(1)
    c = np.full((B * nc, B * nr), 9.0, np.float32)
    g = np.zeros_like(c)
    for k in range(B):
        c[k * nc:(k + 1) * nc, k * nr:(k + 1) * nr] = rng.random((nc, nr), dtype=np.float32)
    g[nc:2 * nc, nr:2 * nr] = rng.standard_normal((nc, nr))
    phi = torch.full((B * nr,), 0.15, device=cuda), torch.full((B * nc,), 0.15, device=cuda)
    adj = _Adjoint(torch.from_numpy(c).to(cuda).view(-1), *phi,
                   [(B * nr, B * nc, B * nr, 0, 0, 0, 0, 1.0, 0.5)])
    z, iters, rel = adj.solve(torch.from_numpy(g).to(cuda).view(-1), 1e-10, 5000)
    z = z.cpu().numpy()
    live = np.r_[nr:2 * nr, B * nr + nc:B * nr + 2 * nc]
    assert iters[0] < 5000 and np.abs(z[live]).max() > 0
    assert not np.delete(z, live).any()
