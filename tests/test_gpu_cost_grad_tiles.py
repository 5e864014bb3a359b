"""GPU: the cost's chain rule (drot_sqeuclidean_cost_grad) at the edges of its
tiles -- 256-row bands, 32-column tiles, chunks of tiles, unaligned leading
dimensions -- against FP64 autograd.  Bar 1e-5 relative, the one of the other
chain-rule tests (FP32 sums of at most a few thousand terms)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("d", [8, 16, 24, 32])
@pytest.mark.parametrize("m,n", [(1, 1), (3, 33), (255, 31), (256, 32), (257, 65), (514, 4099),
                                 (2050, 161)])
@pytest.mark.parametrize("clamp", [True, False])
def test_chain_rule_tile_edges(cuda, m, n, d, clamp):
    from reg_drot.cost import sqeuclidean_cost
    g = torch.Generator(device=cuda).manual_seed(m + n + d)
    x = torch.randn(m, d, generator=g, device=cuda, requires_grad=True)
    y = torch.randn(n, d, generator=g, device=cuda, requires_grad=True)
    up = torch.randn(n, m, generator=g, device=cuda)
    gx, gy = torch.autograd.grad(sqeuclidean_cost(x, y, 0.25, clamp), (x, y), up)
    xd, yd = (t.detach().double().requires_grad_(True) for t in (x, y))
    c = 0.25 * ((yd * yd).sum(1, keepdim=True) + (xd * xd).sum(1)[None, :] - 2.0 * (yd @ xd.T))
    rx, ry = torch.autograd.grad(c, (xd, yd), up.double())
    assert float((gx - rx).norm()) <= 1e-5 * float(rx.norm())
    assert float((gy - ry).norm()) <= 1e-5 * float(ry.norm())
