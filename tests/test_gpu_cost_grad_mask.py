"""GPU: the cost's chain rule on a clamped cost, with zeros of C in it.

Entries where C = 0 pass no gradient.  C holds zeros at random places, on the last
rows and columns among them, independent of the points: reading C from any other
row, column or tile, on the vector path or the scalar one, changes the sums.  The
padding rows are NaN.  Against the FP64 sums of the masked gradient; bar 1e-5
relative, the one of the other chain-rule tests.
"""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("d", [8, 16, 24, 32])
@pytest.mark.parametrize("m,n,ld", [(1, 1, 1), (3, 33, 4), (255, 31, 255), (257, 65, 260),
                                    (514, 4099, 514), (2050, 161, 2052), (640, 300, 640)])
def test_zeros_of_the_cost_pass_no_gradient(cuda, m, n, ld, d):
    from reg_drot.cost import _chain_rule
    g = torch.Generator(device=cuda).manual_seed(m + n + d)
    x = torch.randn(m, d, generator=g, device=cuda)
    y = torch.randn(n, d, generator=g, device=cuda)
    up = torch.full((n, ld), float("nan"), device=cuda)
    c = torch.full((n, ld), float("nan"), device=cuda)
    up[:, :m] = torch.randn(n, m, generator=g, device=cuda)
    on = torch.rand(n, m, generator=g, device=cuda) < 0.5
    on[:, -1] ^= True
    on[-1] ^= True
    on[0, 0] = True
    c[:, :m] = torch.where(on, torch.rand(n, m, generator=g, device=cuda) + 0.5, 0.0)
    gx, gy = _chain_rule([(m, n, ld, 0, 0, 0)], x, y, 0.25, c, up, True)
    gm = torch.where(on, up[:, :m], 0.0).double()
    xd, yd = x.double(), y.double()
    rx = 0.5 * (xd * gm.sum(0)[:, None] - gm.T @ yd)
    ry = 0.5 * (yd * gm.sum(1)[:, None] - gm @ xd)
    assert float((gx - rx).norm()) <= 1e-5 * float(rx.norm())
    assert float((gy - ry).norm()) <= 1e-5 * float(ry.norm())
