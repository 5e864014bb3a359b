"""GPU: batched GL instances whose last 16-byte vector of a column holds rows
of several classes and padding rows, which belong to the caller."""
import math

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nr,G", [(2, 2), (3, 3), (6, 3), (7, 7), (1025, 512)])
def test_padding_beside_two_classes_is_ignored(cuda, nr, G):
    from reg_drot.batch import GLBatch
    nc = 40
    g = torch.Generator(device=cuda).manual_seed(nr)
    b = GLBatch([(nr, nc)], G, 2.0, 1e-3, 0.0, device=cuda, cols_per_tile=16,
                tuning={"tail_quarters": 0})
    cost = torch.rand(nc, nr, generator=g, device=cuda)
    p, q = b.pack_marginals([torch.full((nr,), 1.0 / nr)], [torch.full((nc,), 1.0 / nc)])
    out = []
    for fill in (0.0, float("nan")):
        c = b.pack_c([cost])
        c[:b.lds[0] * nc].view(nc, b.lds[0])[:, nr:] = fill
        x, info = b.solve(c, p, q, 20)
        out.append((b.view(x, 0).clone(), info))
    assert math.isfinite(out[1][1][0]["objective"])
    assert torch.equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
