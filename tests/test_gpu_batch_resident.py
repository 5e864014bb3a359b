"""GPU: batches whose instances run on resident tiles (drot_resident_batch_kernel)
at the edges of their tilings, against the streaming batch kernel.

A tuning record that is not the default selects the streaming kernel, and
plans without the resident tiles' part of the workspace.  Fixed iteration
counts; the bar on X and the duals is the one of the parity tests (1e-5
relative Frobenius: the two differ in the order of FP32 row and column sums
only).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

STREAMING = {"tail_quarters": 0}


def _costs(shapes, device, seed):
    g = torch.Generator(device=device).manual_seed(seed)
    return [torch.rand(nc, nr, generator=g, device=device) + 1e-3 for nr, nc in shapes]


def _marginals(shapes, seed):
    rng = np.random.default_rng(seed)
    return ([torch.from_numpy(rng.dirichlet(np.ones(m)).astype(np.float32)) for m, _ in shapes],
            [torch.from_numpy(rng.dirichlet(np.ones(n)).astype(np.float32)) for _, n in shapes])


def _close(x, y):
    x, y = x.double(), y.double()
    return float((x - y).norm()) <= 1e-5 * float(y.norm())


def _bytes(batch):
    return batch.workspace_for(batch.cols_per_tile)[2]


def _compare(make, shapes, dtype, cuda, iters):
    res, ref = make(None), make(STREAMING)
    assert _bytes(res) > _bytes(ref), "the batch does not run on resident tiles"
    c = res.pack_c(_costs(shapes, cuda, 5), dtype=dtype)
    for k, (nr, nc) in enumerate(shapes):  # padding rows belong to the caller
        ld, off = res.lds[k], res.offsets[k]
        c[off:off + ld * nc].view(nc, ld)[:, nr:] = float("nan")
    p, q = res.pack_marginals(*_marginals(shapes, 6))
    for n in iters:
        out = []
        for b in (res, ref):
            x, info = b.solve(c, p, q, n)
            out.append((b.unpack(x), info, b.state(info)))
        (xs, infos, states), (ys, refs, rstates) = out
        for k, shape in enumerate(shapes):
            assert _close(xs[k], ys[k]), (n, shape)
            for name in ("n_iter", "iters_run", "converged", "objective_valid"):
                assert infos[k][name] == refs[k][name], (n, shape, name)
            assert abs(infos[k]["objective"] - refs[k]["objective"]) <= \
                1e-5 * abs(refs[k]["objective"]), (n, shape)
            for name in ("a", "b"):
                assert _close(states[k][name], rstates[k][name]), (n, shape, name)


# one element; a padding column per warp; both sides of a warp's 128 rows; the
# narrowest and the lowest; ragged bands and chunks; C, then X in global memory
QR_SHAPES = [(1, 1), (5, 3), (96, 80), (128, 65), (129, 64), (255, 257), (1, 500), (500, 1),
             (2047, 130), (1501, 1499), (703, 1402), (2600, 2201)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_qr_batch_tilings_match_streaming(cuda, dtype):
    from reg_drot.batch import QRBatch
    _compare(lambda t: QRBatch(QR_SHAPES, 2.0, 1e-2, 0.0, device=cuda, cols_per_tile=128, tuning=t),
             QR_SHAPES, dtype, cuda, (0, 1, 31, 40))


# classes of one row, a class per warp, classes off the vector boundary, idle
# warps, the tallest classes, C and X in global memory
GL_SHAPES = [(2, 4, 2), (64, 90, 64), (128, 300, 1), (301, 203, 3), (1502, 131, 2), (1024, 77, 1),
             (2040, 1600, 2), (1999, 1203, 10)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gl_batch_tilings_match_streaming(cuda, dtype):
    from reg_drot.batch import GLBatch
    shapes = [(m, n) for m, n, _ in GL_SHAPES]
    _compare(lambda t: GLBatch(shapes, [g for _, _, g in GL_SHAPES], 2.0, 1e-3, 0.0, device=cuda,
                               cols_per_tile=128, tuning=t),
             shapes, dtype, cuda, (0, 1, 31, 40))


def test_instances_that_wait_for_ctas(cuda):
    """More instances than run at once, each with its own stop: the same bits
    whichever CTAs run them, and every one at its stop."""
    from reg_drot.batch import QRBatch
    shapes = [(300 + 37 * (k % 11), 250 + 53 * (k % 7)) for k in range(120)]
    b = QRBatch(shapes, 2.0, 1e-2, 1e-3, device=cuda, cols_per_tile=128)
    assert _bytes(b) > _bytes(QRBatch(shapes, 2.0, 1e-2, 1e-3, device=cuda, cols_per_tile=128,
                                      tuning=STREAMING))
    c = b.pack_c(_costs(shapes, cuda, 8))
    p, q = b.pack_marginals(*_marginals(shapes, 9))
    x, info = b.solve(c, p, q, 20000)
    assert all(i["converged"] == 1 and i["residual"] < 1e-3 for i in info)
    assert len({i["n_iter"] for i in info}) > 1
    for _ in range(2):
        y, again = b.solve(c, p, q, 20000)
        assert again == info
        assert all(torch.equal(u, v) for u, v in zip(b.unpack(x), b.unpack(y)))
    rows = [i["residual"] for i in info]
    for k in range(0, len(shapes), 17):  # the residual is that of the plan handed back
        v = b.view(x, k).double()
        pk = p[sum(m for m, _ in shapes[:k]):][:shapes[k][0]].double()
        qk = q[sum(n for _, n in shapes[:k]):][:shapes[k][1]].double()
        r = float(((v.sum(0) - pk) ** 2).sum() + ((v.sum(1) - qk) ** 2).sum()) ** 0.5
        assert abs(r - rows[k]) <= 1e-2 * rows[k] + 1e-6


def test_an_exchange_that_never_completes_ends_every_wait(cuda, monkeypatch):
    """The first instance's first tile adds nothing: its CTAs, and those that
    wait for work, end within the limit; the next solve runs as ever."""
    import reg_drot
    from reg_drot.batch import QRBatch
    shapes = [(700, 500)] * 40
    b = QRBatch(shapes, 2.0, 1e-2, 0.0, device=cuda, cols_per_tile=128)
    c = b.pack_c(_costs(shapes, cuda, 3))
    p, q = b.pack_marginals(*_marginals(shapes, 4))
    x, _ = b.solve(c, p, q, 30)
    monkeypatch.setenv("DROT_BARRIER_TIMEOUT_MS", "200")
    monkeypatch.setenv("DROT_TEST_STALL_CTA", "0")
    with pytest.raises(reg_drot.DrotError) as err:
        b.solve(c, p, q, 30)
    assert err.value.status == 3 or "timeout" in str(err.value).lower()
    monkeypatch.delenv("DROT_TEST_STALL_CTA")
    monkeypatch.delenv("DROT_BARRIER_TIMEOUT_MS")
    y, _ = b.solve(c, p, q, 30)
    assert all(torch.equal(u, v) for u, v in zip(b.unpack(x), b.unpack(y)))
