"""GPU: the single-problem kernel whose tiles stay on chip (drot_resident.cuh)
at the edges of its tilings, against the FP32 oracle and the streaming kernel.

Fixed iteration counts, so both sides run the same iterations; the bar on X
is the one of the parity tests (1e-5 relative Frobenius: the two differ in
the order of FP32 row and column sums only).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402


def _problem(nr, nc, seed):
    g = torch.Generator().manual_seed(seed)
    c = torch.rand(nc, nr, generator=g) + 1e-3
    rng = np.random.default_rng(seed)
    p = torch.from_numpy(rng.dirichlet(np.ones(nr)).astype(np.float32))
    q = torch.from_numpy(rng.dirichlet(np.ones(nc)).astype(np.float32))
    return c / c.max(), p, q


def _close(x, y):
    x, y = np.asarray(x, np.float64), np.asarray(y, np.float64)
    return np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)


def _streaming(fn, kind, dtype=torch.float32):
    """fn() with the streaming kernel pinned for every shape."""
    from reg_drot import autotune
    autotune.pin(kind, 0, 0, c_dtype=dtype, vectors_per_lane=4)
    try:
        return fn()
    finally:
        autotune.clear()


# one element; one CTA with a padding column per warp; the last one-CTA size
# and the first beyond it; rows on both sides of a warp's 128 and of a band;
# columns that leave warps and CTAs empty; the largest tiles (one copy of X)
QR_SHAPES = [(1, 1), (5, 3), (96, 80), (100, 92), (128, 65), (129, 64), (255, 257), (1, 500),
             (500, 1), (1023, 130), (1501, 1499), (1705, 1700)]


@pytest.mark.parametrize("nr,nc", QR_SHAPES, ids=[f"{a}x{b}" for a, b in QR_SHAPES])
def test_qr_tilings_match_oracle(cuda, nr, nc):
    import reg_drot
    c, p, q = _problem(nr, nc, nr + nc)
    for iters in (31, 40):
        x, info, _ = reg_drot.solve_qr(c.to(cuda), p.to(cuda), q.to(cuda), 2.0, 1e-2, iters, 0.0)
        o = O.quadratic_drot(c.numpy(), p.numpy(), q.numpy(), 2.0, 1e-2, iters, 0.0)
        assert info["status"] == 0 and info["n_iter"] == iters + 1
        assert _close(x.cpu(), o["x"])
        assert abs(info["objective"] - o["objective"]) <= 1e-5 * abs(o["objective"])


# classes of one row, a class per warp, classes off the vector boundary, a
# class of several warps with idle warps, the tallest ones
GL_SHAPES = [(2, 4, 2), (64, 90, 64), (128, 300, 1), (301, 203, 3), (1502, 131, 2),
             (1700, 77, 1)]


@pytest.mark.parametrize("nr,nc,G", GL_SHAPES, ids=[f"{a}x{b}g{g}" for a, b, g in GL_SHAPES])
def test_gl_tilings_match_oracle(cuda, nr, nc, G):
    import reg_drot
    c, p, q = _problem(nr, nc, nr + nc + G)
    rw = 1e-3 / (nr // G)
    x, info, _ = reg_drot.solve_gl(c.to(cuda), p.to(cuda), q.to(cuda), G, 2.0, rw, 40, 0.0)
    o = O.group_lasso_drot(c.numpy(), p.numpy(), q.numpy(), G, 2.0, rw, 40, 0.0)
    assert info["status"] == 0 and info["n_iter"] == 40
    assert _close(x.cpu(), o["x"])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_unaligned_pointers_and_bf16_match_streaming(cuda, dtype):
    """Columns and base pointers off the vector boundary."""
    import reg_drot
    nr, nc = 516, 211
    c, p, q = _problem(nr, nc, 7)
    buf = torch.empty(nr * nc + 1, dtype=dtype, device=cuda)
    cd = buf[1:].view(nc, nr)
    cd.copy_(c)

    def run():
        return reg_drot.solve_qr(cd, p.to(cuda), q.to(cuda), 2.0, 1e-3, 60, 0.0)[0]
    assert _close(run().cpu(), _streaming(run, "qr", dtype).cpu())


def test_mass_beyond_the_exchange_words_range(cuda):
    """A cost of -50 gives a plan of mass 1e4 at first: the rounds that the
    fixed-point words cannot hold are repeated on a coarser scale."""
    import reg_drot
    nr, nc = 600, 500
    c, p, q = _problem(nr, nc, 3)
    c = c - 50.0
    for iters in (1, 2, 9):
        x, info, _ = reg_drot.solve_qr(c.to(cuda), p.to(cuda), q.to(cuda), 2.0, 1e-2, iters, 0.0)
        o = O.quadratic_drot(c.numpy(), p.numpy(), q.numpy(), 2.0, 1e-2, iters, 0.0)
        assert info["status"] == 0
        assert _close(x.cpu(), o["x"])


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_costs_that_are_not_finite_match_streaming(cuda, value):
    """Forbidden pairs (+inf) and invalid costs give the streaming kernel's
    plan entry for entry where that is not finite, and within the bar else."""
    import reg_drot
    nr, nc = 300, 200
    c, p, q = _problem(nr, nc, 9)
    c[5, 7] = c[100, 250] = value

    def run():
        return reg_drot.solve_qr(c.to(cuda), p.to(cuda), q.to(cuda), 2.0, 1e-2, 20, 0.0)[0].cpu()
    x, y = run(), _streaming(run, "qr")
    assert torch.equal(torch.isnan(x), torch.isnan(y))
    assert torch.equal(torch.isinf(x), torch.isinf(y))
    ok = torch.isfinite(y)
    assert float((x[ok].double() - y[ok].double()).norm()) <= 1e-5 * float(y[ok].double().norm())


def test_segments_equal_one_launch(cuda, solver_lib):
    """drot_qr_solve from a returned state: 7 + 12 iterations in two calls and
    19 in one give the same bits."""
    import ctypes
    from reg_drot._lib import DrotResult
    nr, nc = 700, 333
    c, p, q = (t.to(cuda) for t in _problem(nr, nc, 11))
    s = float(np.float32(2.0) / np.float32(nr + nc))
    out = []
    for parts in ((19,), (8, 11)):
        st = {"x": torch.empty(nc, nr, device=cuda), "a": torch.empty(nr, device=cuda),
              "b": torch.empty(nc, device=cuda), "phi1": torch.empty(nr, device=cuda),
              "phi2": torch.empty(nc, device=cuda), "alpha": torch.empty(1, device=cuda)}
        stream = torch.cuda.current_stream().cuda_stream
        assert solver_lib.drot_init_state(nr, nc, s, 1, p.data_ptr(), q.data_ptr(),
                                          *[t.data_ptr() for t in st.values()], stream) == 0
        nbytes = solver_lib.drot_qr_workspace_bytes(nr, nc)
        ws = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
        for n in parts:
            res = DrotResult()
            assert solver_lib.drot_qr_solve(
                c.data_ptr(), p.data_ptr(), q.data_ptr(), nr, nc, s, 1.02, n, -1.0,
                *[t.data_ptr() for t in st.values()], ws.data_ptr(), nbytes, ctypes.byref(res),
                stream) == 0
        out.append(st)
    for k in out[0]:
        assert torch.equal(out[0][k], out[1][k]), k


def test_streamed_gl_iterations_recomputed_singly_give_the_same_bits(cuda, solver_lib):
    """Beyond the chip the streaming kernel alternates the order of its
    columns; a segment recomputed one iteration at a time
    (drot_gl_adjoint_segment) ends in the state of one launch over it."""
    import ctypes
    from reg_drot._lib import DrotResult
    nr, nc, G, n = 2600, 2100, 2, 5
    c, p, q = (t.to(cuda) for t in _problem(nr, nc, 12))
    s = float(np.float32(2.0) / np.float32(nr + nc))
    stream = torch.cuda.current_stream().cuda_stream
    nbytes = solver_lib.drot_gl_workspace_bytes(nr, nc, G)
    ws = torch.empty(nbytes + 256, dtype=torch.uint8, device=cuda)
    wptr = ws.data_ptr() + (-ws.data_ptr()) % 256
    out = []
    for single in (False, True):
        st = {"x": torch.empty(nc, nr, device=cuda), "a": torch.empty(nr, device=cuda),
              "b": torch.empty(nc, device=cuda), "phi1": torch.empty(nr, device=cuda),
              "phi2": torch.empty(nc, device=cuda), "alpha": torch.empty(1, device=cuda)}
        ptrs = [t.data_ptr() for t in st.values()]
        assert solver_lib.drot_init_state(nr, nc, s, 1, p.data_ptr(), q.data_ptr(), *ptrs,
                                          stream) == 0
        if single:
            ab = solver_lib.drot_gl_adjoint_workspace_bytes(nr, nc, G)
            aws = torch.empty(ab + 256, dtype=torch.uint8, device=cuda)
            bars = [torch.zeros(k, device=cuda) for k in
                    (nr * nc, 2 * (nr + nc) + 1, nr * nc, nr, nc)]
            states = torch.empty(n * (nr * nc + nr + nc), device=cuda)
            rc = solver_lib.drot_gl_adjoint_segment(
                c.data_ptr(), 0, p.data_ptr(), q.data_ptr(), nr, nc, G, s, 1e-6, *ptrs, n,
                states.data_ptr(), wptr, nbytes, *[t.data_ptr() for t in bars],
                aws.data_ptr() + (-aws.data_ptr()) % 256, ab, stream)
        else:
            res = DrotResult()
            rc = solver_lib.drot_gl_solve(c.data_ptr(), p.data_ptr(), q.data_ptr(), nr, nc, G, s,
                                          1e-6, n, -1.0, *ptrs, wptr, nbytes, ctypes.byref(res),
                                          stream)
        assert rc == 0
        torch.cuda.synchronize()
        out.append(st)
    for k in out[0]:
        assert torch.equal(out[0][k], out[1][k]), k


# part of X and C in global memory: C alone, both, columns off the vector
# boundary (aligned copies), a ragged last band and chunk, the widest warps
PARTIAL_SHAPES = [(2000, 2000, torch.float32), (2603, 2501, torch.float32),
                  (3004, 2998, torch.float32), (2600, 4100, torch.bfloat16),
                  (4301, 3907, torch.bfloat16), (7000, 900, torch.float32)]


@pytest.mark.parametrize("nr,nc,dtype", PARTIAL_SHAPES,
                         ids=[f"{a}x{b}{'b' if d == torch.bfloat16 else ''}"
                              for a, b, d in PARTIAL_SHAPES])
def test_qr_tilings_partly_in_global_memory_match_oracle(cuda, nr, nc, dtype):
    import reg_drot
    c, p, q = _problem(nr, nc, nr + nc)
    c = c.to(dtype)
    cr = c.float().numpy()
    for iters in (7, 12):
        x, info, _ = reg_drot.solve_qr(c.to(cuda), p.to(cuda), q.to(cuda), 2.0, 1e-2, iters, 0.0)
        o = O.quadratic_drot(cr, p.numpy(), q.numpy(), 2.0, 1e-2, iters, 0.0)
        assert info["status"] == 0 and info["n_iter"] == iters + 1
        assert _close(x.cpu(), o["x"])
        assert abs(info["objective"] - o["objective"]) <= 1e-5 * abs(o["objective"])
    # a stop: the returned plan is unfolded wherever its columns lie
    eps = 1.5 * info["residual"]
    x, info, _ = reg_drot.solve_qr(c.to(cuda), p.to(cuda), q.to(cuda), 2.0, 1e-2, 200, eps)
    o = O.quadratic_drot(cr, p.numpy(), q.numpy(), 2.0, 1e-2, 200, eps)
    assert info["converged"] == 1 and info["n_iter"] == o["n_iter"]
    assert _close(x.cpu(), o["x"])
