"""GPU: duals after an iteration in which some row and column sums are not finite.

A cost of -inf makes one entry of the plan infinite (group lasso: NaN): the sums of
its row, of its column and of the plan are, and those duals with them; the other rows and columns
keep finite sums, and their duals the bar of the parity tests (1e-5 relative)
against the streaming kernel.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _state(lib, kind, c, p, q, iters):
    from reg_drot._lib import DrotResult
    nc, nr = c.shape
    dev = c.device
    s = float(np.float32(2.0) / np.float32(nr + nc))
    st = {"x": torch.empty(nc, nr, device=dev), "a": torch.empty(nr, device=dev),
          "b": torch.empty(nc, device=dev), "phi1": torch.empty(nr, device=dev),
          "phi2": torch.empty(nc, device=dev), "alpha": torch.empty(1, device=dev)}
    ptrs = [t.data_ptr() for t in st.values()]
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.drot_init_state(nr, nc, s, 1, p.data_ptr(), q.data_ptr(), *ptrs, stream) == 0
    nbytes = (lib.drot_qr_workspace_bytes(nr, nc) if kind == "qr" else
              lib.drot_gl_workspace_bytes(nr, nc, 1))
    ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    head = (c.data_ptr(), p.data_ptr(), q.data_ptr(), nr, nc)
    tail = (iters, -1.0, *ptrs, ws.data_ptr(), nbytes, ctypes.byref(DrotResult()), stream)
    rc = (lib.drot_qr_solve(*head, s, 1.02, *tail) if kind == "qr" else
          lib.drot_gl_solve(*head, 1, s, 1e-6, *tail))
    assert rc == 0
    return st


# one CTA; rows and columns over several; a mass that also needs a coarser scale
CASES = [("qr", 96, 80, 0.0), ("qr", 700, 500, 0.0), ("qr", 700, 500, 400.0),
         ("gl", 700, 500, 0.0)]


@pytest.mark.parametrize("kind,nr,nc,shift", CASES, ids=[f"{k}{m}x{n}-{s:.0f}" for k, m, n, s in CASES])
def test_finite_sums_beside_infinite_ones(cuda, solver_lib, kind, nr, nc, shift):
    from reg_drot import autotune
    g = torch.Generator().manual_seed(nr)
    c = (torch.rand(nc, nr, generator=g) - shift).to(cuda)
    c[nc // 3, nr // 2] = float("-inf")
    rng = np.random.default_rng(nr)
    p, q = (torch.from_numpy(rng.dirichlet(np.ones(k)).astype(np.float32)).to(cuda)
            for k in (nr, nc))
    autotune.pin(kind, 0, 0, vectors_per_lane=4)  # the streaming kernel
    try:
        ref = _state(solver_lib, kind, c, p, q, 1)
    finally:
        autotune.clear()
    st = _state(solver_lib, kind, c, p, q, 1)
    for k in ("a", "b"):
        u, v = st[k].double(), ref[k].double()
        assert torch.equal(torch.isfinite(u), torch.isfinite(v)), k
        assert int((~torch.isfinite(v)).sum()) == 1, k  # the case is the one described
        ok = torch.isfinite(v)
        assert float((u - v)[ok].norm()) <= 1e-5 * float(v[ok].norm()), k
