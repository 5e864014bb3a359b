"""GPU: the state that a resident solve hands back when it stops on an iteration
whose successor, already run, did not fit the exchange words at first.

A cost of -400 to -360 gives a plan of mass 2e5 after one iteration and above 512
after two.  The residual of the first, about 1.3e4, stops the solve; the returned
state is that of the first iteration.  alpha is alpha0 + 1 - mass in FP32, and the
masses of the two kernels differ by an ulp of theirs at most, so the bar on it is
4 ulp; the duals' is the parity tests' 1e-5 relative.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NR, NC, EPS = 600, 500, 16000.0


def _problem(cuda):
    g = torch.Generator().manual_seed(3)
    c = torch.rand(NC, NR, generator=g) + 1e-3
    rng = np.random.default_rng(3)
    return [t.to(cuda) for t in (40.0 * c / c.max() - 400.0,
                                 torch.from_numpy(rng.dirichlet(np.ones(NR)).astype(np.float32)),
                                 torch.from_numpy(rng.dirichlet(np.ones(NC)).astype(np.float32)))]


def _solve(lib, kind, c, p, q, iters, eps):
    from reg_drot._lib import DrotResult
    dev = c.device
    s = float(np.float32(2.0) / np.float32(NR + NC))
    st = {"x": torch.empty(NC, NR, device=dev), "a": torch.empty(NR, device=dev),
          "b": torch.empty(NC, device=dev), "phi1": torch.empty(NR, device=dev),
          "phi2": torch.empty(NC, device=dev), "alpha": torch.empty(1, device=dev)}
    ptrs = [t.data_ptr() for t in st.values()]
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.drot_init_state(NR, NC, s, 1, p.data_ptr(), q.data_ptr(), *ptrs, stream) == 0
    nbytes = (lib.drot_qr_workspace_bytes(NR, NC) if kind == "qr" else
              lib.drot_gl_workspace_bytes(NR, NC, 2))
    ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    res = DrotResult()
    head = (c.data_ptr(), p.data_ptr(), q.data_ptr(), NR, NC)
    tail = (iters, eps, *ptrs, ws.data_ptr(), nbytes, ctypes.byref(res), stream)
    rc = (lib.drot_qr_solve(*head, s, 1.02, *tail) if kind == "qr" else
          lib.drot_gl_solve(*head, 2, s, 1e-6, *tail))
    assert rc == 0
    return st, res.as_dict()


def _same(st, ref):
    assert abs(float(st["alpha"]) - float(ref["alpha"])) <= 2.0 ** -21 * abs(float(ref["alpha"]))
    for k in ("x", "a", "b"):
        d = (st[k].double() - ref[k].double()).norm()
        assert float(d) <= 1e-5 * float(ref[k].double().norm()), k


@pytest.mark.parametrize("kind", ["qr", "gl"])
def test_state_of_a_stop_before_a_repeated_round(cuda, solver_lib, kind):
    from reg_drot import autotune
    c, p, q = _problem(cuda)
    autotune.pin(kind, 0, 0, vectors_per_lane=4)  # the streaming kernel
    try:
        two, _ = _solve(solver_lib, kind, c, p, q, 2, -1.0)
        ref, rinfo = _solve(solver_lib, kind, c, p, q, 40, EPS)
    finally:
        autotune.clear()
    assert float(two["x"].double().sum()) > 512.0  # the case is the one described
    st, info = _solve(solver_lib, kind, c, p, q, 40, EPS)
    assert rinfo["converged"] == 1 and rinfo["iters_run"] == 1
    for k in ("n_iter", "iters_run", "converged", "status"):
        assert info[k] == rinfo[k]
    _same(st, ref)


def test_batch_state_of_a_stop_before_a_repeated_round(cuda):
    from reg_drot.batch import QRBatch
    c, p, q = _problem(cuda)
    states = []
    for tuning in (None, {"tail_quarters": 0}):  # resident tiles, streaming
        b = QRBatch([(NR, NC)] * 3, 2.0, 1e-2, EPS, device=cuda, cols_per_tile=128, tuning=tuning)
        pc = b.pack_c([c] * 3)
        pp, pq = b.pack_marginals([p] * 3, [q] * 3)
        x, info = b.solve(pc, pp, pq, 40)
        assert all(i["converged"] == 1 and i["iters_run"] == 1 for i in info)
        states.append([dict(t, x=u) for t, u in zip(b.state(info), b.unpack(x))])
    for st, ref in zip(*states):
        _same(st, ref)
