"""GPU: host threads that solve problems of different shapes at the same time, each
on its own stream, do not make each other's launches fail.

Kernels are shared by all shapes, and so is a kernel's shared-memory limit: set to
the size of each launch, 350 of 48,000 such launches were refused.
"""
import threading

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(64 + 40 * k, 60 + 30 * k) for k in range(8)]


@pytest.mark.parametrize("kind", ["qr", "gl"])
def test_threads_with_different_shapes(cuda, solver_lib, kind):
    import reg_drot
    from reg_drot._lib import lib
    failed = []

    def work(k):
        nr, nc = SHAPES[k]
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            c = torch.rand(nc, nr, device=cuda)
            p = torch.full((nr,), 1.0 / nr, device=cuda)
            q = torch.full((nc,), 1.0 / nc, device=cuda)
            if kind == "qr":
                x, _, ws = reg_drot.solve_qr(c, p, q, 2.0, 1e-2, 2, 1e-9)
            else:
                x, _, ws = reg_drot.solve_gl(c, p, q, 2, 2.0, 1e-6, 2, 1e-9)
            want = x.clone()
            pad = (-ws.data_ptr()) % 256
            head = (c.data_ptr(), 0, p.data_ptr(), q.data_ptr(), nr, nc)
            tail = (2.0, 1e-2 if kind == "qr" else 1e-6, 2, 1e-9, x.data_ptr(),
                    ws.data_ptr() + pad, ws.numel() - pad, None, st.cuda_stream)
            fn = (lib().drot_quadratic_drot_ex if kind == "qr" else
                  lib().drot_group_lasso_drot_ex)
            args = head + tail if kind == "qr" else head + (2,) + tail
            for i in range(3000):
                rc = fn(*args)
                if rc:
                    failed.append((k, i, rc))
                if i % 200 == 199:
                    st.synchronize()
            if not torch.equal(x, want):
                failed.append((k, "plan"))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(SHAPES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, (len(failed), failed[:3])
