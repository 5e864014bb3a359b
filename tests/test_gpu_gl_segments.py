"""GPU: a group-lasso solve split into launches at any count ends in the state of
one launch, bit for bit, on tiles and beyond the chip, where the streaming kernel
walks its columns one way and the other in turn."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _problem(nr, nc, seed, cuda):
    g = torch.Generator(device=cuda).manual_seed(seed)
    c = torch.rand(nc, nr, generator=g, device=cuda) + 1e-3
    rng = np.random.default_rng(seed)
    p = torch.from_numpy(rng.dirichlet(np.ones(nr)).astype(np.float32))
    q = torch.from_numpy(rng.dirichlet(np.ones(nc)).astype(np.float32))
    return c, p.to(cuda), q.to(cuda)


def _run(lib, c, p, q, G, parts):
    from reg_drot._lib import DrotResult
    nc, nr = c.shape
    dt = 1 if c.dtype == torch.bfloat16 else 0
    s = float(np.float32(2.0) / np.float32(nr + nc))
    dev = c.device
    st = {"x": torch.empty(nc, nr, device=dev), "a": torch.empty(nr, device=dev),
          "b": torch.empty(nc, device=dev), "phi1": torch.empty(nr, device=dev),
          "phi2": torch.empty(nc, device=dev), "alpha": torch.empty(1, device=dev)}
    ptrs = [t.data_ptr() for t in st.values()]
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.drot_init_state(nr, nc, s, 1, p.data_ptr(), q.data_ptr(), *ptrs, stream) == 0
    nbytes = lib.drot_gl_workspace_bytes(nr, nc, G)
    ws = torch.empty(nbytes + 256, dtype=torch.uint8, device=dev)
    objective = None
    for n in parts:
        res = DrotResult()
        assert lib.drot_gl_solve_ex(
            c.data_ptr(), dt, p.data_ptr(), q.data_ptr(), nr, nc, G, s, 1e-6, n, -1.0, *ptrs,
            ws.data_ptr() + (-ws.data_ptr()) % 256, nbytes, ctypes.byref(res), stream) == 0
        objective = res.as_dict()["objective_f64"]
    return dict(st, objective=torch.tensor(objective))


# tiles; in L2; beyond it: teams of 4 and of 8 vectors, a class per warp (two CTAs
# per SM), unaligned columns, fewer columns per warp than blocks, a BF16 cost
SHAPES = [(500, 400, 2, torch.float32), (2600, 2100, 2, torch.float32),
          (6000, 5000, 3, torch.float32), (10000, 2000, 2, torch.float32),
          (8192, 2600, 16, torch.float32), (5003, 4001, 2, torch.float32),
          (40000, 450, 10, torch.float32), (7000, 6000, 7, torch.bfloat16)]


@pytest.mark.parametrize("nr,nc,G,dtype", SHAPES, ids=[f"{a}x{b}g{g}" for a, b, g, _ in SHAPES])
def test_any_split_gives_the_bits_of_one_launch(cuda, solver_lib, nr, nc, G, dtype):
    c, p, q = _problem(nr, nc, nr + nc, cuda)
    c = c.to(dtype)
    one = _run(solver_lib, c, p, q, G, (6,))
    for parts in ((1, 5), (3, 3), (1, 1, 1, 1, 1, 1)):
        st = _run(solver_lib, c, p, q, G, parts)
        for k in one:
            assert torch.equal(one[k], st[k]), (parts, k)


def test_plan_and_gradient_do_not_depend_on_the_checkpoint_spacing(cuda):
    from reg_drot.autograd import group_lasso_drot_fn
    nr, nc, G = 5200, 4800, 3
    c, p, q = _problem(nr, nc, 1, cuda)
    up = torch.randn(nc, nr, device=cuda)
    out = []
    for segment, last_k in ((4, None), (3, None), (5, 4), (6, 4)):
        cc = c.clone().requires_grad_(True)
        x = group_lasso_drot_fn(cc, p, q, G, 2.0, 1e-9, 6, -1.0, segment=segment, last_k=last_k)
        out.append((x.detach(), torch.autograd.grad(x, cc, up)[0]))
    assert int((out[0][0] > 0).sum()) > nr
    for x, _ in out[1:]:
        assert torch.equal(x, out[0][0])
    assert torch.equal(out[1][1], out[0][1])
    assert torch.equal(out[3][1], out[2][1])
