"""GPU: plan and duals of a resident solve where the numbers are small -- a cold
start with zero duals, marginals with entries of 1e-8 and 1e-11, a cost in small
units -- against the iteration in FP64.

The exchange words hold sums to 2^-47 per CTA (GC of them: below 2^-42 here), an
absolute bound, against FP32 roundings of the sums and duals.  Both kernels are
measured, and the bar on the resident one is twice the streaming kernel's error
plus one FP32 rounding: per vector, and over the rows of the small marginals plus
the words' resolution.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

EPS32 = 2.0 ** -24


def _solve(lib, c, p, q, s, kappa, iters):
    from reg_drot._lib import DrotResult
    nc, nr = c.shape
    dev = c.device
    st = {"x": torch.empty(nc, nr, device=dev), "a": torch.empty(nr, device=dev),
          "b": torch.empty(nc, device=dev), "phi1": torch.empty(nr, device=dev),
          "phi2": torch.empty(nc, device=dev), "alpha": torch.empty(1, device=dev)}
    ptrs = [t.data_ptr() for t in st.values()]
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.drot_init_state(nr, nc, s, 0, p.data_ptr(), q.data_ptr(), *ptrs, stream) == 0
    start = {k: v.double().clone() for k, v in st.items()}
    nbytes = lib.drot_qr_workspace_bytes(nr, nc)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    assert lib.drot_qr_solve(c.data_ptr(), p.data_ptr(), q.data_ptr(), nr, nc, s, kappa, iters,
                             -1.0, *ptrs, ws.data_ptr(), nbytes, ctypes.byref(DrotResult()),
                             stream) == 0
    return start, st


@pytest.mark.parametrize("small", [1e-8, 1e-11])
@pytest.mark.parametrize("unit", [1e-6, 1.0, 30.0])
@pytest.mark.parametrize("nr,nc", [(96, 80), (700, 500), (1500, 1400)])
def test_errors_at_small_scales_are_the_streaming_kernels(cuda, solver_lib, nr, nc, unit, small):
    from reg_drot import autotune
    rng = np.random.default_rng(5)
    c = torch.from_numpy(rng.random((nc, nr), dtype=np.float32) * np.float32(unit)).to(cuda)
    marg = []
    for k in (nr, nc):
        v = rng.dirichlet(np.ones(k))
        v[::7] = small * (1 + rng.random(len(v[::7])))
        marg.append(torch.from_numpy((v / v.sum()).astype(np.float32)).to(cuda))
    p, q = marg
    s, kappa, iters = float(np.float32(2.0) / np.float32(nr + nc)), float(np.float32(1.02)), 8
    start, st = _solve(solver_lib, c, p, q, s, kappa, iters)
    autotune.pin("qr", 0, 0, vectors_per_lane=4)  # the streaming kernel
    try:
        _, ref = _solve(solver_lib, c, p, q, s, kappa, iters)
    finally:
        autotune.clear()
    d = start
    c64, p64, q64 = c.double(), p.double(), q.double()
    for _ in range(iters):
        d["x"] = (d["x"] + d["phi1"][None] + d["phi2"][:, None] - s * c64).clamp_min(0) / kappa
        r, k = d["x"].sum(0) - p64, d["x"].sum(1) - q64
        total = d["x"].sum()
        gamma = (2 * (total - 1) - d["alpha"]) / (nr + nc)
        d["a"], d["b"] = d["a"] - r, d["b"] - k
        d["phi1"], d["phi2"] = (d["a"] - r + gamma) / nc, (d["b"] - k + gamma) / nr
        d["alpha"] = d["alpha"] + 1 - total
    # a cost in small units leaves a mass of 1 up to rounding: alpha and the duals are
    # then sums of the roundings of the float mass (2^-25 each, twice that in gamma,
    # kept by alpha from one iteration to the next)
    mass = iters ** 2 * 2.0 ** -24 / min(nr, nc) if unit < 1.0 else 0.0
    for name in ("x", "a", "b", "phi1", "phi2"):
        size, n = float(d[name].norm()), d[name].numel()
        mine, theirs = (float((t[name].double() - d[name]).norm()) for t in (st, ref))
        assert mine <= 2 * theirs + EPS32 * size + mass * n ** 0.5, (name, mine / size, theirs / size)
    for name in ("a", "b"):
        rows = slice(None, None, 7)
        size, n = float(d[name][rows].norm()), d[name][rows].numel()
        mine, theirs = (float((t[name].double() - d[name])[rows].norm()) for t in (st, ref))
        words = iters * 2.0 ** -42 * n ** 0.5
        assert mine <= 2 * theirs + EPS32 * size + words + mass * n ** 0.5, name
