"""The prior transform on both sides of the row counts from which a warp takes tiles of rows: the same
bits row by row."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tril", [True, False])
@pytest.mark.parametrize("D", [1, 3, 8, 17, 32, 33, 64, 65, 100, 128])
def test_both_sides(gpu_lib, D, tril, dtype):
    from jaxns_gb300 import _ffi
    g = np.random.default_rng(D)
    dev = lambda x: torch.as_tensor(x, device="cuda")
    kind = dev((g.random(D) < 0.7).astype(np.int32))
    a, b, ln, c = dev(g.standard_normal(D)), dev(0.5 + g.random(D)), dev(g.standard_normal(D)), dev(g.standard_normal(D))
    A = dev(np.tril(g.standard_normal((D, D))))
    rs = dev(np.maximum(0, np.arange(D) - g.integers(0, D + 1, D)).astype(np.int32))
    tab = _ffi.PriorTable(D=D, kind=kind.data_ptr(), a=a.data_ptr(), b=b.data_ptr(), log_norm=ln.data_ptr(),
                          A=A.data_ptr() if tril else None, row_start=rs.data_ptr(), c=c.data_ptr(), log_det=0.25)
    line = (16 if D <= 32 else 8) * torch.cuda.get_device_properties(0).multi_processor_count
    U = torch.rand(line + 7, D, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(D)).to(dtype)
    U.view(-1)[::7] = 2.0 ** -24
    L = torch.rand(line + 7, dtype=torch.float64, device="cuda")
    p = lambda x: ctypes.c_void_p(x.data_ptr() if x is not None else 0)

    def run(M):
        X, out = torch.empty(M, D, dtype=torch.float64, device="cuda"), torch.empty(M, dtype=torch.float64, device="cuda")
        f32 = dtype == torch.float32
        _ffi.call("gbns_prior_transform", ctypes.byref(tab), p(U if f32 else None), p(None if f32 else U),
                  ctypes.c_longlong(M), p(L), p(X), p(out), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return X.cpu().numpy(), out.cpu().numpy()

    few = run(line)  # a warp per row
    for M in (line + 1, line + 7):  # tiles
        many = run(M)
        for x, y in zip(many, few):
            np.testing.assert_array_equal(x[:line], y)
