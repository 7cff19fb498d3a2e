"""The register's log X of a long sample set is summed in FP64 between threads and blocks."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("live", [2, 14, 29, 64])
def test_register_log_X_is_fp64(gpu_lib, live):
    """One sample per thread of every block, all with the same live-point count: the exact sum of the
    table's entries (fp32 pairs, exact in FP64) against the register.  Roundings of 2^-53 of the sum at
    most: five levels of a warp, four levels or sixteen in turn over the warps (8.5 at most, each the size
    of its partial sum), five blocks per lane (3), five levels.  As fp32 pairs these counts are off by up to
    42 2^-53."""
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import ncoef_table
    N = 512 * torch.cuda.get_device_properties(0).multi_processor_count - 1
    table = ncoef_table(live)
    L = (-50.0 * np.exp(-np.arange(N) / (4.0 * N))).astype(np.float32)
    dev = lambda x: torch.as_tensor(x, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    tL, tn, tab = dev(L), torch.full((N,), live, dtype=torch.int32, device="cuda"), dev(table)
    fin, lX = torch.empty(8, dtype=torch.float64, device="cuda"), torch.empty(N, dtype=torch.float64, device="cuda")
    _ffi.call("gbns_evidence_stats", p(tL), p(tn), ctypes.c_longlong(N), p(tab), ctypes.c_int(live), p(fin), p(lX),
              ctypes.c_void_p(0), ctypes.c_void_p(0), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    pairs = table[live, 8:].view(np.float32)
    final = fin.cpu().numpy()
    for got, k in ((final[1], 0), (final[2], 4)):  # log X, log X2
        exact = N * (Fraction(float(pairs[k])) + Fraction(float(pairs[k + 1])))
        assert abs((Fraction(float(got)) - exact) / exact) <= 22 * 2.0 ** -53


@pytest.mark.parametrize("N,at", [(3000, 2999), (3001, 3000), (3001, 1500), (20000, 19999), (300001, 300000), (300001, 77777)])
def test_a_count_of_zero_leaves_the_samples_before_it(gpu_lib, N, at):
    """X is 0 after a sample with no live point; log X before it is what it is without it."""
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import ncoef_table
    dev = lambda x: torch.as_tensor(x, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    n = np.random.default_rng(N).integers(1, 60, N).astype(np.int32)
    n[at] = 0
    tL, tn, tab = dev(np.sort(np.random.default_rng(at).standard_normal(N)).astype(np.float32)), dev(n), dev(ncoef_table(64))
    fin, lX, ldZ = (torch.empty(k, dtype=torch.float64, device="cuda") for k in (8, N, N))
    _ffi.call("gbns_evidence_stats", p(tL), p(tn), ctypes.c_longlong(N), p(tab), ctypes.c_int(64), p(fin), p(lX), p(ldZ),
              ctypes.c_void_p(0), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    ref = np.cumsum(-np.log1p(1.0 / n[:at].astype(np.longdouble))).astype(np.float64)
    np.testing.assert_allclose(lX.cpu().numpy()[:at], ref, rtol=1e-12, atol=1e-12)
    assert np.isfinite(ldZ.cpu().numpy()[:at]).all()
