"""The device's uniforms and normals from their 64 bits: the fp32 roundings of the exact values, and
the fp32 oracle's quantile, at every leading-bit count the draws reach."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_uniforms_and_normals_bit_exact(gpu_lib, oracle_mod):
    from jaxns_gb300 import _ffi
    n = 1 << 24                                       # down to ~24 leading zeros: both conversions' paths
    key = torch.tensor([7, 11], dtype=torch.int32, device="cuda")
    bits = torch.empty(n, dtype=torch.int64, device="cuda")
    u, z = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(2))
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    for fn, out in (("gbns_random_bits64", bits), ("gbns_uniform", u), ("gbns_normal", z)):
        _ffi.call(fn, p(key), p(out), ctypes.c_longlong(n), ctypes.c_void_p(0))
    torch.cuda.synchronize()
    M = bits.cpu().numpy().view(np.uint64) >> np.uint64(12)
    want = M.astype(np.float32) * np.float32(2.0 ** -52)
    np.testing.assert_array_equal(u.cpu().numpy().view(np.uint32), want.view(np.uint32))
    z = z.cpu().numpy()
    fn = oracle_mod.lib().orc32_fm_normal_from_bits
    fn.restype, fn.argtypes = ctypes.c_float, [ctypes.c_uint64]
    from_half = np.abs(M.astype(np.int64) - (1 << 51))
    order = np.argsort(M)
    rows = np.concatenate([np.arange(20000), np.argsort(from_half)[:3000], order[:3000], order[-3000:]])
    ref = np.array([fn(int(M[i]) << 12) for i in rows], np.float32)
    np.testing.assert_array_equal(z[rows].view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("runs", [1, 20, 100, 1100])  # 32, 8 and 4 lanes per chain, one thread per chain
@pytest.mark.parametrize("D", [1, 3, 9, 15])
def test_odd_dimensions_of_the_shells(gpu_lib, oracle_mod, runs, D):
    """The shells' likelihood takes the dimensions in pairs."""
    from conftest import assert_shell_exact
    from jaxns_gb300.engine import NSBatch, RunSpec, shells_offset, shells_params
    n, c = 42, np.zeros(D)
    c[0] = 3.5
    spec = RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=7, family=1, params=shells_params(c, -c, 2.0, 0.1),
                   prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -6.0), prior_b=np.full(D, 12.0), max_samples=40 * n,
                   term_cond={"max_samples": 40 * n}, key=oracle_mod.PRNGKey(D), log_L_offset=shells_offset(0.1))
    b = NSBatch([spec] * runs, device="cuda")
    b.init()
    b.iterate(5)
    live = b.live_view(0)["log_L_raw"].cpu().numpy()
    key = oracle_mod.PRNGKey(8)
    b.slice_shell(torch.full((runs,), float(live[20])), torch.tensor(key.view(np.int32)).repeat(runs, 1))
    torch.cuda.synchronize()
    for r in {0, runs - 1}:
        assert_shell_exact(oracle_mod, b, r, live[20], key)
