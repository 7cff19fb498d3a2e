"""Runs whose store is smaller than what one iteration appends."""
import ctypes

import numpy as np
import pytest

from conftest import corr_gauss

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _spec(oracle_mod, n, s, K, cap, limit=False):
    from jaxns_gb300.engine import RunSpec, mvn_offset, mvn_params
    D = 2
    mu, cov = corr_gauss(D, 1)
    return RunSpec(D=D, num_live_points=n, shell_size=s, num_slices=K + 1, family=0, params=mvn_params(mu, cov),
                   prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -10.0), prior_b=np.full(D, 20.0), max_samples=cap,
                   term_cond={"max_samples": float(cap)} if limit else {"dlogZ": 1e-30}, key=oracle_mod.PRNGKey(5), num_phantom=K,
                   log_L_offset=float(mvn_offset(cov)))


@pytest.mark.parametrize("limit", [False, True])  # with the sample limit the run ends before its first shell
@pytest.mark.parametrize("n,s,K,cap", [(16, 8, 0, 4), (16, 8, 0, 8), (16, 8, 2, 8), (300, 150, 0, 150), (9, 8, 3, 5)])
def test_appends_stay_in_the_store(gpu_lib, oracle_mod, n, s, K, cap, limit):
    """A capacity below one shell, its phantoms or the live set: the run's appends end at its own
    last slot, and the next run's store holds what it holds alone."""
    from jaxns_gb300.engine import NSBatch
    small, big = _spec(oracle_mod, n, s, K, cap, limit), _spec(oracle_mod, 64, 32, 1, 64 * 40)
    alone, both = NSBatch([big]), NSBatch([small, big])
    for b in (alone, both):
        b.init()
        b.iterate(1)
        b.finalize()
    st = both.state()
    assert st["iterations"][0] == (0 if limit else 1) and st["iterations"][1] == 1
    assert st["num_samples"][1] == alone.state()["num_samples"][0]
    for f in ("store_L", "store_S", "store_E", "store_P"):
        np.testing.assert_array_equal(getattr(both, f)[cap:].cpu().numpy(), getattr(alone, f).cpu().numpy(), err_msg=f)
    np.testing.assert_array_equal(both.store_U[2 * cap:].cpu().numpy(), alone.store_U.cpu().numpy())
    if st["done"][0]:  # (a store of exactly one shell goes on) the live points, appended last, fill the whole store
        live = both.live_view(0)["log_L_raw"].cpu().numpy()
        np.testing.assert_array_equal(both.store_L[:cap].cpu().numpy(), live[:cap])


@pytest.mark.parametrize("runs", [1, 60, 320])  # many, two and one block per run
def test_phantoms_overwrite_the_shell_they_overlap(gpu_lib, oracle_mod, runs):
    """Capacity 18 for a shell of 8 and 16 phantoms: the phantoms start at slot 2, over the shell
    written before them, and the live points follow at slot 6."""
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import NSBatch
    n, s, K, cap = 9, 8, 2, 18
    b = NSBatch([_spec(oracle_mod, n, s, K, cap)] * runs)
    b.init()
    old = b.live_view(runs - 1)
    old = {k: old[k].cpu().numpy().copy() for k in ("log_L_raw", "U")}
    _ffi.call("gbns_batch_shell", ctypes.byref(b._b), b._stream())
    pL = b.ph_L[-s * K:].cpu().numpy()
    pU = b.ph_U[-s * K * 2:].view(-1, 2).cpu().numpy()
    _ffi.call("gbns_batch_merge", ctypes.byref(b._b), b._stream())
    new = b.live_view(runs - 1)
    L, U = b.store_L[-cap:].cpu().numpy(), b.store_U[-2 * cap:].view(-1, 2).cpu().numpy()
    for got, shell, ph, live in ((L, old["log_L_raw"], pL, new["log_L_raw"]), (U, old["U"], pU, new["U"])):
        np.testing.assert_array_equal(got[:2], shell[:2])
        np.testing.assert_array_equal(got[2:6], ph[:4])
        np.testing.assert_array_equal(got[6:15], live.cpu().numpy())
        np.testing.assert_array_equal(got[15:], ph[13:])
    np.testing.assert_array_equal(b.store_P[-cap:].cpu().numpy(), [0] * 2 + [1] * 4 + [0] * 9 + [1] * 3)
