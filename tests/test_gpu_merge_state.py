"""The merge on a state whose work word holds anything: a caller of the C ABI fills the run states
itself, and only the documented fields count."""
import ctypes

import numpy as np
import pytest

from conftest import corr_gauss

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["gbns_batch_merge", "gbns_batch_iterate"])
@pytest.mark.parametrize("runs", [1, 9, 100, 400])  # 16, 16, one and one block per run
def test_any_work_word(gpu_lib, oracle_mod, runs, entry):
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import _STATE_DTYPE, NSBatch, RunSpec, mvn_offset, mvn_params
    D, n = 2, 64
    mu, cov = corr_gauss(D, 1)
    spec = RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=3, family=0, params=mvn_params(mu, cov),
                   prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -10.0), prior_b=np.full(D, 20.0),
                   max_samples=40 * n, term_cond={"dlogZ": 1e-30}, key=oracle_mod.PRNGKey(3),
                   log_L_offset=float(mvn_offset(cov)))
    out = []
    for fill in (False, True):
        b = NSBatch([spec] * runs)
        b.init()
        for _ in range(3):
            if fill:
                st = b.state().copy()
                st["pad1"] = np.random.default_rng(1).integers(-2 ** 31, 2 ** 31, runs)
                b.t_state.copy_(torch.frombuffer(bytearray(st.tobytes()), dtype=torch.uint8))
            if entry == "gbns_batch_merge":
                _ffi.call("gbns_batch_shell", ctypes.byref(b._b), b._stream())
                _ffi.call(entry, ctypes.byref(b._b), b._stream())
            else:
                _ffi.call(entry, ctypes.byref(b._b), 2, b._stream())
        out.append((b.state(), b.live_L[0].cpu().numpy(), b.live_L[1].cpu().numpy(), b.store_L.cpu().numpy()))
    assert _STATE_DTYPE.names[-1] == "pad1"
    fields = [f for f in _STATE_DTYPE.names if f != "pad1"]
    assert np.all(out[0][0]["iterations"] == (3 if entry == "gbns_batch_merge" else 6))
    for f in fields:
        np.testing.assert_array_equal(out[0][0][f], out[1][0][f], err_msg=f)
    for x, y in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(x, y)
