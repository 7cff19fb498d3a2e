"""Host threads that drive batches and transforms of different sizes at the same time."""
import ctypes
import threading

import numpy as np
import pytest

from conftest import corr_gauss

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _together(calls, times):
    """Runs the calls in a thread each, in their own streams, and returns what they raised."""
    errors, start = [], threading.Barrier(len(calls))

    def work(f):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(times):
                    f()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 - handed to the test
            errors.append(e)

    threads = [threading.Thread(target=work, args=(f,)) for f in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_merges_of_different_sizes(gpu_lib, oracle_mod):
    """Live sets above 32 KB of shared memory, of three sizes, merged side by side."""
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import NSBatch, RunSpec, mvn_offset, mvn_params
    mu, cov = corr_gauss(2, 1)
    batches = []
    for n in (2100, 3000, 4096):
        b = NSBatch([RunSpec(D=2, num_live_points=n, shell_size=n // 2, num_slices=2, family=0, params=mvn_params(mu, cov),
                             prior_kind=np.zeros(2, np.int32), prior_a=np.full(2, -10.0), prior_b=np.full(2, 20.0),
                             max_samples=4 * n, term_cond={"max_samples": 1.0}, key=oracle_mod.PRNGKey(n), store_U=False,
                             log_L_offset=float(mvn_offset(cov)))])
        b.init()
        b.iterate(1)  # done: the merges below only launch
        batches.append(b)
    torch.cuda.synchronize()
    assert not _together([lambda b=b: _ffi.call("gbns_batch_merge", ctypes.byref(b._b), b._stream()) for b in batches], 3000)


def test_transforms_of_different_sizes(gpu_lib):
    """MultivariateNormalTriL maps of 46 to 64 dimensions transformed side by side."""
    import jaxns_gb300 as gb
    calls = []
    for D in (46, 55, 64):
        def prior_model(D=D):
            x = yield gb.Prior(gb.MultivariateNormalTriL(np.zeros(D), np.eye(D)), name="x")
            return x
        m = gb.Model(prior_model, gb.MultivariateNormalLikelihood(np.zeros(D), np.eye(D)))
        U = torch.rand(4, D, device="cuda").clamp(0.01, 0.99)
        m.transform_device(U)
        calls.append(lambda m=m, U=U: m.transform_device(U))
    torch.cuda.synchronize()
    assert not _together(calls, 2000)
