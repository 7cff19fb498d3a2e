"""A stream that owns some of the device's SMs only (a green context): the results passes run there with
one block per run, and give what they give on the whole device."""
import contextlib
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _part_stream(min_sms):
    """A stream of a green context of at least min_sms SMs (skips where the driver has none)."""
    try:
        cu = ctypes.CDLL("libcuda.so.1")
        names = ("cuDeviceGetDevResource", "cuDevSmResourceSplitByCount", "cuDevResourceGenerateDesc", "cuGreenCtxCreate",
                 "cuGreenCtxStreamCreate", "cuGreenCtxDestroy", "cuStreamDestroy_v2")
        get, split, describe, create, stream_create, destroy, stream_destroy = (getattr(cu, n) for n in names)
    except (OSError, AttributeError) as e:
        pytest.skip(f"no green contexts: {e}")
    torch.zeros(1, device="cuda")  # the primary context
    res, part = (ctypes.c_ubyte * 144)(), (ctypes.c_ubyte * 144)()  # CUdevResource
    n, desc, ctx, stream = ctypes.c_uint(1), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    dev = ctypes.c_int(torch.cuda.current_device())
    for rc in (get(dev, res, 1), split(part, ctypes.byref(n), res, None, 0, min_sms), describe(ctypes.byref(desc), part, 1),
               create(ctypes.byref(ctx), desc, dev, 1), stream_create(ctypes.byref(stream), ctx, 1, 0)):
        if rc != 0:
            pytest.skip(f"no green context here (driver error {rc})")
    try:
        yield torch.cuda.ExternalStream(stream.value)
        torch.cuda.synchronize()
    finally:
        stream_destroy(stream)
        destroy(ctx)


def test_results_of_few_runs(gpu_lib):
    from test_gpu_team import _batch
    ref_b, ref = _batch(100, 3, True)  # one block per run
    b, _ = _batch(2, 3, True)
    torch.cuda.synchronize()
    with _part_stream(16) as s:
        with torch.cuda.stream(s):
            out = b.results(with_U=True)
        s.synchronize()
        for r in range(2):
            v, w = b.run_slices(r, out), ref_b.run_slices(r, ref)
            for f in v:
                np.testing.assert_array_equal(v[f].cpu().numpy(), w[f].cpu().numpy(), err_msg=f)


def test_long_sets(gpu_lib, oracle_mod):
    from test_gpu_team import test_long_sets_match_the_oracle
    with _part_stream(16) as s:
        with torch.cuda.stream(s):
            test_long_sets_match_the_oracle(gpu_lib, oracle_mod, 6001, 100, True, True)
            test_long_sets_match_the_oracle(gpu_lib, oracle_mod, 6001, 100, False, False)
