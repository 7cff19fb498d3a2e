"""The prior transform's row tiles, bit for bit the oracle, at the edges of their sizes; and
sample_evidence at the edges of its threads, tiles, clusters and replica groups."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("D,M,tril", [(1, 1, False), (2, 513, True), (5, 127, True), (8, 10001, True), (8, 4864, False),
                                      (16, 33, True), (31, 1000, True), (32, 5, False), (33, 301, True), (64, 1001, True),
                                      (65, 7, True), (96, 300, False), (97, 77, True), (128, 1300, True), (129, 301, True)])
def test_transform_tiles(gpu_lib, oracle_mod, D, M, tril, dtype):
    import ctypes
    from jaxns_gb300 import _ffi
    g = np.random.default_rng(D * M)
    kind = (g.random(D) < 0.7).astype(np.int32)
    a, b, ln = g.standard_normal(D), 0.5 + g.random(D), g.standard_normal(D)
    A = np.tril(g.standard_normal((D, D))) if tril else None
    row_start = np.maximum(0, np.arange(D) - g.integers(0, D + 1, D)).astype(np.int32)
    c = g.standard_normal(D)
    U = g.random((M, D)).astype(dtype)
    U[0, 0], U[-1, -1] = 0.0, 1.0                     # infinite normals
    U.flat[:: 7] = np.float32(2.0 ** -24)             # many tails in one warp's tile
    lL = g.standard_normal(M)
    lL[M // 2] = -np.inf
    dev = {k: torch.tensor(v, device="cuda") for k, v in dict(kind=kind, a=a, b=b, ln=ln, rs=row_start, c=c, U=U, L=lL).items()}
    Ad = torch.tensor(A, device="cuda") if tril else None
    X = torch.full((M, D), 7.0, dtype=torch.float64, device="cuda")
    out = torch.full((M,), 7.0, dtype=torch.float64, device="cuda")
    p = lambda x: ctypes.c_void_p(x.data_ptr() if x is not None else 0)  # (a bare int would be cut to 32 bits)
    tab = _ffi.PriorTable(D=D, kind=dev["kind"].data_ptr(), a=dev["a"].data_ptr(), b=dev["b"].data_ptr(),
                          log_norm=dev["ln"].data_ptr(), A=Ad.data_ptr() if tril else None,
                          row_start=dev["rs"].data_ptr() if tril else None, c=dev["c"].data_ptr() if tril else None,
                          log_det=0.25)
    f32 = dtype == np.float32
    _ffi.call("gbns_prior_transform", ctypes.byref(tab), p(dev["U"] if f32 else None), p(None if f32 else dev["U"]),
              ctypes.c_longlong(M), p(dev["L"]), p(X), p(out), p(None))
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        Xo, oo = oracle_mod.prior_transform(kind, a, b, ln, U, A=A, row_start=row_start, c=c, log_det=0.25, log_L=lL)
    np.testing.assert_array_equal(X.cpu().numpy(), Xo)
    np.testing.assert_array_equal(out.cpu().numpy(), oo)


@pytest.mark.parametrize("N,S", [(1, 1), (2, 300), (511, 5), (1024, 101), (2049, 607), (4097, 100), (33001, 3), (40000, 1300)])
def test_sample_evidence_edges(gpu_lib, oracle_mod, N, S):
    from jaxns_gb300 import sample_evidence
    g = np.random.default_rng(N + S)
    n = g.integers(N // 40 + 1, N // 20 + 3, N)
    n[N // 2] = 1                                     # a large step of log X
    n[-min(N, 5):] = np.arange(min(N, 5), 0, -1)
    L = np.sort(-0.5 * g.chisquare(6, N) * 20.0)
    L[: N // 9] = -np.inf                             # samples that add nothing
    got = sample_evidence(np.array([3, N], np.uint32), n, L, S=S).cpu().numpy()
    ref = oracle_mod.sample_evidence(np.array([3, N], np.uint32), n, L, S=S)
    # each log X is a sum of N terms and each log Z one of N terms: N roundings of the largest size
    tol = 4 * (N + 8) * 2.0 ** -53 * max(1.0, np.sum(1.0 / n) * 2 + 80, np.abs(L[np.isfinite(L)]).max(initial=0.0))
    assert np.isfinite(ref).all()
    np.testing.assert_allclose(got, ref, rtol=0, atol=tol)
