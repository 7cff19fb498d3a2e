"""The results of few or long runs on a team of blocks: block counts from one to all, in-order and
out-of-order stores, the same as one block per run."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _batch(runs, K, with_U):
    import jaxns_gb300 as gb
    from jaxns_gb300.engine import NSBatch, RunSpec, shells_offset, shells_params
    D, n = 3, 300
    c = np.zeros(D)
    c[0] = 3.5
    cap = n * 40 * (1 + K)
    specs = [RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=4, family=1,
                     params=shells_params(c, -c, 2.0, 0.1), prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -6.0),
                     prior_b=np.full(D, 12.0), max_samples=cap, term_cond={"dlogZ": 1e-4, "max_samples": float(cap)},
                     num_phantom=K, key=gb.random.PRNGKey(100 + r % 2), store_U=with_U, log_L_offset=shells_offset(0.1))
             for r in range(runs)]
    b = NSBatch(specs)
    b.run(block=8)
    return b, b.results(with_U=with_U)


@pytest.mark.parametrize("K", [0, 3])
def test_teams_match_one_block(gpu_lib, K):
    ref_b, ref = _batch(100, K, True)  # more than half as many runs as SMs: one block per run
    for runs in (1, 2, 7, 60):
        b, out = _batch(runs, K, True)
        for r in {0, runs - 1}:
            v, w = b.run_slices(r, out), ref_b.run_slices(r % 2, ref)
            for f in ("samples_indices", "num_live_points", "log_L_samples", "nevals_sorted", "U_sorted"):
                np.testing.assert_array_equal(v[f].cpu().numpy(), w[f].cpu().numpy(), err_msg=f)
            # sums of the same fp32-pair terms in another grouping: a few units of 2^-48 per sample
            for f in ("log_X_mean", "log_dp_mean", "scalars"):
                np.testing.assert_allclose(v[f].cpu().numpy(), w[f].cpu().numpy(), rtol=1e-11, atol=1e-11, err_msg=f)


@pytest.mark.parametrize("N,live,shuffle", [(16383, 64, True), (16384, 64, False), (16384, 500, True), (77825, 1000, False),
                                            (77825, 1000, True), (300001, 100, True)])
@pytest.mark.parametrize("lz", [True, False])
def test_long_sets_match_the_oracle(gpu_lib, oracle_mod, N, live, shuffle, lz):
    """Around the size at which one block hands over to the team, through gbns_count_crossed_edges and
    gbns_evidence_stats (with and without the per-sample log Z)."""
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import ncoef_table
    g = np.random.default_rng(N + live)
    L = np.sort((-50.0 * np.exp(-np.arange(N) / (4.0 * live))).astype(np.float32))
    sender = np.maximum(np.arange(N) - g.integers(live // 2, live, N), 0).astype(np.int32)
    if shuffle:
        order = np.argsort(np.arange(N) + g.integers(0, live, N), kind="stable")
        L, sender = L[order], np.minimum(sender, np.arange(N)).astype(np.int32)
    dev = lambda x: torch.as_tensor(x, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    tL, ts, i32 = dev(L), dev(sender), dict(dtype=torch.int32, device="cuda")
    si, nl, deg = torch.empty(N, **i32), torch.empty(N, **i32), torch.empty(N + 1, **i32)
    sll = torch.empty(2 * (N + 1), dtype=torch.int64, device="cuda")
    n = ctypes.c_longlong(N)
    _ffi.call("gbns_count_crossed_edges", p(ts), p(tL), n, p(si), p(nl), p(sll), p(deg), s)
    osi, onl = oracle_mod.count_crossed_edges(sender, L.astype(np.float64))
    np.testing.assert_array_equal(si.cpu().numpy(), osi)
    np.testing.assert_array_equal(nl.cpu().numpy(), onl)
    Ls = np.ascontiguousarray(L[osi])
    counts = np.clip(onl, 1, 2 * live).astype(np.int32)
    f64 = dict(dtype=torch.float64, device="cuda")
    fin, lX, ldZ = torch.empty(8, **f64), torch.empty(N, **f64), torch.empty(N, **f64)
    lZ = torch.empty(N, **f64) if lz else None
    tab, tLs, tn = dev(ncoef_table(live)), dev(Ls), dev(counts)  # counts beyond the table are computed
    _ffi.call("gbns_evidence_stats", p(tLs), p(tn), n, p(tab), ctypes.c_int(live), p(fin), p(lX), p(ldZ), p(lZ), s)
    ofin, per = oracle_mod.compute_evidence_stats(Ls.astype(np.float64), counts.astype(np.float64))
    # log X against an extended-precision running sum: the oracle's own FP64 one, 300,000 additions of
    # nearly equal terms, is off by up to N 2^-53 of its value
    np.testing.assert_allclose(lX.cpu().numpy(), np.cumsum(-np.log1p(1.0 / counts.astype(np.longdouble))).astype(np.float64),
                               rtol=1e-12, atol=1e-12)
    # terms carry fp32 mantissas: ~1e-7 each, as in the one-block scan's test
    np.testing.assert_allclose(ldZ.cpu().numpy(), per["log_dZ_mean"], rtol=1e-6, atol=1e-6)
    np.testing.assert_allclose(fin.cpu().numpy(), [ofin[f] for f in oracle_mod.EV_FIELDS], rtol=1e-6, atol=1e-6)
    if lz:
        np.testing.assert_allclose(lZ.cpu().numpy(), per["log_Z_mean"], rtol=1e-6, atol=1e-6)


def test_team_launches_are_capturable(gpu_lib):
    """The results pass of one run replayed from a CUDA graph gives the same scalars."""
    b, out = _batch(1, 0, False)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        again = b.results(with_U=False)
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(again["scalars"].cpu().numpy(), out["scalars"].cpu().numpy())


@pytest.mark.parametrize("N,live,shuffle", [(2999, 50, True), (3000, 50, False), (3000, 400, True), (3001, 100, True),
                                            (7001, 300, True)])
@pytest.mark.parametrize("lz", [True, False])
def test_sets_at_the_hand_over_match_the_oracle(gpu_lib, oracle_mod, N, live, shuffle, lz):
    test_long_sets_match_the_oracle(gpu_lib, oracle_mod, N, live, shuffle, lz)
