"""The merge with several blocks per run (few runs) and with one narrow block per run (many runs):
the same permutation, store and phantoms as numpy's stable argsort, the same register."""
import ctypes

import numpy as np
import pytest

from conftest import corr_gauss

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _merge(oracle_mod, runs, n, s, K, ordered):
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import NSBatch, RunSpec, mvn_offset, mvn_params
    D = 3
    mu, cov = corr_gauss(D, 1)
    cap = 6 * s * (1 + K) + 2 * n
    cap += -cap % (s * (1 + K))
    spec = RunSpec(D=D, num_live_points=n, shell_size=s, num_slices=K + 1, family=0, params=mvn_params(mu, cov),
                   prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -10.0), prior_b=np.full(D, 20.0),
                   max_samples=cap, term_cond={"max_samples": float(cap)}, key=oracle_mod.PRNGKey(3),
                   num_phantom=K, log_L_offset=float(mvn_offset(cov)))
    b = NSBatch([spec] * runs)
    b.init()
    g = np.random.default_rng(n + s)
    live = np.round(g.standard_normal(n) * 3, 1).astype(np.float32)
    live = np.sort(live) if ordered else live
    new = np.round(g.standard_normal(s) * 3, 1).astype(np.float32)
    U, nU = g.random((n, D), np.float32), g.random((s, D), np.float32)
    pL, pU = g.random(s * K, np.float32), g.random(s * K * D, np.float32)
    for r in range(runs):
        b.set_live(r, U, live)
    rep = lambda x: torch.from_numpy(np.tile(np.ravel(x), runs))
    b.new_L.copy_(rep(new))
    b.new_U.copy_(rep(nU))
    b.new_E.copy_(rep(np.arange(s, dtype=np.int32) + 1))
    if K:
        b.ph_L.copy_(rep(pL))
        b.ph_U.copy_(rep(pU))
    _ffi.call("gbns_batch_merge", ctypes.byref(b._b), b._stream())
    torch.cuda.synchronize()
    if s == n:  # no seed points above the contour: the run ended at its start and the merge leaves it
        rec = b.state()[runs - 1]
        assert rec["done"] == 1 and rec["iterations"] == 0
        np.testing.assert_array_equal(b.live_view(runs - 1)["log_L_raw"].cpu().numpy(), live)
        return rec
    key = np.concatenate([new, live[s:]])
    perm = np.argsort(key + 0.0, kind="stable")
    r = runs - 1
    v = b.live_view(r)
    np.testing.assert_array_equal(v["log_L_raw"].cpu().numpy(), key[perm])
    np.testing.assert_array_equal(v["U"].cpu().numpy(), np.concatenate([nU, U[s:]])[perm])
    st = b.store_view(r)
    np.testing.assert_array_equal(st["log_L_raw"][:s].cpu().numpy(), live[:s])
    np.testing.assert_array_equal(st["U"][:s].cpu().numpy(), U[:s])
    np.testing.assert_array_equal(st["log_L_raw"][s:s + s * K].cpu().numpy(), pL)
    np.testing.assert_array_equal(st["U"][s:s + s * K].cpu().numpy().ravel(), pU)
    np.testing.assert_array_equal(st["phantom"][:s + s * K].cpu().numpy(), np.repeat([0, 1], [s, s * K]))
    rec = b.state()[r]
    assert rec["pad1"] == 0 and rec["iterations"] == 1 and rec["next_sample_idx"] == s * (1 + K)
    return rec


@pytest.mark.parametrize("n,s,K,ordered", [(2, 1, 0, True), (9, 9, 0, True), (33, 1, 2, True), (240, 120, 0, True),
                                           (513, 256, 1, True), (1001, 500, 0, False), (4096, 2048, 0, True)])
def test_blocks_per_run(gpu_lib, oracle_mod, n, s, K, ordered):
    recs = [_merge(oracle_mod, runs, n, s, K, ordered) for runs in (1, 40, 320)]
    for rec in recs[1:]:
        for f in ("num_samples", "num_likelihood_evaluations", "plateau", "no_seed_points", "done", "termination_reason",
                  "log_L_contour", "absolute_spread", "relative_spread"):
            assert rec[f] == recs[0][f], f
        np.testing.assert_array_equal(rec["key"], recs[0]["key"])
        for f in ("ev", "ev_rem"):  # sums of pairs in another grouping: a few units of 2^-48
            for x, y in zip(rec[f].tolist(), recs[0][f].tolist()):
                assert x == y or abs(x - y) < 1e-11 * max(1.0, abs(y)), (f, x, y)
