"""The sampler chosen by the chains at work at once: every choice, with the host's count, without one
and with any other, runs the same chains."""
import numpy as np
import pytest

from conftest import assert_shell_exact
from test_gpu_spec import _spec

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("D,family,runs,n,kw,lane,warp", [
    (8, "uniform", 3, 42, {}, 3 * 32, 0),                            # 21 chains a run: two groups of 16
    (10, "shells", 5, 402, {}, 5 * (64 * 3 + 16), 0),                # 201 chains: three items of 64 and one of 9
    (10, "shells", 2, 402, dict(chains_per_lane=2), 2 * (64 + 64), 0),   # 128 + 73 chains on 64 lanes
    (24, "uniform", 4, 402, {}, 0, 4 * 201), (40, "uniform", 4, 1002, {}, 0, 4 * 501),
    (24, "uniform", 2, 1402, dict(wide_chains_per_item=4096), 0, 2 * 512)])
def test_the_host_counts_the_chains_at_work(oracle_mod, D, family, runs, n, kw, lane, warp):
    from jaxns_gb300.engine import NSBatch
    b = NSBatch([_spec(oracle_mod, D, 2, 0, family, True, n=n)] * runs, device="cpu", **kw)
    assert (b._b.lane_chains, b._b.warp_chains) == (lane, warp)


# runs of 21 chains, counted as 32: 32, 8 and 4 lanes per chain and one thread per chain
@pytest.mark.gpu
@pytest.mark.parametrize("D,S,prior,runs", [(6, 7, "normal", (22, 23, 112, 113, 625, 626)), (16, 5, "uniform", (22, 112, 626)),
                                            (24, 5, "shells", (468, 469)), (48, 3, "shells", (390, 391))])
def test_lane_lines(gpu_lib, oracle_mod, D, S, prior, runs):
    from jaxns_gb300.engine import NSBatch
    spec = _spec(oracle_mod, D, S, 1, prior, True)
    for R in runs:
        _shell(oracle_mod, NSBatch([spec] * R, device="cuda"), spec, R)


# runs of 201 chains: 16, 8 and 4 proposals per round and the warp-cooperative kernel
@pytest.mark.gpu
@pytest.mark.parametrize("D,S,runs", [(20, 5, (5, 6, 10, 11, 109, 110)), (40, 3, (5, 7, 8, 69, 70))])
def test_warp_lines(gpu_lib, oracle_mod, D, S, runs):
    from jaxns_gb300.engine import NSBatch
    spec = _spec(oracle_mod, D, S, 1, "uniform", True, n=402)
    for R in runs:
        _shell(oracle_mod, NSBatch([spec] * R, device="cuda"), spec, R)


@pytest.mark.gpu
@pytest.mark.parametrize("D,prior", [(6, "normal"), (24, "uniform"), (24, "shells")])
@pytest.mark.parametrize("count", [0, -7, 1, 1500, 10000, 2 ** 31 - 1])
def test_any_count(gpu_lib, oracle_mod, D, prior, count):
    """The count chooses the kernel and nothing else."""
    from jaxns_gb300.engine import NSBatch
    spec = _spec(oracle_mod, D, 6, 1, prior, True, n=64)
    b = NSBatch([spec] * 3, device="cuda")
    b._b.lane_chains = b._b.warp_chains = count
    _shell(oracle_mod, b, spec, 3)


def _shell(oracle_mod, b, spec, R):
    b.init()
    b.iterate(3)
    live = b.live_view(0)["log_L_raw"].cpu().numpy()
    at, key = spec.shell_size - 1, oracle_mod.PRNGKey(7)
    b.slice_shell(torch.full((R,), float(live[at])), torch.tensor(key.view(np.int32)).repeat(R, 1))
    torch.cuda.synchronize()
    for r in {0, R - 1}:
        assert_shell_exact(oracle_mod, b, r, live[at], key)
