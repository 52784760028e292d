"""The give-up path of the kernels' bounded waits (opencnn_b200/csrc/ptx.cuh), which a healthy run
never takes: a test-only kernel (tests/wait_probe.cu) waits on an mbarrier on which, by a host flag,
nobody arrives.  The wait must run out after its limit, set the status word, let the other waiter
of the CTA fall through, and the kernel must return with the context intact - checked by running
the real operator afterwards and comparing it with the oracle bit for bit."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from conftest import wait_probe_lib_path  # noqa: E402
from opencnn_b200 import api  # noqa: E402

pytestmark = pytest.mark.gpu
LIMIT_NS = 2_000_000          # 2 ms per wait


@pytest.fixture(scope="module")
def probe():
    lib = ctypes.CDLL(wait_probe_lib_path())
    lib.wait_probe_run.argtypes = [ctypes.c_int, ctypes.c_ulonglong, ctypes.POINTER(ctypes.c_longlong)]
    lib.wait_probe_last_status.restype = ctypes.c_int
    return lib


def _run(lib, skip_arrive):
    out = (ctypes.c_longlong * 8)()
    assert lib.wait_probe_run(int(skip_arrive), LIMIT_NS, out) == 0
    keys = ("issuer_ok", "waiter_ok", "waiter_second_ok", "drain_ok", "drain_timeout_ok", "issuer_wait_ns",
            "waiter_second_ns", "drain_timeout_ns")
    return dict(zip(keys, list(out)))


def test_healthy_wait_leaves_status_clear(probe):
    r = _run(probe, skip_arrive=False)
    assert r["issuer_ok"] == 1 and r["waiter_ok"] == 1
    assert r["drain_ok"] == 1
    assert r["drain_timeout_ok"] == 1 and r["drain_timeout_ns"] >= LIMIT_NS       # the drain's own limit
    assert probe.wait_probe_last_status() == 0


def test_wait_that_runs_out_sets_status_and_returns(oracle, libs, probe):
    r = _run(probe, skip_arrive=True)
    assert r["issuer_ok"] == 0, "nobody arrived: the wait must give up"
    assert LIMIT_NS <= r["issuer_wait_ns"] < 50 * LIMIT_NS
    assert r["waiter_ok"] == 0, "the second waiter must come back through the CTA's dead word"
    assert r["waiter_second_ok"] == 0 and r["waiter_second_ns"] < LIMIT_NS, "later waits return at once"
    assert r["drain_ok"] == 1 and r["drain_timeout_ok"] == 1
    assert probe.wait_probe_last_status() == 1          # kStatusWaitTimeout
    assert probe.wait_probe_last_status() == 0          # reading resets it
    # the context is intact: the operator runs and is bit-exact
    N, C, K, H, W = 32, 16, 64, 6, 6
    x, g = oracle.input_chwn(N, C, H, W), oracle.filter_crsk(C, K)
    dy = torch.full((K, H, W, N), float("nan"), device="cuda")
    dws = torch.empty((C, 4, 4, K), device="cuda")
    assert api.conv3x3(torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda(), dy, dws, N, C, H, W, K) == 0
    assert api.last_device_status() == 0
    assert np.array_equal(dy.cpu().numpy(), oracle.forward(x, g))


@pytest.mark.parametrize("skip_arrive", [False, True])
def test_wait_that_runs_out_in_one_cta_of_a_pair_ends_the_other(oracle, libs, probe, skip_arrive):
    """A CTA that gave up no longer reports to the pair's leader, so that the leader's wait runs out as well (it must not
    take what was never written for ready); both return, and the operator on CTA pairs still runs."""
    out = (ctypes.c_longlong * 3)()
    assert probe.wait_probe_pair_run(int(skip_arrive), LIMIT_NS, out) == 0
    worker_ok, leader_ok, leader_wait_ns = list(out)
    assert probe.wait_probe_last_status() == int(skip_arrive)
    assert (worker_ok, leader_ok) == ((0, 0) if skip_arrive else (1, 1))
    if skip_arrive:
        assert 4 * LIMIT_NS <= leader_wait_ns < 200 * LIMIT_NS
    N, C, K, H, W = 32, 64, 128, 4, 4
    x, g = oracle.input_int(N, C, H, W), oracle.filter_int(C, K)
    ws, dy = torch.empty((C, 4, 4, K), device="cuda"), torch.full((K, H, W, N), float("nan"), device="cuda")
    assert api.filter_transform(torch.from_numpy(g).cuda(), ws, C, K, precision="bf16") == 0
    assert api.winograd_forward_kernel(torch.from_numpy(x).cuda(), ws, dy, N, C, H, W, K, precision="bf16", kernel="pair_local") == 0
    assert api.last_device_status() == 0
    assert np.array_equal(dy.cpu().numpy().astype(np.float64), oracle.direct_f64(x, g))


@pytest.mark.parametrize("skip_arrive", [False, True])
def test_wait_of_a_whole_warp(probe, skip_arrive):
    """All lanes get the same answer; the wait that nobody ends runs out after its limit, or at once where one before it has."""
    out = (ctypes.c_longlong * 4)()
    assert probe.wait_probe_warp_run(int(skip_arrive), LIMIT_NS, out) == 0
    first_ok, second_ok, first_ns, second_ns = list(out)
    assert probe.wait_probe_last_status() == 1 and probe.wait_probe_last_status() == 0
    assert (first_ok, second_ok) == (0 if skip_arrive else 32, 0)
    waited_ns = first_ns if skip_arrive else second_ns
    assert LIMIT_NS <= waited_ns < 50 * LIMIT_NS
    if skip_arrive:
        assert second_ns < LIMIT_NS
