"""GPU: the self-test of the bounded waits reaches every kind of wait that the kernels use, and
gives the context's pivot record back."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_every_kind_of_wait_runs_out(hs, ctx):
    lib = hs._lib.load()
    ctx.set_problem(128, 128)
    A = torch.eye(128, dtype=torch.float64, device="cuda:0").reshape(-1)
    A[5 * 129] = -1.0
    ctx.take_info()
    hs.MatrixOperations.cholesky(ctx, A, 0, 0)
    st = lib.hs_selftest_bounded_wait(ctx.handle, 20_000_000)
    text = lib.hs_last_error().decode()
    assert hs._lib.STATUS_NAMES[st] == "HS_ERR_TIMEOUT", text
    for kind in ("thread_wait", "warp_wait", "suspended_wait", "suspended_wait_warp", "warp_count", "warp_pairs",
                 "mbar_wait_for"):
        assert kind in text
    assert ctx.take_info() == 5
    assert ctx.take_info() == -1


def test_copies_in_flight_are_waited_for_after_an_expiry(hs, ctx):
    """A CTA that gives up must not leave while a copy still writes its shared memory: the wait
    for it ignores the failure mark, and has a limit of its own."""
    lib = hs._lib.load()
    ctx.set_problem(128, 128)
    assert hs._lib.STATUS_NAMES[lib.hs_selftest_bounded_wait(ctx.handle, 5_000_000)] == "HS_ERR_TIMEOUT"
    assert "landed" in lib.hs_last_error().decode()


def test_limit_counts_from_when_every_cta_is_resident(hs, ctx):
    """A sweep is no cooperative launch: while other streams' kernels hold SMs that it still
    needs, its CTAs wait on; once all are resident the limit counts."""
    lib = hs._lib.load()
    ctx.set_problem(128, 128)
    assert hs._lib.STATUS_NAMES[lib.hs_selftest_bounded_wait(ctx.handle, 100_000_000)] == "HS_ERR_TIMEOUT"
    text = lib.hs_last_error().decode()
    assert "absent CTAs" in text and "all CTAs" in text
