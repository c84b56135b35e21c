"""The bounded waits of the fused two-pass kernel (fft_flow.cu): a row tile whose
transform's column tiles nobody counts.  The loader, the scheduler, both groups
and the counter warp must each give up, report it and return."""
import pytest

pytestmark = pytest.mark.gpu


def test_queue_that_never_moves_ends_and_reports(torch_cuda, ctx_cache, lib):
    from ckfft_gb300 import binding

    ctx = ctx_cache(1024)
    for _ in range(3):
        assert lib.CkFftCudaSelfTestWait(ctx.handle, 2) == 1, binding.last_error()
    assert lib.CkFftCudaSelfTestWait(ctx.handle, 3) == 0
