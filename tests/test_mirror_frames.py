"""Real transforms of one block (n = 2^7 .. 2^15), whose split and merge pass
mirrors between lanes: a frame inside a warp (16 or 32 threads), frames of
several warps, with a last block that is partly empty (its idle threads take part
in the shuffles), and bins and samples that mirror themselves.  Every output
against FP64, and untouched memory behind the last frame.

Tolerance as in test_mirror_passes.py: eight standard deviations of
2^-24 sqrt(4 log2 n) of the outputs' rms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2n", range(7, 16))
@pytest.mark.parametrize("count", [1, 7, 33])
def test_forward_and_inverse(torch_cuda, ctx_cache, log2n, count):
    torch, n = torch_cuda, 1 << log2n
    rng = np.random.default_rng(100 * log2n + count)
    ctx = ctx_cache(n)
    x = rng.uniform(-1, 1, (count, n)).astype(np.float32)
    b = (rng.uniform(-1, 1, (count, n // 2 + 1)) + 1j * rng.uniform(-1, 1, (count, n // 2 + 1))).astype(np.complex64)
    b[:, [0, -1]] = b[:, [0, -1]].real
    X = torch.full((count + 1, n // 2 + 1), 7 + 0j, dtype=torch.complex64, device="cuda")
    y = torch.full((count + 1, n), 7.0, device="cuda")
    ctx.check(ctx.batch("rfwd", n, count, torch.from_numpy(x).cuda(), X))
    ctx.check(ctx.batch("rinv", n, count, torch.from_numpy(b).cuda(), y))
    for got, want in ((X.cpu().numpy(), 2 * np.fft.rfft(x.astype(np.float64))),
                      (y.cpu().numpy(), n * np.fft.irfft(b.astype(np.complex128), n))):
        rms = float(np.sqrt(np.mean(np.abs(want) ** 2)))
        assert (got[count] == 7).all()
        assert np.abs(got[:count] - want).max() <= 8 * 2.0 ** -24 * np.sqrt(4 * log2n) * rms
