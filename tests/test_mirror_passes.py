"""Real transforms of several passes (n >= 2^16): the column pass that stores
mirrored rows conjugated, the row pass with the split in its registers and the
column pass with the merge in its registers.  Every sub-length (2^7 .. 2^10),
the cluster kernel with eight and with four blocks a transform, the two- and the
three-pass plans, and the rows and columns that mirror themselves (bins 0, M/2, M and the middle rows): every output against FP64.  The larger
counts of 2^18 .. 2^21 take the chained launches: two whole panels, a partial
last one, and one transform more than the panels hold.

Tolerance: each of the log2 n levels rounds a handful of times at 2^-24 of a
value whose size is the output's rms, and the errors add as a random walk: a
standard deviation of at most 2^-24 sqrt(4 log2 n) rms.  Eight of them bound
the largest of 2^25 outputs; a wrong or missing partner is off by about 1 rms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(got, want, log2n):
    rms = float(np.sqrt(np.mean(np.abs(want) ** 2)))
    tol = 8 * 2.0 ** -24 * np.sqrt(4 * log2n) * rms
    err = np.abs(got - want)
    assert np.isfinite(got).all()
    assert err.max() <= tol, (int(err.argmax()), float(err.max()), tol)


@pytest.mark.parametrize("log2n,count", [(16, 2), (16, 385), (17, 3), (18, 3), (18, 32), (18, 43), (19, 2), (19, 17), (20, 2), (20, 9), (21, 1), (21, 5), (22, 2), (23, 1), (24, 1), (25, 1)])
def test_forward_and_inverse(torch_cuda, ctx_cache, log2n, count):
    torch, n = torch_cuda, 1 << log2n
    rng = np.random.default_rng(log2n)
    ctx = ctx_cache(n)
    x = rng.uniform(-1, 1, (count, n)).astype(np.float32)
    X = torch.full((count, n // 2 + 1), float("nan"), dtype=torch.complex64, device="cuda")
    ctx.check(ctx.batch("rfwd", n, count, torch.from_numpy(x).cuda(), X))
    some = range(count) if count < 5 else sorted({0, 1, count // 2, count - 2, count - 1})
    assert not torch.isnan(torch.view_as_real(X)).any()
    for f in some:
        check(X[f].cpu().numpy(), 2 * np.fft.rfft(x[f].astype(np.float64)), log2n)
    b = (rng.uniform(-1, 1, (count, n // 2 + 1)) + 1j * rng.uniform(-1, 1, (count, n // 2 + 1))).astype(np.complex64)
    b[:, [0, -1]] = b[:, [0, -1]].real
    y = torch.full((count, n), float("nan"), device="cuda")
    ctx.check(ctx.batch("rinv", n, count, torch.from_numpy(b).cuda(), y))
    assert not torch.isnan(y).any()
    for f in some:
        check(y[f].cpu().numpy(), n * np.fft.irfft(b[f].astype(np.complex128), n), log2n)
