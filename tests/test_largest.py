"""The largest three-pass sizes (complex to 2^28, real to 2^30): every pair of
sub-lengths beyond the half length 2^24 the other tests reach.

Forward: chosen bins against an FP64 sum over the whole input.  Inverse: every
value of the round trip.  Tolerance as in test_mirror_passes.py: each of the
log2 n levels rounds a handful of times at 2^-24, a standard deviation of at most
2^-24 sqrt(4 log2 n) of the outputs' rms, sqrt(2) times that for the round trip;
eight of them bound the largest of 2^31 values."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(lib):
    from ckfft_gb300 import binding

    c = binding.Context(1 << 30)
    yield c
    c.close()
    gc.collect()


def bins(torch, x, ks):
    """sum_n x[n] W_N^(k n) in FP64: n = B a + b, first over a, then over b."""
    n = x.numel()
    b = 1 << 15
    a = n // b
    k = torch.tensor(ks, device="cuda", dtype=torch.int64)[:, None]
    ia, ib = torch.arange(a, device="cuda"), torch.arange(b, device="cuda")
    unit = lambda num, den: torch.exp(-2j * np.pi * (num % den).double() / den)
    wa, wb = unit(k * ia, a), unit(k * ib, n)
    s = torch.zeros((len(ks), b), dtype=torch.complex128, device="cuda")
    rows = x.view(a, b)
    step = min(a, 1 << 12)
    for r in range(0, a, step):
        s += wa[:, r:r + step] @ rows[r:r + step].to(torch.complex128)
    return (s * wb).sum(1)


@pytest.mark.parametrize("real,log2n", [(False, 26), (False, 28), (True, 27), (True, 29), (True, 30)])
def test_forward_bins_and_round_trip(torch_cuda, ctx, real, log2n):
    torch, n = torch_cuda, 1 << log2n
    g = torch.Generator(device="cuda")
    g.manual_seed(log2n + real)
    x = torch.rand((n, 1 if real else 2), generator=g, device="cuda").mul_(2).sub_(1)
    x = x[:, 0] if real else torch.view_as_complex(x)
    X = torch.full((n // 2 + 1 if real else n,), float("nan"), dtype=torch.complex64, device="cuda")
    y = torch.full_like(x, float("nan"))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx.check(ctx.batch("rfwd" if real else "cfwd", n, 1, x, X, s))
    ctx.check(ctx.batch("rinv" if real else "cinv", n, 1, X, y, s))
    s.synchronize()
    top = n // 2 if real else n - 1
    ks = [0, 1, 1023, 1 << 10, (1 << 20) + 1, n // 2, n // 2 - 1, top, top - 1]
    ks += np.random.default_rng(log2n).integers(0, top, 15).tolist()
    scale = 2 if real else 1
    rms = scale * (n / (3 if real else 1.5)) ** 0.5
    tol = 8 * 2.0 ** -24 * (4 * log2n) ** 0.5
    err = (X[torch.tensor(ks, device="cuda")].to(torch.complex128) - scale * bins(torch, x, ks)).abs()
    assert err.max().item() <= tol * rms, (ks[int(err.argmax())], err.max().item(), tol * rms)
    # in slices: the arrays are up to 4 GiB
    worst = 0.0
    for lo in range(0, n, 1 << 26):
        d = y[lo:lo + (1 << 26)] / (2 * n if real else n) - x[lo:lo + (1 << 26)]
        assert torch.isfinite(torch.view_as_real(d) if not real else d).all()
        worst = max(worst, d.abs().max().item())
    assert worst <= tol * 2 ** 0.5 * (1 / (3 if real else 1.5)) ** 0.5, worst
