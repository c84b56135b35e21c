"""Calls one after the other on one stream, each reading what the one before
wrote a moment ago, with the input changed between rounds: kernels start before
the one ahead is done and must still read its results.  Row segments that are not
aligned for pairs and rows read twice, through the cached loads; steps of the
chained and queued passes.  Against the same calls with the stream waited for."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real,log2n,count,columns", [
    (False, 9, 301, True), (False, 12, 33, True), (True, 10, 301, True), (True, 13, 35, True),
    (True, 5, 2001, False), (True, 7, 1001, False), (True, 15, 31, False), (False, 18, 50, False), (True, 19, 17, False),
    (False, 22, 3, False),
])
def test_rounds(torch_cuda, ctx_cache, real, log2n, count, columns):
    torch, n = torch_cuda, 1 << log2n
    ctx = ctx_cache(1 << 22)
    g = torch.Generator(device="cuda")
    g.manual_seed(log2n + count)
    x0 = torch.rand((4, count * n, 1 if real else 2), generator=g, device="cuda") * 2 - 1
    bins = n // 2 + 1 if real else n
    x = torch.empty_like(x0[0])
    X = torch.zeros((count * bins, 2), device="cuda")
    out = torch.empty((8,) + x.shape, device="cuda")
    kinds = ("rfwd", "rinv") if real else ("cfwd", "cinv")
    s = torch.cuda.Stream()

    def rounds(wait):
        out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            for i in range(8):
                x.copy_(x0[i % 4])
                for kind, a, b in ((kinds[0], x, X), (kinds[1], X, out[i])):
                    if columns:
                        ctx.check(ctx.strided(kind, n, count, a, count, 1, b, count, 1, s))
                    else:
                        ctx.check(ctx.batch(kind, n, count, a, b, s))
                    if wait:
                        s.synchronize()
        torch.cuda.synchronize()
        return out.view(torch.int32).clone()

    want = rounds(True)
    for _ in range(3):
        assert torch.equal(rounds(False), want)
