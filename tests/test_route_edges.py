"""Multi-pass batches at the edges of their routes, against the same transforms
one at a time, bit for bit: the cluster kernel's long batches (complex 2^15, four
blocks a transform from 384 on), three-pass and chained batches of more than one
group of 256 MiB of intermediates, and chains on two streams at once."""
import pytest

pytestmark = pytest.mark.gpu


def bits(torch, t):
    return (torch.view_as_real(t) if t.is_complex() else t).contiguous().view(torch.int32)


def make(torch, kind, n, count, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ni, no = (n // 2 + 1 if kind == "rinv" else n), (n // 2 + 1 if kind == "rfwd" else n)
    x = torch.rand((count, ni, 1 if kind == "rfwd" else 2), generator=g, device="cuda") * 2 - 1
    x = x[..., 0] if kind == "rfwd" else torch.view_as_complex(x)
    return x, torch.zeros((count, no), dtype=torch.float32 if kind == "rinv" else torch.complex64, device="cuda")


def check_singles(torch, ctx, kind, n, x, y, stream):
    count = x.shape[0]
    one = torch.empty_like(y[0])
    for f in sorted({0, 1, count // 2, count - 2, count - 1} & set(range(count))):
        ctx.check(ctx.batch(kind, n, 1, x[f], one, stream))
        stream.synchronize()
        assert torch.equal(bits(torch, one), bits(torch, y[f])), (kind, n, count, f)


@pytest.mark.parametrize("kind", ["cfwd", "cinv"])
@pytest.mark.parametrize("count", [383, 384, 601])
def test_long_cluster_batches(torch_cuda, ctx_cache, kind, count):
    torch, n = torch_cuda, 1 << 15
    ctx = ctx_cache(1 << 23)
    x, y = make(torch, kind, n, count, count)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx.check(ctx.batch(kind, n, count, x, y, s))
    s.synchronize()
    check_singles(torch, ctx, kind, n, x, y, s)


@pytest.mark.parametrize("kind,log2n,count", [("cfwd", 22, 9), ("cinv", 22, 9), ("rfwd", 23, 9), ("rinv", 23, 9),
                                              ("rfwd", 20, 65), ("rinv", 20, 67)])
def test_two_groups(torch_cuda, ctx_cache, kind, log2n, count):
    torch, n = torch_cuda, 1 << log2n
    ctx = ctx_cache(1 << 23)
    x, y = make(torch, kind, n, count, log2n)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx.check(ctx.batch(kind, n, count, x, y, s))
    s.synchronize()
    check_singles(torch, ctx, kind, n, x, y, s)


@pytest.mark.parametrize("log2n,kinds", [(18, ("rfwd", "rinv")), (21, ("rfwd", "rinv")), (22, ("cfwd", "cinv")),
                                         (23, ("rfwd", "rinv"))])
def test_two_streams(torch_cuda, ctx_cache, log2n, kinds):
    torch, n = torch_cuda, 1 << log2n
    ctx = ctx_cache(1 << 23)
    count = max(2, (1 << 24) >> log2n)
    work = [(k, *make(torch, k, n, count, i)) for i, k in enumerate(kinds)]
    want = []
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for k, x, y in work:
        ctx.check(ctx.batch(k, n, count, x, y, s[0]))
        s[0].synchronize()
        check_singles(torch, ctx, k, n, x, y, s[0])
        want.append(y.clone())
    got = [[torch.zeros_like(w) for _ in range(4)] for w in want]
    torch.cuda.synchronize()
    for r in range(4):
        for i, (k, x, _) in enumerate(work):
            ctx.check(ctx.batch(k, n, count, x, got[i][r], s[i]))
    torch.cuda.synchronize()
    for w, outs in zip(want, got):
        for o in outs:
            assert torch.equal(bits(torch, o), bits(torch, w))


@pytest.mark.parametrize("log2n,count,offset,in_dist,out_pad,queued", [
    (17, 95, 0, 0, 0, 0), (17, 96, 0, 0, 0, 1), (20, 11, 0, 0, 0, 0), (20, 12, 0, 0, 0, 1), (16, 400, 0, 0, 0, 0), (21, 8, 0, 0, 0, 0),
    (17, 300, 0, 0, 0, 1),                                   # groups of 256 and 44
    (17, 99, 1, 0, 0, 0), (17, 99, 0, 1, 0, 0),              # off 16 bytes: the base, the distance
    (17, 99, 0, 2, 0, 1), (17, 99, 0, 0, 3, 1), (18, 49, 0, 2 - (1 << 18), 0, 0),
])
def test_which_calls_are_queued(torch_cuda, ctx_cache, lib, log2n, count, offset, in_dist, out_pad, queued):
    """The batches the queue kernel takes (in_dist: beyond the size) and those it turns away."""
    import ctypes

    torch, n = torch_cuda, 1 << log2n
    lib.ckg_flow_launches.restype = ctypes.c_longlong
    ctx = ctx_cache(1 << 23)
    x = torch.zeros(offset + (count - 1) * (n + in_dist) + n, dtype=torch.complex64, device="cuda")[offset:]
    y = torch.zeros(count * (n + out_pad), dtype=torch.complex64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    before = lib.ckg_flow_launches()
    ctx.check(ctx.strided("cfwd", n, count, x, 1, n + in_dist, y, 1, n + out_pad, s))
    s.synchronize()
    assert lib.ckg_flow_launches() - before == queued
