"""Batches whose output range overlaps the input's, at sizes whose passes otherwise
run as one queue or chain (complex 2^17 .. 2^20, real 2^18 .. 2^21): all inputs of a
group are read before its first output is written, so the results are those of
disjoint buffers, bit for bit."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def flow_launches(lib):
    lib.ckg_flow_launches.restype = ctypes.c_longlong
    return lib.ckg_flow_launches()


@pytest.mark.parametrize("kind,log2n,count", [("cfwd", 17, 99), ("cinv", 18, 50), ("cfwd", 20, 13), ("rfwd", 18, 50),
                                              ("rinv", 19, 17)])
@pytest.mark.parametrize("shift", [3, -3])
def test_overlapping_batch(torch_cuda, ctx_cache, lib, kind, log2n, count, shift):
    torch, n = torch_cuda, 1 << log2n
    ctx = ctx_cache(1 << 20)
    # in 8-byte units: a transform's input and output, and the shift of the output
    ni = n if kind[0] == "c" else n // 2 if kind == "rfwd" else n // 2 + 1
    no = n if kind[0] == "c" else n // 2 if kind == "rinv" else n // 2 + 1
    gap = 3 * max(ni, no) + 2
    g = torch.Generator(device="cuda")
    g.manual_seed(log2n + count)
    buf = torch.rand((gap + count * max(ni, no), 2), generator=g, device="cuda") * 2 - 1
    at_in, at_out = (0, gap) if shift > 0 else (gap, 0)
    src = buf[at_in:at_in + count * ni].clone()
    want = torch.empty((count * no, 2), device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    before = flow_launches(lib)
    ctx.check(ctx.batch(kind, n, count, src, want, s))
    assert flow_launches(lib) - before == (1 if kind[0] == "c" else 0)
    ctx.check(ctx.batch(kind, n, count, buf[at_in:], buf[at_out:], s))
    assert flow_launches(lib) - before == (1 if kind[0] == "c" else 0)
    s.synchronize()
    got = buf[at_out:at_out + count * no]
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
