"""Large layout calls whose input is page-locked host memory, which the kernels
read in place with plain loads and never with bulk copies: complex 2^17 .. 2^20
must not take the queue kernel, whose column tiles are TMA copies of the input.
A page-locked output, which every kernel stores to, leaves the route as it is."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log2n,count", [("cfwd", 17, 97), ("cinv", 20, 12)])
@pytest.mark.parametrize("host_in,host_out", [(True, False), (True, True), (False, True), (False, False)])
def test_page_locked_sides(torch_cuda, ctx_cache, lib, kind, log2n, count, host_in, host_out):
    torch, n = torch_cuda, 1 << log2n
    lib.ckg_flow_launches.restype = ctypes.c_longlong
    ctx = ctx_cache(1 << 20)
    x = torch.randn((count, n), dtype=torch.complex64, device="cuda")
    want = torch.empty_like(x)
    ctx.check(ctx.batch(kind, n, count, x, want))
    src = x.cpu().pin_memory() if host_in else x
    dst = torch.empty((count, n), dtype=torch.complex64, pin_memory=True) if host_out else torch.empty_like(x)
    before = lib.ckg_flow_launches()
    ctx.check(ctx.strided(kind, n, count, src, 1, n, dst, 1, n))
    assert lib.ckg_flow_launches() - before == (0 if host_in else 1)
    assert torch.equal(torch.view_as_real(dst).cpu().view(torch.int32), torch.view_as_real(want).cpu().view(torch.int32))
