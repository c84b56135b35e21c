"""Layouts that are distance 1 on both sides (fft_columns.cu and, next to its
range, fft_inter.cu) give the bits of the same transforms in a contiguous
batch: every size of the rule and one beyond each end, counts around a tile
and far from one, even and odd strides, padded rows, bases off by a value."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(k, l) for k in ("cfwd", "cinv") for l in (7, 8, 9, 10, 11, 12, 13)]
SIZES += [(k, l) for k in ("rfwd", "rinv") for l in (8, 9, 10, 11, 12, 13, 14)]


@pytest.mark.parametrize("kind,log2n", SIZES)
@pytest.mark.parametrize("count,pad_in,pad_out,off_in,off_out", [
    (48, 0, 0, 0, 0), (2, 0, 0, 0, 0), (17, 0, 0, 0, 0), (37, 1, 2, 0, 0), (64, 4, 6, 0, 1), (33, 3, 1, 1, 0), (8, 1, 0, 1, 1),
])
def test_matches_contiguous(torch_cuda, kind, log2n, count, pad_in, pad_out, off_in, off_out):
    torch = torch_cuda
    from ckfft_gb300 import binding

    n = 1 << log2n
    rows_in = n // 2 + 1 if kind == "rinv" else n
    rows_out = n // 2 + 1 if kind == "rfwd" else n
    tin = torch.float32 if kind == "rfwd" else torch.complex64
    tout = torch.float32 if kind == "rinv" else torch.complex64
    si, so = count + pad_in, count + pad_out
    g = torch.Generator(device="cuda")
    g.manual_seed(n + count)
    x = torch.empty((count, rows_in), dtype=tin, device="cuda")
    r = torch.rand((count, rows_in, 1 if tin == torch.float32 else 2), generator=g, device="cuda") * 2 - 1
    x.copy_(r[..., 0] if tin == torch.float32 else torch.view_as_complex(r))
    a = torch.zeros(off_in + rows_in * si, dtype=tin, device="cuda")
    a[off_in:].view(rows_in, si)[:, :count] = x.t()
    b = torch.zeros(off_out + rows_out * so + 8, dtype=tout, device="cuda")
    want = torch.empty((count, rows_out), dtype=tout, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx = binding.Context(n)
    ctx.check(ctx.batch(kind, n, count, x, want, s))
    ctx.check(ctx.strided(kind, n, count, a[off_in:], si, 1, b[off_out:], so, 1, s))
    s.synchronize()
    ctx.close()

    def bits(t):
        t = t.contiguous()
        return (torch.view_as_real(t) if t.is_complex() else t).view(torch.int32)

    got = b[off_out:off_out + rows_out * so].view(rows_out, so)
    assert torch.equal(bits(got[:, :count].t()), bits(want))
    assert not got[:, count:].any() and not b[:off_out].any() and not b[off_out + rows_out * so:].any()
