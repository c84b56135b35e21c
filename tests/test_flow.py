"""Batches large enough for the fused two-pass kernel (fft_flow.cu) give the
bits of the same transforms run one at a time (the passes as launches of their
own, which the parity tests hold to the oracle), in every form the rule lets in
or turns away: sizes, kinds, odd counts, groups, bases that are not 16-byte
aligned, padded and overlapping frames."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(t):
    import torch

    return (torch.view_as_real(t) if t.is_complex() else t).contiguous().view(torch.int32)


def _run(torch, kind, n, count, offset, pad_in, pad_out, overlap=False):
    from ckfft_gb300 import binding

    ni = no = n
    di = 2 if overlap else ni + pad_in
    do = no + pad_out
    g = torch.Generator(device="cuda")
    g.manual_seed(7 * n + count)
    raw = torch.rand(2 * (offset + (count - 1) * di + ni), generator=g, device="cuda") * 2 - 1
    x = torch.view_as_complex(raw.view(-1, 2))[offset:]
    y = torch.zeros(offset + count * do, dtype=torch.complex64, device="cuda")[offset:]
    one = torch.zeros(no, dtype=torch.complex64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx = binding.Context(n)
    ctx.check(ctx.strided(kind, n, count, x, 1, di, y, 1, do, s))
    picks = sorted({0, 1, count // 2, count - 2, count - 1} & set(range(count)))
    for f in picks:
        src = x[f * di:f * di + ni].clone()
        torch.cuda.synchronize()
        ctx.check(ctx.batch(kind, n, 1, src, one, s))
        s.synchronize()
        got = y[f * do:f * do + no]
        assert torch.equal(_bits(got), _bits(one)), (kind, n, count, f)
        if pad_out:
            assert not y[f * do + no:(f + 1) * do].any(), "padding was written"
    s.synchronize()
    ctx.close()


# both sides of the size the rule starts at, odd counts, more than one group of
# 256 MiB of intermediates (2^17 x 300: 256 and 44, the second group below it)
@pytest.mark.parametrize("kind,log2n,count", [
    ("cfwd", 17, 95), ("cfwd", 17, 97), ("cinv", 17, 300), ("cfwd", 18, 49), ("cinv", 18, 47), ("cfwd", 19, 25),
    ("cinv", 19, 24), ("cfwd", 20, 13), ("cinv", 20, 12), ("cfwd", 20, 41),
])
def test_matches_single_transforms(torch_cuda, kind, log2n, count):
    _run(torch_cuda, kind, 1 << log2n, count, 0, 0, 0)


@pytest.mark.parametrize("kind,log2n,count", [("cfwd", 17, 99), ("cinv", 20, 13)])
@pytest.mark.parametrize("offset,pad_in,pad_out", [(1, 0, 0), (0, 2, 1), (0, 1, 0), (0, 0, 3)])
def test_alignment_and_padding(torch_cuda, kind, log2n, count, offset, pad_in, pad_out):
    _run(torch_cuda, kind, 1 << log2n, count, offset, pad_in, pad_out)


def test_overlapping_frames(torch_cuda):
    _run(torch_cuda, "cfwd", 1 << 18, 49, 0, 0, 0, overlap=True)


def test_two_streams(torch_cuda):
    """Two large batches in flight at once, each with its own intermediates and counters."""
    torch = torch_cuda
    from ckfft_gb300 import binding

    n, count = 1 << 18, 50
    x = [torch.randn(count, n, dtype=torch.complex64, device="cuda") for _ in range(2)]
    ref = [torch.empty_like(v) for v in x]
    got = [torch.empty_like(v) for v in x]
    streams = [torch.cuda.Stream() for _ in x]
    torch.cuda.synchronize()
    ctx = binding.Context(n)
    for i in range(2):
        ctx.check(ctx.batch("cfwd", n, count, x[i], ref[i]))
    for _ in range(5):
        for i in range(2):
            ctx.check(ctx.batch("cfwd", n, count, x[i], got[i], streams[i]))
    torch.cuda.synchronize()
    for i in range(2):
        assert torch.equal(_bits(got[i]), _bits(ref[i]))
        want = np.fft.fft(x[i][count - 1].cpu().numpy().astype(np.complex128))
        d = got[i][count - 1].cpu().numpy() - want
        assert np.linalg.norm(d) <= 1e-6 * np.linalg.norm(want)
    ctx.close()
