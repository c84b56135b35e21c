"""Memory of the stream-ordered pool behind multi-pass calls: what lies idle is
bounded however many streams a process uses (with the bound set low, in a process
of its own), captures work beyond it, the last context gives everything back,
and a server request that needs the memory gets it."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HEAD = f"""
import sys, time, torch
sys.path.insert(0, {ROOT!r})
from ckfft_gb300 import binding
free = lambda: torch.cuda.mem_get_info()[0] >> 20
n, count = 1 << 20, 32                        # 256 MiB of intermediates a call
x = torch.randn((count, n), dtype=torch.complex64, device="cuda")
ctx = binding.Context(n)
want = torch.empty_like(x)
ctx.check(ctx.batch("cfwd", n, count, x, want))         # (blocking: a lane's scratch, not the pool's)
y = torch.empty_like(x)
bits = lambda t: torch.view_as_real(t).view(torch.int32)
def spread(streams):
    for s in streams:                         # each call is done long before the next, but nobody waits for it
        ctx.check(ctx.batch("cfwd", n, count, x, y, s))
        time.sleep(0.005)
"""

BOUNDED = HEAD + """
streams = [torch.cuda.Stream() for _ in range(16)]
torch.cuda.synchronize()
spread(streams[:1])
before = free()
for _ in range(3):
    spread(streams)
held = before - free()
assert held <= 512, held                      # 512 MiB idle, one block of which was there before
# two streams at once, far more often than the bound lets them keep blocks
outs = [torch.empty_like(x) for _ in range(8)]
for _ in range(6):
    for s, o in zip(streams, outs):
        ctx.check(ctx.batch("cfwd", n, count, x, o, s))
torch.cuda.synchronize()
assert all(torch.equal(bits(o), bits(want)) for o in outs)
# a capture while the pool is over its bound
g = torch.cuda.CUDAGraph()
y.zero_()
torch.cuda.synchronize()
with torch.cuda.graph(g, stream=streams[0]):
    ctx.check(ctx.batch("cfwd", n, count, x, y, streams[0]))
g.replay()
torch.cuda.synchronize()
assert torch.equal(bits(y), bits(want))
del g
ctx.close()
print("ok")
"""

GIVEN_BACK = HEAD + """
streams = [torch.cuda.Stream() for _ in range(6)]
other = binding.Context(1024)
torch.cuda.synchronize()
before = free()
spread(streams)
torch.cuda.synchronize()
assert before - free() >= 6 * 256, before - free()
ctx.close()
assert before - free() >= 5 * 256, before - free()      # another context is open
other.close()
assert before - free() <= 64, before - free()
print("ok")
"""

SERVER = HEAD + """
streams = [torch.cuda.Stream() for _ in range(12)]
big = torch.zeros((256, n), dtype=torch.complex64, device="cuda")
out = torch.empty_like(big)
server = binding.Server(ctx, scratch_budget_bytes=64 << 20, max_inflight=1, direct_threshold_bytes=0)
torch.cuda.synchronize()
spread(streams)                               # 3 GiB idle in the pool
torch.cuda.synchronize()
# leave 1.5 GiB: less than the request's 2 GiB of intermediates
filler = torch.empty((free() - 1536) << 20, dtype=torch.uint8, device="cuda")
t = server.submit("cfwd", n, 256, big, out)
ok, _ = server.wait(t, 10.0)
del filler
torch.cuda.empty_cache()
if ok != 1:
    server.wait(t, 60.0)
server.close()
assert ok == 1, "the request was not admitted"
print("ok")
"""


@pytest.mark.parametrize("child,env", [(BOUNDED, {"CKFFT_CUDA_POOL_IDLE_MIB": "512"}), (GIVEN_BACK, {}), (SERVER, {})],
                         ids=["bounded", "given_back", "server"])
def test_pool(torch_cuda, child, env):
    torch_cuda.cuda.empty_cache()
    r = subprocess.run([sys.executable, "-c", child], env=dict(os.environ, **env), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
