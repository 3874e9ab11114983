"""flash_forward_host sends its last chunk in pieces: every split of the heads gives the bits of one call on all heads that
lie on the device, and the pieces land where they belong."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,n,d,chunk,causal,wl",
                         [(1, 8192, 128, 1, True, -1),     # one head: nothing to take apart
                          (2, 8192, 128, 2, True, -1),     # pieces of exactly 2 MiB a tensor
                          (2, 8191, 128, 2, True, -1),     # just below: whole
                          (5, 8200, 64, 5, False, -1),     # 3 heads and 2
                          (7, 8200, 128, 7, True, 300),    # 4, 2, 1
                          (3, 16384, 64, 8, True, -1),     # fewer heads than a chunk may have
                          (19, 4100, 128, 8, True, -1),    # the last chunk is short
                          (24, 4096, 128, 8, False, -1),   # three whole chunks: slots used again
                          (40, 333, 128, 40, True, -1)])   # small heads
def test_host_call_equals_the_device_call(pkg, heads, n, d, chunk, causal, wl):
    import torch

    nbytes = pkg.lib().flash_forward_host_workspace_bytes(n, d, chunk)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    g = torch.Generator()
    for turn in range(2):  # the second call must not see what the first left in the workspace
        g.manual_seed(10 * n + turn)
        q, k, v = (torch.randn(1, heads, n, d, generator=g).half().pin_memory() for _ in range(3))
        out = torch.full_like(q, float("nan")).pin_memory()
        pkg.flash_forward_host(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), 1, heads, n, d, ws.data_ptr(),
                               nbytes, chunk_heads=chunk, is_causal=causal, window_left=wl)
        want = pkg.attention_forward(q.cuda(), k.cuda(), v.cuda(), causal=causal, window_left=wl)
        assert torch.equal(out, want.cpu())
