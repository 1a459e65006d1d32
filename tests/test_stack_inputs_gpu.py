"""What the native stack call is given: cache buffers that start anywhere, and whatever stands before it in a CUDA graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import dart_pytorch_b200 as dp
from dart_pytorch_b200.nn.attention import EncoderCache
from dart_pytorch_b200.nn.transformer import TransformerEncoder


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hd", [32, 96])
@pytest.mark.parametrize("offset", [0, 1, 8])
def test_cache_buffers_start_anywhere(dtype, hd, offset):
    m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=64, embed_dim=2 * hd, num_layers=2, num_heads=2, device="cuda", dtype=dtype,
                            init_std=0.2)).eval()
    toks = torch.randint(0, 97, (2, 9), device="cuda")

    def steps(cache):
        with torch.no_grad():
            return torch.cat([m.hidden(toks[:, :7], 0, cache)] + [m.hidden(toks[:, i:i + 1], i, cache) for i in (7, 8)], 1)
    want, cache = steps(EncoderCache.empty(2, 2)), EncoderCache.empty(2, 2)
    for c in cache.layers:
        c.k_buf, c.v_buf = (torch.zeros(2 * 128 * 2 * hd + offset, device="cuda", dtype=dtype)[offset:].view(2, 128, 2 * hd)
                            for _ in range(2))
    got = steps(cache)
    # the same sums, by other kernels where the rows do not start on 16 bytes
    assert float((got - want).float().norm() / want.float().norm()) < (2e-2 if dtype == torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("before", ["nothing", "fill", "copy", "join"])
def test_recorded_behind_other_work(dtype, before):
    """A short stack starts as a programmatic dependent of what was recorded before it, which need not be a kernel."""
    enc = TransformerEncoder(2, 128, 2, device="cuda", dtype=dtype).eval()
    src, x = torch.randn(5, 128, device="cuda").to(dtype), torch.zeros(5, 128, device="cuda", dtype=dtype)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()

    def body():
        if before == "fill":
            x.zero_()
        elif before == "copy":
            x.copy_(src)
        elif before == "join":
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                x.copy_(src)
                x.mul_(2.0)
            torch.cuda.current_stream().wait_stream(side)
        return enc(x)
    with torch.no_grad():
        body()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            out = body()
        for _ in range(3):
            src.copy_(torch.randn(5, 128, device="cuda"))
            if before == "nothing":
                x.copy_(src)
            graph.replay()
            torch.cuda.synchronize()
            got = out.clone()
            assert torch.equal(got, enc({"nothing": src, "fill": torch.zeros_like(src), "copy": src, "join": src * 2.0}[before]))
