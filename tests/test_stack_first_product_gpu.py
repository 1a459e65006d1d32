"""A stack that opens with a product (post-norm blocks on given hidden states), right behind a kernel of this package that writes the
product's weight: the product reads what was written."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.models.bert import BertConfig, BertModel
from dart_pytorch_b200.ops import kernels as K
from dart_pytorch_b200.ops import stack


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [1, 8, 23])
def test_weight_written_right_ahead(dtype, rows):
    D = 512
    m = BertModel(BertConfig(vocab_size=50, max_position_embeddings=64, embed_dim=D, num_layers=2, num_heads=8, intermediate_size=1024,
                             device="cuda", dtype=dtype)).eval()
    layers = [stack.Layer(b.attention, b.attention_output_ln, b.output_ln, b.intermediate.weight, b.intermediate.bias, b.output.weight,
                          b.output.bias) for b in m.layers]
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(rows, D, device="cuda", generator=g).to(dtype)
    w = m.layers[0].attention.w_qkv
    factors = [(torch.randn(w.shape[0], 2048, device="cuda", generator=g).to(dtype), (torch.randn(2048, D, device="cuda", generator=g) * 1e-3).to(dtype))
               for _ in range(2)]

    def run(wait):
        outs = []
        with torch.no_grad():
            for i in range(12):
                K.gemm(*factors[i % 2], w.data)
                if wait:
                    torch.cuda.synchronize()
                outs.append(stack.run(layers, x, post_norm=True, act="gelu_tanh"))
                if wait:
                    torch.cuda.synchronize()
        return outs
    want, got = run(True), run(False)
    assert all(o is not None for o in want) and not torch.equal(want[0], want[1])
    for a, b in zip(got, want):
        assert torch.equal(a, b)
