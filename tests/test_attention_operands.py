"""Attention on keys and values that do not go with the queries: never by a kernel, which takes their sizes from them."""
import pytest
import torch

from dart_pytorch_b200 import ops
from dart_pytorch_b200.ops import flash as A

B, H, Sq, hd = 2, 4, 5, 16
OTHERS = {"value_rows": ((2, 2, 7, 16), (2, 2, 3, 16)), "value_heads": ((2, 2, 7, 16), (2, 1, 7, 16)),
          "batch": ((1, 2, 7, 16), (1, 2, 7, 16)), "larger_batch": ((3, 2, 7, 16), (3, 2, 7, 16)),
          "head_size": ((2, 2, 7, 8), (2, 2, 7, 8)), "narrow_values": ((2, 2, 7, 16), (2, 2, 7, 8)),
          "wide_values": ((2, 2, 7, 16), (2, 2, 7, 24))}


@pytest.fixture
def calls(monkeypatch):
    seen = []
    monkeypatch.setattr(A, "attn_f32", lambda *a, **k: seen.append("kernel"))
    monkeypatch.setattr(A, "_attention_composed", lambda q, k, v, *a: (seen.append("composed"), q)[1])
    return seen


@pytest.mark.parametrize("name", sorted(OTHERS))
@pytest.mark.parametrize("grad", [True, False])
def test_other_shapes(calls, name, grad):
    k, v = (torch.randn(s) for s in OTHERS[name])
    A.attention_bhsd(torch.randn(B, H, Sq, hd, requires_grad=grad), k, v, True)
    assert calls == ["composed"]


def test_other_devices_and_types(calls):
    q = torch.randn(B, H, Sq, hd)
    for t in (torch.empty(2, 2, 7, 16, device="meta"), torch.randn(2, 2, 7, 16).double(), torch.zeros(2, 2, 7, 16, dtype=torch.long)):
        A.attention_bhsd(q, t, t, True)
        A.attention_bhsd(q, q[:, :2], t[:, :, :Sq], True)
    assert calls == ["composed"] * 6
    calls.clear()
    for t in (torch.randn(2, 2, 7, 16), torch.randn(2, 2, 7, 16).bfloat16()):
        A.attention_bhsd(q, t, t, True)
    assert calls == ["kernel"] * 2


def test_bf16_rows_of_another_width(monkeypatch):
    """Heads that are no kernel size of their own: rows of another width than the heads take up are refused."""
    seen = []
    monkeypatch.setattr(A, "attn_fwd", lambda q, *a, **k: (seen.append(1), (q, None))[1])

    def rows(n, width):
        return torch.zeros(n, width, dtype=torch.bfloat16)
    with torch.no_grad():
        for widths in ((4 * 24, 2 * 16, 2 * 24), (4 * 24, 2 * 24, 2 * 32), (4 * 16, 2 * 24, 2 * 24), (4 * 32, 2 * 24, 2 * 24)):
            with pytest.raises(RuntimeError):
                A.attention_tokens(rows(10, widths[0]), rows(14, widths[1]), rows(14, widths[2]), 2, 5, 7, 4, 2, 24, False)
        assert not seen
        A.attention_tokens(rows(10, 96), rows(14, 48), rows(14, 48), 2, 5, 7, 4, 2, 24, False)
        assert seen == [1]


@pytest.mark.gpu
@pytest.mark.parametrize("dv", [8, 64, 80])
def test_values_of_another_size(dv):
    q, k, v = (torch.randn(n, d, device="cuda", requires_grad=True) for n, d in ((9, 64), (33, 64), (33, dv)))
    o = ops.sdpa(q, k, v)
    do = torch.randn(9, dv, device="cuda")
    got = (o, *torch.autograd.grad(o, (q, k, v), do))
    d = [t.detach().double().requires_grad_(True) for t in (q, k, v)]
    ref = (d[0] @ d[1].t() / 8.0).softmax(-1) @ d[2]
    want = (ref, *torch.autograd.grad(ref, d, do.double()))
    for a, b in zip(got, want):      # (sums of up to 80 terms, two of them in a row for the gradients)
        assert a.shape == b.shape and float((a.double() - b).norm().detach() / b.norm().detach()) < 3e-6


@pytest.mark.gpu
def test_operands_that_do_not_go_together_are_refused():
    q = torch.randn(B, H, Sq, hd, device="cuda")
    for name in ("value_rows", "value_heads", "batch", "head_size"):
        k, v = (torch.randn(s, device="cuda") for s in OTHERS[name])
        with pytest.raises((ValueError, IndexError)):
            A.attention_bhsd(q, k, v, False)
