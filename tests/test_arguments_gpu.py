"""GPU: operands that hold more than a call reads stay accepted, and only the part that the call names is read."""
import pytest
import torch

from gpu_util import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hkv", [2, 8])
def test_caches_and_keys_for_more_sequences_than_q(Hkv):
    from tinytorch_b200 import op
    q = make((2, 8, 1, 64), torch.bfloat16, 71)[0]
    k, v = make((5, Hkv, 300, 64), torch.bfloat16, 72)[0], make((5, Hkv + 1, 310, 64), torch.bfloat16, 73)[0]
    lens = torch.tensor([300, 17, 5, 5, 5], dtype=torch.int32, device="cuda")
    want, _ = op.sdpAttentionDecode(q, k[:2].contiguous(), v[:2, :Hkv, :300].contiguous(), lens[:2].contiguous())
    assert torch.equal(op.sdpAttentionDecode(q, k, v, lens)[0], want)
    q = make((2, 8, 40, 64), torch.bfloat16, 74)[0]
    want, _ = op.sdpAttentionFwd(q, k[:2].contiguous(), v[:2, :Hkv, :300].contiguous())
    assert torch.equal(op.sdpAttentionFwd(q, k, v)[0], want)


def test_lengths_in_pinned_memory():
    from tinytorch_b200 import op
    q, k, v = (make((3, 4, 150, 64), torch.bfloat16, s)[0] for s in (75, 76, 77))
    lens = torch.tensor([150, 20, 3], dtype=torch.int32)
    got, _ = op.sdpAttentionFwd(q, k, v, kvLens=lens.pin_memory())
    assert torch.equal(got, op.sdpAttentionFwd(q, k, v, kvLens=lens.cuda())[0])


def test_bias_with_a_stride():
    from tinytorch_b200 import fused
    x, w = make((40, 64), torch.bfloat16, 78)[0], make((24, 64), torch.bfloat16, 79)[0]
    b = make((24, 3), torch.bfloat16, 80)[0]
    for call in (fused.linear, fused._linear_raw):
        assert torch.equal(call(x, w, b[:, 1]), call(x, w, b[:, 1].contiguous()))
    leaf = b[:, 1].requires_grad_()
    fused.linear(x, w, leaf).float().sum().backward()
    assert torch.equal(leaf.grad, torch.full_like(leaf, 40))
