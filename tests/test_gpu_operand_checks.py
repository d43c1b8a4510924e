"""Operands whose sizes do not go together are refused on the host: a kernel that trusted them would read past a tensor."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def mk(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("kv", [(1, 77, 256), (3, 77, 256), (2, 77, 128), (2, 77, 320)])
@pytest.mark.parametrize("grad", [False, True])
def test_cross_attention_refuses_keys_of_another_batch_or_width(kv, grad):
    q, kv = mk(2, 32, 128).requires_grad_(grad), mk(*kv)
    with pytest.raises((RuntimeError, ValueError)):
        F.attention_kv(q, kv, 2)


def test_attention_refuses_keys_of_another_head_count():
    from eridiffusion_b200.ops import _native as N
    q, k = mk(2, 32, 2, 64), mk(1, 32, 2, 64)
    with pytest.raises(ValueError):
        N.ops().attention(q, k, k, 1.0, None, -1)
    with pytest.raises(ValueError):
        N.ops().attention(q, mk(2, 32, 2, 64), mk(2, 48, 2, 64), 1.0, None, -1)


def test_no_keys_at_all_is_the_librarys_answer():
    q = mk(2, 32, 128)
    assert torch.equal(F.attention_kv(q, mk(2, 0, 256), 2),
                       F.R.attention(q.view(2, 32, 2, 64), *(mk(2, 0, 2, 64) for _ in range(2))).reshape(2, 32, 128))
