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


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("name,shape", [("weight", (56,)), ("bias", (56,)), ("pre_c", (8,)), ("pre_c", (1, 128)), ("pre_nc", (2, 56)),
                                        ("pre_nc", (3, 64)), ("pre_nc", (128,)), ("pre_nc", (1, 128))])
def test_group_norm_refuses_addends_of_another_size(grad, name, shape):
    kw = dict(weight=mk(64), bias=mk(64))
    kw[name] = mk(*shape)
    with pytest.raises(ValueError):
        F.group_norm_silu(mk(2, 64, 16, 4).contiguous(memory_format=torch.channels_last).requires_grad_(grad), groups=8, **kw)


@pytest.mark.parametrize("name", ["bias", "bias2"])
def test_add_bias_refuses_a_bias_of_another_size(name):
    with pytest.raises(ValueError):
        F.add_bias(mk(2, 16, 64), mk(2, 16, 64), **{name: mk(56)})


def test_one_embedding_for_every_sample():
    """[1, C] adds the same embedding to every sample, as a broadcast sum did, and its gradient is the sum over them."""
    x, w, b, emb = mk(3, 64, 4, 4).contiguous(memory_format=torch.channels_last), mk(64), mk(64), mk(1, 64).requires_grad_()
    wide = emb.detach().expand(3, 64).contiguous().requires_grad_()
    dy = mk(3, 64, 4, 4)
    y, z = F.group_norm_silu(x, w, b, 8, pre_nc=emb), F.group_norm_silu(x, w, b, 8, pre_nc=wide)
    y.backward(dy)
    z.backward(dy)
    assert torch.equal(y, z) and emb.grad.shape == (1, 64)
    want = wide.grad.double().sum(0, keepdim=True)
    # three bf16 values added and rounded once: 2^-8 of the largest partial sum
    assert (emb.grad.double() - want).abs().max() <= 2.0 ** -8 * wide.grad.double().abs().sum(0).max()


@pytest.mark.parametrize("n,hw", [(0, 16), (2, 0)])
@pytest.mark.parametrize("grad", [False, True])
def test_group_norm_of_nothing_is_an_error(n, hw, grad):
    with pytest.raises(RuntimeError):
        F.group_norm_silu(mk(n, hw, 64).requires_grad_(grad), mk(64), mk(64), 8)


@pytest.mark.parametrize("buffers", [False, True])
def test_linear_without_rows_has_zero_gradients(buffers):
    x, w, b = mk(2, 0, 64).requires_grad_(), mk(256, 64).requires_grad_(), mk(256).requires_grad_()
    if buffers:
        w.grad, b.grad = torch.ones_like(w), torch.ones_like(b)
    F.linear(x, w, b).backward(mk(2, 0, 256))
    assert x.grad.shape == x.shape and all((p.grad == (1 if buffers else 0)).all() for p in (w, b))
