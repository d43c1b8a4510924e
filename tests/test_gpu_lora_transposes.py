"""Published transposes of adapter matrices are never answered once they are stale."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def mat(*s):
    return torch.nn.Parameter(torch.randn(*s, device="cuda").to(torch.bfloat16))


def right(m):
    return torch.equal(F._lora_transposed(m), m.detach().t())


def test_sets_that_overlap():
    m1, m2 = mat(16, 256), mat(256, 16)
    assert F.prepare_lora_transposes([m1, m2]) == 2 and F.prepare_lora_transposes([m1]) == 1
    with torch.no_grad():
        m1.mul_(2)
        m2.mul_(2)
    F.invalidate_lora_transposes([m1, m2])
    assert right(m1) and right(m2)


@pytest.mark.parametrize("first", ["fp32", "strided"])
def test_first_matrix_outside_every_set(first):
    m0 = mat(16, 64).float() if first == "fp32" else mat(64, 32)[:, ::2]
    m = mat(16, 256)
    assert F.prepare_lora_transposes([m0, m]) == 1
    with torch.no_grad():
        m.mul_(2)
    F.invalidate_lora_transposes([m0, m])
    assert right(m)


def test_matrix_moved_to_another_address():
    m = mat(16, 256)
    old = m.data
    F.prepare_lora_transposes([m])
    m.data = old.clone()
    old.mul_(3)                  # another matrix of that shape at the old address
    assert right(old) and right(m)
    F.prepare_lora_transposes([torch.nn.Parameter(old)])
    assert right(old) and right(m)


def test_prepared_copies_are_used():
    m = mat(16, 256)
    F.prepare_lora_transposes([m])
    assert F._lora_transposed(m).data_ptr() == F._lora_transposed(m).data_ptr() and right(m)
    F.invalidate_lora_transposes([m])
    a, b = F._lora_transposed(m), F._lora_transposed(m)
    assert a.data_ptr() != b.data_ptr()
