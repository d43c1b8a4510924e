"""Every kernel family with bounded waits is among those whose error word training reads."""
import re
from pathlib import Path

import pytest

from eridiffusion_b200.ops import _native as N
from eridiffusion_b200.ops import flash_attn as FA
from eridiffusion_b200.ops import functional as F

FAMILIES = sorted({m for f in Path(N.__file__).parents[1].joinpath("csrc").glob("*.cu")
                   for m in re.findall(r"int eri_(\w+)_check_error\(", f.read_text())} - {"link_probe"})   # (a benchmark's own kernel)


class Fake:
    def __init__(self, failed):
        for f in FAMILIES:
            setattr(self, f"eri_{f}_check_error", lambda v=43 if f == failed else 0: v)


@pytest.mark.parametrize("family", FAMILIES)
def test_a_wait_that_ran_out_is_reported(monkeypatch, family):
    monkeypatch.setattr(N, "require", lambda: Fake(family))
    monkeypatch.setattr(FA, "_bind", lambda lib: None)
    assert F.kernel_error_check() == {family: 43}
    assert (FA.check_error() == 43) == family.startswith("fa")
    assert (F.gemm_error_check() == 43) == (family in ("gemm", "gemm2", "gemm_few"))
