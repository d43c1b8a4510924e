"""The op layer's choices follow this module's switches and rules: there is no second copy of either."""
import re
from pathlib import Path

import pytest
import torch

from eridiffusion_b200.ops import _native as N
from eridiffusion_b200.ops import functional as F

SRC = Path(N.__file__).parents[1] / "csrc" / "torch"
FLAG = {n: int(v) for n, v in re.findall(r"k(\w+) = (\d+)", re.search(r"enum Flag : int \{([^}]*)\}", (SRC / "eri_ops.h").read_text()).group(1))}
SHIFT = int(re.search(r"kFewTilesShift = (\d+)", (SRC / "eri_ops.h").read_text()).group(1))


@pytest.mark.parametrize("switch,flag", [("_RANK_STREAM", "RankStream"), ("_GEMM_PAIR", "Pair"), ("_GEMM_GROUP", "Group"),
                                         ("_WGRAD_NATIVE", "Wgrad"), ("_ACCUM_INTO_GRAD", "AccumGrad")])
def test_switches(monkeypatch, switch, flag):
    for on in (False, True):
        monkeypatch.setattr(F, switch, on)
        assert bool(F._flags() & FLAG[flag]) == on


@pytest.mark.parametrize("tiles", [0, 7, 36, 1000])
def test_tile_limit(monkeypatch, tiles):
    monkeypatch.setattr(F, "_PAIR_MIN_TILES", tiles)
    assert F._flags() >> SHIFT == tiles and max(FLAG.values()) < 1 << SHIFT


def test_activation_rule(monkeypatch):
    x, w = torch.empty(1, device="meta").expand(1, 4096, 3072), torch.empty(1, device="meta").expand(12288, 3072)
    assert F._flags(x, w, "gelu") & FLAG["ActOutside"] and not F._flags(x, w, None) & FLAG["ActOutside"]
    assert not F._flags(x[:, :512], w, "gelu") & FLAG["ActOutside"]
    monkeypatch.setattr(F, "_ACT_EPILOGUE", True)
    assert not F._flags(x, w, "gelu") & FLAG["ActOutside"]


def test_no_second_copy():
    src = "".join(f.read_text() for f in SRC.glob("*.cpp"))
    assert "getenv" not in src
