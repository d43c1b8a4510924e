"""A header that the op layer includes is part of its rebuild digest: both libraries share argument structs, and one side
built against an older layout would pass wrong strides."""
import re

from eridiffusion_b200.csrc import build


def test_every_included_header_is_in_the_digest():
    seen, todo = set(), list((build.CSRC / "torch").glob("*.cpp"))
    while todo:
        f = todo.pop()
        for inc in re.findall(r'#include "([^"]+)"', f.read_text()):
            h = (f.parent / inc).resolve()
            if h not in seen:
                seen.add(h)
                todo.append(h)
    assert {"attn_args.h", "gemm_args.h", "eri_ops.h"} <= {h.name for h in seen}
    assert seen <= {h.resolve() for h in build.torch_headers()}
