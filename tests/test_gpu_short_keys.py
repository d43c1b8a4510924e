"""Key sets shorter than one 128-key tile: the padding bias under graph capture, for more shapes than are kept, and on
several streams."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F
from eridiffusion_b200.ops import reference as R

pytestmark = pytest.mark.gpu


def mk(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16)


def close(o, q, k, v):
    # bf16 probabilities and output: 2^-8 of values of order one
    assert (o.float() - R.attention_fp32(q, k, v)).abs().max().item() < 2.0 ** -6


def test_first_met_while_a_graph_is_captured():
    q, k = mk(1, 64, 2, 64), mk(1, 33, 2, 64)
    F.attention(q, mk(1, 35, 2, 64), mk(1, 35, 2, 64))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        o = F.attention(q, k, k)
    graph.replay()
    close(o, q, k, k)
    close(F.attention(q, k, k), q, k, k)


def test_more_shapes_than_are_kept_on_two_streams():
    q, k = mk(3, 32, 1, 64), mk(3, 127, 1, 64)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    out = []
    for lk in range(20, 120):
        with torch.cuda.stream(streams[lk & 1]):
            out.append((lk, F.attention(q, k[:, :lk].contiguous(), k[:, :lk].contiguous())))
    torch.cuda.synchronize()
    for lk, o in out:
        close(o, q, k[:, :lk], k[:, :lk])
