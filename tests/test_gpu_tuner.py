"""The choice of the FP32 stage kernel: timed again and again on a small grid, where its launches are as short as the gaps
between them, it comes out the same, on the context's own stream and on the caller's."""
import pytest

from dfdm import serve
from dfdm.native import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["tgv", "channel"])
def test_the_choice_repeats(kind):
    import torch
    c = serve.serve_case(kind, 32, 800.0, 1)
    with Solver(c, "fp32") as s:
        first = s.stage_variant()[0]
        for stream in (None, torch.cuda.Stream()):
            if stream is not None:
                s.set_stream(stream.cuda_stream)
            for _ in range(8):
                s.set_stage_variant(-1)
                v, one, pairs = s.stage_variant()
                assert v == first == (1 if pairs < one else 0), (one, pairs)
