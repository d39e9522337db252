"""The autotuner's choices at 256: one x sweep, and the number of the second one it once had."""

import pytest
import torch

import oracle as O
import symcode as S
from symcode import autotune as A
from _util import rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu


def test_the_x_sweep_of_256_has_no_choice_and_takes_its_old_number():
    g = S.Grid(3, 256, dtype=torch.float32, device="cuda:0")
    assert A.num_variants(g)[A.SWEEPS.index("x_sweep")] == 1
    u = [to_dev(c, g) for c in O.random_field(O.Grid(3, 256), seed=50, kpeak=4)]
    out = []
    for v in (0, 1):
        A.set_variants(g, {"x_sweep": v})
        out.append([to_np(c) for c in S.convectiondiffusion_(S.vectorfield(g), u, g, 1e-3)])
    assert rel_l2(out[1], out[0]) == 0.0
    with pytest.raises(S.SymcodeError):
        A.set_variants(g, {"x_sweep": 2})
    g.close()
