"""The decode kernel whose CTAs share out the chunks of all heads (csrc/dec.cuh): CTAs that cross heads, heads met by two or more
CTAs, heads of one chunk, heads that are one CTA's alone, more than two heads per SM."""
import numpy as np
import pytest

import oracle_lib as ol
from gpu_util import bf16_from_dev, bf16_problem, bf16_to_dev

pytestmark = pytest.mark.gpu
TOL = 2e-2   # the bf16 bound of the other decode tests


@pytest.mark.parametrize("shape", [(1, 100, 4, 300, 128), (1, 147, 1, 129, 64), (1, 149, 16, 1000, 128), (1, 150, 3, 513, 64), (2, 150, 2, 200, 128), (1, 3, 32, 4000, 128),
                                   (1, 33, 17, 700, 64), (1, 1, 1, 65, 128), (1, 296, 2, 256, 64)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("pe", [ol.PE_NONE, ol.PE_ROPE_INTERLEAVED])
def test_against_oracle(pkg, cuda, shape, pe):
    B, H, Lq, Lk, D = shape
    bits, up = bf16_problem(B, H, Lq, Lk, D, 110)
    q, k, v = (bf16_to_dev(b, cuda) for b in bits)
    want = ol.attention(*up, pe=pe)
    first = None
    for rep in range(2):
        got = bf16_from_dev(pkg.forward(q, k, v, pe=pe))
        assert pkg.last_path() == "tc_decode"
        assert np.abs(got - want).max() <= TOL, np.abs(got - want).max()
        first = got if first is None else first
    assert np.array_equal(first, got)   # the cut does not depend on timing
