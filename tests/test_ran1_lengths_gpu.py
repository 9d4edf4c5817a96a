"""ran1 fills on both sides of the length from which three warps make the stream, from a new stream, one under way and
the degenerate seed, against the oracle: values and state."""

import numpy as np
import pytest

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import BoxArrays, Ran1State
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [-7, -2147483647])
@pytest.mark.parametrize("n", [100, 2046, 2047, 2048, 2049, 2080, 4097])
def test_lengths_around_the_three_warps(n, seed):
    from epsr_python_translation_b200.device import DeviceBox
    d = DeviceBox(BoxArrays.from_system(configs.c1_water(seed=1, nmol=4)))
    st = Ran1State(idum=seed)
    t = d.ran1_tensor(st)
    for k in (n, 33, n):
        vals = d.ran1_fill(t, k)
        ref, st = oracle.ran1_fill(st, k)
        assert np.array_equal(vals.cpu().numpy().view(np.uint32), ref.view(np.uint32))
        assert np.array_equal(t.cpu().numpy(), st.as_array())
