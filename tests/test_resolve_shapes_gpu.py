"""The speculative cycle's resolver (a pair of CTAs) against the strict walk of the same stream, at the
sizes where its blocks of 32 moves, its ring of 128 far parts and its helpers (56 moves in flight) begin and
end.  The two form the same energy changes from the same pair energies and differ in the rounding of the
sums alone, so they accept the same moves and reach the same coordinates, bit for bit."""

import numpy as np
import pytest

from epsr_python_translation_b200 import configs
from tests.test_walk_gpu import _box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmol", [2, 31, 32, 33, 56, 57, 127, 129, 193, 700])
def test_resolver_accepts_what_the_walk_accepts(nmol):
    s = configs.c1_water(seed=nmol, nmol=nmol)
    a, b = _box(s, False), _box(s, False)
    for _ in range(3):
        for d in (a, b):
            d.molfit(strict=d is b, rotcycle=False)
            d.check_status()
        x, y = a.download_mc(), b.download_mc()
        assert np.array_equal(x["acc"], y["acc"])
        for k in ("xa", "ya", "za", "xadd", "yadd", "zadd"):
            assert np.array_equal(getattr(a, k).cpu().numpy(), getattr(b, k).cpu().numpy()), k
