"""fit_expansion against the C oracle, strict sums, bit for bit, at the edges of its cluster and CTA
forms: one worker CTA and many, the row counts where a CTA is added, terms that fill a thread's
registers exactly and spill past them, the wide CTA (more than 256 rows or perturbed terms a
CTA), and a stream that is never clean (the seed whose Park-Miller sequence is zero)."""

import numpy as np
import pytest
import torch

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import Ran1State
from oracle import oracle
from tests.goldens import assert_bits_equal

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.mark.parametrize("npt,nterms,ncfirst,seed", [
    (5, 3, 1, -7), (160, 16, 1, -8), (161, 17, 2, -9), (320, 128, 1, -10), (321, 129, 3, -11), (1120, 24, 1, -12),
    (1121, 20, 1, -13), (2100, 12, 1, -14), (150, 300, 1, -15), (90, 21, 1, -2147483647)])
def test_fit_shapes_match_oracle(npt, nterms, ncfirst, seed):
    _compare(npt, nterms, ncfirst, seed)


@pytest.mark.parametrize("npt,nterms,seed", [(1464, 300, -16), (2432, 200, -17), (3072, 168, -18)])
def test_largest_rows_match_oracle(npt, nterms, seed):
    """Shapes whose rows take nearly all the shared memory of the largest cluster."""
    _compare(npt, nterms, 1, seed)


def _compare(npt, nterms, ncfirst, seed):
    from epsr_python_translation_b200 import transforms
    rng = np.random.default_rng(npt)
    expr = configs.ep_basis(configs.qgrid(npt, 0.05), nterms)
    yin = np.zeros(npt + 1, f32)
    yin[1:] = (rng.standard_normal(npt) * 0.05).astype(f32)
    wtold = np.zeros(nterms + 1, f32)
    wtold[1:] = (rng.standard_normal(nterms) * 0.01).astype(f32)
    st = Ran1State(idum=seed)
    t = torch.from_numpy(st.as_array()).cuda()
    got = transforms.fit_expansion(yin, expr, wtold, f32(0.01), 1, npt, ncfirst, nterms, 1000, 10, t, strict=True)
    ref, after = oracle.fit_expansion(yin, expr, wtold.copy(), f32(0.01), 1, npt, ncfirst, nterms, 1000, 10, st)
    for k in ("wt", "wtold", "yout"):
        assert_bits_equal(got[k].cpu().numpy()[1:], ref[k][1:], k)
    for k in ("stepr", "acceptr", "rejrat", "chisq"):
        assert_bits_equal(got[k], ref[k], k)
    assert got["trials"] == ref["trials"]
    assert np.array_equal(t.cpu().numpy(), after.as_array())
