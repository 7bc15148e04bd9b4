"""Fields written and read back: one piece, and several pieces of whole planes."""
import numpy as np
import pytest

import cloverleaf3d_ref_b200 as C
import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [C.PRECISION_FP64, C.PRECISION_MIXED])
@pytest.mark.parametrize("n", [(5, 3, 4), (203, 190, 118)])
def test_written_field_comes_back(n, precision):
    ch = C.Chunk(decks.to_deck(decks.shock(*n, 4)), precision)
    rng = np.random.default_rng(7)
    for name in ("density0", "energy0", "xvel0", "vol_flux_x", "vol_flux_y", "mass_flux_z"):
        a = np.asfortranarray(rng.standard_normal(C.field_shape(name, *n)))
        ch.set_field(name, a)
        want = a.astype(np.float32).astype(np.float64) if precision and name != "density0" else a
        assert np.array_equal(ch.field(name), want), name
    ch.close()


def test_summaries_of_each_deck_of_an_ensemble():
    ds = [decks.to_deck(decks.shock(n, n + 1, n + 2, 12, summary_frequency=3)) for n in (8, 11, 9)]
    e = C.Ensemble(ds)
    e.run()
    for i, d in enumerate(ds):
        ch = C.Chunk(d)
        ch.run()
        got, steps = e.deck_summaries(i)
        want, wsteps = ch.summaries()
        assert np.array_equal(steps, wsteps)
        np.testing.assert_allclose(got, want, rtol=5e-16)  # both within one ulp of the exact sum
        short, s2 = e.deck_summaries(i, cap=2)
        assert np.array_equal(short, got[:2]) and np.array_equal(s2, steps[:2])
        ch.close()
    e.close()
