"""Fields written and read back: one piece, and several pieces of whole planes."""
from concurrent.futures import ThreadPoolExecutor

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


@pytest.mark.parametrize("precision", [C.PRECISION_FP64, C.PRECISION_MIXED])
def test_threads_read_one_chunk(precision):
    """Every field of a chunk (each in several pieces), and of an ensemble's decks, read by eight threads at once."""
    n = (150, 190, 190)  # 45 MB of doubles a field
    ch = C.Chunk(decks.to_deck(decks.shock(*n, 4)), precision)
    rng = np.random.default_rng(11)
    for name in C.FIELD_NAMES:
        ch.set_field(name, np.asfortranarray(rng.standard_normal(C.field_shape(name, *n), dtype=np.float32)
                                             .astype(np.float64)))
    e = C.Ensemble([decks.to_deck(decks.shock(*s, 4)) for s in ((8, 9, 10), (70, 61, 50), (33, 20, 90))], precision)
    e.run()
    with ThreadPoolExecutor(8) as pool:
        got = list(pool.map(ch.field, C.FIELD_NAMES))
        jobs = [(i, name) for _ in range(4) for name in C.FIELD_NAMES for i in range(3)]
        parts = list(pool.map(lambda job: e.deck_field(*job), jobs))
    for name, a in zip(C.FIELD_NAMES, got):
        assert np.array_equal(a, ch.field(name)), name
    for (i, name), a in zip(jobs, parts):
        assert np.array_equal(a, e.deck_field(i, name)), (i, name)
    ch.close()
    e.close()
