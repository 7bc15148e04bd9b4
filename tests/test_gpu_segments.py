"""Staged marches whose segments end unevenly.

The planes a staged block marches follow from the launch's tiles and planes, so
the first, last and shortest segments fall on other planes as a grid grows: one
plane per block on the smallest grids, up to 32 on the largest."""
import numpy as np
import pytest
import torch

import cloverleaf3d_ref_b200 as C
import decks
import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (33, 9, 5), (31, 8, 61), (64, 65, 33), (40, 130, 97), (130, 40, 67)])
def test_native_and_dropin_bitwise_over_segments(nx, ny, nz):
    d = decks.shock(nx, ny, nz, 5, states=decks.MIXED_STATES)
    ref = O.run(d, want_fields=True)
    ch = C.Chunk(decks.to_deck(d))
    assert ch.use_tma(True)
    di = C.DropIn(decks.to_deck(d))
    for run in (ch, di):
        assert run.run() == ref["steps"]
        assert np.array_equal(run.dt_history(), ref["dt"])
        for name, want in ref["fields"].items():
            assert np.array_equal(run.field(name), want), name
        run.close()
    # FP32 storage: staged against register forms
    out = []
    for tma in (True, False):
        ch = C.Chunk(decks.to_deck(d), C.PRECISION_MIXED)
        assert ch.use_tma(tma) == tma
        ch.run()
        out.append([ch.field(n) for n in C.FIELD_NAMES])
        ch.close()
    for a, b, name in zip(*out, C.FIELD_NAMES):
        assert np.array_equal(a, b), name


@pytest.mark.parametrize("precision", [C.PRECISION_FP64, C.PRECISION_MIXED])
@pytest.mark.parametrize("graphs", [True, False])
def test_ensemble_staged_and_register_forms(precision, graphs):
    """Decks around the tiles' and warps' edges, side by side: staged and register forms, and each deck alone."""
    sizes = [(3, 3, 3), (33, 9, 5), (31, 8, 61), (32, 32, 32), (29, 17, 40), (64, 3, 12), (62, 31, 7)]
    ds = [decks.to_deck(decks.shock(*n, 6, states=decks.MIXED_STATES)) for n in sizes]
    runs = []
    for tma in (True, False):
        e = C.Ensemble(ds, precision)
        e.use_graphs(graphs)
        assert e.use_tma(tma) == tma
        e.run()
        runs.append(e)
    for i, d in enumerate(ds):
        ch = C.Chunk(d, precision)
        ch.run()
        assert all(e.deck_status(i) == 0 for e in runs)
        assert all(np.array_equal(e.deck_dt_history(i), ch.dt_history()) for e in runs)
        for name in C.FIELD_NAMES:
            want = ch.field(name)
            assert all(np.array_equal(e.deck_field(i, name), want) for e in runs), (i, name)
        ch.close()
    for e in runs:
        e.close()


ROWS = (24, 25, 26, 27, 28, 29, 58, 59, 91)


def test_mixed_forms_agree_at_every_row_length():
    """Flow along x up to the far wall, rows that end at each place in their pitch: staged and register forms of a
    chunk, and of ensembles, whichever decks share them."""
    ds = [decks.to_deck(decks.shock(nx, 9, 6, 14, states=decks.MIXED_STATES)) for nx in ROWS]
    want = []
    for d in ds:
        out = []
        for tma in (True, False):
            ch = C.Chunk(d, C.PRECISION_MIXED)
            assert ch.use_tma(tma) == tma
            ch.run()
            assert ch.status == 0
            out.append({n: ch.field(n) for n in C.FIELD_NAMES})
            ch.close()
        want.append(out[1])
        for n in C.FIELD_NAMES:
            assert np.array_equal(out[0][n], out[1][n]), (d.s.x_cells, n)
    for tma in (True, False):
        for part in (ds, ds[2:4]):
            e = C.Ensemble(part, C.PRECISION_MIXED)
            assert e.use_tma(tma) == tma
            e.run()
            for i, d in enumerate(part):
                ref = want[ds.index(d)]
                for n in C.FIELD_NAMES:
                    assert np.array_equal(e.deck_field(i, n), ref[n]), (d.s.x_cells, n, tma)
            e.close()


@pytest.mark.parametrize("precision", [C.PRECISION_FP64, C.PRECISION_MIXED])
def test_ensembles_one_after_another(precision):
    """Ensembles of other sizes and numbers of decks, whose device memory lies where the last one's lay: each deck of
    each against itself alone."""
    sizes = [(40, 33, 12), (33, 40, 9), (64, 20, 7), (31, 31, 31), (70, 16, 10), (20, 48, 24)]
    ds = [decks.to_deck(decks.shock(*n, 5, states=decks.MIXED_STATES)) for n in sizes]
    want = []
    for d in ds:
        ch = C.Chunk(d, precision)
        ch.run()
        want.append([ch.field(n) for n in C.FIELD_NAMES])
        ch.close()
    for r in range(12):
        part = [(r + i * (1 + r % 2)) % 6 for i in range(1 + r % 4)]
        e = C.Ensemble([ds[i] for i in part], precision)
        assert e.use_tma(True)
        e.run()
        for at, i in enumerate(part):
            assert e.deck_status(at) == 0
            for n, w in zip(C.FIELD_NAMES, want[i]):
                assert np.array_equal(e.deck_field(at, n), w), (r, sizes[i], n)
        e.close()


def test_no_room_for_the_maps():
    """An ensemble whose tensor maps find no room on the device says so, keeps the register forms for every launch and
    runs on; with room again it takes the staged forms."""
    ds = [decks.to_deck(decks.shock(8 + i % 5, 8 + i % 3, 9, 12, states=decks.MIXED_STATES)) for i in range(400)]
    e = C.Ensemble(ds)  # too small for the staged forms by default
    e.step(4)
    e.sync()
    ballast, size = [], 1 << 34
    try:
        while size >= 1 << 18:
            try:
                ballast.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                size //= 2
        assert not e.use_tma(True)
    finally:
        ballast.clear()
        torch.cuda.empty_cache()
    e.step(3)
    assert e.use_tma(True)
    e.step(5)
    for i in range(0, 400, 41):
        ch = C.Chunk(ds[i])
        ch.step(12)
        assert np.array_equal(e.deck_dt_history(i), ch.dt_history())
        for n in C.FIELD_NAMES:
            assert np.array_equal(e.deck_field(i, n), ch.field(n)), (i, n)
        ch.close()
    e.close()
