"""The bulk-copy-fed line passes against the per-thread-load line passes.

The engine runs its row and column passes either with kernels whose threads load the wave
straight from global memory, or with kernels that stage each item's lines in shared memory through
the copy engine and keep the transmission rows resident; MTB_PIPE pins the choice (bit 0 rows,
bit 1 columns), otherwise the engine's autotuner picks the faster per shape. All variants compute
the same transforms with the same rounding, so the waves are bit-identical; the FP64 detector sums
are too where both variants use tiles of the same width, and agree to FP64 rounding (1e-13
relative) where they do not (1024: 8-column tiles in the bulk-copy-fed pass, 16 in the other; the
per-tile partials are then added in a different order). Cases cover:
several line groups per CTA in the row pass (a change of transmission rows inside a CTA), probe
counts that are and are not multiples of the row-pass unit, and the column pass's detector
partials.
"""
import numpy as np
import pytest

from multem_b200 import api, specimens

pytestmark = pytest.mark.gpu



def _stem(p, pipe, monkeypatch):
    monkeypatch.setenv("MTB_PIPE", str(pipe))
    e = api.Engine(p)
    r = e.run()
    e.close()
    return np.stack([np.stack(d["image_tot"]) for d in r["data"]])


@pytest.mark.parametrize("nx,ns", [(512, 4), (512, 3), (64, 4), (128, 4), (256, 4), (384, 4), (1024, 4), (2048, 4)])
def test_stem_pipelined_matches_per_thread_kernels(nx, ns, monkeypatch):
    p = specimens.stem_srtio3(nx=nx, ny=nx, na=4, nb=4, nc=6, ns=ns, nconf=1, seed=3)
    ref = _stem(p, 0, monkeypatch)
    exact = nx < 1024
    for pipe in (1, 2, 3):
        img = _stem(p, pipe, monkeypatch)
        assert img.shape == ref.shape
        if exact:
            np.testing.assert_array_equal(img, ref, err_msg=f"MTB_PIPE={pipe}")
        else:
            np.testing.assert_allclose(img, ref, rtol=1e-13, atol=0, err_msg=f"MTB_PIPE={pipe}")
    monkeypatch.delenv("MTB_PIPE")
    e = api.Engine(p)
    r = e.run()
    e.close()
    np.testing.assert_allclose(np.stack([np.stack(d["image_tot"]) for d in r["data"]]), ref, rtol=0 if exact else 1e-13,
                               atol=0)


@pytest.mark.parametrize("nx", [128, 256, 384, 512, 1024])
def test_exit_wave_pipelined_matches_per_thread_kernels(nx, monkeypatch):
    p = specimens.hrtem_si001(nx=nx, ny=nx, na=4, nb=4, nc=6)
    out = {}
    for pipe in (0, 3):
        monkeypatch.setenv("MTB_PIPE", str(pipe))
        r = api.ilc_multem(None, p)
        out[pipe] = np.stack([np.asarray(d["psi_coh"]) for d in r["data"]])
    np.testing.assert_array_equal(out[3], out[0])


# the lengths that have an alternative shape; probes so that every group of every CTA takes several tiles or units, with and
# without a remainder (columns of 256: 32 tiles of 8 columns per probe over 148 CTAs of six groups; rows of 256 take
# whole groups of eight probes), and other line lengths in the other direction, which set the strides
@pytest.mark.parametrize("nx,ny,shape,ns", [(256, 256, 1 << 2, 4), (256, 256, 1 << 2, 8), (256, 256, 1 << 2, 9), (256, 512, 1 << 2, 7),
                                            (256, 64, 1 << 2, 16), (512, 512, 1 << 2, 4), (512, 512, 1 << 2, 7), (512, 128, 1 << 2, 9),
                                            (512, 1024, 1 << 2, 5), (256, 256, 2, 8), (256, 256, 2, 4), (128, 256, 2, 8),
                                            (2048, 2048, 2, 4), (64, 2048, 2, 4), (384, 384, 2 << 2, 4), (384, 384, 2 << 2, 7),
                                            (384, 256, 2 << 2, 8), (1024, 1024, 2 << 2, 4), (1024, 256, 2 << 2, 5)])
def test_alternative_pipeline_shapes_match(nx, ny, shape, ns, monkeypatch):
    """The autotuner's alternative pipeline shapes of the slice step (columns, bits 2-3: 1 owned by warps at 256 and 512, 2
    early issue with full exchange buffers at 384 and 1024; rows, bits 0-1: 2 the same at 256 and 2048) give the
    waves of the per-thread-load kernels bit for bit."""
    p = specimens.stem_srtio3(nx=nx, ny=ny, na=4, nb=4, nc=6 if max(nx, ny) < 2048 else 2, ns=ns, nconf=1, seed=3)
    monkeypatch.setenv("MTB_BATCH", str(ns * ns))
    ref = _stem(p, 0, monkeypatch)
    monkeypatch.setenv("MTB_SHAPE", str(shape))
    monkeypatch.setenv("MTB_PIPE", "3")
    e = api.Engine(p)
    e.run()
    t = e.tuning()
    e.close()
    assert t["probes_per_launch"] == ns * ns and (t["cols"] == 1 + (shape >> 2) if shape > 3 else t["rows"] == 1 + shape), t
    img = _stem(p, 3, monkeypatch)
    monkeypatch.delenv("MTB_SHAPE")
    if nx == 1024:
        np.testing.assert_allclose(img, ref, rtol=1e-13, atol=0)
    else:
        np.testing.assert_array_equal(img, ref)


def test_autotuner_reports_its_choice():
    p = specimens.stem_srtio3(nx=512, ny=512, na=8, nb=8, nc=3, ns=16, nconf=1, seed=3)
    e = api.Engine(p)
    e.run()
    t = e.tuning()
    e.close()
    assert t["rows"] in (0, 1, 2, 3) and t["cols"] in (0, 1, 2, 3)
    assert t["probes_per_launch"] in (128, 256)


ROWS = {64: (0, 1), 128: (0, 1), 256: (0, 1, 3), 384: (0, 1), 512: (0, 1), 1024: (0, 1), 2048: (0, 1, 3)}
COLS = {64: (0, 1), 128: (0, 1), 256: (0, 1, 2), 384: (0, 1, 3), 512: (0, 1, 2), 1024: (0, 1, 3), 2048: (0, 1)}


@pytest.mark.parametrize("nx,ny", [(64, 2048), (128, 64), (256, 1024), (384, 512), (512, 256), (1024, 384), (2048, 128)])
def test_only_variants_of_the_lengths_are_reported(nx, ny, monkeypatch):
    """The autotuner chooses, and mt_engine_tuning reports, variants that the line lengths have; one wave, or several with
    transmission functions of their own, have no bulk-copy-fed rows."""
    p = specimens.hrtem_si001(nx=nx, ny=ny, na=2, nb=2, nc=2)
    q = specimens.stem_srtio3(nx=nx, ny=ny, na=4, nb=4, nc=2, ns=4, nconf=1, seed=3)
    for spec, rows in ((p, (0,)), (q, ROWS[ny])):
        for pin in (None, "0", "5", "10"):
            if pin is None:
                monkeypatch.delenv("MTB_PIPE", raising=False)
            else:
                monkeypatch.setenv("MTB_PIPE", "3")
                monkeypatch.setenv("MTB_SHAPE", pin)
            e = api.Engine(spec)
            e.run()
            t = e.tuning()
            e.close()
            assert t["rows"] in rows and t["cols"] in COLS[nx], (pin, t)


def test_short_passes_are_tuned_too():
    """Columns of 1024 points are faster bulk-copy fed however few they are (1024 x 128, one wave: 17 us a slice
    with per-thread loads, 13 us)."""
    p = specimens.hrtem_si001(nx=1024, ny=128, na=2, nb=2, nc=4)
    e = api.Engine(p)
    e.run()
    t = e.tuning()
    e.close()
    assert t["cols"] in (1, 3)
