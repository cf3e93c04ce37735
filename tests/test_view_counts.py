"""The backprojection at the lines of its launch rules: few views (tiles are not
sorted by where they lie, fewer registers), more views than the table of views to
pass over holds (4096), and numbers of tiles on both sides of where the tile depth
or the registers change.  Bit for bit the volumes of the persistent batch kernel,
which has none of these rules, and of the same views accumulated in other chunks."""
import numpy as np
import pytest

from test_view_loop import _scan

pytestmark = pytest.mark.gpu


def _persistent(e, raw, vol):
    import torch

    from jenhine_b200.fdk import FDKBatch
    out = torch.empty(tuple(vol[::-1]), device="cuda")
    FDKBatch([e], autotune=False, graph=False, schedule="persistent").run([raw], [out])
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _needs_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


@pytest.mark.parametrize("geo", ["ideal", "flex", "tilted"])
@pytest.mark.parametrize("form,zpt", [("fp32", 8), ("mixed", 8), ("mixed", 16)])
@pytest.mark.parametrize("views", [1, 2, 3, 4, 5, 6, 47, 48])
def test_few_views(geo, form, zpt, views):
    from jenhine_b200 import _lib
    _needs_gpu()
    if geo == "tilted" and views == 1:
        pytest.skip("the orbit's first view is not tilted")
    vol = (41, 77, 27)
    e, raw = _scan(geo, views, 96, 80, 1.0, form, vol, 1.3)
    e.set_option(_lib.OPT_BP_ZPT, zpt)
    got = e.reconstruct(raw).cpu().numpy()
    np.testing.assert_array_equal(got, _persistent(e, raw, vol))
    frames = e.filter_raw(raw, 0, views)
    chunked = []
    for n in {views, 1, 3, min(views, 6)}:
        e.bp_reset()
        for v0 in range(0, views, n):
            e.bp_accumulate(frames[v0:v0 + n], v0)
        chunked.append(e.finalize().cpu().numpy())
    for c in chunked[1:]:
        np.testing.assert_array_equal(c, chunked[0])
    if form == "fp32":
        np.testing.assert_array_equal(chunked[0], got)


# 4 x 32 columns a tile: 148 SMs hold 444 FP32 tiles in half a wave and 592 mixed ones in a wave of four CTAs
@pytest.mark.parametrize("form,slices", [("fp32", 104), ("fp32", 120), ("mixed", 144), ("mixed", 160)])
@pytest.mark.parametrize("geo", ["ideal", "flex", "tilted"])
def test_numbers_of_tiles(geo, form, slices):
    from jenhine_b200 import _lib
    _needs_gpu()
    vol = (64, 64, slices)
    e, raw = _scan(geo, 9, 120, 110, 1.0, form, vol, 0.5)
    got = e.reconstruct(raw).cpu().numpy()
    np.testing.assert_array_equal(got, _persistent(e, raw, vol))
    e.set_option(_lib.OPT_BP_ZPT, 8)
    np.testing.assert_array_equal(e.reconstruct(raw).cpu().numpy(), got)
    e.set_option(_lib.OPT_BP_WEIGHTS, 0)
    np.testing.assert_array_equal(e.reconstruct(raw).cpu().numpy(), got)
    frames = e.filter_raw(raw, 0, 9)
    e.bp_reset()
    for v0 in range(0, 9, 4):
        e.bp_accumulate(frames[v0:v0 + 4], v0)
    if form == "fp32":
        np.testing.assert_array_equal(e.finalize().cpu().numpy(), got)


@pytest.mark.parametrize("form", ["fp32", "mixed"])
def test_more_views_than_the_table_holds(form):
    from jenhine_b200 import _lib
    _needs_gpu()
    vol, views = (12, 40, 9), 4099
    e, raw = _scan("flex", views, 24, 16, 3.0, form, vol, 4.0)
    got = e.reconstruct(raw).cpu().numpy()
    assert np.isfinite(got).any()
    np.testing.assert_array_equal(got, _persistent(e, raw, vol))
    e.set_option(_lib.OPT_BP_WEIGHTS, 0)
    np.testing.assert_array_equal(e.reconstruct(raw).cpu().numpy(), got)
