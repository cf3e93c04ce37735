"""The exact int8 ramp product at widths on both sides of its K blocks (128
columns) and output tiles (64), where the digit planes that a block loads and
multiplies change, and at row counts around its 128-row tiles.

Against the FP64 filter of the oracle, on frames of white noise (the filtered
values are then as large as the weighted ones, nothing cancels): the rows are
rounded to FP32 once when weighted (2^-24 at most, 0.29 of it in the mean
square: 1.7e-8), the pre-weight, the operator's edge column and the result once
each, the fixed point is below 2^-31.  Four such roundings are 3.5e-8; the bar is
three times that, 1e-7, and a digit product left out is 2^-16 or more."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,rows", [(3, 5), (33, 17), (64, 128), (65, 129), (127, 3), (129, 64), (257, 43), (300, 31),
                                        (513, 10), (770, 9), (1025, 6), (1500, 5)])
def test_int8_product_at_the_edges_of_its_blocks(oracle, width, rows):
    import torch

    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    views, pix = 3, 150.0 / width
    g = ScanGeometry(views, 500.0, 800.0, width, rows, pix, pix, seed=3)
    P = g.ptms()
    e = FDKEngine(ScanConfig(views, 500.0, 800.0, width, rows, pix), ReconConfig(8, 8, 8, 1.0, 1.0), P)
    frames = np.random.default_rng(width).standard_normal((views, rows, width)).astype(np.float32)
    got = e.filter(torch.from_numpy(frames).cuda()).cpu().numpy()
    L = oracle.fft_length(width)
    H = oracle.filter_spectrum(L, g.half_sample_rate, 0.0, 0.0, [], [])
    want = oracle.filter_projections_f64(frames, P, H, 500.0)
    assert rel_l2(got, want) <= 1e-7


@pytest.mark.parametrize("u,rows", [(33, 17), (64, 40), (257, 9), (300, 8)])
def test_chunks_of_any_size_give_the_same_volume(u, rows):
    """The default chunk against single views and against chunks that leave a
    remainder, with rows that do and do not fill the packers' runs of eight."""
    import torch

    from jenhine_b200 import _lib
    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    views, pix = 37, 100.0 / u
    P = ScanGeometry(views, 500.0, 800.0, u, rows, pix, pix, seed=4).ptms()
    raw = torch.from_numpy(np.random.default_rng(1).integers(1, 65000, (views, rows, u), dtype=np.uint16)).cuda()
    for form in ("fp32", "mixed"):
        e = FDKEngine(ScanConfig(views, 500.0, 800.0, u, rows, pix), ReconConfig(16, 16, 6, 1.0, 1.0), P, precision=form)
        want = e.reconstruct(raw).cpu().numpy()
        assert e.get_option(_lib.OPT_VIEW_CHUNK) == views
        for chunk in (1, 5, 36):
            e.set_option(_lib.OPT_VIEW_CHUNK, chunk)
            np.testing.assert_array_equal(e.reconstruct(raw).cpu().numpy(), want)
        tight = FDKEngine(ScanConfig(views, 500.0, 800.0, u, rows, pix), ReconConfig(16, 16, 6, 1.0, 1.0), P, precision=form)
        tight.set_option(_lib.OPT_DEVICE_MEMORY_LIMIT, 1 << 34)
        assert tight.get_option(_lib.OPT_VIEW_CHUNK) == 32
        np.testing.assert_array_equal(tight.reconstruct(raw).cpu().numpy(), want)
