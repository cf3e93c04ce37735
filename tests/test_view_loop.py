"""The backprojection's view loops against the persistent batch kernel, which
keeps the loop with a range test for every sample, 64-bit record addresses and
no special case for ideal orbits: the same volumes bit for bit (NaN where no
view sees a voxel included), whatever mixture of tiles inside and across the
detector's border a scan gives, in both forms, for each way a sample's place
depends on the slice (ideal orbit, flexing gantry, tilted orbit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scan(geo, views, u, v, pix, form, vol, vox, **kw):
    import torch

    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    g = ScanGeometry(views, 500.0, 800.0, u, v, pix, pix, seed=11,
                     flex_shift_px=0.0 if geo == "ideal" else 0.5, flex_tilt_deg=0.0 if geo == "ideal" else 0.3,
                     gantry_tilt_deg=2.0 if geo == "tilted" else 0.0)
    P = g.ptms()
    assert (P[:, 10] != 0).any() == (geo == "tilted")
    assert (P[:, 2] != 0).any() == (geo != "ideal")
    scan = ScanConfig(views, 500.0, 800.0, u, v, pix)
    recon = ReconConfig(*vol, vox, vox)
    raw = torch.from_numpy(np.random.default_rng(5).integers(200, 60000, (views, v, u), dtype=np.uint16)).cuda()
    e = FDKEngine(scan, recon, P, precision=form, **kw)
    return e, raw


# all inside (small voxels), all kinds of tile, nothing but the border; ragged
# sizes; frames of more than 2^23 pixels (no float record index)
CASES = [(20, 96, 80, 1.0, (24, 64, 16), 0.6), (20, 96, 80, 1.0, (41, 77, 27), 1.3), (11, 33, 17, 2.0, (13, 37, 5), 2.5),
         (9, 4100, 2051, 0.03, (20, 40, 12), 1.5)]


@pytest.mark.parametrize("geo", ["ideal", "flex", "tilted"])
@pytest.mark.parametrize("form", ["fp32", "mixed"])
@pytest.mark.parametrize("case", CASES, ids=[f"{c[1]}x{c[2]}" + "x".join(map(str, c[4])) for c in CASES])
@pytest.mark.parametrize("zpt", [4, 8, 16])
def test_view_loops_equal_the_range_tested_loop(geo, form, case, zpt):
    import torch

    from jenhine_b200 import _lib
    from jenhine_b200.fdk import FDKBatch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    if form == "fp32" and zpt == 16:
        pytest.skip("the batch kernel has no 16-slice FP32 tiles")
    views, u, v, pix, vol, vox = case
    e, raw = _scan(geo, views, u, v, pix, form, vol, vox)
    e.set_option(_lib.OPT_BP_ZPT, zpt)
    got = e.reconstruct(raw).cpu().numpy()
    out = torch.empty(tuple(vol[::-1]), device="cuda")
    FDKBatch([e], autotune=False, graph=False, schedule="persistent").run([raw], [out])
    torch.cuda.synchronize()
    np.testing.assert_array_equal(got, out.cpu().numpy())
    # per-sample weights: the loops that load the taper too
    e.set_option(_lib.OPT_BP_WEIGHTS, 0)
    np.testing.assert_array_equal(e.reconstruct(raw).cpu().numpy(), got)


@pytest.mark.parametrize("geo", ["ideal", "flex", "tilted"])
def test_accumulated_views_equal_one_launch(geo):
    """FP32: chunks of views, each with its own tiles inside the detector."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    views, u, v, pix, vol, vox = CASES[1]
    e, raw = _scan(geo, views, u, v, pix, "fp32", vol, vox)
    want = e.reconstruct(raw).cpu().numpy()
    e.bp_reset()
    for v0 in range(0, views, 7):
        n = min(7, views - v0)
        e.bp_accumulate(e.filter_raw(raw, v0, n), v0)
    np.testing.assert_array_equal(e.finalize().cpu().numpy(), want)
