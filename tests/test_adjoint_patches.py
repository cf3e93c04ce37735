"""The adjoint backprojection's patches in shared memory, by dot products with
the forward, where they can go wrong: slices less than a row apart (additions
by shared-memory reductions), much more than a row apart (patches that do not
hold the block), blocks across the detector's border and on its last column,
volumes that fill no block, tilted orbits.  <A x, y> = <x, A^T y> on signed random
vectors to 1e-6 of |A x| |y| (test_adjoint.py's bar: both sides are FP32 sums of
a few thousand products in any order, 2^-24 each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "rows_apart": (20, 96, 80, 1.0, (24, 24, 40), 0.9, 0.0),
    "rows_shared": (20, 160, 120, 0.5, (40, 40, 70), 0.15, 0.0),
    "one_row": (20, 128, 96, 0.6, (33, 17, 35), 0.375, 0.0),
    "large_voxels": (12, 300, 280, 0.3, (20, 20, 34), 2.5, 0.0),
    "across_the_border": (20, 64, 40, 1.0, (50, 45, 33), 1.0, 0.0),
    "ragged": (7, 33, 17, 2.0, (13, 37, 5), 2.0, 0.0),
    "tilted": (20, 96, 80, 1.0, (24, 31, 40), 0.9, 3.0),
    "one_slice": (9, 40, 3, 1.0, (9, 9, 1), 0.7, 0.0),
}


@pytest.mark.parametrize("name", CASES)
def test_dot_product(name):
    import torch

    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    views, u, v, pix, vol, vox, tilt = CASES[name]
    P = ScanGeometry(views, 500.0, 800.0, u, v, pix, pix, flex_shift_px=0.5, flex_tilt_deg=0.3, gantry_tilt_deg=tilt,
                     seed=6).ptms()
    e = FDKEngine(ScanConfig(views, 500.0, 800.0, u, v, pix), ReconConfig(*vol, vox, vox), P)
    gen = torch.Generator(device="cuda").manual_seed(8)
    q = torch.randn((views, v, u), generator=gen, device="cuda")
    e.bp_reset()
    e.bp_accumulate(q, 0)
    x = e.finalize(apply_ctnum=False)
    seen = torch.isfinite(x)
    assert seen.any()
    x = torch.nan_to_num(x)
    y = torch.randn(x.shape, generator=gen, device="cuda") * seen
    qb = torch.full_like(q, np.nan)
    for v0 in range(0, views, 8):
        n = min(8, views - v0)
        e.bp_adjoint(y, v0, n, out=qb[v0:v0 + n])
    lhs, rhs = (x.double() * y.double()).sum().item(), (q.double() * qb.double()).sum().item()
    assert abs(lhs - rhs) <= 1e-6 * x.double().norm().item() * y.double().norm().item()


def test_zero_residual_gives_zero():
    import torch

    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    P = ScanGeometry(6, 500.0, 800.0, 32, 24, 2.0, 2.0).ptms()
    e = FDKEngine(ScanConfig(6, 500.0, 800.0, 32, 24, 2.0), ReconConfig(8, 8, 8, 2.0, 2.0), P)
    e.bp_reset()
    e.bp_accumulate(torch.ones((6, 24, 32), device="cuda"), 0)
    qb = torch.full((6, 24, 32), np.nan, device="cuda")
    e.bp_adjoint(torch.zeros((8, 8, 8), device="cuda"), 0, 6, out=qb)
    assert (qb == 0).all()
