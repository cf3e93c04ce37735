"""The adjoint backprojection's two ways, quad space and patches in shared memory.

Which one runs shows in the context's memory: quad space takes 16 bytes a pixel
of scratch, patches none.  The rule is tried at both sides of each of its lines
(size and fill of the volume, pixels a voxel, the detector's border).  Patches
are right for any scan all the same: under a memory limit that leaves no room for
the scratch they run for the shapes where quad space is the faster one, and the
two ways' outputs differ by the order of FP32 sums alone: 1e-6 of the norm of the
sums of moduli, test_adjoint_patches.py's bar (a few thousand products a pixel
at the most, 2^-24 each)."""
import numpy as np
import pytest

from test_adjoint_patches import CASES

pytestmark = pytest.mark.gpu


def _adjoint(scan, vol, vox, tilt=0.0, nv=None, no_scratch=False):
    """The adjoint of nv views, that of the residuals' moduli, the scratch it took, and (volume, residuals, projections)."""
    import torch

    from jenhine_b200 import _lib
    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    views, u, v, pix = scan
    P = ScanGeometry(views, 500.0, 800.0, u, v, pix, pix, flex_shift_px=0.5, flex_tilt_deg=0.3, gantry_tilt_deg=tilt,
                     seed=6).ptms()
    e = FDKEngine(ScanConfig(views, 500.0, 800.0, u, v, pix), ReconConfig(*vol, vox, vox), P)
    gen = torch.Generator(device="cuda").manual_seed(8)
    q = torch.randn((views, v, u), generator=gen, device="cuda")
    e.bp_reset()
    e.bp_accumulate(q, 0)
    x = e.finalize(apply_ctnum=False)
    y = torch.randn(x.shape, generator=gen, device="cuda")
    before = e.device_bytes
    if no_scratch:
        e.set_option(_lib.OPT_DEVICE_MEMORY_LIMIT, before)
    qb = e.bp_adjoint(y, 0, nv or views, out=torch.full((nv or views, v, u), np.nan, device="cuda"))
    scratch = e.device_bytes - before
    moduli = e.bp_adjoint(y.abs(), 0, nv or views)
    return qb, moduli, scratch, (x, y, q)


@pytest.mark.parametrize("name", CASES)
def test_patches_equal_quad_space(name):
    views, u, v, pix, vol, vox, tilt = CASES[name]
    a, m, scratch, _ = _adjoint((views, u, v, pix), vol, vox, tilt)
    assert scratch == 16 * views * u * v
    b, _, none, _ = _adjoint((views, u, v, pix), vol, vox, tilt, no_scratch=True)
    assert none == 0
    assert (a - b).double().norm().item() <= 1e-6 * m.double().norm().item()


# (views, u, v, pixel), volume, voxel, tilt -> patches: voxels of 0.625 mm or more, 1.3 pixels a voxel unless stated
RULE = {
    "128": ((6, 280, 280, 0.77), (128, 128, 128), 0.625, 0.0, True),
    "128_tilted": ((6, 280, 280, 0.77), (128, 128, 128), 0.625, 2.0, True),
    "ragged": ((6, 280, 290, 0.77), (131, 125, 127), 0.625, 0.0, True),
    "too_few_blocks": ((6, 260, 260, 0.77), (120, 120, 120), 0.625, 0.0, False),
    "blocks_half_empty": ((6, 330, 150, 0.77), (176, 176, 48), 0.5, 0.0, False),
    "rows_shared": ((6, 220, 220, 1.0), (128, 128, 128), 0.625, 0.0, False),
    "patch_too_small": ((6, 360, 360, 0.6), (128, 128, 128), 0.625, 0.0, False),
    "across_the_border": ((6, 280, 150, 0.77), (128, 128, 128), 0.625, 0.0, False),
}


@pytest.mark.parametrize("name", RULE)
def test_rule(name):
    scan, vol, vox, tilt, patches = RULE[name]
    qb, m, scratch, (x, y, q) = _adjoint(scan, vol, vox, tilt)
    assert (scratch == 0) == patches
    import torch
    seen = torch.isfinite(x)
    x, y = torch.nan_to_num(x), y * seen
    lhs, rhs = (x.double() * y.double()).sum().item(), (q.double() * qb.double()).sum().item()
    assert abs(lhs - rhs) <= 1e-6 * x.double().norm().item() * y.double().norm().item()
    other = _adjoint(scan, vol, vox, tilt, no_scratch=True)[0]
    assert (qb - other).double().norm().item() <= 1e-6 * m.double().norm().item()
    # fewer views of the same scan, from the scratch of more
    sub = _adjoint(scan, vol, vox, tilt, nv=2)[0]
    assert (qb[:2] - sub).double().norm().item() <= 1e-6 * m[:2].double().norm().item()


def test_a_captured_call_outlives_larger_ones():
    """Quad space captured with its scratch in place, then a call of more views: the
    graph's scratch stays.  Captured before there is any, patches run."""
    import torch

    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    views, u, v = 12, 60, 50
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        e = FDKEngine(ScanConfig(views, 500.0, 800.0, u, v, 1.0), ReconConfig(20, 20, 16, 1.0, 1.0),
                      ScanGeometry(views, 500.0, 800.0, u, v, 1.0, 1.0).ptms(), stream=s.cuda_stream)
        e.bp_reset()
        e.bp_accumulate(torch.ones((views, v, u), device="cuda"), 0)
        y = torch.randn((16, 20, 20), device="cuda")
        outs, graphs = [torch.empty((2, v, u), device="cuda") for _ in range(2)], []
        held = []
        for out in outs:
            torch.cuda.synchronize()
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1], stream=s):
                e.bp_adjoint(y, 0, 2, out=out)
            torch.cuda.synchronize()
            held.append(e.device_bytes)
            want = e.bp_adjoint(y, 0, 2)       # after the first capture: makes the scratch
        assert held[1] == held[0] + 2 * 16 * u * v
        whole = e.bp_adjoint(y)
        for g, out in zip(graphs, outs):
            out.fill_(np.nan)
            g.replay()
            torch.cuda.synchronize()
            bar = 1e-6 * e.bp_adjoint(y.abs(), 0, 2).double().norm().item()
            for other in (want, whole[:2]):
                assert (out - other).double().norm().item() <= bar
    torch.cuda.synchronize()
