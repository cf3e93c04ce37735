"""The adjoint backprojection's bilinear weights, by one voxel alone in front of
a detector where its place is known exactly (matrices with W = 1, the voxel 2^-9
of a pixel from the next column and 2^-10 of one from the next row).  Each of its
four pixels is rt (1 - fx or fx) (1 - fy or fy) times the taper: three roundings of
2^-24 each (1 - f is exact), so the ratio of two pixels, their tapers divided out
in FP64, is that of the weights to six, large and small ones alike.  An infinite
residual makes all four infinite and nothing NaN.  A volume large enough for the
patches in shared memory, and a small one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VIEWS, DET = 4, 200


def _adjoint_of_one_voxel(n, value):
    import torch

    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    e = FDKEngine(ScanConfig(VIEWS, 500.0, 800.0, DET, DET, 1.0), ReconConfig(n, n, n, 1.0, 1.0),
                  ScanGeometry(VIEWS, 500.0, 800.0, DET, DET, 1.0, 1.0).ptms())
    # u = x + 100 - 2^-9 + 0.5, v = 1.25 z + 99.875 - 2^-10 + 0.5: at (0.5, 0.5, 0.5) the places 101 less those
    P = np.array([[1, 0, 0, 100 - 2.0 ** -9], [0, 0, 1.25, 99.875 - 2.0 ** -10], [0, 0, 0, 1]], np.float32)
    e.set_bp_geometry(np.tile(P.reshape(1, 12), (VIEWS, 1)))
    e.bp_reset()
    e.bp_accumulate(torch.ones((VIEWS, DET, DET), device="cuda"), 0)
    y = torch.zeros((n, n, n), device="cuda")
    y[n // 2, n // 2, n // 2] = value
    return e.bp_adjoint(y).cpu().numpy(), e.uweights()


@pytest.mark.parametrize("n", [128, 24])
def test_small_weights_are_as_exact_as_large_ones(n):
    q, w = _adjoint_of_one_voxel(n, 1.0 / 3.0)
    f = np.array([1 - 2.0 ** -9, 1 - 2.0 ** -10])
    want = np.outer([1 - f[1], f[1]], [1 - f[0], f[0]])
    for view in range(VIEWS):
        rows, cols = np.nonzero(q[view])
        assert set(zip(rows, cols)) == {(100, 100), (100, 101), (101, 100), (101, 101)}
        got = q[view, 100:102, 100:102].astype(np.float64) / w[view, 100:102].astype(np.float64)
        ratio = (got / got[1, 1]) / (want / want[1, 1])
        assert np.abs(ratio - 1).max() <= 6.0 * 2.0 ** -24 * 1.001


@pytest.mark.parametrize("n", [128, 24])
def test_an_infinite_residual_stays_infinite(n):
    q, _ = _adjoint_of_one_voxel(n, np.inf)
    want = np.zeros_like(q)
    want[:, 100:102, 100:102] = np.inf
    np.testing.assert_array_equal(q, want)
