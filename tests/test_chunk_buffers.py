"""The filter stage's buffers: the first call of a context makes room for every
later one, so that a captured graph's pointers stay valid and a capture has
nothing to allocate, whichever entry point came first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(form="fp32", views=48, u=40, v=24, stream=None):
    import torch

    from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
    from jenhine_b200.phantom import ScanGeometry
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    P = ScanGeometry(views, 500.0, 800.0, u, v, 2.0, 2.0, seed=2).ptms()
    e = FDKEngine(ScanConfig(views, 500.0, 800.0, u, v, 2.0), ReconConfig(16, 16, 12, 2.0, 2.0), P, precision=form,
                  stream=stream)
    raw = np.random.default_rng(3).integers(200, 60000, (views, v, u), dtype=np.uint16)
    return e, raw, torch.from_numpy(raw).cuda()


@pytest.mark.parametrize("form", ["fp32", "mixed"])
def test_the_first_call_makes_room_for_all(form):
    e, host, raw = _engine(form)
    e.filter_raw(raw, 0, 1)
    held = e.device_bytes
    e.filter_raw(raw, 0, raw.shape[0])
    assert e.device_bytes == held
    e, host, raw = _engine(form)
    want = e.reconstruct_host(host)
    held = e.device_bytes
    np.testing.assert_array_equal(e.reconstruct(raw).cpu().numpy(), want)
    e.filter_raw(raw, 0, raw.shape[0])
    assert e.device_bytes == held


def test_a_captured_call_outlives_larger_ones():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        e, _, raw = _engine(stream=s.cuda_stream)
        torch.cuda.synchronize()
        want = e.filter_raw(raw, 0, raw.shape[0]).clone()   # another context's answer
        torch.cuda.synchronize()
        e, _, raw = _engine(stream=s.cuda_stream)
        torch.cuda.synchronize()
        e.filter_raw(raw, 0, 1)
        out = torch.empty_like(want)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            e.filter_raw(raw, 0, raw.shape[0], out=out)
        e.reconstruct(raw)
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


@pytest.mark.parametrize("views,u,v", [(700, 256, 256), (400, 33, 256), (90, 64, 64), (40, 768, 768)])
def test_a_chunk_is_bounded_and_dealt_evenly(views, u, v):
    """At most the bytes of 32 frames of 768 x 768 (8 a pixel, rows of weighted samples
    padded to 64), and chunks that differ by less than their number."""
    import torch

    from jenhine_b200 import _lib
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    e, _, raw = _engine(views=views, u=u, v=v)
    chunk = e.get_option(_lib.OPT_VIEW_CHUNK)
    last = (views - 1) % chunk + 1
    assert chunk == min(views, 32) or chunk - last < -(-views // chunk)
    before = e.device_bytes
    e.reconstruct(raw)
    held = e.device_bytes - before - 16 * views * u * v - 4 * 16 * 16 * 12
    row = 4 * (-(-u // 64) * 64 + u)
    assert held <= chunk * v * (row + 8) + 4096
    assert chunk == min(views, 32) or chunk * v * row <= 32 * 768 * 768 * 8


def test_another_product_in_the_same_buffers():
    """The parts of the weighted rows take 4 or 8 bytes a sample: a context that changes
    its ramp product gives what one with that product from the start gives."""
    import torch

    from jenhine_b200 import _lib
    e, _, raw = _engine(u=70)
    want = {}
    for product in (_lib.RAMP_I8X14, _lib.RAMP_TF32X3, _lib.RAMP_FP16X3, _lib.RAMP_FP32_SIMT, _lib.RAMP_BF16X3):
        f, _, _ = _engine(u=70)
        f.set_option(_lib.OPT_RAMP_PRODUCT, product)
        want[product] = f.reconstruct(raw)
    for product in (*want, *reversed(want)):
        e.set_option(_lib.OPT_RAMP_PRODUCT, product)
        assert torch.equal(e.reconstruct(raw).nan_to_num(1e30), want[product].nan_to_num(1e30)), product


@pytest.mark.parametrize("later", ["more_views", "another_product", "adjoint"])
def test_buffers_a_graph_names_are_kept(later):
    """A captured filter call, then one that needs larger buffers: more views, rows of
    two TF32 parts, the filter adjoint of many views."""
    import torch

    from jenhine_b200 import _lib
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        e, _, raw = _engine(stream=s.cuda_stream)
        frames = e.preprocess(raw)
        want = e.filter(frames[:2])
        out = torch.empty_like(want)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            e.filter(frames[:2], out=out)
        torch.cuda.synchronize()
        held = e.device_bytes
        if later == "more_views":
            e.filter(frames)
        elif later == "another_product":
            e.set_option(_lib.OPT_RAMP_PRODUCT, _lib.RAMP_TF32X3)
            e.filter(frames[:2])
        else:
            e.filter_adjoint(frames)
        assert e.device_bytes > held
        junk = torch.full((1 << 22,), np.nan, device="cuda")
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and junk.isnan().all()
