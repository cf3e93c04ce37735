"""The autotuner and the views per chunk: the default is among what it times, it
leaves the option alone where it times nothing (compositing), it finds its answers
again, and the default can be had back."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

MAKE = f"""
import sys
sys.path.insert(0, {ROOT!r})
from jenhine_b200 import _lib
from jenhine_b200.fdk import FDKEngine, ReconConfig, ScanConfig
from jenhine_b200.phantom import ScanGeometry
def engine(views, u, v, offset=False):
    P = ScanGeometry(views, 500.0, 800.0, u, v, 1.0, 1.0, offset_u_px=u / 3.0 if offset else 0.0).ptms()
    scan = ScanConfig(views, 500.0, 800.0, u, v, 1.0)
    if offset:
        scan.filter_input_width, scan.detector_on_right = 2 * u, True
    return FDKEngine(scan, ReconConfig(16, 16, 16, 1.0, 1.0), P)
def chunk(e):
    return e.get_option(_lib.OPT_VIEW_CHUNK)
"""


def _child(code, cache):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    r = subprocess.run([sys.executable, "-c", MAKE + code], env=dict(os.environ, JFDK_AUTOTUNE_CACHE=str(cache)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return cache.read_text().splitlines() if cache.exists() else []


def test_the_default_is_a_candidate_and_can_be_had_back(tmp_path):
    lines = _child("""
e = engine(300, 96, 64)
usual = chunk(e)
assert usual > 64, usual
e.autotune()
assert chunk(e) in (usual, 16, 32, 64)
tuned = chunk(e)
f = engine(300, 96, 64)
f.autotune()                       # answered from the cache
assert chunk(f) == tuned
for n in (5, 0):
    f.set_option(_lib.OPT_VIEW_CHUNK, n)
    assert chunk(f) == (n or usual)
for bad in (-1, 4097):
    try:
        f.set_option(_lib.OPT_VIEW_CHUNK, bad)
    except _lib.JfdkError:
        continue
    raise SystemExit("accepted")
""", tmp_path / "t.txt")
    assert len(lines) == 1 and lines[0].split()[2] in ("0", "16", "32", "64"), lines


def test_a_default_from_the_file(tmp_path):
    cache = tmp_path / "t.txt"
    key = _child("engine(300, 96, 64).autotune()", cache)[0].split()[0]
    cache.write_text(f"{key} 8 0 4\n")
    lines = _child("""
e = engine(300, 96, 64)
usual = chunk(e)
e.set_option(_lib.OPT_VIEW_CHUNK, 7)
e.autotune()
assert chunk(e) == usual and e.tile_depth == 8
""", cache)
    assert lines == [f"{key} 8 0 4"]


def test_compositing_leaves_the_option(tmp_path):
    _child("""
for n in (0, 7):
    e = engine(60, 96, 48, offset=True)
    usual = chunk(e)
    assert usual > 32, usual
    e.set_option(_lib.OPT_VIEW_CHUNK, n)
    e.autotune(force=True)
    assert chunk(e) == (n or usual)
    e.autotune()
    assert chunk(e) == (n or usual)
""", tmp_path / "t.txt")
