"""The launch for frames of more than 4 GB of records, on small frames against the
ordinary one: tests/cuda/wide_check.cu, linked with libjfdk.so."""
import os

import pytest

from conftest import ROOT
from test_quotient import build_and_run

pytestmark = pytest.mark.gpu


def test_wide_launches_equal_ordinary_ones(tmp_path):
    lib = os.path.join(ROOT, "jenhine_b200", "libjfdk.so")
    out = build_and_run("wide_check", tmp_path, lib, "-Xlinker", "-rpath=" + os.path.dirname(lib))
    assert "45 launches, 0 differ" in out
