"""The kernels of lines.cuh hold their fourteen radices once each: what a process loads
at its first call.  Copies for every call site made general.cu's object 8 MB."""
import os

import pytest

from conftest import PKG_NAME, ROOT

LIMIT = 5 << 20


@pytest.mark.parametrize("name", ["general", "resample"])
def test_object_size(name):
    obj = os.path.join(ROOT, PKG_NAME, "csrc", "_build", name + ".o")
    if not os.path.exists(obj):
        pytest.skip("not built here")
    assert os.path.getsize(obj) < LIMIT
