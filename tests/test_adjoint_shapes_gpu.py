"""The adjoint's replay over the level ranges whose launch shapes
test_adjoint_gpu's heights do not reach (33 to 64 and 129 to 256 levels), with
whole and partly filled blocks, and the edges of a column's warps: exact
derivatives of the sequential column, as there."""
import ctypes
import os
import subprocess

import pytest

import test_adjoint_pointwise as pointwise
from test_adjoint_gpu import _assert_exact, exact_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(5, 3, 33), (4, 4, 50), (5, 5, 64), (5, 3, 96)])
def test_exact(nx, ny, nz):
    _assert_exact(exact_check(nx, ny, nz, 150.0, 16))


@pytest.fixture(scope="module")
def tall_harness(tmp_path_factory):
    """The harness for columns of up to 256 levels."""
    tmp = tmp_path_factory.mktemp("tall")
    src = os.path.dirname(pointwise.SRC)
    for name in ("harness.cpp", "dual.h", "column.h"):
        text = open(os.path.join(src, name)).read()
        if name == "column.h":
            assert "constexpr int LMAX = 128;" in text
            text = text.replace("constexpr int LMAX = 128;", "constexpr int LMAX = 256;")
        (tmp / name).write_text(text)
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(tmp), "-I",
                        os.path.join(pointwise.ROOT, "pyshield_b200", "csrc"), str(tmp / "harness.cpp"), "-o",
                        str(tmp / "tall.so")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return ctypes.CDLL(str(tmp / "tall.so"))


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 129), (4, 2, 200), (3, 1, 256)])
def test_exact_tall(nx, ny, nz, tall_harness, monkeypatch):
    monkeypatch.setattr(pointwise, "build_harness", lambda: tall_harness)
    _assert_exact(exact_check(nx, ny, nz, 150.0, 16))
