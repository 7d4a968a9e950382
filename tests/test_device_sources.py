"""What the device code takes for granted about its tables and rules, checked by the compiler -- no GPU.

Each check is a small translation unit over the library's own headers that nvcc must accept.
"""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _compiles(tmp_path, text):
    from ifgf2d_gb300 import build
    src = tmp_path / "check.cu"
    src.write_text(text)
    r = subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", os.path.join(ROOT, "ifgf2d_gb300", "csrc"), "-c", str(src),
                        "-o", str(tmp_path / "check.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


def test_green_table_has_the_alignment_of_its_loads(tmp_path):
    """The table of the fixed-point Green values is read 16 bytes at a time: its declared alignment says so."""
    _compiles(tmp_path, """
#include "green_fx.cuh"
#include <type_traits>
using namespace ifgf;
using namespace ifgf::gx;
using Element = std::remove_all_extents_t<decltype(gx_table)>;
static_assert(alignof(Element) >= 16 && sizeof(Element) % 16 == 0, "16-byte loads");
""")


def test_orthogonalisation_work_grows_with_the_length(tmp_path):
    """Each block of the Gram-Schmidt update (64 rows) adds a bounded number of partial dots of a column."""
    _compiles(tmp_path, """
#include "ifgf2d_kernels.cuh"
using namespace ifgf;
static_assert(dot_block_terms(200) == 1 && dot_block_terms(65536) == 32, "few chunks: by the blocks");
static_assert(dot_block_terms(65537) == 1 && dot_block_terms(1 << 19) == 1 && dot_block_terms(1ll << 32) == 1, "more: added up once");
""")


def test_cosine_and_sine_coefficients():
    """The constants of cos_sin are the power series it names."""
    mp = pytest.importorskip("mpmath")
    mp.mp.dps = 40
    text = open(os.path.join(ROOT, "ifgf2d_gb300", "csrc", "green_fx.cuh")).read()
    body = re.search(r"void cos_sin\(.*?\n}\n", text, re.S)[0]
    cos, sin = body.split("const int v5")
    for part, odd, tail, scale in ((cos, 0, 6, 50), (sin, 1, 5, 47)):
        c = [(-1) ** j * (mp.pi / 2) ** (2 * j + odd) / mp.factorial(2 * j + odd) for j in range(tail + 5)]
        for j in range(tail):
            assert f"0x{int(mp.nint(abs(c[j]) * 2 ** 62)):x}ll" in part, j
        assert str(int(mp.nint(abs(c[tail]) * 2 ** scale))) in part
        floats = [float(v) for v in re.findall(r"-?\d+\.\d+(?=[f)])", part)]
        for j in range(tail + 1, tail + 4 + odd):
            assert min(abs(v - float(c[j] * 2 ** scale)) for v in floats) < 1e-6 * abs(float(c[j] * 2 ** scale)), j
