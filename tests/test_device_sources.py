"""What the device code takes for granted about its tables and rules, checked by the compiler -- no GPU.

Each check is a small translation unit over the library's own headers that nvcc must accept.
"""
import os
import subprocess

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
